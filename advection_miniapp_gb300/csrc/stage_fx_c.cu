// Instantiations of the block fixed-point stage kernels: 6 and 7 points per
// direction (split over translation units to compile in parallel).
#include "stage_fx.cuh"
#include "stage_fx_nodal.cuh"

namespace adv
{
cudaError_t upload_tables_fx_c(const DevTables<double> *d, const DevTables<float> *f)
{
  cudaError_t e = upload_tables_local(d, f);
  if (e == cudaSuccess)
    e = upload_fx_local(d);
  return e != cudaSuccess ? e : upload_fx_basis_local(d);
}

cudaError_t launch_stage_fx_c(int n, const StageArgs &args, cudaStream_t stream)
{
  switch (n)
    {
      case 6: return launch_stage_fx_n<6>(args, stream);
      case 7: return launch_stage_fx_n<7>(args, stream);
      default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_stage_fx_nodal_c(int n, const StageArgs &args, cudaStream_t stream)
{
  switch (n)
    {
      case 6: return launch_stage_fx_nodal_n<6>(args, stream);
      case 7: return launch_stage_fx_nodal_n<7>(args, stream);
      default: return cudaErrorInvalidValue;
    }
}
} // namespace adv
