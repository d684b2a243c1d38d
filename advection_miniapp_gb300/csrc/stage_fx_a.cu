// Instantiations of the block fixed-point stage kernels: 2 and 3 points per
// direction (split over translation units to compile in parallel).
#include "stage_fx.cuh"
#include "stage_fx_nodal.cuh"

namespace adv
{
cudaError_t upload_tables_fx_a(const DevTables<double> *d, const DevTables<float> *f)
{
  cudaError_t e = upload_tables_local(d, f);
  if (e == cudaSuccess)
    e = upload_fx_local(d);
  return e != cudaSuccess ? e : upload_fx_basis_local(d);
}

cudaError_t launch_stage_fx_a(int n, const StageArgs &args, cudaStream_t stream)
{
  switch (n)
    {
      case 2: return launch_stage_fx_n<2>(args, stream);
      case 3: return launch_stage_fx_n<3>(args, stream);
      default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_stage_fx_nodal_a(int n, const StageArgs &args, cudaStream_t stream)
{
  switch (n)
    {
      case 2: return launch_stage_fx_nodal_n<2>(args, stream);
      case 3: return launch_stage_fx_nodal_n<3>(args, stream);
      default: return cudaErrorInvalidValue;
    }
}
} // namespace adv
