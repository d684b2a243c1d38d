// Instantiations of the block fixed-point advection-diffusion stage.
#include "stage_fx_visc.cuh"

namespace adv
{
cudaError_t upload_tables_fx_visc(const DevTables<double> *d, const DevTables<float> *f)
{
  cudaError_t e = upload_tables_local(d, f);
  if (e == cudaSuccess)
    e = upload_fx_local(d, kFxViscShift);
  return e != cudaSuccess ? e : upload_fx_visc_local(d);
}

cudaError_t launch_stage_fx_visc(int n, const StageArgs &args, cudaStream_t stream)
{
  switch (n)
    {
      case 2: return launch_stage_fx_visc_n<2>(args, stream);
      case 3: return launch_stage_fx_visc_n<3>(args, stream);
      case 4: return launch_stage_fx_visc_n<4>(args, stream);
      case 5: return launch_stage_fx_visc_n<5>(args, stream);
      case 6: return launch_stage_fx_visc_n<6>(args, stream);
      case 7: return launch_stage_fx_visc_n<7>(args, stream);
      default: return cudaErrorInvalidValue;
    }
}
} // namespace adv
