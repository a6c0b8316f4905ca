// afc_fx_f32.cu -- the compile-time power-of-two kernels in complex64.
#include "afc_fx_kernels.cuh"

namespace afc {

bool fx_ready_f32(const LaunchDesc& d) { return fx_lookup<float>(d).k != nullptr; }
cudaError_t launch_fx_f32(const LaunchDesc& d, cudaStream_t st) { return launch_fx_t<float>(d, st); }

}  // namespace afc
