// afc_fx_f64.cu -- the compile-time power-of-two kernels in complex128.
#include "afc_fx_kernels.cuh"

namespace afc {

bool fx_ready_f64(const LaunchDesc& d) { return fx_lookup<double>(d).k != nullptr; }
cudaError_t launch_fx_f64(const LaunchDesc& d, cudaStream_t st) { return launch_fx_t<double>(d, st); }

}  // namespace afc
