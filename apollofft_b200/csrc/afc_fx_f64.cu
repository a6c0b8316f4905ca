// afc_fx_f64.cu -- the compile-time power-of-two kernels in complex128.
#include "afc_fx_kernels.cuh"

namespace afc {

bool fx_ready_f64(const LaunchDesc& d) { return fx_lookup<double>(d).k != nullptr; }
cudaError_t launch_fx_f64(const LaunchDesc& d, cudaStream_t st) { return launch_fx_t<double>(d, st); }
int fx_batch_kind_f64(const LaunchDesc& d) { return fx_batch_kind_t<double>(d); }
cudaError_t launch_fx_batch_f64(const void* descs, const FxBatchItem* items, int nitems, int* ctr, const void* in,
                                void* out, void* ws, unsigned* err, bool inv, cudaStream_t st) {
  return launch_fx_batch_t<double>(descs, items, nitems, ctr, in, out, ws, err, inv, st);
}

}  // namespace afc
