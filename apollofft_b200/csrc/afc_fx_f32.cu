// afc_fx_f32.cu -- the compile-time power-of-two kernels in complex64.
#include "afc_fx_kernels.cuh"

namespace afc {

bool fx_ready_f32(const LaunchDesc& d) { return fx_lookup<float>(d).k != nullptr; }
cudaError_t launch_fx_f32(const LaunchDesc& d, cudaStream_t st) { return launch_fx_t<float>(d, st); }
int fx_batch_kind_f32(const LaunchDesc& d) { return fx_batch_kind_t<float>(d); }
cudaError_t launch_fx_batch_f32(const void* descs, const FxBatchItem* items, int nitems, int* ctr, const void* in,
                                void* out, void* ws, unsigned* err, bool inv, cudaStream_t st) {
  return launch_fx_batch_t<float>(descs, items, nitems, ctr, in, out, ws, err, inv, st);
}

}  // namespace afc
