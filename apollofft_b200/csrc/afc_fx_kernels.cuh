// afc_fx_kernels.cuh -- plain launches of the compile-time power-of-two engine
// (one tile per CTA).  Included once per precision (afc_fx_f32.cu,
// afc_fx_f64.cu) so the two sets of kernels compile side by side.
#pragma once
#include <cstdlib>
#include "afc_async.cuh"
#include "afc_fx.cuh"

namespace afc {

// CTAs per SM a kernel is built for.  16 points are 32 (complex64) or 64
// (complex128) registers; three 256-thread CTAs leave 80 registers, two 128.
template <class T> constexpr int fx_min_ctas(int threads) {
  return threads > 256 ? 1 : (sizeof(T) == 4 ? 3 : 2) * (256 / threads);
}

template <class T, int N, int FORM, int MODE, int IN, int OUT>
__global__ void __launch_bounds__(FxTile<T, N, FORM>::threads, fx_min_ctas<T>(FxTile<T, N, FORM>::threads))
    fx_kernel(const __grid_constant__ KArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int L = FxTile<T, N, FORM>::L;
  // launched with programmatic stream serialization the CTA may start while
  // the previous launch drains; nothing is read before that one has completed
  griddep_wait();
  griddep_launch_dependents();
  fx_tile<T, N, L, FORM, MODE, IN, OUT>(a, blockIdx.x * (unsigned)L, reinterpret_cast<typename CT<T>::type*>(smraw));
}

struct FxEntry {
  const void* k = nullptr;
  int L = 0, threads = 0;
  size_t smem = 0;
};
template <class T, int N, int FORM, int MODE, int IN, int OUT> static FxEntry fx_entry() {
  using Tl = FxTile<T, N, FORM>;
  return FxEntry{reinterpret_cast<const void*>(&fx_kernel<T, N, FORM, MODE, IN, OUT>), Tl::L, Tl::threads, Tl::smem};
}

// Lane-minor forms stop at 1024 points: rows of 64 bytes at 2048 would need a
// CTA of 1024 threads (64 registers each).
template <class T, int FORM, int MODE, int IN, int OUT> static FxEntry fx_by_length(long long n) {
  switch (n) {
    case 64: return fx_entry<T, 64, FORM, MODE, IN, OUT>();
    case 128: return fx_entry<T, 128, FORM, MODE, IN, OUT>();
    case 256: return fx_entry<T, 256, FORM, MODE, IN, OUT>();
    case 512: return fx_entry<T, 512, FORM, MODE, IN, OUT>();
    case 1024: return fx_entry<T, 1024, FORM, MODE, IN, OUT>();
    default: break;
  }
  if constexpr (FORM == FX_ROWS) {
    if (n == 2048) return fx_entry<T, 2048, FORM, MODE, IN, OUT>();
    if (n == 4096) return fx_entry<T, 4096, FORM, MODE, IN, OUT>();
  }
  return FxEntry{};
}

template <class T> static FxEntry fx_lookup(const LaunchDesc& d) {
  const long long n = d.sl.n;
  bool cin = d.in_op == IN_C || d.in_op == IN_R, cout = d.out_op == OUT_C || d.out_op == OUT_RE;
  if (d.fx_form == FX_ROWS && d.fx_mode != FX_CONV) {
    cin = cin || (d.in_op == IN_HERM && d.herm_n == n);
    cout = cout || (d.out_op == OUT_TRUNC && d.herm_n == n && d.store_cols == d.nlen);
  }
  const bool chin = d.in_op == IN_CHIRP || d.in_op == IN_CHIRP_R;
  const bool chout = d.out_op == OUT_CHIRP || d.out_op == OUT_CHIRP_RE;
  switch (d.fx_form) {
    case FX_ROWS:
      if (d.fx_mode == FX_CONV) {
        if (cin && cout) return fx_by_length<T, FX_ROWS, FX_CONV, IN_C, OUT_C>(n);
        if (chin && chout) return fx_by_length<T, FX_ROWS, FX_CONV, IN_CHIRP, OUT_CHIRP>(n);
      } else if (cin && cout) {
        return d.fx_mode == FX_FWD ? fx_by_length<T, FX_ROWS, FX_FWD, IN_C, OUT_C>(n)
                                   : fx_by_length<T, FX_ROWS, FX_INV, IN_C, OUT_C>(n);
      } else if (d.fx_mode == FX_FWD && d.in_op == IN_FRAME && d.out_op == OUT_C) {
        return fx_by_length<T, FX_ROWS, FX_FWD, IN_FRAME, OUT_C>(n);
      }
      break;
    case FX_COLS:
      if (cin && cout)
        return d.fx_mode == FX_FWD ? fx_by_length<T, FX_COLS, FX_FWD, IN_C, OUT_C>(n)
                                   : fx_by_length<T, FX_COLS, FX_INV, IN_C, OUT_C>(n);
      if (d.fx_mode == FX_FWD && cin && d.out_op == OUT_STEP)
        return fx_by_length<T, FX_COLS, FX_FWD, IN_C, OUT_STEP>(n);
      if (d.fx_mode == FX_INV && cin && d.out_op == OUT_STEP)
        return fx_by_length<T, FX_COLS, FX_INV, IN_C, OUT_STEP>(n);
      if (d.fx_mode == FX_FWD && chin && d.out_op == OUT_STEP)
        return fx_by_length<T, FX_COLS, FX_FWD, IN_CHIRP, OUT_STEP>(n);
      if (d.fx_mode == FX_INV && d.in_op == IN_STEP && chout)
        return fx_by_length<T, FX_COLS, FX_INV, IN_STEP, OUT_CHIRP>(n);
      break;
    case FX_ROWS_T:
      if (d.fx_mode == FX_FWD && cin && cout) return fx_by_length<T, FX_ROWS_T, FX_FWD, IN_C, OUT_C>(n);
      if (d.fx_mode == FX_INV && cin && cout) return fx_by_length<T, FX_ROWS_T, FX_INV, IN_C, OUT_C>(n);
      break;
    default: break;
  }
  return FxEntry{};
}

// Programmatic stream serialization for launches of at most one wave: their
// CTAs set up while the previous launch drains.
static bool fx_pdl(long long grid, int threads) {
  static const int pdl_env = [] {
    const char* e = getenv("AFC_PDL");
    return e && *e ? atoi(e) : 1;
  }();
  return pdl_env >= 2 || (pdl_env == 1 && grid * threads <= 148LL * 512);
}

template <class T> static cudaError_t launch_fx_t(const LaunchDesc& d, cudaStream_t st) {
  const FxEntry e = fx_lookup<T>(d);
  if (!e.k) return cudaErrorInvalidValue;
  cudaError_t ce = kernel_smem_grant(e.k, e.smem);
  if (ce != cudaSuccess) return ce;
  KArgs<T> a = to_kargs<T>(d);
  void* args[] = {&a};
  const long long grid = (d.lanes + e.L - 1) / e.L;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3((unsigned)e.threads, 1, 1);
  cfg.dynamicSmemBytes = e.smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = fx_pdl(grid, e.threads) ? 1 : 0;
  ce = cudaLaunchKernelExC(&cfg, e.k, args);
  count_launch(1);
  return ce;
}

}  // namespace afc
