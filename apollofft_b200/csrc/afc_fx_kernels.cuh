// afc_fx_kernels.cuh -- plain launches of the compile-time power-of-two engine
// (one tile per CTA).  Included once per precision (afc_fx_f32.cu,
// afc_fx_f64.cu) so the two sets of kernels compile side by side.
#pragma once
#include <cstdlib>
#include "afc_async.cuh"
#include "afc_fx.cuh"

namespace afc {

// CTAs per SM a kernel is built for.  16 points are 32 (complex64) or 64
// (complex128) registers; 1024 threads leave 64 registers, 768 80, 512 128.
// Complex64 rows fit 64 without spills (16384 x 4096 both ways 391 -> 369 us);
// the strides of columns of up to 512 points and the convolution's second network
// do not (8 x 2^20 151 -> 164 us) and keep 80.  Columns of 1024 and 2048 points run
// 512 threads, two CTAs of 64 registers and 16 to 24 bytes of spills (one CTA of
// 128: 8 x 2^20 183 us against 148).  The odd lengths hold at most 10 points.
template <class T, int N, int FORM, int MODE> constexpr int fx_min_ctas(int threads) {
  if (!fx_pow2(N)) return (sizeof(T) == 4 ? 1024 : 512) / ((threads + 31) / 32 * 32);
  if (threads > 256) return sizeof(T) == 4 ? 2 : 1;
  return (sizeof(T) == 8 ? 2 : FORM == FX_ROWS && MODE != FX_CONV ? 4 : 3) * (256 / threads);
}

template <class T, int N, int FORM, int MODE, int IN, int OUT, bool HALF>
__global__ void __launch_bounds__(FxTile<T, N, FORM>::threads, fx_min_ctas<T, N, FORM, MODE>(FxTile<T, N, FORM>::threads))
    fx_kernel(const __grid_constant__ KArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int L = FxTile<T, N, FORM>::L;
  // launched with programmatic stream serialization the CTA may start while
  // the previous launch drains; nothing is read before that one has completed
  griddep_wait();
  griddep_launch_dependents();
  fx_tile<T, N, L, FORM, MODE, IN, OUT, HALF>(a, blockIdx.x * (unsigned)L,
                                       reinterpret_cast<typename CT<T>::type*>(smraw));
}

struct FxEntry {
  const void* k = nullptr;
  int L = 0, threads = 0;
  size_t smem = 0;
};
template <class T, int N, int FORM, int MODE, int IN, int OUT, bool HALF> static FxEntry fx_entry() {
  using Tl = FxTile<T, N, FORM>;
  return FxEntry{reinterpret_cast<const void*>(&fx_kernel<T, N, FORM, MODE, IN, OUT, HALF>), Tl::L, Tl::threads, Tl::smem};
}

// Lane-minor forms stop at 1024 points: rows of 64 bytes at 2048 would need a
// CTA of 1024 threads (64 registers each).  Plain complex64 columns of 2048 points
// have a build with rows of 32 bytes (the 2048^2 images: 128 us a pass against 150 on
// the TMA kernel).
template <class T, int FORM, int MODE, int IN, int OUT, bool HALF = false> static FxEntry fx_by_length(long long n) {
  switch (n) {
    case 64: return fx_entry<T, 64, FORM, MODE, IN, OUT, HALF>();
    case 128: return fx_entry<T, 128, FORM, MODE, IN, OUT, HALF>();
    case 256: return fx_entry<T, 256, FORM, MODE, IN, OUT, HALF>();
    case 512: return fx_entry<T, 512, FORM, MODE, IN, OUT, HALF>();
    case 1024: return fx_entry<T, 1024, FORM, MODE, IN, OUT, HALF>();
    default: break;
  }
  if constexpr (FORM == FX_ROWS) {
    if (n == 2048) return fx_entry<T, 2048, FORM, MODE, IN, OUT, HALF>();
    if (n == 4096) return fx_entry<T, 4096, FORM, MODE, IN, OUT, HALF>();
  }
  if constexpr (FORM == FX_COLS && IN == IN_C && OUT == OUT_C && sizeof(T) == 4)
    if (n == 2048) return fx_entry<T, 2048, FORM, MODE, IN, OUT, HALF>();
  if constexpr (FORM != FX_ROWS_T && MODE != FX_CONV && IN == IN_C && OUT == OUT_C) {
    if (n == 243) return fx_entry<T, 243, FORM, MODE, IN, OUT, HALF>();
    if (n == 250) return fx_entry<T, 250, FORM, MODE, IN, OUT, HALF>();
    if (n == 343) return fx_entry<T, 343, FORM, MODE, IN, OUT, HALF>();
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
  // chirped points j = i jmul + col below n jmul / 2 lie in the lower half of every lane
  const bool half = 2 * std::max(d.nlen, d.nlen_out) <= n * d.jmul;
  switch (d.fx_form) {
    case FX_ROWS:
      if (d.fx_mode == FX_CONV) {
        if (cin && cout) return fx_by_length<T, FX_ROWS, FX_CONV, IN_C, OUT_C>(n);
        if (chin && chout)  // half: Bluestein always, a CZT when both of its lengths are at most n / 2
          return half ? fx_by_length<T, FX_ROWS, FX_CONV, IN_CHIRP, OUT_CHIRP, true>(n)
                      : fx_by_length<T, FX_ROWS, FX_CONV, IN_CHIRP, OUT_CHIRP>(n);
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
      if (d.fx_mode == FX_FWD && chin && d.out_op == OUT_STEP && half)
        return fx_by_length<T, FX_COLS, FX_FWD, IN_CHIRP, OUT_STEP, true>(n);
      if (d.fx_mode == FX_INV && d.in_op == IN_STEP && chout && half)
        return fx_by_length<T, FX_COLS, FX_INV, IN_STEP, OUT_CHIRP, true>(n);
      break;
    case FX_ROWS_T:
      if (d.fx_mode == FX_FWD && cin && cout) return fx_by_length<T, FX_ROWS_T, FX_FWD, IN_C, OUT_C>(n);
      if (d.fx_mode == FX_INV && cin && cout) return fx_by_length<T, FX_ROWS_T, FX_INV, IN_C, OUT_C>(n);
      break;
    default: break;
  }
  return FxEntry{};
}

// Programmatic stream serialization: a launch's CTAs set up while the previous
// one drains, and none reads anything before that one has completed (every
// thread waits first).  256^3 complex128 both ways 518 -> 504 us, 16384 x 4096
// complex64 391 -> 381, 4096 CZTs 99 -> 96.  AFC_PDL=0 launches plainly.
static bool fx_pdl() {
  static const int pdl_env = [] {
    const char* e = getenv("AFC_PDL");
    return e && *e ? atoi(e) : 1;
  }();
  return pdl_env != 0;
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
  cfg.numAttrs = fx_pdl() ? 1 : 0;
  ce = cudaLaunchKernelExC(&cfg, e.k, args);
  count_launch(1);
  return ce;
}

// ───────────────────────── persistent batch kernel ─────────────────────────
// Every compile-time tile of an uneven batch in one launch.  A tile is 4096
// points (256 threads) of any length and form; CTAs claim tiles in list order
// from an atomic counter.  A transform of several passes (two-pass lengths,
// large Bluestein) orders them by a counter of its own: each finished tile adds
// one, and a tile of a later pass waits until every tile of the passes before
// it is done.  Waiting is safe without co-residency: a tile waits only for tiles
// earlier in the list, those were claimed earlier by CTAs that are running, and
// the lowest unfinished tile never waits for an unfinished one.  Waits are
// bounded: on timeout the CTA sets the error word and leaves.
//
// One launch instead of one per pass keeps a transform's intermediate in L2
// (the list runs its passes a few hundred tiles apart) and leaves one tail.  The
// next tile's claim and list entry are fetched while the current tile runs.

constexpr int kFxBatchThreads = 256;

template <class T, int N, int FORM, int MODE, int IN, int OUT>
__device__ __forceinline__ void fx_batch_tile(const KArgs<T>& a, unsigned q0, unsigned char* sm) {
  fx_tile<T, N, 4096 / N, FORM, MODE, IN, OUT, IN == IN_CHIRP || OUT == OUT_CHIRP>(
      a, q0, reinterpret_cast<typename CT<T>::type*>(sm));
}

__device__ __forceinline__ void fx_cp16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}

// Long lists (deep): the claims of a CTA run three tiles ahead; while tile i
// runs, the descriptor of tile i + 1, the list entry of tile i + 2 and the claim
// of tile i + 3 are on their way, so none of the three dependent fetches is
// waited for.  Lists under six tiles per CTA claim one tile at a time, which
// balances them better (us one by one -> ahead: 3.1 tiles per CTA, 128 transforms of
// 64 .. 65536 points complex128, 116 -> 123; 3.7, 4096 of 64 .. 4096 complex64, 119 ->
// 127; 6.1, 512 of 64 .. 65536 complex64, 181 -> 181; 7.4, 4096 of 64 .. 4096
// complex128, 266 -> 260; 54, 4096 of 64 .. 65536 complex64, 1096 -> 1071).
// Descriptors are read from shared memory, field by field where they are used
// (read through a global pointer the compiler kept them in registers across the
// tile and spilled 1.7 KB; now 64 bytes, and complex64 fits four CTAs per SM:
// 4096 uneven transforms 1238 us at three, 1177 us at four).
template <class T, bool INV>
__global__ void __launch_bounds__(kFxBatchThreads, sizeof(T) == 4 ? 4 : 2)
    fx_batch_kernel(const KArgs<T>* __restrict__ descs, const FxBatchItem* __restrict__ items, int nitems, int* ctr,
                    const void* in_base, void* out_base, void* ws_base, unsigned* err, int deep) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(16) KArgs<T> s_ka[2];
  __shared__ __align__(16) FxBatchItem s_item[3];
  __shared__ int s_idx[3];
  static_assert(sizeof(KArgs<T>) % 16 == 0 && sizeof(FxBatchItem) % 16 == 0, "copied 16 bytes at a time");
  constexpr int KW = (int)sizeof(KArgs<T>) / 16, IW = (int)sizeof(FxBatchItem) / 16;
  const int tid = threadIdx.x;
  constexpr int DIR = INV ? FX_INV : FX_FWD;
  auto copy_desc = [&](int slot, int item) {
    const char* src = reinterpret_cast<const char*>(descs + s_item[item].desc);
    if (tid < KW) fx_cp16(reinterpret_cast<char*>(&s_ka[slot]) + 16 * tid, src + 16 * tid);
  };
  // thread 0, once the copy has landed: buffer selectors become pointers
  auto resolve = [&](int slot, int item) {
    KArgs<T>& k = s_ka[slot];
    char* bases[4] = {nullptr, (char*)in_base, (char*)out_base, (char*)ws_base};
    k.in = bases[k.in_sel] + (size_t)k.in + s_item[item].in_off;
    k.out = bases[k.out_sel] + (size_t)k.out + s_item[item].out_off;
  };
  if (tid == 0) {
    // one claim after the other: a CTA runs its claims in list order
    s_idx[0] = atomicAdd(ctr, 1);
    s_item[0] = items[min(s_idx[0], nitems - 1)];
    if (deep) {
      s_idx[1] = atomicAdd(ctr, 1);
      s_item[1] = items[min(s_idx[1], nitems - 1)];
      s_idx[2] = atomicAdd(ctr, 1);
    }
  }
  __syncthreads();
  copy_desc(0, 0);
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  if (tid == 0) resolve(0, 0);
  __syncthreads();
  for (int i = 0;; ++i) {
    const int c0 = i % 3, c1 = (i + 1) % 3, c2 = (i + 2) % 3, ks = i & 1;
    if (s_idx[c0] >= nitems) break;
    int nx = 0;
    if (deep) copy_desc(ks ^ 1, c1);
    if (deep && tid == 0) {
      const char* src = reinterpret_cast<const char*>(items + min(s_idx[c2], nitems - 1));
#pragma unroll
      for (int w = 0; w < IW; ++w) fx_cp16(reinterpret_cast<char*>(&s_item[c2]) + 16 * w, src + 16 * w);
      nx = atomicAdd(ctr, 1);
    }
    if (s_item[c0].wait > 0) {  // the passes before this one, of the same transform
      bool ok = true;
      if (tid == 0) {
        const volatile int* c = ctr + s_item[c0].dep;
        const int want = s_item[c0].wait;
        int k = 0;
        while (*c < want && k < (1 << 22)) {
          __nanosleep(64);
          ++k;
        }
        ok = *c >= want;
        __threadfence();
      }
      if (__syncthreads_or(!ok)) {
        if (tid == 0) {
          atomicExch(err, 1u);
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        return;
      }
    }
    const KArgs<T>& a = s_ka[ks];
    const unsigned q0 = s_item[c0].q0;
#define AFC_FXB(OP, LG, FORM, MODE, IN, OUT) \
  case OP * 8 + LG - 6: fx_batch_tile<T, (1 << LG), FORM, MODE, IN, OUT>(a, q0, smraw); break;
#define AFC_FXB5(OP, FORM, MODE, IN, OUT)                                                                     \
  AFC_FXB(OP, 6, FORM, MODE, IN, OUT) AFC_FXB(OP, 7, FORM, MODE, IN, OUT) AFC_FXB(OP, 8, FORM, MODE, IN, OUT) \
  AFC_FXB(OP, 9, FORM, MODE, IN, OUT) AFC_FXB(OP, 10, FORM, MODE, IN, OUT)
#define AFC_FXB7(OP, FORM, MODE, IN, OUT) \
  AFC_FXB5(OP, FORM, MODE, IN, OUT) AFC_FXB(OP, 11, FORM, MODE, IN, OUT) AFC_FXB(OP, 12, FORM, MODE, IN, OUT)
    switch (s_item[c0].kind) {
      AFC_FXB7(FXB_ROWS, FX_ROWS, DIR, IN_C, OUT_C)
      AFC_FXB5(FXB_COLS, FX_COLS, DIR, IN_C, OUT_STEP)
      AFC_FXB5(FXB_ROWS_T, FX_ROWS_T, DIR, IN_C, OUT_C)
      AFC_FXB7(FXB_CONV, FX_ROWS, FX_CONV, IN_CHIRP, OUT_CHIRP)
      AFC_FXB5(FXB_CHIRP_COLS, FX_COLS, FX_FWD, IN_CHIRP, OUT_STEP)
      AFC_FXB5(FXB_CONV_ROWS, FX_ROWS, FX_CONV, IN_C, OUT_C)
      AFC_FXB5(FXB_COLS_CHIRP, FX_COLS, FX_INV, IN_STEP, OUT_CHIRP)
      default: break;
    }
#undef AFC_FXB7
#undef AFC_FXB5
#undef AFC_FXB
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();  // the tile's stores are issued, its shared memory is free, the copies have landed
    if (tid == 0) {
      if (s_item[c0].dep > 0) {
        __threadfence();
        atomicAdd(ctr + s_item[c0].dep, 1);
      }
      if (deep) {
        s_idx[c0] = nx;  // tile i + 3
        resolve(ks ^ 1, c1);
      } else {
        s_idx[c1] = atomicAdd(ctr, 1);
        s_item[c1] = items[min(s_idx[c1], nitems - 1)];
      }
    }
    __syncthreads();
    if (!deep && s_idx[c1] < nitems) {
      copy_desc(ks ^ 1, c1);
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncthreads();
      if (tid == 0) resolve(ks ^ 1, c1);
      __syncthreads();
    }
  }
}

// Tile kind of a descriptor in the batch kernel, -1 when it has none.
template <class T> static int fx_batch_kind_t(const LaunchDesc& d) {
  if (!fx_lookup<T>(d).k || d.store_cols || d.hm_cmax) return -1;
  if ((d.in_op != IN_C && d.in_op != IN_CHIRP && d.in_op != IN_STEP) ||
      (d.out_op != OUT_C && d.out_op != OUT_CHIRP && d.out_op != OUT_STEP))
    return -1;
  int lg = 0;
  while ((1 << lg) < d.sl.n) ++lg;
  if ((1 << lg) != d.sl.n) return -1;
  int op;
  if (d.fx_form == FX_ROWS) op = d.fx_mode != FX_CONV ? FXB_ROWS : d.in_op == IN_CHIRP ? FXB_CONV : FXB_CONV_ROWS;
  else if (d.fx_form == FX_ROWS_T) op = FXB_ROWS_T;
  else if (d.out_op == OUT_STEP) op = d.in_op == IN_CHIRP ? FXB_CHIRP_COLS : FXB_COLS;
  else if (d.in_op == IN_STEP) op = FXB_COLS_CHIRP;
  else return -1;
  if (d.out_op == OUT_CHIRP || d.in_op == IN_CHIRP)  // chirp tiles of the batch kernel are half
    if (2 * std::max(d.nlen, d.nlen_out) > (long long)d.sl.n * d.jmul) return -1;
  if (lg > 10 && op != FXB_ROWS && op != FXB_CONV) return -1;
  return op * 8 + lg - 6;
}

template <class T> constexpr size_t fx_batch_smem() {
  using C = typename CT<T>::type;
  size_t m = 0;
  const int ns[7] = {64, 128, 256, 512, 1024, 2048, 4096};
  for (int n : ns)
    for (int lm = 0; lm < (n <= 1024 ? 2 : 1); ++lm) {
      const size_t b = (size_t)(4096 / n) * fx_ld(n, 4096 / n, lm != 0, (int)sizeof(C)) * sizeof(C);
      if (b > m) m = b;
    }
  return m;
}

template <class T>
static cudaError_t launch_fx_batch_t(const void* descs, const FxBatchItem* items, int nitems, int* ctr, const void* in,
                                     void* out, void* ws, unsigned* err, bool inv, cudaStream_t st) {
  auto k = inv ? fx_batch_kernel<T, true> : fx_batch_kernel<T, false>;
  const size_t smem = fx_batch_smem<T>();
  cudaError_t e = kernel_smem_grant(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  int sms = 148, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long grid = (long long)sms * kernel_ctas_per_sm(reinterpret_cast<const void*>(k), kFxBatchThreads, smem);
  const int deep = nitems >= 6 * grid;
  if (grid > nitems) grid = nitems;
  k<<<(unsigned)grid, kFxBatchThreads, smem, st>>>(static_cast<const KArgs<T>*>(descs), items, nitems, ctr, in, out, ws,
                                                   err, deep);
  count_launch(1);
  return cudaGetLastError();
}

}  // namespace afc
