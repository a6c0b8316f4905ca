// afc_kargs.cuh -- launch arguments of the lanes / convolution kernels and the
// global load / store operators they apply (shared by the general engine and
// the compile-time power-of-two engine).
#pragma once
#include <cuda_runtime.h>
#include <cstring>
#include "afc_engine.cuh"
#include "afc_internal.h"

namespace afc {

// ───────────────────────────── kernel arguments ─────────────────────────────

template <class T> struct alignas(16) KArgs {
  using C = typename CT<T>::type;
  StageList sl;
  const C* tw;
  long long lanes;
  int L, P, ld;
  int in_op, out_op;
  int stage_in, stage_out;
  LaneMap im, om;          // input / output lane maps
  const void* in;
  void* out;
  T scale;
  // element-index map of index-aware operators: j = i * jmul + col(q),
  // col(q) = (q / col_div) % col_mod.
  long long jmul, col_div, col_mod;
  long long nlen;          // valid length (chirp / truncation) or p (Rader)
  long long herm_n;        // full length behind a half spectrum
  T pair_w;                // Hermitian weight of paired bins (adjoints); 1 otherwise
  // four-step twiddle W_N^{(col * i) mod N} = hi[m / B] * lo[m % B], conj if tw_conj
  long long twN, twB;
  int tw_conj;
  const C* tw_hi;
  const C* tw_lo;
  const C* spec;           // pointwise spectrum
  long long spec_ld;       // convolution tiles: lane spectrum = spec + col * spec_ld (0: shared)
  const C* chirp;          // Bluestein chirp (forward sign; conj if chirp_conj)
  int chirp_conj;
  const int* gather;       // Rader: gather[q] = g^q mod p
  const int* scatter;      // Rader: scatter[q] = g^{-q} mod p
  int lane_minor;          // tile kernel: consecutive threads take consecutive lanes
  int in_sel, out_sel;     // batch descriptors: 0 absolute pointer, else base[sel] + offset
  const C* chirp_out;      // OUT_CHIRP: post-multiply table when it differs from chirp (CZT)
  long long nlen_out;      // OUT_CHIRP: outputs kept when > 0 (else nlen)
  const T* window;         // IN_FRAME: analysis window
  long long frame_off;     // IN_FRAME: frame q covers signal[q hop - frame_off + i]
  const C* fx_tw;          // compile-time engine: stage twiddles and step twiddle factors
  const C* fx_a;
  const C* fx_b;
  // log2 of im.d2, om.d2, col_div and col_mod when all four are powers of two
  // (two-pass lengths on contiguous lanes), else fx_sh[0] = -1
  int fx_sh[4];
  int store_cols;          // compile-time rows: > 0 keeps the first store_cols points
  int hm_cmax;             // compile-time columns: columns 1 .. hm_cmax are also stored mirrored
};

template <class T>
__device__ __forceinline__ typename CT<T>::type gload(const KArgs<T>& a, long long base, long long col, int i) {
  using C = typename CT<T>::type;
  const C zero = C{(T)0, (T)0};
  switch (a.in_op) {
    case IN_C:
      return static_cast<const C*>(a.in)[base + (long long)i * a.im.es];
    case IN_R:  // real input widened (reference RealFftData, real_storage.rs:186-303)
      return C{static_cast<const T*>(a.in)[base + (long long)i * a.im.es], (T)0};
    case IN_HERM: {  // half spectrum (n/2+1 bins) expanded by Hermitian symmetry
      const C* p = static_cast<const C*>(a.in);
      const long long n = a.herm_n;
      const long long j = (long long)i * a.jmul + col;  // index in the full spectrum
      C v;
      if (2 * j <= n) {
        v = p[base + (long long)i * a.im.es];
      } else {  // a two-pass column starts col elements into the lane
        const long long es = a.im.es / a.jmul;
        v = p[base + (n - j - col) * es];
        v.y = -v.y;
      }
      if (j > 0 && 2 * j != n) v = cscale(v, a.pair_w);
      return v;
    }
    case IN_CHIRP:
    case IN_CHIRP_R: {  // Bluestein premultiply x[j] * chirp[j], zero for j >= nlen
      const long long j = (long long)i * a.jmul + col;
      if (j >= a.nlen) return zero;
      const long long off = base + (long long)i * a.im.es;
      C x = a.in_op == IN_CHIRP ? static_cast<const C*>(a.in)[off] : C{static_cast<const T*>(a.in)[off], (T)0};
      const C c = a.chirp[j];
      return a.chirp_conj ? cmulc(x, c) : cmul(x, c);
    }
    case IN_GATHER:
    case IN_GATHER_R: {  // Rader: x[g^i] for i < p-1, zero padding beyond
      if (i >= a.nlen - 1) return zero;
      const long long off = base + (long long)a.gather[i] * a.im.es;
      return a.in_op == IN_GATHER ? static_cast<const C*>(a.in)[off] : C{static_cast<const T*>(a.in)[off], (T)0};
    }
    case IN_FRAME: {  // STFT analysis frame: signal[base - frame_off + i] * window[i], zero outside the signal
      const long long j = base - a.frame_off + i;
      if (j < 0 || j >= a.nlen) return zero;
      return C{static_cast<const T*>(a.in)[j] * a.window[i], (T)0};
    }
  }
  return zero;
}

template <class T>
__device__ __forceinline__ void gstore(const KArgs<T>& a, long long base, long long col, int i,
                                       typename CT<T>::type v, typename CT<T>::type x0) {
  using C = typename CT<T>::type;
  const long long off = base + (long long)i * a.om.es;
  switch (a.out_op) {
    case OUT_C:
      static_cast<C*>(a.out)[off] = cscale(v, a.scale);
      return;
    case OUT_RE:  // real part (reference C2R: full inverse then .re)
      static_cast<T*>(a.out)[off] = v.x * a.scale;
      return;
    case OUT_TRUNC: {  // keep j < nlen (half spectrum); paired bins weighted by pair_w
      const long long j = (long long)i * a.jmul + col;
      if (j < a.nlen) {
        const bool paired = (j > 0) && (2 * j != a.herm_n);
        static_cast<C*>(a.out)[off] = cscale(v, paired ? a.scale * a.pair_w : a.scale);
      }
      return;
    }
    case OUT_TW: {  // four-step: multiply by W_N^{col * i}; twB is a power of two
      unsigned long long m = (unsigned long long)col * (unsigned long long)i;
      if (m >= (unsigned long long)a.twN) m %= (unsigned long long)a.twN;  // col * i < N in every four-step pass
      const int sh = __ffsll(a.twB) - 1;
      const C w = cmul(a.tw_hi[m >> sh], a.tw_lo[m & (unsigned long long)(a.twB - 1)]);
      v = a.tw_conj ? cmulc(v, w) : cmul(v, w);
      static_cast<C*>(a.out)[off] = cscale(v, a.scale);
      return;
    }
    case OUT_MUL: {  // pointwise spectrum at natural index j
      const long long j = (long long)i * a.jmul + col;
      static_cast<C*>(a.out)[off] = cmul(v, a.spec[j]);
      return;
    }
    case OUT_CHIRP:
    case OUT_CHIRP_RE: {  // Bluestein / CZT post-multiply, keep j < nlen (nlen_out when set)
      const long long j = (long long)i * a.jmul + col;
      if (j < (a.nlen_out > 0 ? a.nlen_out : a.nlen)) {
        const C c = a.chirp_out ? a.chirp_out[j] : a.chirp[j];
        v = cscale(a.chirp_conj ? cmulc(v, c) : cmul(v, c), a.scale);
        if (a.out_op == OUT_CHIRP) static_cast<C*>(a.out)[off] = v;
        else static_cast<T*>(a.out)[off] = v.x;
      }
      return;
    }
    case OUT_SCATTER:
    case OUT_SCATTER_RE: {  // Rader: X[g^{-i}] = x0 + conv[i]
      if (i < a.nlen - 1) {
        const long long o2 = base + (long long)a.scatter[i] * a.om.es;
        const C y = cscale(cadd(x0, v), a.scale);
        if (a.out_op == OUT_SCATTER) static_cast<C*>(a.out)[o2] = y;
        else static_cast<T*>(a.out)[o2] = y.x;
      }
      return;
    }
  }
}

template <class T> __device__ __forceinline__ long long col_of(const KArgs<T>& a, long long q) {
  return (q / a.col_div) % a.col_mod;
}

template <class T> inline KArgs<T> to_kargs(const LaunchDesc& d) {
  using C = typename CT<T>::type;
  KArgs<T> a;
  memset(&a, 0, sizeof(a));
  a.sl = d.sl;
  a.tw = static_cast<const C*>(d.tw);
  a.lanes = d.lanes;
  a.L = d.L;
  a.P = d.P;
  a.ld = d.ld;
  a.in_op = d.in_op;
  a.out_op = d.out_op;
  a.stage_in = d.stage_in;
  a.stage_out = d.stage_out;
  a.im = d.im;
  a.om = d.om;
  a.in = d.in;
  a.out = d.out;
  a.scale = (T)d.scale;
  a.jmul = d.jmul ? d.jmul : 1;
  a.col_div = d.col_div ? d.col_div : 1;
  a.col_mod = d.col_mod ? d.col_mod : 1;
  a.nlen = d.nlen;
  a.herm_n = d.herm_n;
  a.pair_w = (T)d.pair_w;
  a.twN = d.twN ? d.twN : 1;
  a.twB = d.twB ? d.twB : 1;
  a.tw_conj = d.tw_conj;
  a.tw_hi = static_cast<const C*>(d.tw_hi);
  a.tw_lo = static_cast<const C*>(d.tw_lo);
  a.spec = static_cast<const C*>(d.spec);
  a.spec_ld = d.spec_ld;
  a.window = static_cast<const T*>(d.window);
  a.chirp_out = static_cast<const C*>(d.chirp_out);
  a.nlen_out = d.nlen_out;
  a.frame_off = d.frame_off;
  a.chirp = static_cast<const C*>(d.chirp);
  a.chirp_conj = d.chirp_conj;
  a.gather = d.gather;
  a.scatter = d.scatter;
  a.lane_minor = d.lane_minor;
  a.fx_tw = static_cast<const C*>(d.fx_tw);
  a.fx_a = static_cast<const C*>(d.fx_a);
  a.fx_b = static_cast<const C*>(d.fx_b);
  const long long pw[4] = {a.im.d2, a.om.d2, a.col_div, a.col_mod};
  for (int i = 0; i < 4; ++i) {
    int sh = 0;
    while ((1ll << sh) < pw[i]) ++sh;
    a.fx_sh[i] = sh;
  }
  for (int i = 0; i < 4; ++i)
    if ((1ll << a.fx_sh[i]) != pw[i]) a.fx_sh[0] = -1;
  a.store_cols = d.store_cols;
  a.hm_cmax = d.hm_cmax;
  a.in_sel = d.in_sel;
  a.out_sel = d.out_sel;
  return a;
}

}  // namespace afc
