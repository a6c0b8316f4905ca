// afc_fx.cuh -- compile-time power-of-two engine: lanes of n = 64 .. 4096
// points, 16 points per thread in registers, every stride a template constant.
//
// The general engine (afc_engine.cuh) walks a runtime stage list: an index
// division, a padding term and a 64-bit twiddle index per butterfly, an
// operator switch and a lane-map lookup per element, and a shared-memory copy
// on each side of the stages.  Its passes are instruction-bound (large-prime
// Bluestein: about 300 thread-instructions per point and pass, 8-10 % of the
// DRAM bandwidth).  Here a thread holds points t + P q (q < 16, P = n / 16
// threads per lane) on load and on store, in every form: global memory goes
// straight to registers through an operator fixed at compile time, stages
// exchange through one shared buffer, and the result goes straight back.
//
// Two networks over the same stage list and twiddle table:
//  * forward order (Stockham, as the general engine): stage s reads
//    j + r n/R, twiddles, R-point DFT, writes (j - k) R + k + r Ns;
//  * its transpose (the DFT matrix is symmetric): stages in reverse order, each
//    reading the forward write pattern, DFT, twiddle, writing the forward read
//    pattern.  It starts from the registers the forward order ends with, so a
//    convolution multiplies by its spectrum without touching shared memory.
//
// Shared layout: element i of lane l at l LD + i + i / 16.  For powers of two
// the padded index of a + r c with a < c (or both multiples of 16) splits into
// pad(a) + pad(r c), so every access is one base plus a constant.
#pragma once
#include "afc_kargs.cuh"

namespace afc {

// Radix 16 first, the rest of the power in the last stage: the fewest twiddle
// loads for the stage count (1024 as 16 16 4: 1.7 per point, as 16 8 8: 1.75),
// and the general engine's stage list, so results round alike.
template <int N> struct FxRad;
template <> struct FxRad<64> { static constexpr int n = 2, r0 = 16, r1 = 4, r2 = 1, e = 16; };
template <> struct FxRad<128> { static constexpr int n = 2, r0 = 16, r1 = 8, r2 = 1, e = 16; };
template <> struct FxRad<256> { static constexpr int n = 2, r0 = 16, r1 = 16, r2 = 1, e = 16; };
template <> struct FxRad<512> { static constexpr int n = 3, r0 = 16, r1 = 16, r2 = 2, e = 16; };
template <> struct FxRad<1024> { static constexpr int n = 3, r0 = 16, r1 = 16, r2 = 4, e = 16; };
template <> struct FxRad<2048> { static constexpr int n = 3, r0 = 16, r1 = 16, r2 = 8, e = 16; };
template <> struct FxRad<4096> { static constexpr int n = 3, r0 = 16, r1 = 16, r2 = 16, e = 16; };
// Three odd lengths, plain rows and columns only: e points per thread, a multiple
// of every radix.  They took the place of TMA builds for the same lengths; other
// smooth lengths have none (complex64 volumes both ways, of the copy rate over six
// passes: 243 x 250 x 343 0.61; 240 x 252 x 350 0.47, 225 x 240 x 245 0.34, 288^3 0.45).
template <> struct FxRad<243> { static constexpr int n = 3, r0 = 9, r1 = 9, r2 = 3, e = 9; };
template <> struct FxRad<250> { static constexpr int n = 3, r0 = 10, r1 = 5, r2 = 5, e = 10; };
template <> struct FxRad<343> { static constexpr int n = 3, r0 = 7, r1 = 7, r2 = 7, e = 7; };

__host__ __device__ constexpr bool fx_pow2(int n) { return (n & (n - 1)) == 0; }

// Lane stride in shared memory.  Powers of two are padded by one element every
// 16; the odd lengths' strides spread over the banks by themselves.  Lane-major
// tiles (consecutive threads walk one lane): the (padded) length.  Tiles with a
// lane-minor side (consecutive threads take consecutive lanes): the next length
// congruent to (elements per 128 bytes) / L, so the lanes of a wavefront fall in
// distinct banks.
__host__ __device__ constexpr int fx_ld(int n, int lanes, bool lane_minor, int csz) {
  const int ld = n + (fx_pow2(n) ? n / 16 : 0);
  if (!lane_minor) return ld;
  const int per = 128 / csz;
  const int want = lanes >= per ? 1 : per / lanes;
  int v = ld;
  while (v % per != want) ++v;
  return v;
}

template <class T, int N> struct FxEng {
  using C = typename CT<T>::type;
  static constexpr int EP = FxRad<N>::e;  // points per thread
  static constexpr int P = N / EP, NST = FxRad<N>::n;
  __host__ __device__ static constexpr int pad(int i) { return fx_pow2(N) ? i + (i >> 4) : i; }
  __host__ __device__ static constexpr int R(int s) {
    return s == 0 ? FxRad<N>::r0 : s == 1 ? FxRad<N>::r1 : FxRad<N>::r2;
  }
  __host__ __device__ static constexpr int NS(int s) { return s == 0 ? 1 : R(s - 1) * NS(s - 1); }
  __host__ __device__ static constexpr int twoff(int s) { return s <= 1 ? 0 : twoff(s - 1) + (R(s - 1) - 1) * NS(s - 1); }

  // Butterfly b of stage S holds points q = b + r NB, r < R (NB = EP / R).
  template <int S, bool INV> __device__ __forceinline__ static void dft(C (&v)[EP]) {
    constexpr int RR = R(S), NB = EP / RR;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      C u[RR];
#pragma unroll
      for (int r = 0; r < RR; ++r) u[r] = v[b + r * NB];
      DFT<RR, INV>::run(u);
#pragma unroll
      for (int r = 0; r < RR; ++r) v[b + r * NB] = u[r];
    }
  }
  template <int S, bool INV>
  __device__ __forceinline__ static void twiddle(C (&v)[EP], const C* __restrict__ tw, int t) {
    constexpr int RR = R(S), NB = EP / RR, Ns = NS(S);
    if constexpr (Ns > 1) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const C* w = tw + twoff(S) + ((t + b * P) % Ns);
#pragma unroll
        for (int r = 1; r < RR; ++r) {
          const C wr = __ldg(w + (r - 1) * Ns);
          v[b + r * NB] = INV ? cmulc(v[b + r * NB], wr) : cmul(v[b + r * NB], wr);
        }
      }
    }
  }
  // forward write pattern of stage S: (j - k) R + k + r Ns
  template <int S> __device__ __forceinline__ static int wbase(int t, int b) {
    constexpr int RR = R(S), Ns = NS(S);
    const int j = t + b * P, k = j % Ns;
    return pad((j - k) * RR + k);
  }
  template <int S> __device__ __forceinline__ static void put_w(const C (&v)[EP], C* sm, int t) {
    constexpr int RR = R(S), NB = EP / RR, Ns = NS(S);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      C* p = sm + wbase<S>(t, b);
#pragma unroll
      for (int r = 0; r < RR; ++r) p[pad(r * Ns)] = v[b + r * NB];
    }
  }
  template <int S> __device__ __forceinline__ static void get_w(C (&v)[EP], const C* sm, int t) {
    constexpr int RR = R(S), NB = EP / RR, Ns = NS(S);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const C* p = sm + wbase<S>(t, b);
#pragma unroll
      for (int r = 0; r < RR; ++r) v[b + r * NB] = p[pad(r * Ns)];
    }
  }
  // forward read pattern of every stage: t + P q
  __device__ __forceinline__ static void put_r(const C (&v)[EP], C* sm, int t) {
    C* p = sm + pad(t);
#pragma unroll
    for (int q = 0; q < EP; ++q) p[pad(P * q)] = v[q];
  }
  __device__ __forceinline__ static void get_r(C (&v)[EP], const C* sm, int t) {
    const C* p = sm + pad(t);
#pragma unroll
    for (int q = 0; q < EP; ++q) v[q] = p[pad(P * q)];
  }
};

// Barrier of the threads sharing a lane: a warp when lane-major lanes of at
// most 32 threads lie inside one warp, else the CTA.
template <bool WARP> __device__ __forceinline__ void fx_sync() {
  if constexpr (WARP) __syncwarp();
  else __syncthreads();
}

// Forward-order network.  Before the last exchange the thread is (lane slot
// smA, position tA), after it (smB, tB): the two differ only in FX_ROWS_T
// tiles, whose store side is lane-minor.  Every thread of the CTA calls it.
// HALF: points q >= 8 (the upper half of the lane) are zero on input.
template <class T, int N, bool INV, bool WARP, bool HALF>
__device__ __forceinline__ void fx_fwd(typename CT<T>::type (&v)[FxEng<T, N>::EP], typename CT<T>::type* smA, int tA,
                                       typename CT<T>::type* smB, int tB,
                                       const typename CT<T>::type* __restrict__ tw) {
  using E = FxEng<T, N>;
  static_assert(!HALF || E::R(0) == 16, "the power-of-two lists start with radix 16");
  if constexpr (HALF) dft16_half<INV>(v);
  else E::template dft<0, INV>(v);
  E::template put_w<0>(v, smA, tA);
  fx_sync<WARP>();
  if constexpr (E::NST == 3) {
    E::get_r(v, smA, tA);
    E::template twiddle<1, INV>(v, tw, tA);
    E::template dft<1, INV>(v);
    fx_sync<WARP>();
    E::template put_w<1>(v, smA, tA);
    fx_sync<WARP>();
  }
  E::get_r(v, smB, tB);
  E::template twiddle<E::NST - 1, INV>(v, tw, tB);
  E::template dft<E::NST - 1, INV>(v);
}

// Transposed network, from the registers fx_fwd leaves.
template <class T, int N, bool INV, bool WARP>
__device__ __forceinline__ void fx_transposed(typename CT<T>::type (&v)[FxEng<T, N>::EP], typename CT<T>::type* sm, int t,
                                              const typename CT<T>::type* __restrict__ tw) {
  using E = FxEng<T, N>;
  E::template dft<E::NST - 1, INV>(v);
  E::template twiddle<E::NST - 1, INV>(v, tw, t);
  fx_sync<WARP>();
  E::put_r(v, sm, t);
  fx_sync<WARP>();
  if constexpr (E::NST == 3) {
    E::template get_w<1>(v, sm, t);
    E::template dft<1, INV>(v);
    E::template twiddle<1, INV>(v, tw, t);
    fx_sync<WARP>();
    E::put_r(v, sm, t);
    fx_sync<WARP>();
  }
  E::template get_w<0>(v, sm, t);
  E::template dft<0, INV>(v);
}

// Lane base of a three-level lane map in 32-bit lane arithmetic (the planner
// keeps lane counts below 2^31); sh = log2 d2 when d2 is a power of two, else -1.
__device__ __forceinline__ long long fx_base(const LaneMap& m, unsigned q, int sh) {
  if (m.d2 == 1) {
    if (m.off) return m.off[q];
    if (m.d1 == 1) return (long long)q * m.s0;
  }
  const unsigned d2 = (unsigned)m.d2;
  const unsigned t = sh >= 0 ? q >> sh : q / d2, c = q - t * d2;
  if (m.off) return m.off[t] + (long long)c * m.s2;
  const unsigned d1 = (unsigned)m.d1;
  if (d1 == 1) return t * m.s0 + c * m.s2;
  const unsigned a = t / d1, b = t - a * d1;
  return a * m.s0 + b * m.s1 + c * m.s2;
}

// Column of a lane: (q / col_div) mod col_mod.
template <class T> __device__ __forceinline__ unsigned fx_col(const KArgs<T>& a, unsigned q) {
  if (a.fx_sh[0] >= 0) return (q >> a.fx_sh[2]) & ((unsigned)a.col_mod - 1u);
  return (q / (unsigned)a.col_div) % (unsigned)a.col_mod;
}

// One tile of L lanes starting at lane q0; L P threads, all of them call it.
// HALF (chirp operators): the valid inputs and the kept outputs all lie in the
// lower half of the lane, as in every Bluestein convolution (n <= M / 2), so
// points q >= 8 are never loaded nor stored.
// Plain complex data are read through L2: each point is read once, and a batch tile
// may read what another CTA of the same launch wrote.
// IN: IN_C (also IN_R, and IN_HERM on contiguous lanes), IN_FRAME, IN_CHIRP
// (also IN_CHIRP_R), IN_STEP; OUT: OUT_C (also OUT_RE; on contiguous lanes
// OUT_TRUNC and the first store_cols points; on strided lanes the mirrored
// columns of a Hermitian pass), OUT_STEP, OUT_CHIRP (also OUT_CHIRP_RE).
template <class T, int N, int L, int FORM, int MODE, int IN, int OUT, bool HALF = false>
__device__ __forceinline__ void fx_tile(const KArgs<T>& a, unsigned q0, typename CT<T>::type* sm) {
  using C = typename CT<T>::type;
  using E = FxEng<T, N>;
  constexpr int P = E::P, EP = E::EP;
  constexpr bool LMA = FORM == FX_COLS, LMB = FORM != FX_ROWS;
  constexpr int LD = fx_ld(N, L, LMB, (int)sizeof(C));
  constexpr bool WARP = FORM == FX_ROWS && P <= 32 && 32 % P == 0;
  const int tid = threadIdx.x;
  const int lA = LMA ? tid % L : tid / P, tA = LMA ? tid / L : tid % P;
  const int lB = LMB ? tid % L : tid / P, tB = LMB ? tid / L : tid % P;
  const unsigned lanes = (unsigned)a.lanes;
  const unsigned qA = q0 + lA, qB = q0 + lB;
  constexpr int QN = HALF ? EP / 2 : EP;
  C v[EP];
  // ── load: points tA + P q of lane lA ──
  if (qA < lanes) {
    const long long ib = fx_base(a.im, qA, a.fx_sh[0] >= 0 ? a.fx_sh[0] : -1);
    const long long es = FORM == FX_COLS ? a.im.es : 1;
    if constexpr (IN == IN_C) {
      if (a.in_op == IN_R) {
        const T* p = static_cast<const T*>(a.in) + ib + tA * es;
#pragma unroll
        for (int q = 0; q < EP; ++q) v[q] = C{p[(long long)(P * q) * es], (T)0};
      } else if (FORM == FX_ROWS && a.in_op == IN_HERM) {
        // half spectrum (N / 2 + 1 bins) expanded by Hermitian symmetry
        const C* p = static_cast<const C*>(a.in) + ib;
#pragma unroll
        for (int q = 0; q < EP; ++q) {
          const int i = tA + P * q;
          const bool up = 2 * i > N;
          C x = p[up ? N - i : i];
          if (up) x.y = -x.y;
          if (i > 0 && 2 * i != N) x = cscale(x, a.pair_w);
          v[q] = x;
        }
      } else {
        const C* p = static_cast<const C*>(a.in) + ib + tA * es;
#pragma unroll
        for (int q = 0; q < EP; ++q) v[q] = __ldcg(p + (long long)(P * q) * es);
      }
    } else if constexpr (IN == IN_FRAME) {
      const long long s = ib - a.frame_off + tA;
      const T* p = static_cast<const T*>(a.in) + s;
      const T* w = a.window + tA;
      if (s - tA >= 0 && s - tA + N <= a.nlen) {
#pragma unroll
        for (int q = 0; q < EP; ++q) v[q] = C{p[P * q] * __ldg(w + P * q), (T)0};
      } else {
#pragma unroll
        for (int q = 0; q < EP; ++q) {
          const long long j = s + P * q;
          v[q] = C{j >= 0 && j < a.nlen ? p[P * q] * w[P * q] : (T)0, (T)0};
        }
      }
    } else if constexpr (IN == IN_CHIRP) {
      // Bluestein / CZT premultiply: x[j] chirp[j], zero from nlen on
      const unsigned jm = FORM == FX_COLS ? (unsigned)a.jmul : 1u;
      const unsigned col = FORM == FX_COLS ? fx_col(a, qA) : 0u;
      const unsigned nlen = (unsigned)a.nlen;
      const unsigned j0 = (unsigned)tA * jm + col;
      const long long o0 = ib + tA * es;
      const bool cj = a.chirp_conj != 0, re = a.in_op == IN_CHIRP_R;
#pragma unroll
      for (int q = 0; q < QN; ++q) {
        const unsigned j = j0 + (unsigned)(P * q) * jm;
        C x = C{(T)0, (T)0};
        if (j < nlen) {
          const long long o = o0 + (long long)(P * q) * es;
          x = re ? C{static_cast<const T*>(a.in)[o], (T)0} : static_cast<const C*>(a.in)[o];
          const C c = __ldg(a.chirp + j);
          x = cj ? cmulc(x, c) : cmul(x, c);
        }
        v[q] = x;
      }
    } else {  // IN_STEP: times the conjugate step twiddle of (column, tA + P q)
      const unsigned cm = (unsigned)a.col_mod;
      const unsigned col = fx_col(a, qA);
      const C* p = static_cast<const C*>(a.in) + ib + tA * es;
#pragma unroll
      for (int q = 0; q < EP; ++q) v[q] = __ldcg(p + (long long)(P * q) * es);
      const C wa = __ldg(a.fx_a + (unsigned)tA * cm + col);
#pragma unroll
      for (int q = 0; q < EP; ++q) v[q] = cmulc(v[q], cmul(wa, __ldg(a.fx_b + (unsigned)q * cm + col)));
    }
  } else {
#pragma unroll
    for (int q = 0; q < EP; ++q) v[q] = C{(T)0, (T)0};
  }
  // ── stages ──
  C* const smA = sm + lA * LD;
  C* const smB = sm + lB * LD;
  if constexpr (MODE == FX_CONV) {
    fx_fwd<T, N, false, WARP, HALF>(v, smA, tA, smB, tB, a.fx_tw);
    const unsigned qc = qB < lanes ? qB : 0u;
    const C* sp = a.spec + tB;
    if (a.spec_ld) sp += (long long)fx_col(a, qc) * a.spec_ld;
#pragma unroll
    for (int q = 0; q < EP; ++q) v[q] = cmul(v[q], __ldg(sp + P * q));
    fx_transposed<T, N, true, WARP>(v, smB, tB, a.fx_tw);
  } else {
    fx_fwd<T, N, MODE == FX_INV, WARP, HALF && IN == IN_CHIRP>(v, smA, tA, smB, tB, a.fx_tw);
  }
  // ── store: points tB + P q of lane lB ──
  if (qB >= lanes) return;
  const long long es = FORM == FX_ROWS ? 1 : a.om.es;
  const long long ob = fx_base(a.om, qB, a.fx_sh[0] >= 0 ? a.fx_sh[1] : -1) + tB * es;
  const T sc = a.scale;
  if constexpr (OUT == OUT_C) {
    if (a.out_op == OUT_RE) {
      T* p = static_cast<T*>(a.out) + ob;
#pragma unroll
      for (int q = 0; q < EP; ++q) p[(long long)(P * q) * es] = v[q].x * sc;
    } else if (FORM == FX_ROWS && a.store_cols > 0) {
      // the first store_cols points (OUT_TRUNC: a half spectrum, paired bins weighted)
      C* p = static_cast<C*>(a.out) + ob;
      const T pw = a.out_op == OUT_TRUNC ? sc * a.pair_w : sc;
#pragma unroll
      for (int q = 0; q < EP; ++q) {
        const int i = tB + P * q;
        if (i < a.store_cols) p[P * q] = cscale(v[q], i > 0 && 2 * i != N ? pw : sc);
      }
    } else {
      C* p = static_cast<C*>(a.out) + ob;
#pragma unroll
      for (int q = 0; q < EP; ++q) p[(long long)(P * q) * es] = cscale(v[q], sc);
      if (FORM == FX_COLS && a.hm_cmax > 0) {
        // Hermitian input rows: column es - c is the conjugate of this one
        // read backwards, Y[k][es - c] = conj(Y[(N - k) mod N][c])
        const int c = (int)(qB % (unsigned)a.om.d2);
        if (c >= 1 && c <= a.hm_cmax) {
          C* m = static_cast<C*>(a.out) + fx_base(a.om, qB, a.fx_sh[0] >= 0 ? a.fx_sh[1] : -1) + a.om.es - 2 * c;
#pragma unroll
          for (int q = 0; q < EP; ++q) {
            const int k = tB + P * q;
            const C y = cscale(v[q], sc);
            m[(long long)(k ? N - k : 0) * es] = C{y.x, -y.y};
          }
        }
      }
    }
  } else if constexpr (OUT == OUT_STEP) {
    const unsigned cm = (unsigned)a.col_mod;
    const unsigned col = fx_col(a, qB);
    const bool cj = a.tw_conj != 0;
    C* p = static_cast<C*>(a.out) + ob;
    const C wa = __ldg(a.fx_a + (unsigned)tB * cm + col);
#pragma unroll
    for (int q = 0; q < EP; ++q) {
      const C w = cmul(wa, __ldg(a.fx_b + (unsigned)q * cm + col));
      p[(long long)(P * q) * es] = cscale(cj ? cmulc(v[q], w) : cmul(v[q], w), sc);
    }
  } else {  // OUT_CHIRP: postmultiply, outputs below nlen (nlen_out when set)
    const unsigned jm = FORM == FX_COLS ? (unsigned)a.jmul : 1u;
    const unsigned col = FORM == FX_COLS ? fx_col(a, qB) : 0u;
    const unsigned nlen = (unsigned)(a.nlen_out > 0 ? a.nlen_out : a.nlen);
    const C* ch = a.chirp_out ? a.chirp_out : a.chirp;
    const unsigned j0 = (unsigned)tB * jm + col;
    const bool cj = a.chirp_conj != 0, re = a.out_op == OUT_CHIRP_RE;
#pragma unroll
    for (int q = 0; q < QN; ++q) {
      const unsigned j = j0 + (unsigned)(P * q) * jm;
      if (j < nlen) {
        const C c = __ldg(ch + j);
        const C y = cscale(cj ? cmulc(v[q], c) : cmul(v[q], c), sc);
        const long long o = ob + (long long)(P * q) * es;
        if (re) static_cast<T*>(a.out)[o] = y.x;
        else static_cast<C*>(a.out)[o] = y;
      }
    }
  }
}

// Lanes per tile of each length and form.  Powers of two: 128 threads for
// contiguous lanes (more CTAs of fewer lanes overlap their load, compute and
// store phases better: STFT frames of 1024 points complex128 87 -> 78 us against
// 256 threads), 256 threads with a lane-minor side, whose rows keep at least 64
// bytes (512 threads for 1024 complex64).  Odd lengths: about 256 threads, rows
// of 128 bytes while that takes at most 512 threads.
template <class T, int N, int FORM> struct FxTile {
  static constexpr int P = FxEng<T, N>::P;
  static constexpr bool P2 = fx_pow2(N);
  static constexpr int base = FORM == FX_ROWS && P2 ? 128 : 256;
  static constexpr int wide = sizeof(T) == 8 ? 8 : 16;  // 128-byte rows
  static constexpr int minL = FORM == FX_ROWS ? 1 : P2 ? (N > 1024 ? wide / 4 : wide / 2) : wide * P <= 512 ? wide : 8;
  static constexpr int L = FORM != FX_ROWS && !P2 ? minL : base / P > minL ? base / P : minL;
  static constexpr int threads = L * P;
  static constexpr size_t smem =
      (size_t)L * fx_ld(N, L, FORM != FX_ROWS, (int)sizeof(typename CT<T>::type)) * sizeof(typename CT<T>::type);
};

}  // namespace afc
