// afc_engine.cuh -- the shared-memory Stockham engine behind every transform.
//
// One CTA transforms L lanes (independent 1D transforms of length n).  Each
// lane is worked on by P threads (lane-major: tid = l * P + t).  A transform
// is a list of Stockham stages; stage s has radix R and Ns = product of the
// radices before it (the formulation of radix_composite/core.rs:169-183):
//
//   butterfly j in [0, n/R), k = j mod Ns
//   read    x[j + r * n/R]                     r = 0..R-1
//   twiddle x_r *= W_{Ns R}^{r k}               (forward W = exp(-2 pi i / .))
//   R-point DFT
//   write   y[(j - k) * R + k + r * Ns]
//
// Stages ping-pong between two shared buffers per lane (or read global memory
// directly in stage 0 and write it directly in the last stage).  Each thread
// walks its butterflies j = t, t + P, ... one at a time, so only one radix-R
// butterfly is live in registers and one barrier separates stages.  For
// contiguous lanes the direct stage-0 read and last-stage write are coalesced
// (consecutive threads touch consecutive elements); strided lanes and
// operators with index maps (chirps, gathers, twiddles, truncation) are staged
// through shared memory by cooperative copies in the kernels.
//
// Shared index of element i: i + (i >> psh), see StageList.
#pragma once
#include <cstdint>
#include "afc_butterfly.cuh"

namespace afc {

constexpr int kMaxStages = 24;

struct StageDesc {
  int R;
  int Ns;
  int twoff;  // offset (in complex elements) of this stage's twiddles, stored r-major: [(r-1) Ns + k]
  unsigned mg;  // ceil(2^32 / Ns) for Ns > 1: j / Ns = umulhi(j, mg) while j Ns < 2^32
};

struct StageList {
  int n;
  int nst;
  // shared index of element i: i + (i >> psh).  Powers of two: 4 (one pad
  // element every 16 breaks the stride-R conflicts of stage outputs); other
  // lengths start with an odd or composite radix whose outputs spread over the
  // banks, and run unpadded (31: no element).
  int psh;
  StageDesc st[kMaxStages];
};

// j mod Ns for a butterfly index j.
__device__ __forceinline__ int stage_mod(int j, int Ns, unsigned mg) {
  return Ns > 1 ? j - Ns * (int)__umulhi((unsigned)j, mg) : 0;
}
// Distance of r strides d in the shared layout.  For powers of two spad(i + r d)
// splits into spad(i) + spad(r d) (i below d or both multiples of 16), and
// unpadded lists are linear, so a butterfly's addresses are one base plus terms
// that do not depend on the thread.
template <bool PAD> __device__ __forceinline__ int stage_off(int r, int d) { return r * d + (PAD ? (r * d) >> 4 : 0); }
template <bool PAD> __device__ __forceinline__ int stage_idx(int i) { return i + (PAD ? i >> 4 : 0); }
// A stride the compiler cannot lift out of the butterfly loop: a thread runs one
// or two butterflies per stage, and R lifted offsets cost R registers each way.
__device__ __forceinline__ int stage_stride(int d) {
  asm volatile("" : "+r"(d));
  return d;
}

// Lane q -> base offset (in elements):  c = q % d2, b = (q / d2) % d1, a = q / (d1 d2),
// base = a*s0 + b*s1 + c*s2.  Element i of the lane lives at base + i*es.
// With an offset table (uneven batches): base = off[q / d2] + (q % d2) * s2.
struct LaneMap {
  long long d1, d2;
  long long s0, s1, s2;
  long long es;
  const long long* off;
  __host__ __device__ __forceinline__ long long base(long long q) const {
    if (off) return off[q / d2] + (q % d2) * s2;
    long long c = q % d2;
    long long t = q / d2;
    long long b = t % d1;
    long long a = t / d1;
    return a * s0 + b * s1 + c * s2;
  }
};

__host__ __device__ __forceinline__ int spad(int i, int psh) { return i + (i >> psh); }

// Number of shared buffers a stage list needs per lane, given whether the
// input is staged into shared memory and whether the output is staged out.
__host__ __device__ inline int engine_buffers(int nst, bool stage_in, bool stage_out) {
  if (nst == 0) return 1;
  int in_buf = stage_in ? 0 : -1, maxb = stage_in ? 0 : -1;
  for (int i = 0; i < nst; ++i) {
    const bool last = i == nst - 1;
    if (last && !stage_out) break;
    const int ob = in_buf == 0 ? 1 : 0;
    maxb = ob > maxb ? ob : maxb;
    in_buf = ob;
  }
  return maxb + 1 > 0 ? maxb + 1 : 1;
}

// One stage of one lane.  src == nullptr: read global through cx; dst ==
// nullptr: write global through cx.  Index arithmetic per butterfly, not per
// element: a multiply for j mod Ns, one base on each side.
template <int R, bool INV, bool PAD, class Ctx, class C>
__device__ __forceinline__ void stage(const Ctx& cx, const C* __restrict__ src, C* __restrict__ dst, int n,
                                      const StageDesc& sd, const C* __restrict__ tw, int t, int P) {
  const int nb = n / R;
  for (int j = t; j < nb; j += P) {
    const int d = stage_stride(nb), Ns = stage_stride(sd.Ns);
    C v[R];
    if (src) {
      const C* p = src + stage_idx<PAD>(j);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[stage_off<PAD>(r, d)];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = cx.gload(j + r * d);
    }
    const int k = stage_mod(j, Ns, sd.mg);
    if (Ns > 1) {
      const C* w = tw + k;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        const C wr = w[(r - 1) * Ns];
        v[r] = INV ? cmulc(v[r], wr) : cmul(v[r], wr);
      }
    }
    DFT<R, INV>::run(v);
    const int o = (j - k) * R + k;
    if (dst) {
      C* p = dst + stage_idx<PAD>(o);
#pragma unroll
      for (int r = 0; r < R; ++r) p[stage_off<PAD>(r, Ns)] = v[r];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) cx.gstore(o + r * Ns, v[r]);
    }
  }
}

// Runs every stage of `sl` for this thread's lane.  buf0/buf1: the lane's
// shared buffers; stage_in: the input already sits in buf0; stage_out: leave
// the result in shared memory.  Returns the buffer holding the result when
// stage_out (nullptr otherwise).  Ends with a barrier after every stage.
template <bool INV, class Ctx, class C>
__device__ __forceinline__ C* run_stages(const Ctx& cx, const StageList& sl, const C* __restrict__ tw, int t, int P,
                                         C* buf0, C* buf1, bool stage_in, bool stage_out) {
  const int nst = sl.nst;
  C* cur = stage_in ? buf0 : nullptr;
  if (nst == 0) {  // n = 1: a (scaled / converted) copy
    if (t == 0) {
      const C v = cur ? cur[0] : cx.gload(0);
      if (stage_out) buf0[0] = v;
      else cx.gstore(0, v);
    }
    __syncthreads();
    return stage_out ? buf0 : nullptr;
  }
  for (int i = 0; i < nst; ++i) {
    const bool last = i == nst - 1;
    C* nxt = (last && !stage_out) ? nullptr : (cur == buf0 ? buf1 : buf0);
    const StageDesc s = sl.st[i];
    const C* twi = tw + s.twoff;
#define AFC_ST(R, PAD) stage<R, INV, PAD>(cx, cur, nxt, sl.n, s, twi, t, P)
    if (sl.psh == 4) {  // a power of two
      switch (s.R) {
        case 2: AFC_ST(2, true); break;
        case 4: AFC_ST(4, true); break;
        case 8: AFC_ST(8, true); break;
        case 16: AFC_ST(16, true); break;
        default: break;
      }
    } else {
      switch (s.R) {
        case 2: AFC_ST(2, false); break;
        case 3: AFC_ST(3, false); break;
        case 4: AFC_ST(4, false); break;
        case 5: AFC_ST(5, false); break;
        case 6: AFC_ST(6, false); break;
        case 7: AFC_ST(7, false); break;
        case 8: AFC_ST(8, false); break;
        case 9: AFC_ST(9, false); break;
        case 10: AFC_ST(10, false); break;
        case 12: AFC_ST(12, false); break;
        case 14: AFC_ST(14, false); break;
        case 15: AFC_ST(15, false); break;
        case 11: AFC_ST(11, false); break;
        case 13: AFC_ST(13, false); break;
        case 16: AFC_ST(16, false); break;
        default: break;
      }
    }
#undef AFC_ST
    __syncthreads();
    cur = nxt;
  }
  return cur;
}

}  // namespace afc
