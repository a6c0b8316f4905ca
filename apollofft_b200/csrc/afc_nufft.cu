// afc_nufft.cu -- Kaiser-Bessel spreading / interpolation for the 1D NUFFT
// (apollo-nufft NufftPlan1D, transform/dimension_1d.rs:156-272), and below for
// the 3D one.
//
// Type 1: every non-uniform point adds value * phi(p - d) to the 2w+1
// oversampled grid cells around round(m x / L) (atomic adds, after sorting where
// that pays), the grid goes through this library's forward FFT, and the n output
// bins are the grid bins k_signed mod m times the deconvolution factors.
// Type 2: the n coefficients times the deconvolution factors are placed at
// k_signed mod m, the grid goes through the unnormalized inverse FFT, and every
// point gathers its 2w+1 cells weighted by phi.  phi is the reference's kernel
// phi(x) = I0(beta sqrt(1 - (x/w)^2)) / I0(beta), |x| < w, with I0 by its power
// series (kaiser_bessel.rs:55-116), evaluated in FP64 per tap as one polynomial.
#include <cuda_runtime.h>
#include "afc_internal.h"

namespace afc {

// I0(z) = sum_k ((z/2)^2)^k / (k!)^2: term_k = term_{k-1} (z/2)^2 / k^2, the
// ratios from a table of 1/k^2 (so the running product is a chain of
// multiplies, not divides), summed four terms at a time until the last of them
// drops below epsilon of the sum (at most 256 terms).  The terms the reference
// would not add are below epsilon of the sum.
struct NuInvSquares {
  double v[257];
  constexpr NuInvSquares() : v() {
    for (int k = 1; k <= 256; ++k) v[k] = 1.0 / ((double)k * (double)k);
  }
};
__constant__ NuInvSquares c_nu_inv_k2 = NuInvSquares();

__device__ __forceinline__ double nu_i0(double z) {
  const double scaled = 0.25 * z * z;
  double sum = 1.0, term = 1.0;
  for (int k = 1; k <= 256; k += 4) {
    const double q0 = scaled * c_nu_inv_k2.v[k], q1 = scaled * c_nu_inv_k2.v[k + 1];
    const double q2 = scaled * c_nu_inv_k2.v[k + 2], q3 = scaled * c_nu_inv_k2.v[k + 3];
    term *= q0;
    sum += term;
    term *= q1;
    sum += term;
    term *= q2;
    sum += term;
    term *= q3;
    sum += term;
    if (term <= 2.220446049250313e-16 * sum) break;
  }
  return sum;
}

__device__ __forceinline__ double nu_kb(double x, double w, double beta, double i0b) {
  const double u = x / w;
  const double u2 = u * u;
  if (u2 >= 1.0) return 0.0;
  return nu_i0(beta * sqrt(1.0 - u2)) / i0b;
}

// phi as a polynomial: I0's series in (z/2)^2 = (beta / 2w)^2 s, s = w^2 - x^2,
// divided by I0(beta), has the fixed positive coefficients NuPoly::c, so Horner
// needs one FMA per term instead of the running product's three operations, no
// division and no square root; s = (w - x)(w + x) does not cancel at the edge.  The
// first dropped term is below 2^-60 of phi(0) = 1.  At w = 6 (44 terms) the series'
// weights were about half of a 1D call.  K = 0 (kernels too wide for the table): the
// series.
__device__ __forceinline__ double nu_phi(const NuPoly& f, double x, double w, double beta, double i0b) {
  if (f.K == 0) return nu_kb(x, w, beta, i0b);
  const double s = (w - x) * (w + x);
  if (s <= 0.0) return 0.0;  // a NaN position gives NaN weights
  double a = f.c[f.K - 1];
#pragma unroll 5
  for (int k = f.K - 2; k >= 0; --k) a = fma(a, s, f.c[k]);
  return a;
}

// Taps p0 .. p0 + 3 of one axis at once (four independent chains per coefficient).
__device__ __forceinline__ void nu_phi4(const NuPoly& f, int p0, double d, int w, double beta, double i0b, double* o) {
  if (f.K == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = nu_kb((double)(p0 + i - w) - d, (double)w, beta, i0b);
    return;
  }
  double s[4], a[4];
  const double c0 = f.c[f.K - 1];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double x = (double)(p0 + i - w) - d;
    s[i] = ((double)w - x) * ((double)w + x);
    a[i] = c0;
  }
#pragma unroll 5
  for (int k = f.K - 2; k >= 0; --k) {
    const double c = f.c[k];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = fma(a[i], s[i], c);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = s[i] <= 0.0 ? 0.0 : a[i];
}

// All T taps of one axis in one walk over the coefficients (T independent chains:
// a coefficient load feeds T FMAs instead of four, and no tap is evaluated past
// the kernel).
template <int T>
__device__ __forceinline__ void nu_phi_all(const NuPoly& f, double d, double beta, double i0b, double (&o)[T]) {
  constexpr int w = T / 2;
  if (f.K == 0) {
#pragma unroll
    for (int i = 0; i < T; ++i) o[i] = nu_kb((double)(i - w) - d, (double)w, beta, i0b);
    return;
  }
  double s[T];
  const double c0 = f.c[f.K - 1];
#pragma unroll
  for (int i = 0; i < T; ++i) {
    const double x = (double)(i - w) - d;
    s[i] = ((double)w - x) * ((double)w + x);
    o[i] = c0;
  }
#pragma unroll 2
  for (int k = f.K - 2; k >= 0; --k) {
    const double c = f.c[k];
#pragma unroll
    for (int i = 0; i < T; ++i) o[i] = fma(o[i], s[i], c);
  }
#pragma unroll
  for (int i = 0; i < T; ++i) o[i] = s[i] <= 0.0 ? 0.0 : o[i];
}

struct NuGeom {
  long long m;     // oversampled length
  int w;           // kernel half width
  double beta, i0b;
  double len;      // periodic domain length n dx
  NuPoly f;
};

// Position -> (m0, d): x mod L (Euclidean), t = m x / L, m0 = round(t) (half
// away from zero), d = t - m0.
__device__ __forceinline__ void nu_place(const NuGeom& g, double x, long long& m0, double& d) {
  double r = fmod(x, g.len);
  if (r < 0.0) r += g.len;
  const double t = (double)g.m * r / g.len;
  const double rt = round(t);
  m0 = (long long)rt;
  d = t - rt;
}

__device__ __forceinline__ long long nu_wrap(long long i, long long m) {
  long long r = i % m;
  return r < 0 ? r + m : r;
}

__global__ void nu_spread(const __grid_constant__ NuGeom g, const double* __restrict__ pos, const double2* __restrict__ val, long long npts,
                          double2* grid) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < npts; j += (long long)gridDim.x * blockDim.x) {
    long long m0;
    double d;
    nu_place(g, pos[j], m0, d);
    const double2 v = val[j];
    long long cell = nu_wrap(m0 - g.w, g.m);
    for (int p = 0; p <= 2 * g.w; p += 4) {
      double wt[4];
      nu_phi4(g.f, p, d, g.w, g.beta, g.i0b, wt);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (p + i <= 2 * g.w && wt[i] != 0.0) {
          double2* c = grid + cell;
          atomicAdd(&c->x, v.x * wt[i]);
          atomicAdd(&c->y, v.y * wt[i]);
        }
        if (++cell >= g.m) cell -= g.m;
      }
    }
  }
}

// Spreading of sorted points.  The kernel above is bound by its FP64 atomics
// (2 (2w + 1) per point, about 140 G/s), and crowded points contend for the same
// cells.  Sorted by bins of cells, the 32 points of a warp fall within a few
// cells of each other: each lane evaluates its point's weights, then the warp
// takes a window of 32 cells, one per lane, and every lane sums what the points
// of the window add to its cell before one atomic add: about 20 cells per 32
// points and window instead of 32 (2w + 1).  Points too far from the first one
// wait for the next window.
constexpr int kNu1Warps = 4;
__host__ __device__ constexpr size_t nu1_smem(int T) {
  return (size_t)kNu1Warps * ((size_t)T * 33 * sizeof(double) + 32 * (sizeof(double2) + sizeof(int)));
}

__global__ void nu1_bin(const __grid_constant__ NuGeom g, int width, const double* __restrict__ pos, long long npts,
                        int* __restrict__ cnt, int* __restrict__ bin, int* __restrict__ rank) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < npts; j += (long long)gridDim.x * blockDim.x) {
    long long m0;
    double d;
    nu_place(g, pos[j], m0, d);
    const int b = (int)nu_wrap(m0, g.m) / width;
    bin[j] = b;
    rank[j] = atomicAdd(&cnt[b], 1);
  }
}

// TC: taps at compile time (0: any width)
template <int TC>
__global__ void __launch_bounds__(32 * kNu1Warps) nu1_spread(const __grid_constant__ NuGeom g, const int* __restrict__ idx,
                                                             const double* __restrict__ pos,
                                                             const double2* __restrict__ val, long long npts,
                                                             double2* grid) {
  extern __shared__ __align__(16) unsigned char nu_smem[];
  const int T = TC ? TC : 2 * g.w + 1, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double2* const sv = reinterpret_cast<double2*>(nu_smem) + 32 * wid;
  double* const sw = reinterpret_cast<double*>(reinterpret_cast<double2*>(nu_smem) + 32 * kNu1Warps) + wid * T * 33;
  int* const sc = reinterpret_cast<int*>(reinterpret_cast<double*>(reinterpret_cast<double2*>(nu_smem) + 32 * kNu1Warps) +
                                         kNu1Warps * T * 33) + 32 * wid;
  const long long step = (long long)gridDim.x * kNu1Warps * 32;
  for (long long base = ((long long)blockIdx.x * kNu1Warps + wid) * 32; base < npts; base += step) {
    const bool valid = base + lane < npts;
    int c = 0;
    if (valid) {
      const int j = idx[base + lane];
      long long m0;
      double d;
      nu_place(g, pos[j], m0, d);
      c = (int)nu_wrap(m0, g.m);
      sv[lane] = val[j];
      if constexpr (TC > 0) {
        double o[TC];
        nu_phi_all<TC>(g.f, d, g.beta, g.i0b, o);
#pragma unroll
        for (int i = 0; i < TC; ++i) sw[i * 33 + lane] = o[i];
      } else {
        for (int p = 0; p < T; p += 4) {
          double o[4];
          nu_phi4(g.f, p, d, g.w, g.beta, g.i0b, o);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (p + i < T) sw[(p + i) * 33 + lane] = o[i];
        }
      }
      sc[lane] = c;
    }
    __syncwarp();
    unsigned rem = __ballot_sync(0xffffffffu, valid);
    while (rem) {
      const bool left = rem >> lane & 1;
      const int c0 = (int)__reduce_min_sync(0xffffffffu, left ? (unsigned)c : 0xffffffffu);
      const bool hit = left && c - c0 <= 31 - 2 * g.w;
      unsigned mask = __ballot_sync(0xffffffffu, hit);
      rem &= ~mask;
      double ax = 0.0, ay = 0.0;
      while (mask) {
        const int p = __ffs(mask) - 1;
        mask &= mask - 1;
        const int tap = lane - (sc[p] - c0);  // cell c0 - w + lane of point p
        const double2 v = sv[p];
        const double wt = tap >= 0 && tap < T ? sw[tap * 33 + p] : 0.0;
        if (wt != 0.0) {
          ax = fma(v.x, wt, ax);
          ay = fma(v.y, wt, ay);
        }
      }
      if (ax != 0.0 || ay != 0.0) {
        long long cell = (long long)c0 - g.w + lane;
        if (cell < 0) cell += g.m;
        if (cell >= g.m) cell -= g.m;
        atomicAdd(&grid[cell].x, ax);
        atomicAdd(&grid[cell].y, ay);
      }
    }
    __syncwarp();
  }
}

// TC: taps at compile time (0: any width)
template <int TC>
__global__ void __launch_bounds__(256) nu_interp(const __grid_constant__ NuGeom g, const double2* __restrict__ grid, const double* __restrict__ pos, long long npts,
                          double2* out) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < npts; j += (long long)gridDim.x * blockDim.x) {
    long long m0;
    double d;
    nu_place(g, pos[j], m0, d);
    double2 acc = make_double2(0.0, 0.0);
    long long cell = nu_wrap(m0 - g.w, g.m);
    if constexpr (TC > 0) {
      double wt[TC];
      nu_phi_all<TC>(g.f, d, g.beta, g.i0b, wt);
#pragma unroll
      for (int i = 0; i < TC; ++i) {
        const double2 c = grid[cell];
        if (wt[i] != 0.0) {
          acc.x += c.x * wt[i];
          acc.y += c.y * wt[i];
        }
        if (++cell >= g.m) cell -= g.m;
      }
      out[j] = acc;
      continue;
    }
    for (int p = 0; p <= 2 * g.w; p += 4) {
      double2 c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // the loads fly while the weights are evaluated
        c[i] = p + i <= 2 * g.w ? grid[cell] : make_double2(0.0, 0.0);
        if (++cell >= g.m) cell -= g.m;
      }
      double wt[4];
      nu_phi4(g.f, p, d, g.w, g.beta, g.i0b, wt);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (wt[i] != 0.0) {  // a tap outside the kernel adds nothing, whatever its cell holds
          acc.x += c[i].x * wt[i];
          acc.y += c[i].y * wt[i];
        }
      }
    }
    out[j] = acc;
  }
}

// k -> k_signed mod m (fft_signed_index: k <= n/2 stays, else k - n).
__device__ __forceinline__ long long nu_bin(long long k, long long n, long long m) {
  const long long ks = k <= n / 2 ? k : k - n;
  return nu_wrap(ks, m);
}

__global__ void nu_deconv_out(const double2* __restrict__ grid, const double* __restrict__ deconv, long long n,
                              long long m, double2* out) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const double2 c = grid[nu_bin(k, n, m)];
    const double f = deconv[k];
    out[k] = make_double2(c.x * f, c.y * f);
  }
}

__global__ void nu_place_coeffs(const double2* __restrict__ coeffs, const double* __restrict__ deconv, long long n,
                                long long m, double2* grid) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const double2 c = coeffs[k];
    const double f = deconv[k];
    grid[nu_bin(k, n, m)] = make_double2(c.x * f, c.y * f);
  }
}

// ─── 3D (apollo-nufft NufftPlan3D, transform/dimension_3d.rs:193-620) ───
// Separable kernel: weight = phi_x phi_y phi_z over T^3 taps, T = 2w + 1; grid
// C-order [ix][iy][iz] of size mx x my x mz, every m a power of two.
// One warp per point: the lanes evaluate the 3T axis weights into shared
// memory, then walk the T x T (py, pz) plane flattened over the 32 lanes for
// every px, so one warp instruction touches two or three contiguous runs of T
// cells (T = 13: 6 instructions per plane) instead of 32 scattered cells.
struct NuGeom3 {
  long long mx, my, mz;
  int w;
  double beta, i0b;
  double lx, ly, lz;
  NuPoly f;
};

constexpr int kNuMaxTaps = 65;       // T for w <= 32
constexpr int kNuWarps = 8;          // warps (points in flight) per 256-thread CTA

__device__ __forceinline__ double nu_axis_t(double x, double len, long long m) {
  double r = fmod(x, len);
  if (r < 0.0) r += len;
  return (double)m * r / len;
}

// Lanes fill wt[0..T) for one axis and return m0 (the same in every lane).
__device__ __forceinline__ long long nu_axis_weights(double x, double len, long long m, const NuGeom3& g, int lane,
                                                     double* wt) {
  const double t = nu_axis_t(x, len, m);
  const double rt = round(t);
  const double d = t - rt;
  for (int p = lane; p <= 2 * g.w; p += 32) wt[p] = nu_phi(g.f, (double)(p - g.w) - d, (double)g.w, g.beta, g.i0b);
  return (long long)rt;
}

struct NuPlaneWalk {  // lane's (py, pz) start and the constant stride of 32 flattened cells
  int py0, pz0, dpy, dpz, iters;
  __device__ NuPlaneWalk(int T, int lane)
      : py0(lane / T), pz0(lane % T), dpy(32 / T), dpz(32 % T), iters((T * T + 31) / 32) {}
};

__global__ void __launch_bounds__(32 * kNuWarps) nu_spread3(const __grid_constant__ NuGeom3 g, const double* __restrict__ pos,
                                                              const double2* __restrict__ val, long long npts,
                                                              double2* grid) {
  __shared__ double sw[kNuWarps][3][kNuMaxTaps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int T = 2 * g.w + 1;
  const NuPlaneWalk pw(T, lane);
  const long long mxm = g.mx - 1, mym = g.my - 1, mzm = g.mz - 1;
  double* wx = sw[wid][0];
  double* wy = sw[wid][1];
  double* wz = sw[wid][2];
  const long long warps = (long long)gridDim.x * kNuWarps;
  for (long long j = (long long)blockIdx.x * kNuWarps + wid; j < npts; j += warps) {
    const long long m0x = nu_axis_weights(pos[3 * j], g.lx, g.mx, g, lane, wx);
    const long long m0y = nu_axis_weights(pos[3 * j + 1], g.ly, g.my, g, lane, wy);
    const long long m0z = nu_axis_weights(pos[3 * j + 2], g.lz, g.mz, g, lane, wz);
    const double2 v = val[j];
    __syncwarp();
    for (int px = 0; px < T; ++px) {
      const double wxv = wx[px];
      if (wxv == 0.0) continue;
      double2* plane = grid + ((m0x + px - g.w) & mxm) * g.my * g.mz;
      int py = pw.py0, pz = pw.pz0;
      for (int it = 0; it < pw.iters; ++it) {
        if (py < T) {
          const double wt = wxv * wy[py] * wz[pz];
          if (wt != 0.0) {
            double2* c = plane + ((m0y + py - g.w) & mym) * g.mz + ((m0z + pz - g.w) & mzm);
            atomicAdd(&c->x, v.x * wt);
            atomicAdd(&c->y, v.y * wt);
          }
        }
        py += pw.dpy;
        pz += pw.dpz;
        if (pz >= T) pz -= T, ++py;
      }
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(32 * kNuWarps) nu_interp3(const __grid_constant__ NuGeom3 g, const double2* __restrict__ grid,
                                                              const double* __restrict__ pos, long long npts,
                                                              double2* out) {
  __shared__ double sw[kNuWarps][3][kNuMaxTaps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int T = 2 * g.w + 1;
  const NuPlaneWalk pw(T, lane);
  const long long mxm = g.mx - 1, mym = g.my - 1, mzm = g.mz - 1;
  double* wx = sw[wid][0];
  double* wy = sw[wid][1];
  double* wz = sw[wid][2];
  const long long warps = (long long)gridDim.x * kNuWarps;
  for (long long j = (long long)blockIdx.x * kNuWarps + wid; j < npts; j += warps) {
    const long long m0x = nu_axis_weights(pos[3 * j], g.lx, g.mx, g, lane, wx);
    const long long m0y = nu_axis_weights(pos[3 * j + 1], g.ly, g.my, g, lane, wy);
    const long long m0z = nu_axis_weights(pos[3 * j + 2], g.lz, g.mz, g, lane, wz);
    __syncwarp();
    double ax = 0.0, ay = 0.0;
    for (int px = 0; px < T; ++px) {
      const double wxv = wx[px];
      if (wxv == 0.0) continue;
      const double2* plane = grid + ((m0x + px - g.w) & mxm) * g.my * g.mz;
      int py = pw.py0, pz = pw.pz0;
      for (int it = 0; it < pw.iters; ++it) {
        if (py < T) {
          const double wt = wxv * wy[py] * wz[pz];
          if (wt != 0.0) {
            const double2 c = plane[((m0y + py - g.w) & mym) * g.mz + ((m0z + pz - g.w) & mzm)];
            ax += c.x * wt;
            ay += c.y * wt;
          }
        }
        py += pw.dpy;
        pz += pw.dpz;
        if (pz >= T) pz -= T, ++py;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, o);
      ay += __shfl_xor_sync(0xffffffffu, ay, o);
    }
    if (lane == 0) out[j] = make_double2(ax, ay);
    __syncwarp();
  }
}

// ─── tiled 3D spreading / interpolation ───
// Points are bucketed by the B^3 tile of cells that holds their centre cell
// round(t) mod m (the reference bucket-sorts its points too, sort_points_3d,
// dimension_3d.rs:74-117); one CTA per tile keeps the tile and its w-cell halo,
// E^3 cells with E = B + 2w, in shared memory.  Spreading: warp k owns the
// x-planes lx = k mod 16 of the tile and adds every point's taps on its planes
// with plain shared-memory read-modify-writes (no two warps share a cell),
// then the CTA adds its E^3 cells to the grid with coalesced atomics (tiles'
// halos overlap); grid atomics drop from (2w+1)^3 per point to E^3 per tile.
// Interpolation: the CTA loads its E^3 cells once, stages the weights of 64
// points at a time with all its threads, and one warp per point gathers from
// shared memory.
constexpr int kNuTileThreads = 512;
constexpr int kNuTileWarps = kNuTileThreads / 32;
constexpr int kNuChunk = 64;  // points whose weights a tile CTA stages at once

struct NuTiles {
  int B, E, nty, ntz;
  const int* off;  // ntiles + 1 offsets into idx
  const int* idx;  // point indices grouped by tile
};

__device__ __forceinline__ int nu_centre(double x, double len, long long m) {
  return (int)((long long)round(nu_axis_t(x, len, m)) & (m - 1));
}

__global__ void nu3_bin(const __grid_constant__ NuGeom3 g, int B, int nty, int ntz, const double* __restrict__ pos, long long npts,
                        int* __restrict__ cnt, int* __restrict__ tile, int* __restrict__ rank) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < npts; j += (long long)gridDim.x * blockDim.x) {
    const int cx = nu_centre(pos[3 * j], g.lx, g.mx);
    const int cy = nu_centre(pos[3 * j + 1], g.ly, g.my);
    const int cz = nu_centre(pos[3 * j + 2], g.lz, g.mz);
    const int t = ((cx / B) * nty + cy / B) * ntz + cz / B;
    tile[j] = t;
    rank[j] = atomicAdd(&cnt[t], 1);
  }
}

// Exclusive prefix sum of cnt[0..n) into off[0..n], one CTA of 1024 threads,
// each over a contiguous chunk.
__global__ void __launch_bounds__(1024) nu3_scan(const int* __restrict__ cnt, int* __restrict__ off, int n) {
  __shared__ int wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int per = (n + 1023) / 1024;
  const int lo = min(n, tid * per), hi = min(n, lo + per);
  int s = 0;
  for (int i = lo; i < hi; ++i) s += cnt[i];
  int v = s;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) wsum[wid] = v;
  __syncthreads();
  if (wid == 0) {
    int w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  int ex = v - s + (wid > 0 ? wsum[wid - 1] : 0);
  for (int i = lo; i < hi; ++i) {
    off[i] = ex;
    ex += cnt[i];
  }
  if (tid == 1023) off[n] = ex;
}

__global__ void nu3_scatter(const int* __restrict__ tile, const int* __restrict__ rank, const int* __restrict__ off,
                            long long npts, int* __restrict__ idx) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < npts; j += (long long)gridDim.x * blockDim.x)
    idx[off[tile[j]] + rank[j]] = (int)j;
}

struct NuTileCoord {
  int tx, ty, tz;
  __device__ NuTileCoord(int tile, const NuTiles& tl)
      : tx(tile / (tl.nty * tl.ntz)), ty((tile / tl.ntz) % tl.nty), tz(tile % tl.ntz) {}
};

// Axis-a weight of tap `tap` for the point at pos, and (lc non-null) the
// point's centre cell relative to the tile origin, in [0, B).
__device__ __forceinline__ double nu_tile_weight(const NuGeom3& g, const NuTiles& tl, const NuTileCoord& tc,
                                                 const double* pos, int a, int tap, int* lc) {
  const double len = a == 0 ? g.lx : a == 1 ? g.ly : g.lz;
  const long long m = a == 0 ? g.mx : a == 1 ? g.my : g.mz;
  const int t0 = a == 0 ? tc.tx : a == 1 ? tc.ty : tc.tz;
  const double t = nu_axis_t(pos[a], len, m);
  const double rt = round(t);
  if (lc) *lc = (int)((long long)rt & (m - 1)) - t0 * tl.B;
  return nu_phi(g.f, (double)(tap - g.w) - (t - rt), (double)g.w, g.beta, g.i0b);
}

// The lane's cells of a T x T (py, pz) plane: at most kNuTileIters, packed
// py << 8 | pz (-1 past the plane), fixed for the whole kernel.
constexpr int kNuTileIters = 12;  // ceil(T^2 / 32) for T <= 19 (w <= 9)

struct NuLaneCells {
  int pyz[kNuTileIters];
  __device__ NuLaneCells(int T, int lane) {
#pragma unroll
    for (int it = 0; it < kNuTileIters; ++it) {
      const int f = it * 32 + lane;
      pyz[it] = f < T * T ? ((f / T) << 8) | (f % T) : -1;
    }
  }
};

__global__ void __launch_bounds__(kNuTileThreads) nu3_spread_tiles(const __grid_constant__ NuGeom3 g, NuTiles tl,
                                                                    const double* __restrict__ pos,
                                                                    const double2* __restrict__ val, double2* grid) {
  extern __shared__ __align__(16) unsigned char nu_smem[];
  const int tile = blockIdx.x;
  const int start = tl.off[tile], end = tl.off[tile + 1];
  if (start == end) return;
  const int T = 2 * g.w + 1, E = tl.E, E2 = E * E, E3 = E2 * E;
  double2* acc = reinterpret_cast<double2*>(nu_smem);
  double* wts = reinterpret_cast<double*>(acc + E3);       // kNuChunk x 3 x T
  int* loc = reinterpret_cast<int*>(wts + kNuChunk * 3 * T);  // kNuChunk x 3
  for (int c = threadIdx.x; c < E3; c += kNuTileThreads) acc[c] = make_double2(0.0, 0.0);
  const NuTileCoord tc(tile, tl);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const NuLaneCells lc(T, lane);
  for (int base = start; base < end; base += kNuChunk) {
    const int cnt = min(kNuChunk, end - base);
    __syncthreads();  // zeroing done / previous chunk's weights consumed
    for (int e = threadIdx.x; e < cnt * 3 * T; e += kNuTileThreads) {
      const int p = e / (3 * T), r = e - p * 3 * T, a = r / T, tap = r - a * T;
      const long long j = tl.idx[base + p];
      wts[e] = nu_tile_weight(g, tl, tc, pos + 3 * j, a, tap, tap == 0 ? &loc[p * 3 + a] : nullptr);
    }
    __syncthreads();
    for (int p = 0; p < cnt; ++p) {
      const int lx0 = loc[p * 3], ly0 = loc[p * 3 + 1], lz0 = loc[p * 3 + 2];
      int px = (wid - lx0) % kNuTileWarps;
      if (px < 0) px += kNuTileWarps;
      if (px >= T) continue;  // warp-uniform: none of this point's planes is ours
      const double* wx = wts + p * 3 * T;
      const double* wy = wx + T;
      const double* wz = wy + T;
      const double2 v = val[tl.idx[base + p]];
      for (; px < T; px += kNuTileWarps) {
        const double wxv = wx[px];
        double2* plane = acc + (lx0 + px) * E2 + ly0 * E + lz0;
        // six of the lane's cells at a time: all loads first, then the adds and
        // stores (the lane's cells are distinct, and so are different lanes'),
        // so six shared-memory loads are in flight instead of one
#pragma unroll
        for (int h = 0; h < kNuTileIters; h += 6) {
          if (h * 32 >= T * T) break;
          double2 cv[6];
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            const int f = lc.pyz[h + i];
            if (f >= 0) cv[i] = plane[(f >> 8) * E + (f & 255)];
          }
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            const int f = lc.pyz[h + i];
            if (f >= 0) {
              const double wt = wxv * wy[f >> 8] * wz[f & 255];
              cv[i].x += v.x * wt;
              cv[i].y += v.y * wt;
              plane[(f >> 8) * E + (f & 255)] = cv[i];
            }
          }
        }
      }
      __syncwarp();  // the next point's lanes may touch the cells written here
    }
  }
  __syncthreads();
  const long long mxm = g.mx - 1, mym = g.my - 1, mzm = g.mz - 1;
  const long long gx0 = (long long)tc.tx * tl.B - g.w, gy0 = (long long)tc.ty * tl.B - g.w,
                  gz0 = (long long)tc.tz * tl.B - g.w;
  for (int c = threadIdx.x; c < E3; c += kNuTileThreads) {
    const double2 a = acc[c];
    if (a.x == 0.0 && a.y == 0.0) continue;
    const int cx = c / E2, cy = (c / E) % E, cz = c % E;
    double2* d = grid + (((gx0 + cx) & mxm) * g.my + ((gy0 + cy) & mym)) * g.mz + ((gz0 + cz) & mzm);
    atomicAdd(&d->x, a.x);
    atomicAdd(&d->y, a.y);
  }
}

// ─── 3D spreading and interpolation by boxes of cells ───
// The tile kernels are bound by shared memory (a 16-byte cell per tap, read and
// for spreading written back) and spreading adds every tile's halo to the grid
// with atomics, 15 times the cells at w = 6.  Here the cells stay in registers
// and the points move: a warp owns a box of 8 x 4 x 8 cells and meets every
// point whose taps reach it (25 boxes per point at w = 6).  Per box the sums are
// small FP64 matrix products (mma m8n8k4):
//   spreading      C[x][z] += wx[point][x] (v wy wz)[point][z], 4 points at a
//                  time, for each y and for both parts of v;
//   interpolation  D[point][z] = sum_x wx[point][x] cell[x][z], 8 points at a
//                  time, then summed over y and z with their weights.
// One operand element per lane feeds 8 FMAs.  Measured at 2^18 uniform points on
// 128^3 cells, w = 6 (kernel alone): spreading by tiles 1650 us, by boxes with scalar
// FMAs, bound by the broadcast weight loads, 1095, by these 612; interpolation by
// tiles 784 us, by boxes 713 and 23 for the sums, bound by the shared-memory loads
// ahead of each group (the FP64 pipe is 6-8 % busy).  Tiles are one CTA each, so for
// crowded points the boxes are up to 40 times as fast at spreading and 14 at
// interpolation (16^3 modes, w = 6, 2^17 points).
//  nu3_points: one record per point in tile order: value, centre, index, and the
//              axis weights between runs of seven zeros, so no tap is range-checked;
//  nu3_boxes:  a CTA of 8 warps owns 16 x 8 x 16 cells and streams the records of
//              the tiles within w cells of it through shared memory, the next chunk
//              in flight while one is worked on.  Each warp lists the records that
//              meet its box and takes them in groups.
//  nu3_collect: interpolation only.  A CTA adds up its eight boxes' parts of a
//              point in one order and stores the sum in a slot of the point that
//              its place relative to the point's first tap determines (7.7 CTAs
//              per point on average at w = 6); this adds the slots in order.  So a
//              value is the same bits whatever the order the CTAs ran in.
// Boxes partition the grid: spreading writes each cell once, without atomics
// unless a box's points are split over CTAs.
constexpr int kNuBoxThreads = 256;
// chunk and CTAs per SM measured at 2^18 points on 128^3 cells, w = 6 (spreading /
// interpolation with atomics): 32 points, three CTAs 798 / 900 us for the whole
// call, 64 points, two CTAs 845 / 927, 32 points, two CTAs 917 / 1027
constexpr int kNuBoxChunk = 32;
constexpr int kNuBoxRuns = 64;  // contiguous runs of candidate points per CTA

// Record: v.x, v.y, centre cells and index (four ints), then x, y and z weights.
__host__ __device__ constexpr int nu_xo(int) { return 11; }
__host__ __device__ constexpr int nu_yo(int T) { return 18 + T; }
__host__ __device__ constexpr int nu_zo(int T) { return 25 + 2 * T; }
__host__ __device__ constexpr int nu_rec(int T) { return (32 + 3 * T + 1) / 2 * 2; }
constexpr int kNuZeros = 16;  // a block of zeros: the record of the slots that fill up a group
__host__ __device__ constexpr int nu_list() { return (kNuBoxChunk + 16) * 4; }  // ints per warp
// The CTA blocks of 16 x 8 x 16 cells that the taps of a point with centre cell c
// reach along an axis of nb blocks of 2^sh cells: the first (c - w) >> sh, then
// upward, wrapping.
__host__ __device__ constexpr int nu_slots(int w, int sh) { return ((2 * w + (1 << sh) - 1) >> sh) + 1; }  // at most
__host__ __device__ constexpr int nu_slots3(int w) { return nu_slots(w, 4) * nu_slots(w, 3) * nu_slots(w, 4); }
__device__ __forceinline__ int nu_blocks(int c, int w, int sh, int nb) {
  return min(nb, ((c + w) >> sh) - ((c - w) >> sh) + 1);
}

__device__ __forceinline__ void nu_cp16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}

// Block of kNuPts points, three threads each (one per axis): the records are put
// together in shared memory and stored whole (rows written straight to global
// memory were 13 eight-byte stores per thread to 32 places each: 97 us at 2^18
// points).  val null (interpolation): no value in the record.
constexpr int kNuPts = 64;
template <int T>
__global__ void __launch_bounds__(3 * kNuPts) nu3_points(const __grid_constant__ NuGeom3 g, const int* __restrict__ idx,
                                                         const double* __restrict__ pos,
                                                         const double2* __restrict__ val, int npts,
                                                         double* __restrict__ rec) {
  constexpr int R = nu_rec(T);
  __shared__ __align__(16) double sm[kNuPts * R];
  for (int i = threadIdx.x; i < kNuPts * R; i += 3 * kNuPts) sm[i] = 0.0;
  const int p = threadIdx.x / 3, a = threadIdx.x - 3 * p;
  for (int base = blockIdx.x * kNuPts; base < npts; base += gridDim.x * kNuPts) {
    const int cnt = min(kNuPts, npts - base);
    __syncthreads();  // zeroed / the previous records are stored
    if (p < cnt) {
      const int j = idx[base + p];
      const long long m = a == 0 ? g.mx : a == 1 ? g.my : g.mz;
      const double t = nu_axis_t(pos[3ll * j + a], a == 0 ? g.lx : a == 1 ? g.ly : g.lz, m);
      const double rt = round(t);
      double* r = sm + p * R;
      double* w = r + (a == 0 ? nu_xo(T) : a == 1 ? nu_yo(T) : nu_zo(T));
      double o[T];
      nu_phi_all<T>(g.f, t - rt, g.beta, g.i0b, o);
#pragma unroll
      for (int i = 0; i < T; ++i) w[i] = o[i];
      int* c = reinterpret_cast<int*>(r + 2);
      c[a] = (int)((long long)rt & (m - 1));
      if (a == 0) {
        const double2 v = val ? val[j] : make_double2(0.0, 0.0);
        r[0] = v.x;
        r[1] = v.y;
        c[3] = j;
      }
    }
    __syncthreads();
    const double2* s2 = reinterpret_cast<const double2*>(sm);
    double2* d2 = reinterpret_cast<double2*>(rec + (long long)base * R);
    for (int i = threadIdx.x; i < cnt * R / 2; i += 3 * kNuPts) d2[i] = s2[i];
  }
}

// D += A B: A 8 x 4 (row lane / 4, column lane % 4), B 4 x 8 (row lane % 4,
// column lane / 4), D 8 x 8 (row lane / 4, columns 2 (lane % 4) and the next).
__device__ __forceinline__ void nu_mma(double2& d, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d.x), "+d"(d.y)
               : "d"(a), "d"(b));
}

// SPREAD: records -> cells (add: the cells may be shared with other CTAs);
// else: cells -> a slot of `out` per point and CTA that its taps reach.
template <bool SPREAD>
__global__ void __launch_bounds__(kNuBoxThreads, 3)
    nu3_boxes(int mx, int my, int mz, int w, const int* __restrict__ off, const double* __restrict__ rec,
              double2* __restrict__ grid, double2* __restrict__ out, int add) {
  extern __shared__ __align__(16) double nu_sm[];
  __shared__ int run_start[kNuBoxRuns], run_pre[kNuBoxRuns + 1];
  __shared__ int s_dst[2][kNuBoxChunk];  // !SPREAD: where the CTA's sum of each point goes, by chunk parity
  const int T = 2 * w + 1, S = nu_rec(T);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nby = my / 8, nbz = mz / 16;
  const int b = blockIdx.x;
  const int gx0 = b / (nby * nbz) * 16, gy0 = b / nbz % nby * 8, gz0 = b % nbz * 16;
  // candidate tiles (8 cells a side): rows along z are runs of the sorted points
  const int tx = mx / 8, ty = my / 8, tz = mz / 8, wt = (w + 7) / 8;
  const int cx = min(tx, 2 + 2 * wt), cy = min(ty, 1 + 2 * wt), cz = min(tz, 2 + 2 * wt);
  const int bx = gx0 / 8 - wt, by = gy0 / 8 - wt, bz = (gz0 / 8 - wt) & (tz - 1);
  const int nrun = cx * cy * 2;  // a run may wrap: two pieces
  if (tid < nrun) {
    const int row = tid >> 1;
    const int base = (((bx + row / cy) & (tx - 1)) * ty + ((by + row % cy) & (ty - 1))) * tz;
    const int first = min(cz, tz - bz);  // tiles before the wrap
    const int lo = tid & 1 ? base : base + bz, hi = tid & 1 ? base + cz - first : base + bz + first;
    run_start[tid] = off[lo];
    run_pre[tid + 1] = off[hi] - off[lo];
  }
  const int ZB = 2 * kNuBoxChunk * S;  // the zero block
  if (tid < kNuZeros) nu_sm[ZB + tid] = 0.0;
  int4* const list = reinterpret_cast<int4*>(nu_sm + ZB + kNuZeros) + wid * (kNuBoxChunk + 16);
  __syncthreads();
  if (tid == 0) {
    run_pre[0] = 0;
    for (int i = 0; i < nrun; ++i) run_pre[i + 1] += run_pre[i];
  }
  __syncthreads();
  const int total = run_pre[nrun];
  const int nchunk = (total + kNuBoxChunk - 1) / kNuBoxChunk;
  int c = blockIdx.y;
  if (c >= nchunk) return;
  // a few threads per record, 16 bytes a copy.  The points of a chunk are nchunk
  // apart, so it samples all candidate tiles and the warps of the CTA meet about
  // as many of its points each (in run order a chunk is a tile, which some boxes
  // meet whole and others not at all)
  auto stage = [&](int ch, int slot) {
    constexpr int TPP = kNuBoxThreads / kNuBoxChunk;  // threads per record
    const int p = tid / TPP, ord = p * nchunk + ch;
    if (ord < total) {
      int lo = 0, hi = nrun;  // last run with run_pre <= ord
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (run_pre[mid] <= ord) lo = mid;
        else hi = mid;
      }
      const double* r = rec + (long long)(run_start[lo] + ord - run_pre[lo]) * S;
      double* d = nu_sm + (slot * kNuBoxChunk + p) * S;
      for (int i = 2 * (tid % TPP); i < S; i += 2 * TPP) nu_cp16(d + i, r + i);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // this warp's box; the lane's row and column in the products
  const int x0 = gx0 + (wid >> 2) * 8, y0 = gy0 + ((wid >> 1) & 1) * 4, z0 = gz0 + (wid & 1) * 8;
  const int lr = lane >> 2, lk = lane & 3;
  stage(c, 0);
  double2 acc[4][2];     // SPREAD: C[x = lr][z = 2 lk, 2 lk + 1] of row y, real and imaginary
  double cell[4][2][2];  // else: B[x = lk + 4 s][z = lr] of row y, real and imaginary
  // else: the boxes' parts of a chunk's points, by chunk parity, box and point
  double2* const part = reinterpret_cast<double2*>(nu_sm + ZB + kNuZeros + (kNuBoxThreads / 32) * nu_list() / 2);
  const long long sx = (long long)my * mz;
  if constexpr (SPREAD) {
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = make_double2(0.0, 0.0);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const double2 v = grid[(x0 + 4 * s + lk) * sx + (long long)(y0 + j) * mz + z0 + lr];
        cell[j][s][0] = v.x;
        cell[j][s][1] = v.y;
      }
  }
  // the parts of the chunk of this parity, by one warp, a lane per point; they are
  // next written two chunks on
  auto sum_parts = [&](int slot) {
    const int dst = s_dst[slot][lane];
    if (dst < 0) return;
    const double2* q = part + slot * 8 * kNuBoxChunk + lane;
    double2 v = q[0];
#pragma unroll
    for (int b8 = 1; b8 < 8; ++b8) {
      v.x += q[b8 * kNuBoxChunk].x;
      v.y += q[b8 * kNuBoxChunk].y;
    }
    out[dst] = v;
  };
  static_assert(kNuBoxThreads == 256 && kNuBoxChunk == 32, "8 boxes of a warp each, a lane per point of the chunk");
  bool any = false;
  int k = 0;
  for (; c < nchunk; ++k, c += gridDim.y) {
    const int slot = k & 1;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // this chunk is here, the one before it done by every warp
    if (c + (int)gridDim.y < nchunk) stage(c + gridDim.y, slot ^ 1);
    if (!SPREAD && k > 0 && wid == (k & 7)) sum_parts(slot ^ 1);
    // the chunk's records that meet this box: offsets of its first weights (in
    // doubles from nu_sm; a box may start up to seven zeros before a row)
    double2* const mine = part + (slot * 8 + wid) * kNuBoxChunk;
    const bool slots = !SPREAD && wid == (k + 4 & 7);  // this warp works out the points' slots
    int n = 0;
    {
      const int p = lane, rp = (slot * kNuBoxChunk + p) * S;
      bool hit = false;
      int4 e = make_int4(0, 0, 0, 0);
      if (p * nchunk + c < total) {
        const int4 cc = *reinterpret_cast<const int4*>(nu_sm + rp + 2);
        const int dx = (x0 - cc.x + w) & (mx - 1), dy = (y0 - cc.y + w) & (my - 1), dz = (z0 - cc.z + w) & (mz - 1);
        hit = (dx < T || dx > mx - 8) && (dy < T || dy > my - 4) && (dz < T || dz > mz - 8);
        e = make_int4(rp + nu_xo(T) + (dx < T ? dx : dx - mx), rp + nu_yo(T) + (dy < T ? dy : dy - my),
                      rp + nu_zo(T) + (dz < T ? dz : dz - mz), SPREAD ? rp : p);
        if (slots) {
          int dst = -1;
          const int nbx = mx / 16;
          const int bxr = (gx0 / 16 - ((cc.x - w) >> 4)) & (nbx - 1), byr = (gy0 / 8 - ((cc.y - w) >> 3)) & (nby - 1);
          const int bzr = (gz0 / 16 - ((cc.z - w) >> 4)) & (nbz - 1);
          if (bxr < nu_blocks(cc.x, w, 4, nbx) && byr < nu_blocks(cc.y, w, 3, nby) && bzr < nu_blocks(cc.z, w, 4, nbz))
            dst = cc.w * nu_slots3(w) + (bxr * nu_slots(w, 3) + byr) * nu_slots(w, 4) + bzr;
          s_dst[slot][p] = dst;
        }
      } else if (slots) {
        s_dst[slot][p] = -1;
      }
      const unsigned mask = __ballot_sync(0xffffffffu, hit);
      if (hit) list[__popc(mask & ((1u << lane) - 1))] = e;
      else if (!SPREAD) mine[p] = make_double2(0.0, 0.0);
      n = __popc(mask);
    }
    // fills up the last group, and one group past it for the loop's look-ahead
    if (lane < 16) list[n + lane] = make_int4(ZB, ZB, ZB, SPREAD ? ZB : -1);
    __syncwarp();
    constexpr int G = SPREAD ? 4 : 8;
    int4 e = list[SPREAD ? lk : lr];
#pragma unroll 2
    for (int i = 0; i < n; i += G) {
      const int4 e_next = list[i + G + (SPREAD ? lk : lr)];
      if constexpr (SPREAD) {
        const double2 v = *reinterpret_cast<const double2*>(nu_sm + e.w);
        const double wz = nu_sm[e.z + lr], ax = nu_sm[e.x + lr];
        const double vr = v.x * wz, vi = v.y * wz;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double wy = nu_sm[e.y + j];
          nu_mma(acc[j][0], ax, vr * wy);
          nu_mma(acc[j][1], ax, vi * wy);
        }
      } else {
        const double a0 = nu_sm[e.x + lk], a1 = nu_sm[e.x + 4 + lk];
        const double w0 = nu_sm[e.z + 2 * lk], w1 = nu_sm[e.z + 2 * lk + 1];
        double re = 0.0, im = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          double2 dr = make_double2(0.0, 0.0), di = dr;
          nu_mma(dr, a0, cell[j][0][0]);
          nu_mma(di, a0, cell[j][0][1]);
          nu_mma(dr, a1, cell[j][1][0]);
          nu_mma(di, a1, cell[j][1][1]);
          const double wy = nu_sm[e.y + j];
          re = fma(wy, fma(w1, dr.y, w0 * dr.x), re);
          im = fma(wy, fma(w1, di.y, w0 * di.x), im);
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          re += __shfl_xor_sync(0xffffffffu, re, o);
          im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lk == 0 && e.w >= 0) mine[e.w] = make_double2(re, im);
      }
      e = e_next;
    }
    any = any || n;
  }
  if constexpr (!SPREAD) {
    __syncthreads();
    if (wid == 0) sum_parts(k & 1 ^ 1);
  }
  if constexpr (SPREAD) {
    if (!any) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double2* o = grid + (x0 + lr) * sx + (long long)(y0 + j) * mz + z0 + 2 * lk;
      const double2 c0 = make_double2(acc[j][0].x, acc[j][1].x), c1 = make_double2(acc[j][0].y, acc[j][1].y);
      if (add) {
        atomicAdd(&o[0].x, c0.x);
        atomicAdd(&o[0].y, c0.y);
        atomicAdd(&o[1].x, c1.x);
        atomicAdd(&o[1].y, c1.y);
      } else {
        o[0] = c0;
        o[1] = c1;
      }
    }
  }
}

// The slots of each point: four lanes take its x and y blocks in turn, then add up
// in one order.  Centre and index come from the record (three fmod per point
// otherwise).
__global__ void nu3_collect(int mx, int my, int mz, int w, const double* __restrict__ rec,
                            const double2* __restrict__ slots, int npts, double2* __restrict__ out) {
  const int ny = nu_slots(w, 3), nz = nu_slots(w, 4);
  const int t = blockIdx.x * blockDim.x + threadIdx.x, i0 = min(t >> 2, npts - 1), l = t & 3;
  const int4 cc = *reinterpret_cast<const int4*>(rec + (long long)i0 * nu_rec(2 * w + 1) + 2);
  const int bx = nu_blocks(cc.x, w, 4, mx / 16), by = nu_blocks(cc.y, w, 3, my / 8), bz = nu_blocks(cc.z, w, 4, mz / 16);
  const double2* q = slots + (long long)cc.w * nu_slots3(w);
  double2 v = make_double2(0.0, 0.0);
  for (int i = l; i < bx * by; i += 4) {
    const double2* r = q + (i / by * ny + i % by) * nz;
    for (int z = 0; z < bz; ++z) {
      v.x += r[z].x;
      v.y += r[z].y;
    }
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  if (l == 0 && t >> 2 < npts) out[cc.w] = v;
}

// T: taps per axis at compile time.  A lane holds the point's x-weights in
// registers and sums its (py, pz) columns over x first, two FMAs and one
// shared-memory load per tap (with the weight product inside the loop and the
// cell list checked at run time it was 936 instructions per lane and point at
// w = 6).  The shared loads (4 wavefronts per 32 cells) bound it.
template <int T>
__global__ void __launch_bounds__(kNuTileThreads) nu3_interp_tiles(const __grid_constant__ NuGeom3 g, NuTiles tl,
                                                                    const double2* __restrict__ grid,
                                                                    const double* __restrict__ pos, double2* out) {
  extern __shared__ __align__(16) unsigned char nu_smem[];
  const int tile = blockIdx.x;
  const int start = tl.off[tile], end = tl.off[tile + 1];
  if (start == end) return;
  constexpr int IT = (T * T + 31) / 32, G4 = (T + 3) / 4;
  const int E = tl.E, E2 = E * E, E3 = E2 * E;
  double2* cells = reinterpret_cast<double2*>(nu_smem);
  double* wts = reinterpret_cast<double*>(cells + E3);       // kNuChunk x 3 x T
  int* loc = reinterpret_cast<int*>(wts + kNuChunk * 3 * T);  // kNuChunk x 3
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const NuTileCoord tc(tile, tl);
  const long long mxm = g.mx - 1, mym = g.my - 1, mzm = g.mz - 1;
  const long long gx0 = (long long)tc.tx * tl.B - g.w, gy0 = (long long)tc.ty * tl.B - g.w,
                  gz0 = (long long)tc.tz * tl.B - g.w;
  for (int c = threadIdx.x; c < E3; c += kNuTileThreads) {
    const int cx = c / E2, cy = (c / E) % E, cz = c % E;
    cells[c] = grid[(((gx0 + cx) & mxm) * g.my + ((gy0 + cy) & mym)) * g.mz + ((gz0 + cz) & mzm)];
  }
  int coff[IT];  // the lane's columns; past the plane: column 0 with weight 0
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int f = it * 32 + lane;
    coff[it] = f < T * T ? (f / T) * E + f % T : 0;
  }
  for (int base = start; base < end; base += kNuChunk) {
    const int cnt = min(kNuChunk, end - base);
    __syncthreads();  // cells loaded / previous chunk's weights consumed
    // the chunk's axis weights, four taps of one point and axis per thread
    for (int e = threadIdx.x; e < cnt * 3 * G4; e += kNuTileThreads) {
      const int p = e / (3 * G4), r = e - p * 3 * G4, a = r / G4, t0 = (r - a * G4) * 4;
      const double* ps = pos + 3 * (long long)tl.idx[base + p];
      const long long m = a == 0 ? g.mx : a == 1 ? g.my : g.mz;
      const double t = nu_axis_t(ps[a], a == 0 ? g.lx : a == 1 ? g.ly : g.lz, m);
      const double rt = round(t);
      if (t0 == 0) loc[p * 3 + a] = (int)((long long)rt & (m - 1)) - (a == 0 ? tc.tx : a == 1 ? tc.ty : tc.tz) * tl.B;
      double o[4];
      nu_phi4(g.f, t0, t - rt, g.w, g.beta, g.i0b, o);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (t0 + i < T) wts[p * 3 * T + a * T + t0 + i] = o[i];
    }
    __syncthreads();
    for (int p = wid; p < cnt; p += kNuTileWarps) {
      const double* wp = wts + p * 3 * T;
      double wx[T];
#pragma unroll
      for (int i = 0; i < T; ++i) wx[i] = wp[i];
      double ax = 0.0, ay = 0.0;
      const double2* corner = cells + loc[p * 3] * E2 + loc[p * 3 + 1] * E + loc[p * 3 + 2];
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int f = it * 32 + lane;
        const double wyz = f < T * T ? wp[T + f / T] * wp[2 * T + f % T] : 0.0;
        const double2* col = corner + coff[it];
        double sx = 0.0, sy = 0.0;
#pragma unroll
        for (int px = 0; px < T; ++px) {
          const double2 c = col[px * E2];
          sx = fma(wx[px], c.x, sx);
          sy = fma(wx[px], c.y, sy);
        }
        if (f < T * T) {
          ax = fma(wyz, sx, ax);
          ay = fma(wyz, sy, ay);
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
      }
      if (lane == 0) out[tl.idx[base + p]] = make_double2(ax, ay);
    }
  }
}

// modes[kx][ky][kz] <-> grid[kx_signed mod mx][ky_signed mod my][kz_signed mod mz], times dx dy dz deconvolution.
__global__ void nu_modes3(long long nx, long long ny, long long nz, long long mx, long long my, long long mz,
                          const double* __restrict__ dcx, const double* __restrict__ dcy, const double* __restrict__ dcz,
                          const double2* src, double2* dst, int to_grid) {
  const long long total = nx * ny * nz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const long long kz = e % nz, ky = (e / nz) % ny, kx = e / (ny * nz);
    const long long gi = (nu_bin(kx, nx, mx) * my + nu_bin(ky, ny, my)) * mz + nu_bin(kz, nz, mz);
    const double f = dcx[kx] * dcy[ky] * dcz[kz];
    if (to_grid) {
      const double2 c = src[e];
      dst[gi] = make_double2(c.x * f, c.y * f);
    } else {
      const double2 c = src[gi];
      dst[e] = make_double2(c.x * f, c.y * f);
    }
  }
}

static unsigned nu_grid(long long work) {
  long long b = (work + 255) / 256;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return (unsigned)b;
}

// Sorting costs three passes over the points (about 60 us per million) and three
// launches, and saves atomics: about 20 per window of 32 cells and 32 points
// instead of 2 T per point, and the contention of crowded points.  Measured at
// uniform / crowded points (the middle sampled most), us unsorted -> sorted:
//  * from two million taps on, w = 4, n = 4096, 2^20 points 160 -> 195 / 978 -> 312,
//    n = 65536 156 -> 146 / 328 -> 210, w = 6 219 -> 166 / 479 -> 233;
//  * from 16 points a cell on, w = 4, n = 1024, 2^16 points 35 -> 51 / 136 -> 52;
//  * below six taps a cell the windows hold a point or two: w = 4, n = 2^22, 2^22
//    points 1112 -> 1116 / 1101 -> 1345: unsorted;
//  * w = 3 from 16 points a cell on only: n = 1024, 2^20 points 286 -> 365 / 1366 -> 388,
//    n = 4096 139 -> 197 / 744 -> 307; n = 65536 (8 a cell) 122 -> 146 / 267 -> 206;
//  * w = 2: n = 1024, 2^20 points 136 -> 357 / 917 -> 371: unsorted, but for the few
//    cells whose atomics serialize (n = 128, 2^18 points 183 -> 116 / 562 -> 164).
bool nufft_sorted(const NuLaunch& L, long long npts) {
  const long long T = 2 * L.w + 1;
  if (T > 25 || L.m < 64 || L.m >= (1ll << 31) - 64 || npts > INT32_MAX) return false;
  const bool crowd = npts >= 16 * L.m && npts >= 4096;
  if (T < 7) return L.m <= 256 && npts >= 256 * L.m;
  if (T < 9) return crowd;
  return crowd || (npts * T >= 6 * L.m && npts * T >= (1 << 21));
}

cudaError_t nufft_spread_dev(const NuLaunch& L, const NuTileLaunch& TL, const double* pos, const void* val,
                             long long npts, void* grid, cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  const NuGeom g{L.m, L.w, L.beta, L.i0b, L.len, L.f};
  if (TL.idx && nufft_sorted(L, npts)) {
    const int width = nufft_bin_width(L.m), bins = (int)((L.m + width - 1) / width);
    cudaError_t e = cudaMemsetAsync(TL.cnt, 0, (size_t)bins * sizeof(int), st);
    if (e != cudaSuccess) return e;
    nu1_bin<<<nu_grid(npts), 256, 0, st>>>(g, width, pos, npts, TL.cnt, TL.tile, TL.rank);
    nu3_scan<<<1, 1024, 0, st>>>(TL.cnt, TL.off, bins);
    nu3_scatter<<<nu_grid(npts), 256, 0, st>>>(TL.tile, TL.rank, TL.off, npts, TL.idx);
    const size_t smem = nu1_smem(2 * L.w + 1);
    auto k = nu1_spread<0>;
    switch (L.w) {
      case 4: k = nu1_spread<9>; break;
      case 5: k = nu1_spread<11>; break;
      case 6: k = nu1_spread<13>; break;
      case 7: k = nu1_spread<15>; break;
      case 8: k = nu1_spread<17>; break;
      default: break;
    }
    e = kernel_smem_grant(reinterpret_cast<const void*>(k), smem);
    if (e != cudaSuccess) return e;
    const long long blocks = (npts + 32 * kNu1Warps - 1) / (32 * kNu1Warps);
    k<<<(unsigned)std::min<long long>(blocks, 1 << 20), 32 * kNu1Warps, smem, st>>>(
        g, TL.idx, pos, static_cast<const double2*>(val), npts, static_cast<double2*>(grid));
    count_launch(4);
    return cudaGetLastError();
  }
  nu_spread<<<nu_grid(npts), 256, 0, st>>>(g, pos, static_cast<const double2*>(val), npts, static_cast<double2*>(grid));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t nufft_interp_dev(const NuLaunch& L, const void* grid, const double* pos, long long npts, void* out,
                             cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  const NuGeom g{L.m, L.w, L.beta, L.i0b, L.len, L.f};
  auto k = nu_interp<0>;
  switch (L.w) {
    case 4: k = nu_interp<9>; break;
    case 5: k = nu_interp<11>; break;
    case 6: k = nu_interp<13>; break;
    case 7: k = nu_interp<15>; break;
    case 8: k = nu_interp<17>; break;
    default: break;
  }
  k<<<nu_grid(npts), 256, 0, st>>>(g, static_cast<const double2*>(grid), pos, npts, static_cast<double2*>(out));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t nufft_deconv_out_dev(const void* grid, const double* deconv, long long n, long long m, void* out,
                                 cudaStream_t st) {
  nu_deconv_out<<<nu_grid(n), 256, 0, st>>>(static_cast<const double2*>(grid), deconv, n, m, static_cast<double2*>(out));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t nufft_place_coeffs_dev(const void* coeffs, const double* deconv, long long n, long long m, void* grid,
                                   cudaStream_t st) {
  nu_place_coeffs<<<nu_grid(n), 256, 0, st>>>(static_cast<const double2*>(coeffs), deconv, n, m,
                                              static_cast<double2*>(grid));
  count_launch(1);
  return cudaGetLastError();
}

static NuGeom3 geom3(const NuLaunch3& L) {
  return NuGeom3{L.mx, L.my, L.mz, L.w, L.beta, L.i0b, L.lx, L.ly, L.lz, L.f};
}

static unsigned nu_warp_grid(long long npts) {
  long long b = (npts + kNuWarps - 1) / kNuWarps;
  return (unsigned)(b < 148 * 8 ? b : 148 * 8);
}

cudaError_t nufft3_spread_dev(const NuLaunch3& L, const double* pos, const void* val, long long npts, void* grid,
                              cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  nu_spread3<<<nu_warp_grid(npts), 32 * kNuWarps, 0, st>>>(geom3(L), pos, static_cast<const double2*>(val), npts,
                                            static_cast<double2*>(grid));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t nufft3_interp_dev(const NuLaunch3& L, const void* grid, const double* pos, long long npts, void* out,
                              cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  nu_interp3<<<nu_warp_grid(npts), 32 * kNuWarps, 0, st>>>(geom3(L), static_cast<const double2*>(grid), pos, npts,
                                            static_cast<double2*>(out));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t nufft3_modes_dev(const NuLaunch3& L, const double* dcx, const double* dcy, const double* dcz,
                             const void* src, void* dst, bool to_grid, cudaStream_t st) {
  nu_modes3<<<nu_grid(L.nx * L.ny * L.nz), 256, 0, st>>>(L.nx, L.ny, L.nz, L.mx, L.my, L.mz, dcx, dcy, dcz,
                                                         static_cast<const double2*>(src), static_cast<double2*>(dst),
                                                         to_grid ? 1 : 0);
  count_launch(1);
  return cudaGetLastError();
}

int nufft3_tile_size(int w) {
  if ((2 * w + 1) * (2 * w + 1) > 32 * kNuTileIters) return 0;  // more plane cells than a lane's list holds
  for (int B : {8, 4})
    if (nufft3_tile_smem(B, w) <= 220 * 1024) return B;
  return 0;
}

size_t nufft3_tile_smem(int B, int w) {
  const size_t E = (size_t)(B + 2 * w), T = (size_t)(2 * w + 1);
  const size_t cells = E * E * E * sizeof(double2);
  // both kernels stage the axis weights and centre cells of kNuChunk points
  return cells + kNuChunk * 3 * T * sizeof(double) + kNuChunk * 3 * sizeof(int);
}

// The box kernel serves grids whose axes hold a kernel and a box side by side
// (a padded x row is not periodic) and whose candidate runs fit its table.
bool nufft3_boxes(const NuLaunch3& L) {
  const long long lo = std::min(L.mx, std::min(L.my, L.mz)), hi = std::max(L.mx, std::max(L.my, L.mz));
  const int T = 2 * L.w + 1, wt = (L.w + 7) / 8;
  return lo >= 16 && lo >= T + 8 && hi < (1 << 20) && (2 + 2 * wt) * (1 + 2 * wt) * 2 <= kNuBoxRuns &&
         nufft3_box_smem(L.w, false) <= 112 * 1024;
}
// Interpolation with few taps costs the tile kernel less than the boxes' records
// and sums: from a point per 32 cells on, w = 2 takes the tiles.  Measured at
// uniform / crowded points, us tiles -> boxes: w = 2, 2^20 points on 128^3 cells
// 491 / 3818 -> 2310 / 6525, 2^17 on 64^3 123 / 1019 -> 346 / 469 (a tile is one CTA, so
// crowded points on a small grid would prefer boxes); 2^15 on 256^3 767 / 571 -> 537 /
// 739: boxes.  Wider kernels gain less from tiles and lose more: w = 3, 2^17 on 64^3
// 182 / 1599 -> 366 / 507, w = 4, 2^17 on 128^3 325 / 1249 -> 408 / 1088, w = 6 518 / 2353 ->
// 489 / 1347: boxes.
bool nufft3_boxes_interp(const NuLaunch3& L, long long npts) {
  return nufft3_boxes(L) && (L.w > 2 || 32 * npts < L.mx * L.my * L.mz);
}
size_t nufft3_box_smem(int w, bool spread) {
  return ((size_t)2 * kNuBoxChunk * nu_rec(2 * w + 1) + kNuZeros) * sizeof(double) +
         (size_t)(kNuBoxThreads / 32) * nu_list() * sizeof(int) +
         (spread ? 0 : (size_t)2 * (kNuBoxThreads / 32) * kNuBoxChunk * sizeof(double2));
}
size_t nufft3_slot_bytes(int w) { return (size_t)nu_slots3(w) * sizeof(double2); }
size_t nufft3_rec_bytes(int w) { return (size_t)nu_rec(2 * w + 1) * sizeof(double); }

// Spreads npts points onto the zeroed grid, or interpolates the grid at them
// into out; kNu3Slice points at a time (their records take nufft3_rec_bytes each
// and, interpolating, their slots nufft3_slot_bytes).
cudaError_t nufft3_boxes_dev(const NuLaunch3& L, const NuTileLaunch& TL, bool spread, const double* pos,
                             const void* val, long long npts, void* grid, void* out, cudaStream_t st) {
  const NuGeom3 g = geom3(L);
  const int nty = (int)(L.my / 8), ntz = (int)(L.mz / 8), ntiles = (int)(L.mx / 8) * nty * ntz;
  const size_t smem = nufft3_box_smem(L.w, spread);
  auto k = spread ? nu3_boxes<true> : nu3_boxes<false>;
  cudaError_t e = kernel_smem_grant(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  const int boxes = (int)(L.mx / 16) * (int)(L.my / 8) * (int)(L.mz / 16);
  for (long long p0 = 0; p0 < npts; p0 += kNu3Slice) {
    const long long n = std::min<long long>(kNu3Slice, npts - p0);
    const double* ps = pos + 3 * p0;
    e = cudaMemsetAsync(TL.cnt, 0, (size_t)ntiles * sizeof(int), st);
    if (e != cudaSuccess) return e;
    nu3_bin<<<nu_grid(n), 256, 0, st>>>(g, 8, nty, ntz, ps, n, TL.cnt, TL.tile, TL.rank);
    nu3_scan<<<1, 1024, 0, st>>>(TL.cnt, TL.off, ntiles);
    nu3_scatter<<<nu_grid(n), 256, 0, st>>>(TL.tile, TL.rank, TL.off, n, TL.idx);
    void (*points)(const NuGeom3, const int*, const double*, const double2*, int, double*) = nullptr;
    switch (L.w) {  // nufft3_tile_size: 2 <= w <= 9
      case 2: points = nu3_points<5>; break;
      case 3: points = nu3_points<7>; break;
      case 4: points = nu3_points<9>; break;
      case 5: points = nu3_points<11>; break;
      case 6: points = nu3_points<13>; break;
      case 7: points = nu3_points<15>; break;
      case 8: points = nu3_points<17>; break;
      case 9: points = nu3_points<19>; break;
      default: return cudaErrorInvalidValue;
    }
    points<<<(unsigned)((n + kNuPts - 1) / kNuPts), 3 * kNuPts, 0, st>>>(
        g, TL.idx, ps, spread ? static_cast<const double2*>(val) + p0 : nullptr, (int)n, TL.rec);
    // a box's chunks are dealt to `split` CTAs: about 4096 CTAs in all, so a
    // grid of few boxes, or points crowded into some of them, still fills the chip.
    // Type 1 at w = 6, us with 1 / 2 / 4 / 8 / 32 CTAs a box: 2^18 points on 64^3 modes
    // (1024 boxes) uniform 716 / 705 / 728 / 789 / 1189, crowded about the middle 15388 /
    // 8781 / 5017 / 2910 / 1273; 2^15 on 32^3 (128 boxes) 199 / 154 / 154 / 145 / 191 and
    // 2031 / 1129 / 639 / 422 / 202; 2^18 on 16^3 (16 boxes) 8863 / 4564 / 2367 / 1269 / 874
    const long long chunks = (n + kNuBoxChunk - 1) / kNuBoxChunk;
    const int split = (int)std::max<long long>(1, std::min<long long>(chunks, std::min(32, 4096 / boxes)));
    k<<<dim3((unsigned)boxes, (unsigned)split), kNuBoxThreads, smem, st>>>(
        (int)L.mx, (int)L.my, (int)L.mz, L.w, TL.off, TL.rec, static_cast<double2*>(grid), TL.slots,
        split > 1 || npts > kNu3Slice);
    if (!spread)
      nu3_collect<<<(unsigned)((4 * n + 255) / 256), 256, 0, st>>>((int)L.mx, (int)L.my, (int)L.mz, L.w, TL.rec, TL.slots,
                                                                   (int)n, static_cast<double2*>(out) + p0);
    count_launch(spread ? 5 : 6);
  }
  return cudaGetLastError();
}

cudaError_t nufft3_tiled_dev(const NuLaunch3& L, const NuTileLaunch& TL, bool spread, const double* pos,
                             const void* src, long long npts, void* dst, cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  const NuGeom3 g = geom3(L);
  const int ntiles = TL.ntx * TL.nty * TL.ntz;
  cudaError_t e = cudaMemsetAsync(TL.cnt, 0, (size_t)ntiles * sizeof(int), st);
  if (e != cudaSuccess) return e;
  nu3_bin<<<nu_grid(npts), 256, 0, st>>>(g, TL.B, TL.nty, TL.ntz, pos, npts, TL.cnt, TL.tile, TL.rank);
  nu3_scan<<<1, 1024, 0, st>>>(TL.cnt, TL.off, ntiles);
  nu3_scatter<<<nu_grid(npts), 256, 0, st>>>(TL.tile, TL.rank, TL.off, npts, TL.idx);
  const NuTiles tl{TL.B, TL.B + 2 * L.w, TL.nty, TL.ntz, TL.off, TL.idx};
  const size_t smem = nufft3_tile_smem(TL.B, L.w);
  if (spread) {
    e = kernel_smem_grant(reinterpret_cast<const void*>(nu3_spread_tiles), smem);
    if (e != cudaSuccess) return e;
    nu3_spread_tiles<<<ntiles, kNuTileThreads, smem, st>>>(g, tl, pos, static_cast<const double2*>(src),
                                                           static_cast<double2*>(dst));
  } else {
    void (*k)(const NuGeom3, NuTiles, const double2*, const double*, double2*) = nullptr;
    switch (L.w) {  // nufft3_tile_size: 2 <= w <= 9
      case 2: k = nu3_interp_tiles<5>; break;
      case 3: k = nu3_interp_tiles<7>; break;
      case 4: k = nu3_interp_tiles<9>; break;
      case 5: k = nu3_interp_tiles<11>; break;
      case 6: k = nu3_interp_tiles<13>; break;
      case 7: k = nu3_interp_tiles<15>; break;
      case 8: k = nu3_interp_tiles<17>; break;
      case 9: k = nu3_interp_tiles<19>; break;
      default: return cudaErrorInvalidValue;
    }
    e = kernel_smem_grant(reinterpret_cast<const void*>(k), smem);
    if (e != cudaSuccess) return e;
    k<<<ntiles, kNuTileThreads, smem, st>>>(g, tl, static_cast<const double2*>(src), pos, static_cast<double2*>(dst));
  }
  count_launch(4);
  return cudaGetLastError();
}

// ───────────────────── exact direct non-uniform DFTs ─────────────────────
// apollo-nufft's exact direct sums (transform/dimension_1d.rs:428-472,
// dimension_3d.rs:677-712): every output is the full sum over the inputs with
// the phase (2 pi / L) k x, k the FFT-signed index (k <= n/2 stays, else
// k - n; kaiser_bessel.rs:152-158), evaluated in FP64 like the reference.
// One thread per output; the inputs stream through shared memory in chunks of
// the block size, so each is read from global memory once per block.

constexpr int kDirectThreads = 256;
constexpr double kTwoPi = 6.283185307179586476925286766559;  // 2 pi

__device__ __forceinline__ long long direct_signed(long long k, long long n) { return k <= n / 2 ? k : k - n; }

// out[k] = sum_j v_j exp(-i (2 pi / L) k_s x_j), k < n
__global__ void __launch_bounds__(kDirectThreads) nudft1_type1(const double* __restrict__ pos,
                                                               const double2* __restrict__ val, long long npts,
                                                               long long n, double two_pi_over_l, double2* out) {
  __shared__ double sx[kDirectThreads];
  __shared__ double2 sv[kDirectThreads];
  const long long k = (long long)blockIdx.x * kDirectThreads + threadIdx.x;
  const double ks = (double)direct_signed(k < n ? k : 0, n);
  double re = 0.0, im = 0.0;
  for (long long j0 = 0; j0 < npts; j0 += kDirectThreads) {
    const long long j = j0 + threadIdx.x;
    __syncthreads();
    if (j < npts) {
      sx[threadIdx.x] = pos[j];
      sv[threadIdx.x] = val[j];
    }
    __syncthreads();
    const int cnt = (int)(npts - j0 < kDirectThreads ? npts - j0 : kDirectThreads);
    for (int i = 0; i < cnt; ++i) {
      const double angle = -two_pi_over_l * ks * sx[i];
      double sn, cs;
      sincos(angle, &sn, &cs);
      const double2 v = sv[i];
      re += v.x * cs - v.y * sn;
      im += v.x * sn + v.y * cs;
    }
  }
  if (k < n) out[k] = make_double2(re, im);
}

// out[j] = sum_k c_k exp(+i (2 pi / L) k_s x_j), j < npts
__global__ void __launch_bounds__(kDirectThreads) nudft1_type2(const double2* __restrict__ coeffs, long long n,
                                                               const double* __restrict__ pos, long long npts,
                                                               double two_pi_over_l, double2* out) {
  __shared__ double2 sc[kDirectThreads];
  const long long j = (long long)blockIdx.x * kDirectThreads + threadIdx.x;
  const double x = j < npts ? pos[j] : 0.0;
  double re = 0.0, im = 0.0;
  for (long long k0 = 0; k0 < n; k0 += kDirectThreads) {
    __syncthreads();
    if (k0 + threadIdx.x < n) sc[threadIdx.x] = coeffs[k0 + threadIdx.x];
    __syncthreads();
    const int cnt = (int)(n - k0 < kDirectThreads ? n - k0 : kDirectThreads);
    for (int i = 0; i < cnt; ++i) {
      const double angle = two_pi_over_l * (double)direct_signed(k0 + i, n) * x;
      double sn, cs;
      sincos(angle, &sn, &cs);
      const double2 c = sc[i];
      re += c.x * cs - c.y * sn;
      im += c.x * sn + c.y * cs;
    }
  }
  if (j < npts) out[j] = make_double2(re, im);
}

// out[kx, ky, kz] = sum_j v_j exp(-i (wx kx_s x_j + wy ky_s y_j + wz kz_s z_j))
__global__ void __launch_bounds__(kDirectThreads) nudft3_type1(const double* __restrict__ pos,
                                                               const double2* __restrict__ val, long long npts,
                                                               long long nx, long long ny, long long nz, double wx,
                                                               double wy, double wz, double2* out) {
  __shared__ double sp[3 * kDirectThreads];
  __shared__ double2 sv[kDirectThreads];
  const long long total = nx * ny * nz;
  const long long m = (long long)blockIdx.x * kDirectThreads + threadIdx.x;
  const long long mm = m < total ? m : 0;
  const double kx = (double)direct_signed(mm / (ny * nz), nx);
  const double ky = (double)direct_signed((mm / nz) % ny, ny);
  const double kz = (double)direct_signed(mm % nz, nz);
  double re = 0.0, im = 0.0;
  for (long long j0 = 0; j0 < npts; j0 += kDirectThreads) {
    const long long j = j0 + threadIdx.x;
    __syncthreads();
    if (j < npts) {
      sp[3 * threadIdx.x] = pos[3 * j];
      sp[3 * threadIdx.x + 1] = pos[3 * j + 1];
      sp[3 * threadIdx.x + 2] = pos[3 * j + 2];
      sv[threadIdx.x] = val[j];
    }
    __syncthreads();
    const int cnt = (int)(npts - j0 < kDirectThreads ? npts - j0 : kDirectThreads);
    for (int i = 0; i < cnt; ++i) {
      const double angle = -(wx * kx * sp[3 * i] + wy * ky * sp[3 * i + 1] + wz * kz * sp[3 * i + 2]);
      double sn, cs;
      sincos(angle, &sn, &cs);
      const double2 v = sv[i];
      re += v.x * cs - v.y * sn;
      im += v.x * sn + v.y * cs;
    }
  }
  if (m < total) out[m] = make_double2(re, im);
}

cudaError_t nudft1_type1_dev(const double* pos, const void* val, long long npts, long long n, double len, void* out,
                             cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((n + kDirectThreads - 1) / kDirectThreads);
  nudft1_type1<<<grid, kDirectThreads, 0, st>>>(pos, static_cast<const double2*>(val), npts, n, kTwoPi / len,
                                                static_cast<double2*>(out));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t nudft1_type2_dev(const void* coeffs, long long n, const double* pos, long long npts, double len, void* out,
                             cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((npts + kDirectThreads - 1) / kDirectThreads);
  nudft1_type2<<<grid, kDirectThreads, 0, st>>>(static_cast<const double2*>(coeffs), n, pos, npts, kTwoPi / len,
                                                static_cast<double2*>(out));
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t nudft3_type1_dev(const double* pos, const void* val, long long npts, long long nx, long long ny,
                             long long nz, double lx, double ly, double lz, void* out, cudaStream_t st) {
  const long long total = nx * ny * nz;
  if (total <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((total + kDirectThreads - 1) / kDirectThreads);
  nudft3_type1<<<grid, kDirectThreads, 0, st>>>(pos, static_cast<const double2*>(val), npts, nx, ny, nz,
                                                kTwoPi / lx, kTwoPi / ly, kTwoPi / lz,
                                                static_cast<double2*>(out));
  count_launch(1);
  return cudaGetLastError();
}

}  // namespace afc
