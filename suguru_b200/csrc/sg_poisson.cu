// sg_poisson.cu -- solver1d (solver.f90:43-157) after initsolver(e)
// (initsolver.f90:11-130) on the GPU: periodic x and y by a real 2-D FFT of
// every z plane, then for every (x, y) mode the reference's tridiagonal
// elimination in z in FP64, then the inverse FFT.
//
// The FFTs are the library's own (the reference's fft.f / 2DECOMP transforms
// are FFTPACK-style mixed-radix FFTs): self-sorting (Stockham) passes, FP64,
// with twiddle factors tabulated once on the host.  Both directions are
// unnormalised, so that the pair multiplies by itot * jtot (the convention of
// the callers).  Any itot/2 and jtot whose prime factors are at most
// kMaxRadix are accepted.
//
// Modes lie [m][k][j] (x mode, level, y): the rows' kernels transpose as they
// write and read (runs of the CTA's rows), so that the y transforms run on
// contiguous sequences and the elimination on tiles of neighbouring columns.
// A solve is five launches: rows_r2c, cols, tri_tile, cols, rows_c2r.
// (A cluster of eight CTAs holding one x mode's whole plane over distributed
// shared memory, for cols, tri_tile, cols in one launch, moves a third of
// the bytes but took 119 us against 89 us at 256 x 256 x 128: 33 clusters
// fit at once, and their loads, exchanges and sweeps run in lockstep.)
//
// The rows of initsolver(e), built in the kernel in the reference's order:
//   a = c = dzi^2, b = -(a + c);
//   e = 0, 1: b(1) += a(1), b(kmax) += c(kmax), a(1) = c(kmax) = 0 (Neumann);
//   e = 2:    b(1) -= a(1), b(kmax) -= c(kmax), a(1) = c(kmax) = 0 (the
//             no-slip ghost rows of u and v), then b -= Rep/dt;
//   e = 3:    b(kmax) = 1, a(1) = a(kmax) = c(kmax) = 0 (w = 0 at the top
//             face), then b -= Rep/dt and b(kmax) = 1 again;
// the eigenvalues xrt + yrt of the mode join b except in the last row of
// e = 3.  The pivots keep the reference's operations and roundings (no
// fused multiply-add): for e = 0, 1 the mean mode's last pivot is then
// exactly zero whenever it is in exact arithmetic, and that mode's top value
// is set to zero, as the reference does.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "sg_common.cuh"
#include "sg_ctx.h"

namespace sg {
namespace {

constexpr double kPi = 3.14159265358979323846264338327950288;

struct Rows {
  double a, b, c;
};

__device__ __forceinline__ Rows solver_row(int k, int kmax, int e, double dzi, double shift) {
  Rows r;
  r.a = __dmul_rn(dzi, dzi);
  r.c = __dmul_rn(dzi, dzi);
  r.b = -__dadd_rn(r.a, r.c);
  const bool first = k == 0, last = k == kmax - 1;
  if (e <= 1) {
    if (first) r.b = __dadd_rn(r.b, r.a);
    if (last) r.b = __dadd_rn(r.b, r.c);
    if (first) r.a = 0.;
    if (last) r.c = 0.;
  } else {
    if (e == 2) {
      if (first) r.b = __dsub_rn(r.b, r.a);
      if (last) r.b = __dsub_rn(r.b, r.c);
      if (first) r.a = 0.;
      if (last) r.c = 0.;
    } else {
      if (last) {
        r.b = 1.;
        r.a = 0.;
        r.c = 0.;
      }
      if (first) r.a = 0.;
    }
    r.b = __dsub_rn(r.b, shift);
    if (e == 3 && last) r.b = 1.;
  }
  return r;
}

// The elimination split in two.  Its pivots depend only on the mode's
// eigenvalue, the row type e and the shift, not on the right-hand side, so
// tri_coeff_kernel runs the reference's forward recurrence for them once per
// (e, shift) and tabulates, per x mode m, level k and y mode j ([m][k][j]),
//   z_k = 1 / (b_k + lam - a_k d_{k-1})  (k < kmax-1; d_{-1} = 0),
//   z_{kmax-1} = bb - a d_{kmax-2}        (the last pivot itself, bb = b + lam
//                                          except for e = 3),
// with the same operations in the same order (no fused multiply-add: the mean
// mode's exact zero depends on it).  The multipliers d_k = c_k z_k = dzi^2 z_k
// (k < kmax-1) are one multiplication and are not stored.  A solve with the
// table is two first-order sweeps per mode,
//   q_0 = r_0 z_0, q_k = (r_k - a_k q_{k-1}) z_k, the last row divided by its
//   pivot (or set to zero when the pivot is exactly zero: the mean mode of
//   the Neumann rows, as the reference does), then x_k = q_k - d_k x_{k+1}.
__global__ void __launch_bounds__(128) tri_coeff_kernel(int kmax, int jtot, int nxm, int e, double dzi, double shift,
                                                        const double* __restrict__ xrt,
                                                        const double* __restrict__ yrt, double* __restrict__ zt) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nxm * jtot) return;
  const int m = q / jtot, j = q - m * jtot;
  const double lam = __dadd_rn(xrt[m], yrt[j]);
  double* zm = zt + (long)m * kmax * jtot + j;
  Rows r = solver_row(0, kmax, e, dzi, shift);
  double z = __drcp_rn(__dadd_rn(r.b, lam));
  double dk = __dmul_rn(r.c, z);
  zm[0] = z;
  for (int k = 1; k < kmax - 1; ++k) {
    r = solver_row(k, kmax, e, dzi, shift);
    z = __drcp_rn(__dsub_rn(__dadd_rn(r.b, lam), __dmul_rn(r.a, dk)));
    dk = __dmul_rn(r.c, z);
    zm[(long)k * jtot] = z;
  }
  r = solver_row(kmax - 1, kmax, e, dzi, shift);
  const double bb = e == 3 ? r.b : __dadd_rn(r.b, lam);
  zm[(long)(kmax - 1) * jtot] = __dsub_rn(bb, __dmul_rn(r.a, dk));
}

template <int V>
using Const = std::integral_constant<int, V>;

// The two sweeps of one real column (the real or the imaginary parts of a
// mode's levels: the elimination's coefficients are real) at c[k cs], its
// pivots at z[k zs]; a = dzi^2 is both a_k (k = 1 .. kmax-2) and c_k.  Bound
// by the chain from level to level, so each sweep is one fused multiply-add
// per level on it (8 cycles; the products r_k z_k and a z_k are off it) and
// runs in blocks of B levels without branches, the next block's loads ahead
// of the block's arithmetic.  (The three dependent operations of the
// unfused form with a guarded load per level took 97 cycles a level.)
// cs, zs: the strides, as constants (tri_tile_kernel) or values.
template <int B, class SC, class SZ>
__device__ __forceinline__ void tri_sweeps(double* c, const double* z, SC cs, SZ zs, int kmax, int e, double a) {
  const int last = kmax - 1;
  double r[B], w[B], rn[B], wn[B];
#pragma unroll
  for (int t = 0; t < B; ++t) {
    const int k = min(1 + t, last);
    r[t] = c[k * cs];
    w[t] = z[k * zs];
  }
  double p = c[0] * z[0];
  c[0] = p;
  int k = 1;
  for (; k + B <= last; k += B) {
#pragma unroll
    for (int t = 0; t < B; ++t) {
      const int q = min(k + B + t, last);
      rn[t] = c[q * cs];
      wn[t] = z[q * zs];
    }
#pragma unroll
    for (int t = 0; t < B; ++t) {
      p = fma(-(a * w[t]), p, r[t] * w[t]);
      c[(k + t) * cs] = p;
    }
#pragma unroll
    for (int t = 0; t < B; ++t) {
      r[t] = rn[t];
      w[t] = wn[t];
    }
  }
#pragma unroll
  for (int t = 0; t < B; ++t)
    if (k + t < last) {
      p = fma(-(a * w[t]), p, r[t] * w[t]);
      c[(k + t) * cs] = p;
    }
  {
    const double zk = z[last * zs], al = e == 3 ? 0.0 : a;  // e = 3: the identity row of w at the top
    p = zk != 0.0 ? fma(-al, p, c[last * cs]) / zk : 0.0;
    c[last * cs] = p;
  }
#pragma unroll
  for (int t = 0; t < B; ++t) {
    const int q = max(last - 1 - t, 0);
    r[t] = c[q * cs];
    w[t] = z[q * zs];
  }
  k = last - 1;
  for (; k - B >= -1; k -= B) {
#pragma unroll
    for (int t = 0; t < B; ++t) {
      const int q = max(k - B - t, 0);
      rn[t] = c[q * cs];
      wn[t] = z[q * zs];
    }
#pragma unroll
    for (int t = 0; t < B; ++t) {
      p = fma(-(a * w[t]), p, r[t]);
      c[(k - t) * cs] = p;
    }
#pragma unroll
    for (int t = 0; t < B; ++t) {
      r[t] = rn[t];
      w[t] = wn[t];
    }
  }
#pragma unroll
  for (int t = 0; t < B; ++t)
    if (k - t >= 0) {
      p = fma(-(a * w[t]), p, r[t]);
      c[(k - t) * cs] = p;
    }
}

// C neighbouring columns of one x mode, all levels, per CTA: copied to shared
// memory with their pivots, swept there by 2 C threads (real and imaginary
// parts), written back: each mode is read and written once.  Bound by memory
// (24 bytes in and 16 out per mode) with the sweeps' latency hidden by the
// other CTAs on the SM: at 256 x 256 x 128, 40 us with C = 16 (4.4 TB/s)
// against 46 us with C = 8, 69 us with C = 4 (short runs) and 41 us with
// C = 32 (fewer CTAs); a thread per column on global memory with a register
// ring, which stores and reloads the forward values, took 80 us.
constexpr int kTriThreads = 64;

template <int C>
__global__ void __launch_bounds__(kTriThreads) tri_tile_kernel(int kmax, int jtot, int e, double a,
                                                               const double* __restrict__ zt,
                                                               double2* __restrict__ c) {
  extern __shared__ __align__(16) double2 tsm[];  // [kmax][C] modes, then [kmax][C] pivots
  double* zs = (double*)(tsm + kmax * C);
  const int j0 = blockIdx.x * C, nj = min(C, jtot - j0);
  const long o = (long)blockIdx.y * kmax * jtot + j0;
  const int jl = threadIdx.x % C, k0 = threadIdx.x / C;
  if (jl < nj)
    for (int k = k0; k < kmax; k += kTriThreads / C) {
      stage_async(&tsm[k * C + jl], &c[o + (long)k * jtot + jl]);
      stage_async(&zs[k * C + jl], &zt[o + (long)k * jtot + jl]);
    }
  stage_wait();
  __syncthreads();
  if (threadIdx.x < 2 * nj)
    tri_sweeps<8>((double*)tsm + threadIdx.x, zs + (threadIdx.x >> 1), Const<2 * C>{}, Const<C>{}, kmax, e, a);
  __syncthreads();
  if (jl < nj)
    for (int k = k0; k < kmax; k += kTriThreads / C) c[o + (long)k * jtot + jl] = tsm[k * C + jl];
}

// Columns too long for a tile in shared memory: a thread per real column of
// the modes in global memory.
__global__ void __launch_bounds__(128) tri_apply_kernel(int kmax, int jtot, int nxm, int e, double a,
                                                        const double* __restrict__ zt, double2* __restrict__ c) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= 2L * nxm * jtot) return;
  const int part = (int)(q & 1), m = (int)((q >> 1) / jtot), j = (int)((q >> 1) % jtot);
  const long o = (long)m * kmax * jtot + j;
  tri_sweeps<16>((double*)(c + o) + part, zt + o, 2L * jtot, (long)jtot, kmax, e, a);
}

// ---------------------------------------------------------------- FFT ---
constexpr int kMaxRadix = 61;
constexpr int kMaxPasses = 8;
constexpr int kMaxLength = 2048;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cswap(double2 a) { return make_double2(a.y, a.x); }

// ------------------------------------------------- power-of-two FFTs ---
// Lengths N = 32, 64, 128, 256: a sequence belongs to TPS = N/8 consecutive
// lanes of one warp, each holding 8 values in registers.  A Stockham pass of
// radix R after sub-transforms of length NS gives thread tau the butterflies
// j = tau + b TPS (b < 8/R); butterfly j reads x[j + r N/R], twiddles it by
// W_{NS R}^{r (j mod NS)}, forms the R-point DFT and writes V[q] to
// (j / NS) NS R + j mod NS + q NS.  Between passes the values go through the
// sequence's slot in shared memory, element e at e ^ ((e >> 3) & 7): every
// read and write pattern of the passes then puts the 8 lanes of a quarter
// warp on 8 different 16-byte bank groups.  Radices: 32 = 8.4, 64 = 8.8,
// 128 = 8.4.4, 256 = 8.8.4.  Twiddles come from per-pass tables in shared
// memory (TwTab); the 8-point DFT uses sqrt(1/2) as a constant.
__device__ __forceinline__ int swz(int e) { return e ^ ((e >> 3) & 7); }

template <int R>
__device__ __forceinline__ void dft_reg(double2* v, int sign) {
  if constexpr (R == 2) {
    const double2 a = v[0], b = v[1];
    v[0] = make_double2(a.x + b.x, a.y + b.y);
    v[1] = make_double2(a.x - b.x, a.y - b.y);
  } else if constexpr (R == 4) {
    const double2 s02 = make_double2(v[0].x + v[2].x, v[0].y + v[2].y);
    const double2 d02 = make_double2(v[0].x - v[2].x, v[0].y - v[2].y);
    const double2 s13 = make_double2(v[1].x + v[3].x, v[1].y + v[3].y);
    const double2 d13 = make_double2(v[1].x - v[3].x, v[1].y - v[3].y);
    const double sx = sign > 0 ? -d13.y : d13.y, sy = sign > 0 ? d13.x : -d13.x;  // sign * i * d13
    v[0] = make_double2(s02.x + s13.x, s02.y + s13.y);
    v[1] = make_double2(d02.x + sx, d02.y + sy);
    v[2] = make_double2(s02.x - s13.x, s02.y - s13.y);
    v[3] = make_double2(d02.x - sx, d02.y - sy);
  } else {
    static_assert(R == 8, "radix");
    // V_q = E_q + W^q O_q, V_{q+4} = E_q - W^q O_q, W = exp(sign 2 pi i / 8)
    double2 E[4] = {v[0], v[2], v[4], v[6]}, O[4] = {v[1], v[3], v[5], v[7]};
    dft_reg<4>(E, sign);
    dft_reg<4>(O, sign);
    constexpr double h = 0.70710678118654752440;
    double2 t1, t2, t3;
    if (sign < 0) {
      t1 = make_double2(h * (O[1].x + O[1].y), h * (O[1].y - O[1].x));
      t2 = make_double2(O[2].y, -O[2].x);
      t3 = make_double2(h * (O[3].y - O[3].x), -h * (O[3].x + O[3].y));
    } else {
      t1 = make_double2(h * (O[1].x - O[1].y), h * (O[1].x + O[1].y));
      t2 = make_double2(-O[2].y, O[2].x);
      t3 = make_double2(-h * (O[3].x + O[3].y), h * (O[3].x - O[3].y));
    }
    v[0] = make_double2(E[0].x + O[0].x, E[0].y + O[0].y);
    v[4] = make_double2(E[0].x - O[0].x, E[0].y - O[0].y);
    v[1] = make_double2(E[1].x + t1.x, E[1].y + t1.y);
    v[5] = make_double2(E[1].x - t1.x, E[1].y - t1.y);
    v[2] = make_double2(E[2].x + t2.x, E[2].y + t2.y);
    v[6] = make_double2(E[2].x - t2.x, E[2].y - t2.y);
    v[3] = make_double2(E[3].x + t3.x, E[3].y + t3.y);
    v[7] = make_double2(E[3].x - t3.x, E[3].y - t3.y);
  }
}

// Twiddles of a pass (NS > 1) as their own table, tp[(r-1) NS + k] =
// W_{NS R}^{r k}: the lanes of a quarter warp (consecutive k) read
// consecutive 16-byte values.  Tables of a length's passes lie one after the
// other: 32: 24 values; 64: 56; 128: 24 + 96; 256: 56 + 192.
template <int N> struct TwTab;
template <> struct TwTab<32> { static constexpr int size = 24; };
template <> struct TwTab<64> { static constexpr int size = 56; };
template <> struct TwTab<128> { static constexpr int size = 120, off2 = 0, off3 = 24; };
template <> struct TwTab<256> { static constexpr int size = 248, off2 = 0, off3 = 56; };

template <int N, int R, int NS>
__device__ __forceinline__ void fill_pass_tw(double2* tp, const double2* __restrict__ tw_g, int tid, int nthr) {
  for (int i = tid; i < (R - 1) * NS; i += nthr) {
    const int r = i / NS + 1, k = i % NS;
    tp[i] = tw_g[r * k * (N / (NS * R))];
  }
}

// the pass tables of length N from the table W_N^t (t < N) in global memory
template <int N>
__device__ __forceinline__ void fill_tw(double2* tp, const double2* __restrict__ tw_g, int tid, int nthr) {
  if constexpr (N == 32) {
    fill_pass_tw<32, 4, 8>(tp, tw_g, tid, nthr);
  } else if constexpr (N == 64) {
    fill_pass_tw<64, 8, 8>(tp, tw_g, tid, nthr);
  } else if constexpr (N == 128) {
    fill_pass_tw<128, 4, 8>(tp + TwTab<128>::off2, tw_g, tid, nthr);
    fill_pass_tw<128, 4, 32>(tp + TwTab<128>::off3, tw_g, tid, nthr);
  } else {
    fill_pass_tw<256, 8, 8>(tp + TwTab<256>::off2, tw_g, tid, nthr);
    fill_pass_tw<256, 4, 64>(tp + TwTab<256>::off3, tw_g, tid, nthr);
  }
}

// v[b R + r] = x[j_b + r N/R] on entry; V[q] of butterfly b in v[b R + q] on
// exit; tp: this pass's twiddle table (unused when NS = 1)
template <int N, int R, int NS>
__device__ __forceinline__ void pass_reg(double2 (&v)[8], int tau, const double2* __restrict__ tp, int sign) {
  constexpr int TPS = N / 8, NB = 8 / R;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j = tau + b * TPS, k = j & (NS - 1);
    if constexpr (NS > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) {
        double2 t = tp[(r - 1) * NS + k];
        if (sign > 0) t = cconj(t);
        v[b * R + r] = cmul(v[b * R + r], t);
      }
    }
    dft_reg<R>(&v[b * R], sign);
  }
}

template <int N, int R>
__device__ __forceinline__ void load_pass(double2 (&v)[8], const double2* seq, int tau) {
  constexpr int TPS = N / 8, NB = 8 / R;
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int r = 0; r < R; ++r) v[b * R + r] = seq[swz(tau + b * TPS + r * (N / R))];
}

template <int N, int R, int NS>
__device__ __forceinline__ int out_pos(int tau, int b, int q) {
  const int j = tau + b * (N / 8);
  return (j / NS) * NS * R + (j & (NS - 1)) + q * NS;
}

template <int N, int R, int NS>
__device__ __forceinline__ void store_pass(const double2 (&v)[8], double2* seq, int tau) {
  constexpr int NB = 8 / R;
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int q = 0; q < R; ++q) seq[swz(out_pos<N, R, NS>(tau, b, q))] = v[b * R + q];
}

// The last pass of each length, for the callers' output positions.
template <int N> struct LastPass;
template <> struct LastPass<32> { static constexpr int R = 4, NS = 8; };
template <> struct LastPass<64> { static constexpr int R = 8, NS = 8; };
template <> struct LastPass<128> { static constexpr int R = 4, NS = 32; };
template <> struct LastPass<256> { static constexpr int R = 4, NS = 64; };

// v holds x[tau + r TPS] (the first pass's inputs); on exit v[b R + q] holds
// the transform at out_pos<N, LastPass R, LastPass NS>(tau, b, q).  Every lane
// of the warp calls it (the passes synchronise the warp); seq is the
// sequence's shared-memory slot (N values, swizzled), tw the pass tables
// (fill_tw).
template <int N>
__device__ __forceinline__ void fft_reg(double2 (&v)[8], double2* seq, int tau, const double2* __restrict__ tw,
                                        int sign) {
  pass_reg<N, 8, 1>(v, tau, tw, sign);
  __syncwarp();  // every lane has read its inputs (the caller's, if from seq)
  store_pass<N, 8, 1>(v, seq, tau);
  __syncwarp();
  if constexpr (N == 32) {
    load_pass<N, 4>(v, seq, tau);
    pass_reg<N, 4, 8>(v, tau, tw, sign);
  } else if constexpr (N == 64) {
    load_pass<N, 8>(v, seq, tau);
    pass_reg<N, 8, 8>(v, tau, tw, sign);
  } else if constexpr (N == 128) {
    load_pass<N, 4>(v, seq, tau);
    pass_reg<N, 4, 8>(v, tau, tw + TwTab<N>::off2, sign);
    __syncwarp();
    store_pass<N, 4, 8>(v, seq, tau);
    __syncwarp();
    load_pass<N, 4>(v, seq, tau);
    pass_reg<N, 4, 32>(v, tau, tw + TwTab<N>::off3, sign);
  } else {
    static_assert(N == 256, "length");
    load_pass<N, 8>(v, seq, tau);
    pass_reg<N, 8, 8>(v, tau, tw + TwTab<N>::off2, sign);
    __syncwarp();
    store_pass<N, 8, 8>(v, seq, tau);
    __syncwarp();
    load_pass<N, 4>(v, seq, tau);
    pass_reg<N, 4, 64>(v, tau, tw + TwTab<N>::off3, sign);
  }
}

template <int N>
__device__ __forceinline__ void store_last(const double2 (&v)[8], double2* seq, int tau) {
  store_pass<N, LastPass<N>::R, LastPass<N>::NS>(v, seq, tau);
}

// ------------------------------------------------- mixed-radix FFTs ---
// Every other length: Stockham passes between two buffers in shared memory,
// with radices up to 16 whose butterflies stay in registers (composite ones
// built from their factors), so that most lengths take two passes: one pass
// per prime factor spent its time in shared memory and in barriers (a 150-
// point transform had four).  Forward transforms only: an inverse transform
// swaps the real and imaginary parts of its input and of its output.
//
// x / d for x < 2^16 and 1 <= d <= 2^15 as a multiplication: m = floor(2^32 / d) + 1.
struct FastDiv {
  unsigned d, m;
};
__device__ __forceinline__ int fdiv_u(int x, FastDiv f) { return f.d == 1 ? x : (int)__umulhi((unsigned)x, f.m); }

// Pass of radix p after sub-transforms of length ns: np = n / p butterflies;
// its twiddles tw[off + (r-1) ns + k] = exp(-2 pi i r k / (ns p)).
struct FftPass {
  int p, off;
  FastDiv np, ns;
};
struct FftPlan {
  int n, nf;
  FftPass pass[kMaxPasses];
  const double2* tw;
};

// buffer position of element e: one slot of padding after every eight, so
// that the passes' strided writes (stride p) spread over the banks
__host__ __device__ constexpr int fpad(int e) { return e + (e >> 3); }
__host__ __device__ constexpr int fld(int n) { return fpad(n) + 1; }

// forward DFTs of P values in registers, V_q = sum_r v_r exp(-2 pi i q r / P)
template <int P>
__device__ __forceinline__ void dft_fwd(double2* v);

// coprime A, B (the prime-factor map: input n = B a + A b mod A B, output q
// with q = qa mod A and q = qb mod B): no twiddles between the factors
template <int A, int B>
__device__ __forceinline__ void dft_coprime(double2* v) {
  constexpr int N = A * B;
  double2 t[N];
#pragma unroll
  for (int b = 0; b < B; ++b) {
    double2 u[A];
#pragma unroll
    for (int a = 0; a < A; ++a) u[a] = v[(B * a + A * b) % N];
    dft_fwd<A>(u);
#pragma unroll
    for (int a = 0; a < A; ++a) t[a * B + b] = u[a];
  }
#pragma unroll
  for (int a = 0; a < A; ++a) dft_fwd<B>(&t[a * B]);
#pragma unroll
  for (int q = 0; q < N; ++q) v[q] = t[(q % A) * B + q % B];
}

// odd prime P from the cosines and sines c[r], s[r] of 2 pi r / P: the sums
// and differences of v_r and v_{P-r} take real factors
template <int P>
__device__ __forceinline__ void dft_odd(double2* v, const double (&c)[P / 2 + 1], const double (&s)[P / 2 + 1]) {
  constexpr int H = P / 2;
  double2 a[H], b[H];
#pragma unroll
  for (int r = 1; r <= H; ++r) {
    a[r - 1] = cadd(v[r], v[P - r]);
    b[r - 1] = csub(v[r], v[P - r]);
  }
  const double2 v0 = v[0];
  double2 sum = v0;
#pragma unroll
  for (int r = 0; r < H; ++r) sum = cadd(sum, a[r]);
  v[0] = sum;
#pragma unroll
  for (int q = 1; q <= H; ++q) {
    double2 e = v0, o = make_double2(0.0, 0.0);
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      const int qr = (q * r) % P, i = qr <= H ? qr : P - qr;
      const double sn = qr <= H ? s[i] : -s[i];
      e.x += c[i] * a[r - 1].x;
      e.y += c[i] * a[r - 1].y;
      o.x += sn * b[r - 1].x;
      o.y += sn * b[r - 1].y;
    }
    v[q] = make_double2(e.x + o.y, e.y - o.x);  // e - i o
    v[P - q] = make_double2(e.x - o.y, e.y + o.x);
  }
}

// A x B values with the twiddles exp(-2 pi i a b / (A B)) between the factors
template <int A, int B>
__device__ __forceinline__ void dft_square(double2* v, const double2 (&w)[A][B]) {
  double2 t[A * B];
#pragma unroll
  for (int b = 0; b < B; ++b) {  // input n = B a + b
    double2 u[A];
#pragma unroll
    for (int a = 0; a < A; ++a) u[a] = v[B * a + b];
    dft_fwd<A>(u);
#pragma unroll
    for (int a = 0; a < A; ++a) t[a * B + b] = a && b ? cmul(u[a], w[a][b]) : u[a];
  }
#pragma unroll
  for (int a = 0; a < A; ++a) {
    dft_fwd<B>(&t[a * B]);
#pragma unroll
    for (int b = 0; b < B; ++b) v[a + A * b] = t[a * B + b];
  }
}

template <> __device__ __forceinline__ void dft_fwd<2>(double2* v) { dft_reg<2>(v, -1); }
template <> __device__ __forceinline__ void dft_fwd<4>(double2* v) { dft_reg<4>(v, -1); }
template <> __device__ __forceinline__ void dft_fwd<8>(double2* v) { dft_reg<8>(v, -1); }
template <> __device__ __forceinline__ void dft_fwd<3>(double2* v) {
  const double c[2] = {1.0, -0.5}, s[2] = {0.0, 0.86602540378443864676};
  dft_odd<3>(v, c, s);
}
template <> __device__ __forceinline__ void dft_fwd<5>(double2* v) {
  const double c[3] = {1.0, 0.30901699437494742410, -0.80901699437494742410};
  const double s[3] = {0.0, 0.95105651629515357212, 0.58778525229247312917};
  dft_odd<5>(v, c, s);
}
template <> __device__ __forceinline__ void dft_fwd<7>(double2* v) {
  const double c[4] = {1.0, 0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
  const double s[4] = {0.0, 0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
  dft_odd<7>(v, c, s);
}
template <> __device__ __forceinline__ void dft_fwd<6>(double2* v) { dft_coprime<2, 3>(v); }
template <> __device__ __forceinline__ void dft_fwd<10>(double2* v) { dft_coprime<2, 5>(v); }
template <> __device__ __forceinline__ void dft_fwd<12>(double2* v) { dft_coprime<4, 3>(v); }
template <> __device__ __forceinline__ void dft_fwd<14>(double2* v) { dft_coprime<2, 7>(v); }
template <> __device__ __forceinline__ void dft_fwd<15>(double2* v) { dft_coprime<3, 5>(v); }
template <> __device__ __forceinline__ void dft_fwd<9>(double2* v) {
  constexpr double c1 = 0.76604444311897803520, s1 = 0.64278760968653932632;  // 2 pi / 9
  constexpr double c2 = 0.17364817766693034885, s2 = 0.98480775301220805937;
  constexpr double c4 = -0.93969262078590838405, s4 = 0.34202014332566873304;
  const double2 w[3][3] = {{{1, 0}, {1, 0}, {1, 0}}, {{1, 0}, {c1, -s1}, {c2, -s2}}, {{1, 0}, {c2, -s2}, {c4, -s4}}};
  dft_square<3, 3>(v, w);
}
template <> __device__ __forceinline__ void dft_fwd<16>(double2* v) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, h = 0.70710678118654752440;
  const double2 w[4][4] = {{{1, 0}, {1, 0}, {1, 0}, {1, 0}},
                           {{1, 0}, {c1, -s1}, {h, -h}, {s1, -c1}},
                           {{1, 0}, {h, -h}, {0, -1}, {-h, -h}},
                           {{1, 0}, {s1, -c1}, {-h, -h}, {-c1, s1}}};
  dft_square<4, 4>(v, w);
}

template <int P>
__device__ __forceinline__ void any_pass(const double2* in, double2* out, int nb, int ld, const FftPass& F,
                                         const double2* __restrict__ tw) {
  const int np = (int)F.np.d, ns = (int)F.ns.d;
  const double2* t = tw + F.off;
  for (int idx = threadIdx.x; idx < nb * np; idx += blockDim.x) {
    const int sq = fdiv_u(idx, F.np), j = idx - sq * np, k = j - fdiv_u(j, F.ns) * ns;
    const double2* src = in + sq * ld;
    double2 v[P];
#pragma unroll
    for (int r = 0; r < P; ++r) v[r] = src[fpad(j + r * np)];
    if (ns > 1)
#pragma unroll
      for (int r = 1; r < P; ++r) v[r] = cmul(v[r], t[(r - 1) * ns + k]);
    dft_fwd<P>(v);
    double2* dst = out + sq * ld;
    const int o = (j - k) * P + k;
#pragma unroll
    for (int q = 0; q < P; ++q) dst[fpad(o + q * ns)] = v[q];
  }
}

// any prime radix up to kMaxRadix, straight from its definition: a thread per
// output; the P-point roots are twiddles too (wroot[t] = exp(-2 pi i t / p))
__device__ __forceinline__ void prime_pass(const double2* in, double2* out, int nb, int ld, const FftPass& F,
                                           const double2* __restrict__ tw) {
  const int p = F.p, np = (int)F.np.d, ns = (int)F.ns.d, n = np * p;
  const double2* t = tw + F.off;
  const double2* root = t + (p - 1) * ns;
  for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
    const int bq = fdiv_u(idx, F.np), j = idx - bq * np, sq = bq / p, q = bq - sq * p;
    const int k = j - fdiv_u(j, F.ns) * ns;
    const double2* src = in + sq * ld;
    double2 acc = src[fpad(j)];
    int qr = 0;
    for (int r = 1; r < p; ++r) {
      qr += q;
      if (qr >= p) qr -= p;
      const double2 x = cmul(src[fpad(j + r * np)], cmul(t[(r - 1) * ns + k], root[qr]));
      acc = cadd(acc, x);
    }
    out[sq * ld + fpad((j - k) * p + k + q * ns)] = acc;
  }
}

// nb sequences of length P.n in shared memory, sequence s at b0 + s ld
// (element e at fpad(e)), transformed forward between b0 and b1; returns the
// buffer that holds the result.  Begins and ends with a block barrier.
__device__ __forceinline__ double2* fft_any(double2* b0, double2* b1, int nb, int ld, const FftPlan& P) {
  double2* in = b0;
  double2* out = b1;
  for (int f = 0; f < P.nf; ++f) {
    const FftPass& F = P.pass[f];
    __syncthreads();
    switch (F.p) {
      case 2: any_pass<2>(in, out, nb, ld, F, P.tw); break;
      case 3: any_pass<3>(in, out, nb, ld, F, P.tw); break;
      case 4: any_pass<4>(in, out, nb, ld, F, P.tw); break;
      case 5: any_pass<5>(in, out, nb, ld, F, P.tw); break;
      case 6: any_pass<6>(in, out, nb, ld, F, P.tw); break;
      case 7: any_pass<7>(in, out, nb, ld, F, P.tw); break;
      case 8: any_pass<8>(in, out, nb, ld, F, P.tw); break;
      case 9: any_pass<9>(in, out, nb, ld, F, P.tw); break;
      case 10: any_pass<10>(in, out, nb, ld, F, P.tw); break;
      case 12: any_pass<12>(in, out, nb, ld, F, P.tw); break;
      case 14: any_pass<14>(in, out, nb, ld, F, P.tw); break;
      case 15: any_pass<15>(in, out, nb, ld, F, P.tw); break;
      case 16: any_pass<16>(in, out, nb, ld, F, P.tw); break;
      default: prime_pass(in, out, nb, ld, F, P.tw); break;
    }
    double2* t = in;
    in = out;
    out = t;
  }
  __syncthreads();
  return in;
}

// Where the inverse rows put the solution: dense (f == nullptr: into the
// transform's own real array), or scaled into the interior of a field with a
// one-cell halo, value (i, j, k) (0-based) at f[(k+1) plane + (j+1) ldi + i+1].
struct RowsOut {
  double* f;
  long ldi, plane;
  double scale;
  int jtot;
};

// Forward real-to-complex transform of nb rows of nx = 2 n reals per CTA:
// z_m = x_2m + i x_2m+1, Z = FFT_n(z), then for k = 0 .. n:
// X_k = (Z_k + conj Z_{n-k}) / 2 - (i/2) W^k (Z_k - conj Z_{n-k}),
// W = exp(-2 pi i / nx), Z_n = Z_0; mode k of row r at dst[k nrows + r].
constexpr int kAnyThreads = 128;

__global__ void __launch_bounds__(kAnyThreads, 4) rows_r2c_any(long nrows, FastDiv nb, FftPlan P,
                                                            const double2* __restrict__ wpost,
                                                            const double* __restrict__ src, double2* __restrict__ dst) {
  extern __shared__ __align__(16) double2 fsm[];
  const int n = P.n, ld = fld(n);
  const long r0 = (long)blockIdx.x * nb.d;
  const int rows = (int)min((long)nb.d, nrows - r0);
  double2* b0 = fsm;
  double2* b1 = fsm + nb.d * ld;
  const double2* s2 = (const double2*)src + r0 * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < rows; r += kAnyThreads / 32)
    for (int t = lane; t < n; t += 32) b0[r * ld + fpad(t)] = s2[(long)r * n + t];
  const double2* Z = fft_any(b0, b1, rows, ld, P);
  for (int t = threadIdx.x; t < (n + 1) * (int)nb.d; t += kAnyThreads) {
    const int k = fdiv_u(t, nb), r = t - k * nb.d;
    if (r >= rows) continue;
    const double2 zk = Z[r * ld + fpad(k == n ? 0 : k)], zc = cconj(Z[r * ld + fpad(k == 0 ? 0 : n - k)]);
    const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y + zc.y));
    const double2 o = make_double2(0.5 * (zk.x - zc.x), 0.5 * (zk.y - zc.y));
    const double2 wo = cmul(wpost[k], o);  // W^k o; times -i: (wo.y, -wo.x)
    dst[(long)k * nrows + r0 + r] = make_double2(e.x + wo.y, e.y - wo.x);
  }
}

// Inverse complex-to-real rows: from the n + 1 modes X_k of a row,
// Z_k = (X_k + conj X_{n-k}) + i conj(W^k) (X_k - conj X_{n-k}), k < n,
// z = unnormalised inverse FFT_n(Z), x_2m = Re z_m, x_2m+1 = Im z_m (nx x).
__global__ void __launch_bounds__(kAnyThreads, 4) rows_c2r_any(long nrows, FastDiv nb, FftPlan P,
                                                            const double2* __restrict__ wpost,
                                                            const double2* __restrict__ src, double* __restrict__ dst,
                                                            RowsOut out) {
  extern __shared__ __align__(16) double2 fsm[];
  const int n = P.n, ld = fld(n);
  const long r0 = (long)blockIdx.x * nb.d;
  const int rows = (int)min((long)nb.d, nrows - r0);
  double2* b0 = fsm;
  double2* b1 = fsm + nb.d * ld;
  for (int t = threadIdx.x; t < (n / 2 + 1) * (int)nb.d; t += kAnyThreads) {
    const int k = fdiv_u(t, nb), r = t - k * nb.d;
    if (r >= rows) continue;
    const double2 a = src[(long)k * nrows + r0 + r], b = src[(long)(n - k) * nrows + r0 + r];
    auto z = [&](double2 x, double2 y, int q) {  // Z_q from X_q = x and X_{n-q} = y
      const double2 yc = cconj(y);
      const double2 sum = cadd(x, yc), t2 = cmul(cconj(wpost[q]), csub(x, yc));  // times i: (-t2.y, t2.x)
      return make_double2(sum.x - t2.y, sum.y + t2.x);
    };
    b0[r * ld + fpad(k)] = cswap(z(a, b, k));
    if (k > 0) b0[r * ld + fpad(n - k)] = cswap(z(b, a, n - k));
  }
  const double2* z = fft_any(b0, b1, rows, ld, P);  // swapped: (Im, Re)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < rows; r += kAnyThreads / 32) {
    const long row = r0 + r;
    if (!out.f) {
      double2* d2 = (double2*)dst + row * n;
      for (int t = lane; t < n; t += 32) d2[t] = cswap(z[r * ld + fpad(t)]);
    } else {
      const int j = (int)(row % out.jtot);
      const long k = row / out.jtot;
      double* f = out.f + (k + 1) * out.plane + (j + 1) * out.ldi + 1;
      for (int i = lane; i < 2 * n; i += 32) {
        const double2 v = z[r * ld + fpad(i >> 1)];
        f[i] = (i & 1 ? v.x : v.y) * out.scale;
      }
    }
  }
}

// y transforms: nseq contiguous sequences, nb per CTA, in place; an inverse by
// swapping parts
__global__ void __launch_bounds__(kAnyThreads, 4) cols_any(long nseq, int nb, FftPlan P, bool inv,
                                                        double2* __restrict__ data) {
  extern __shared__ __align__(16) double2 fsm[];
  const int n = P.n, ld = fld(n);
  const long s0 = (long)blockIdx.x * nb;
  const int ns = (int)min((long)nb, nseq - s0);
  double2* d = data + s0 * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < ns; r += kAnyThreads / 32)
    for (int t = lane; t < n; t += 32) {
      const double2 x = d[(long)r * n + t];
      fsm[r * ld + fpad(t)] = inv ? cswap(x) : x;
    }
  const double2* y = fft_any(fsm, fsm + nb * ld, ns, ld, P);
  for (int r = warp; r < ns; r += kAnyThreads / 32)
    for (int t = lane; t < n; t += 32) {
      const double2 x = y[r * ld + fpad(t)];
      d[(long)r * n + t] = inv ? cswap(x) : x;
    }
}

constexpr int kRegThreads = 256;

// Real-to-complex rows (complex length N = nx / 2), 256 / (N / 8) rows per
// CTA, the post-processing split of rows_r2c_any.  Loads go straight from
// global memory into the first pass's registers (a half-row run of 16-byte
// values per group of lanes); the modes are written transposed, a run of the
// CTA's rows per mode (128 to 1024 bytes).
template <int N>
__global__ void __launch_bounds__(kRegThreads) rows_r2c_reg(long nrows, const double2* __restrict__ tw_g,
                                                           const double2* __restrict__ wp_g,
                                                           const double* __restrict__ src, double2* __restrict__ dst) {
  constexpr int TPS = N / 8, SPC = kRegThreads / TPS, LD = N + 1;
  __shared__ double2 tw[TwTab<N>::size], wp[N + 1];
  __shared__ double2 buf[SPC * LD];
  fill_tw<N>(tw, tw_g, threadIdx.x, kRegThreads);
  for (int t = threadIdx.x; t <= N; t += kRegThreads) wp[t] = wp_g[t];
  const int sq = threadIdx.x / TPS, tau = threadIdx.x % TPS;
  const long row0 = (long)blockIdx.x * SPC, row = row0 + sq;
  const bool ok = row < nrows;
  const double2* s = (const double2*)src + row * N;
  double2 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = ok ? s[tau + r * TPS] : make_double2(0.0, 0.0);
  __syncthreads();  // the tables
  double2* seq = buf + sq * LD;
  fft_reg<N>(v, seq, tau, tw, -1);
  __syncwarp();
  store_last<N>(v, seq, tau);
  __syncthreads();
  const int rr = threadIdx.x % SPC, k0 = threadIdx.x / SPC;
  if (row0 + rr >= nrows) return;
  const double2* q = buf + rr * LD;
#pragma unroll
  for (int i = 0; i <= 8; ++i) {
    const int k = k0 + i * TPS;
    if (k <= N) {
      const double2 zk = q[swz(k & (N - 1))], zc = cconj(q[swz((N - k) & (N - 1))]);
      const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y + zc.y));
      const double2 od = make_double2(0.5 * (zk.x - zc.x), 0.5 * (zk.y - zc.y));
      const double2 wo = cmul(wp[k], od);
      dst[(long)k * nrows + row0 + rr] = make_double2(e.x + wo.y, e.y - wo.x);
    }
  }
}

// Complex-to-real rows, the pre-processing of rows_c2r_any: the modes of the
// CTA's rows come in transposed through shared memory (row pairs X_k,
// X_{n-k}), the first pass's inputs are formed in registers, the last pass
// writes the reals straight to global memory (16-byte runs, or pairs of
// 8-byte values into a halo field).
template <int N>
__global__ void __launch_bounds__(kRegThreads) rows_c2r_reg(long nrows, const double2* __restrict__ tw_g,
                                                           const double2* __restrict__ wp_g,
                                                           const double2* __restrict__ src, double* __restrict__ dst,
                                                           RowsOut out) {
  constexpr int TPS = N / 8, SPC = kRegThreads / TPS, LD = N + 1;
  __shared__ double2 tw[TwTab<N>::size], wp[N + 1];
  __shared__ double2 buf[SPC * LD];
  fill_tw<N>(tw, tw_g, threadIdx.x, kRegThreads);
  for (int t = threadIdx.x; t <= N; t += kRegThreads) wp[t] = wp_g[t];
  const int sq = threadIdx.x / TPS, tau = threadIdx.x % TPS;
  const long row0 = (long)blockIdx.x * SPC, row = row0 + sq;
  const bool ok = row < nrows;
  {
    const int rr = threadIdx.x % SPC, k0 = threadIdx.x / SPC;
    const bool in = row0 + rr < nrows;
#pragma unroll
    for (int i = 0; i <= 8; ++i) {
      const int k = k0 + i * TPS;
      if (k <= N) buf[rr * LD + k] = in ? src[(long)k * nrows + row0 + rr] : make_double2(0.0, 0.0);
    }
  }
  double2* seq = buf + sq * LD;  // first the row's N + 1 modes (linear), then the FFT slot
  __syncthreads();  // the tables and the modes
  double2 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int k = tau + r * TPS;
    const double2 xk = seq[k], xc = cconj(seq[N - k]);
    const double2 sum = make_double2(xk.x + xc.x, xk.y + xc.y), dif = make_double2(xk.x - xc.x, xk.y - xc.y);
    const double2 t2 = cmul(cconj(wp[k]), dif);
    v[r] = make_double2(sum.x - t2.y, sum.y + t2.x);
  }
  fft_reg<N>(v, seq, tau, tw, +1);
  if (!ok) return;
  constexpr int R = LastPass<N>::R, NS = LastPass<N>::NS;
  if (!out.f) {
    double2* d2 = (double2*)dst + row * N;
#pragma unroll
    for (int b = 0; b < 8 / R; ++b)
#pragma unroll
      for (int q = 0; q < R; ++q) d2[out_pos<N, R, NS>(tau, b, q)] = v[b * R + q];
  } else {
    const long j = row % out.jtot, k = row / out.jtot;
    double* f = out.f + (k + 1) * out.plane + (j + 1) * out.ldi + 1;
#pragma unroll
    for (int b = 0; b < 8 / R; ++b)
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int m = out_pos<N, R, NS>(tau, b, q);
        f[2 * m] = v[b * R + q].x * out.scale;
        f[2 * m + 1] = v[b * R + q].y * out.scale;
      }
  }
}

// y transforms: contiguous sequences of length N in place, 256 / (N / 8) per
// CTA, registers to registers
template <int N>
__global__ void __launch_bounds__(kRegThreads) cols_reg(long nseq, const double2* __restrict__ tw_g, int sign,
                                                       double2* __restrict__ data) {
  constexpr int TPS = N / 8, SPC = kRegThreads / TPS, LD = N + 1;
  __shared__ double2 tw[TwTab<N>::size];
  __shared__ double2 buf[SPC * LD];
  fill_tw<N>(tw, tw_g, threadIdx.x, kRegThreads);
  const int sq = threadIdx.x / TPS, tau = threadIdx.x % TPS;
  const long s = (long)blockIdx.x * SPC + sq;
  const bool ok = s < nseq;
  double2* d = data + s * N;
  double2 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = ok ? d[tau + r * TPS] : make_double2(0.0, 0.0);
  __syncthreads();
  fft_reg<N>(v, buf + sq * LD, tau, tw, sign);
  if (!ok) return;
  constexpr int R = LastPass<N>::R, NS = LastPass<N>::NS;
#pragma unroll
  for (int b = 0; b < 8 / R; ++b)
#pragma unroll
    for (int q = 0; q < R; ++q) d[out_pos<N, R, NS>(tau, b, q)] = v[b * R + q];
}

}  // namespace

namespace {

FastDiv fast_div(int d) { return FastDiv{(unsigned)d, (unsigned)((1ull << 32) / (unsigned)d) + 1u}; }

// The fewest radices whose product is n, and among those the smallest largest
// one; prime factors above 7 are passes of their own.
void best_radices(int n, std::vector<int>& cur, std::vector<int>& best) {
  static const int radices[] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  if (n == 1) {
    auto key = [](const std::vector<int>& v) { return v.empty() ? 0 : *std::max_element(v.begin(), v.end()); };
    if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && key(cur) < key(best))) best = cur;
    return;
  }
  if (!best.empty() && cur.size() + 1 > best.size()) return;
  for (int r : radices)
    if (n % r == 0 && (cur.empty() || r <= cur.back())) {
      cur.push_back(r);
      best_radices(n / r, cur, best);
      cur.pop_back();
    }
}

// passes of length n and their twiddles (appended to tw as (re, im) pairs);
// false when a prime factor is above kMaxRadix or there are too many passes
bool make_plan(int n, FftPlan& P, std::vector<double>& tw) {
  std::vector<int> rad, primes;
  int m = n;
  for (int p = 11; p <= m; p += 2)
    while (m % p == 0) {
      if (p > kMaxRadix) return false;
      primes.push_back(p);
      m /= p;
    }
  std::vector<int> cur;
  if (m > 1) best_radices(m, cur, rad);
  rad.insert(rad.end(), primes.begin(), primes.end());
  if ((int)rad.size() > kMaxPasses) return false;
  P.n = n;
  P.nf = (int)rad.size();
  int ns = 1;
  auto put = [&](double t) {  // exp(-2 pi i t)
    tw.push_back(std::cos(2.0 * kPi * t));
    tw.push_back(-std::sin(2.0 * kPi * t));
  };
  const int base = (int)(tw.size() / 2);
  for (int f = 0; f < P.nf; ++f) {
    const int p = rad[f];
    P.pass[f] = FftPass{p, (int)(tw.size() / 2) - base, fast_div(n / p), fast_div(ns)};
    for (int r = 1; r < p; ++r)
      for (int k = 0; k < ns; ++k) put((double)(r * k) / (double)(ns * p));
    if (p > 16 || p == 11 || p == 13)
      for (int t = 0; t < p; ++t) put((double)t / (double)p);
    ns *= p;
  }
  return true;
}

std::vector<double> twiddles(int n) {  // exp(-2 pi i t / n) as (re, im) pairs
  std::vector<double> w(2 * (size_t)n);
  for (int t = 0; t < n; ++t) {
    w[2 * t] = std::cos(2.0 * kPi * t / n);
    w[2 * t + 1] = -std::sin(2.0 * kPi * t / n);
  }
  return w;
}

bool pow2_fast(int n) { return n == 32 || n == 64 || n == 128 || n == 256; }

size_t tri_tile_smem(int kmax, int C) { return (sizeof(double2) + sizeof(double)) * (size_t)kmax * C; }

// sequences per CTA of the mixed-radix row and column kernels: about 1280
// values (two padded buffers: 46 KB, four CTAs of 128 threads on an SM)
int any_rows(int n) { return std::max(1, std::min(16, 1280 / n)); }
size_t any_smem(int n) { return sizeof(double2) * 2 * any_rows(n) * fld(n); }

#define SG_POW2_DISPATCH(n, call) \
  switch (n) {                    \
    case 32: call(32); break;     \
    case 64: call(64); break;     \
    case 128: call(128); break;   \
    default: call(256); break;    \
  }

struct Plans {
  FftPlan x, y;
};

}  // namespace

int poisson_setup(sg_ctx* c, unsigned types) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  const long nxm = f.itot / 2 + 1, nslots = nxm * f.jtot;
  void* p = nullptr;
  auto tables = [&]() -> int {
    for (int e = 0; e < 4; ++e)
      if ((types >> e & 1u) && !s.zt[e]) {
        SG_TRY(dalloc(c, p, sizeof(double) * nslots * f.ktot), "alloc");
        s.zt[e] = (double*)p;
      }
    return SG_OK;
  };
  if (s.ready) return tables();
  if (f.itot % 2 != 0 || f.ktot < 4) return fail(c, SG_ERR_CONFIG, "solver1d here needs an even itot and ktot >= 4");
  const long nreal = (long)f.itot * f.jtot * f.ktot;
  SG_TRY(dalloc(c, p, sizeof(double) * nreal), "alloc");
  s.r = (double*)p;
  SG_TRY(dalloc(c, p, sizeof(double2) * nslots * f.ktot), "alloc");
  s.c = p;
  SG_RET(tables());
  // initsolver.f90:111-130: xrt(2m) = xrt(2m+1) = -4 dxi^2 sin(2m pi / (2 itot))^2, the
  // modes of a real transform in x; in y the complex modes j and jtot - j share yrt
  std::vector<double> tab(nxm + f.jtot);
  const double dxi = 1.0 / (f.lx / f.itot), dyi = 1.0 / (f.ly / f.jtot);
  for (long m = 0; m < nxm; ++m) tab[m] = -4. * dxi * dxi * std::pow(std::sin((double)(2 * m) * kPi / (2. * f.itot)), 2.);
  for (int j = 0; j < f.jtot; ++j) {
    const int jm = std::min(j, f.jtot - j);
    tab[nxm + j] = -4. * dyi * dyi * std::pow(std::sin((double)(2 * jm) * kPi / (2. * f.jtot)), 2.);
  }
  SG_TRY(dalloc(c, p, sizeof(double) * tab.size()), "alloc");
  s.tab = (double*)p;
  SG_TRY(cudaMemcpy(s.tab, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice), "upload");
  // FFT plans: complex length itot/2 for the rows (real length itot), jtot
  // for the y transforms.  Tables, one after the other: the register
  // transforms' exp(-2 pi i t / n) of both lengths, the row split's
  // W^k = exp(-2 pi i k / itot), k <= itot/2, then the mixed-radix passes' own.
  Plans pl{};
  const int n = f.itot / 2;
  std::vector<double> w = twiddles(n), wy = twiddles(f.jtot), wp(2 * (size_t)nxm), px, py;
  if (n > kMaxLength || f.jtot > kMaxLength || !make_plan(n, pl.x, px) || !make_plan(f.jtot, pl.y, py))
    return fail(c, SG_ERR_CONFIG, "solver1d here needs itot/2 and jtot of at most 2048 whose prime factors are "
                                  "at most 61");
  for (long k = 0; k < nxm; ++k) {
    wp[2 * k] = std::cos(2.0 * kPi * k / f.itot);
    wp[2 * k + 1] = -std::sin(2.0 * kPi * k / f.itot);
  }
  const size_t opx = w.size() / 2 + wy.size() / 2 + wp.size() / 2, opy = opx + px.size() / 2;
  w.insert(w.end(), wy.begin(), wy.end());
  w.insert(w.end(), wp.begin(), wp.end());
  w.insert(w.end(), px.begin(), px.end());
  w.insert(w.end(), py.begin(), py.end());
  SG_TRY(dalloc(c, p, sizeof(double) * w.size()), "alloc");
  SG_TRY(cudaMemcpy(p, w.data(), sizeof(double) * w.size(), cudaMemcpyHostToDevice), "upload");
  s.w = (double2*)p;
  pl.x.tw = s.w + opx;
  pl.y.tw = s.w + opy;
  s.wpost = s.w + n + f.jtot;
  static_assert(sizeof(Plans) <= sizeof(s.plans), "plan storage");
  std::memcpy(s.plans, &pl, sizeof(pl));
  s.ready = true;
  return SG_OK;
}

void poisson_free(sg_ctx* c) { (void)c; }

namespace {

template <int N>
void launch_r2c(long nrows, const double2* tw, const double2* wp, const double* r, double2* m, cudaStream_t st) {
  constexpr int SPC = kRegThreads / (N / 8);
  rows_r2c_reg<N><<<(unsigned)((nrows + SPC - 1) / SPC), kRegThreads, 0, st>>>(nrows, tw, wp, r, m);
}
template <int N>
void launch_c2r(long nrows, const double2* tw, const double2* wp, const double2* m, double* r, const RowsOut& o,
                cudaStream_t st) {
  constexpr int SPC = kRegThreads / (N / 8);
  rows_c2r_reg<N><<<(unsigned)((nrows + SPC - 1) / SPC), kRegThreads, 0, st>>>(nrows, tw, wp, m, r, o);
}
template <int N>
void launch_cols(long nseq, const double2* tw, int sign, double2* m, cudaStream_t st) {
  constexpr int SPC = kRegThreads / (N / 8);
  cols_reg<N><<<(unsigned)((nseq + SPC - 1) / SPC), kRegThreads, 0, st>>>(nseq, tw, sign, m);
}

template <int C>
cudaError_t launch_tri_tile(int kmax, int jtot, int nxm, int e, double a, const double* zt, double2* c,
                            cudaStream_t st) {
  const size_t smem = tri_tile_smem(kmax, C);
  cudaError_t err = smem_limit(tri_tile_kernel<C>, smem);
  if (err != cudaSuccess) return err;
  tri_tile_kernel<C><<<dim3((unsigned)((jtot + C - 1) / C), (unsigned)nxm), kTriThreads, smem, st>>>(kmax, jtot, e, a,
                                                                                                   zt, c);
  return cudaGetLastError();
}

// The widest tile of which at least three fit an SM (runs of 256, 128 or 64
// bytes); tiles of four columns as long as one fits, then global memory.
cudaError_t launch_tri(int kmax, int jtot, int nxm, int e, double a, const double* zt, double2* c, cudaStream_t st) {
  constexpr size_t third = 72 * 1024, most = 220 * 1024;
  if (tri_tile_smem(kmax, 16) <= third) return launch_tri_tile<16>(kmax, jtot, nxm, e, a, zt, c, st);
  if (tri_tile_smem(kmax, 8) <= third) return launch_tri_tile<8>(kmax, jtot, nxm, e, a, zt, c, st);
  if (tri_tile_smem(kmax, 4) <= most) return launch_tri_tile<4>(kmax, jtot, nxm, e, a, zt, c, st);
  tri_apply_kernel<<<(unsigned)((2L * nxm * jtot + 127) / 128), 128, 0, st>>>(kmax, jtot, nxm, e, a, zt, c);
  return cudaGetLastError();
}

}  // namespace

int poisson_solve(sg_ctx* c, double* r, int e, double shift, cudaStream_t st, const PoisOut* out) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  Plans pl;
  std::memcpy(&pl, s.plans, sizeof(pl));
  const int n = f.itot / 2, nxm = n + 1;
  const long nrows = (long)f.jtot * f.ktot;
  const RowsOut ro{out ? out->f : nullptr, out ? out->ldi : 0, out ? out->plane : 0, out ? out->scale : 0.0, f.jtot};
  const double dzi = 1.0 / (f.lz / f.ktot);
  double2* modes = (double2*)s.c;
  const double2* twx = s.w;
  const double2* twy = s.w + n;
  int launches = 5;
  if (e < 0 || e > 3 || !s.zt[e]) return fail(c, SG_ERR_STATE, "solver1d: tables of this row type were not set up");
  if (!s.tvalid[e] || s.tshift[e] != shift) {
    // (re)build the tables for this shift; inside a stream capture the build
    // is recorded but has not run, so they are not marked valid for the
    // direct calls that may come before the graph's first launch
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    SG_TRY(cudaStreamIsCapturing(st, &cap), "solver1d");
    tri_coeff_kernel<<<(unsigned)((nxm * f.jtot + 127) / 128), 128, 0, st>>>(f.ktot, f.jtot, nxm, e, dzi, shift, s.tab,
                                                                             s.tab + nxm, s.zt[e]);
    s.tvalid[e] = cap == cudaStreamCaptureStatusNone;
    s.tshift[e] = shift;
    launches += 1;
  }
  // x rows to modes
  const int rx = any_rows(n);
  const unsigned gx = (unsigned)((nrows + rx - 1) / rx);
  if (pow2_fast(n)) {
#define SG_R2C(N) launch_r2c<N>(nrows, twx, s.wpost, r, modes, st)
    SG_POW2_DISPATCH(n, SG_R2C)
#undef SG_R2C
  } else {
    SG_TRY(smem_limit(rows_r2c_any, any_smem(n)), "fft");
    rows_r2c_any<<<gx, kAnyThreads, any_smem(n), st>>>(nrows, fast_div(rx), pl.x, s.wpost, r, modes);
  }
  // y transforms, elimination, inverse y transforms
  const long nseq = (long)nxm * f.ktot;
  const int ry = any_rows(f.jtot);
  auto cols = [&](int sign) -> int {
    if (pow2_fast(f.jtot)) {
#define SG_COLS(N) launch_cols<N>(nseq, twy, sign, modes, st)
      SG_POW2_DISPATCH(f.jtot, SG_COLS)
#undef SG_COLS
    } else {
      SG_TRY(smem_limit(cols_any, any_smem(f.jtot)), "fft");
      cols_any<<<(unsigned)((nseq + ry - 1) / ry), kAnyThreads, any_smem(f.jtot), st>>>(nseq, ry, pl.y, sign > 0, modes);
    }
    return SG_OK;
  };
  SG_RET(cols(-1));
  SG_TRY(launch_tri(f.ktot, f.jtot, nxm, e, dzi * dzi, s.zt[e], modes, st), "solver1d");
  SG_RET(cols(+1));
  // modes to x rows
  if (pow2_fast(n)) {
#define SG_C2R(N) launch_c2r<N>(nrows, twx, s.wpost, modes, r, ro, st)
    SG_POW2_DISPATCH(n, SG_C2R)
#undef SG_C2R
  } else {
    SG_TRY(smem_limit(rows_c2r_any, any_smem(n)), "fft");
    rows_c2r_any<<<gx, kAnyThreads, any_smem(n), st>>>(nrows, fast_div(rx), pl.x, s.wpost, modes, r, ro);
  }
  SG_TRY(cudaGetLastError(), "solver1d");
  c->launches += launches;
  return SG_OK;
}

}  // namespace sg
