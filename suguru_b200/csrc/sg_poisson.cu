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
// A solve is five launches: rows_r2c, cols, tri_tile, cols, rows_c2r.  The
// flow step's four solves and its projection run together in mode space
// (poisson_project): the three right-hand sides are transformed in one launch
// per direction, tri_flow_tile solves u, v, w, takes their divergence, solves
// the pressure correction and corrects the three on chip, and the inverse
// rows write the fields with their halos.
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

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cswap(double2 a) { return make_double2(a.y, a.x); }

// x / d for x < 2^16 and 1 <= d <= 2^15 as a multiplication: m = floor(2^32 / d) + 1.
struct FastDiv {
  unsigned d, m;
};
__device__ __forceinline__ int fdiv_u(int x, FastDiv f) { return f.d == 1 ? x : (int)__umulhi((unsigned)x, f.m); }

// A tile of C neighbouring columns of one x mode in shared memory, and the
// elimination on it.  The sweeps are first-order recurrences
//   q_k = al_k q_{k-1} + z_k r_k,  x_k = q_k + al_k x_{k+1},  al_k = -a z_k
// (a = dzi^2 is both a_k, k >= 1, and c_k), the same for the real and the
// imaginary parts.  A chain of all levels takes 34 cycles a level, 8,700 for
// 128 levels up and down, with two warps busy; so the levels are cut into 16
// segments, and a warp sweeps two columns, lane = 2 segment + column: from a
// zero start for the segment's end value and the product of its al, which
// shuffles compose into the true starts, then from those.  The way up from the
// true start also sums what the segment hands down (x at its first level from
// a zero above it is the sum of q_k times the al below k), so the levels are
// read three times.  |al| <= 1, so the composition loses nothing.  Bound by
// shared memory: eight segments with a lane per real column and four reads
// took half as many wavefronts again (the flow step's kernel 170 us at
// 256 x 256 x 128, now 155 us).  Rows of a segment are shifted by 32 bytes per
// segment (pivots: 16), so that the warp's lanes fall on different banks.
constexpr int kSegs = 16;

template <int C>
struct Tile {
  FastDiv len;  // levels per segment
  __device__ __forceinline__ int at(int k, int jl) const { return k * C + jl + 2 * fdiv_u(k, len); }
};
__host__ __device__ constexpr int tile_size(int kmax, int C) { return kmax * C + 2 * kSegs; }

// (f, p) <- the maps x -> f x + p of the segments up to the lane's own
// (down: from the top), composed; returns what enters the lane's segment.
template <bool DOWN>
__device__ __forceinline__ double2 compose_segments(double f, double2 p, int seg) {
#pragma unroll
  for (int d = 1; d < kSegs; d *= 2) {
    double ft, px, py;
    if (DOWN) {
      ft = __shfl_down_sync(0xffffffffu, f, 2 * d);
      px = __shfl_down_sync(0xffffffffu, p.x, 2 * d);
      py = __shfl_down_sync(0xffffffffu, p.y, 2 * d);
    } else {
      ft = __shfl_up_sync(0xffffffffu, f, 2 * d);
      px = __shfl_up_sync(0xffffffffu, p.x, 2 * d);
      py = __shfl_up_sync(0xffffffffu, p.y, 2 * d);
    }
    if (DOWN ? seg + d < kSegs : seg >= d) {
      p = make_double2(fma(f, px, p.x), fma(f, py, p.y));
      f *= ft;
    }
  }
  const bool first = seg == (DOWN ? kSegs - 1 : 0);
  const double2 in = DOWN ? make_double2(__shfl_down_sync(0xffffffffu, p.x, 2), __shfl_down_sync(0xffffffffu, p.y, 2))
                          : make_double2(__shfl_up_sync(0xffffffffu, p.x, 2), __shfl_up_sync(0xffffffffu, p.y, 2));
  return first ? make_double2(0.0, 0.0) : in;
}

// Columns 2 col2 and 2 col2 + 1 of the tile; whole warps.
template <int C>
__device__ __forceinline__ void tri_tile_sweeps(double2* tile, const double* zs, int col2, int kmax, int len, int e,
                                                double a) {
  const int lane = threadIdx.x & 31, seg = lane >> 1, k0 = seg * len;
  const int n = min(len, kmax - k0), nu = min(n, kmax - 1 - k0), o = k0 * C + 2 * seg + 2 * col2 + (lane & 1);
  double2* c = tile + o;
  const double* z = zs + o;
  double f = 1.0;
  double2 p = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int t = 0; t < nu; ++t) {
    const double w = z[t * C], al = -(a * w);
    const double2 r = c[t * C];
    p = make_double2(fma(al, p.x, r.x * w), fma(al, p.y, r.y * w));
    f *= al;
  }
  __syncwarp();
  p = compose_segments<false>(f, p, seg);
  double g = 1.0;
  double2 d = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int t = 0; t < nu; ++t) {
    const double w = z[t * C], al = -(a * w);
    const double2 r = c[t * C];
    p = make_double2(fma(al, p.x, r.x * w), fma(al, p.y, r.y * w));
    c[t * C] = p;
    d = make_double2(fma(g, p.x, d.x), fma(g, p.y, d.y));
    g *= al;
  }
  if (n > 0 && k0 + n == kmax) {  // the top row: its pivot itself is tabulated; e = 3: the identity row of w
    const double w = z[nu * C], al = e == 3 ? 0.0 : -a;
    const double2 r = c[nu * C];
    p = w != 0.0 ? make_double2(fma(al, p.x, r.x) / w, fma(al, p.y, r.y) / w) : make_double2(0.0, 0.0);
    c[nu * C] = p;
    d = make_double2(fma(g, p.x, d.x), fma(g, p.y, d.y));
  }
  __syncwarp();
  p = compose_segments<true>(f, d, seg);
#pragma unroll 4
  for (int t = n - 1; t >= 0; --t) {  // (the top row's al only meets zeros)
    const double al = -(a * z[t * C]);
    const double2 r = c[t * C];
    p = make_double2(fma(al, p.x, r.x), fma(al, p.y, r.y));
    c[t * C] = p;
  }
}

// C columns, all levels, per CTA: copied to shared memory with their pivots,
// solved there, written back; each mode is read and written once.  Memory-
// bound (24 bytes in and 16 out per mode, 176 MB at 256 x 256 x 128); runs of
// 256 bytes (C = 16) beat 128 and 64.
template <int C>
__global__ void __launch_bounds__(16 * C) tri_tile_kernel(int kmax, int jtot, FastDiv len, int e, double a,
                                                          const double* __restrict__ zt, double2* __restrict__ c) {
  extern __shared__ __align__(16) double2 tsm[];  // modes, then pivots
  const Tile<C> T{len};
  double* zs = (double*)(tsm + tile_size(kmax, C));
  const int j0 = blockIdx.x * C, nj = min(C, jtot - j0);
  const long o = (long)blockIdx.y * kmax * jtot + j0;
  const int jl = threadIdx.x % C, k0 = threadIdx.x / C;
  if (jl < nj)
    for (int k = k0; k < kmax; k += 16) {
      stage_async(&tsm[T.at(k, jl)], &c[o + (long)k * jtot + jl]);
      stage_async(&zs[T.at(k, jl)], &zt[o + (long)k * jtot + jl]);
    }
  stage_wait();
  __syncthreads();
  tri_tile_sweeps<C>(tsm, zs, threadIdx.x >> 5, kmax, len.d, e, a);
  __syncthreads();
  if (jl < nj)
    for (int k = k0; k < kmax; k += 16) c[o + (long)k * jtot + jl] = tsm[T.at(k, jl)];
}

// The two sweeps of one real column in global memory, at c[k cs] with its
// pivots at z[k zs], in blocks of B levels, the next block's loads ahead of
// the block's arithmetic in the other of two register sets.
template <int B>
__device__ __forceinline__ void tri_sweeps(double* c, const double* z, long cs, long zs, int kmax, int e, double a) {
  const int last = kmax - 1, nb = (last - 1) / B;  // full blocks of rows 1 .. last - 1
  double r0[B], w0[B], r1[B], w1[B], p;
  auto load = [&](double(&r)[B], double(&w)[B], int k, int dir) {
    const double *ck = c + k * cs, *zk = z + k * zs;
#pragma unroll
    for (int t = 0; t < B; ++t) {
      r[t] = ck[dir * t * cs];
      w[t] = zk[dir * t * zs];
    }
  };
  auto up = [&](const double(&r)[B], const double(&w)[B], int k) {
    double* ck = c + k * cs;
#pragma unroll
    for (int t = 0; t < B; ++t) {
      p = fma(-(a * w[t]), p, r[t] * w[t]);
      ck[t * cs] = p;
    }
  };
  auto down = [&](const double(&r)[B], const double(&w)[B], int k) {
    double* ck = c + k * cs;
#pragma unroll
    for (int t = 0; t < B; ++t) {
      p = fma(-(a * w[t]), p, r[t]);
      ck[-t * cs] = p;
    }
  };
  int k = 1;
  if (nb > 0) load(r0, w0, k, 1);
  p = c[0] * z[0];
  c[0] = p;
  for (int b = 0; b < nb; b += 2) {
    if (b + 1 < nb) load(r1, w1, k + B, 1);
    up(r0, w0, k);
    k += B;
    if (b + 1 < nb) {
      if (b + 2 < nb) load(r0, w0, k + B, 1);
      up(r1, w1, k);
      k += B;
    }
  }
  for (; k < last; ++k) {
    const double w = z[k * zs];
    p = fma(-(a * w), p, c[k * cs] * w);
    c[k * cs] = p;
  }
  {
    const double zk = z[last * zs], al = e == 3 ? 0.0 : a;  // e = 3: the identity row of w at the top
    p = zk != 0.0 ? fma(-al, p, c[last * cs]) / zk : 0.0;
    c[last * cs] = p;
  }
  k = last - 1;
  for (int t = (last - 1) - nb * B; t > 0; --t, --k) {
    p = fma(-(a * z[k * zs]), p, c[k * cs]);
    c[k * cs] = p;
  }
  if (nb > 0) load(r0, w0, k, -1);
  for (int b = 0; b < nb; b += 2) {
    if (b + 1 < nb) load(r1, w1, k - B, -1);
    down(r0, w0, k);
    k -= B;
    if (b + 1 < nb) {
      if (b + 2 < nb) load(r0, w0, k - B, -1);
      down(r1, w1, k);
      k -= B;
    }
  }
  c[0] = fma(-(a * z[0]), p, c[0]);
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

// The flow step's solves and projection for C columns of one x mode, all
// levels: u and v (e = 2), w (e = 3), the divergence over dt (fillps), the
// pressure correction (e = 1) and the corrected velocities (correc), on the
// modes in shared memory.  A difference along x or y is a factor per mode,
// with ex = exp(-2 pi i m / itot) and ey = exp(-2 pi i j / jtot):
//   u(i) - u(i-1) -> (1 - ex) u,   p(i+1) - p(i) -> (conj(ex) - 1) p;
// w(0) = 0 in the divergence, and the top row of w, zero, takes no
// correction (p(k1) = p(kmax)).  72 bytes in and 64 out per mode, 590 MB at
// 256 x 256 x 128 (91 us; 155 measured): shared memory and the phases' barriers
// bound it.  In physical space the same steps moved the modes of all four
// fields twice more, and u, v, w and p once each through fillps and correc.
struct FlowModes {
  double2 *u, *v, *w, *p;                      // [m][k][j]
  const double *z2, *z3, *z1;                  // pivots of e = 2, 3, 1
  const double2 *ex, *ey;
  double sx, sy, sz;                           // dxi / dt, dyi / dt, dzi / dt
  double gx, gy, gz;                           // dt dxi, dt dyi, dt dzi
};

__device__ __forceinline__ double2 mode_divergence(const FlowModes& F, double2 dx, double2 dy, double2 u, double2 v,
                                                   double2 w, double2 wl) {
  const double2 a = cmul(dx, u), b = cmul(dy, v);
  return make_double2((w.x - wl.x) * F.sz + b.x * F.sy + a.x * F.sx, (w.y - wl.y) * F.sz + b.y * F.sy + a.y * F.sx);
}

// u -= dt dxi (conj(ex) - 1) p, with dx = 1 - ex: conj(ex) - 1 = -conj(dx)
__device__ __forceinline__ double2 mode_corrected(double2 u, double2 dx, double2 p, double g) {
  const double2 q = cmul(cconj(dx), p);
  return make_double2(u.x + g * q.x, u.y + g * q.y);
}

template <int C>
__global__ void __launch_bounds__(48 * C) tri_flow_tile_kernel(int kmax, int jtot, FastDiv len, double a, FlowModes F) {
  extern __shared__ __align__(16) double2 tsm[];  // u, v, w, then the pivots z2, z3, z1
  const Tile<C> T{len};
  const int n = tile_size(kmax, C);
  double2 *su = tsm, *sv = su + n, *sw = sv + n;
  double *z2 = (double*)(sw + n), *z3 = z2 + n, *z1 = z3 + n;
  double2* sp = (double2*)z2;  // the pressure correction takes the place of z2, z3 after their use
  const int j0 = blockIdx.x * C, nj = min(C, jtot - j0), m = blockIdx.y;
  const long o = (long)m * kmax * jtot + j0;
  const int jl = threadIdx.x % C, k0 = threadIdx.x / C, warp = threadIdx.x >> 5;
  if (jl < nj)
    for (int k = k0; k < kmax; k += 48) {
      const int q = T.at(k, jl);
      const long g = o + (long)k * jtot + jl;
      stage_async(&su[q], &F.u[g]);
      stage_async(&sv[q], &F.v[g]);
      stage_async(&sw[q], &F.w[g]);
      stage_async(&z2[q], &F.z2[g]);
      stage_async(&z3[q], &F.z3[g]);
      stage_async(&z1[q], &F.z1[g]);
    }
  stage_wait();
  __syncthreads();
  {  // C / 2 warps (two columns each) for each of u, v, w
    const int f = warp / (C / 2), c2 = warp - f * (C / 2);
    tri_tile_sweeps<C>(f == 0 ? su : f == 1 ? sv : sw, f == 2 ? z3 : z2, c2, kmax, len.d, f == 2 ? 3 : 2, a);
  }
  __syncthreads();
  const double2 ex = F.ex[m], ey = F.ey[min(j0 + jl, jtot - 1)];
  const double2 dx = make_double2(1.0 - ex.x, -ex.y), dy = make_double2(1.0 - ey.x, -ey.y);
  if (jl < nj)
    for (int k = k0; k < kmax; k += 48) {
      const int q = T.at(k, jl);
      sp[q] = mode_divergence(F, dx, dy, su[q], sv[q], sw[q], k ? sw[T.at(k - 1, jl)] : make_double2(0.0, 0.0));
    }
  __syncthreads();
  if (warp < C / 2) tri_tile_sweeps<C>(sp, z1, warp, kmax, len.d, 1, a);
  __syncthreads();
  if (jl < nj)
    for (int k = k0; k < kmax; k += 48) {
      const int q = T.at(k, jl);
      const long g = o + (long)k * jtot + jl;
      const double2 p = sp[q], pu = k + 1 < kmax ? sp[T.at(k + 1, jl)] : p;
      F.u[g] = mode_corrected(su[q], dx, p, F.gx);
      F.v[g] = mode_corrected(sv[q], dy, p, F.gy);
      F.w[g] = make_double2(sw[q].x - F.gz * (pu.x - p.x), sw[q].y - F.gz * (pu.y - p.y));
      F.p[g] = p;
    }
}

// The same on global memory, for columns too long for a tile: the divergence
// of the solved velocities, and after the pressure solve their correction
__global__ void mode_divergence_kernel(int kmax, int jtot, long n, FlowModes F) {
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const int j = (int)(g % jtot), k = (int)(g / jtot % kmax), m = (int)(g / ((long)jtot * kmax));
  const double2 ex = F.ex[m], ey = F.ey[j];
  F.p[g] = mode_divergence(F, make_double2(1.0 - ex.x, -ex.y), make_double2(1.0 - ey.x, -ey.y), F.u[g], F.v[g], F.w[g],
                           k ? F.w[g - jtot] : make_double2(0.0, 0.0));
}
__global__ void mode_correct_kernel(int kmax, int jtot, long n, FlowModes F) {
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const int j = (int)(g % jtot), k = (int)(g / jtot % kmax), m = (int)(g / ((long)jtot * kmax));
  const double2 ex = F.ex[m], ey = F.ey[j], p = F.p[g], pu = k + 1 < kmax ? F.p[g + jtot] : p;
  F.u[g] = mode_corrected(F.u[g], make_double2(1.0 - ex.x, -ex.y), p, F.gx);
  F.v[g] = mode_corrected(F.v[g], make_double2(1.0 - ey.x, -ey.y), p, F.gy);
  const double2 w = F.w[g];
  F.w[g] = make_double2(w.x - F.gz * (pu.x - p.x), w.y - F.gz * (pu.y - p.y));
}

// ---------------------------------------------------------------- FFT ---
constexpr int kMaxRadix = 61;
constexpr int kMaxPasses = 8;
constexpr int kMaxLength = 2048;

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
// transform's own real array), or scaled into a field with a one-cell halo,
// halo cells included: the periodic images in x and y, and the wall planes by
// bounduvw's and boundp's rules (bound.f90:7-139).
struct RowsOut {
  double* f;
  long ldi, plane;
  double scale, lo, hi;  // wall values: f(0) = lo - f(1), f(k1) = hi - f(kmax) (u, v)
  int itot, jtot, ktot;
  int kind;              // 0: u or v; 1: w (zero at the bottom, f(k1) = f(kmax-1)); 2: pressure, added to f
};
struct RowsOuts {
  RowsOut o[4];
};

// Row (j, k) (0-based) of a field and the rows it is copied to: its periodic
// image in y, and beside a wall the halo plane's row and that row's image.
// Consecutive lanes put consecutive cells (a thread that stored its own pairs
// of cells filled half of each sector it touched: 161 against 127 us for the
// four fields of a flow step at 256 x 256 x 128).
struct RowTarget {
  double *f, *img, *wall, *wall_img;
  double scale, wa, wc;  // wall value: wc + wa x
  int nx;
  bool add;
  __device__ __forceinline__ RowTarget(const RowsOut& o, int j, int k) {
    const int jh = j == 0 ? o.jtot + 1 : (j == o.jtot - 1 ? 0 : -1);
    int kh = -1;
    wa = 1.0;
    wc = 0.0;
    if (o.kind == 1) {
      if (k == 0) { kh = 0; wa = 0.0; }
      if (k == o.ktot - 2) kh = o.ktot + 1;
    } else if (k == 0 || k == o.ktot - 1) {
      kh = k == 0 ? 0 : o.ktot + 1;
      if (o.kind == 0) { wa = -1.0; wc = k == 0 ? o.lo : o.hi; }
    }
    auto row = [&](int jj, int kk) { return o.f + kk * o.plane + jj * o.ldi; };
    f = row(j + 1, k + 1);
    img = jh >= 0 ? row(jh, k + 1) : nullptr;
    wall = kh >= 0 ? row(j + 1, kh) : nullptr;
    wall_img = kh >= 0 && jh >= 0 ? row(jh, kh) : nullptr;
    scale = o.scale;
    nx = o.itot;
    add = o.kind == 2;
  }
  __device__ __forceinline__ void store(double* r, int i, double x) const {
    r[i] = x;
    if (i == 1) r[nx + 1] = x;
    if (i == nx) r[0] = x;
  }
  __device__ __forceinline__ void copies(int i, double x) const {
    if (img) store(img, i, x);
    if (wall) {
      x = wa == 0.0 ? 0.0 : wc + wa * x;
      store(wall, i, x);
      if (wall_img) store(wall_img, i, x);
    }
  }
};

// Forward real-to-complex transform of nb rows of nx = 2 n reals per CTA:
// z_m = x_2m + i x_2m+1, Z = FFT_n(z), then for k = 0 .. n:
// X_k = (Z_k + conj Z_{n-k}) / 2 - (i/2) W^k (Z_k - conj Z_{n-k}),
// W = exp(-2 pi i / nx), Z_n = Z_0; mode k of row r at dst[k nrows + r].
constexpr int kAnyThreads = 128;

// The CTA's rows of n values, contiguous in global memory, into its padded
// slots.  Ten loads of a thread are issued before their stores (up to 1280
// values, what any_rows gives a CTA, in one round): these kernels hold 16
// warps an SM and wait for memory first.  With a load at a time, and a pair or
// a cell at a time in rows_c2r_any, 180 x 150 x 99 took 65 us (forward rows of
// three fields), 108 (columns), 116 (inverse rows of four); now 47, 88, 85.
// SWAP: real and imaginary parts exchanged.
template <bool SWAP>
__device__ __forceinline__ void stage_rows(double2* s, const double2* g, int rows, int ld, FastDiv n) {
  constexpr int H = 10;
  const int total = rows * (int)n.d;
  for (int t0 = threadIdx.x; t0 < total; t0 += H * kAnyThreads) {
    double2 x[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int t = t0 + h * kAnyThreads;
      x[h] = t < total ? g[t] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int t = t0 + h * kAnyThreads;
      if (t >= total) break;
      const int r = fdiv_u(t, n);
      s[r * ld + fpad(t - r * (int)n.d)] = SWAP ? cswap(x[h]) : x[h];
    }
  }
}

__global__ void __launch_bounds__(kAnyThreads, 4) rows_r2c_any(long nrows, FastDiv nb, FastDiv nd, FftPlan P,
                                                            const double2* __restrict__ wpost,
                                                            const double* __restrict__ src, double2* __restrict__ dst) {
  extern __shared__ __align__(16) double2 fsm[];
  const int n = P.n, ld = fld(n);
  src += (long)blockIdx.y * nrows * 2 * n;  // field
  dst += (long)blockIdx.y * nrows * (n + 1);
  const long r0 = (long)blockIdx.x * nb.d;
  const int rows = (int)min((long)nb.d, nrows - r0);
  double2* b0 = fsm;
  double2* b1 = fsm + nb.d * ld;
  stage_rows<false>(b0, (const double2*)src + r0 * n, rows, ld, nd);
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
                                                            RowsOuts outs) {
  extern __shared__ __align__(16) double2 fsm[];
  const int n = P.n, ld = fld(n);
  const RowsOut& out = outs.o[blockIdx.y];  // field
  src += (long)blockIdx.y * nrows * (n + 1);
  const long r0 = (long)blockIdx.x * nb.d;
  const int rows = (int)min((long)nb.d, nrows - r0);
  double2* b0 = fsm;
  double2* b1 = fsm + nb.d * ld;
  // mode pairs (k, n - k) of the rows, six of a thread loaded before they are used
  constexpr int H = 6;
  const int total = (n / 2 + 1) * (int)nb.d;
  for (int t0 = threadIdx.x; t0 < total; t0 += H * kAnyThreads) {
    double2 a[H], b[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int t = t0 + h * kAnyThreads, k = fdiv_u(t, nb), r = t - k * (int)nb.d;
      const bool in = t < total && r < rows;
      a[h] = in ? src[(long)k * nrows + r0 + r] : make_double2(0.0, 0.0);
      b[h] = in ? src[(long)(n - k) * nrows + r0 + r] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int t = t0 + h * kAnyThreads, k = fdiv_u(t, nb), r = t - k * (int)nb.d;
      if (t >= total || r >= rows) continue;
      auto z = [&](double2 x, double2 y, int q) {  // Z_q from X_q = x and X_{n-q} = y
        const double2 yc = cconj(y);
        const double2 sum = cadd(x, yc), t2 = cmul(cconj(wpost[q]), csub(x, yc));  // times i: (-t2.y, t2.x)
        return make_double2(sum.x - t2.y, sum.y + t2.x);
      };
      b0[r * ld + fpad(k)] = cswap(z(a[h], b[h], k));
      if (k > 0) b0[r * ld + fpad(n - k)] = cswap(z(b[h], a[h], n - k));
    }
  }
  const double2* z = fft_any(b0, b1, rows, ld, P);  // swapped: (Im, Re)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < rows; r += kAnyThreads / 32) {
    const long row = r0 + r;
    if (!out.f) {
      double2* d2 = (double2*)dst + row * n;
      for (int t = lane; t < n; t += 32) d2[t] = cswap(z[r * ld + fpad(t)]);
    } else {
      const int kr = (int)row / out.jtot;  // a field has less than 2^31 rows
      const RowTarget t(out, (int)row - kr * out.jtot, kr);
      const double* zr = (const double*)(z + r * ld);
      for (int i0 = lane; i0 < 2 * n; i0 += H * 32) {
        double x[H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const int i = i0 + 32 * h;
          x[h] = i < 2 * n ? t.scale * zr[2 * fpad(i >> 1) + 1 - (i & 1)] : 0.0;
        }
        if (t.add)
#pragma unroll
          for (int h = 0; h < H; ++h)
            if (i0 + 32 * h < 2 * n) x[h] = t.f[i0 + 32 * h + 1] + x[h];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const int i = i0 + 32 * h + 1;
          if (i > 2 * n) continue;
          t.store(t.f, i, x[h]);
          t.copies(i, x[h]);
        }
      }
    }
  }
}

// y transforms: nseq contiguous sequences, nb per CTA, in place; an inverse by
// swapping parts
__global__ void __launch_bounds__(kAnyThreads, 4) cols_any(long nseq, int nb, FastDiv nd, FftPlan P, bool inv,
                                                        double2* __restrict__ data) {
  extern __shared__ __align__(16) double2 fsm[];
  const int n = P.n, ld = fld(n);
  const long s0 = (long)blockIdx.x * nb;
  const int ns = (int)min((long)nb, nseq - s0);
  double2* d = data + s0 * n;
  if (inv)
    stage_rows<true>(fsm, d, ns, ld, nd);
  else
    stage_rows<false>(fsm, d, ns, ld, nd);
  const double2* y = fft_any(fsm, fsm + nb * ld, ns, ld, P);
  for (int t = threadIdx.x; t < ns * n; t += kAnyThreads) {
    const int r = fdiv_u(t, nd);
    const double2 x = y[r * ld + fpad(t - r * n)];
    d[t] = inv ? cswap(x) : x;
  }
}

constexpr int kRegThreads = 256;

// Real-to-complex rows (complex length N = nx / 2), 256 / (N / 8) rows per
// CTA, the post-processing split of rows_r2c_any.  Loads go straight from
// global memory into the first pass's registers (a half-row run of 16-byte
// values per group of lanes); the modes are written transposed, a run of the
// CTA's rows per mode (128 to 1024 bytes).  Bound by shared memory (83 % of its
// wavefronts; DRAM half busy): a thread forms modes k and N - k from one read
// of Z_k and Z_{N-k} (three fields of 256 x 256 x 128: 73 us, 79 with each
// mode reading both for itself).
template <int N>
__global__ void __launch_bounds__(kRegThreads) rows_r2c_reg(long nrows, const double2* __restrict__ tw_g,
                                                           const double2* __restrict__ wp_g,
                                                           const double* __restrict__ src, double2* __restrict__ dst) {
  constexpr int TPS = N / 8, SPC = kRegThreads / TPS, LD = N + 1;
  src += (long)blockIdx.y * nrows * 2 * N;  // field
  dst += (long)blockIdx.y * nrows * (N + 1);
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
  double2* d = dst + row0 + rr;
#pragma unroll
  for (int i = 0; i <= 4; ++i) {  // the pair k, N - k, k <= N / 2
    const int k = k0 + i * TPS;
    if (k > N / 2) continue;
    const double2 a = q[swz(k)], b = q[swz((N - k) & (N - 1))];
    auto mode = [&](double2 zk, double2 zn, double2 w) {
      const double2 zc = cconj(zn);
      const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y + zc.y));
      const double2 od = make_double2(0.5 * (zk.x - zc.x), 0.5 * (zk.y - zc.y));
      const double2 wo = cmul(w, od);
      return make_double2(e.x + wo.y, e.y - wo.x);
    };
    d[(long)k * nrows] = mode(a, b, wp[k]);
    if (k < N / 2) d[(long)(N - k) * nrows] = mode(b, a, wp[N - k]);
  }
}

// Complex-to-real rows, the pre-processing of rows_c2r_any: a thread reads the
// modes X_k and X_{N-k} of a row (runs of the CTA's rows per mode), forms Z_k
// and Z_{N-k}, and hands them over through shared memory to the lanes of the
// row; the last pass writes the reals straight to global memory in 16-byte
// runs, or through the slot into a field and its halo (RowTarget).  Bound by
// shared memory: with the modes handed over instead, each read twice, four
// fields of 256 x 256 x 128 took 134 us, now 127.
template <int N>
__global__ void __launch_bounds__(kRegThreads) rows_c2r_reg(long nrows, const double2* __restrict__ tw_g,
                                                           const double2* __restrict__ wp_g,
                                                           const double2* __restrict__ src, double* __restrict__ dst,
                                                           RowsOuts outs) {
  constexpr int TPS = N / 8, SPC = kRegThreads / TPS, LD = N + 1;
  const RowsOut& out = outs.o[blockIdx.y];  // field
  src += (long)blockIdx.y * nrows * (N + 1);
  __shared__ double2 tw[TwTab<N>::size], wp[N + 1];
  __shared__ double2 buf[SPC * LD];
  fill_tw<N>(tw, tw_g, threadIdx.x, kRegThreads);
  for (int t = threadIdx.x; t <= N; t += kRegThreads) wp[t] = wp_g[t];
  const int sq = threadIdx.x / TPS, tau = threadIdx.x % TPS;
  const long row0 = (long)blockIdx.x * SPC, row = row0 + sq;
  const bool ok = row < nrows;
  double2* seq = buf + sq * LD;  // first Z of the row (linear), then the FFT slot
  double2 v[8];
  {
    const int rr = threadIdx.x % SPC, k0 = threadIdx.x / SPC;
    const bool in = row0 + rr < nrows;
    const double2* g = src + row0 + rr;
    double2 xa[5], xb[5];  // X_k and X_{N-k}, k <= N / 2
#pragma unroll
    for (int i = 0; i <= 4; ++i) {
      const int k = k0 + i * TPS;
      const bool h = in && k <= N / 2;
      xa[i] = h ? g[(long)k * nrows] : make_double2(0.0, 0.0);
      xb[i] = h ? g[(long)(N - k) * nrows] : make_double2(0.0, 0.0);
    }
    __syncthreads();  // the tables
    double2* q = buf + rr * LD;
#pragma unroll
    for (int i = 0; i <= 4; ++i) {
      const int k = k0 + i * TPS;
      if (k > N / 2) continue;
      auto z = [&](double2 x, double2 y, double2 w) {  // Z_k from X_k = x and X_{N-k} = y
        const double2 c = cconj(y), t = cmul(cconj(w), csub(x, c));
        return make_double2((x.x + c.x) - t.y, (x.y + c.y) + t.x);
      };
      q[k] = z(xa[i], xb[i], wp[k]);
      if (k > 0 && k < N / 2) q[N - k] = z(xb[i], xa[i], wp[N - k]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = seq[tau + r * TPS];
  fft_reg<N>(v, seq, tau, tw, +1);
  if (!out.f) {
    if (!ok) return;
    constexpr int R = LastPass<N>::R, NS = LastPass<N>::NS;
    double2* d2 = (double2*)dst + row * N;
#pragma unroll
    for (int b = 0; b < 8 / R; ++b)
#pragma unroll
      for (int q = 0; q < R; ++q) d2[out_pos<N, R, NS>(tau, b, q)] = v[b * R + q];
    return;
  }
  __syncwarp();
  store_last<N>(v, seq, tau);
  __syncwarp();
  if (!ok) return;
  const int kr = (int)row / out.jtot;  // a field has less than 2^31 rows
  const RowTarget t(out, (int)row - kr * out.jtot, kr);
  const double* xs = (const double*)seq;
  double x[16];  // cells tau + q TPS + 1
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int i = tau + q * TPS;
    x[q] = t.scale * xs[2 * swz(i >> 1) + (i & 1)];
  }
  double* f = t.f + 1 + tau;
  if (t.add)
#pragma unroll
    for (int q = 0; q < 16; ++q) x[q] = f[q * TPS] + x[q];
#pragma unroll
  for (int q = 0; q < 16; ++q) f[q * TPS] = x[q];
  if (tau == 0) t.f[2 * N + 1] = x[0];
  if (tau == TPS - 1) t.f[0] = x[15];
  if (t.img || t.wall)
#pragma unroll
    for (int q = 0; q < 16; ++q) t.copies(tau + q * TPS + 1, x[q]);
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
  int big = n;  // without its factors 2, 3, 5 and 7
  for (int p : {2, 3, 5, 7})
    while (big % p == 0) big /= p;
  const int m = n / big;
  for (int p = 11; p <= big; p += 2)
    while (big % p == 0) {
      if (p > kMaxRadix) return false;
      primes.push_back(p);
      big /= p;
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

size_t tri_tile_smem(int kmax, int C) { return (sizeof(double2) + sizeof(double)) * (size_t)tile_size(kmax, C); }
FastDiv segment_length(int kmax) { return fast_div((kmax + kSegs - 1) / kSegs); }

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

int poisson_setup(sg_ctx* c, unsigned types, int nfields) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  const long nxm = f.itot / 2 + 1, nslots = nxm * f.jtot;
  void* p = nullptr;
  auto tables = [&]() -> int {
    for (int e = 0; e < 4; ++e)
      if ((types >> e & 1u) && s.zt[e].empty()) {
        SG_TRY(dalloc(c, p, sizeof(double) * nslots * f.ktot), "alloc");
        s.zt[e].push_back({(double*)p, 0.0, false, false});
      }
    return SG_OK;
  };
  const long nreal = (long)f.itot * f.jtot * f.ktot;
  auto fields = [&]() -> int {  // real and mode arrays for nfields fields at once
    if (s.nfields >= nfields) return SG_OK;
    SG_TRY(dalloc(c, p, sizeof(double) * nreal * std::min(nfields, 3)), "alloc");
    s.r = (double*)p;
    SG_TRY(dalloc(c, p, sizeof(double2) * nslots * f.ktot * nfields), "alloc");
    s.c = p;
    s.nfields = nfields;
    return SG_OK;
  };
  if (s.ready) {
    SG_RET(fields());
    return tables();
  }
  if (f.itot % 2 != 0 || f.ktot < 4) return fail(c, SG_ERR_CONFIG, "solver1d here needs an even itot and ktot >= 4");
  SG_RET(fields());
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



namespace {

template <int N>
void launch_r2c(long nrows, int nf, const double2* tw, const double2* wp, const double* r, double2* m,
                cudaStream_t st) {
  constexpr int SPC = kRegThreads / (N / 8);
  rows_r2c_reg<N><<<dim3((unsigned)((nrows + SPC - 1) / SPC), nf), kRegThreads, 0, st>>>(nrows, tw, wp, r, m);
}
template <int N>
void launch_c2r(long nrows, int nf, const double2* tw, const double2* wp, const double2* m, double* r,
                const RowsOuts& o, cudaStream_t st) {
  constexpr int SPC = kRegThreads / (N / 8);
  rows_c2r_reg<N><<<dim3((unsigned)((nrows + SPC - 1) / SPC), nf), kRegThreads, 0, st>>>(nrows, tw, wp, m, r, o);
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
  tri_tile_kernel<C><<<dim3((unsigned)((jtot + C - 1) / C), (unsigned)nxm), 16 * C, smem, st>>>(
      kmax, jtot, segment_length(kmax), e, a, zt, c);
  return cudaGetLastError();
}

constexpr size_t kThirdOfSm = 75 * 1024, kTileMost = 220 * 1024;

cudaError_t launch_tri_apply(int kmax, int jtot, int nxm, int e, double a, const double* zt, double2* c,
                             cudaStream_t st) {
  tri_apply_kernel<<<(unsigned)((2L * nxm * jtot + 127) / 128), 128, 0, st>>>(kmax, jtot, nxm, e, a, zt, c);
  return cudaGetLastError();
}

// The widest tile of which at least three fit an SM (runs of 256, 128 or 64
// bytes); tiles of four columns as long as one fits, then global memory.
cudaError_t launch_tri(int kmax, int jtot, int nxm, int e, double a, const double* zt, double2* c, cudaStream_t st) {
  if (tri_tile_smem(kmax, 16) <= kThirdOfSm) return launch_tri_tile<16>(kmax, jtot, nxm, e, a, zt, c, st);
  if (tri_tile_smem(kmax, 8) <= kThirdOfSm) return launch_tri_tile<8>(kmax, jtot, nxm, e, a, zt, c, st);
  if (tri_tile_smem(kmax, 4) <= kTileMost) return launch_tri_tile<4>(kmax, jtot, nxm, e, a, zt, c, st);
  return launch_tri_apply(kmax, jtot, nxm, e, a, zt, c, st);
}

template <int C>
cudaError_t launch_flow_tile(int kmax, int jtot, int nxm, double a, const FlowModes& F, cudaStream_t st) {
  const size_t smem = 3 * tri_tile_smem(kmax, C);
  cudaError_t err = smem_limit(tri_flow_tile_kernel<C>, smem);
  if (err != cudaSuccess) return err;
  tri_flow_tile_kernel<C><<<dim3((unsigned)((jtot + C - 1) / C), (unsigned)nxm), 48 * C, smem, st>>>(
      kmax, jtot, segment_length(kmax), a, F);
  return cudaGetLastError();
}

// Likewise for the flow step's four solves, three times the tile's memory: eight
// columns to 129 levels, then four.  Up to 193 levels two tiles of eight fit an
// SM, beyond one; a flow step with them against four columns took 715 and 740 us
// at 256 x 256 x 130, 857 and 867 at 160 levels, 1,147 and 1,094 at 200 (one tile),
// 1,465 and 1,431 at 256; 180 x 150 x 132 460 and 475, x 200 702 and 668: the line
// costs up to 4 % just above 129 levels.
cudaError_t launch_flow_tri(int kmax, int jtot, int nxm, double a, const FlowModes& F, cudaStream_t st, int& launches) {
  launches += 1;
  if (3 * tri_tile_smem(kmax, 8) <= kThirdOfSm) return launch_flow_tile<8>(kmax, jtot, nxm, a, F, st);
  if (3 * tri_tile_smem(kmax, 4) <= kTileMost) return launch_flow_tile<4>(kmax, jtot, nxm, a, F, st);
  const long n = (long)nxm * kmax * jtot;
  const unsigned nb = (unsigned)((n + 255) / 256);
  cudaError_t e = launch_tri(kmax, jtot, nxm, 2, a, F.z2, F.u, st);
  if (e == cudaSuccess) e = launch_tri(kmax, jtot, nxm, 2, a, F.z2, F.v, st);
  if (e == cudaSuccess) e = launch_tri(kmax, jtot, nxm, 3, a, F.z3, F.w, st);
  if (e != cudaSuccess) return e;
  mode_divergence_kernel<<<nb, 256, 0, st>>>(kmax, jtot, n, F);
  e = launch_tri(kmax, jtot, nxm, 1, a, F.z1, F.p, st);
  if (e != cudaSuccess) return e;
  mode_correct_kernel<<<nb, 256, 0, st>>>(kmax, jtot, n, F);
  launches += 5;
  return cudaGetLastError();
}

// The pivots z of row type e for this shift, (re)built if there are none.  An
// eager solve takes the table of the shift or rebuilds the free one, or
// another when graphs have pinned all.  A solve that is being captured pins
// the table of its shift; with none made yet, or when kMostPinned others are
// pinned, the graph builds its own in `graph` each time it runs (a flow step
// of 256 x 256 x 128 then takes 758 us against 720, of 64^3 58 against 49),
// which is for graphs of a time step never taken eagerly or of a third one.
// The Neumann rows have one shift, zero: whoever builds their table writes
// the same values, so a graph may build it where eager solves read.
int poisson_tables(sg_ctx* c, int e, double shift, cudaStream_t st, const double*& z) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  const int nxm = f.itot / 2 + 1;
  if (e < 0 || e > 3 || s.zt[e].empty())
    return fail(c, SG_ERR_STATE, "solver1d: tables of this row type were not set up");
  auto& T = s.zt[e];
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  SG_TRY(cudaStreamIsCapturing(st, &cap), "solver1d");
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  const size_t bytes = sizeof(double) * nxm * f.jtot * f.ktot;
  int pinned = 0;
  for (const auto& t : T) pinned += t.pinned;
  for (auto& t : T)
    if (t.made && t.shift == shift && (!capturing || t.pinned || pinned < s.kMostPinned)) {
      t.pinned = t.pinned || capturing;
      z = t.z;
      return SG_OK;
    }
  double* to = nullptr;
  sg_ctx::PoissonState::Pivots* own = nullptr;  // the eager table that is rebuilt
  if (capturing && e < 2) {
    to = T[0].z;
  } else if (capturing) {
    if (!s.graph[e]) {
      // an allocation is not part of the capture
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      SG_TRY(cudaThreadExchangeStreamCaptureMode(&mode), "solver1d");
      const cudaError_t err = dalloc(c, s.graph[e], bytes);
      SG_TRY(cudaThreadExchangeStreamCaptureMode(&mode), "solver1d");
      SG_TRY(err, "alloc");
    }
    to = s.graph[e];
  } else {
    auto free = std::find_if(T.begin(), T.end(), [](const auto& t) { return !t.pinned; });
    if (free == T.end()) {
      SG_TRY(dalloc(c, to, bytes), "alloc");
      T.push_back({to, 0.0, false, false});
      free = T.end() - 1;
    }
    own = &*free;
    *own = {free->z, shift, false, false};
    to = own->z;
  }
  tri_coeff_kernel<<<(unsigned)((nxm * f.jtot + 127) / 128), 128, 0, st>>>(
      f.ktot, f.jtot, nxm, e, 1.0 / (f.lz / f.ktot), shift, s.tab, s.tab + nxm, to);
  SG_TRY(cudaGetLastError(), "solver1d");
  if (own) own->made = true;
  c->launches += 1;
  z = to;
  return SG_OK;
}

// nf real fields [nf][ktot][jtot][itot] to their modes [nf][m][k][j]
int rows_forward(sg_ctx* c, int nf, const double* r, double2* modes, cudaStream_t st) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  Plans pl;
  std::memcpy(&pl, s.plans, sizeof(pl));
  const int n = f.itot / 2, nb = any_rows(n);
  const long nrows = (long)f.jtot * f.ktot;
  if (pow2_fast(n)) {
#define SG_R2C(N) launch_r2c<N>(nrows, nf, s.w, s.wpost, r, modes, st)
    SG_POW2_DISPATCH(n, SG_R2C)
#undef SG_R2C
  } else {
    SG_TRY(smem_limit(rows_r2c_any, any_smem(n)), "fft");
    rows_r2c_any<<<dim3((unsigned)((nrows + nb - 1) / nb), nf), kAnyThreads, any_smem(n), st>>>(nrows, fast_div(nb), fast_div(n),
                                                                                              pl.x, s.wpost, r, modes);
  }
  SG_TRY(cudaGetLastError(), "solver1d");
  c->launches += 1;
  return SG_OK;
}

int rows_inverse(sg_ctx* c, int nf, const double2* modes, double* r, const RowsOuts& out, cudaStream_t st) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  Plans pl;
  std::memcpy(&pl, s.plans, sizeof(pl));
  const int n = f.itot / 2, nb = any_rows(n);
  const long nrows = (long)f.jtot * f.ktot;
  if (pow2_fast(n)) {
#define SG_C2R(N) launch_c2r<N>(nrows, nf, s.w, s.wpost, modes, r, out, st)
    SG_POW2_DISPATCH(n, SG_C2R)
#undef SG_C2R
  } else {
    SG_TRY(smem_limit(rows_c2r_any, any_smem(n)), "fft");
    rows_c2r_any<<<dim3((unsigned)((nrows + nb - 1) / nb), nf), kAnyThreads, any_smem(n), st>>>(nrows, fast_div(nb), pl.x,
                                                                                              s.wpost, modes, r, out);
  }
  SG_TRY(cudaGetLastError(), "solver1d");
  c->launches += 1;
  return SG_OK;
}

// y transforms of the modes of nf fields, in place
int cols_transform(sg_ctx* c, int nf, int sign, double2* modes, cudaStream_t st) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  Plans pl;
  std::memcpy(&pl, s.plans, sizeof(pl));
  const int n = f.itot / 2, nb = any_rows(f.jtot);
  const long nseq = (long)nf * (n + 1) * f.ktot;
  if (pow2_fast(f.jtot)) {
#define SG_COLS(N) launch_cols<N>(nseq, s.w + n, sign, modes, st)
    SG_POW2_DISPATCH(f.jtot, SG_COLS)
#undef SG_COLS
  } else {
    SG_TRY(smem_limit(cols_any, any_smem(f.jtot)), "fft");
    cols_any<<<(unsigned)((nseq + nb - 1) / nb), kAnyThreads, any_smem(f.jtot), st>>>(nseq, nb, fast_div(f.jtot),
                                                                                     pl.y, sign > 0, modes);
  }
  SG_TRY(cudaGetLastError(), "solver1d");
  c->launches += 1;
  return SG_OK;
}

}  // namespace

int poisson_solve(sg_ctx* c, double* r, int e, double shift, cudaStream_t st) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  const double dzi = 1.0 / (f.lz / f.ktot);
  double2* modes = (double2*)s.c;
  const double* zt = nullptr;
  SG_RET(poisson_tables(c, e, shift, st, zt));
  SG_RET(rows_forward(c, 1, r, modes, st));
  SG_RET(cols_transform(c, 1, -1, modes, st));
  SG_TRY(launch_tri(f.ktot, f.jtot, f.itot / 2 + 1, e, dzi * dzi, zt, modes, st), "solver1d");
  c->launches += 1;
  SG_RET(cols_transform(c, 1, +1, modes, st));
  return rows_inverse(c, 1, modes, r, RowsOuts{}, st);
}

int poisson_project(sg_ctx* c, const double* r3, double dt, double shift, double* u, double* v, double* w, double* p,
                    double vb2, double vt2, cudaStream_t st) {
  auto& s = c->pois;
  const sg_config& f = c->cfg;
  const int nxm = f.itot / 2 + 1;
  const double dxi = 1.0 / (f.lx / f.itot), dyi = 1.0 / (f.ly / f.jtot), dzi = 1.0 / (f.lz / f.ktot), dti = 1.0 / dt;
  const long nm = (long)nxm * f.ktot * f.jtot;
  double2* M = (double2*)s.c;
  const double *z1 = nullptr, *z2 = nullptr, *z3 = nullptr;
  SG_RET(poisson_tables(c, 2, shift, st, z2));
  SG_RET(poisson_tables(c, 3, shift, st, z3));
  SG_RET(poisson_tables(c, 1, 0.0, st, z1));
  SG_RET(rows_forward(c, 3, r3, M, st));
  SG_RET(cols_transform(c, 3, -1, M, st));
  const FlowModes F{M,        M + nm,   M + 2 * nm, M + 3 * nm,   z2,         z3,         z1,         s.wpost,
                    s.w + f.itot / 2, dti * dxi, dti * dyi, dti * dzi, dt * dxi, dt * dyi, dt * dzi};
  int launches = 0;
  SG_TRY(launch_flow_tri(f.ktot, f.jtot, nxm, dzi * dzi, F, st, launches), "solver1d");
  c->launches += launches;
  SG_RET(cols_transform(c, 4, +1, M, st));
  const IBGrid& g = c->grid;
  const long plane = (long)g.ldi * g.ldj;
  const double scale = 1.0 / ((double)f.itot * f.jtot);
  const RowsOuts o{{{u, g.ldi, plane, scale, 0.0, 0.0, f.itot, f.jtot, f.ktot, 0},
                    {v, g.ldi, plane, scale, vb2, vt2, f.itot, f.jtot, f.ktot, 0},
                    {w, g.ldi, plane, scale, 0.0, 0.0, f.itot, f.jtot, f.ktot, 1},
                    {p, g.ldi, plane, scale, 0.0, 0.0, f.itot, f.jtot, f.ktot, 2}}};
  return rows_inverse(c, 4, M, nullptr, o, st);
}

}  // namespace sg
