// sg_flow_solver.cu -- one step of the reference's FFT flow solver
// (fsolver = 'f', main.f90:333-347) on the GPU, FP64:
//
//  fftuvw (fftuvw.f90:13-127): per interior cell the right-hand sides
//      Rep (-(momxp) - (momxad) - uo / dt), and likewise for v and w:
//      momxp = -dxi (p(i+1) - p(i)) + forcex (mom.f90:113-134), momxad the
//      Adams-Bashforth convection 1.5 (level n) - 0.5 (level n-1) of the
//      face fluxes (mom.f90:9-54, 136-181, 266-311); the w right-hand side
//      is zero in the top row; then the Helmholtz solves of solver1d after
//      initsolver(3) for w and initsolver(2) for u and v (sg_poisson.cu);
//  bounduvw (bound.f90:7-86): wall rows and periodic x, y halos;
//  fillps (fillps.f90): the divergence over dt, solver1d after
//      initsolver(1), boundp;
//  correc (correc.f90): the velocity minus dt times the pressure gradient,
//      bounduvw; pnew += p, boundp.
//
// Two parts: the right-hand sides here, then everything from the solves to
// the updated pressure in mode space (poisson_project, sg_poisson.cu).
#include <cmath>

#include "sg_common.cuh"
#include "sg_ctx.h"

namespace sg {
namespace {

struct FGrid {
  int itot, jtot, ktot, ldi, ldj;
  long plane;
  double dxi, dyi, dzi;
};

__device__ __forceinline__ long at(const FGrid& g, int i, int j, int k) {
  return (long)k * g.plane + (long)j * g.ldi + i;
}

struct Fields {
  const double* f[7];   // u, v, w of level n, of level n-1, p
  const double* fb[3];  // IB force
};

// fftuvw's right-hand sides of u, v and w into the solver's layout
// [field][k-1][j-1][i-1].
//
// The convection of the three components shares six products per grid point
// and level: with the sums U_x = u(i) + u(i+1) and so on, the fluxes through
// the faces between the point and its upper neighbours are (times 1/4)
//   U_x U_x,  U_y V_x,  U_z W_x,  V_y V_y,  V_z W_y,  W_z W_z,
// and every component's face flux is one of them, here or at the lower
// neighbour.  A thread per point forms them for both levels, combined as
// 1.5 (n) - 0.5 (n-1) at once, and takes the lower neighbours' in x and y
// from shared memory and in z from its own previous step: about 80 FP64
// operations a cell instead of 270 when each component's stencil was
// evaluated by itself.  Blocks of 32 x 8 cells march up kMomZ levels, the
// first step for the z fluxes below only; the threads hold the block's points
// with one more column and row on either side, each loads its point of every
// field once per level, one level ahead of its use, and the upper neighbours
// in x and y come through shared memory too (loading them from global memory
// kept 24 loads a cell in the way of the arithmetic: 250 us at
// 256 x 256 x 128; the arrays' 870 MB take 134 us).
constexpr int kMomX = 32, kMomY = 8, kMomZ = 16;
constexpr int kMomW = kMomX + 2, kMomPts = kMomW * (kMomY + 2), kMomThreads = (kMomPts + 31) / 32 * 32;

constexpr int kMomRow = kMomPts + kMomW;  // slots per array, the last row's upper neighbours included
constexpr size_t kMomSmem = sizeof(double) * 2 * (7 + 5) * kMomRow;

__global__ void __launch_bounds__(kMomThreads, 2) momentum_rhs_kernel(FGrid g, Fields F, double dt, double rep,
                                                                   double* __restrict__ r) {
  // two levels of: the seven fields, then XX, XY, XZ, YY, YZ of the points
  extern __shared__ __align__(16) double smom[];
  const int nbx = (g.itot + kMomX - 1) / kMomX, t = threadIdx.x;
  const int fx = t % kMomW, fy = t / kMomW;
  const int i = (int)(blockIdx.x % nbx) * kMomX + fx, j = (int)(blockIdx.x / nbx) * kMomY + fy;
  const bool cell = t < kMomPts && fx > 0 && fy > 0 && fx <= kMomX && fy <= kMomY && i <= g.itot && j <= g.jtot;
  const int k0 = (int)blockIdx.y * kMomZ + 1, k1 = min(k0 + kMomZ, g.ktot + 1);
  const int plane = (int)g.plane;  // a field has less than 2^31 values
  int o = (int)at(g, min(i, g.itot + 1), min(j, g.jtot + 1), k0 - 1);
  const long n = (long)g.itot * g.jtot * g.ktot;
  double* q = r + ((long)(k0 - 1) * g.jtot + (j - 1)) * g.itot + (i - 1);
  const double dti = 1.0 / dt;
  double cur[7], nx[7], zprev[3] = {0.0, 0.0, 0.0};  // XZ, YZ, ZZ of the level below
  double fo[3] = {0.0, 0.0, 0.0};
  double part[3] = {0.0, 0.0, 0.0};  // the previous level's right-hand sides but for its lower neighbours' fluxes
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    cur[c] = F.f[c][o];
    nx[c] = F.f[c][o + plane];
  }
  // the level's fluxes at the lower neighbours complete its right-hand sides
  auto finish = [&](int k) {
    const double* se = smom + (14 + 5 * (k & 1)) * kMomRow + t;
    auto at = [&](int h, int d) { return se[h * kMomRow - d]; };
    q[0] = (part[0] - (g.dxi * at(0, 1) + g.dyi * at(1, kMomW))) * rep;
    q[n] = (part[1] - (g.dxi * at(1, 1) + g.dyi * at(3, kMomW))) * rep;
    // dwdt(i,j,kmax) = 0 (fftuvw.f90:86-92)
    q[2 * n] = k == g.ktot ? 0.0 : (part[2] - (g.dxi * at(2, 1) + g.dyi * at(4, kMomW))) * rep;
    q += (long)g.jtot * g.itot;
  };
  for (int k = k0 - 1; k < k1; ++k) {
    // the level after the next, and the next level's forces, ahead of their use
    double nn[7], fn[3];
    const bool more = k + 1 < k1;
    o += plane;
#pragma unroll
    for (int c = 0; c < 7; ++c) nn[c] = more ? F.f[c][o + plane] : 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) fn[c] = more && cell ? F.fb[c][o] : 0.0;
    double* s = smom + 7 * (k & 1) * kMomRow + t;
    double* se = smom + (14 + 5 * (k & 1)) * kMomRow + t;
    if (t < kMomPts)
#pragma unroll
      for (int c = 0; c < 7; ++c) s[c * kMomRow] = cur[c];
    __syncthreads();  // this level's fields and the previous level's fluxes
    if (cell && k > k0) finish(k - 1);
    if (t < kMomPts) {
      // XX, XY, XZ, YY, YZ, ZZ of both levels, 1/4 (1.5 (n) - 0.5 (n-1))
      double e[6];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const int a = 3 * l, b = a + 1, c = a + 2;
        const double ux = cur[a] + s[a * kMomRow + 1], uy = cur[a] + s[a * kMomRow + kMomW], uz = cur[a] + nx[a];
        const double vx = cur[b] + s[b * kMomRow + 1], vy = cur[b] + s[b * kMomRow + kMomW], vz = cur[b] + nx[b];
        const double wx = cur[c] + s[c * kMomRow + 1], wy = cur[c] + s[c * kMomRow + kMomW], wz = cur[c] + nx[c];
        const double m[6] = {ux * ux, uy * vx, uz * wx, vy * vy, vz * wy, wz * wz};
#pragma unroll
        for (int h = 0; h < 6; ++h) e[h] = l == 0 ? 0.375 * m[h] : e[h] - 0.125 * m[h];
      }
#pragma unroll
      for (int h = 0; h < 5; ++h) se[h * kMomRow] = e[h];
      const double dp[3] = {s[6 * kMomRow + 1] - cur[6], s[6 * kMomRow + kMomW] - cur[6], nx[6] - cur[6]};
      const double dd[3] = {g.dxi, g.dyi, g.dzi};
      const double up[3] = {g.dxi * e[0] + g.dyi * e[1] + g.dzi * (e[2] - zprev[0]),
                            g.dxi * e[1] + g.dyi * e[3] + g.dzi * (e[4] - zprev[1]),
                            g.dxi * e[2] + g.dyi * e[4] + g.dzi * (e[5] - zprev[2])};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double v = cur[c] * dti;
        v = fma(fma(-v, dt, cur[c]), dti, v);  // cur / dt: the product and one residual correction
        part[c] = dd[c] * dp[c] - fo[c] + up[c] - v;
      }
      zprev[0] = e[2];
      zprev[1] = e[4];
      zprev[2] = e[5];
    }
#pragma unroll
    for (int c = 0; c < 7; ++c) {
      cur[c] = nx[c];
      nx[c] = nn[c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) fo[c] = fn[c];
  }
  __syncthreads();
  if (cell) finish(k1 - 1);
}

}  // namespace

int flow_setup(sg_ctx* c, double rep, double vb2, double vt2) {
  if (c->mixed) return fail(c, SG_ERR_CONFIG, "the flow solver runs on FP64 contexts");
  if (!(rep > 0.0) || !std::isfinite(rep) || !std::isfinite(vb2) || !std::isfinite(vt2))
    return fail(c, SG_ERR_ARG, "rep must be positive and finite, the wall values finite");
  SG_RET(poisson_setup(c, (1u << 1) | (1u << 2) | (1u << 3), 4));
  auto& s = c->flow;
  s.rep = rep;
  s.vb2 = vb2;
  s.vt2 = vt2;
  if (s.ready) return SG_OK;
  const sg_config& f = c->cfg;
  if (f.mem == SG_MEM_HOST)
    for (int q = 0; q < 13; ++q) SG_TRY(dalloc(c, s.stage[q], sizeof(double) * c->nfield), "alloc");
  s.ready = true;
  return SG_OK;
}

int flow_run(sg_ctx* c, double dt, const double* uo, const double* vo, const double* wo, const double* uoo,
             const double* voo, const double* woo, double* p, const double* fx, const double* fy, const double* fz,
             double* u, double* v, double* w) {
  const sg_config& f = c->cfg;
  auto& s = c->flow;
  cudaStream_t st = c->st;
  const IBGrid& ib = c->grid;
  FGrid g{f.itot, f.jtot, f.ktot, ib.ldi, ib.ldj, (long)ib.ldi * ib.ldj, 1.0 / (f.lx / f.itot),
          1.0 / (f.ly / f.jtot), 1.0 / (f.lz / f.ktot)};
  const Fields F{{uo, vo, wo, uoo, voo, woo, p}, {fx, fy, fz}};
  const dim3 mgrid((unsigned)(((f.itot + kMomX - 1) / kMomX) * ((f.jtot + kMomY - 1) / kMomY)),
                   (unsigned)((f.ktot + kMomZ - 1) / kMomZ));
  SG_TRY(smem_limit(momentum_rhs_kernel, kMomSmem), "momentum");
  momentum_rhs_kernel<<<mgrid, kMomThreads, kMomSmem, st>>>(g, F, dt, s.rep, c->pois.r);
  SG_TRY(cudaGetLastError(), "momentum");
  c->launches += 1;
  SG_RET(poisson_project(c, c->pois.r, dt, s.rep / dt, u, v, w, p, s.vb2, s.vt2, st));
  return SG_OK;
}

}  // namespace sg
