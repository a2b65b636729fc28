// sg_bending.cu -- the membrane kernel with the bending terms of ibend = 1
// (param.f90:90-91) on the GPU.
//
// With bending, cal_spectral_force (sph.f90:1523-1755) also synthesises the
// third and fourth derivatives of the shape (cal_co_tang_basis2 with
// ibend = 1, sph3.f90:137-180) and adds the moment's transverse shear and its
// divergence to the equilibrium (sph.f90:1705-1709), in the form of
// bending_force (sg_mechanics.cuh).
//
// Here: a fourth Legendre synthesis problem per degree group (the third and
// fourth theta derivatives of the shape's series, one extra contraction launch
// after the analysis), and a membrane kernel that evaluates the whole chain per
// point.  The kernel computes every capsule of the context (capsules with a
// zero bending modulus skip the bending terms), one point per thread.
#include <algorithm>
#include <vector>

#include "sg_ctx.h"
#include "sg_longitude.cuh"
#include "sg_mechanics.cuh"

namespace sg {

namespace {

// Staged values per (row, m): G's 18 (ccs = 2c + cos/sin, kind P, dP, d2P at
// 3 ccs + kind) then GB's 12 (kind d3P, d4P at 18 + 2 ccs + kind), padded to 32
// so that a component's values are read in pairs.
constexpr int kBK = 32;

// Force and normal of one point from its synthesised derivative sums (x_t, x_p,
// x_tt, x_tp, x_pp, then the four third and five fourth derivatives), the
// reference sphere at (st, ct, cp, sp) added to them.
template <class T>
__device__ __forceinline__ void bend_point(T (&acc)[14][3], T st, T ct, T cp, T sp, T R, const RefSphere<T>& S, T hf,
                                           T csk, int law, T eb, bool normals_only, T* f, T* nrm) {
  // x = R u, u = (st sp, st cp, ct)
  const T u[3] = {st * sp, st * cp, ct};
  const T ut[3] = {ct * sp, ct * cp, -st};
  const T up[3] = {st * cp, -st * sp, T(0)};
  const T utp[3] = {ct * cp, -ct * sp, T(0)};
  const T upp[3] = {-st * sp, -st * cp, T(0)};
  const T utpp[3] = {-ct * sp, -ct * cp, T(0)};
  // derivatives of u in the order of acc: u_t, u_p, u_tt = -u, u_tp, u_pp,
  // u_ttt = -u_t, u_ttp = -u_p, u_tpp, u_ppp = -u_p, u_tttt = u,
  // u_tttp = -u_tp, u_ttpp = -u_pp, u_tppp = -u_tp, u_pppp = -u_pp
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T sph[14] = {ut[c], up[c], -u[c], utp[c], upp[c], -ut[c], -up[c], utpp[c], -up[c],
                       u[c], -utp[c], -upp[c], -utp[c], -upp[c]};
#pragma unroll
    for (int q = 0; q < 14; ++q) acc[q][c] += R * sph[q];
  }
  f[0] = f[1] = f[2] = T(0);
  if (normals_only) {
    T cc[3];
    cross3(acc[0], acc[1], cc);
    const T sm = sqrt(dot3(cc, cc));
    for (int c = 0; c < 3; ++c) nrm[c] = fdiv(cc[c], sm);
  } else {
    membrane_force<T>(acc[0], acc[1], acc[2], acc[3], acc[4], S, hf, csk, law, nrm, f);
    if (eb != T(0)) bending_force<T>(acc[0], acc[1], acc[2], acc[3], acc[4], acc + 5, acc + 9, S, eb, f);
  }
}

// FP64, one point per thread.
__global__ void __launch_bounds__(256, 1) membrane_bend_kernel(const RowWork* __restrict__ work, int nwork,
                                                            const CapInfo* __restrict__ caps,
                                                            const GroupDev* __restrict__ groups,
                                                            const int* __restrict__ sur_flag) {
  using T = double;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x;
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const RowWork it = work[w];
    const CapInfo ci = caps[it.cap];
    const T hf = (T)(0.5 * ci.gs), csk = (T)ci.csk, eb = (T)ci.eb;
    const bool normals_only = sur_flag && sur_flag[it.cap];
    const GroupDev gd = groups[it.group];
    const int N = gd.N, nD = gd.nD, mD = gd.mD, H = mD >> 1, HP = dft_hp<T>(H), TS = dft_ts<T>(H);
    const int RP = (int)blockDim.x / mD > 0 ? (int)blockDim.x / mD : 1;  // rows per chunk, one point per thread
    const int SR = N * kBK + 16 / (int)sizeof(T);
    T* sG = (T*)smem_raw;               // [RP][SR]
    T* sTrig = sG + RP * SR;            // [2N][TS]: cos m phi_j (rows m), sin (rows N + m), j < H
    T* sOut = sTrig + 2 * N * TS;       // [RP][6][2 HP]: points j < H, then half a turn on; then their sums and differences
    int* sOff = (int*)(sOut + RP * 12 * HP);  // [30N]: staged offsets of G's then GB's elements
    const T* Gs = (const T*)gd.buf.G + (long long)ci.gidx * (18 * N * nD);   // [ccs][m][kind][lat]
    const T* Gb = (const T*)gd.buf.GB + (long long)ci.gidx * (12 * N * nD);  // [ccs][m][kind][lat]
    const T* trig = (const T*)gd.trigD[0];
    const T* lat = (const T*)gd.latD[0];
    T* Fout = (T*)gd.buf.Fout + (long long)ci.gidx * 12 * N * nD;
    const T R = (T)ci.R;
    __syncthreads();  // the previous item's reads of shared memory are done
    stage_dft<T>(sTrig, trig, mD, N, H, sOut, RP * 12);
    for (int e = tid; e < 18 * N; e += blockDim.x) {  // e = (ccs N + m) 3 + kind
      const int kind = e % 3, cm_ = e / 3, m = cm_ % N, ccs = cm_ / N;
      sOff[e] = m * kBK + 3 * ccs + kind;
    }
    for (int e = tid; e < 12 * N; e += blockDim.x) {  // e = (ccs N + m) 2 + kind
      const int kind = e & 1, cm_ = e >> 1, m = cm_ % N, ccs = cm_ / N;
      sOff[18 * N + e] = m * kBK + 18 + 2 * ccs + kind;
    }
    const int sr = tid % RP, se0 = tid / RP, ses = (int)blockDim.x / RP;
    const bool son = tid < ses * RP;
    for (int rb = it.row0; rb < it.row0 + it.nrows; rb += RP) {
      const int rows = min(RP, it.row0 + it.nrows - rb);
      __syncthreads();  // the previous chunk's staged rows and outputs are consumed
      if (son && sr < rows) {
        for (int e = se0; e < 18 * N; e += ses) stage_async(&sG[sr * SR + sOff[e]], &Gs[(long long)e * nD + rb + sr]);
        for (int e = se0; e < 12 * N; e += ses)
          stage_async(&sG[sr * SR + sOff[18 * N + e]], &Gb[(long long)e * nD + rb + sr]);
      }
      stage_wait();
      __syncthreads();
      {
        const int r = tid / mD, j = tid - (tid / mD) * mD;
        if (r < rows) {
          const int i = rb + r;
          // a1, a2, d11, d12, d22, S1..S4, Q1..Q5 per component
          T acc[14][3];
#pragma unroll
          for (int q = 0; q < 14; ++q) acc[q][0] = acc[q][1] = acc[q][2] = T(0);
          const T* g = sG + r * SR;
          // half a turn on, cos and sin of an odd m change sign
          const int jh = j < H ? j : j - H;
          const T turn = j < H ? T(1) : T(-1);
          for (int m = 0; m < N; ++m) {
            const T sg = m & 1 ? turn : T(1);
            const T cm = sg * sTrig[m * TS + jh], sm = sg * sTrig[(N + m) * TS + jh], fm = (T)m, fm2 = fm * fm;
            const T* gm = g + m * kBK;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              T ga[5], gb[5];  // P^(k) series of the cos and sin rows, k = 0..4
              const double2 *lo = (const double2*)(gm + 6 * c), *hi = (const double2*)(gm + 18 + 4 * c);
              const double2 x0 = lo[0], x1 = lo[1], x2 = lo[2], x3 = hi[0], x4 = hi[1];
              ga[0] = x0.x, ga[1] = x0.y, ga[2] = x1.x, ga[3] = x3.x, ga[4] = x3.y;
              gb[0] = x1.y, gb[1] = x2.x, gb[2] = x2.y, gb[3] = x4.x, gb[4] = x4.y;
              T t0[5], t1[5];  // parthe0 and parthe1 forms of the P^(k) series
#pragma unroll
              for (int k = 0; k < 5; ++k) {
                t0[k] = ga[k] * cm - gb[k] * sm;
                t1[k] = fm * (ga[k] * (-sm) - gb[k] * cm);
              }
              acc[0][c] += t0[1];               // x_t
              acc[1][c] += t1[0];               // x_p
              acc[2][c] += t0[2];               // x_tt
              acc[3][c] += t1[1];               // x_tp
              acc[4][c] += -fm2 * t0[0];        // x_pp
              acc[5][c] += t0[3];               // x_ttt
              acc[6][c] += t1[2];               // x_ttp
              acc[7][c] += -fm2 * t0[1];        // x_tpp
              acc[8][c] += -fm2 * t1[0];        // x_ppp (m^3 (a sin + b cos))
              acc[9][c] += t0[4];               // x_tttt
              acc[10][c] += t1[3];              // x_tttp
              acc[11][c] += -fm2 * t0[2];       // x_ttpp
              acc[12][c] += -fm2 * t1[1];       // x_tppp
              acc[13][c] += fm2 * fm2 * t0[0];  // x_pppp
            }
          }
          const T st = lat[4 * i], ct = lat[4 * i + 1];
          const T cp = turn * sTrig[1 * TS + jh], sp = turn * sTrig[(N + 1) * TS + jh];
          T f[3], nrm[3];
          bend_point<T>(acc, st, ct, cp, sp, R, RefSphere<T>(R, st, ct), hf, csk, ci.law, eb, normals_only, f, nrm);
          T* o = sOut + r * 12 * HP + (j < H ? 0 : HP) + jh;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            o[2 * c * HP] = f[c];
            o[2 * (3 + c) * HP] = nrm[c];
          }
        }
      }
      __syncthreads();
      // points half a turn apart to their sum and difference, then the forward
      // DFT (shagc.f:364-380) of the six outputs per row; the staged rows are
      // consumed, their memory takes the results
      for (int q = tid; q < rows * 6 * H; q += blockDim.x) {
        const int line = q / H, j = q - line * H;
        T* o = sOut + line * 2 * HP + j;
        const T a = o[0], b = o[HP];
        o[0] = a + b;
        o[HP] = a - b;
      }
      __syncthreads();
      dft_chunk<T, 6, 3, false>(sOut, sTrig, N, H, rows, RP, sG, Fout + rb, nD);
    }
  }
}

// its shared memory (bytes) for degrees up to nmax
size_t bend_smem(int nmax) {
  using T = double;
  size_t e = 0;
  for (size_t n = 1; n <= (size_t)nmax; ++n) {
    const size_t RP = 256 / (4 * n) > 0 ? 256 / (4 * n) : 1;
    e = std::max(e, RP * (n * kBK + 16 / sizeof(T)) + 2 * n * dft_ts<T>(2 * (int)n) + RP * 12 * dft_hp<T>(2 * (int)n) +
                        (30 * n * sizeof(int) + sizeof(T) - 1) / sizeof(T) + 8);
  }
  return sizeof(T) * e;
}

// The FP32 kernel: two points half a turn apart per thread, as in
// membrane_kernel_f2.  The synthesis sums the even and the odd m of every
// series as a packed pair (f32x2), the points j and j + mD/2 are their sum and
// difference: one load and one packed operation serve two m and two points.
// The second point's 42 sums wait in shared memory while the first is
// evaluated, so that 128 registers suffice.  Staged values [m pair][k][m
// parity], k as above, padded to 64 floats; trig (cos m, cos m+1, sin m,
// sin m+1) per point.  68 us at 524,288 points (64 in the bending force's form
// without the frame, 96 in that form with a point per thread).
constexpr int kBP = 64;

__global__ void __launch_bounds__(256, 2) membrane_bend_kernel_f2(const RowWork* __restrict__ work, int nwork,
                                                                  const CapInfo* __restrict__ caps,
                                                                  const GroupDev* __restrict__ groups,
                                                                  const int* __restrict__ sur_flag) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x;
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const RowWork it = work[w];
    const CapInfo ci = caps[it.cap];
    const float hf = (float)(0.5 * ci.gs), csk = (float)ci.csk, eb = (float)ci.eb;
    const bool normals_only = sur_flag && sur_flag[it.cap];
    const GroupDev gd = groups[it.group];
    const int N = gd.N, nD = gd.nD, mD = gd.mD, H = mD >> 1, NP = (N + 1) >> 1;
    const int HP = dft_hp<float>(H), TS = dft_ts<float>(H);
    const int RP = (int)blockDim.x / H > 0 ? (int)blockDim.x / H : 1;
    const int SR = NP * kBP + 4;
    float* sG = (float*)smem_raw;            // [RP][SR], then the DFT's results
    float4* sTP = (float4*)(sG + RP * SR);   // [NP][H]
    float* sTrig = (float*)(sTP + NP * H);   // [2N][TS]
    float* sOut = sTrig + 2 * N * TS;        // [RP][6][2 HP]
    float* sB = sOut + RP * 12 * HP;         // [42][256]: the second points' sums
    int* sOff = (int*)(sB + 42 * 256);       // [30N]
    const float* Gs = (const float*)gd.buf.G + (long long)ci.gidx * (18 * N * nD);
    const float* Gb = (const float*)gd.buf.GB + (long long)ci.gidx * (12 * N * nD);
    const float* trig = (const float*)gd.trigD[1];
    const float* lat = (const float*)gd.latD[1];
    float* Fout = (float*)gd.buf.Fout + (long long)ci.gidx * 12 * N * nD;
    const float R = (float)ci.R;
    __syncthreads();  // the previous item's reads of shared memory are done
    {
      const StageMap tm = stage_map(H);
      if (tm.on)
        for (int mp = tm.e0; mp < NP; mp += tm.es) {
          const int j = tm.r, m = 2 * mp;
          const bool odd = m + 1 < N;
          sTP[mp * H + j] = make_float4(trig[m * mD + j], odd ? trig[(m + 1) * mD + j] : 0.0f, trig[(N + m) * mD + j],
                                        odd ? trig[(N + m + 1) * mD + j] : 0.0f);
        }
    }
    stage_dft<float>(sTrig, trig, mD, N, H, sOut, RP * 12);
    for (int e = tid; e < 18 * N; e += blockDim.x) {  // e = (ccs N + m) 3 + kind
      const int kind = e % 3, cm_ = e / 3, m = cm_ % N, ccs = cm_ / N;
      sOff[e] = (m >> 1) * kBP + 2 * (3 * ccs + kind) + (m & 1);
    }
    for (int e = tid; e < 12 * N; e += blockDim.x) {  // e = (ccs N + m) 2 + kind
      const int kind = e & 1, cm_ = e >> 1, m = cm_ % N, ccs = cm_ / N;
      sOff[18 * N + e] = (m >> 1) * kBP + 2 * (18 + 2 * ccs + kind) + (m & 1);
    }
    const StageMap sm = stage_map(RP);
    for (int rb = it.row0; rb < it.row0 + it.nrows; rb += RP) {
      const int rows = min(RP, it.row0 + it.nrows - rb);
      __syncthreads();  // the previous chunk's staged rows and outputs are consumed
      if (sm.on && sm.r < rows) {
        for (int e = sm.e0; e < 18 * N; e += sm.es)
          stage_async(&sG[sm.r * SR + sOff[e]], &Gs[(long long)e * nD + rb + sm.r]);
        for (int e = sm.e0; e < 12 * N; e += sm.es)
          stage_async(&sG[sm.r * SR + sOff[18 * N + e]], &Gb[(long long)e * nD + rb + sm.r]);
      }
      if (N & 1)  // the last pair's odd m
        for (int q = tid; q < 30 * rows; q += blockDim.x) {
          const int r = q / 30, k = q - r * 30;
          sG[r * SR + (N >> 1) * kBP + 2 * k + 1] = 0.0f;
        }
      stage_wait();
      __syncthreads();
      const int r = tid / H, j = tid - (tid / H) * H;
      if (r < rows) {
        const int i = rb + r;
        float2 acc[14][3];
#pragma unroll
        for (int q = 0; q < 14; ++q) acc[q][0] = acc[q][1] = acc[q][2] = make_float2(0.0f, 0.0f);
        const float* g = sG + r * SR;
        for (int mp = 0; mp < NP; ++mp) {
          const float4 t = sTP[mp * H + j];
          const float m0 = (float)(2 * mp), m1 = m0 + 1.0f;
          const float2 cm = make_float2(t.x, t.y), sn = make_float2(t.z, t.w), nsn = make_float2(-t.z, -t.w);
          const float2 nfm = make_float2(-m0, -m1), nf2 = make_float2(-m0 * m0, -m1 * m1);
          const float2 f4 = __fmul2_rn(nf2, nf2);
          const float4* gq = (const float4*)(g + mp * kBP);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float4 x0 = gq[3 * c], x1 = gq[3 * c + 1], x2 = gq[3 * c + 2], x3 = gq[9 + 2 * c], x4 = gq[10 + 2 * c];
            // P^(k) series of the cos and sin rows, k = 0..4
            const float2 ga[5] = {make_float2(x0.x, x0.y), make_float2(x0.z, x0.w), make_float2(x1.x, x1.y),
                                  make_float2(x3.x, x3.y), make_float2(x3.z, x3.w)};
            const float2 gb[5] = {make_float2(x1.z, x1.w), make_float2(x2.x, x2.y), make_float2(x2.z, x2.w),
                                  make_float2(x4.x, x4.y), make_float2(x4.z, x4.w)};
            float2 t0[5], t1[4];  // parthe0 and parthe1 forms
#pragma unroll
            for (int k = 0; k < 5; ++k) t0[k] = __ffma2_rn(ga[k], cm, __fmul2_rn(gb[k], nsn));
#pragma unroll
            for (int k = 0; k < 4; ++k) t1[k] = __fmul2_rn(nfm, __ffma2_rn(ga[k], sn, __fmul2_rn(gb[k], cm)));
            acc[0][c] = __fadd2_rn(acc[0][c], t0[1]);            // x_t
            acc[1][c] = __fadd2_rn(acc[1][c], t1[0]);            // x_p
            acc[2][c] = __fadd2_rn(acc[2][c], t0[2]);            // x_tt
            acc[3][c] = __fadd2_rn(acc[3][c], t1[1]);            // x_tp
            acc[4][c] = __ffma2_rn(nf2, t0[0], acc[4][c]);       // x_pp
            acc[5][c] = __fadd2_rn(acc[5][c], t0[3]);            // x_ttt
            acc[6][c] = __fadd2_rn(acc[6][c], t1[2]);            // x_ttp
            acc[7][c] = __ffma2_rn(nf2, t0[1], acc[7][c]);       // x_tpp
            acc[8][c] = __ffma2_rn(nf2, t1[0], acc[8][c]);       // x_ppp
            acc[9][c] = __fadd2_rn(acc[9][c], t0[4]);            // x_tttt
            acc[10][c] = __fadd2_rn(acc[10][c], t1[3]);          // x_tttp
            acc[11][c] = __ffma2_rn(nf2, t0[2], acc[11][c]);     // x_ttpp
            acc[12][c] = __ffma2_rn(nf2, t1[1], acc[12][c]);     // x_tppp
            acc[13][c] = __ffma2_rn(f4, t0[0], acc[13][c]);      // x_pppp
          }
        }
        float x[14][3];
#pragma unroll
        for (int q = 0; q < 14; ++q)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            x[q][c] = acc[q][c].x + acc[q][c].y;
            sB[(3 * q + c) * 256 + tid] = acc[q][c].x - acc[q][c].y;
          }
        const float st = lat[4 * i], ct = lat[4 * i + 1];
        const RefSphere<float> S(R, st, ct);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {  // h = 1: half a turn on (cos p, sin p change sign)
          if (h)
#pragma unroll
            for (int q = 0; q < 14; ++q)
#pragma unroll
              for (int c = 0; c < 3; ++c) x[q][c] = sB[(3 * q + c) * 256 + tid];
          const float sg = h ? -1.0f : 1.0f, cp = sg * sTrig[TS + j], sp = sg * sTrig[(N + 1) * TS + j];
          float fo[3], no[3];
          bend_point<float>(x, st, ct, cp, sp, R, S, hf, csk, ci.law, eb, normals_only, fo, no);
          float* o = sOut + r * 12 * HP + h * HP + j;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            o[2 * c * HP] = fo[c];
            o[2 * (3 + c) * HP] = no[c];
          }
        }
        // the thread's own two points to their sum and difference
        float* o = sOut + r * 12 * HP + j;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const float a = o[2 * q * HP], b = o[(2 * q + 1) * HP];
          o[2 * q * HP] = a + b;
          o[(2 * q + 1) * HP] = a - b;
        }
      }
      __syncthreads();
      dft_chunk<float, 6, 3, true>(sOut, sTrig, N, H, rows, RP, sG, Fout + rb, nD);
    }
  }
}

// Shared memory of membrane_bend_kernel_f2 (bytes) for degrees up to nmax
size_t bend_f2_smem(int nmax) {
  size_t e = 0;
  for (size_t n = 1; n <= (size_t)nmax; ++n) {
    const size_t H = 2 * n, NP = (n + 1) / 2, RP = 256 / H > 0 ? 256 / H : 1;
    e = std::max(e, RP * (NP * kBP + 4) + NP * H * 4 + 2 * n * dft_ts<float>((int)H) + RP * 12 * dft_hp<float>((int)H) +
                        42 * 256 + 30 * n + 8);
  }
  return sizeof(float) * e;
}

}  // namespace

template <class K>
static cudaError_t launch_bend(K kernel, size_t smem, const RowWork* work, int nwork, const CapInfo* caps,
                               const GroupDev* groups, const int* sur_flag, cudaStream_t st) {
  cudaError_t err = smem_limit(kernel, smem);
  if (err != cudaSuccess) return err;
  int dev = 0, sms = 148, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 256, smem) != cudaSuccess || per < 1) per = 1;
  const int grid = std::min(nwork, sms * per);
  launch_pdl(kernel, dim3(grid), dim3(256), smem, st, work, nwork, caps, groups, sur_flag);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_membrane_bend(const RowWork* work, int nwork, const CapInfo* caps, const GroupDev* groups,
                                 const int* sur_flag, int nmax, cudaStream_t st) {
  if (nwork <= 0) return cudaSuccess;
  if constexpr (sizeof(T) == 4)
    return launch_bend(membrane_bend_kernel_f2, bend_f2_smem(nmax), work, nwork, caps, groups, sur_flag, st);
  else
    return launch_bend(membrane_bend_kernel, bend_smem(nmax), work, nwork, caps, groups, sur_flag, st);
}

template cudaError_t launch_membrane_bend<double>(const RowWork*, int, const CapInfo*, const GroupDev*, const int*, int,
                                                  cudaStream_t);
template cudaError_t launch_membrane_bend<float>(const RowWork*, int, const CapInfo*, const GroupDev*, const int*, int,
                                                 cudaStream_t);

}  // namespace sg
