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

template <class T>
struct VecPair {
  using type = float2;
};
template <>
struct VecPair<double> {
  using type = double2;
};

template <class T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1) membrane_bend_kernel(const RowWork* __restrict__ work, int nwork,
                                                            const CapInfo* __restrict__ caps,
                                                            const GroupDev* __restrict__ groups,
                                                            const int* __restrict__ sur_flag) {
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
    const T* trig = (const T*)gd.trigD[sizeof(T) == 8 ? 0 : 1];
    const T* lat = (const T*)gd.latD[sizeof(T) == 8 ? 0 : 1];
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
              using T2 = typename VecPair<T>::type;
              const T2 *lo = (const T2*)(gm + 6 * c), *hi = (const T2*)(gm + 18 + 4 * c);
              const T2 x0 = lo[0], x1 = lo[1], x2 = lo[2], x3 = hi[0], x4 = hi[1];
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
          // the reference sphere: x = R u, u = (st sp, st cp, ct)
          const T st = lat[4 * i], ct = lat[4 * i + 1];
          const T cp = turn * sTrig[1 * TS + jh], sp = turn * sTrig[(N + 1) * TS + jh];
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
          T f[3] = {T(0), T(0), T(0)}, nrm[3];
          if (normals_only) {
            T cc[3];
            cross3(acc[0], acc[1], cc);
            const T sm = sqrt(dot3(cc, cc));
            for (int c = 0; c < 3; ++c) nrm[c] = fdiv(cc[c], sm);
          } else {
            membrane_force<T>(acc[0], acc[1], acc[2], acc[3], acc[4], RefSphere<T>(R, st, ct), hf, csk, ci.law, nrm, f);
            if (eb != T(0)) bending_force<T>(acc[0], acc[1], acc[2], acc[3], acc[4], acc + 5, acc + 9, eb, f);
          }
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
      dft_chunk<T, 6, 3, sizeof(T) == 4>(sOut, sTrig, N, H, rows, RP, sG, Fout + rb, nD);
    }
  }
}

}  // namespace

template <class T>
cudaError_t launch_membrane_bend(const RowWork* work, int nwork, const CapInfo* caps, const GroupDev* groups,
                                 const int* sur_flag, int nmax, cudaStream_t st) {
  if (nwork <= 0) return cudaSuccess;
  size_t e = 0;  // shared memory (elements of T) over the degrees up to nmax
  for (size_t n = 1; n <= (size_t)nmax; ++n) {
    const size_t RP = 256 / (4 * n) > 0 ? 256 / (4 * n) : 1;
    const size_t en = RP * (n * kBK + 16 / sizeof(T)) + 2 * n * dft_ts<T>(2 * (int)n) + RP * 12 * dft_hp<T>(2 * (int)n) +
                      (30 * n * sizeof(int) + sizeof(T) - 1) / sizeof(T) + 8;
    e = std::max(e, en);
  }
  const size_t smem = sizeof(T) * e;
  cudaError_t err = smem_limit(membrane_bend_kernel<T>, smem);
  if (err != cudaSuccess) return err;
  int dev = 0, sms = 148, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, membrane_bend_kernel<T>, 256, smem) != cudaSuccess || per < 1)
    per = 1;
  const int grid = std::min(nwork, sms * per);
  launch_pdl(membrane_bend_kernel<T>, dim3(grid), dim3(256), smem, st, work, nwork, caps, groups, sur_flag);
  return cudaGetLastError();
}

template cudaError_t launch_membrane_bend<double>(const RowWork*, int, const CapInfo*, const GroupDev*, const int*, int,
                                                  cudaStream_t);
template cudaError_t launch_membrane_bend<float>(const RowWork*, int, const CapInfo*, const GroupDev*, const int*, int,
                                                 cudaStream_t);

}  // namespace sg
