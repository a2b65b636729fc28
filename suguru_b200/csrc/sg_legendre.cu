// sg_legendre.cu -- batched Legendre contractions (the theta half of the
// SPHEREPACK Gauss-grid analysis shagc.f:384-470 and synthesis shsgc.f:329-470)
// on CUDA cores, for the FP64 plain path and as the FP32 fallback.
//
// Each LegWork item is one (problem, m, tile of 32 data rows), with the
// problems chained to it: D[q][j] = sum_k A[q][k] B_m[j][k], and for each
// chained problem the same with D as its A.  The tables of the whole chain
// and the tile's A rows are copied to shared memory by asynchronous copies,
// all issued before any is waited for, the tables before the predecessor
// kernel has finished (they do not depend on it).  A warp forms four rows,
// lane = j, two k at a time: one 16-byte load of the table serves four rows,
// the rows' values are broadcasts.  Rows are an even number of elements apart
// whose half is odd (leg_ld), so that the lanes' table loads meet different
// banks.  The sums run over k in order, from k = m in a synthesis, whose
// coefficients vanish for n < m.
//
// What bounds it: latency and the intermediates' traffic in L2 (about 100 MB
// per step at 256 capsules of degree 15); the sums themselves are 6 us of FP64.
// Copying row after row through registers, one row per load, with a launch
// per stage, took 146 us a step there in six launches; chained in three
// launches, 64 us.
#include "sg_common.cuh"
#include "sg_kernels.h"

namespace sg {

constexpr int LEG_QT = 32;
constexpr int kLegRows = 4;  // rows per warp: 8 warps x 4 = LEG_QT

template <class T>
struct Pair;
template <>
struct Pair<double> {
  using type = double2;
};
template <>
struct Pair<float> {
  using type = float2;
};

__host__ __device__ constexpr int leg_ld(int K) {
  const int e = (K + 1) & ~1;
  return (e >> 1) & 1 ? e : e + 2;
}

// nr rows of K elements into shared rows of leg_ld(K), a zero after an odd
// row; src(r) is row r's first element.  16 or 32 lanes per row.
template <class T, class Src>
__device__ __forceinline__ void stage_rows(T* dst, int nr, int K, const Src& src) {
  const int ld = leg_ld(K), w = K <= 16 ? 16 : 32;
  const int r0 = (int)threadIdx.x / w, k0 = (int)threadIdx.x % w, step = (int)blockDim.x / w;
  for (int r = r0; r < nr; r += step) {
    const T* s = src(r);
    for (int k = k0; k < K; k += w) stage_async(&dst[r * ld + k], &s[k]);
    if ((K & 1) && k0 == 0) dst[r * ld + K] = T(0);
  }
}

// One problem on the tile: rows sA (leg_ld(K)), table sB; results to D (row
// offsets off, -1 past the last row) and, when sD is given, to its rows.
template <class T>
__device__ __forceinline__ void contract_tile(const T* sA, const T* sB, int K, int J, int k0, T* D,
                                              const long long* off, T* sD) {
  using T2 = typename Pair<T>::type;
  const int ld = leg_ld(K), ldd = leg_ld(J), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool narrow = J <= 16;  // two halves of the warp take two rows each
  const int q0 = warp * kLegRows + (narrow ? (lane >> 4) * 2 : 0), nr = narrow ? 2 : 4;
  const T* a = sA + q0 * ld;
  for (int jb = 0; jb < J; jb += 32) {
    const int j = jb + (narrow ? lane & 15 : lane);
    const T* b = sB + min(j, J - 1) * ld;
    T acc[kLegRows] = {T(0), T(0), T(0), T(0)};
    int k = k0;
    if (k & 1) {
#pragma unroll
      for (int i = 0; i < kLegRows; ++i)
        if (i < nr) acc[i] += a[i * ld + k] * b[k];
      ++k;
    }
    if (narrow) {
#pragma unroll 2
      for (; k < K; k += 2) {
        const T2 bk = *(const T2*)(b + k);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const T2 ak = *(const T2*)(a + i * ld + k);
          acc[i] += ak.x * bk.x;
          acc[i] += ak.y * bk.y;
        }
      }
    } else {
#pragma unroll 2
      for (; k < K; k += 2) {
        const T2 bk = *(const T2*)(b + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const T2 ak = *(const T2*)(a + i * ld + k);
          acc[i] += ak.x * bk.x;
          acc[i] += ak.y * bk.y;
        }
      }
    }
    if (j < J)
#pragma unroll
      for (int i = 0; i < kLegRows; ++i)
        if (i < nr) {
          const long long o = off[q0 + i];
          if (o >= 0) D[o + j] = acc[i];
          if (sD) {
            sD[(q0 + i) * ldd + j] = acc[i];
            if ((J & 1) && j == J - 1) sD[(q0 + i) * ldd + J] = T(0);
          }
        }
  }
}

template <class T>
__global__ void __launch_bounds__(256) legendre_kernel(const LegProblem* __restrict__ probs,
                                                       const LegWork* __restrict__ work, int nwork) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long s_off[4][LEG_QT];  // row offsets: the root's A, the three D's
  if ((int)blockIdx.x >= nwork) return;
  const LegWork wk = work[blockIdx.x];
  const int m = wk.m, q0 = wk.q0;
  const int lvl[3] = {wk.prob, wk.lvl1, wk.lvl1 >= 0 ? wk.lvl2 : -1};
  const LegProblem& R = probs[wk.prob];
  const int K = R.K, J = R.J;
  const int nq = min(LEG_QT, R.Q - q0);
  T* sA = (T*)smem_raw;                // [QT][ld(K)]
  T* sD = sA + LEG_QT * leg_ld(K);     // [QT][ld(J)] when chained
  T* sB[3];
  sB[0] = sD + (lvl[1] >= 0 ? LEG_QT * leg_ld(J) : 0);
  sB[1] = sB[0] + J * leg_ld(K);
  sB[2] = sB[1] + (lvl[1] >= 0 ? probs[lvl[1]].J * leg_ld(J) : 0);
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    if (lvl[l] < 0) continue;
    const LegProblem& P = probs[lvl[l]];
    const T* B = (const T*)P.B + (long long)m * P.sBm;
    const int Kl = P.K;
    stage_rows(sB[l], P.J, Kl, [&](int j) { return B + (long long)j * Kl; });
  }
  if (threadIdx.x < 4 * LEG_QT) {
    const int l = (int)threadIdx.x / LEG_QT - 1, q = (int)threadIdx.x % LEG_QT;
    if (l < 0 || lvl[l] >= 0) {
      const LegProblem& P = probs[l < 0 ? wk.prob : lvl[l]];
      long long o = -1;
      if (q < nq) {
        const int qq = q0 + q, c = qq / P.rpc, r = qq - c * P.rpc;
        o = l < 0 ? (long long)c * P.sAc + (long long)r * P.sAr + (long long)m * P.sAm
                  : (long long)c * P.sDc + (long long)r * P.sDr + (long long)m * P.sDm;
      }
      s_off[l + 1][q] = o;
    }
  }
  __syncthreads();
  pdl_enter();  // the data rows come from the predecessor
  const T* A = (const T*)R.A;
  stage_rows(sA, nq, K, [&](int q) { return A + s_off[0][q]; });
  stage_wait();
  __syncthreads();
  contract_tile<T>(sA, sB[0], K, J, R.tri ? m : 0, (T*)R.D, s_off[1], lvl[1] >= 0 ? sD : nullptr);
  if (lvl[1] < 0) return;
  __syncthreads();
#pragma unroll
  for (int l = 1; l < 3; ++l) {
    if (lvl[l] < 0) continue;
    const LegProblem& P = probs[lvl[l]];
    contract_tile<T>(sD, sB[l], J, P.J, P.tri ? m : 0, (T*)P.D, s_off[l + 1], nullptr);
  }
}

// Shared-memory elements of a chain: J and K of its root, the chained
// problems' J (0: none; their K is the root's J).
size_t legendre_elems(int J, int K, int J1, int J2) {
  size_t n = (size_t)(LEG_QT + J) * leg_ld(K);
  if (J1 > 0) n += (size_t)(LEG_QT + J1 + J2) * leg_ld(J);
  return n;
}

template <class T>
cudaError_t launch_legendre(const LegProblem* d_probs, const LegWork* d_work, int nwork, size_t elems,
                            cudaStream_t st) {
  if (nwork <= 0) return cudaSuccess;
  const size_t smem = sizeof(T) * elems;
  // the chain's tables and rows must fit the device's opt-in limit (SH degree
  // 31 in FP64: 113 KB); refuse on the host rather than launch with a request
  // the device cannot grant
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  if (smem > (size_t)optin) return cudaErrorInvalidValue;
  e = smem_limit(legendre_kernel<T>, smem);
  if (e != cudaSuccess) return e;
  launch_pdl(legendre_kernel<T>, dim3(nwork), dim3(256), smem, st, d_probs, d_work, nwork);
  return cudaGetLastError();
}

template cudaError_t launch_legendre<double>(const LegProblem*, const LegWork*, int, size_t, cudaStream_t);
template cudaError_t launch_legendre<float>(const LegProblem*, const LegWork*, int, size_t, cudaStream_t);

}  // namespace sg
