// sg_longitude.cuh -- staging and the forward longitude DFTs of the pointwise
// kernels (sg_spectral.cu, sg_bending.cu).
#pragma once
#include "sg_common.cuh"

namespace sg {

// Thread mapping of the staging loops: thread t takes row r = t % RP of every
// (t / RP + k blockDim / RP)-th staged element, so that no loop iteration
// divides by a runtime value; the threads past the last whole group of RP
// stay idle.  Element offsets come from per-item tables in shared memory.
struct StageMap {
  int r, e0, es;
  bool on;
};
__device__ __forceinline__ StageMap stage_map(int RP) {
  StageMap m;
  m.es = (int)blockDim.x / RP;
  m.r = (int)threadIdx.x % RP;
  m.e0 = (int)threadIdx.x / RP;
  m.on = (int)threadIdx.x < m.es * RP;
  return m;
}

// The trig table rows hm < nrow, columns j < H, of a [nrow][ld] global table
// into [nrow][ts] shared rows.
template <class T>
__device__ __forceinline__ void stage_trig(T* dst, int ts, const T* src, int ld, int nrow, int H) {
  const StageMap sm = stage_map(H);
  if (sm.on)
    for (int hm = sm.e0; hm < nrow; hm += sm.es) dst[hm * ts + sm.r] = src[hm * ld + sm.r];
}

// The forward longitude DFTs of the pointwise kernels.  A row's values lie
// as half-turn sums at [j] and differences at [HP + j] per field, the trig
// rows p < 2N (cos m = p, then sin m = p - N) at stride TS; lane p sums its
// trig row against the sums (even m) or the differences (odd m), 16 bytes of
// each at a time: HP = H rounded up to whole vectors, zeros after H, and TS an
// odd number of vectors, so that eight lanes' trig loads meet all banks.  The
// data are broadcasts; with PAIR (FP32) the even and the odd j are two partial
// sums in a packed pair, otherwise the sum runs over j in order.  The
// results go through shared memory ([f 2N + p][row], an odd number of rows
// apart) and out as runs of the chunk's rows: lanes that stored their own
// result filled 4 bytes of 32 sectors at a time.  Together: membrane 35 -> 33,
// posfwd 16 -> 14, shgrid 16 -> 15 us at 524,288 points in FP32, 194 -> 174,
// 68 -> 64, 66 -> 54 us at 1.6 million; FP64 membrane 65 -> 57 us.
template <class T>
__host__ __device__ constexpr int dft_vec() {
  return 16 / (int)sizeof(T);
}
template <class T>
__host__ __device__ constexpr int dft_hp(int H) {
  return (H + dft_vec<T>() - 1) / dft_vec<T>() * dft_vec<T>();
}
template <class T>
__host__ __device__ constexpr int dft_ts(int H) {
  return (dft_hp<T>(H) / dft_vec<T>() & 1) ? dft_hp<T>(H) : dft_hp<T>(H) + dft_vec<T>();
}
__host__ __device__ constexpr int dft_rows(int RP) { return RP | 1; }

// F fields at o, o + os, ...; t: the lane's trig row
template <class T, int F, bool PAIR>
__device__ __forceinline__ void dft_lane(const T* o, int os, const T* t, int HP, T (&a)[F]) {
  if constexpr (PAIR) {
    float2 s[F];
#pragma unroll
    for (int f = 0; f < F; ++f) s[f] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int j = 0; j < HP; j += 4) {
      const float4 w = *(const float4*)(t + j);
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const float4 x = *(const float4*)(o + f * os + j);
        s[f] = __ffma2_rn(make_float2(x.x, x.y), make_float2(w.x, w.y), s[f]);
        s[f] = __ffma2_rn(make_float2(x.z, x.w), make_float2(w.z, w.w), s[f]);
      }
    }
#pragma unroll
    for (int f = 0; f < F; ++f) a[f] = s[f].x + s[f].y;
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int f = 0; f < F; ++f) a[f] = T(0);
#pragma unroll 2
    for (int j = 0; j < HP; j += 4) {
      const float4 w = *(const float4*)(t + j);
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const float4 x = *(const float4*)(o + f * os + j);
        a[f] = fma(x.w, w.w, fma(x.z, w.z, fma(x.y, w.y, fma(x.x, w.x, a[f]))));
      }
    }
  } else {
#pragma unroll
    for (int f = 0; f < F; ++f) a[f] = T(0);
#pragma unroll 2
    for (int j = 0; j < HP; j += 2) {
      const double2 w = *(const double2*)(t + j);
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const double2 x = *(const double2*)(o + f * os + j);
        a[f] = fma(x.x, w.x, a[f]);
        a[f] = fma(x.y, w.y, a[f]);
      }
    }
  }
}

// The whole chunk: `rows` rows of NF fields in groups of F, lines of 2 HP
// values at sOut + (row NF + field) 2 HP; results through sRes to
// out[(field 2N + p) ld + row].
template <class T, int NF, int F, bool PAIR>
__device__ __forceinline__ void dft_chunk(const T* sOut, const T* sTrig, int N, int H, int rows, int RP, T* sRes,
                                          T* out, int ld) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int HP = dft_hp<T>(H), TS = dft_ts<T>(H), RS = dft_rows(RP);
  const T sf = T(1) / T(H);  // 2 / nlon, H = nlon / 2
  for (int line = warp; line < rows * (NF / F); line += nwarp) {
    const int rr = line / (NF / F), f0 = F * (line - rr * (NF / F));
    const T* o = sOut + (rr * NF + f0) * 2 * HP;
    for (int p = lane; p < 2 * N; p += 32) {
      const int m = p < N ? p : p - N;
      T a[F];
      dft_lane<T, F, PAIR>(o + ((m & 1) ? HP : 0), 2 * HP, sTrig + p * TS, HP, a);
#pragma unroll
      for (int f = 0; f < F; ++f) sRes[((f0 + f) * 2 * N + p) * RS + rr] = (p < N ? sf : -sf) * a[f];
    }
  }
  __syncthreads();
  const StageMap m = stage_map(RP);
  if (m.on && m.r < rows)
    for (int e = m.e0; e < NF * 2 * N; e += m.es) out[(long long)e * ld + m.r] = sRes[e * RS + m.r];
}

// Trig rows at the DFT's stride with zeros after H, and the zeros after H of
// the chunk's lines (2 per row and field).
template <class T>
__device__ __forceinline__ void stage_dft(T* sTrig, const T* trig, int ld, int N, int H, T* sOut, int lines) {
  const int HP = dft_hp<T>(H), TS = dft_ts<T>(H);
  stage_trig<T>(sTrig, TS, trig, ld, 2 * N, H);
  if (HP > H)
    for (int q = threadIdx.x; q < (HP - H) * (2 * N + lines); q += blockDim.x) {
      const int r = q / (HP - H), j = H + q - r * (HP - H);
      if (r < 2 * N)
        sTrig[r * TS + j] = T(0);
      else
        sOut[(r - 2 * N) * HP + j] = T(0);
    }
}

}  // namespace sg
