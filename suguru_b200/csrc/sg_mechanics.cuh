// sg_mechanics.cuh -- membrane mechanics of one surface point (device code
// shared by the spectral force kernels): the membrane force of
// cal_spectral_force (sph.f90:1668-1715 with sph1.f90:581-651, the unit
// normal, and the laws of membmodel.c) and the bending force added by
// ibend = 1.
#pragma once
#include "sg_common.cuh"

namespace sg {

// Division in the pointwise geometry and mechanics: the FP32 path uses the
// fast reciprocal-based division (2 ulp), the FP64 path the IEEE division.
template <class T>
__device__ __forceinline__ T fdiv(T a, T b);
template <>
__device__ __forceinline__ float fdiv<float>(float a, float b) {
  return __fdividef(a, b);
}
template <>
__device__ __forceinline__ double fdiv<double>(double a, double b) {
  return a / b;
}

// The reference sphere of radius R at colatitude t (st = sin t, ct = cos t):
// contravariant metric A^11 = 1/R^2, A^22 = 1/(R st)^2 (A^12 = 0), the root of
// A^11 A^22, and cot t.
template <class T>
struct RefSphere {
  T A1, A2, rA, cot;
  __device__ __forceinline__ RefSphere(T R, T st, T ct) {
    const T is = fdiv(T(1), st), q = ct * is;
    cot = fma(fma(-q, st, ct), is, q);
    A1 = fdiv(T(1), R * R);
    A2 = A1 * (is * is);
    rA = A1 * is;
  }
};

// Unit normal and membrane force per area of one point (cal_spectral_force's
// equilibrium, sph.f90:1668-1715, with cal_Js_I1_I2_deri, sph.f90:1115-1156,
// the laws of membmodel.c and calculate_cauchy_tensor_deri, sph.f90:1179-1234).
// The reference forms the contravariant basis with its derivatives and the
// Christoffel symbols, takes the tension's covariant divergence and its
// contraction with the curvature, and sums q1 a1 + q2 a2 + q3 n.  With
// x_ab = G^c_ab a_c + b_ab n those sums are
//   f = (sq T^ab)_,a / sq a_b + T^ab x_ab,   sq = sqrt(det a_ab).
// With the stretches E1 = A^11 a_11, E2 = A^22 a_22, G = A^11 A^22 a_12 and
// J^2 = E1 E2 - G a_12 the tension is
//   T^11 = 2/J A^11 (W1 + W2 E2), T^22 = 2/J A^22 (W1 + W2 E1), T^12 = -2/J W2 G,
// and sq = J / sqrt(A^11 A^22), so J drops out of the divergence:
//   J/2 f = (A^11 (p1_,t + cot p1) - (W2 G)_,p) a1 + (A^22 p2_,p - (W2 G)_;t) a2
//           + A^11 p1 x_tt - 2 W2 G x_tp + A^22 p2 x_pp,
// p1 = W1 + W2 E2, p2 = W1 + W2 E1, the t derivatives of E2 and G taken with
// the sphere's own (of A^22, cot) removed: through y = x_tp - cot x_p, zero on
// the sphere.  For the Skalak law p1 = hf (E1 - 1 + C I2 E2): every quantity is
// of the size of the strain and the terms of the sphere's tension, which would
// cancel, do not appear.  A point's rounding error is 0.6 to 0.7 of the reference
// form's in FP32 and FP64; written with T^ab_,a + (q_,a / 2 q) T^ab it was 1.1 to
// 1.3 times that.  About 170 operations with one division and one root instead of
// 500 with a dozen divisions: the membrane kernel 41 -> 35 us in FP32 and 83 -> 65
// us in FP64 at 524,288 points.
// law 0: Skalak W1 = hf (1 + I1), W2 = hf (C I2 - 1) (membmodel.c:81-99);
// law 1: neo-Hookean W1 = hf, W2 = -hf (I2 + 1)^-2 (membmodel.c:60-79, the
// reference's -DNONHOOK build).
// Every sum is an explicit fused multiply-add, and a product that leaves the
// function is rounded, so that the staged and the fused force stage, which
// both inline this, give the same bits.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <class T>
__device__ __forceinline__ T dot3_fma(const T* u, const T* v) {
  return fma(u[2], v[2], fma(u[1], v[1], u[0] * v[0]));
}

template <class T>
__device__ __forceinline__ void membrane_force(const T* a1, const T* a2, const T* d11, const T* d12, const T* d22,
                                               const RefSphere<T>& S, T hf, T csk, int law, T* n, T* f) {
  const T cc[3] = {fma(a1[1], a2[2], -(a1[2] * a2[1])), fma(a1[2], a2[0], -(a1[0] * a2[2])),
                   fma(a1[0], a2[1], -(a1[1] * a2[0]))};
  const T y[3] = {fma(-S.cot, a2[0], d12[0]), fma(-S.cot, a2[1], d12[1]), fma(-S.cot, a2[2], d12[2])};
  const T g11 = dot3_fma(a1, a1), g22 = dot3_fma(a2, a2), g12 = dot3_fma(a1, a2), q = dot3_fma(cc, cc);
  const T AA = S.A1 * S.A2, J2 = AA * q, iJ2 = fdiv(T(1), J2), iJ = sqrt(J2) * iJ2;
  const T isq = iJ * S.rA;  // over the normal's length
  for (int c = 0; c < 3; ++c) n[c] = mul_rn(cc[c], isq);
  const T E1 = S.A1 * g11, E2 = S.A2 * g22, G = AA * g12;
  const T e1 = fma(S.A1, g11, -T(1)), e2 = fma(S.A2, g22, -T(1)), I2 = fma(AA, q, -T(1));
  // derivatives along t and p (index 0, 1), half of E1's and E2's
  const T E1d[2] = {S.A1 * dot3_fma(a1, d11), S.A1 * dot3_fma(a1, d12)};
  const T E2d[2] = {S.A2 * dot3_fma(a2, y), S.A2 * dot3_fma(a2, d22)};
  const T Gd[2] = {AA * (dot3_fma(a2, d11) + dot3_fma(a1, y)), AA * (dot3_fma(a1, d22) + dot3_fma(a2, d12))};
  const bool nh = law == 1;
  const T hc = hf * csk, iJ4 = iJ2 * iJ2;
  const T V = nh ? -(hf * iJ4) : hc * I2;  // W2, but for Skalak's -hf, which is in p1 and p2
  const T W2 = nh ? V : fma(hc, I2, -hf);
  T Vd[2];
#pragma unroll
  for (int al = 0; al < 2; ++al) {
    const T J2d = T(2) * fma(E1d[al], E2, fma(E1, E2d[al], -(g12 * Gd[al])));
    Vd[al] = nh ? (T(2) * hf * J2d) * (iJ4 * iJ2) : hc * J2d;
  }
  const T p1 = fma(V, E2, nh ? hf : hf * e1), p2 = fma(V, E1, nh ? hf : hf * e2);
  const T p1d = fma(Vd[0], E2, T(2) * fma(V, E2d[0], nh ? T(0) : hf * E1d[0]));
  const T p2d = fma(Vd[1], E1, T(2) * fma(V, E1d[1], nh ? T(0) : hf * E2d[1]));
  const T c0 = T(2) * iJ, k12 = -T(2) * (W2 * G), k11 = S.A1 * p1, k22 = S.A2 * p2;
  const T k1 = fma(S.A1, fma(S.cot, p1, p1d), -fma(Vd[1], G, W2 * Gd[1]));
  const T k2 = fma(S.A2, p2d, -fma(Vd[0], G, W2 * Gd[0]));
  for (int c = 0; c < 3; ++c)
    f[c] = mul_rn(c0, fma(k1, a1[c], fma(k2, a2[c], fma(k11, d11[c], fma(k12, d12[c], k22 * d22[c])))));
}

// The bending force of ibend = 1 (sph.f90:1705-1709), added to f.  The
// reference forms the moment M^ba = eb a^bg (A^ga B_gg' - a^ga b_gg') with its
// first and second derivatives (cal_moment_deri, sph.f90:1236-1372, from the
// twice differentiated curvature, contravariant metric and Christoffel
// symbols, sph.f90:479-1111, sph1.f90:299-542), its divergence Q^b = M^ab_|a
// and Q^b_|b (cal_Q, :1375-1424), and adds Q^b_|b n - Q^b b_b^a a_a
// (cal_bcurmix, :1427-1454).  On the sphere A^ga B_gg' is delta / R, so M^ba =
// eb (a^ba / R - b^ba); the metric is covariantly constant and by Codazzi's
// equations b^ab_|a = a^bg h_,g with h = a^ab b_ab, hence
//   Q^b = -eb a^bg h_,g  and  f += -eb Lap(h) n + eb a^bg h_,g b_b^a a_a.
// h = S / q^(3/2) with S = g22 L - 2 g12 M + g11 N, L, M, N = x_ab . m,
// m = a1 x a2 and q = m . m: its value and five derivatives follow from
// products, about 450 operations instead of 2,500 and no tensors to keep.
// S3 = x_ttt, x_ttp, x_tpp, x_ppp; S4 = x_tttt, x_tttp, x_ttpp, x_tppp, x_pppp.
template <class T>
struct Jet2 {  // a function of (t, p): value and derivatives t, p, tt, tp, pp
  T v, t, p, tt, tp, pp;
};
template <class T>
__device__ __forceinline__ Jet2<T> operator*(const Jet2<T>& a, const Jet2<T>& b) {
  return {a.v * b.v,
          a.t * b.v + a.v * b.t,
          a.p * b.v + a.v * b.p,
          a.tt * b.v + T(2) * (a.t * b.t) + a.v * b.tt,
          a.tp * b.v + a.t * b.p + a.p * b.t + a.v * b.tp,
          a.pp * b.v + T(2) * (a.p * b.p) + a.v * b.pp};
}

template <class T>
__device__ __forceinline__ void bending_force(const T* a1, const T* a2, const T* x11, const T* x12, const T* x22,
                                              const T (*S3)[3], const T (*S4)[3], T eb, T* f) {
  auto dot = [](const T* u, const T* v) { return dot3(u, v); };
  T m[3], mt[3], mp[3], mtt[3], mtp[3], mpp[3];
  {
    T u[3], v[3], w[3];
    cross3(a1, a2, m);
    cross3(x11, a2, u);
    cross3(a1, x12, v);
    for (int c = 0; c < 3; ++c) mt[c] = u[c] + v[c];
    cross3(x12, a2, u);
    cross3(a1, x22, v);
    for (int c = 0; c < 3; ++c) mp[c] = u[c] + v[c];
    cross3(S3[0], a2, u);
    cross3(x11, x12, v);
    cross3(a1, S3[1], w);
    for (int c = 0; c < 3; ++c) mtt[c] = u[c] + T(2) * v[c] + w[c];
    cross3(S3[1], a2, u);
    cross3(x11, x22, v);
    cross3(a1, S3[2], w);
    for (int c = 0; c < 3; ++c) mtp[c] = u[c] + v[c] + w[c];
    cross3(S3[2], a2, u);
    cross3(x12, x22, v);
    cross3(a1, S3[3], w);
    for (int c = 0; c < 3; ++c) mpp[c] = u[c] + T(2) * v[c] + w[c];
  }
  const T q = dot(m, m), iq = fdiv(T(1), q);
  const T lt = T(2) * dot(m, mt) * iq, lp = T(2) * dot(m, mp) * iq;  // q_,t / q, q_,p / q
  const T ltt = T(2) * (dot(mt, mt) + dot(m, mtt)) * iq, ltp = T(2) * (dot(mt, mp) + dot(m, mtp)) * iq,
          lpp = T(2) * (dot(mp, mp) + dot(m, mpp)) * iq;
  // x_ab . m with its derivatives, from x_ab and its derivatives
  auto proj = [&](const T* x, const T* xt, const T* xp, const T* xtt, const T* xtp, const T* xpp) {
    Jet2<T> j;
    j.v = dot(x, m);
    j.t = dot(xt, m) + dot(x, mt);
    j.p = dot(xp, m) + dot(x, mp);
    j.tt = dot(xtt, m) + T(2) * dot(xt, mt) + dot(x, mtt);
    j.tp = dot(xtp, m) + dot(xt, mp) + dot(xp, mt) + dot(x, mtp);
    j.pp = dot(xpp, m) + T(2) * dot(xp, mp) + dot(x, mpp);
    return j;
  };
  const T x1212 = dot(x12, x12);
  const T a1x111 = dot(a1, S3[0]), a1x112 = dot(a1, S3[1]), a1x122 = dot(a1, S3[2]), a1x222 = dot(a1, S3[3]);
  const T a2x111 = dot(a2, S3[0]), a2x112 = dot(a2, S3[1]), a2x122 = dot(a2, S3[2]), a2x222 = dot(a2, S3[3]);
  const T x1112 = dot(x11, x12), x1122 = dot(x11, x22), x1222 = dot(x12, x22);
  const T a1x11 = dot(a1, x11), a1x12 = dot(a1, x12), a1x22 = dot(a1, x22);
  const T a2x11 = dot(a2, x11), a2x12 = dot(a2, x12), a2x22 = dot(a2, x22);
  const Jet2<T> g11 = {dot(a1, a1), T(2) * a1x11, T(2) * a1x12, T(2) * (dot(x11, x11) + a1x111),
                       T(2) * (x1112 + a1x112), T(2) * (x1212 + a1x122)};
  const Jet2<T> g22 = {dot(a2, a2), T(2) * a2x12, T(2) * a2x22, T(2) * (x1212 + a2x112), T(2) * (x1222 + a2x122),
                       T(2) * (dot(x22, x22) + a2x222)};
  // -2 g12
  const Jet2<T> g12 = {-T(2) * dot(a1, a2),
                       -T(2) * (a2x11 + a1x12),
                       -T(2) * (a2x12 + a1x22),
                       -T(2) * (a2x111 + T(2) * x1112 + a1x112),
                       -T(2) * (a2x112 + x1122 + x1212 + a1x122),
                       -T(2) * (a2x122 + T(2) * x1222 + a1x222)};
  const Jet2<T> L = proj(x11, S3[0], S3[1], S4[0], S4[1], S4[2]);
  const Jet2<T> M = proj(x12, S3[1], S3[2], S4[1], S4[2], S4[3]);
  const Jet2<T> N = proj(x22, S3[2], S3[3], S4[2], S4[3], S4[4]);
  const Jet2<T> A = g22 * L, B = g12 * M, C = g11 * N;
  const T s = A.v + B.v + C.v, st = A.t + B.t + C.t, sp = A.p + B.p + C.p;
  const T stt = A.tt + B.tt + C.tt, stp = A.tp + B.tp + C.tp, spp = A.pp + B.pp + C.pp;
  // h = s r with r = q^(-3/2): r_,t / r = -3/2 lt, r_,tt / r = 15/4 lt^2 - 3/2 ltt
  const T isq = sqrt(iq), r = iq * isq;
  const T ht = r * (st - T(1.5) * s * lt), hp = r * (sp - T(1.5) * s * lp);
  const T htt = r * (stt - T(3) * st * lt + s * (T(3.75) * lt * lt - T(1.5) * ltt));
  const T htp = r * (stp - T(1.5) * (st * lp + sp * lt) + s * (T(3.75) * lt * lp - T(1.5) * ltp));
  const T hpp = r * (spp - T(3) * sp * lp + s * (T(3.75) * lp * lp - T(1.5) * lpp));
  // contravariant metric, u^a = a^ab h_,b, and Lap(h) = a^ab (h_,ab - x_ab . u)
  const T c11 = g22.v * iq, c22 = g11.v * iq, c12 = T(0.5) * g12.v * iq;
  const T u1 = c11 * ht + c12 * hp, u2 = c12 * ht + c22 * hp;
  const T k11 = htt - (u1 * a1x11 + u2 * a2x11), k12 = htp - (u1 * a1x12 + u2 * a2x12),
          k22 = hpp - (u1 * a1x22 + u2 * a2x22);
  const T lap = c11 * k11 + T(2) * c12 * k12 + c22 * k22;
  const T w1 = (u1 * L.v + u2 * M.v) * isq, w2 = (u1 * M.v + u2 * N.v) * isq;  // u^b b_ba
  const T d1 = eb * (c11 * w1 + c12 * w2), d2 = eb * (c12 * w1 + c22 * w2), dn = -eb * lap * isq;
  for (int c = 0; c < 3; ++c) f[c] += dn * m[c] + d1 * a1[c] + d2 * a2[c];
}

}  // namespace sg
