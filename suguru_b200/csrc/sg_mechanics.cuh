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
// A^11 A^22, cot t, and the power of two c with 1 <= c st < 2.
__device__ __forceinline__ float pow2_inv(float x) {
  return __int_as_float(0x7F000000 - (__float_as_int(x) & 0x7F800000));
}
__device__ __forceinline__ double pow2_inv(double x) {
  return __hiloint2double(0x7FE00000 - (__double2hiint(x) & 0x7FF00000), 0);
}
template <class T>
struct RefSphere {
  T A1, A2, rA, cot, c;
  __device__ __forceinline__ RefSphere(T R, T st, T ct) {
    const T is = fdiv(T(1), st), q = ct * is;
    cot = fma(fma(-q, st, ct), is, q);
    c = pow2_inv(st);
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
// h = S / q^(3/2) with S = g22 L - 2 g12 M + g11 N, L, M, N the second
// derivatives of x along m = e1 x e2 and q = m . m: its value and five
// derivatives follow from products, about 500 operations instead of 2,500 and
// no tensors to keep.  The frame is e1 = x_t, e2 = c x_p with c'/c = -cot t,
// as 1 / sin t has, and the derivatives are D1 = d/dt, D2 = c d/dp (D1 D2 =
// D2 D1 - cot D2; both obey the product rule), so that the powers of sin t,
// whose derivatives would have to cancel in h, do not appear: from x_p itself
// (450 operations) a point's rounding error was 3.7 times the reference form's in
// FP32 and FP64, a mixed step's force at degree 5 off by 1.4e-6 against 0.8e-6;
// now 0.7 of that form's, and 0.75e-6.  c is a power of two on each row and the
// factors cot are applied one at a time: a rounded constant in common to a row's
// points would leave an error that does not average out over them.
// S3 = x_ttt, x_ttp, x_tpp, x_ppp; S4 = x_tttt, x_tttp, x_ttpp, x_tppp, x_pppp.
template <class T>
struct Jet2 {  // a function on the surface: value and derivatives D1, D2, D1 D1, D1 D2, D2 D2
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
__device__ __forceinline__ void bending_force(const T* a1, const T* x_p, const T* x11, const T* x_tp, const T* x_pp,
                                              const T (*S3)[3], const T (*S4)[3], const RefSphere<T>& R, T eb, T* f) {
  auto dot = [](const T* u, const T* v) { return dot3(u, v); };
  const T c1 = R.c, c2 = c1 * c1, c3 = c2 * c1, c4 = c2 * c2, k = R.cot, k2 = T(2) * k;
  // derivatives of x11 = D1 e1, of e2, u = D2 e1 and v = D2 e2: _1 = D1 and so on
  T e2[3], u[3], v[3], e2_1[3], e2_11[3], x11_2[3], x11_12[3], x11_22[3];
  T u_1[3], u_2[3], u_11[3], u_12[3], u_22[3], v_1[3], v_2[3], v_11[3], v_12[3], v_22[3];
  const T *x11_1 = S3[0], *x11_11 = S4[0];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    e2[i] = x_p[i] * c1;
    u[i] = x_tp[i] * c1;
    v[i] = x_pp[i] * c2;
    e2_1[i] = u[i] - k * e2[i];
    x11_2[i] = S3[1][i] * c1;
    u_1[i] = x11_2[i] - k * u[i];
    e2_11[i] = x11_2[i] - k2 * e2_1[i] + e2[i];
    u_2[i] = S3[2][i] * c2;
    v_1[i] = u_2[i] - k2 * v[i];
    v_2[i] = S3[3][i] * c3;
    const T t = S4[1][i] * c1;
    x11_12[i] = t - k * x11_2[i];
    u_11[i] = t - k2 * u_1[i] + u[i];
    x11_22[i] = S4[2][i] * c2;
    u_12[i] = x11_22[i] - k2 * u_2[i];
    v_11[i] = x11_22[i] - T(4) * k * (v_1[i] + T(0.5) * k * v[i]) + T(2) * v[i];
    u_22[i] = S4[3][i] * c3;
    v_12[i] = u_22[i] - k * (T(3) * v_2[i]);
    v_22[i] = S4[4][i] * c4;
  }
  T m[3], m1[3], m2[3], m11[3], m12[3], m22[3];
  {
    T p[3], q[3], r[3], s[3];
    cross3(a1, e2, m);
    cross3(x11, e2, p);
    cross3(a1, e2_1, q);
    for (int c = 0; c < 3; ++c) m1[c] = p[c] + q[c];
    cross3(u, e2, p);
    cross3(a1, v, q);
    for (int c = 0; c < 3; ++c) m2[c] = p[c] + q[c];
    cross3(x11_1, e2, p);
    cross3(x11, e2_1, q);
    cross3(a1, e2_11, r);
    for (int c = 0; c < 3; ++c) m11[c] = p[c] + T(2) * q[c] + r[c];
    cross3(u_1, e2, p);
    cross3(x11, v, q);
    cross3(u, e2_1, r);
    cross3(a1, v_1, s);
    for (int c = 0; c < 3; ++c) m12[c] = p[c] + q[c] + r[c] + s[c];
    cross3(u_2, e2, p);
    cross3(u, v, q);
    cross3(a1, v_2, r);
    for (int c = 0; c < 3; ++c) m22[c] = p[c] + T(2) * q[c] + r[c];
  }
  // 1 / q by the fast division and one correction (the IEEE division's call for
  // its rare cases would spill)
  const T q = dot(m, m), iq0 = fdiv(T(1), q), iq = fma(fma(-q, iq0, T(1)), iq0, iq0);
  const T l1 = T(2) * dot(m, m1) * iq, l2 = T(2) * dot(m, m2) * iq;  // D1 q / q, D2 q / q
  const T l11 = T(2) * (dot(m1, m1) + dot(m, m11)) * iq, l12 = T(2) * (dot(m1, m2) + dot(m, m12)) * iq,
          l22 = T(2) * (dot(m2, m2) + dot(m, m22)) * iq;
  // x . m with its derivatives, from x and its derivatives
  auto proj = [&](const T* x, const T* x1, const T* x2, const T* x11, const T* x12, const T* x22) {
    Jet2<T> j;
    j.v = dot(x, m);
    j.t = dot(x1, m) + dot(x, m1);
    j.p = dot(x2, m) + dot(x, m2);
    j.tt = dot(x11, m) + T(2) * dot(x1, m1) + dot(x, m11);
    j.tp = dot(x12, m) + dot(x1, m2) + dot(x2, m1) + dot(x, m12);
    j.pp = dot(x22, m) + T(2) * dot(x2, m2) + dot(x, m22);
    return j;
  };
  const T a1x11 = dot(a1, x11);
  const Jet2<T> g11 = {dot(a1, a1), T(2) * a1x11, T(2) * dot(a1, u), T(2) * (dot(x11, x11) + dot(a1, x11_1)),
                       T(2) * (dot(u, x11) + dot(a1, u_1)), T(2) * (dot(u, u) + dot(a1, u_2))};
  const Jet2<T> g22 = {dot(e2, e2), T(2) * dot(e2, e2_1), T(2) * dot(e2, v), T(2) * (dot(e2_1, e2_1) + dot(e2, e2_11)),
                       T(2) * (dot(e2_1, v) + dot(e2, v_1)), T(2) * (dot(v, v) + dot(e2, v_2))};
  // -2 g12
  const T g12v = dot(a1, e2);
  const Jet2<T> g12 = {-T(2) * g12v,
                       -T(2) * (dot(x11, e2) + dot(a1, e2_1)),
                       -T(2) * (dot(u, e2) + dot(a1, v)),
                       -T(2) * (dot(x11_1, e2) + T(2) * dot(x11, e2_1) + dot(a1, e2_11)),
                       -T(2) * (dot(u_1, e2) + dot(x11, v) + dot(u, e2_1) + dot(a1, v_1)),
                       -T(2) * (dot(u_2, e2) + T(2) * dot(u, v) + dot(a1, v_2))};
  const Jet2<T> L = proj(x11, x11_1, x11_2, x11_11, x11_12, x11_22);
  const Jet2<T> M = proj(u, u_1, u_2, u_11, u_12, u_22);
  const Jet2<T> N = proj(v, v_1, v_2, v_11, v_12, v_22);
  const Jet2<T> A = g22 * L, B = g12 * M, C = g11 * N;
  const T s = A.v + B.v + C.v, s1 = A.t + B.t + C.t, s2 = A.p + B.p + C.p;
  const T s11 = A.tt + B.tt + C.tt, s12 = A.tp + B.tp + C.tp, s22 = A.pp + B.pp + C.pp;
  // h = s r with r = q^(-3/2): D1 r / r = -3/2 l1, D1 D1 r / r = 15/4 l1^2 - 3/2 l11
  const T isq = sqrt(iq), r = iq * isq;
  const T h1 = r * (s1 - T(1.5) * s * l1), h2 = r * (s2 - T(1.5) * s * l2);
  const T h11 = r * (s11 - T(3) * s1 * l1 + s * (T(3.75) * l1 * l1 - T(1.5) * l11));
  const T h12 = r * (s12 - T(1.5) * (s1 * l2 + s2 * l1) + s * (T(3.75) * l1 * l2 - T(1.5) * l12));
  const T h22 = r * (s22 - T(3) * s2 * l2 + s * (T(3.75) * l2 * l2 - T(1.5) * l22));
  // contravariant metric, g^a = a^ab D_b h, and Lap(h) = a^ab (D_a D_b h - D_a e_b . g)
  const T c11 = g22.v * iq, c22 = g11.v * iq, c12 = -g12v * iq;
  const T u1 = c11 * h1 + c12 * h2, u2 = c12 * h1 + c22 * h2;
  const T k11 = h11 - (u1 * a1x11 + u2 * dot(x11, e2)), k12 = h12 - (u1 * dot(a1, e2_1) + u2 * dot(e2, e2_1)),
          k22 = h22 - (u1 * dot(a1, v) + u2 * dot(e2, v));
  const T lap = c11 * k11 + T(2) * c12 * k12 + c22 * k22;
  const T w1 = (u1 * L.v + u2 * M.v) * isq, w2 = (u1 * M.v + u2 * N.v) * isq;  // g^b b_ba
  const T d1 = eb * (c11 * w1 + c12 * w2), d2 = eb * (c12 * w1 + c22 * w2), dn = -eb * lap * isq;
  for (int c = 0; c < 3; ++c) f[c] += dn * m[c] + d1 * a1[c] + d2 * e2[c];
}

}  // namespace sg
