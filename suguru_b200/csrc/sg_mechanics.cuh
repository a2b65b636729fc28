// sg_mechanics.cuh -- pointwise geometry and membrane mechanics of one
// surface point (device code shared by the spectral force kernels).
//
// sph1.f90:581-651 (unit normal and its derivatives), sph.f90:442-476
// (curvature), sph1.f90:197-297 with co2contra (capsulesolid.f90:106-146:
// contravariant basis and derivatives), sph.f90:735-893 (Christoffel
// symbols), sph.f90:896-961 (metric tensors and derivatives), for the
// bending terms, in the reference's operation order; and the membrane force
// itself (cal_spectral_force's equilibrium, sph.f90:1668-1715) in the shorter
// form of membrane_force.
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

// ------------------------------------------------- geometry + mechanics ---
// The geometry that the bending terms differentiate (sg_bending.cu).
template <class T>
struct Geo {
  T a1[3], a2[3], d11[3], d12[3], d22[3];
  T n[3];
  T c1[3], c2[3];
  T conat[3], conatd1[2][3], bcur[3], chf[8];
  // derivatives of the unit normal and of the contravariant basis along
  // xi^al (cderi3, conderi1, conderi2 of the reference)
  T nde[2][3], cdc1[2][3], cdc2[2][3];
};

// sph1.f90:581-651 (normal), sph.f90:442-476 (curvature), sph1.f90:197-297
// with co2contra (capsulesolid.f90:106-146), sph.f90:735-893 (christof),
// sph.f90:896-961 (metrics).  Same operation order as the reference.
template <class T>
__device__ __forceinline__ void geometry(Geo<T>& G) {
  const T* cd1[2] = {G.d11, G.d12};
  const T* cd2[2] = {G.d12, G.d22};
  T cc[3];
  cross3(G.a1, G.a2, cc);
  const T sm = sqrt(cc[0] * cc[0] + cc[1] * cc[1] + cc[2] * cc[2]);
  for (int c = 0; c < 3; ++c) G.n[c] = fdiv(cc[c], sm);
  T (&nde)[2][3] = G.nde;
#pragma unroll
  for (int al = 0; al < 2; ++al) {
    T x1[3], x2[3], dc[3];
    cross3(cd1[al], G.a2, x1);
    cross3(G.a1, cd2[al], x2);
    for (int c = 0; c < 3; ++c) dc[c] = x1[c] + x2[c];
    const T tmp = fdiv(dot3(cc, dc), sqrt(cc[0] * cc[0] + cc[1] * cc[1] + cc[2] * cc[2]));
    for (int c = 0; c < 3; ++c) nde[al][c] = fdiv(T(1), sm) * (x1[c] + x2[c] - tmp * G.n[c]);
  }
  G.bcur[0] = dot3(G.n, G.d11);
  G.bcur[1] = dot3(G.n, G.d22);
  G.bcur[2] = dot3(G.n, G.d12);
  T a2n[3], na1[3];
  cross3(G.a2, G.n, a2n);
  cross3(G.n, G.a1, na1);
  const T hyb1 = dot3(G.a1, a2n), hyb2 = dot3(G.a2, na1);
  for (int c = 0; c < 3; ++c) {
    G.c1[c] = fdiv(a2n[c], hyb1);
    G.c2[c] = fdiv(na1[c], hyb2);
  }
  const T g = hyb1;
  T (&cdc1)[2][3] = G.cdc1;
  T (&cdc2)[2][3] = G.cdc2;
#pragma unroll
  for (int al = 0; al < 2; ++al) {
    T a2de_n3[3], a2_n3de[3], n3de_a1[3], n3_a1de[3], vt[3];
    cross3(cd2[al], G.n, a2de_n3);
    cross3(G.a2, nde[al], a2_n3de);
    cross3(nde[al], G.a1, n3de_a1);
    cross3(G.n, cd1[al], n3_a1de);
    for (int c = 0; c < 3; ++c) vt[c] = a2de_n3[c] + a2_n3de[c];
    const T gde = dot3(cd1[al], a2n) + dot3(G.a1, vt);
    for (int c = 0; c < 3; ++c) {
      cdc1[al][c] = fdiv(T(1), g) * (-gde * G.c1[c] + a2de_n3[c] + a2_n3de[c]);
      cdc2[al][c] = fdiv(T(1), g) * (-gde * G.c2[c] + n3de_a1[c] + n3_a1de[c]);
    }
  }
  // christof(gamma,beta,alpha) at [(gamma-1) + 2(beta-1) + 4(alpha-1)]
  G.chf[0 + 0 + 0] = dot3(G.d11, G.c1);  // (1,1,1)
  G.chf[1 + 0 + 0] = dot3(G.d12, G.c1);  // (2,1,1)
  G.chf[0 + 2 + 0] = dot3(G.d11, G.c2);  // (1,2,1)
  G.chf[1 + 2 + 0] = dot3(G.d12, G.c2);  // (2,2,1)
  G.chf[1 + 0 + 4] = dot3(G.d22, G.c1);  // (2,1,2)
  G.chf[1 + 2 + 4] = dot3(G.d22, G.c2);  // (2,2,2)
  G.chf[0 + 0 + 4] = G.chf[1];           // (1,1,2) = (2,1,1)
  G.chf[0 + 2 + 4] = G.chf[3];           // (1,2,2) = (2,2,1)
  G.conat[0] = G.c1[0] * G.c1[0] + G.c1[1] * G.c1[1] + G.c1[2] * G.c1[2];
  G.conat[1] = G.c2[0] * G.c2[0] + G.c2[1] * G.c2[1] + G.c2[2] * G.c2[2];
  G.conat[2] = dot3(G.c1, G.c2);
#pragma unroll
  for (int al = 0; al < 2; ++al) {
    G.conatd1[al][0] = T(2) * dot3(G.c1, cdc1[al]);
    G.conatd1[al][1] = T(2) * dot3(G.c2, cdc2[al]);
    G.conatd1[al][2] = dot3(G.c1, cdc2[al]) + dot3(G.c2, cdc1[al]);
  }
}

// The reference sphere of radius R at colatitude t (st = sin t, ct = cos t):
// contravariant metric A^11 = 1/R^2, A^22 = 1/(R st)^2 (A^12 = 0), its only
// derivative d_t A^22 = -2 ct / (R^2 st^3), and 1/(A^11 A^22), its root.
template <class T>
struct RefSphere {
  T A1, A2, A2t, iA, rA;
  __device__ __forceinline__ RefSphere(T R, T st, T ct) {
    const T is = fdiv(T(1), st), R2 = R * R;
    A1 = fdiv(T(1), R2);
    A2 = A1 * (is * is);
    A2t = (-T(2) * ct) * is * A2;
    rA = R2 * st;
    iA = rA * rA;
  }
};

// Unit normal and membrane force per area of one point (cal_spectral_force's
// equilibrium, sph.f90:1668-1715, with cal_Js_I1_I2_deri, sph.f90:1115-1156,
// the laws of membmodel.c and calculate_cauchy_tensor_deri, sph.f90:1179-1234).
// The reference forms the contravariant basis with its derivatives and the
// Christoffel symbols, takes the tension's covariant divergence and its
// contraction with the curvature, and sums q1 a1 + q2 a2 + q3 n.  With
// x_ab = G^c_ab a_c + b_ab n those sums are
//   f = (T^ab_,a + (q_,a / 2 q) T^ab) a_b + T^ab x_ab,   q = det a_ab,
// which needs the metric and its first derivatives only (six dot products
// beside the metric's three), the basis vectors and the second derivatives
// as they are: about 170 operations with one division and one root instead of
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
  const T g11 = dot3_fma(a1, a1), g22 = dot3_fma(a2, a2), g12 = dot3_fma(a1, a2), q = dot3_fma(cc, cc);
  const T a2d12 = dot3_fma(a2, d12), a1d12 = dot3_fma(a1, d12);
  const T g11d[2] = {T(2) * dot3_fma(a1, d11), T(2) * a1d12}, g22d[2] = {T(2) * a2d12, T(2) * dot3_fma(a2, d22)};
  const T g12d[2] = {dot3_fma(a2, d11) + a1d12, dot3_fma(a1, d22) + a2d12};
  const T iq = fdiv(T(1), q);
  const T AA = S.A1 * S.A2, J = sqrt(AA * q);    // sqrt(1 + I2) = Js
  const T iJ2 = iq * S.iA, iJ = J * iJ2;
  const T isq = (J * S.rA) * iq;                 // 1 / sqrt(q): over the normal's length
  for (int c = 0; c < 3; ++c) n[c] = mul_rn(cc[c], isq);
  const T I1 = fma(S.A1, g11, fma(S.A2, g22, -T(2)));
  const bool nh = law == 1;
  const T W1 = nh ? hf : fma(hf, I1, hf);
  const T W2 = nh ? -((hf * iJ2) * iJ2) : hf * fma(csk, fma(AA, q, -T(1)), -T(1));
  const T t1 = T(2) * W1 * iJ, s2 = T(2) * J * W2 * iq;  // T^ab = t1 A^ab + s2 adj(a)^ab
  T t1d[2], s2d[2], gam[2];
#pragma unroll
  for (int al = 0; al < 2; ++al) {
    const T A2d = al == 0 ? S.A2t : T(0);
    const T qd = fma(g11d[al], g22, fma(g11, g22d[al], (-T(2) * g12) * g12d[al]));
    const T I1d = fma(S.A1, g11d[al], fma(A2d, g22, S.A2 * g22d[al]));
    const T J2d = S.A1 * fma(A2d, q, S.A2 * qd);
    const T Jd = (T(0.5) * J2d) * iJ;
    const T W1d = nh ? T(0) : hf * I1d;
    const T W2d = nh ? (T(2) * hf * J2d) * (iJ2 * iJ2 * iJ2) : (hf * csk) * J2d;
    t1d[al] = fma(T(2), W1d, -(t1 * Jd)) * iJ;
    s2d[al] = fma(T(2), fma(Jd, W2, J * W2d), -(s2 * qd)) * iq;
    gam[al] = (T(0.5) * qd) * iq;
  }
  const T T11 = fma(t1, S.A1, s2 * g22), T22 = fma(t1, S.A2, s2 * g11), T12 = -(s2 * g12);
  const T T11d1 = fma(t1d[0], S.A1, fma(s2d[0], g22, s2 * g22d[0]));
  const T T22d2 = fma(t1d[1], S.A2, fma(s2d[1], g11, s2 * g11d[1]));
  const T T12d1 = -fma(s2d[0], g12, s2 * g12d[0]);
  const T T12d2 = -fma(s2d[1], g12, s2 * g12d[1]);
  const T c1 = fma(gam[0], T11, fma(gam[1], T12, T11d1 + T12d2));
  const T c2 = fma(gam[0], T12, fma(gam[1], T22, T12d1 + T22d2));
  for (int c = 0; c < 3; ++c)
    f[c] = fma(c1, a1[c], fma(c2, a2[c], fma(T11, d11[c], fma(T(2) * T12, d12[c], T22 * d22[c]))));
}

}  // namespace sg
