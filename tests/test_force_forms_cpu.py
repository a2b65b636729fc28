"""Rounding errors of the pointwise membrane and bending forces, on the CPU.

sg_mechanics.cuh is compiled as C++ (fused multiply-adds only where it writes them) and its force of a
point evaluated in 32 and 64 bits on surfaces with exact derivatives: spheres displaced by 5 % by random
polynomials of degree 4 in the Cartesian coordinates, at the force grids' points of degrees 3 to 8.  The error
is the difference from the same function in long double, rms over the points weighted by area, relative
to the rms force.  The reference's own form (basis, Christoffel symbols, covariant divergence; moment
tensor with its first and second derivatives), compiled and evaluated in the same way on the same
surfaces, has the errors of REFERENCE: the kernels' shorter forms may have no larger ones.
"""
import ctypes
import functools
import os
import shutil
import subprocess

import numpy as np
import pytest

from suguru_b200 import workloads as W

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "suguru_b200", "csrc")
REFERENCE = {("f", 0.0): 1.83e-6, ("f", 0.3): 4.04e-6, ("d", 0.0): 3.46e-15, ("d", 0.3): 7.65e-15}

SHIM = """
#pragma once
#include <cmath>
#include <cstring>
#define __device__
#define __forceinline__ inline
using std::fma;
using std::sqrt;
inline float __fdividef(float a, float b) { return a / b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline int __float_as_int(float x) { int i; memcpy(&i, &x, 4); return i; }
inline float __int_as_float(int i) { float x; memcpy(&x, &i, 4); return x; }
inline int __double2hiint(double x) { long long i; memcpy(&i, &x, 8); return (int)(i >> 32); }
inline double __hiloint2double(int h, int l) {
  long long i = ((long long)h << 32) | (unsigned)l; double x; memcpy(&x, &i, 8); return x;
}
namespace sg {
using E = long double;
inline E mul_rn(E a, E b) { return a * b; }
inline E pow2_inv(E x) { return std::exp2(-std::floor(std::log2(x))); }
template <class T> T dot3(const T* u, const T* v) { return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]; }
template <class T> void cross3(const T* u, const T* v, T* w) {
  w[0] = u[1] * v[2] - u[2] * v[1]; w[1] = u[2] * v[0] - u[0] * v[2]; w[2] = u[0] * v[1] - u[1] * v[0];
}
}
"""
HARNESS = """
#include "sg_mechanics.cuh"
namespace sg {
template <> inline E fdiv<E>(E a, E b) { return a / b; }
template <class T>
void run(long n, const double* x, const double* sc, double R, double eb, int law, double* out) {
  for (long p = 0; p < n; ++p) {
    T d[14][3], f[3], nrm[3];
    for (int q = 0; q < 14; ++q)
      for (int c = 0; c < 3; ++c) d[q][c] = (T)x[(p * 14 + q) * 3 + c];
    const RefSphere<T> S((T)R, (T)sc[2 * p], (T)sc[2 * p + 1]);
    membrane_force<T>(d[0], d[1], d[2], d[3], d[4], S, T(0.5), T(1), law, nrm, f);
    if (eb != 0.0) bending_force<T>(d[0], d[1], d[2], d[3], d[4], d + 5, d + 9, S, (T)eb, f);
    for (int c = 0; c < 3; ++c) out[3 * p + c] = (double)f[c];
  }
}
}
#define RUN(name, T) extern "C" void name(long n, const double* x, const double* sc, double R, double eb, int law, \\
                                          double* out) { sg::run<T>(n, x, sc, R, eb, law, out); }
RUN(run_f, float)
RUN(run_d, double)
RUN(run_e, long double)
"""
ORDER = [(1, 0), (0, 1), (2, 0), (1, 1), (0, 2), (3, 0), (2, 1), (1, 2), (0, 3), (4, 0), (3, 1), (2, 2), (1, 3), (0, 4)]


def _derivative(poly, along_p):
    """Of sums {(m, sin?, a, b): coefficient} of sin^a t cos^b t (cos or sin)(m p)."""
    out = {}
    for (m, s, a, b), v in poly.items():
        terms = [((m, 1 - s, a, b), v * (m if s else -m))] if along_p else \
            [((m, s, a - 1, b + 1), v * a), ((m, s, a + 1, b - 1), -v * b)]
        for k, w in terms:
            if w:
                out[k] = out.get(k, 0.0) + w
    return out


def _value(poly, st, ct, p):
    v = np.zeros(np.broadcast(st, p).shape, np.longdouble)
    for (m, s, a, b), c in poly.items():
        v += c * st ** a * ct ** b * (np.sin(m * p) if s else np.cos(m * p))
    return v


@functools.cache
def surfaces(dtype, count=24, deg=4):
    """(R, derivatives [nlat][nlon][14][3], (sin t, cos t), weights), inputs rounded to dtype."""
    rng, out = np.random.default_rng(17), []
    for q in range(count):
        t, w, p = W.force_grid(3 + q % 6)
        nlat, nlon = t.size, p.size
        st, ct = np.sin(t.astype(np.longdouble))[:, None], np.cos(t.astype(np.longdouble))[:, None]
        p = p.astype(np.longdouble)[None, :]
        R = rng.uniform(0.05, 0.2)
        d = np.zeros((nlat, nlon, 14, 3))
        for c in range(3):
            poly = {(1, 1, 1, 0): R} if c == 0 else {(1, 0, 1, 0): R} if c == 1 else {(0, 0, 0, 1): R}
            for m in range(deg + 1):
                for b in range(deg + 1 - m):
                    for s in range(2 if m else 1):
                        k = (m, s, m, b)
                        poly[k] = poly.get(k, 0.0) + 0.05 * R * rng.normal() / (1 + m + b) ** 2
            for k, (i, j) in enumerate(ORDER):
                f = poly
                for _ in range(i):
                    f = _derivative(f, False)
                for _ in range(j):
                    f = _derivative(f, True)
                d[:, :, k, c] = _value(f, st, ct, p)
        sc = np.ascontiguousarray(np.broadcast_to(np.stack([st, ct], -1), (nlat, nlon, 2)), dtype=np.float64)
        out.append((float(dtype(R)), d.astype(dtype).astype(np.float64), sc.astype(dtype).astype(np.float64), w))
    return out


def error(run, exact, dtype, cbend, law=0):
    num = den = 0.0
    for R, d, sc, w in surfaces(dtype):
        eb = float(dtype(cbend * R * R))
        n = d.shape[0] * d.shape[1]
        ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        f = [np.zeros((*d.shape[:2], 3)) for _ in range(2)]
        for o, fn in zip(f, (run, exact)):
            fn(ctypes.c_long(n), ptr(d), ptr(sc), ctypes.c_double(R), ctypes.c_double(eb), law, ptr(o))
        num += (w[:, None, None] * (f[0] - f[1]) ** 2).sum() / R ** 2
        den += (w[:, None, None] * f[1] ** 2).sum() / R ** 2
    return np.sqrt(num / den)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("forms")
    shutil.copy(os.path.join(CSRC, "sg_mechanics.cuh"), d)
    (d / "sg_common.cuh").write_text(SHIM)
    (d / "forms.cpp").write_text(HARNESS)
    so = str(d / "forms.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", so, str(d / "forms.cpp")],
                   check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("prec, dtype", [("f", np.float32), ("d", np.float64)])
@pytest.mark.parametrize("cbend", [0.0, 0.3])
def test_error_is_the_reference_forms_or_less(lib, prec, dtype, cbend):
    assert error(getattr(lib, "run_" + prec), lib.run_e, dtype, cbend) <= REFERENCE[prec, cbend]
