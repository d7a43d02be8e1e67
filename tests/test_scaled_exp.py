"""The exponential of an argument in table steps (fexp_s of pjg_math.cuh), which
the kernels take for rate constants, k0 / kinf and the fall-off terms, on the
CPU: the header's own code compiled for the host, its intrinsics being the
IEEE operations that they name.

Against 2^(xs / 1024) 2^(n0 / 1024) in extended precision.  Its error in ulp:
1/2 for the table entry, 1/2 for the last FMA, and the polynomial's 9.4e-17,
which is 0.85 at most; products inside are scaled by |r| <= 3.4e-4: below 2.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
using std::fma; using std::exp; using std::log; using std::pow;
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __align__(n) alignas(n)
struct { int x; } threadIdx, blockDim;
struct int2 { int x, y; };
struct int4 { int x, y, z, w; };
template <class T> inline T __ldg(const T* p) { return *p; }
inline long long __double_as_longlong(double x) { long long b; memcpy(&b, &x, 8); return b; }
inline double __longlong_as_double(long long b) { double x; memcpy(&x, &b, 8); return x; }
inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
inline int __double2loint(double x) { return (int)__double_as_longlong(x); }
inline double __hiloint2double(int h, int l) { return __longlong_as_double((long long)h << 32 | (unsigned)l); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
#include "pjg_math.cuh"
extern "C" void scaled_exp(const double* xs, const int* n0, double* y, double* ref, int n)
{
    for (int i = 0; i < n; ++i) {
        y[i] = pjg::fexp_s(xs[i], n0[i], pjg_exp2_table);
        ref[i] = (double)(exp2l((long double)xs[i] / PJG_EXP_TAB) * exp2l((long double)n0[i] / PJG_EXP_TAB));
    }
}
extern "C" double exp_max() { return EXP_MAX; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("scaled_exp")
    src, so = d / "scaled_exp.cpp", d / "scaled_exp.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "pyjac-v2_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def evaluate(lib, xs, n0):
    xs = np.ascontiguousarray(xs, dtype=np.float64)
    n0 = np.ascontiguousarray(np.broadcast_to(n0, xs.shape), dtype=np.int32)
    y, ref = np.empty_like(xs), np.empty_like(xs)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    lib.scaled_exp(p(xs), p(n0), p(y), p(ref), xs.size)
    return y, ref


def test_error_over_the_range(lib):
    rng = np.random.default_rng(3)
    k = np.arange(-3000, 3000)
    top = 2.0 ** 20
    near = np.concatenate([k + 0.5, np.nextafter(k + 0.5, np.inf), np.nextafter(k + 0.5, -np.inf), k, k + 1e-9])
    parts = [(rng.uniform(-2, 2, 100000), 0), (near, 0),
             (rng.uniform(-1, 1, 100000) * 10.0 ** rng.uniform(-320, 5, 100000), 0),
             (np.array([0.0, -0.0, 5e-324, -5e-324, 0.5, -0.5, 1.0, -1.0, np.nextafter(top, 0), -np.nextafter(top, 0)]), 0)]
    xs = rng.uniform(-top, top, 300000)
    parts.append((xs, (rng.uniform(-1.04e6, 1.02e6, xs.size) - xs).astype(np.int32)))  # e^-704 .. e^690
    for xs, n0 in parts:
        total = xs + n0
        y, ref = evaluate(lib, xs, n0)
        ok = (total > -1.04e6) & (total < 996 * 1024.0)
        assert ok.any()
        assert float((np.abs(y[ok] - ref[ok]) / np.spacing(ref[ok])).max()) <= 2.0
        # from 2^996 to the clamp the library takes exp of the argument as a double:
        # half an ulp of 691 for it and 691 2^-53 for the step's own rounding
        far = (total >= 996 * 1024.0) & (total < 1.02e6)
        assert float(np.abs(y[far] / ref[far] - 1.0).max(initial=0.0)) <= 2e-13


def test_outside_the_range(lib):
    """The library exponential with the clamp at EXP_MAX (rounding of the
    argument's product aside: 710 2^-52), zero below, and special values."""
    lib.exp_max.restype = ctypes.c_double
    top = np.exp(lib.exp_max())
    y, _ = evaluate(lib, [1.1e6, 1e9, np.inf, -1.2e6, -1e300, -np.inf, np.nan], 0)
    assert np.allclose(y[:3], top, rtol=1e-13, atol=0)
    assert (y[3:6] == 0.0).all() and np.isnan(y[6])
    y, ref = evaluate(lib, [-1.05e6, -1.06e6, -1.08e6], 0)  # around the smallest normal number
    assert float(np.abs(y / ref - 1.0).max()) < 1e-12
