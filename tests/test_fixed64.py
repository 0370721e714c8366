"""The fixed-point functions of the plain FP64 walks (csrc/fixed64.hpp, compiled for the host)
against extended precision."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53
SOURCE = r"""
#include "fixed64.hpp"
extern "C" void turn(const uint64_t *t, double *s, double *c, long n) { for (long i = 0; i < n; i++) vmc::sincos_turn(t[i], s[i], c[i]); }
extern "C" void nlog(const uint32_t *w, double *y, long n) { for (long i = 0; i < n; i++) y[i] = vmc::neg_log_open(w[i]); }
extern "C" void expx(const double *x, double *y, long n) { for (long i = 0; i < n; i++) y[i] = vmc::one_minus_exp_over_x(x[i]); }
extern "C" void frac(const double *x, uint64_t *y, long n) { for (long i = 0; i < n; i++) y[i] = vmc::fixed_of_double(x[i]); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if np.finfo(np.longdouble).eps > 2e-19:
        pytest.skip("long double is no wider than double here")
    d = tmp_path_factory.mktemp("fixed64")
    (d / "f.cpp").write_text(SOURCE)
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "valomc_gb300", "csrc"),
                    str(d / "f.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def call(fn, x, *outs):
    fn(x.ctypes.data_as(C.c_void_p), *[o.ctypes.data_as(C.c_void_p) for o in outs], C.c_long(len(x)))
    return outs


def test_sine_and_cosine_of_a_turn(lib):
    rng = np.random.default_rng(1)
    eighth = (np.arange(8, dtype=np.uint64) << np.uint64(61))
    near = np.concatenate([eighth + np.uint64(k) for k in range(0, 40)] + [eighth - np.uint64(k) for k in range(1, 40)])
    t = np.concatenate([near, rng.integers(0, 2 ** 64, 400000, dtype=np.uint64)])
    s, c = call(lib.turn, t, np.empty(len(t)), np.empty(len(t)))
    a = t.astype(np.longdouble) / np.longdouble(2) ** 64
    a = (a - np.rint(a)) * (8 * np.arctan(np.longdouble(1)))
    # one rounding of a result below 1 (half a unit of 2^-53) and the truncation, below 2^-56
    assert np.max(np.abs(s - np.sin(a))) < 1.1 * U and np.max(np.abs(c - np.cos(a))) < 1.1 * U
    for k, (es, ec) in enumerate([(0, 1), (1, 0), (0, -1), (-1, 0)]):
        assert s[2 * k] == es and c[2 * k] == ec


def test_exponential_sample(lib):
    rng = np.random.default_rng(2)
    edges = np.concatenate([np.arange(300), 2 ** 32 - 1 - np.arange(300), 2 ** np.arange(32) - 1, 2 ** np.arange(32)])
    w = np.concatenate([edges, rng.integers(0, 2 ** 32, 400000), 2 ** 32 - 1 - rng.integers(0, 2 ** 24, 100000)])
    w = w.astype(np.uint32)
    (y,) = call(lib.nlog, w, np.empty(len(w)))
    want = -np.log((w.astype(np.longdouble) + np.longdouble(0.5)) / np.longdouble(2) ** 32)
    want[w >= 2 ** 31] = -np.log1p(-((2 ** 32 - 1 - w[w >= 2 ** 31].astype(np.longdouble)) + np.longdouble(0.5)) / np.longdouble(2) ** 32)
    # -log x from a table entry and a series, 2^-60 each, next to 0.0039 at the least: 2^-52
    assert np.max(np.abs(y - want) / want) < 2.5 * U
    assert np.all(y > 0)


def test_absorbed_fraction_over_its_depth(lib):
    rng = np.random.default_rng(3)
    x = np.concatenate([[0.0, 5e-324, 1e-300, 2.0 ** -64, 2.0 ** -53], np.nextafter(0.0625, 0) * np.ones(1),
                        rng.uniform(0, 0.0625, 300000), 10.0 ** rng.uniform(-20, -1.3, 100000)])
    (y,) = call(lib.expx, x, np.empty(len(x)))
    xl = x.astype(np.longdouble)
    want = np.where(xl > 1e-15, -np.expm1(-xl) / np.where(xl > 0, xl, 1), 1 - xl / 2)
    assert np.max(np.abs(y - want) / want) < 1.1 * U


def test_fraction_of_a_double(lib):
    rng = np.random.default_rng(4)
    x = np.concatenate([[0.0, 5e-324, 0.5, 1.0, 1.5, 2.0 ** 40 + 0.25, 2.0 ** -64, 2.0 ** -65], rng.uniform(0, 3, 1000)])
    (y,) = call(lib.frac, x, np.empty(len(x), np.uint64))
    want = [int(np.floor(np.ldexp(np.longdouble(v) - np.floor(np.longdouble(v)), 64))) for v in x]
    assert [int(v) for v in y] == want
