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
extern "C" void turn60(const uint64_t *t, int64_t *s, int64_t *c, long n) { for (long i = 0; i < n; i++) vmc::sincos_turn_fixed(t[i], s[i], c[i]); }
extern "C" void to60(const double *x, int64_t *y, double *z, long n) { for (long i = 0; i < n; i++) z[i] = vmc::double_of_60(y[i] = vmc::fixed60_of(x[i])); }
extern "C" void prod(const int64_t *x, int64_t *p, int64_t *q, long n) {
  for (long i = 0; i + 3 < n; i += 4) {
    const vmc::Split60 a = vmc::split60(x[i]), b = vmc::split60(x[i + 1]), c = vmc::split60(x[i + 2]), d = vmc::split60(x[i + 3]);
    p[i] = vmc::mul60(a, b);
    q[i] = vmc::dot60(a, b, vmc::neg60(c), d);
  }
}
extern "C" void rcp(const uint64_t *d, uint64_t *y, long n) { for (long i = 0; i < n; i++) y[i] = vmc::rcp_fixed(d[i]); }
extern "C" void root(const int64_t *s, int64_t *r, int64_t *y, int32_t *k, long n) {
  for (long i = 0; i < n; i++) { const vmc::Root60 q = vmc::sqrt60(s[i]); r[i] = q.r; y[i] = q.y; k[i] = q.k; }
}
extern "C" void hg(const uint32_t *u, const double *g, int64_t *c, long n) { for (long i = 0; i < n; i++) c[i] = vmc::hg_cosine(u[i], g[i], vmc::hg_inverse(g[i])); }
extern "C" void turn2(const uint32_t *u, const double *g, int64_t *c, int64_t *s, int32_t *ok, long n) {
  for (long i = 0; i < n; i++) ok[i] = vmc::turn_2d(u[i], g[i], vmc::turn_ratio(g[i]), c[i], s[i]);
}
extern "C" void unit(int64_t *v, int32_t *ok, long n) { for (long i = 0; i < n; i++) ok[i] = vmc::unit60(v + 3 * i, 3); }
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


ONE = 2 ** 60


def test_fixed_sine_and_cosine_are_the_double_ones(lib):
    rng = np.random.default_rng(5)
    t = np.concatenate([np.arange(8, dtype=np.uint64) << np.uint64(61), rng.integers(0, 2 ** 64, 200000, dtype=np.uint64)])
    s, c = call(lib.turn60, t, np.empty(len(t), np.int64), np.empty(len(t), np.int64))
    sd, cd = call(lib.turn, t, np.empty(len(t)), np.empty(len(t)))
    for a, b in ((s, sd), (c, cd)):  # the double's rounding and a unit of 2^-62
        assert np.max(np.abs(a.astype(np.longdouble) / np.longdouble(4 * ONE) - b)) <= 0.5 * U + 2.0 ** -62


def test_fixed_numbers_and_their_products(lib):
    rng = np.random.default_rng(6)
    x = np.concatenate([[0.0, -0.0, 1.0, -1.0, 2.0 ** -60, -(2.0 ** -60), 2.0 ** -61, 5e-324, np.nextafter(2, 0)],
                        rng.uniform(-1, 1, 100000), rng.uniform(-1, 1, 1000) * 10.0 ** rng.uniform(-20, 0, 1000)])
    y, z = call(lib.to60, x, np.empty(len(x), np.int64), np.empty(len(x)))
    exact = [int(np.trunc(np.ldexp(np.longdouble(v), 60))) for v in x]
    assert [int(v) for v in y] == exact
    assert np.all(np.abs(z - x) < 2.0 ** -60)
    v = np.concatenate([np.array([ONE, ONE, -ONE, ONE, -ONE, -1, ONE - 1, 1 - ONE], np.int64), y[np.abs(x) <= 1][:80000]])
    v = v[:len(v) // 4 * 4]
    p, q = call(lib.prod, v, np.zeros(len(v), np.int64), np.zeros(len(v), np.int64))
    for i in range(0, len(v), 4):
        a, b, c, d = (int(w) for w in v[i:i + 4])
        # the lower halves' product (below a unit each) and the shift's remainder
        assert 0 <= a * b - (int(p[i]) << 60) < 2 << 60
        assert abs(a * b - c * d - (int(q[i]) << 60)) < 3 << 60


def test_reciprocal_and_root(lib):
    rng = np.random.default_rng(7)
    d = np.concatenate([np.uint64(2 ** 63) + np.arange(64, dtype=np.uint64), np.uint64(2 ** 64 - 1) - np.arange(64, dtype=np.uint64),
                        rng.integers(2 ** 63, 2 ** 64, 100000, dtype=np.uint64)])
    (y,) = call(lib.rcp, d, np.empty(len(d), np.uint64))
    for a, b in zip(d.tolist(), y.tolist()):
        # e is cut to 2 units of 2^-61, times y0 <= 2, and the two shifts: 6 units; the series 2^-66
        assert abs(b * a - (1 << 125)) < 7 * a
    s = np.concatenate([np.arange(1, 300), ONE - np.arange(300), 2 ** np.arange(60) + 1, 2 ** np.arange(61), rng.integers(1, ONE, 100000),
                        (ONE * 10.0 ** rng.uniform(-15, 0, 20000)).astype(np.int64) + 1]).astype(np.int64)
    s = s[s <= ONE]
    r, y, k = call(lib.root, s, np.empty(len(s), np.int64), np.empty(len(s), np.int64), np.empty(len(s), np.int32))
    t = s.astype(np.longdouble) / ONE * np.longdouble(4) ** k
    assert t.min() >= 0.25 and t.max() <= 1
    # h and e are cut to 2 and 5 units of 2^-60, u to 1 more; times h <= 1 and y0 <= 2
    assert np.max(np.abs(r / np.longdouble(ONE) - np.sqrt(t))) < 10 / np.longdouble(ONE)
    assert np.max(np.abs(y / np.longdouble(ONE) - 1 / np.sqrt(t))) < 18 / np.longdouble(ONE)


def test_henyey_greenstein_cosine(lib):
    rng = np.random.default_rng(8)
    n = 200000
    u = np.concatenate([np.arange(1, 50), 2 ** 32 - 2 - np.arange(50), [0, 2 ** 32 - 1], rng.integers(0, 2 ** 32, n)]).astype(np.uint32)
    g = rng.uniform(-0.999, 0.999, len(u))
    g[::5] = rng.choice([0.0, 0.8, 0.9, -0.5, 0.99, 0.01, 1e-6, 2.0 ** -30], len(g[::5]))
    c = call(lib.hg, u, g, np.empty(len(u), np.int64))[-1]
    gl, c0 = g.astype(np.longdouble), 2 * (u.astype(np.longdouble) / np.longdouble(2 ** 32 - 1)) - 1
    d = 1 + gl * c0
    q = (1 - gl * gl) / d
    with np.errstate(divide="ignore", invalid="ignore"):
        want = np.where(gl == 0, c0, (1 + gl * gl - q * q) / (2 * gl))
        # d is cut to 4 units of 2^-60, the other terms to 8
        bound = np.where(gl == 0, 4, np.abs(0.5 / g) * (2 * q * q * (4 / d + 8) + 8) + 4) / np.longdouble(ONE)
    inner = (u > 0) & (u < 2 ** 32 - 1)
    assert np.all(np.abs(c / np.longdouble(ONE) - want)[inner] <= bound[inner] + 2.0 ** -62)
    assert np.all(c[u == 0] == -ONE) and np.all(c[u == 2 ** 32 - 1] == ONE)
    edge = np.array([1.0, -1.0, 0.9995, 1e-10, np.nan, 2.0])
    c = call(lib.hg, np.full(6, 12345, np.uint32), edge, np.empty(6, np.int64))[-1]
    assert np.all(c == np.iinfo(np.int64).min)


def test_turn_in_the_plane(lib):
    rng = np.random.default_rng(10)
    n = 200000
    u = np.concatenate([np.arange(50), 2 ** 32 - 1 - np.arange(50), 2 ** 31 + np.arange(-20, 20), rng.integers(0, 2 ** 32, n)]).astype(np.uint32)
    g = rng.uniform(-0.998, 0.998, len(u))
    g[::5] = rng.choice([0.0, 0.8, 0.9, -0.5, 0.99, 0.01, 1e-6, -0.998], len(g[::5]))
    c, s, ok = call(lib.turn2, u, g, np.empty(len(u), np.int64), np.empty(len(u), np.int64), np.empty(len(u), np.int32))[1:]
    assert np.all(ok == 1)
    a = u.astype(np.longdouble) / np.longdouble(2 ** 32) * (4 * np.arctan(np.longdouble(1)))
    k = (1 - np.abs(g.astype(np.longdouble))) / (1 + np.abs(g.astype(np.longdouble)))
    x, y = np.cos(a) * np.where(g < 0, k, 1), np.sin(a) * np.where(g < 0, 1, k)
    d = x * x + y * y
    # x and y are cut to 2 units of 2^-60 when the larger is brought to [1/2, 1), from units of 2^-62
    # and k's own 5 of 2^-61; each square to 6, times 1 / d <= 4, and the
    # quotient's own 8
    bound = (4 * (6 + 6 + 4 / (4 * np.maximum(np.abs(x), np.abs(y))) * 4) + 8) / np.longdouble(ONE)
    iso = g == 0
    wc, ws = np.where(iso, np.cos(2 * a), (x * x - y * y) / d), np.where(iso, np.sin(2 * a), 2 * x * y / d)
    assert np.all(np.abs(c / np.longdouble(ONE) - wc) < bound) and np.all(np.abs(s / np.longdouble(ONE) - ws) < bound)
    edge = np.array([1.0, -1.0, 0.9999, 1e-300, 2.0, -2.0, np.nan])
    ok = call(lib.turn2, np.full(7, 12345, np.uint32), edge, np.empty(7, np.int64), np.empty(7, np.int64), np.empty(7, np.int32))[-1]
    assert not ok.any()


def test_unit_vectors(lib):
    rng = np.random.default_rng(9)
    v = rng.normal(size=(100000, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    v *= 1 + rng.uniform(-0.45, 0.45, (len(v), 1)) * 2.0 ** -30
    f = np.rint(v * ONE).astype(np.int64)
    ok = np.zeros(len(v), np.int32)
    lib.unit(f.ctypes.data_as(C.c_void_p), ok.ctypes.data_as(C.c_void_p), C.c_long(len(v)))
    assert np.all(ok == 1)
    length = np.sqrt(np.sum((f / np.longdouble(ONE)) ** 2, axis=1))
    assert np.max(np.abs(length - 1)) < 8 / np.longdouble(ONE)  # the sum is cut to 2 units, a component to 1 each
    f = np.array([[ONE, ONE >> 14, 0], [ONE + (1 << 31), 0, 0]], np.int64)
    lib.unit(f.ctypes.data_as(C.c_void_p), ok.ctypes.data_as(C.c_void_p), C.c_long(2))
    assert np.all(ok[:2] == 0)
