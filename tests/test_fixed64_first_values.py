"""The fixed-point functions of the plain FP64 walks with what the device gives them: FP32 first values
with the errors that CUDA documents, table entries read by 16-byte loads."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "fixed64.hpp"
extern "C" int log_align() { return (int)alignof(vmc::LogEntry); }
extern "C" void rcp(const uint64_t *d, int ulps, uint64_t *y, long n) {
  for (long i = 0; i < n; i++) {
    float f = vmc::rcp_first(d[i]);
    for (int u = 0; u < (ulps < 0 ? -ulps : ulps); u++) f = nextafterf(f, ulps < 0 ? 0.0f : 1e30f);
    y[i] = vmc::rcp_refined(d[i], f);
  }
}
extern "C" void root(const int64_t *s, int ulps, int64_t *r, int64_t *y, int32_t *k, long n) {
  for (long i = 0; i < n; i++) {
    k[i] = vmc::root_shift(s[i]);
    const int64_t t = s[i] << (2 * k[i]);
    float f = vmc::root_first(t);
    for (int u = 0; u < (ulps < 0 ? -ulps : ulps); u++) f = nextafterf(f, ulps < 0 ? 0.0f : 1e30f);
    const vmc::Root60 q = vmc::root_refined(t, k[i], f);
    r[i] = q.r;
    y[i] = q.y;
  }
}
extern "C" int log_size() { return (int)sizeof(vmc::LogEntry); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed64")
    (d / "f.cpp").write_text(SOURCE)
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "valomc_gb300", "csrc"),
                    str(d / "f.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def test_logarithm_table_is_aligned_for_its_loads(lib):
    """The device reads an entry with one 16-byte load."""
    assert lib.log_align() == 16 and lib.log_size() == 16


ONE = 2 ** 60


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("ulps", [-1, 0, 1])  # CUDA's reciprocal: one ulp
def test_reciprocal_from_the_first_value_of_the_device(lib, ulps):
    rng = np.random.default_rng(71)
    d = np.concatenate([np.uint64(2 ** 63) + np.arange(3000, dtype=np.uint64) * np.uint64(2 ** 30),
                        np.uint64(2 ** 64 - 1) - np.arange(3000, dtype=np.uint64) * np.uint64(2 ** 30),
                        rng.integers(2 ** 63, 2 ** 64, 100000, dtype=np.uint64)])
    y = np.empty(len(d), np.uint64)
    lib.rcp(ptr(d), ulps, ptr(y), C.c_long(len(d)))
    for a, b in zip(d.tolist(), y.tolist()):
        assert abs(b * a - (1 << 125)) < 7 * a  # as with an exact first value: e^3 < 2^-63


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])  # CUDA's reciprocal root: two ulps
def test_root_from_the_first_value_of_the_device(lib, ulps):
    if np.finfo(np.longdouble).eps > 2e-19:
        pytest.skip("long double is no wider than double here")
    rng = np.random.default_rng(72)
    s = np.concatenate([ONE - np.arange(3000), ONE - np.arange(3000) * 2 ** 40, ONE // 4 + np.arange(3000) * 2 ** 30,
                        rng.integers(1, ONE, 100000), (ONE * 10.0 ** rng.uniform(-15, 0, 20000)).astype(np.int64) + 1])
    s = s.astype(np.int64)
    s = s[(s > 0) & (s <= ONE)]
    r, y, k = np.empty(len(s), np.int64), np.empty(len(s), np.int64), np.empty(len(s), np.int32)
    lib.root(ptr(s), ulps, ptr(r), ptr(y), ptr(k), C.c_long(len(s)))
    t = s.astype(np.longdouble) / ONE * np.longdouble(4) ** k
    # the bounds of an exact first value: e^3 < 2^-60
    assert np.max(np.abs(r / np.longdouble(ONE) - np.sqrt(t))) < 10 / np.longdouble(ONE)
    assert np.max(np.abs(y / np.longdouble(ONE) - 1 / np.sqrt(t))) < 18 / np.longdouble(ONE)
