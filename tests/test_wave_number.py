"""The wave number per turn that the plain FP64 walks advance their phase by (csrc/host_setup.cpp,
compiled for the host): as near to f n / c as a double can be."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "host_setup.hpp"
extern "C" double turns_per_mm(double f) {
  // a triangle whose first edge emits
  static const int64_t H[3] = {0, 1, 2}, BH[6] = {0, 1, 2, 1, 2, 0};
  static const double r[6] = {0, 1, 0, 0, 0, 1}, one[3] = {1, 1, 1};
  vmc_input in{};
  in.dim = 2; in.Ne = 1; in.Nb = 3; in.Nr = 3;
  in.H = H; in.BH = BH; in.r = r;
  in.mua = in.mus = in.g = in.n = one;
  in.n_mua = in.n_mus = in.n_g = in.n_n = 1;
  in.BCType = "caa"; in.n_BCType = 3;
  in.BCn = one; in.n_BCn = 3;
  in.f = f; in.Nphoton = 1;
  vmc::HostMesh m;
  vmc::HostJob j;
  if (vmc::build_mesh(&in, 1, m, true) || vmc::build_job(&in, m, j)) return -1.0;
  return j.k_turn;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("wave")
    (d / "f.cpp").write_text(SOURCE)
    csrc = os.path.join(ROOT, "valomc_gb300", "csrc")
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fopenmp", "-ffp-contract=off", "-I" + csrc,
                    "-I" + os.path.join(ROOT, "include"), str(d / "f.cpp"), os.path.join(csrc, "host_setup.cpp"), "-o", so],
                   check=True)
    L = C.CDLL(so)
    L.turns_per_mm.restype, L.turns_per_mm.argtypes = C.c_double, [C.c_double]
    return L


@pytest.mark.parametrize("f", [100e6, 73e6, 1.5e8, 37e6, 1.0, 3.3e9])
def test_turns_per_millimetre(lib, f):
    got = Fraction(lib.turns_per_mm(f))
    want = Fraction(f) / Fraction(299792458000)  # mm/s
    assert abs(got / want - 1) <= Fraction(1, 2 ** 53)
