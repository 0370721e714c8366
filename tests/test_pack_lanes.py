"""Where the photons of a CTA go when its lanes are packed (csrc/vmc_types.hpp, compiled for the
host): every photon to a thread of its own, for each block size and each count of live photons."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "vmc_types.hpp"
extern "C" int warps_for(int all, int warps) { return vmc::pack_warps(all, warps); }
extern "C" void targets(int all, int warps, int turn, int *to) {
  const int want = vmc::pack_warps(all, warps);
  for (int k = 0; k < all; k++) to[k] = vmc::pack_thread(k, all, want, turn, warps);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pack")
    (d / "f.cpp").write_text(SOURCE)
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "valomc_gb300", "csrc"),
                    str(d / "f.cpp"), "-o", so], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("warps", range(1, 9))
def test_every_photon_has_a_thread_of_its_own(lib, warps):
    for n in range(1, 32 * warps + 1):
        want = lib.warps_for(n, warps)
        assert (n + 31) // 32 <= want <= min(warps, max(n, 1))
        for turn in range(warps):
            to = (C.c_int * n)()
            lib.targets(n, warps, turn, to)
            got = list(to)
            assert len(set(got)) == n, (n, turn)
            assert 0 <= min(got) and max(got) < 32 * warps, (n, turn)
            assert len({t // 32 for t in got}) <= want
