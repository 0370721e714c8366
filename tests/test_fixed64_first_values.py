"""The fixed-point functions of the plain FP64 walks with the device's own operands: the alignment of
its table loads."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "fixed64.hpp"
extern "C" int log_align() { return (int)alignof(vmc::LogEntry); }
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
