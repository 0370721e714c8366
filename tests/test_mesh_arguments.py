"""vmc_mesh_create refuses a geometry whose sizes make no sense before anything reads its arrays."""
import ctypes as C

import pytest

import valomc_gb300 as V
from golden.make_golden import cases
from valomc_gb300 import api

INVALID = 32


@pytest.mark.parametrize("field,value", [("dim", 0), ("dim", 1), ("dim", 4), ("Ne", -1), ("Nb", -1), ("Nr", -5)])
def test_sizes_of_a_geometry(built, field, value):
    m = api._Marshal(cases()["square2d"][0])
    assert V.lib().vmc_status_string(INVALID) == b"invalid argument"
    if field == "dim" and value > 1:  # room for the columns that a reader would expect
        m = api._Marshal(cases()["jitter3d"][0])
        m.s.Ne, m.s.Nb, m.s.Nr = 8, 8, 8
    setattr(m.s, field, value)
    h = C.c_void_p()
    assert V.lib().vmc_mesh_create(C.byref(m.s), V.VMC_FP64, 0, C.byref(h)) == INVALID
    assert not h.value
