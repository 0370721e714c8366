"""Results written over the arrays that the job was given."""
import ctypes as C

import numpy as np
import pytest

import valomc_gb300 as V
from golden.make_golden import cases
from valomc_gb300 import api

pytestmark = pytest.mark.gpu
KEYS = ("ER", "EI", "EBR", "EBI", "DEBR", "DEBI")


def over(m, out, arrays, fields):
    """Points results of `out` at the optics arrays of `m`."""
    for k, nm in fields.items():
        a = np.ctypeslib.as_array(getattr(m.s, nm), shape=(len(arrays[k]),))
        setattr(out, k, api._ptr(a))
        arrays[k] = a


@pytest.mark.parametrize("name", ["jitter3d", "mixed3d", "mixed3d_fd", "mixed2d_fd", "square2d"])
@pytest.mark.parametrize("fields", [{"ER": "mua"}, {"ER": "n", "EI": "mua"}, {"EI": "mua"}])
def test_results_over_the_optics(built, name, fields):
    p = cases()[name][0].copy(Nphoton=1500)
    want = V.run(p)
    m = api._Marshal(p)
    out, arr, _ = api._outputs(p.Ne, p.Nb, p.dim, False)
    over(m, out, arr, fields)
    st, o = api.VmcStats(), api.options()
    assert V.lib().vmc_run(C.byref(m.s), C.byref(o), C.byref(out), C.byref(st)) == 0
    for k in KEYS:
        np.testing.assert_allclose(arr[k], getattr(want, k), rtol=1e-9, atol=1e-12)
    if p.f == 0.0:
        assert abs(st.ledger[1] - want.stats["ledger"]["absorbed"]) < 1e-6


def test_results_of_one_job_over_the_optics_of_another(built):
    """A continuous-wave job's results over the arrays of a modulated one, which is launched after it."""
    p, q = (cases()[n][0].copy(Nphoton=1500) for n in ("mixed3d", "mixed3d_fd"))
    mesh = V.Mesh(p)
    want, _ = V.run_batch([mesh, mesh], [p, q])
    ms = [api._Marshal(x, geometry=False) for x in (p, q)]
    pairs = [api._outputs(p.Ne, p.Nb, 3, False)[:2] for _ in ms]
    over(ms[1], pairs[0][0], pairs[0][1], {"ER": "mua", "EI": "mus"})
    jobs = (api.VmcInput * 2)(*[m.s for m in ms])
    outs = (api.VmcOutput * 2)(*[o for o, _ in pairs])
    hs = (C.c_void_p * 2)(mesh.h, mesh.h)
    st, o = api.VmcStats(), api.options()
    assert V.lib().vmc_run_batch(hs, jobs, 2, C.byref(o), outs, C.byref(st), None) == 0
    for (_, arr), w in zip(pairs, want):
        for k in KEYS:
            np.testing.assert_allclose(arr[k], getattr(w, k), rtol=1e-9, atol=1e-12)
    mesh.close()
