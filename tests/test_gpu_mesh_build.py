"""Meshes from 1,000 elements have neighbours and records made on the device: the same ones as the
host's, in neighbours, errors and walks."""
import numpy as np
import pytest

import valomc_gb300 as V
from valomc_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu
DEVICE_FROM = 1000


def jittered(dim, n, origin, seed):
    if dim == 3:
        r, H, BH = mg.box_mesh_3d(n, n, n)
    else:
        r, H, BH = mg.rectangular_mesh(n, n, 1)
    r = r.astype(float)
    lo, hi = r.min(0), r.max(0)
    inner = np.all((r > lo + 1e-9) & (r < hi - 1e-9), axis=1)
    r[inner] += np.random.default_rng(seed).uniform(-0.2, 0.2, (int(inner.sum()), dim))
    return r + origin, H, BH


def problem(dim, extra=0):
    """A mesh below the limit; a second body apart from it, of `extra` cells a side, whose elements,
    nodes and faces come after its own, puts it above."""
    r, H, BH = jittered(dim, 5 if dim == 3 else 20, 0.0, 1)
    ne, nb = len(H), len(BH)
    if extra:
        r2, H2, BH2 = jittered(dim, extra, 500.0, 2)
        H, BH, r = np.vstack([H, H2 + len(r)]), np.vstack([BH, BH2 + len(r)]), np.vstack([r, r2])
    assert (len(H) >= DEVICE_FROM) == (extra > 0)
    types = np.full(len(BH), ord("a"), np.uint8)
    mid = r[BH].mean(1)
    types[:nb][np.abs(mid[:nb, -1] - r[:, -1].min()) < 1e-7] = ord("c")
    el = np.arange(len(H))
    return mg.Problem(dim=dim, H=H, BH=BH, r=r, mua=0.02 + 0.01 * (el % 3), mus=np.full(len(H), 2.0),
                      g=np.full(len(H), 0.7), n=np.where(el % 32 < 1, 1.45, 1.37), BCType=types, BCn=np.ones(len(BH)),
                      Nphoton=20000, seed=5), ne, nb


@pytest.mark.parametrize("precision", [V.VMC_FP64, V.VMC_FP32])
# extra bodies with fewer nodes than the 1024 threads of the scan, and with many more
@pytest.mark.parametrize("dim,extra", [(2, 15), (2, 80), (3, 4), (3, 20)])
def test_same_neighbours_and_walks_as_the_hosts(built, dim, extra, precision):
    small, ne, nb = problem(dim)
    large, _, _ = problem(dim, extra)
    a = V.run(small, precision=precision)
    b = V.run(large, precision=precision, want_hn=True)
    np.testing.assert_array_equal(b.HN, V.build_neighbourhood(large)[1])
    assert (a.stats["steps"], a.stats["scatters"]) == (b.stats["steps"], b.stats["scatters"])
    mesh = V.Mesh(large, precision=precision)
    given = large.copy()
    given.HN = b.HN
    res, _ = V.run_batch([mesh], [large], precision=precision)
    mesh.close()
    for r in (b, res[0], V.run(given, precision=precision)):
        for k, cut in (("ER", ne), ("EBR", nb)):
            x, y = getattr(a, k), getattr(r, k)
            # the same deposits, added in another order; the totals they are normalised by are sums too
            np.testing.assert_allclose(y[:cut], x, rtol=1e-9, atol=1e-15 * np.abs(x).max())
            assert not y[cut:].any()


@pytest.mark.parametrize("dim", [2, 3])
def test_same_errors_as_the_hosts(built, dim):
    p, _, _ = problem(dim, 15 if dim == 2 else 4)
    twice = p.copy(H=np.vstack([p.H, p.H[7:8]]))  # a second element on the faces of element 7
    for k in ("mua", "mus", "g", "n"):
        setattr(twice, k, np.append(getattr(p, k), getattr(p, k)[7]))
    cases = [twice]
    bare = p.copy(BH=p.BH[1:], BCType=p.BCType[1:], BCn=p.BCn[1:])  # a face without its boundary element
    if dim == 2:
        cases.append(bare)
    for q in cases:
        status, _ = V.build_neighbourhood(q)
        with pytest.raises(V.VmcError) as run:
            V.run(q)
        with pytest.raises(V.VmcError) as mesh:
            V.Mesh(q)
        assert status and run.value.status == mesh.value.status == status
    if dim == 3:
        np.testing.assert_array_equal(V.run(bare, want_hn=True).HN, V.build_neighbourhood(bare)[1])
