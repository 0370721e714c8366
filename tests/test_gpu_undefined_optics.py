"""Elements whose optics are no numbers: the plain FP64 walks do there what the reference does."""
import numpy as np
import pytest

import oracle
import valomc_gb300 as V
from golden.make_golden import cases

pytestmark = pytest.mark.gpu


def few(p, field, seed):
    """p with one element in fifty of field `field` undefined (a few percent of the faces: the plain
    walk), and sources into some of them"""
    x = getattr(p, field).copy()
    x[np.random.default_rng(seed).random(p.Ne) < 0.02] = np.nan
    return p.copy(**{field: x})


@pytest.mark.parametrize("field", ["mus", "n", "g", "mua"])
@pytest.mark.parametrize("name", ["jitter3d", "circles2d"])
def test_undefined_optics_in_some_elements(built, name, field):
    p = cases()[name][0].copy(Nphoton=2000)
    # optics of one medium, so that what changes across faces is the undefined elements alone
    p = few(p.copy(mus=np.full(p.Ne, 1.3), n=np.full(p.Ne, 1.3), g=np.full(p.Ne, 0.6)), field, 4)
    want = oracle.run(p, rng=oracle.RNG_PHILOX, normalize=False)
    got = V.run(p, precision=V.VMC_FP64, normalize=False)
    assert got.stats["steps"] == want.steps and got.stats["loss"] == want.loss
    for k in ("ER", "EBR"):
        a, b = getattr(got, k), np.asarray(getattr(want, k))
        assert np.array_equal(np.isnan(a), np.isnan(b)), k
        np.testing.assert_allclose(np.nan_to_num(a), np.nan_to_num(b), rtol=1e-7, atol=1e-7, err_msg=k)


@pytest.mark.parametrize("name", ["jitter3d", "circles2d"])
def test_an_undefined_index_around_the_source(built, name):
    """Photons that start in a corner of an undefined index are lost where they first leave an element."""
    p = cases()[name][0].copy(Nphoton=2000)
    lo, hi = p.r.min(axis=0), p.r.max(axis=0)
    corner = lambda x: np.all((x - lo) / (hi - lo) < 0.26, axis=1)
    inside, lit = corner(p.r[p.H].mean(axis=1)), corner(p.r[p.BH].mean(axis=1))
    assert 0.01 < inside.mean() < 0.1 and lit.any()  # few of the faces: the plain walk
    p = p.copy(mus=np.full(p.Ne, 1.3), n=np.where(inside, np.nan, 1.3), g=np.full(p.Ne, 0.6),
               BCType=np.where(lit, ord("c"), ord("a")).astype(np.uint8))
    want = oracle.run(p, rng=oracle.RNG_PHILOX, normalize=False)
    got = V.run(p, precision=V.VMC_FP64, normalize=False)
    assert want.loss > p.Nphoton / 2
    assert got.stats["steps"] == want.steps and got.stats["loss"] == want.loss
    np.testing.assert_allclose(got.EBR, want.EBR, rtol=1e-7, atol=1e-7)
