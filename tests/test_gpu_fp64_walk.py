"""The plain FP64 walk's choice of the exit face, on meshes where its FP32 half cannot serve (tiny
elements), has little to go by (large coordinates, slivers) or is exact, against the oracle on the
same Philox streams."""
import os
import sys

import numpy as np
import pytest

import valomc_gb300 as V
from valomc_gb300 import meshgen as mg

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def problem(dim, shape, inclusion, f):
    rng = np.random.default_rng(5)
    if dim == 3:
        r, H, BH = mg.box_mesh_3d(6, 5, 4)
    else:
        r, H, BH = mg.rectangular_mesh(7, 6, 1)
    r = r.astype(float)
    size = 1.0
    if shape == "slivers":  # interior nodes moved: thin elements, no grid-aligned faces
        lo, hi = r.min(0), r.max(0)
        inner = np.all((r > lo + 1e-9) & (r < hi - 1e-9), axis=1)
        r[inner] += rng.uniform(-0.3, 0.3, (int(inner.sum()), dim))
    elif shape == "far":
        r += 1e5
    elif shape in ("tiny", "huge"):
        size = 1e-6 if shape == "tiny" else 1e6
        r *= size
    ne, nb = len(H), len(BH)
    cen, mid = r[H].mean(1), r[BH].mean(1)
    inside = np.linalg.norm((cen - r.mean(0)) / size, axis=1) < (0.9 if inclusion else 0.0)
    types = np.full(nb, ord("a"), np.uint8)
    types[np.abs(mid[:, -1] - r[:, -1].min()) < 1e-7 * size] = ord("c")
    return mg.Problem(dim=dim, H=H, BH=BH, r=r, mua=np.where(inside, 0.2, 0.05) / size,
                      mus=np.where(inside, 1.0, 3.0) / size, g=np.where(inside, 0.0, 0.8), n=np.where(inside, 1.5, 1.35),
                      BCType=types, BCn=np.ones(nb), Nphoton=3000, seed=99, f=f / size, phase0=3.0 if f else 0.0)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("shape,inclusion,f", [("grid", False, 0.0), ("grid", True, 1e9), ("slivers", True, 0.0),
                                               ("slivers", False, 1e9), ("far", True, 0.0), ("tiny", True, 1e9),
                                               ("huge", True, 0.0)])
def test_walk_matches_the_oracle(built, dim, shape, inclusion, f):
    p = problem(dim, shape, inclusion, f)
    gpu = V.run(p, precision=V.VMC_FP64)
    ref = oracle.run(p, rng=oracle.RNG_PHILOX, nthreads=4)
    assert gpu.stats["photons_done"] == p.Nphoton and gpu.stats["loss"] == ref.loss
    # a position holds 53 bits of its coordinate: at 1e5 an element's exit may turn on 1e-11
    slack = 1e-3 if shape == "far" else 0.0
    assert abs(gpu.stats["steps"] - ref.steps) <= slack * ref.steps
    for k in ("ER", "EI", "EBR", "EBI", "DEBR", "DEBI"):
        a, b = getattr(gpu, k), getattr(ref, k)
        assert np.abs(a - b).sum() <= (1e-2 if shape == "far" else 1e-6) * np.abs(b).sum(), k


@pytest.mark.parametrize("dim", [2, 3])
def test_jobs_of_both_fp64_walks_share_a_batch(built, dim):
    """Optics drawn per element take the literal walk, uniform ones the other: a batch of both
    equals single runs, and each the oracle."""
    p = problem(dim, "slivers", False, 0.0)
    rng = np.random.default_rng(6)
    rough = p.copy(mus=rng.uniform(2.0, 4.0, p.Ne), seed=7)
    mesh = V.Mesh(p, precision=V.VMC_FP64)
    res, _ = V.run_batch([mesh, mesh], [p, rough], precision=V.VMC_FP64)
    for q, r in zip((p, rough), res):
        one = V.run(q, precision=V.VMC_FP64)
        ref = oracle.run(q, rng=oracle.RNG_PHILOX, nthreads=4)
        for k in ("ER", "EBR"):
            np.testing.assert_allclose(getattr(r, k), getattr(one, k), rtol=1e-9, atol=1e-15)
            a, b = getattr(r, k), getattr(ref, k)
            assert np.abs(a - b).sum() <= 1e-6 * np.abs(b).sum(), k
    mesh.close()


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("g", [0.02, -0.9, 0.9995, -0.9995])
def test_scattering_angles_at_the_ends_of_fixed_point(built, dim, g):
    """|g| above 0.999 leaves the fixed-point angles for FP64 ones."""
    p = problem(dim, "slivers", False, 0.0)
    p.g[:] = g
    gpu = V.run(p, precision=V.VMC_FP64)
    ref = oracle.run(p, rng=oracle.RNG_PHILOX, nthreads=4)
    assert gpu.stats["photons_done"] == p.Nphoton and gpu.stats["loss"] == ref.loss
    assert gpu.stats["steps"] == ref.steps
    for k in ("ER", "EBR"):
        a, b = getattr(gpu, k), getattr(ref, k)
        assert np.abs(a - b).sum() <= 1e-6 * np.abs(b).sum(), k


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("source", ["c", "i"])
@pytest.mark.parametrize("n_out", [1.35, 1.0, 1.36, 0.2, 6.0])
def test_interfaces_and_launches(built, dim, source, n_out):
    """The choice at an interface in FP32, where it is certain (index ratios of 1/4 to 4), and in
    FP64 elsewhere; the launches' directions."""
    p = problem(dim, "slivers", True, 0.0)
    p.BCn[:] = n_out
    p.BCType[p.BCType == ord("c")] = ord(source)
    gpu = V.run(p, precision=V.VMC_FP64)
    ref = oracle.run(p, rng=oracle.RNG_PHILOX, nthreads=4)
    assert gpu.stats["photons_done"] == p.Nphoton and gpu.stats["loss"] == ref.loss
    assert gpu.stats["steps"] == ref.steps
    for k in ("ER", "EBR", "DEBR"):
        a, b = getattr(gpu, k), getattr(ref, k)
        assert np.abs(a - b).sum() <= 1e-6 * np.abs(b).sum(), k


@pytest.mark.parametrize("sigma", [0.02, 0.2, 1.0, 5.0, 100.0])
def test_gaussian_launch_angles(built, sigma):
    """The bisection's halvings are decided by the inverse error function where it is certain."""
    p = problem(2, "slivers", False, 0.0)
    p.BCType[p.BCType == ord("c")] = ord("g")
    p.GaussianSigma = np.full(p.Nb, sigma)
    gpu = V.run(p, precision=V.VMC_FP64)
    ref = oracle.run(p, rng=oracle.RNG_PHILOX, nthreads=4)
    assert (gpu.stats["steps"], gpu.stats["loss"]) == (ref.steps, ref.loss)
    for k in ("ER", "EBR", "DEBR"):
        a, b = getattr(gpu, k), getattr(ref, k)
        assert np.abs(a - b).sum() <= 1e-6 * np.abs(b).sum(), k
