"""Batched launches, the serving loop, cancellation / timeout, progress, and the drop-in
executables, on the GPU through the C ABI."""
import os
import subprocess
import tempfile
import threading
import time

import numpy as np
import pytest

import valomc_gb300 as V
from golden.make_golden import cases
from valomc_gb300 import build as vbuild
from valomc_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu
RTOL = 1e-9  # same photons, same draws: only the order of the FP64 atomic additions differs


def small_jobs():
    c = cases()
    jobs = [c["phantom3d"][0].copy(Nphoton=30000, seed=21), c["pencil3d"][0].copy(Nphoton=20000, seed=22),
            mg.pencil_box(10, 0.03, 8.0, 0.9, 1.37, (4.3, 5.2), 25000, seed=23),
            mg.pencil_box(14, 0.08, 15.0, 0.85, 1.41, (6.6, 2.3), 15000, seed=24)]
    return jobs


@pytest.mark.parametrize("precision", [V.VMC_FP64, V.VMC_FP32])
def test_batch_equals_individual_runs(built, precision):
    jobs = small_jobs()
    meshes = [V.Mesh(p, precision=precision) for p in jobs]
    res, tot = V.run_batch(meshes, jobs, precision=precision)
    assert tot["photons_done"] == sum(p.Nphoton for p in jobs)
    for p, r in zip(jobs, res):
        one = V.run(p, precision=precision)
        np.testing.assert_allclose(r.ER, one.ER, rtol=RTOL, atol=1e-300)
        np.testing.assert_allclose(r.EBR, one.EBR, rtol=RTOL, atol=1e-300)
        assert r.stats["steps"] == one.stats["steps"] > 0  # per-job step counts
    assert sum(r.stats["steps"] for r in res) == tot["steps"]


@pytest.mark.parametrize("use_graph", [False, True])
def test_calls_from_two_threads_overlap_and_equal_sequential_runs(built, use_graph):
    # each call runs on a stream of its own; ctypes drops the GIL for the call
    jobs = small_jobs()[:2]
    opts = V.options(use_graph=use_graph)
    seq = [V.run(p, precision=V.VMC_FP32, opts=opts) for p in jobs]
    out = [None, None]
    errs = []

    def work(i):
        try:
            out[i] = [V.run(jobs[i], precision=V.VMC_FP32, opts=opts) for _ in range(3)]
        except Exception as e:  # noqa: BLE001 -- reported below
            errs.append(e)

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join(timeout=300)
    assert not errs and all(o is not None for o in out)
    for i in range(2):
        for r in out[i]:
            np.testing.assert_allclose(r.ER, seq[i].ER, rtol=RTOL, atol=1e-300)
            np.testing.assert_allclose(r.DEBR, seq[i].DEBR, rtol=RTOL, atol=1e-300)
            assert r.stats["steps"] == seq[i].stats["steps"]


@pytest.mark.parametrize("precision", [V.VMC_FP64, V.VMC_FP32])
def test_zero_photon_jobs(built, precision):
    """An empty run launches nothing and normalises to NaN as the reference does; an empty
    job inside a batch leaves the others as they are alone."""
    p = cases()["square2d"][0]
    r = V.run(p, precision=precision, nphoton=0)
    assert r.stats["photons_done"] == 0 and r.stats["steps"] == 0
    assert np.isnan(r.ER).all() and np.isnan(r.EBR).all()
    raw = V.run(p, precision=precision, nphoton=0, normalize=False)
    assert not raw.ER.any() and not raw.EBR.any()
    # a negative count runs no photon and divides by itself, as MonteCarlo does: -0.0
    neg = V.run(p, precision=precision, nphoton=-5)
    assert neg.stats["photons_done"] == 0 and not neg.ER.any() and np.signbit(neg.ER).all()
    jobs = small_jobs()[:2]
    jobs = [jobs[0].copy(Nphoton=0), jobs[1]]
    meshes = [V.Mesh(q, precision=precision) for q in jobs]
    res, tot = V.run_batch(meshes, jobs, precision=precision)
    assert tot["photons_done"] == jobs[1].Nphoton
    assert np.isnan(res[0].ER).all()
    one = V.run(jobs[1], precision=precision)
    np.testing.assert_allclose(res[1].ER, one.ER, rtol=RTOL, atol=1e-300)


def test_batch_through_a_cuda_graph_equals_the_plain_launch(built):
    jobs = small_jobs()
    meshes = [V.Mesh(p) for p in jobs]
    plain, _ = V.run_batch(meshes, jobs)
    for _ in range(2):  # the second launch updates the instantiated graph in place
        g, tot = V.run_batch(meshes, jobs, opts=V.options(use_graph=True))
        assert tot["photons_done"] == sum(p.Nphoton for p in jobs)
        for a, b in zip(plain, g):
            np.testing.assert_allclose(b.ER, a.ER, rtol=RTOL, atol=1e-300)


def staging_case(name):
    if name == "box5":  # 750 tets, 300 boundary triangles: the whole set fits a CTA's stage
        return mg.pencil_box(5, 0.05, 6.0, 0.9, 1.4, (2.2, 2.9), 50000, seed=31)
    return cases()[name][0].copy(Nphoton=50000, seed=31)


@pytest.mark.parametrize("precision", [V.VMC_FP64, V.VMC_FP32])
@pytest.mark.parametrize("slots", [64, 2048, 0])
@pytest.mark.parametrize("name", ["phantom3d", "box5", "square2d", "mixed2d_fd"])
def test_shared_memory_staging_equals_global_atomics(built, slots, name, precision):
    # slots > 0: hashed element table (3D FP32 continuous wave); 0: the whole accumulator set
    # of a small mesh; -1: global reductions only
    if precision == V.VMC_FP64 and slots != 0:
        pytest.skip("the hashed table is a tracking-form option")
    p = staging_case(name)
    mesh = V.Mesh(p, precision=precision)
    o = dict(precision=precision)
    plain, _ = V.run_batch([mesh], [p], opts=V.options(stage_slots=-1, **o))
    staged, _ = V.run_batch([mesh], [p], opts=V.options(stage_slots=slots, **o))
    for k in ("ER", "EI", "EBR", "EBI", "DEBR", "DEBI"):
        np.testing.assert_allclose(getattr(staged[0], k), getattr(plain[0], k), rtol=RTOL, atol=1e-300, err_msg=k)
    assert staged[0].stats["steps"] == plain[0].stats["steps"]


@pytest.mark.parametrize("name", ["square2d", "phantom3d"])
def test_refill_threshold_leaves_results_unchanged(built, name):
    # a photon's draws depend on its index only, so launching idle lanes one at a time or in
    # groups changes nothing but the order of the FP64 additions
    p = cases()[name][0].copy(Nphoton=40000, seed=41)
    ref = V.run(p, opts=V.options(refill_lanes=1))
    for k in (4, 32):
        r = V.run(p, opts=V.options(refill_lanes=k))
        np.testing.assert_allclose(r.ER, ref.ER, rtol=RTOL, atol=1e-300)
        np.testing.assert_allclose(r.EBR, ref.EBR, rtol=RTOL, atol=1e-300)
        assert r.stats["steps"] == ref.stats["steps"] and r.stats["photons_done"] == p.Nphoton


def test_autotuner_returns_a_valid_shape(built):
    jobs = small_jobs()
    meshes = [V.Mesh(p) for p in jobs]
    o = V.autotune(meshes, jobs, budget_s=1.0)
    assert o.block_size in (64, 128, 256) and o.fetch_chunk in (32, 64, 128)
    res, _ = V.run_batch(meshes, jobs, opts=o)
    assert all(r.ER.sum() > 0 for r in res)


@pytest.mark.parametrize("precision", [V.VMC_FP64, V.VMC_FP32])
def test_server_result_alone_equals_result_in_the_mix(built, precision):
    jobs = small_jobs()
    meshes = [V.Mesh(p, precision=precision) for p in jobs]
    # alone: one request at a time, small epochs so requests are sliced across launches
    srv = V.Server(precision=precision, max_slots=8, memory_budget=1 << 30, epoch_photons=7000)
    ids = [srv.add_mesh(m) for m in meshes]
    alone = []
    for k, p in enumerate(jobs):
        rid = srv.submit(ids[k], p)
        alone.append(srv.wait(rid))
    # mixed: everything in flight together, submitted while others run
    rids = [srv.submit(ids[k], p) for k, p in enumerate(jobs)]
    mixed = [srv.wait(r) for r in rids]
    srv.close()
    for p, a, m in zip(jobs, alone, mixed):
        one = V.run(p, precision=precision)
        np.testing.assert_allclose(a.ER, m.ER, rtol=RTOL, atol=1e-300)
        np.testing.assert_allclose(a.ER, one.ER, rtol=RTOL, atol=1e-300)
        np.testing.assert_allclose(m.EBR, one.EBR, rtol=RTOL, atol=1e-300)
        assert m.stats["photons_done"] == p.Nphoton
        assert a.stats["steps"] == m.stats["steps"] == one.stats["steps"]


def test_server_default_epochs_keep_each_result(built):
    """Epochs sized by the backlog and water-filled slices (the server's defaults): requests
    of very different sizes submitted together each equal their run alone."""
    jobs = small_jobs()
    sizes = [400, 60000, 3000, 25000]
    meshes = [V.Mesh(p) for p in jobs]
    srv = V.Server(max_slots=8, memory_budget=1 << 30)
    ids = [srv.add_mesh(m) for m in meshes]
    rids = [srv.submit(ids[k], p, nphoton=n) for k, (p, n) in enumerate(zip(jobs, sizes))]
    res = [srv.wait(r, timeout_s=120) for r in rids]
    srv.close()
    for p, n, r in zip(jobs, sizes, res):
        one = V.run(p, nphoton=n)
        assert r.stats["photons_done"] == n and r.stats["steps"] == one.stats["steps"]
        np.testing.assert_allclose(r.ER, one.ER, rtol=RTOL, atol=1e-300)
        np.testing.assert_allclose(r.EBR, one.EBR, rtol=RTOL, atol=1e-300)


def test_server_admission_by_memory_footprint(built):
    p = cases()["phantom3d"][0]
    mesh = V.Mesh(p)
    srv = V.Server(max_slots=4, memory_budget=200_000)  # smaller than one request's state
    mid = srv.add_mesh(mesh)
    rid = srv.submit(mid, p, nphoton=1000)
    with pytest.raises(V.VmcError) as e:
        srv.wait(rid, timeout_s=30)
    assert e.value.status == 39  # VMC_ERR_ADMISSION
    srv.close()


def test_server_releases_memory_of_finished_requests(built):
    """A budget that holds one request at a time: every request is admitted in turn, so the
    memory of finished requests (returned to the server's pool) is accounted back."""
    p = cases()["phantom3d"][0]
    mesh = V.Mesh(p)
    one = V.run(p, nphoton=3000, seed=5)
    srv = V.Server(max_slots=4, memory_budget=900_000)  # one request's state (~0.6 MB) fits, two do not
    mid = srv.add_mesh(mesh)
    rids = [srv.submit(mid, p, nphoton=3000, seed=5) for _ in range(6)]
    res = [srv.wait(r, timeout_s=120) for r in rids]
    srv.close()
    for r in res:
        assert r is not None and r.stats["photons_done"] == 3000
        np.testing.assert_allclose(r.ER, one.ER, rtol=RTOL, atol=1e-300)


def test_server_poll_before_finish(built):
    p = mg.config_3d_phantom(nphoton=1, seed=2)
    mesh = V.Mesh(p)
    srv = V.Server(max_slots=4, memory_budget=1 << 30)
    mid = srv.add_mesh(mesh)
    rid = srv.submit(mid, p, nphoton=5_000_000)
    assert srv.poll(rid) is None
    r = srv.wait(rid, timeout_s=120)
    assert r is not None and r.stats["photons_done"] == 5_000_000
    assert r.stats["seconds_total"] >= r.stats["seconds_kernel"] > 0
    srv.close()


def test_timeout_stops_the_kernel_and_the_context_stays_usable(built):
    p = mg.config_3d_phantom(nphoton=2_000_000_000, seed=3)
    t0 = time.time()
    r = V.run(p, check=False, timeout_s=0.5)
    assert r.stats["status"] == 37  # VMC_ERR_TIMEOUT
    assert time.time() - t0 < 30
    assert 0 < r.stats["photons_done"] < p.Nphoton
    ok = V.run(cases()["phantom3d"][0], nphoton=1000)
    assert ok.stats["photons_done"] == 1000


def test_cancel_flag_and_progress_callback(built):
    p = mg.config_3d_phantom(nphoton=2_000_000_000, seed=4)
    flag = np.zeros(1, np.int32)
    threading.Timer(0.4, lambda: flag.__setitem__(0, 1)).start()
    r = V.run(p, check=False, cancel=flag)
    assert r.stats["status"] == 36  # VMC_ERR_CANCELLED
    seen = []

    def prog(pct):
        seen.append(pct)
        return len(seen) < 3  # abort at the third report, like the MEX waitbar's cancel

    r = V.run(p, check=False, progress=prog)
    assert r.stats["status"] == 36 and len(seen) == 3
    assert all(0 <= s <= 100 for s in seen)


@pytest.mark.parametrize("dim", [3, 2])
def test_executable_writes_the_reference_format(built, dim):
    p = cases()["phantom3d" if dim == 3 else "square2d"][0].copy(Nphoton=20000, seed=77)
    exe = os.path.join(vbuild.BUILD, f"MC{dim}D")
    with tempfile.TemporaryDirectory() as td:
        fin, fout = os.path.join(td, "in.txt"), os.path.join(td, "out.txt")
        mg.write_input(fin, p)
        res = subprocess.run([exe, fin, fout] + (["-s"] if dim == 2 else []), capture_output=True, text=True,
                             timeout=300)
        assert res.returncode == 0, res.stdout + res.stderr
        assert "Computation took" in res.stdout
        lines = open(fout).read().splitlines()
    assert len(lines) == 1 + p.Ne + p.Nb
    assert lines[0].endswith(" 0")
    if dim == 3:
        assert len(lines[1]) == 37  # "%18.10e %18.10e"
    vals = np.array([[float(x) for x in ln.split()] for ln in lines[1:]])
    one = V.run(p)
    rt = 1e-9 if dim == 3 else 1e-5
    np.testing.assert_allclose(vals[:p.Ne, 0], one.ER, rtol=rt, atol=1e-300)
    np.testing.assert_allclose(vals[p.Ne:, 0], one.EBR, rtol=rt, atol=1e-300)


@pytest.mark.parametrize("name,cap", [("phantom3d", 1), ("phantom3d", 60), ("phantom3d_fd", 60), ("mixed3d", 9),
                                      ("square2d", 1), ("square2d", 13)])
def test_step_limit_of_the_tracking_form(built, name, cap):
    """Photons at the step limit are lost with the weight they have then: no walk is longer, the
    ledger closes, and a limit that no walk reaches changes nothing.  One-job and per-job forms."""
    p = cases()[name][0].copy(Nphoton=4000)
    free = V.run(p, normalize=False)
    out = V.run(p, normalize=False, max_steps=cap)
    assert free.stats["capped"] == 0 and 0 < out.stats["capped"] <= p.Nphoton
    assert out.stats["steps"] <= cap * p.Nphoton
    assert out.stats["steps"] >= cap * out.stats["capped"]
    if p.f == 0.0:
        lg = out.stats["ledger"]
        total = lg["absorbed"] + lg["exited"] + lg["roulette_kill"] - lg["roulette_gain"] + lg["lost"]
        assert abs(total / p.Nphoton - 1.0) < 1e-6  # FP32 weights: w - dep and dep round alike
    mesh = V.Mesh(p)
    both, st = V.run_batch([mesh, mesh], [p, p.copy(Nphoton=0)], max_steps=cap, normalize=False)
    assert st["capped"] == out.stats["capped"] and st["steps"] == out.stats["steps"]
    if p.f == 0.0:  # the one-job and per-job forms round a modulated source's phase differently
        for k in ("ER", "EBR"):
            np.testing.assert_allclose(getattr(both[0], k), getattr(out, k), rtol=1e-9, atol=1e-9)
    wide, _ = V.run_batch([mesh], [p], max_steps=free.stats["steps"], normalize=False)
    np.testing.assert_allclose(wide[0].ER, free.ER, rtol=1e-9, atol=1e-9)
    mesh.close()


@pytest.mark.parametrize("name,precision", [("phantom3d", V.VMC_FP32), ("phantom3d_fd", V.VMC_FP32),
                                            ("square2d", V.VMC_FP32), ("mixed2d_fd", V.VMC_FP32),
                                            ("phantom3d", V.VMC_FP64), ("mixed2d_fd", V.VMC_FP64)])
@pytest.mark.parametrize("n,block", [(1, 0), (33, 0), (609, 64), (2500, 0), (19457, 128), (160001, 0)])
def test_photons_dealt_and_moved_between_lanes_walk_alike(built, name, precision, n, block):
    """n photons in one launch equal the same photons in two launches of other sizes, whose lanes,
    warps and packing differ: only the order of the FP64 additions does."""
    if precision == V.VMC_FP64 and n > 20000:
        pytest.skip("the FP64 forms run the smaller counts")
    p = cases()[name][0].copy(Nphoton=n, seed=4242)
    one = V.run(p, precision=precision, normalize=False, block_size=block)
    assert one.stats["photons_done"] == n
    cut = n // 3
    parts = [V.run(p, precision=precision, nphoton=k, seed=4242, normalize=False, photon_offset=o)
             for k, o in ((cut, 0), (n - cut, cut))]
    assert one.stats["steps"] == sum(x.stats["steps"] for x in parts)
    assert one.stats["scatters"] == sum(x.stats["scatters"] for x in parts)
    for k in ("ER", "EI", "EBR", "EBI", "DEBR", "DEBI"):
        total = sum(getattr(x, k) for x in parts)
        np.testing.assert_allclose(getattr(one, k), total, rtol=1e-9, atol=1e-9)
    mesh = V.Mesh(p, precision=precision)  # per-job form: photons of two jobs in the lanes of a warp
    both, st = V.run_batch([mesh, mesh], [p.copy(Nphoton=cut), p.copy(Nphoton=n - cut, seed=77)], precision=precision,
                           normalize=False)
    assert st["photons_done"] == n
    if p.f == 0.0 or precision == V.VMC_FP64:  # the FP32 one-job form rounds the phase differently
        np.testing.assert_allclose(both[0].EBR, parts[0].EBR, rtol=1e-9, atol=1e-9)
    mesh.close()


@pytest.mark.parametrize("block", [32, 64, 96])
@pytest.mark.parametrize("name,precision,n", [("phantom3d", V.VMC_FP32, 20000), ("phantom3d_fd", V.VMC_FP32, 6001),
                                              ("phantom3d", V.VMC_FP64, 5000), ("mixed2d_fd", V.VMC_FP64, 5003)])
def test_blocks_of_few_warps_lose_no_photon(built, name, precision, n, block):
    """CTAs of one to three warps pack their last photons without dropping one: the walks of the
    default block, in steps, scatters and sums."""
    p = cases()[name][0].copy(Nphoton=n, seed=31)
    want = V.run(p, precision=precision, normalize=False)
    one = V.run(p, precision=precision, normalize=False, block_size=block)
    assert one.stats["photons_done"] == want.stats["photons_done"] == n
    assert one.stats["steps"] == want.stats["steps"] and one.stats["scatters"] == want.stats["scatters"]
    for k in ("ER", "EI", "EBR", "EBI"):
        np.testing.assert_allclose(getattr(one, k), getattr(want, k), rtol=1e-9, atol=1e-9)
    mesh = V.Mesh(p, precision=precision)
    _, st = V.run_batch([mesh, mesh], [p.copy(Nphoton=n // 3), p.copy(Nphoton=n - n // 3)], precision=precision,
                        block_size=block)
    assert st["photons_done"] == n
    mesh.close()


@pytest.mark.parametrize("mua", [1e-38, 2e-38, 1e-37])  # subnormal in FP32, and with depths that are
@pytest.mark.parametrize("f", [0.0, 1e-27])
def test_deposits_of_the_smallest_absorption(built, mua, f):
    """Absorption next to none, in FP32's smallest numbers, gives the fluence of none: the walks are
    the same, and a visit to an element loses its deposit only where that is below 1.18e-38."""
    r, H, BH = mg.box_mesh_3d(3, 3, 3)
    r = 20.0 * r
    ne, nb = len(H), len(BH)
    types = np.full(nb, ord("a"), np.uint8)
    types[np.all(r[BH][:, :, 2] == r[:, 2].min(), axis=1)] = ord("c")
    p = mg.Problem(dim=3, H=H, BH=BH, r=r, mua=np.zeros(ne), mus=np.full(ne, 2.0), g=np.zeros(ne), n=np.full(ne, 1.0),
                   BCType=types, BCn=np.full(nb, 1.0), Nphoton=2000, seed=5)
    none = V.run(p, normalize=False)
    out = V.run(p.copy(mua=np.full(ne, mua), f=f), normalize=False)
    assert out.stats["steps"] == none.stats["steps"]
    path = none.ER.sum()  # of all photons, weight 1
    if f == 0.0:
        got, least = out.ER / mua, mua
    else:  # MonteCarlo's normalisation, without volume and number
        k = 2 * np.pi * f / 2.99792458e11
        got, least = (out.EI * k + out.ER * mua) / (k * k + mua * mua), min(k, mua)
    visits = none.stats["steps"] - none.stats["scatters"] + p.Nphoton
    lost = 1.18e-38 / least * visits
    assert lost < 0.75 * path
    # FP32 sums of up to some hundred steps a visit: 1e-4
    assert path * (1 - 1e-4) - lost < got.sum() < path * (1 + 1e-4)
    assert np.all(got <= none.ER * (1 + 1e-4) + 1e-300)


@pytest.mark.parametrize("precision", [V.VMC_FP32, V.VMC_FP64])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_photons_without_a_position_are_lost_at_once(built, precision, bad):
    """Pencil beams, into the body from all sides, from points that are no numbers: no face is ever
    found, as in the reference."""
    p = cases()["jitter3d"][0].copy(Nphoton=500)
    p = p.copy(BCType=np.full(p.Nb, ord("p"), np.uint8), BCLightDirectionType=np.full(p.Nb, ord("p"), np.uint8),
               BCLNormal=np.full((p.Nb, 3), bad))
    out = V.run(p, precision=precision, normalize=False, max_steps=2000)
    assert out.stats["loss"] == p.Nphoton and out.stats["steps"] == 0 and out.stats["capped"] == 0
    assert np.all(out.ER == 0) and np.all(out.EBR == 0)
    assert out.stats["ledger"]["lost"] == p.Nphoton


@pytest.mark.parametrize("precision", [V.VMC_FP32, V.VMC_FP64])
def test_trace_of_a_photon_that_finds_no_face(built, precision):
    """A replayed photon without a direction is lost before it has walked an element: the trace
    holds that event and no element, as the reference's."""
    p = cases()["jitter3d"][0].copy(Nphoton=6)
    p = p.copy(BCType=np.full(p.Nb, ord("l"), np.uint8), BCLightDirectionType=np.full(p.Nb, ord("a"), np.uint8),
               BCLNormal=np.zeros((p.Nb, 3)))
    tape = np.random.default_rng(3).integers(0, 2 ** 32, 6 * 50, dtype=np.uint64).astype(np.uint32)
    off = np.arange(7, dtype=np.int64) * 50
    out = V.run(p, precision=precision, tape=tape, tape_off=off, trace_photons=6, trace_stride=100)
    assert out.stats["loss"] == 6 and out.stats["steps"] == 0
    lost = -2 ** 63 + 2
    assert [list(t) for t in out.traces] == [[lost]] * 6


@pytest.mark.parametrize("mus", [2e-38, 5e-38, 1e-37, 1e-20])
def test_path_left_on_entering_a_scattering_element(built, mus):
    """A layer that scatters next to nothing before one that does: the path left there is the path of
    a vacuum, whose draw is independent, so that sums over layers agree within their noise."""
    r, H, BH = mg.box_mesh_3d(4, 4, 6)
    ne, nb, n = len(H), len(BH), 1000000
    z = r[H].mean(axis=1)[:, 2]
    types = np.full(nb, ord("a"), np.uint8)
    types[np.all(r[BH][:, :, 2] == 0, axis=1)] = ord("l")
    base = mg.Problem(dim=3, H=H, BH=BH, r=r, mua=np.full(ne, 0.2), mus=np.where(z < 2, mus, 2.0), g=np.zeros(ne),
                      n=np.full(ne, 1.0), BCType=types, BCn=np.full(nb, 1.0), Nphoton=n, seed=5)
    tiny = V.run(base, normalize=False)
    none = V.run(base.copy(mus=np.where(z < 2, 0.0, 2.0), seed=6), normalize=False)
    for k in range(6):
        a, b = (x.ER[(z >= k) & (z < k + 1)].sum() for x in (tiny, none))
        assert abs(a - b) < 6 * np.sqrt(2 * n / 4)  # a photon leaves between 0 and 1 there
    assert abs(tiny.stats["scatters"] / none.stats["scatters"] - 1) < 0.02


def test_a_path_that_is_no_number(built):
    """Elements without a scattering coefficient (NaN): what becomes of the photons there is the same
    in a launch of one job and in one of several, and none leaves through a boundary element that
    it has not come to."""
    r, H, BH = mg.box_mesh_3d(4, 4, 6)
    ne, nb = len(H), len(BH)
    z = r[H].mean(axis=1)[:, 2]
    zb = r[BH].mean(axis=1)[:, 2]
    types = np.full(nb, ord("a"), np.uint8)
    types[zb == 6] = ord("l")
    p = mg.Problem(dim=3, H=H, BH=BH, r=r, mua=np.full(ne, 0.2), mus=np.where((z > 2) & (z < 4), np.nan, 2.0), g=np.zeros(ne),
                   n=np.full(ne, 1.0), BCType=types, BCn=np.full(nb, 1.0), Nphoton=5000, seed=5)
    one = V.run(p, normalize=False, max_steps=300)
    mesh = V.Mesh(p)
    two, _ = V.run_batch([mesh, mesh], [p, p.copy(Nphoton=0)], normalize=False, max_steps=300)
    mesh.close()
    assert zb[0] < 1 and one.EBR[0] == 0
    np.testing.assert_allclose(one.EBR, two[0].EBR, rtol=1e-9, atol=1e-9)
    np.testing.assert_allclose(np.nan_to_num(one.ER), np.nan_to_num(two[0].ER), rtol=1e-9, atol=1e-9)
