"""Device memory that the library keeps between calls."""
import glob
import os
import subprocess
import sys

import numpy as np
import pytest

import valomc_gb300 as V
from valomc_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
AFTER_RESET = r"""
import ctypes as C, sys
import numpy as np
import valomc_gb300 as V
from golden.make_golden import cases
rt = C.CDLL(sys.argv[1])
p = cases()["jitter3d"][0].copy(Nphoton=2000)
want = V.run(p)
for precision in (V.VMC_FP32, V.VMC_FP64):
    assert rt.cudaSetDevice(0) == 0 and rt.cudaDeviceReset() == 0
    got = V.run(p)
    np.testing.assert_allclose(got.ER, want.ER, rtol=1e-9)
    mesh = V.Mesh(p, precision=precision)
    both, st = V.run_batch([mesh, mesh], [p, p.copy(seed=9)], precision=precision)
    assert st["photons_done"] == 2 * p.Nphoton
    mesh.close()
print("done")
"""


def test_calls_after_a_device_reset(built):
    """The pool of calls belongs to the context that it was made in: after cudaDeviceReset calls
    make another one."""
    runtimes = sorted(glob.glob("/usr/local/cuda/lib64/libcudart.so*"))
    if not runtimes:
        pytest.skip("no CUDA runtime library to reset the device with")
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.path.join(ROOT, "oracle")]))
    r = subprocess.run([sys.executable, "-c", AFTER_RESET, runtimes[0]], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), r.stdout + r.stderr


def test_a_server_counts_the_memory_of_finished_calls_as_free(built):
    """vmc_server_create limits its budget to the free memory: not less what calls before it have
    left in their pool."""
    torch = pytest.importorskip("torch")
    p = mg.config_3d_phantom(nphoton=10, seed=1)
    V.run(p)  # 648k tetrahedra: 52 MB of records and more
    before = torch.cuda.mem_get_info()[0]
    with_calls_memory = V.Server(memory_budget=1 << 30)
    after = torch.cuda.mem_get_info()[0]
    with_calls_memory.close()
    assert after - before > 32 << 20


# 1.11 GB with planes, in a memory where that leaves less than half; 1.00 GB where it does not fit
@pytest.mark.parametrize("layers,left", [(90, 2200 << 20), (81, 500 << 20)])
def test_fp64_mesh_without_room_for_plane_records(built, layers, left):
    """An FP64 mesh whose vertex records and job fit the device's memory runs, though its plane
    records (three times as much again) would not fit or would leave no room: by the walk that
    needs none of them."""
    torch = pytest.importorskip("torch")
    r, H, BH = mg.box_mesh_3d(80, 80, layers)
    ne, nb = len(H), len(BH)
    types = np.full(nb, ord("a"), np.uint8)
    types[np.all(r[BH][:, :, 2] == 0, axis=1)] = ord("c")
    p = mg.Problem(dim=3, H=H, BH=BH, r=r, mua=np.full(ne, 0.05), mus=np.full(ne, 1.0), g=np.full(ne, 0.8),
                   n=np.full(ne, 1.4), BCType=types, BCn=np.full(nb, 1.0), Nphoton=300, seed=3)
    mesh = V.Mesh(p, precision=V.VMC_FP64)
    assert mesh.device_bytes >= 320 * ne
    want, _ = V.run_batch([mesh], [p], precision=V.VMC_FP64, normalize=False)
    mesh.close()
    V.Server(memory_budget=1 << 30).close()  # gives back what the calls' pool keeps
    free = torch.cuda.mem_get_info()[0]
    try:
        held = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    except RuntimeError:
        pytest.skip("the device's free memory cannot be held in one piece")
    try:
        mesh = V.Mesh(p, precision=V.VMC_FP64)
        assert 112 * ne <= mesh.device_bytes < 200 * ne
        got, st = V.run_batch([mesh, mesh], [p, p.copy(seed=4)], precision=V.VMC_FP64, normalize=False)
        mesh.close()
        assert st["photons_done"] == 2 * p.Nphoton
        one = V.run(p, precision=V.VMC_FP64, normalize=False)
    finally:
        del held
        torch.cuda.empty_cache()
    for x in (got[0], one):
        np.testing.assert_allclose(x.ER, want[0].ER, rtol=1e-8, atol=1e-9)
        np.testing.assert_allclose(x.EBR, want[0].EBR, rtol=1e-8, atol=1e-9)
