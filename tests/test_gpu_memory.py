"""Device memory that the library keeps between calls."""
import glob
import os
import subprocess
import sys

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
