"""A call that keeps its scratch in the library's pool works again after its process has reset the device
(which ends the process's own context, and the pool with it)."""
import glob
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = r"""
import ctypes as C, sys
import numpy as np
from segtaco_gb300 import native as N
L, rt = N.lib(), C.CDLL(sys.argv[1])
def up(a):
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
    return p.value
M, n = 100_000, 64  # past the size that needs no scratch
rng = np.random.default_rng(0)
rp = np.arange(M + 1, dtype=np.int32) * 4
col, val = rng.integers(0, M, 4 * M).astype(np.int32), rng.random(4 * M, dtype=np.float32)
B = rng.random((M, n), dtype=np.float32)
want = (val.reshape(M, 4, 1).astype(np.float64) * B[col].reshape(M, 4, n)).sum(1)
cfg = N.Config.make(schedule="eb_pr")
for _ in range(3):
    d, c = [up(x) for x in (rp, col, val, B)], up(np.zeros((M, n), np.float32))
    for _ in range(2):
        N.check(L.segtaco_spmm(M, M, 4 * M, d[0], d[1], d[2], d[3], N.F32, n, c, n, n, C.byref(cfg), None, 0, None))
    out = np.empty((M, n), np.float32)
    assert rt.cudaMemcpy(out.ctypes.data_as(C.c_void_p), C.c_void_p(c), C.c_size_t(out.nbytes), 2) == 0
    assert np.allclose(out, want, rtol=1e-5, atol=0)
    L.segtaco_taco_release()
    assert rt.cudaDeviceReset() == 0
L.segtaco_taco_release()
print("done")
"""


def test_pool_after_a_reset(cuda):
    runtimes = sorted(glob.glob("/usr/local/cuda/lib64/libcudart.so*"))
    if not runtimes:
        pytest.skip("no CUDA runtime library beside the toolkit")
    r = subprocess.run([sys.executable, "-c", SCRIPT, runtimes[0]], cwd=ROOT, capture_output=True, text=True,
                       timeout=120, env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stdout + r.stderr
