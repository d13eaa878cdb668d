"""SpMSpV over columns of every length: the flat range of a warp's short columns, columns at and past
the length that the cluster shares, and every number of entries per warp."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from segtaco_gb300 import ops, synth

from gpu_util import TOL, dev

pytestmark = pytest.mark.gpu


def _columns(lengths, M, seed):
    """The CSR of A^T: row j holds the `lengths[j]` distinct sorted rows of column j."""
    rng = np.random.default_rng(seed)
    ptr = np.zeros(len(lengths) + 1, np.int32)
    np.cumsum(lengths, out=ptr[1:])
    col = np.concatenate([np.sort(rng.choice(M, n, replace=False)) for n in lengths] + [[]])
    val = rng.uniform(-1, 1, ptr[-1]).astype(np.float32)
    return synth.CSR(ptr, col.astype(np.int32), val, len(lengths), M)


def _check(At, idx, x, with_values=True):
    val = At.val if with_values else np.ones_like(At.val)
    y = ops.spmspv(dev(At, with_values), torch.from_numpy(idx).cuda(), torch.from_numpy(x).cuda(),
                   At.K, torch.full((At.K,), float("nan"), device="cuda"))
    ref, bound = O.spmspv_f64(At.row_ptr, At.col, val, At.K, idx, x)
    err = np.abs(y.cpu().numpy() - ref)
    assert (err <= TOL * bound).all(), err.max()


@pytest.mark.parametrize("edge", [511, 512, 513, 1024, 1025, 33_000])
@pytest.mark.parametrize("with_values", [True, False])
def test_long_columns(cuda, edge, with_values):
    lengths = np.array([0, 1, edge, 7, edge, 0, 32, 31, 33, edge + 5] * 3)
    At = _columns(lengths, 40_000, seed=edge)
    idx = np.arange(At.M, dtype=np.int32)
    x = np.random.default_rng(1).uniform(-1, 1, idx.size).astype(np.float32)
    _check(At, idx, x, with_values)
    _check(At, idx[2:3], x[2:3], with_values)  # one entry


@pytest.mark.parametrize("nx", [1, 31, 33, 9728, 9729, 40_000, 311_297, 640_001])
def test_entries_per_warp(cuda, nx):
    """Past 64 warps per SM a warp takes 2, 4, .. 32 entries; some columns long, some repeated."""
    rng = np.random.default_rng(nx)
    lengths = rng.choice([0, 1, 2, 5, 11], size=5000)
    lengths[rng.choice(5000, 3, replace=False)] = 700
    At = _columns(lengths, 20_000, seed=nx + 1)
    idx = np.sort(rng.integers(0, At.M, nx)).astype(np.int32)
    x = rng.uniform(-1, 1, nx).astype(np.float32)
    _check(At, idx, x)
