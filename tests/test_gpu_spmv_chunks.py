"""SpMV over rows that end at and around the edges of batches (32), steps (128) and chunks (128 to 1024
nonzeros), long runs of empty rows, and rows over many chunks."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from gpu_util import TOL, dev
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu


def _matrix(lengths, K, seed):
    rng = np.random.default_rng(seed)
    ptr = np.zeros(len(lengths) + 1, np.int32)
    np.cumsum(lengths, out=ptr[1:])
    col = rng.integers(1, K, ptr[-1]).astype(np.int32)  # column 0 unused; columns may repeat
    return synth.CSR(ptr, col, rng.uniform(-1, 1, ptr[-1]).astype(np.float32), len(lengths), K)


def _check(A, with_values=True):
    x = np.random.default_rng(1).uniform(-1, 1, A.K).astype(np.float32)
    val = A.val if with_values else np.ones_like(A.val)
    ref = O.spmm_f64(A.row_ptr, A.col, val, x[:, None])[:, 0]
    bound = O.spmm_absbound(A.row_ptr, A.col, val, x[:, None])[:, 0]
    x[0] = np.nan  # idle lanes gather nothing
    y = torch.full((A.M,), float("nan"), device="cuda")
    ops.spmv(dev(A, with_values), torch.from_numpy(x).cuda(), y)
    err = np.abs(y.cpu().numpy() - ref)
    assert (err <= TOL * bound).all(), err.max()


@pytest.mark.parametrize("total", [1, 31, 32, 33, 127, 128, 129, 1023, 1024, 1025, 300_000])
@pytest.mark.parametrize("kind", ["ones", "empties", "edges", "one_row", "mixed"])
def test_row_ends(cuda, total, kind):
    rng = np.random.default_rng(total)
    if kind == "ones":
        lengths = np.ones(total, np.int64)
    elif kind == "empties":  # runs of up to 100 empty rows between short ones
        lengths = []
        while sum(lengths) < total:
            lengths += [0] * int(rng.integers(0, 100)) + [min(int(rng.integers(1, 4)), total - sum(lengths))]
            if len(lengths) > 20_000:
                lengths += [total - sum(lengths)]
        lengths = np.array(lengths + [0] * 70)
    elif kind == "edges":  # rows that end at multiples of 32
        lengths = np.append(rng.choice([32, 64, 96, 128, 1024], size=total // 32 + 1), [])
        lengths = np.diff(np.minimum(np.append(0, np.cumsum(lengths)), total)).astype(np.int64)
    elif kind == "one_row":
        lengths = np.array([0, 0, total, 0])
    else:
        lengths = rng.choice([0, 1, 2, 5, 30, 33, 200, 3000], size=total // 50 + 2)
    A = _matrix(lengths, 5000, seed=total)
    _check(A)
    _check(A, with_values=False)


def test_two_waves_of_chunks(cuda):
    """Enough nonzeros for chunks of 256 and more."""
    rng = np.random.default_rng(5)
    lengths = rng.choice([0, 1, 7, 40, 500, 9000], p=[.1, .5, .2, .1, .09, .01], size=40_000)
    _check(_matrix(lengths, 100_000, seed=6))
