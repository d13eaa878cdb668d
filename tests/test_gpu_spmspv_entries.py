"""SpMSpV: every number of entries per warp, long columns listed in a cluster of several, a y that begins
off a 16-byte boundary, and products that follow each other on a stream and in a graph."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from segtaco_gb300 import ops, synth

from gpu_util import TOL, dev

pytestmark = pytest.mark.gpu


def _matrix(seed, mean):
    rng = np.random.default_rng(seed)
    lengths = np.minimum(rng.poisson(mean, 3000), 4000)
    lengths[rng.choice(3000, 40, replace=False)] = rng.choice([512, 513, 2000, 3999], 40)
    ptr = np.zeros(3001, np.int32)
    np.cumsum(lengths, out=ptr[1:])
    col = np.concatenate([np.sort(rng.choice(4000, n, replace=False)) for n in lengths] + [[]])
    return synth.CSR(ptr, col.astype(np.int32), rng.uniform(-1, 1, ptr[-1]).astype(np.float32), 3000, 4000)


def _close(At, idx, x, y):
    ref, bound = O.spmspv_f64(At.row_ptr, At.col, At.val, At.K, idx, x)
    err = np.abs(y.cpu().numpy() - ref)
    assert (err <= TOL * bound).all(), err.max()


@pytest.mark.parametrize("mean", [1, 20, 90])
@pytest.mark.parametrize("nx", [1, 64, 65, 2048, 2049, 9000, 60_000])
def test_entries_and_alignment(cuda, mean, nx):
    At = _matrix(mean, mean)
    rng = np.random.default_rng(nx)
    idx = rng.integers(0, At.M, nx).astype(np.int32)
    x = rng.uniform(-1, 1, nx).astype(np.float32)
    for off in (0, 1, 3):
        y = torch.full((At.K + 8,), 7.0, device="cuda")
        part = y[off:off + At.K]
        ops.spmspv(dev(At), torch.from_numpy(idx).cuda(), torch.from_numpy(x).cuda(), At.K, part)
        _close(At, idx, x, part)
        assert (y[:off] == 7.0).all() and (y[off + At.K:] == 7.0).all()


@pytest.mark.parametrize("m", [1, 2, 3, 5])
def test_few_rows(cuda, m):
    ptr = np.array([0, 1, 1, 2], np.int32)
    At = synth.CSR(ptr, np.array([0, m - 1], np.int32), np.array([2.0, 3.0], np.float32), 3, m)
    idx, x = np.array([0, 2], np.int32), np.array([1.0, 1.0], np.float32)
    y = torch.full((m + 4,), float("nan"), device="cuda")
    ops.spmspv(dev(At), torch.from_numpy(idx).cuda(), torch.from_numpy(x).cuda(), m, y[1:1 + m])
    _close(At, idx, x, y[1:1 + m])
    assert torch.isnan(y[0]) and torch.isnan(y[1 + m:]).all()


def test_each_call_sees_what_the_stream_did_before(cuda):
    """x is made on the stream just before the call, and y of one call is read and reused by the next."""
    At = _matrix(5, 8)
    Ad, n = dev(At), At.M
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    base = torch.rand(n, device="cuda") - 0.5
    y, total = torch.empty(At.K, device="cuda"), torch.zeros(At.K, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())

    def steps():
        total.zero_()
        for k in range(6):
            ops.spmspv(Ad, idx.flip(0), (base * float(k + 1)).flip(0), At.K, y, stream=s)
            total.add_(y)

    with torch.cuda.stream(s):
        steps()
        s.synchronize()
        _close(At, np.arange(n, dtype=np.int32), 21.0 * base.cpu().numpy(), total)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            steps()
        for _ in range(3):
            g.replay()
        s.synchronize()
        _close(At, np.arange(n, dtype=np.int32), 21.0 * base.cpu().numpy(), total)
