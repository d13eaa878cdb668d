"""SDDMM with X and Y on either side of the size from which X's rows leave L2 first."""
import pytest
import torch

from segtaco_gb300 import ops, synth

from gpu_util import TOL, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d", [37, 64, 128, 256])
@pytest.mark.parametrize("side", [-1, 0])
def test_either_side(cuda, dtype, d, side):
    rows = (64 << 20) // (d * dtype.itemsize * 2) + 1 + side  # X and Y: 64 MB at most, or just more
    A = synth.power_law(rows, rows, 1.8, 200, 0.02, seed=d)
    g = torch.Generator(device="cuda").manual_seed(d)
    X, Y = (torch.rand(rows, d, generator=g, device="cuda").sub_(0.5).to(dtype) for _ in range(2))
    Ad = dev(A)
    out = ops.sddmm(Ad, X, Y, torch.full((A.nnz,), float("nan"), device="cuda")).double()
    i = torch.repeat_interleave(torch.arange(rows, device="cuda"), Ad.row_ptr.diff().long())
    step = 1 << 19
    for p in range(0, A.nnz, step):
        x, y = X[i[p:p + step]].double(), Y[Ad.col[p:p + step].long()].double()
        v = Ad.val[p:p + step].double()
        bound = v.abs() * (x.abs() * y.abs()).sum(1)
        assert ((out[p:p + step] - v * (x * y).sum(1)).abs() <= TOL * bound).all()
