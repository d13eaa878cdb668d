"""The default SDDMM kernel: every lane shape, warp blocks, rows that end inside a step, runs of empty
rows, and the row search of a warp's first nonzero."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from gpu_util import TOL, dev, small_cases, to_torch_bf16
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu

CASES = small_cases()


def _factor(rows, D, pad, bf16, seed):
    X = synth.dense(rows, D + pad, seed)
    bits = synth.to_bf16_bits(X)
    Xd = to_torch_bf16(bits) if bf16 else torch.from_numpy(X).cuda()
    host = synth.bf16_bits_to_f32(bits) if bf16 else X
    return np.ascontiguousarray(host[:, :D]), Xd[:, :D]


def _check(A, D, pad, bf16, config=None, with_values=True):
    X, Xd = _factor(A.M, D, pad, bf16, 1)
    Y, Yd = _factor(A.K, D, pad, bf16, 2)
    out = torch.full((A.nnz,), float("nan"), device="cuda")
    ops.sddmm(dev(A, with_values), Xd, Yd, out=out, config=config)
    rows = np.repeat(np.arange(A.M), np.diff(A.row_ptr))
    val = A.val.astype(np.float64) if with_values else np.ones(A.nnz)
    x, y = X[rows].astype(np.float64), Y[A.col].astype(np.float64)
    err = np.abs(out.cpu().numpy() - val * (x * y).sum(1))
    assert (err <= TOL * np.abs(val) * np.abs(x * y).sum(1) + 1e-30).all(), err.max()


# 32- and 16-byte lanes (bf16: 8-byte ones), 2- and 1-element chunks with one to five per lane, idle
# lanes, and D past the lanes' reach (more than one pass)
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("D,pad", [(1, 0), (2, 0), (3, 0), (4, 0), (6, 0), (7, 0), (8, 0), (12, 0),
                                   (16, 0), (17, 0), (20, 0), (25, 0), (32, 0), (33, 0), (37, 0),
                                   (40, 0), (46, 0), (61, 0), (64, 0), (64, 1), (70, 0), (82, 0),
                                   (85, 0), (96, 0), (100, 0), (126, 0), (127, 0), (128, 0),
                                   (128, 4), (129, 0), (200, 0), (256, 0), (260, 0), (300, 1),
                                   (515, 0), (1024, 0), (1025, 0)])
def test_lane_shapes(cuda, D, pad, bf16):
    _check(CASES["half_empty"], D, pad, bf16)


@pytest.mark.parametrize("block", [32, 64, 256, 4096])
@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("D", [8, 13, 64])
def test_blocks_and_rows(cuda, name, block, D):
    _check(CASES[name], D, 0, False, N.SddmmConfig.make(N.SDDMM_AUTO, block), with_values=D != 13)


@pytest.mark.parametrize("D", [8, 37, 64])
def test_rows_outside_the_pattern_stay_out(cuda, D):
    """Idle positions read row 0 of Y: infinities and NaN there reach no result."""
    A = synth.random_csr(300, 200, 0.05, seed=3)
    A.col[:] = np.maximum(A.col, 1)
    X, Xd = _factor(A.M, D, 0, False, 1)
    Y, Yd = _factor(A.K, D, 0, False, 2)
    want = ops.sddmm(dev(A), Xd, Yd)
    Yd[0, ::2], Yd[0, 1::2] = float("inf"), float("nan")
    assert torch.equal(ops.sddmm(dev(A), Xd, Yd), want)


@pytest.mark.parametrize("nnz", [1_250_003, 2_600_017])
@pytest.mark.parametrize("per_row", [1, 16, 33])
@pytest.mark.parametrize("D,bf16", [(5, False), (64, False), (64, True), (128, False)])
def test_blocks_fitted_to_the_waves(cuda, D, bf16, per_row, nnz):
    """From one to four waves of warps a block is not a power of two, and the last one is short."""
    M, K = (nnz + per_row - 1) // per_row, 500
    rng = np.random.default_rng(3)
    A = synth.CSR(np.minimum(np.arange(M + 1) * per_row, nnz).astype(np.int32),
                  rng.integers(0, K, nnz).astype(np.int32),
                  rng.standard_normal(nnz).astype(np.float32), M, K)
    X, Y = (torch.randn(n, D, device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)
            for n in (M, K))
    Ad = dev(A)
    out = ops.sddmm(Ad, X, Y, out=torch.full((nnz,), float("nan"), device="cuda"))
    rows, cols = torch.arange(nnz, device="cuda") // per_row, Ad.col.long()
    for p in range(0, nnz, 1 << 18):
        q = slice(p, min(p + (1 << 18), nnz))
        xy = X[rows[q]].double() * Y[cols[q]].double()
        v = Ad.val[q].double()
        err = (out[q].double() - v * xy.sum(1)).abs()
        assert (err <= TOL * v.abs() * xy.abs().sum(1) + 1e-30).all(), err.max()
