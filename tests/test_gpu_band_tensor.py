"""The band kernels' tensor-core tiles: values that need all three bf16 parts, window sizes that are not
whole steps, and infinities and NaN, which take the rows that hold them and no others."""
import numpy as np
import pytest
import torch

from gpu_util import TOL, assert_spmm_close, dev, to_torch_bf16
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu

A0 = synth.banded_plus_random(1500, 32, 8, seed=5)


def _spmm(A, Bd, halo=32):
    cfg = N.Config.make(schedule=N.RB_PR, items_per_unit=halo, flags=N.FLAG_WINDOW)
    Ad = dev(A)
    assert " band " in ops.plan_name(Ad, Bd, cfg)
    C = torch.full((A.M, Bd.shape[1]), float("nan"), device="cuda")
    return ops.spmm(Ad, Bd, C, cfg).cpu().numpy()


@pytest.mark.parametrize("scale", [1.0, 1e-30, 3e37])
@pytest.mark.parametrize("halo", [1, 5, 31, 32, 33, 111, 112])
def test_spmm_bf16_parts_and_windows(cuda, halo, scale):
    """Values with 24 significant bits, ordinary, tiny and near the largest."""
    rng = np.random.default_rng(halo)
    bits = rng.integers(0, 1 << 23, A0.nnz, dtype=np.int64) | 1
    val = ((1.0 + bits / 2.0 ** 23) * rng.choice([-1, 1], A0.nnz) * scale).astype(np.float32)
    A = synth.CSR(A0.row_ptr, A0.col, val, A0.M, A0.K)
    B = synth.to_bf16_bits(synth.dense(A.K, 80, seed=6) / np.float32(80))
    assert_spmm_close(_spmm(A, to_torch_bf16(B), halo), A, B, bf16=True)


def _same(got, want, bound):
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~finite], want[~finite].astype(np.float32), equal_nan=True)
    assert (np.abs(got - want)[finite] <= TOL * bound[finite] + 1e-30).all()


@pytest.mark.parametrize("where", ["value", "operand", "both"])
def test_spmm_bf16_infinities(cuda, where):
    A = synth.CSR(A0.row_ptr, A0.col, A0.val.copy(), A0.M, A0.K)
    B = synth.bf16_bits_to_f32(synth.to_bf16_bits(synth.dense(A.K, 64, seed=7)))
    if where != "operand":
        A.val[A.row_ptr[300] + 20] = np.inf
        A.val[A.row_ptr[700] + 3] = np.nan
    if where != "value":
        B[400, 5], B[900, 6], B[901, 6] = np.inf, -np.inf, np.nan
    rows = np.repeat(np.arange(A.M), np.diff(A.row_ptr))
    want, bound = np.zeros((A.M, 64)), np.zeros((A.M, 64))
    with np.errstate(invalid="ignore"):
        terms = A.val.astype(np.float64)[:, None] * B[A.col].astype(np.float64)
        np.add.at(want, rows, terms)
        np.add.at(bound, rows, np.abs(terms))
    _same(_spmm(A, to_torch_bf16(synth.to_bf16_bits(B))), want, bound)


@pytest.mark.parametrize("scale", [1.0, 1e-15, 1e18])
@pytest.mark.parametrize("rows", [1500, 33, 1])
def test_sddmm_parts(cuda, rows, scale):
    A = A0 if rows == 1500 else synth.random_csr(rows, 60, 0.5, seed=rows)
    X, Y = synth.dense(A.M, 64, seed=8) * np.float32(scale), synth.dense(A.K, 64, seed=9)
    out = ops.sddmm(dev(A), torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda(),
                    config=N.SddmmConfig.make(N.SDDMM_BAND)).cpu().numpy()
    r = np.repeat(np.arange(A.M), np.diff(A.row_ptr))
    t = X[r].astype(np.float64) * Y[A.col].astype(np.float64)
    v = A.val.astype(np.float64)
    assert (np.abs(out - v * t.sum(1)) <= TOL * np.abs(v) * np.abs(t).sum(1)).all()


def test_sddmm_infinities(cuda):
    X, Y = synth.dense(A0.M, 64, seed=8), synth.dense(A0.K, 64, seed=9)
    X[100, 3], X[800, 9] = np.inf, np.nan
    Y[120, 7], Y[1200, 60] = -np.inf, np.nan
    out = ops.sddmm(dev(A0), torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda(),
                    config=N.SddmmConfig.make(N.SDDMM_BAND)).cpu().numpy()
    r = np.repeat(np.arange(A0.M), np.diff(A0.row_ptr))
    with np.errstate(invalid="ignore"):
        t = X[r].astype(np.float64) * Y[A0.col].astype(np.float64)
        v = A0.val.astype(np.float64)
        _same(out, v * t.sum(1), np.abs(v) * np.abs(t).sum(1))
