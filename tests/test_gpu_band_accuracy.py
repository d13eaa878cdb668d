"""The band kernels against 64 bits where the tensor cores' split of fp32 values shows: factors with one
element that matters, and factors that are all alike."""
import numpy as np
import pytest
import torch

from gpu_util import dev, to_torch_bf16
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu

A0 = synth.banded_plus_random(1500, 32, 8, seed=5)
D = 64


def _sddmm(A, X, Y):
    out = ops.sddmm(dev(A), torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda(),
                    config=N.SddmmConfig.make(N.SDDMM_BAND)).cpu().numpy()
    rows = np.repeat(np.arange(A.M), np.diff(A.row_ptr))
    t = X[rows].astype(np.float64) * Y[A.col].astype(np.float64)
    v = A.val.astype(np.float64)
    return out, v * t.sum(1), np.abs(v) * np.abs(t).sum(1)


def _ones(A):  # values that scale without rounding
    return synth.CSR(A.row_ptr, A.col, np.ones(A.nnz, np.float32), A.M, A.K)


def _mantissas(rng, shape):
    return ((1.0 + rng.integers(0, 1 << 23, shape) / 2.0 ** 23) *
            rng.choice([-1, 1], shape)).astype(np.float32)


def test_sddmm_one_element(cuda):
    """One product: 2^-24 of it left out, 2^-24 rounded off."""
    rng = np.random.default_rng(1)
    A = _ones(A0)
    X, Y = np.zeros((A.M, D), np.float32), np.zeros((A.K, D), np.float32)
    X[:, 21], Y[:, 21] = _mantissas(rng, A.M), _mantissas(rng, A.K)
    X[::7, 21] = Y[::5, 21] = np.float32(1 + 2.0 ** -7 - 2.0 ** -23)
    out, want, bound = _sddmm(A, X, Y)
    assert (np.abs(out - want) <= 1.02 * 2.0 ** -23 * bound).all()


def test_sddmm_equal_factors(cuda):
    """64 equal products: the sums of 16 are exact; rounded are each with its small parts (2^-24), and
    the running sum at 2, 3 and 4 quarters."""
    A = _ones(A0)
    X = np.full((A.M, D), 1 + 2.0 ** -7 - 2.0 ** -23, np.float32)
    out, want, bound = _sddmm(A, X, X)
    assert (np.abs(out - want) <= 1.02 * 3.25 * 2.0 ** -24 * bound).all()


@pytest.mark.parametrize("sx,sy", [(1e-36, 1e30), (1e-30, 1e-3), (1e30, 1e-37), (1e-20, 1e-18), (1e-39, 1e38),
                                   (3e-19, 3e-19), (1e-44, 1e38)])
def test_sddmm_small_magnitudes(cuda, sx, sy):
    """Dot products as near as 68 fp32 operations bring them (2^-24 each, and 2^-149 where the result is
    subnormal), whatever the factors' magnitudes."""
    rng = np.random.default_rng(2)
    A = _ones(A0)
    X = (_mantissas(rng, (A.M, D)) * np.float64(sx)).astype(np.float32)
    Y = (_mantissas(rng, (A.K, D)) * np.float64(sy)).astype(np.float32)
    out, want, bound = _sddmm(A, X, Y)
    assert (np.abs(out - want) <= 68 * (2.0 ** -24 * bound + 2.0 ** -149)).all()


def test_sddmm_one_small_element(cuda):
    """Tiny factors among ordinary ones; blocks of rows with and without them."""
    rng = np.random.default_rng(3)
    A = _ones(A0)
    X, Y = np.zeros((A.M, D), np.float32), _mantissas(rng, (A.K, D))
    X[:, 5] = _mantissas(rng, A.M)
    X[40::200, 5] *= np.float32(1e-36)
    out, want, bound = _sddmm(A, X, Y)
    assert (np.abs(out - want) <= 1.02 * 2.0 ** -23 * bound + 2.0 ** -149).all()


def _spmm(A, B, bf16):
    cfg = N.Config.make(schedule=N.RB_PR, items_per_unit=32, flags=N.FLAG_WINDOW)
    Bd = torch.from_numpy(B).cuda()
    if bf16:
        bits = synth.to_bf16_bits(B)
        B, Bd = synth.bf16_bits_to_f32(bits), to_torch_bf16(bits)
    Ad = dev(A)
    assert " band " in ops.plan_name(Ad, Bd, cfg)
    C = ops.spmm(Ad, Bd, torch.full((A.M, B.shape[1]), float("nan"), device="cuda"), cfg).cpu().numpy()
    rows = np.repeat(np.arange(A.M), np.diff(A.row_ptr))
    with np.errstate(invalid="ignore"):
        t = A.val.astype(np.float64)[:, None] * B[A.col].astype(np.float64)
        want, bound = np.zeros(C.shape), np.zeros(C.shape)
        np.add.at(want, rows, t)
        np.add.at(bound, rows, np.abs(t))
    return C, want, bound


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("sa,sb", [(1e-30, 1.0), (1e-33, 1e10), (1e-36, 1e30), (1e-39, 1e38), (1e-44, 1e38),
                                   (1.0, 1e-39), (1e-20, 1e-18)])
def test_spmm_small_magnitudes(cuda, sa, sb, bf16):
    """Rows of at most 73 nonzeros as near as their multiply-adds, whatever the magnitudes."""
    rng = np.random.default_rng(4)
    A = synth.CSR(A0.row_ptr, A0.col, (_mantissas(rng, A0.nnz) * np.float64(sa)).astype(np.float32),
                  A0.M, A0.K)
    C, want, bound = _spmm(A, (_mantissas(rng, (A.K, 64)) * np.float64(sb)).astype(np.float32), bf16)
    assert (np.abs(C - want) <= 73 * (2.0 ** -24 * bound + 2.0 ** -149)).all()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n", [64, 80])
def test_spmm_infinities_of_unused_rows(cuda, n, bf16):
    """Infinities and NaN of B and A reach the rows that hold them, by the window and off the band, and
    no others; values near the largest stay finite."""
    rng = np.random.default_rng(6)
    keep = np.ones(A0.nnz, bool)
    keep[np.isin(A0.col, (250, 251, 900))] = False  # unused rows of B
    rows = np.repeat(np.arange(A0.M), np.diff(A0.row_ptr))
    ptr = np.append(0, np.cumsum(np.bincount(rows[keep], minlength=A0.M))).astype(np.int32)
    A = synth.CSR(ptr, A0.col[keep].copy(), _mantissas(rng, int(keep.sum())), A0.M, A0.K)
    A.val[A.row_ptr[600] + 20], A.val[A.row_ptr[700] + 2] = np.inf, np.nan
    A.val[A.row_ptr[1300] + 30] = np.float32(3.4e38)
    B = rng.uniform(0.25, 0.5, (A.K, n)).astype(np.float32)
    B[250], B[251, ::2], B[900, 1::3] = np.inf, np.nan, -np.inf
    B[1000, 7], B[1100, 9] = np.inf, np.nan
    C, want, bound = _spmm(A, B, bf16)
    finite = np.isfinite(want)
    assert finite.mean() > 0.9
    assert np.array_equal(C[~finite], want[~finite].astype(np.float32), equal_nan=True)
    assert (np.abs(C - want)[finite] <= 73 * 2.0 ** -24 * bound[finite]).all()
