"""The band kernels against 64 bits where the tensor cores' split of fp32 values shows: factors with one
element that matters, and factors that are all alike."""
import numpy as np
import pytest
import torch

from gpu_util import dev
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
