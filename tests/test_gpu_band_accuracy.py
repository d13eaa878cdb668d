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
