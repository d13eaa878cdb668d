"""The split walk's sums against 64 bits: a row whose terms all round the same way."""
import numpy as np
import pytest
import torch

from gpu_util import dev, to_torch_bf16
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n", [8, 37, 64, 97, 127, 128])
@pytest.mark.parametrize("sched", ["eb_sr", "eb_pr"])
def test_long_row_rounds_once_a_step(cuda, sched, n, bf16):
    """480 equal terms in one chunk: at most 120 additions of four terms to a growing sum, half a unit of
    the sum each, and three roundings in each four."""
    terms = 480
    x = np.float32(1 + 0.45 * 2.0 ** -15)
    ptr = np.array([0, terms], np.int32)
    A = synth.CSR(ptr, np.arange(terms, dtype=np.int32), np.full(terms, x, np.float32), 1, terms)
    B = np.ones((terms, n), np.float32)
    Bd = to_torch_bf16(synth.to_bf16_bits(B)) if bf16 else torch.from_numpy(B).cuda()
    cfg = N.Config.make(schedule=sched, items_per_unit=512)
    Ad = dev(A)
    assert " walk=5 " in ops.plan_name(Ad, Bd, cfg)
    C = ops.spmm(Ad, Bd, None, cfg).cpu().numpy().astype(np.float64)
    sums = 4 * np.float64(x) * np.arange(1, terms // 4 + 1)
    half = np.spacing(sums.astype(np.float32)).astype(np.float64) / 2
    bound = half.sum() + terms // 4 * 3 * 2.0 ** -22
    assert (np.abs(C - terms * np.float64(x)) <= bound).all()
