"""The row-slot walk of row blocks (depth 4): rb_sr bit for bit the sequential FMA order,
rb_pr within the bound and the same from run to run; rows of every length side by side."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from gpu_util import assert_spmm_close, dev, small_cases, to_torch_bf16
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu

CASES = small_cases()
CASES["steps"] = synth.random_csr(600, 700, 0.0, seed=21, long_rows={
    i: n for i, n in enumerate([0, 1, 7, 8, 9, 15, 16, 17, 0, 0, 31, 127, 128, 129, 500] * 40)})


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("n,pad", [(4, 0), (8, 0), (16, 0), (32, 0), (64, 0), (60, 0), (1, 0), (2, 0),
                                   (3, 0), (6, 0), (13, 0), (17, 0), (37, 0), (61, 0), (64, 1),
                                   (126, 0), (127, 0), (200, 2)])
def test_row_slots(cuda, name, n, pad):
    A = CASES[name]
    B = synth.dense(A.K, n + pad, seed=n)
    Ad, Bd = dev(A), torch.from_numpy(B).cuda()[:, :n]
    host = np.ascontiguousarray(B[:, :n])
    for sched in ("rb_sr", "rb_pr"):
        cfg = N.Config.make(schedule=sched, depth=4)
        if sched == "rb_sr" or A.nnz <= 32 * A.M or n % 4:  # rb_pr's long rows: the row walk
            assert " walk=6 " in ops.plan_name(Ad, Bd, cfg), ops.plan_name(Ad, Bd, cfg)
        C = [ops.spmm(Ad, Bd, torch.full((A.M, n), float("nan"), device="cuda"), cfg).cpu().numpy()
             for _ in range(2)]
        assert np.array_equal(C[0], C[1])
        if sched == "rb_sr":
            want = O.spmm_f32_rowseq(A.row_ptr, A.col, A.val, host, fma=True)
            assert np.array_equal(C[0], want)
        else:
            assert_spmm_close(C[0], A, host)


@pytest.mark.parametrize("n", [8, 36, 37, 64])
@pytest.mark.parametrize("sched", ["rb_sr", "rb_pr"])
def test_row_slots_bf16_and_unused_rows(cuda, sched, n):
    """bf16 B; idle lanes read B row 0, whose infinities reach no row of C."""
    A = synth.random_csr(900, 500, 0.02, seed=22, p_empty=0.2)
    A.col[:] = np.maximum(A.col, 1)
    bits = synth.to_bf16_bits(synth.dense(A.K, n, seed=23))
    bad = bits.copy()
    bad[0, ::2], bad[0, 1::2] = 0x7F80, 0x7FC0
    cfg = N.Config.make(schedule=sched, depth=4)
    C = torch.full((A.M, n), float("nan"), device="cuda")
    ops.spmm(dev(A), to_torch_bf16(bad), C, cfg)
    assert_spmm_close(C.cpu().numpy(), A, bits, bf16=True)
