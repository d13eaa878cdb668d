"""rb_pr over uneven rows as merge-path chunks whose cut rows are joined in order: rows over many chunks
and over exactly two, rows that end at a chunk edge, ragged N, bf16; the same from run to run; callers'
workspaces that hold the chunks' sums, only the pieces, or nothing."""
import numpy as np
import pytest
import torch

from gpu_util import assert_spmm_close, dev, small_cases, spmm_ref, to_torch_bf16
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu

CASES = small_cases()
# chunks of 32 items: a row of 40 chunks (two by two warps and more), rows that end where a chunk does
CASES["edges"] = synth.random_csr(300, 3000, 0.0, seed=31, long_rows={
    0: 31, 1: 31, 2: 30, 3: 0, 4: 64, 9: 1300, 10: 1, 50: 95, 51: 33, 52: 63, 200: 2900, 299: 700})
BIG = synth.power_law(60_000, 50_000, 1.8, 40_000, 0.02, seed=35)  # 1.09M nonzeros


def _cfg(flags=0, **kw):
    return N.Config.make(schedule="rb_pr", depth=8, flags=N.FLAG_LONG_ROWS | flags, **kw)


def _nan(A, n):
    return torch.full((A.M, n), float("nan"), device="cuda")


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n,pad", [(1, 0), (3, 0), (8, 0), (14, 0), (37, 0), (64, 0), (64, 1), (97, 0),
                                   (128, 0), (130, 0), (200, 0), (256, 0)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_joined_chunks(cuda, name, n, pad, bf16):
    A = CASES[name]
    B = synth.dense(A.K, n + pad, seed=n)
    bits = synth.to_bf16_bits(B)
    Bd = (to_torch_bf16(bits) if bf16 else torch.from_numpy(B).cuda())[:, :n]
    Ad = dev(A)
    if A.nnz:
        assert " walk=7 " in ops.plan_name(Ad, Bd, _cfg())
    C = [ops.spmm(Ad, Bd, _nan(A, n), _cfg()).cpu().numpy() for _ in range(2)]
    assert np.array_equal(C[0], C[1])
    assert_spmm_close(C[0], A, np.ascontiguousarray((bits if bf16 else B)[:, :n]), bf16=bf16)


def test_workspaces_and_capture(cuda):
    """A workspace of the full size, one that only holds the pieces' arrays, none under capture, and
    the two halves of a call; all within the bound and each the same when run again."""
    A, n = BIG, 40
    B = synth.dense(A.K, n, seed=36)
    Ad, Bd = dev(A), torch.from_numpy(B).cuda()
    ref = spmm_ref(A, B)
    full = ops.spmm_workspace_size(Ad, n, N.F32, _cfg())
    pieces = ops.spmm_workspace_size(Ad, n, N.F32, N.Config.make(schedule="rb_pr", flags=N.FLAG_LONG_ROWS))
    assert pieces < full
    want = ops.spmm(Ad, Bd, _nan(A, n), _cfg())
    assert_spmm_close(want.cpu().numpy(), A, B, ref=ref)
    ready = _cfg(N.FLAG_PARTITION_READY)
    for size in (full, pieces):
        ws = torch.full((size,), 0xff, dtype=torch.uint8, device="cuda")
        C = _nan(A, n)
        ops.spmm(Ad, Bd, C, _cfg(), ws)
        assert_spmm_close(C.cpu().numpy(), A, B, ref=ref)
        assert size != full or torch.equal(C, want)
        C2 = _nan(A, n)
        ops.spmm_partition(Ad, C2, _cfg(), ws)
        ops.spmm(Ad, Bd, C2, ready, ws)
        assert torch.equal(C, C2)
    with pytest.raises(Exception, match="needs the caller's workspace"):
        ops.spmm(Ad, Bd, _nan(A, n), ready)
    with pytest.raises(Exception, match="workspace too small"):
        ops.spmm(Ad, Bd, _nan(A, n), _cfg(), torch.empty(256, dtype=torch.uint8, device="cuda"))
    C = _nan(A, n)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            ops.spmm(Ad, Bd, C, _cfg(), stream=s)
        for _ in range(2):
            C.fill_(float("nan"))
            g.replay()
            s.synchronize()
            assert torch.equal(C, want)


def test_small_products_need_no_workspace(cuda):
    """Below 1M nonzeros a caller's workspace of any size, and a prepared partition without one, stay
    accepted."""
    A = CASES["edges"]
    B = synth.dense(A.K, 24, seed=5)
    Ad, Bd = dev(A), torch.from_numpy(B).cuda()
    ws = torch.empty(256, dtype=torch.uint8, device="cuda")
    odd = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")[4:]  # not 256-byte aligned
    ops.spmm_partition(Ad, _nan(A, 24), _cfg(), ws)
    for C in (ops.spmm(Ad, Bd, _nan(A, 24), _cfg(), ws), ops.spmm(Ad, Bd, _nan(A, 24), _cfg(), odd),
              ops.spmm(Ad, Bd, _nan(A, 24), _cfg(N.FLAG_PARTITION_READY))):
        assert_spmm_close(C.cpu().numpy(), A, B)


@pytest.mark.parametrize("n", [8, 37, 64])
def test_unused_rows_of_b_do_not_reach_c(cuda, n):
    A = synth.random_csr(700, 400, 0.03, seed=3, p_empty=0.1)
    A.col[:] = np.maximum(A.col, 1)
    B = synth.dense(A.K, n, seed=4)
    bad = B.copy()
    bad[0, ::2], bad[0, 1::2] = np.inf, np.nan
    got = ops.spmm(dev(A), torch.from_numpy(bad).cuda(), _nan(A, n), _cfg())
    assert_spmm_close(got.cpu().numpy(), A, B)
