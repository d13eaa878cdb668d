"""The split walk of merge-path chunks (eb_sr, eb_pr): every lane shape, chunk sizes down to one item,
rows that span runs and chunks, empty rows, and positions outside a chunk that must not touch C."""
import numpy as np
import pytest
import torch

from gpu_util import assert_spmm_close, dev, small_cases, spmm_ref, to_torch_bf16
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu

CASES = small_cases()


def _dense(A, n, pad, bf16, seed):
    """B (K x n) with a row pitch of n + pad elements, and its host values."""
    B = synth.dense(A.K, n + pad, seed)
    Bd = to_torch_bf16(synth.to_bf16_bits(B)) if bf16 else torch.from_numpy(B).cuda()
    host = synth.to_bf16_bits(B) if bf16 else B
    return np.ascontiguousarray(host[:, :n]), Bd[:, :n]


def _run(A, Bd, cfg):
    Ad = dev(A)
    assert " walk=5 " in ops.plan_name(Ad, Bd, cfg), ops.plan_name(Ad, Bd, cfg)
    C = torch.full((A.M, Bd.shape[1]), float("nan"), device="cuda")
    return ops.spmm(Ad, Bd, C, cfg).cpu().numpy()


# N and pitch: chunks of 16 bytes on 1 .. 32 lanes, bf16's 8-byte chunks, 2- and 1-element chunks with
# one to four of them per lane, partly idle lanes, and a second, narrower slab
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n,pad", [(4, 0), (8, 0), (16, 0), (20, 0), (32, 0), (64, 0), (100, 0),
                                   (128, 0), (132, 4), (1, 0), (2, 0), (2, 1), (3, 0), (5, 0),
                                   (6, 0), (7, 0), (9, 0), (14, 0), (17, 0), (25, 0), (33, 0),
                                   (37, 0), (46, 0), (50, 0), (63, 0), (64, 1), (65, 0), (97, 0),
                                   (126, 0), (127, 0), (129, 0), (200, 2)])
def test_lane_shapes(cuda, n, pad, bf16):
    A = CASES["powerlaw"]
    host, Bd = _dense(A, n, pad, bf16, seed=n + 7 * pad)
    assert_spmm_close(_run(A, Bd, N.Config.make(schedule="eb_pr")), A, host, bf16)


@pytest.mark.parametrize("items", [1, 2, 3, 7, 31, 64, 100, 512])
@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("sched,n", [("eb_pr", 36), ("eb_sr", 128), ("eb_sr", 8), ("eb_pr", 13)])
def test_chunk_sizes(cuda, name, items, sched, n):
    A = CASES[name]
    B = synth.dense(A.K, n, seed=items)
    cfg = N.Config.make(schedule=sched, items_per_unit=items)
    assert_spmm_close(_run(A, torch.from_numpy(B).cuda(), cfg), A, B, ref=spmm_ref(A, B))


@pytest.mark.parametrize("n", [8, 33, 64, 128])
def test_unused_rows_of_b_do_not_reach_c(cuda, n):
    """Positions outside a chunk read B row 0: infinities and NaN there stay out of C."""
    A = synth.random_csr(700, 400, 0.03, seed=3, p_empty=0.1)
    A.col[:] = np.maximum(A.col, 1)
    B = synth.dense(A.K, n, seed=4)
    ref = spmm_ref(A, B)
    bad = B.copy()
    bad[0, ::2], bad[0, 1::2] = np.inf, np.nan
    for items in (5, 64, 256):
        cfg = N.Config.make(schedule="eb_pr", items_per_unit=items)
        assert_spmm_close(_run(A, torch.from_numpy(bad).cuda(), cfg), A, B, ref=ref)


@pytest.mark.parametrize("rows,n", [(1, 8), (2, 33), (700, 64), (16_384, 128), (16_385, 128)])
def test_edges_searched_or_partitioned(cuda, rows, n):
    """Up to 2M elements of C the kernel searches its chunk edges; with prepared partition arrays, and
    past that, it reads them.  The same product, also into a strided C, with the padding left alone."""
    A = synth.random_csr(rows, 300, 0.02, seed=rows, p_empty=0.2, long_rows={0: 250, rows - 1: 300})
    B = synth.dense(A.K, n, seed=1)
    ref = spmm_ref(A, B)
    Ad, Bd = dev(A), torch.from_numpy(B).cuda()
    cfg = N.Config.make(schedule="eb_sr")
    ws = torch.empty(ops.spmm_workspace_size(Ad, n, N.F32, cfg), dtype=torch.uint8, device="cuda")
    wide = torch.full((A.M, n + 4), 7.0, device="cuda")
    for C in (torch.full((A.M, n), float("nan"), device="cuda"), wide[:, :n]):
        ops.spmm(Ad, Bd, C, cfg)
        assert_spmm_close(C.cpu().numpy(), A, B, ref=ref)
        ops.spmm_partition(Ad, C, cfg, ws)
        ready = N.Config.make(schedule="eb_sr", flags=N.FLAG_PARTITION_READY)
        ops.spmm(Ad, Bd, C, ready, ws)
        assert_spmm_close(C.cpu().numpy(), A, B, ref=ref)
    assert (wide[:, n:] == 7.0).all()


@pytest.mark.parametrize("n,pad,bf16", [(64, 0, False), (37, 0, False), (126, 0, True), (40, 4, True)])
def test_batches_of_the_split_walk(cuda, n, pad, bf16):
    mats = list(CASES.values()) + [synth.random_csr(50, 60, 0.0, seed=9)]
    items, want = [], []
    for k, A in enumerate(mats):
        host, Bd = _dense(A, n, pad, bf16, seed=k)
        items.append((dev(A), Bd, torch.full((A.M, n), float("nan"), device="cuda")))
        want.append((A, host))
    batch = ops.Batch(items, [N.Config.make(schedule="eb_pr")] * len(items))
    for graph in (False, True):
        for _, _, C in items:
            C.fill_(float("nan"))
        batch.run(graph=graph)
        torch.cuda.synchronize()
        for (A, host), (_, _, C) in zip(want, items):
            assert_spmm_close(C.cpu().numpy(), A, host, bf16)
    batch.close()
