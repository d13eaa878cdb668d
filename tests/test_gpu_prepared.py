"""A prepared partition (segtaco_spmm_partition, SEGTACO_FLAG_PARTITION_READY) followed by a product
whose B takes another plan than the partition could know: a row pitch of 4 GB, or a B that allows no
16-byte loads.  The product then makes what it needs itself."""
import numpy as np
import pytest
import torch

from gpu_util import assert_spmm_close, dev, spmm_ref
from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu

LR, READY = N.FLAG_LONG_ROWS, N.FLAG_PARTITION_READY


def _prepared(A, Bd, **cfg):
    Ad = dev(A)
    flags = cfg.pop("flags", 0)
    C = torch.full((A.M, Bd.shape[1]), float("nan"), device="cuda")
    ws = torch.full((64 << 20,), 0xff, dtype=torch.uint8, device="cuda")
    ops.spmm_partition(Ad, C, N.Config.make(flags=flags, **cfg), ws)
    ops.spmm(Ad, Bd, C, N.Config.make(flags=flags | READY, **cfg), ws)
    return C.cpu().numpy()


def test_row_pitch_of_4_gb(cuda):
    """Joined chunks need nothing prepared; a pitch of 4 GB takes the pieces, which do."""
    rng = np.random.default_rng(1)
    lens = np.r_[np.full(1500, 700), np.full(3000, 3)]
    ptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    nnz, n = int(ptr[-1]), 32
    A = synth.CSR(ptr, rng.integers(0, 3, nnz).astype(np.int32),
                  rng.uniform(-1, 1, nnz).astype(np.float32), len(lens), 3)
    B = synth.dense(3, n, seed=2)
    pitch = 1 << 30
    Bd = torch.empty(2 * pitch + n, device="cuda").as_strided((3, n), (pitch, 1))
    Bd.copy_(torch.from_numpy(B))
    assert_spmm_close(_prepared(A, Bd, schedule="rb_pr", depth=8, flags=LR), A, B)


@pytest.mark.parametrize("cfg", [dict(schedule="rb_pr", flags=LR), dict(schedule="rb_pr", depth=8, flags=LR),
                                 dict(schedule="eb_pr", flags=N.FLAG_SLOT_WALK)],
                         ids=["pieces", "joined", "slot_walk"])
def test_b_without_16_byte_rows(cuda, cfg):
    A = synth.power_law(60_000, 50_000, 1.8, 40_000, 0.02, seed=35)  # 1.09M nonzeros
    B = synth.dense(A.K, 33, seed=3)
    Bd = torch.from_numpy(B).cuda()[:, 1:]
    host = np.ascontiguousarray(B[:, 1:])
    assert_spmm_close(_prepared(A, Bd, **dict(cfg)), A, host, ref=spmm_ref(A, host))


@pytest.mark.parametrize("n", [40, 64, 200])
def test_large_sums_run_as_pieces(cuda, n):
    """Rows of 100 nonzeros and more whose joined sums would pass 64 MB: the size query, the partition and
    the product agree on the pieces (n = 200); below, on joined chunks."""
    rng = np.random.default_rng(n)
    lens = np.minimum(rng.lognormal(np.log(450.0) - 0.5, 1.0, 50_000).astype(np.int64), 20_000)
    ptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    K = 2000
    A = synth.CSR(ptr, rng.integers(0, K, int(ptr[-1])).astype(np.int32),
                  rng.uniform(-1, 1, int(ptr[-1])).astype(np.float32), len(lens), K)
    B = synth.dense(K, n, seed=n)
    Ad, Bd = dev(A), torch.from_numpy(B).cuda()
    cfg = N.Config.make(schedule="rb_pr", depth=8, flags=LR)
    assert ops.plan_name(Ad, Bd, cfg).startswith("rb_pr pieces ") == (n == 200)
    ref = spmm_ref(A, B)
    want = ops.spmm(Ad, Bd, None, cfg)
    assert_spmm_close(want.cpu().numpy(), A, B, ref=ref)
    ws = torch.full((ops.spmm_workspace_size(Ad, n, N.F32, cfg),), 0xff, dtype=torch.uint8, device="cuda")
    C = torch.full((A.M, n), float("nan"), device="cuda")
    ops.spmm_partition(Ad, C, cfg, ws)
    ops.spmm(Ad, Bd, C, N.Config.make(schedule="rb_pr", depth=8, flags=LR | READY), ws)
    assert torch.equal(C, want)
