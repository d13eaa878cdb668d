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
