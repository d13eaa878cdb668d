"""Plans of rb_pr over uneven rows: when joined chunks apply, and what takes their place."""
import ctypes as C

import pytest

from segtaco_gb300 import native as N

LR = N.FLAG_LONG_ROWS


def tuned(L, M, nnz, n, dtype, longest, K=None):
    c = N.Config()
    c.schedule = N.RB_PR
    assert L.segtaco_autotune_heuristic(M, K or M, nnz, n, dtype, longest, C.byref(c)) == N.OK
    return c


def plan(L, M, nnz, n, dtype, cfg, K=None, ldb=None):
    out = C.create_string_buffer(256)
    assert L.segtaco_spmm_plan_name(M, K or M, nnz, n, dtype, None, ldb or n, C.byref(cfg), out, 256) == N.OK
    return out.value.decode()


def workspace(L, M, nnz, n, dtype, cfg, K=None):
    out = C.c_size_t()
    assert L.segtaco_spmm_workspace_size(M, K or M, nnz, n, dtype, C.byref(cfg), C.byref(out)) == N.OK
    return out.value


@pytest.mark.parametrize("threshold,joined", [(0, True), (512, True), (300, False), (4000, False)])
def test_an_explicit_threshold_asks_for_pieces(native_lib, threshold, joined):
    c = N.Config.make(schedule="rb_pr", depth=8, flags=LR, items_per_unit=threshold)
    name = plan(native_lib, 100_000, 1_200_000, 64, N.F32, c)
    assert (" walk=7 " in name) == joined and name.startswith("rb_pr pieces ") != joined
    # below 1M nonzeros no rows are taken out and the threshold says nothing
    assert " walk=7 " in plan(native_lib, 50_000, 600_000, 64, N.F32, c)


@pytest.mark.parametrize("M,n,dtype,V,W", [(400_000, 64, N.F32, 8, 32), (400_000, 128, N.F32, 8, 32),
                                           (100_000, 64, N.F32, 4, 64), (100_000, 128, N.F32, 8, 32),
                                           (100_000, 128, N.BF16, 8, 128), (400_000, 128, N.BF16, 16, 64)])
def test_pieces_of_a_joined_configuration_keep_their_lanes(native_lib, M, n, dtype, V, W):
    """Where joined chunks cannot run (here: a row pitch of 4 GB) the tuned configuration leads to the
    pieces with the lanes they are the fastest with."""
    L, nnz = native_lib, 12 * M
    c = tuned(L, M, nnz, n, dtype, 700)
    assert " walk=7 " in plan(L, M, nnz, n, dtype, c)
    name = plan(L, M, nnz, n, dtype, c, ldb=1 << 31)
    assert name.startswith("rb_pr pieces V=%d " % V) and " W=%d " % W in name, name


@pytest.mark.parametrize("dtype", [N.F32, N.BF16])
@pytest.mark.parametrize("n", [4, 12, 16, 20, 36, 37, 48, 60, 64])
def test_the_pieces_slab_leaves_the_chunks_as_they_are(native_lib, dtype, n):
    L, M = native_lib, 60_000
    c = tuned(L, M, 12 * M * 2, n, dtype, 700)
    bare = N.Config.make(schedule="rb_pr", depth=8, flags=LR)
    a, b = plan(L, M, 24 * M, n, dtype, c), plan(L, M, 24 * M, n, dtype, bare)
    assert " walk=7 " in a and a.split(" rows_per_unit")[0] == b.split(" rows_per_unit")[0]


def test_large_sums_give_way_to_pieces(native_lib):
    """Two rows of N sums per chunk are no more than 64 MB where rows are long and N <= 256."""
    L = native_lib
    c = N.Config.make(schedule="rb_pr", depth=8, flags=LR)
    for M, mean, n, joined in ((233_000, 500, 128, False), (50_000, 1500, 64, False), (200_000, 100, 256, False),
                               (200_000, 100, 128, True), (233_000, 500, 512, True), (400_000, 20, 256, True)):
        name = plan(L, M, M * mean, n, N.F32, c, K=200_000)
        assert (" walk=7 " in name) == joined, name
        ws = workspace(L, M, M * mean, n, N.F32, c, K=200_000)
        if not joined:
            assert name.startswith("rb_pr pieces ") and ws < 64 << 20
