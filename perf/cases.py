"""What the framework is timed on: its public operations over the range in which they are used.

A case names an operation, its sizes, the structure of the sparse matrix, the dense type and whether
the caller tuned the call (a caller that repeats a product keeps a configuration, a workspace and an
output; one that calls once passes none).  The listed cases:

* ``spmm_call_1k_n16``        one untuned product with a small matrix of the uneven pool: call latency
* ``spmm_uniform16_rb_sr_n32`` the plain fp32 product of 16,384 x 16,384, 16 per row, sequential row blocks
* ``spmm_ragged_n37``         an untuned rectangular product whose dense width allows no vector load
* ``spmm_power_law_n128``     the large power-law product (1M x 1M, Zipf rows), the schedule tuned
* ``spmm_power_law_eb_sr_n64`` a mid-size power-law product, sequential reduction over equal chunks
* ``spmm_banded_bf16_n64``    the banded matrix with a bf16 dense operand
* ``spmv_power_law``          the large power-law matrix times a vector, as an iterative solver calls it
* ``spmspv_power_law``        a power-law matrix by columns times a sparse vector, 10 % of it set (a frontier)
* ``sddmm_banded_d64``        sampled dense-dense product on the banded pattern, fp32 factors, tuned
* ``sddmm_power_law_bf16_d128`` the same on a power-law pattern (edge scores), bf16 factors, untuned
* ``batch_pool_48``           48 uneven products planned once and run together as a graph
* ``dropin_eb_sr_n64``        a segTACO-named call on host buffers, copies included

``draw`` spreads over the same operations, structures, types and options between the smallest and the
largest of these sizes.  Inputs are made on the GPU from the seed: uniform columns and values, rows
sorted and distinct, row lengths by structure.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from segtaco_gb300 import native, ops, taco

ZIPF_S, ZIPF_CAP, P_EMPTY = 1.8, 50_000, 0.02
LOG_MEAN, LOG_SIGMA = 12.0, 1.0
HALF_BAND, OFF_BAND = 32, 8
POOL_NS = (16, 32, 64, 128)


def listed():
    return [
        dict(name="spmm_call_1k_n16", op="spmm", structure="lognormal", M=1000, K=1000, N=16,
             dtype="f32", tuned=False, schedule="auto"),
        dict(name="spmm_uniform16_rb_sr_n32", op="spmm", structure="uniform16", M=16_384, K=16_384,
             N=32, dtype="f32", tuned=True, schedule="rb_sr"),
        dict(name="spmm_ragged_n37", op="spmm", structure="lognormal", M=77_777, K=50_001, N=37,
             dtype="f32", tuned=False, schedule="auto"),
        dict(name="spmm_power_law_n128", op="spmm", structure="zipf", M=1_000_000, K=1_000_000,
             N=128, dtype="f32", tuned=True, schedule="auto"),
        dict(name="spmm_power_law_eb_sr_n64", op="spmm", structure="zipf", M=250_000, K=250_000,
             N=64, dtype="f32", tuned=True, schedule="eb_sr"),
        dict(name="spmm_banded_bf16_n64", op="spmm", structure="banded", M=262_144, K=262_144, N=64,
             dtype="bf16", tuned=True, schedule="auto"),
        dict(name="spmv_power_law", op="spmv", structure="zipf", M=1_000_000, K=1_000_000),
        dict(name="spmspv_power_law", op="spmspv", structure="zipf", M=1_000_000, K=1_000_000,
             nx=100_000),
        dict(name="sddmm_banded_d64", op="sddmm", structure="banded", M=262_144, K=262_144, D=64,
             dtype="f32", tuned=True),
        dict(name="sddmm_power_law_bf16_d128", op="sddmm", structure="zipf", M=300_000, K=300_000,
             D=128, dtype="bf16", tuned=False),
        dict(name="batch_pool_48", op="batch", count=48, first=0),
        dict(name="dropin_eb_sr_n64", op="dropin", structure="lognormal", M=100_000, K=100_000,
             N=64, kernel="spmm_eb_sr"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi):
    """A structure and a size of it: square three times in four, banded ones always and smaller."""
    structure = rng.choice(("lognormal", "uniform16", "zipf", "banded"))
    M = _log_int(rng, lo, min(hi, 200_000) if structure == "banded" else hi)
    K = M if structure == "banded" or rng.random() < 0.75 else _log_int(rng, lo, hi)
    return dict(structure=structure, M=M, K=K)


def draw(rng):
    op = rng.choice(("spmm",) * 6 + ("sddmm",) * 3 + ("spmv", "spmspv", "batch", "dropin"))
    if op == "batch":
        return dict(op=op, count=rng.randint(8, 48), first=rng.randint(1, 10_000))
    if op == "dropin":
        case = dict(op=op, **_shape(rng, 1000, 80_000))
        case["N"] = rng.choice((16, 32, 64, rng.randint(1, 64)))
        case["kernel"] = rng.choice(("spmm_rb_sr", "spmm_rb_pr", "spmm_eb_sr", "spmm_eb_pr"))
        return case
    case = dict(op=op, **_shape(rng, 1000, 400_000))
    if op == "spmspv":
        case["nx"] = max(1, int(case["K"] * rng.choice((0.001, 0.01, 0.1, rng.uniform(0.001, 0.3)))))
    if op in ("spmm", "sddmm"):
        width = rng.choice((8, 16, 32, 64, 128, rng.randint(1, 128), rng.randint(1, 128)))
        case["N" if op == "spmm" else "D"] = width
        case["dtype"] = rng.choice(("f32", "f32", "bf16"))
        case["tuned"] = rng.random() < 0.6
    if op == "spmm":
        case["schedule"] = "auto" if not case["tuned"] else rng.choice(
            ("auto", "auto", "rb_sr", "rb_pr", "eb_sr", "eb_pr"))
    return case


# ---- inputs ------------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _uniform(shape, g, dtype=torch.float32):
    return torch.rand(shape, generator=g, device="cuda").mul_(2.0).sub_(1.0).to(dtype)


def _zipf_cdf(cap):
    w = np.arange(1, cap + 1, dtype=np.float64) ** -ZIPF_S
    return np.cumsum(w) / w.sum()


def _lengths(structure, M, K, g):
    """Nonzeros of each row: drawn from the sizes alone and dealt to the rows by the seed, so that
    matrices of the same sizes have the same number of nonzeros."""
    fixed = _generator(M * 31 + K)
    if structure == "zipf":
        cdf = torch.from_numpy(_zipf_cdf(min(ZIPF_CAP, K))).cuda()
        u = torch.rand(M, generator=fixed, device="cuda", dtype=torch.float64)
        n = torch.searchsorted(cdf, u).clamp_(max=cdf.numel() - 1) + 1
        n.masked_fill_(torch.rand(M, generator=fixed, device="cuda") < P_EMPTY, 0)
    elif structure == "uniform16":
        return torch.full((M,), min(16, K), dtype=torch.int64, device="cuda")
    else:
        z = torch.randn(M, generator=fixed, device="cuda", dtype=torch.float64)
        n = torch.exp(z * LOG_SIGMA + math.log(LOG_MEAN) - LOG_SIGMA ** 2 / 2).round_()
        n = n.clamp_(0, 64 if structure == "blockdiag" else K).long()
    return n[torch.randperm(M, generator=g, device="cuda")]


def _csr(structure, M, K, g):
    i = torch.arange(M, device="cuda")
    if structure == "banded":
        n = torch.full((M,), OFF_BAND, dtype=torch.int64, device="cuda")
    else:
        n = _lengths(structure, M, K, g)
    low, width = torch.zeros_like(i), torch.full_like(i, K)
    if structure == "blockdiag":  # blocks of 64 x 64 on the diagonal
        low = i // 64 * 64
        width = (K - low).clamp(max=64)
        n = torch.minimum(n, width)
    elif structure == "banded":  # the columns outside the band, which is put back below
        first = (i - HALF_BAND).clamp(min=0, max=K)
        inside = (i + HALF_BAND + 1).clamp(max=K) - first
        width = K - inside
    rows = torch.repeat_interleave(i, n)
    k = torch.arange(rows.numel(), device="cuda") - (torch.cumsum(n, 0) - n)[rows]
    if structure == "band":  # each row's nonzeros side by side around the diagonal
        cols = rows - n[rows] // 2 + k
        keep = (cols >= 0) & (cols < K)
        rows, cols = rows[keep], cols[keep]
    else:  # one column at random in each of the row's n equal parts: distinct and in order
        a = k * width[rows] // n[rows]
        b = (k + 1) * width[rows] // n[rows]
        cols = a + torch.randint(0, 1 << 40, (rows.numel(),), generator=g, device="cuda") % (b - a)
        cols += low[rows]
    if structure == "banded":
        cols += torch.where(cols >= first[rows], inside[rows], 0)
        band = i[:, None] + torch.arange(-HALF_BAND, HALF_BAND + 1, device="cuda")
        keys = (i[:, None] * K + band)[(band >= 0) & (band < K)]
        keys = torch.sort(torch.cat([keys, rows * K + cols]))[0]
        rows = keys // K
        cols = keys - rows * K
    ptr = torch.zeros(M + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=M), 0)
    return ops.DeviceCSR(ptr, cols.int(), _uniform(cols.numel(), g), M, K)


def _pool(case):
    """Sizes, structures and dense widths of a batch's matrices, the same for every seed."""
    for m in range(case["count"]):
        rng = random.Random(case["first"] * 1009 + m)
        yield (_log_int(rng, 1000, 200_000), rng.choice(("lognormal", "band", "blockdiag", "zipf")),
               rng.choice(POOL_NS))


def _inputs(case, seed):
    """The operands, on the GPU: what prepare() hands to run() and exact() to plain torch."""
    g = _generator(seed)
    op = case["op"]
    if op == "batch":
        items = []
        for M, structure, N in _pool(case):
            A = _csr(structure, M, M, g)
            items.append((A, _uniform((M, N), g)))
        return items
    if op == "spmspv":  # the matrix by columns: its K columns are the rows of the CSR
        At = _csr(case["structure"], case["K"], case["M"], g)
        idx = torch.randperm(case["K"], generator=g, device="cuda")[:case["nx"]].sort()[0].int()
        return At, idx, _uniform(case["nx"], g)
    A = _csr(case["structure"], case["M"], case["K"], g)
    if op == "spmv":
        return A, _uniform(case["K"], g)
    dtype = torch.bfloat16 if case.get("dtype") == "bf16" else torch.float32
    if op == "sddmm":
        return A, _uniform((case["M"], case["D"]), g, dtype), _uniform((case["K"], case["D"]), g, dtype)
    return A, _uniform((case["K"], case["N"]), g, dtype)


# ---- the calls ---------------------------------------------------------------------------------


def prepare(case, seed):
    op, x = case["op"], _inputs(case, seed)
    state = {"op": op, "case": case, "in": x}
    if op == "spmm" and case["tuned"]:
        A, B = x
        schedule = native.SCHEDULES.get(case["schedule"], native.AUTO)
        dt = native.BF16 if case["dtype"] == "bf16" else native.F32
        cfg = ops.autotune(A, case["N"], dt, schedule)
        size = ops.spmm_workspace_size(A, case["N"], dt, cfg)
        state.update(cfg=cfg, C=torch.empty((A.M, case["N"]), device="cuda"),
                     ws=torch.empty(size, dtype=torch.uint8, device="cuda") if size else None)
    elif op == "sddmm" and case["tuned"]:
        A, X, _ = x
        dt = native.BF16 if case["dtype"] == "bf16" else native.F32
        state.update(cfg=ops.sddmm_autotune(A, case["D"], dt), out=torch.empty(A.nnz, device="cuda"))
    elif op == "spmv":
        A = x[0]
        state.update(y=torch.empty(A.M, device="cuda"),
                     ws=torch.empty(ops.spmv_workspace_size(A), dtype=torch.uint8, device="cuda"))
    elif op == "batch":
        outs = [torch.empty((A.M, B.shape[1]), device="cuda") for A, B in x]
        state.update(out=outs, batch=ops.Batch([(A, B, C) for (A, B), C in zip(x, outs)]))
    elif op == "dropin":
        A, B = x
        C = np.empty((A.M, case["N"]), np.float32)
        state["tensors"] = (taco.dense(C), taco.csr(A.row_ptr.cpu().numpy(), A.col.cpu().numpy(),
                                                    A.val.cpu().numpy(), A.M, A.K),
                            taco.dense(B.cpu().numpy()))
        state["C"] = C
        state["in"] = None
    return state


def run(state):
    op, x = state["op"], state["in"]
    if op == "spmm":
        A, B = x
        if "cfg" in state:
            return ops.spmm(A, B, state["C"], config=state["cfg"], workspace=state["ws"])
        return ops.spmm(A, B)
    if op == "sddmm":
        A, X, Y = x
        if "cfg" in state:
            return ops.sddmm(A, X, Y, out=state["out"], config=state["cfg"])
        return ops.sddmm(A, X, Y)
    if op == "spmv":
        return ops.spmv(x[0], x[1], state["y"], workspace=state["ws"])
    if op == "spmspv":
        At, idx, val = x
        return ops.spmspv(At, idx, val, state["case"]["M"])
    if op == "batch":
        state["batch"].run(graph=True)
        return state["out"]
    (tC, _), (tA, _), (tB, _) = state["tensors"]
    taco.call(state["case"]["kernel"], tC, tA, tB)
    return state["C"]


# ---- what a pass cannot do without -------------------------------------------------------------


def _mean_nnz(structure, K):
    """Expected nonzeros per row."""
    if structure == "zipf":
        cap = min(ZIPF_CAP, K)
        w = np.arange(1, cap + 1, dtype=np.float64) ** -ZIPF_S
        return float((w * np.arange(1, cap + 1)).sum() / w.sum()) * (1.0 - P_EMPTY)
    if structure == "banded":
        return min(2 * HALF_BAND + 1 + OFF_BAND, K)
    return min(16 if structure == "uniform16" else LOG_MEAN, K)


def _spmm_work(M, K, N, nnz, esz):
    return nnz * 8 + (M + 1) * 4 + K * N * esz + M * N * 4, 2 * nnz * N


def work(case):
    op = case["op"]
    esz = 2 if case.get("dtype") == "bf16" else 4
    if op == "batch":
        parts = [_spmm_work(M, M, N, M * _mean_nnz(s, M), 4) for M, s, N in _pool(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    M, K = case["M"], case["K"]
    if op == "spmspv":
        nnz = case["nx"] * _mean_nnz(case["structure"], M)
        return {"bytes": case["nx"] * 16 + nnz * 8 + M * 4, "flops": 2 * nnz}
    nnz = M * _mean_nnz(case["structure"], K)
    if op == "sddmm":
        return {"bytes": nnz * 12 + (M + 1) * 4 + (M + K) * case["D"] * esz,
                "flops": 2 * nnz * case["D"]}
    b, f = _spmm_work(M, K, case.get("N", 1), nnz, esz)
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, without the library --------------------------------------------------


def _product(A, B):
    sparse = torch.sparse_csr_tensor(A.row_ptr, A.col, A.val.double(), (A.M, A.K),
                                     check_invariants=False)
    return sparse @ B.double()


def exact(case, seed):
    op, x = case["op"], _inputs(case, seed)
    if op == "batch":
        return [_product(A, B) for A, B in x]
    if op == "spmspv":
        At, idx, val = x
        n = (At.row_ptr[1:] - At.row_ptr[:-1]).long()
        xs = torch.zeros(At.M, dtype=torch.float64, device="cuda")
        xs[idx.long()] = val.double()
        terms = At.val.double() * torch.repeat_interleave(xs, n)
        y = torch.zeros(At.K, dtype=torch.float64, device="cuda")
        return y.index_add_(0, At.col.long(), terms)
    if op == "spmv":
        return _product(x[0], x[1][:, None])[:, 0]
    if op == "sddmm":
        A, X, Y = x
        n = (A.row_ptr[1:] - A.row_ptr[:-1]).long()
        rows = torch.repeat_interleave(torch.arange(A.M, device="cuda"), n)
        out = torch.empty(A.nnz, dtype=torch.float64, device="cuda")
        step = 1 << 20
        for p in range(0, A.nnz, step):
            q = slice(p, p + step)
            dots = (X[rows[q]].double() * Y[A.col[q].long()].double()).sum(1)
            out[q] = A.val[q].double() * dots
        return out
    C = _product(*x)
    return C.cpu().numpy() if op == "dropin" else C
