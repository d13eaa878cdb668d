"""Scratch of calls that bring no workspace: kept by the library between calls, shared by threads
and streams, given back by segtaco_taco_release, and part of the graph when a call is captured."""
import threading

import pytest
import torch

from segtaco_gb300 import native as N
from segtaco_gb300 import ops, synth

from gpu_util import assert_spmm_close

pytestmark = pytest.mark.gpu


def _problem(seed, n):
    A = synth.power_law(3000, 2500, 1.8, 1500, 0.02, seed=seed)
    B = synth.dense(A.K, n, seed=seed + 1)
    return A, B, ops.DeviceCSR.from_host(A), torch.from_numpy(B).cuda()


def test_threads_and_streams_share_the_scratch():
    problems = [_problem(s, n) for s, n in ((1, 16), (2, 33), (3, 64))]
    results = [[] for _ in problems]

    def work(i):
        _, _, Ad, Bd = problems[i]
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.default_stream())
        outs = [torch.full((Ad.M, Bd.shape[1]), float("nan"), device="cuda") for _ in range(8)]
        torch.cuda.synchronize()
        for C in outs:
            ops.spmm(Ad, Bd, C, stream=stream)
        stream.synchronize()
        results[i] = outs

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(problems))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (A, B, _, _), outs in zip(problems, results):
        assert len(outs) == 8
        for C in outs:
            assert_spmm_close(C.cpu().numpy(), A, B)


def test_release_and_capture():
    A, B, Ad, Bd = _problem(5, 32)
    ops.spmm(Ad, Bd)
    torch.cuda.synchronize()
    N.lib().segtaco_taco_release()
    assert_spmm_close(ops.spmm(Ad, Bd).cpu().numpy(), A, B)
    C = torch.full((A.M, 32), float("nan"), device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ops.spmm(Ad, Bd, C)
        for _ in range(3):
            C.fill_(float("nan"))
            graph.replay()
            stream.synchronize()
            assert_spmm_close(C.cpu().numpy(), A, B)
