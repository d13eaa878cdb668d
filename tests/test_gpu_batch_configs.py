"""A batch made from the configurations that another batch reports is that batch again."""
import numpy as np
import pytest
import torch

from gpu_util import assert_spmm_close, dev, to_torch_bf16
from segtaco_gb300 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
def test_reported_configs_rebuild_the_batch(cuda, bf16):
    mats = [synth.power_law(m, m, 1.8, 3000, 0.02, seed=m) for m in (3000, 9000, 30_000)]
    mats += [synth.random_csr(2000, 1500, 0.01, seed=5), synth.banded_plus_random(4000, 16, 4, seed=6)]
    items, refs = [], []
    for k, A in enumerate(mats):
        for n in (16, 32, 64, 128, 37):
            B = synth.dense(A.K, n, seed=k)
            bits = synth.to_bf16_bits(B)
            refs.append((A, bits if bf16 else B))
            items.append((dev(A), to_torch_bf16(bits) if bf16 else torch.from_numpy(B).cuda(),
                          torch.full((A.M, n), float("nan"), device="cuda")))
    first = ops.Batch(items)
    groups, total, configs = first.info()
    again = ops.Batch(items, configs)
    g2, t2, c2 = again.info()
    assert (groups, total) == (g2, t2)
    for a, b in zip(configs, c2):
        assert bytes(a) == bytes(b)
    again.run()
    for (A, B), (_, _, C) in zip(refs, items):
        assert_spmm_close(C.cpu().numpy(), A, B, bf16=bf16)
