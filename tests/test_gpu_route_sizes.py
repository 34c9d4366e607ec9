"""Routing sort on both sides of its block-size rule (tokens, and experts against the SM count) against the oracle's sort: steps
that end inside a block, slot counts with and without vector loads, strided ids, experts without tokens."""
import numpy as np
import pytest
import torch

from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [255, 1023, 1024, 2500])
@pytest.mark.parametrize("E, k", [(16, 8), (160, 8), (40, 3)])
@pytest.mark.parametrize("idt", [torch.int32, torch.int64])
def test_route(T, E, k, idt):
    from orin_qwen_lossless_b200 import ops
    ops.init()
    ids = np.random.default_rng(T + E).random((T, E)).argsort(axis=1)[:, :k].astype(np.int64)
    ids[ids == 7] = 1 << 20    # no expert: routed nowhere
    want = o.route(ids, E, 1, 1)
    dev = torch.from_numpy(ids).to(idt).cuda()
    wide = torch.empty(T, k + 5, dtype=idt, device="cuda")
    wide[:, :k] = dev
    n = want[2][-1]
    for given in (dev, wide[:, :k]):
        got = [t.cpu().numpy() for t in ops.moe_route(given, E, False)]
        assert np.array_equal(got[2], want[2])
        assert np.array_equal(got[0][:n], want[0][:n]) and np.array_equal(got[1][:n], want[1][:n])
