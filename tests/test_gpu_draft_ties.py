"""Candidates of scores that are the same in many rows: the lowest rows of those, on the path of the short lists (up to 8192 rows) and on the
cluster's, in about the time that scores without ties take."""
import numpy as np
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


def _head(ops, rows, cands):
    src = to_bf16_tensor(o.weights_like(rows, 2048, rows))
    return ops.upload(*ops.encode(src, ops.FMT_HUFPAIR, 16, False), "cuda"), ops.DraftHead(2, *ops.int2_quantize(src.cuda()), cands)


@pytest.mark.parametrize("rows", [144, 2048, 8192, 8208, 62080])
@pytest.mark.parametrize("cands", [1, 128])
def test_all_alike(rows, cands):
    from orin_qwen_lossless_b200 import ops
    ops.init()
    w, head = _head(ops, rows, cands)
    h = torch.zeros(3, 2048, device="cuda", dtype=torch.bfloat16)
    h[1] = torch.randn(2048, device="cuda")
    y = ops.draft_logits(h, w, head, rows + 5)
    for t in (0, 2):
        assert torch.equal(y[t].isfinite().nonzero()[:, 0].cpu(), torch.arange(cands)), t
    assert int(y[1].isfinite().sum()) == cands


@pytest.mark.parametrize("rows,values", [(4096, 1), (4096, 3), (8192, 40), (1024, 500)])
def test_few_values(rows, values):
    """Scores of `values` different values: rows of the 2-bit copy that are the same."""
    from orin_qwen_lossless_b200 import ops
    ops.init()
    w, head = _head(ops, rows, 100)
    pick = torch.from_numpy(np.random.default_rng(rows).integers(0, values, rows)).cuda()
    head = ops.DraftHead(2, head.q[pick].contiguous(), head.s[pick].contiguous(), 100)
    h = torch.randn(2, 2048, device="cuda").to(torch.bfloat16)
    scores = head.scores(h).cpu().numpy()
    y = ops.draft_logits(h, w, head, rows)
    for t in range(2):
        want = np.lexsort((np.arange(rows), -scores[t].astype(np.float64)))[:100]
        assert sorted(want) == y[t].isfinite().nonzero()[:, 0].tolist()


def test_ties_cost_no_more_than_scores_without():
    """A rank by comparison with every entry took 2109 us of 8192 rows, against 22 without ties."""
    from orin_qwen_lossless_b200 import ops
    ops.init()
    w, head = _head(ops, 8192, 128)
    took = []
    for h in (torch.randn(1, 2048, device="cuda").to(torch.bfloat16), torch.zeros(1, 2048, device="cuda", dtype=torch.bfloat16)):
        runs = []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(8):
                ops.draft_logits(h, w, head, 8192)
            b.record()
            b.synchronize()
            runs.append(a.elapsed_time(b))
        took.append(sorted(runs)[4])
    assert took[1] < 4 * took[0]
