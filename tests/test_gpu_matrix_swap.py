"""Calls that read a matrix behind everything before them on the stream: the matrix is overwritten by a kernel right in front of
the call (as an in-place swap does), and the result is the new matrix's."""
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


def _two(ops, rows, K, R, cm=False, fo=False):
    """One device matrix to be overwritten, and two encodings of equal size to overwrite it with."""
    enc = []
    for seed in (1, 2):
        plane, aux, meta = ops.encode(to_bf16_tensor(o.weights_like(rows, K, rows + K + seed)), 3, R, cm, fo)
        enc.append((plane.cuda(), aux.cuda(), meta))
    n = max(a.numel() for _, a, _ in enc)
    enc = [(p, torch.nn.functional.pad(a, (0, n - a.numel())), m) for p, a, m in enc]
    return ops.Weight(enc[0][0].clone(), enc[0][1].clone(), enc[0][2]), enc


def _swap(w, to):
    for dst, src in ((w.plane, to[0]), (w.aux, to[1])):
        torch.bitwise_or(src, 0, out=dst)       # an elementwise kernel, not a copy


def _check(weights, call):
    got = []
    for i in (1, 0, 1):
        for w, enc in weights:
            _swap(w, enc[i])
        got.append(call([w for w, _ in weights]))
    torch.cuda.synchronize()
    for g, i in zip(got, (1, 0, 1)):
        assert torch.equal(g, call([type(w)(*enc[i]) for w, enc in weights]))


def test_row_gather_and_draft():
    from orin_qwen_lossless_b200 import ops
    ops.init()
    ids = torch.arange(0, 512, 7, device="cuda", dtype=torch.int32)
    rows = _two(ops, 4096, 2048, 16)
    _check([rows], lambda ws: ops.get_rows(ids, ws[0]))
    head = ops.DraftHead(2, *ops.int2_quantize(to_bf16_tensor(o.weights_like(4096, 2048, 3)).cuda()), 32)
    x = torch.randn(2, 2048, device="cuda").to(torch.bfloat16)
    _check([rows], lambda ws: ops.draft_logits(x, ws[0], head, 4096))


@pytest.mark.parametrize("fo", [False, True])
def test_batched_product(fo):
    from orin_qwen_lossless_b200 import ops
    ops.init()
    E, T = 8, 96
    gate, up = (_two(ops, E * 512, 2048, 16 if fo else 8, not fo, fo) for _ in range(2))
    x = torch.randn(T, 2048, device="cuda").to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, device="cuda")[:4] for _ in range(T)]).to(torch.int32)
    route = ops.moe_route(ids, E, False)
    if not fo:
        ops.ensure_workspace((gate[0], up[0]))
    try:
        _check([gate, up], lambda ws: ops.moe_mm_ids(x, ids, ws[0], E, up=ws[1], out_dtype=torch.bfloat16, route=route))
    finally:
        ops.set_workspace(None)
