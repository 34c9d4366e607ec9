"""Units cut into parts by marks: the same bits as without marks, whatever the marks hold (they are checked where they are used), at the
sizes where a part, a unit or a block begins: one to sixteen parts, several units to a block, a last block that is partly empty."""
import numpy as np
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu

# rows, K, R, chunk-major: parts of a unit = R K / 4096
SHAPES = [(16 * 5, 512, 16, False), (16 * 9, 1024, 16, False), (16 * 7, 2048, 16, False), (16 * 3, 4096, 16, False), (8 * 11, 2048, 8, False),
          (8 * 5, 4096, 8, False), (4 * 13, 2048, 4, False), (4 * 6, 4096, 4, False), (16 * 3, 1536, 16, False), (8 * 9, 2048, 8, True),
          (16 * 5, 1024, 16, True)]


@pytest.fixture(scope="module")
def ops():
    from orin_qwen_lossless_b200 import ops as m
    m.init()
    return m


def _made(ops, rows, K, R, cm, wide=False):
    bits = o.weights_like(rows, K, rows + K + R)
    if wide:    # exponents all over the range: codes of up to 12 bits, streams longer than a unit's buffer
        bits = (bits & 0x807F) | (np.random.default_rng(rows).integers(60, 124, bits.shape, dtype=np.uint16) << 7).astype(np.uint16)
    src = to_bf16_tensor(bits)
    enc = ops.encode(src, ops.FMT_HUFPAIR, R, cm)
    assert enc[2].format == ops.FMT_HUFPAIR
    return src, ops.upload(*enc, "cuda")


def _marks(ops, w):
    """The right marks, no marks that were ever written, marks that are wrong in one lane of one part, and marks of other streams."""
    good = w.marks.view(torch.int16)
    one = good.clone()
    one[good.numel() // 2 + 7] ^= 1
    last = good.clone()
    last[-1] += 64
    return [good, torch.zeros_like(good), torch.full_like(good, -1), torch.randint(-32768, 32767, good.shape, device="cuda").to(torch.int16), one, last, good.roll(32)]


@pytest.mark.parametrize("rows,K,R,cm", SHAPES)
@pytest.mark.parametrize("wide", [False, True])
def test_marks_change_nothing(ops, rows, K, R, cm, wide):
    src, w = _made(ops, rows, K, R, cm, wide)
    plain = ops.Weight(w.plane, w.aux, w.meta)
    parts = R * K // 4096
    assert w.marks.numel() == rows // R * (parts - 1) * 64 and plain.marks is None
    xs = [torch.randn(T, K, device="cuda").to(torch.bfloat16) for T in (1, 2, 3, 8)] + [torch.randn(2, K, device="cuda")]
    if K == 1536:
        xs = []         # reconstruction only: no product has this width
    want = [ops.mmv(x, plain) for x in xs]
    ids = torch.randperm(rows)[:300]
    for marks in _marks(ops, w):
        w.marks = marks.view(torch.uint8)
        if not cm:
            assert torch.equal(ops.get_rows(ids.cuda(), w).cpu().view(torch.int16), src[ids].view(torch.int16))
            assert torch.equal(ops.get_rows(ids.int().cuda(), w, torch.float32).cpu(), src[ids].float())
        assert torch.equal(ops.dequant(w).cpu().view(torch.int16), src.view(torch.int16))
        assert torch.equal(ops.dequant(w, R, rows - 2 * R).cpu().view(torch.int16), src[R:rows - R].view(torch.int16))
        for x, y in zip(xs, want):
            assert torch.equal(ops.mmv(x, w), y)
    assert ops.fault_status() == 0


@pytest.mark.parametrize("T", [1, 3, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_decode_step_of_experts(ops, T, dtype):
    E, k, lo, n = 12, 4, 3, 7       # a slice of the experts: slots routed elsewhere are zeros
    ws = [_made(ops, n * r, K, R, cm)[1] for r, K, R, cm in ((512, 2048, 8, True), (512, 2048, 8, True), (2048 - 16, 512, 16, False))]
    x = torch.randn(T, 2048, device="cuda").to(dtype)
    ids = torch.stack([torch.randperm(E, device="cuda")[:k] for _ in range(T)]).to(torch.int32)
    weights = torch.rand(T, k, device="cuda")
    routed = (ids - lo).clamp(0, n - 1)

    def call():
        step = ops.moe_decode(x, *ws, E, k, topk_weights=weights, topk_ids=ids, expert_lo=lo, n_experts_local=n)[0]
        return [step, ops.mmv(x, ws[0], routed, 512), ops.mmv(torch.randn(T, k, 512, generator=torch.Generator().manual_seed(1)).cuda().to(dtype), ws[2], routed, 2032)]

    good, ws = ws, [ops.Weight(w.plane, w.aux, w.meta) for w in ws]
    want = call()
    for marks in zip(*(_marks(ops, w) for w in good)):
        ws = [ops.Weight(w.plane, w.aux, w.meta, m.view(torch.uint8)) for w, m in zip(good, marks)]
        assert all(torch.equal(a, b) for a, b in zip(call(), want))
    assert ops.fault_status() == 0


@pytest.mark.parametrize("rows,K,R", [(148 * 28 * 16 + 16 * 333, 512, 16), (148 * 20 * 16 + 16 * 700, 1024, 16), (148 * 24 * 8 + 8 * 149, 2048, 8),
                                      (62080, 2048, 16)])
def test_last_round_of_a_large_product(ops, rows, K, R):
    _, w = _made(ops, rows, K, R, False)
    plain = ops.Weight(w.plane, w.aux, w.meta)
    xs = [torch.randn(T, K, device="cuda").to(torch.bfloat16) for T in (1, 2, 4)]
    want = [ops.mmv(x, plain) for x in xs]
    for marks in _marks(ops, w):
        w.marks = marks.view(torch.uint8)
        assert all(torch.equal(ops.mmv(x, w), y) for x, y in zip(xs, want))


@pytest.mark.parametrize("T", [1, 3])
def test_candidates_of_a_draft_step(ops, T):
    src, w = _made(ops, 4096, 2048, 16, False)
    plain = ops.Weight(w.plane, w.aux, w.meta)
    head = ops.DraftHead(2, *ops.int2_quantize(src.cuda()), 128)
    h = torch.randn(T, 2048, device="cuda").to(torch.bfloat16)
    want = ops.draft_logits(h, plain, head, 4100)
    for marks in _marks(ops, w):
        w.marks = marks.view(torch.uint8)
        assert torch.equal(ops.draft_logits(h, w, head, 4100), want)


def test_a_swapped_matrix_needs_no_new_marks(ops):
    rows, K = 1024, 2048
    _, a = _made(ops, rows, K, 16, False)
    other = ops.encode(to_bf16_tensor(o.weights_like(rows, K, 7)), ops.FMT_HUFPAIR, 16, False)
    aux = torch.zeros(max(a.aux.numel(), other[1].numel()), dtype=torch.uint8, device="cuda")
    aux[:a.aux.numel()] = a.aux
    w = ops.Weight(a.plane.clone(), aux, a.meta, a.marks)
    x = torch.randn(1, K, device="cuda").to(torch.bfloat16)
    ops.mmv(x, w)
    w.plane.copy_(other[0])
    w.aux[:other[1].numel()].copy_(other[1])
    assert torch.equal(ops.mmv(x, w), ops.mmv(x, ops.Weight(w.plane, w.aux, w.meta)))


def test_layouts_without_marks(ops):
    src = to_bf16_tensor(o.weights_like(64, 512, 1))
    assert ops.upload(*ops.encode(src, ops.FMT_NIBBLE, 0, False), "cuda").marks is None
    assert ops.upload(*ops.encode(src, ops.FMT_HUFPAIR, 16, False, True), "cuda").marks is None
    assert ops.upload(*ops.encode(src, ops.FMT_HUFPAIR, 8, False), "cuda").marks is None       # one part
    assert ops.upload(*ops.encode(src, ops.FMT_HUFPAIR, 16, False), "cpu").marks is None
