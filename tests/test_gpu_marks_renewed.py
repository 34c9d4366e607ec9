"""Marks after the matrix was overwritten in place: made again by the first call through the Weight, in the memory that captured calls read,
so that an update costs no call after it more than it cost before there were marks."""
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from orin_qwen_lossless_b200 import ops as m
    m.init()
    return m


def _pair(ops, rows=2048, K=2048, R=16, cm=False):
    """A matrix on the GPU with room in aux, and another of the same shape to overwrite it with."""
    a, b = (ops.encode(to_bf16_tensor(o.weights_like(rows, K, seed)), ops.FMT_HUFPAIR, R, cm) for seed in (1, 2))
    n = max(a[1].numel(), b[1].numel())
    return ops.upload(a[0], torch.nn.functional.pad(a[1], (0, n - a[1].numel())), a[2], "cuda"), ops.upload(*b, "cuda")


def _overwrite(w, new):
    w.plane.copy_(new.plane)
    w.aux[:new.aux.numel()].copy_(new.aux)


X = {T: torch.randn(T, 2048).to(torch.bfloat16) for T in (1, 2, 8, 20)}
CALLS = {"mmv": lambda ops, w: ops.mmv(X[1].cuda(), w), "mmv f32": lambda ops, w: ops.mmv(X[2].cuda().float(), w),
         "mmv out": lambda ops, w: ops.mmv(X[1].cuda(), w, out=torch.empty(1, w.meta.rows, device="cuda")), "linear": lambda ops, w: ops.linear(X[8].cuda(), w),
         "linear long": lambda ops, w: ops.linear(X[20].cuda(), w), "dequant": lambda ops, w: ops.dequant(w),
         "get_rows": lambda ops, w: ops.get_rows(torch.arange(0, 2048, 9, device="cuda"), w)}


@pytest.mark.parametrize("name", CALLS)
def test_first_call_makes_them_again(ops, name):
    w, new = _pair(ops)
    memory = w.marks.data_ptr()
    CALLS[name](ops, w)
    assert not torch.equal(w.marks, new.marks)
    _overwrite(w, new)
    for _ in range(2):
        assert torch.equal(CALLS[name](ops, w), CALLS[name](ops, new))
        assert torch.equal(w.marks, new.marks) and w.marks.data_ptr() == memory and w.marks_at == w.aux._version


def test_draft_and_experts(ops):
    w, new = _pair(ops)
    head = ops.DraftHead(2, *ops.int2_quantize(to_bf16_tensor(o.weights_like(2048, 2048, 2)).cuda()), 32)
    _overwrite(w, new)
    assert torch.equal(ops.draft_logits(X[2].cuda(), w, head, 2048), ops.draft_logits(X[2].cuda(), new, head, 2048)) and torch.equal(w.marks, new.marks)
    ws, news = zip(*(_pair(ops, 4 * r, K, R, cm) for r, K, R, cm in ((512, 2048, 8, True), (512, 2048, 8, True), (2048, 512, 16, False))))
    for w, new in zip(ws, news):
        _overwrite(w, new)
    logits = torch.randn(2, 4, device="cuda")
    a, b = (ops.moe_decode(X[2].cuda(), *m, 4, 2, router_logits=logits)[0] for m in (ws, news))
    assert torch.equal(a, b) and all(torch.equal(w.marks, new.marks) for w, new in zip(ws, news))


def test_captured_calls_read_the_renewed_marks(ops):
    w, new = _pair(ops)
    x, y = X[1].cuda(), torch.empty(1, 2048, device="cuda")
    ops.mmv(x, w, out=y)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.mmv(x, w, out=y)
    _overwrite(w, new)
    graph.replay()
    assert torch.equal(y, ops.mmv(x, new)) and not torch.equal(w.marks, new.marks)    # right, and slow
    assert ops.make_marks(w) and torch.equal(w.marks, new.marks)
    graph.replay()
    assert torch.equal(y, ops.mmv(x, new))


def test_under_capture_nothing_is_made(ops):
    w, new = _pair(ops)
    x, y = X[1].cuda(), torch.empty(1, 2048, device="cuda")
    ops.mmv(x, w, out=y)
    _overwrite(w, new)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.mmv(x, w, out=y)
        assert not ops.make_marks(w)
    graph.replay()
    assert torch.equal(y, ops.mmv(x, new))


def test_inference_tensors_and_weights_made_by_hand(ops):
    w, new = _pair(ops)
    with torch.inference_mode():
        i = ops.upload(w.plane.cpu(), w.aux.cpu(), w.meta, "cuda")
        assert torch.equal(i.marks, w.marks) and i.marks_at is None and torch.equal(ops.mmv(X[1].cuda(), i), ops.mmv(X[1].cuda(), w))
        _overwrite(i, new)
        assert torch.equal(ops.mmv(X[1].cuda(), i), ops.mmv(X[1].cuda(), new))
    hand = ops.Weight(w.plane, w.aux, w.meta)
    assert ops.make_marks(hand) and torch.equal(hand.marks, w.marks)
    assert not ops.make_marks(ops.upload(*ops.encode(to_bf16_tensor(o.weights_like(64, 512, 1)), ops.FMT_NIBBLE, 0, False), "cuda"))
