"""The native forms of mmv, linear and draft_logits against the Python functions that they stand in front of: the same results for what
they take, and the same refusals, copies and wrappers for what they leave alone."""
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


class Left:     # stands in for the native module: leaves every call to the Python functions
    mmv = linear = draft_logits = staticmethod(lambda *a: None)


@pytest.fixture(scope="module")
def ops():
    from orin_qwen_lossless_b200 import ops as m
    m.init()
    return m


def _both(ops, monkeypatch, call):
    got = []
    for native in (ops._native(), Left):
        monkeypatch.setattr(ops, "_calls", native)
        try:
            got.append(call())
        except Exception as e:
            got.append((type(e), str(e)))
    a, b = got
    if isinstance(b, torch.Tensor):
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)
    else:
        assert a == b and isinstance(a, tuple)
    return b


@pytest.fixture(scope="module", params=[(3, 16, False), (1, 0, False), (3, 16, True)])
def weight(request, ops):
    return ops.upload(*ops.encode(to_bf16_tensor(o.weights_like(320, 512, 5)), request.param[0], request.param[1], False, request.param[2]), "cuda")


def test_taken(ops, monkeypatch, weight):
    g = torch.Generator(device="cuda").manual_seed(1)
    bias = torch.randn(320, device="cuda", generator=g).to(torch.bfloat16)
    for shape in [(1, 512), (3, 512), (8, 512), (9, 512), (2, 7, 512), (1, 1, 512), (512,), (0, 512)]:
        x = torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
        for b in (None, bias, bias.float()):
            _both(ops, monkeypatch, lambda: ops.linear(x, weight, b))
        _both(ops, monkeypatch, lambda: ops.mmv(x, weight))
        _both(ops, monkeypatch, lambda: ops.mmv(x.float(), weight, out_dtype=torch.bfloat16))


def test_left_alone(ops, monkeypatch, weight):
    x = torch.randn(4, 1024, device="cuda").to(torch.bfloat16)
    flat = torch.randn(5000, device="cuda").to(torch.bfloat16)
    wrong = ops.Weight(weight.plane[:-1], weight.aux, weight.meta)
    cases = [lambda: ops.linear(x[:, :512], weight), lambda: ops.linear(x[:, ::2], weight), lambda: ops.linear(flat[1:513].view(1, 512), weight),
             lambda: ops.mmv(x[:, :512], weight), lambda: ops.mmv(flat[1:513].view(1, 512), weight), lambda: ops.mmv(x, weight), lambda: ops.linear(x, weight),
             lambda: ops.linear(x[:, :512].float(), weight), lambda: ops.mmv(x[:, :512].half(), weight), lambda: ops.mmv(x[:, :512].contiguous(), wrong),
             lambda: ops.linear(x[:, :512].contiguous().cpu(), weight), lambda: ops.mmv(x[:, :512].contiguous().cpu(), weight),
             lambda: ops.mmv(x[:, :512].contiguous().cpu().pin_memory(), weight),
             lambda: ops.linear(flat[:4608].view(9, 512).requires_grad_(), weight), lambda: ops.linear(flat[:512].view(1, 512).requires_grad_(), weight)]
    kinds = [isinstance(_both(ops, monkeypatch, c), torch.Tensor) for c in cases]
    assert kinds == [True, True, False, True, False] + [False] * 7 + [True, False, True]


def test_modes_and_subclasses(ops, monkeypatch, weight):
    x = torch.randn(2, 512, device="cuda").to(torch.bfloat16)

    class Sub(torch.Tensor):
        pass

    seen = []

    class Mode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    want = ops.linear(x, weight)
    assert torch.equal(ops.linear(x.as_subclass(Sub), weight), want)
    with Mode():
        assert torch.equal(ops.linear(x, weight), want)
    assert seen
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda r: ops.linear(r[None], weight))(x)


def test_draft(ops, monkeypatch):
    src = to_bf16_tensor(o.weights_like(1024, 2048, 9))
    w = ops.upload(*ops.encode(src, 3, 16, False), "cuda")
    for bits in (2, 4):
        head = ops.make_draft_head(src.cuda(), bits)
        for T in (1, 4, 5):     # five tokens are refused
            h = torch.randn(T, 2048, device="cuda").to(torch.bfloat16)
            for vocab in (1024, 1030):
                _both(ops, monkeypatch, lambda: ops.draft_logits(h, w, head, vocab))
            _both(ops, monkeypatch, lambda: ops.draft_logits(h.float(), w, head, 1024))
            _both(ops, monkeypatch, lambda: ops.draft_logits(h.t().contiguous().t(), w, head, 1024))
    graded = torch.randn(1, 2048, device="cuda").to(torch.bfloat16).requires_grad_()
    assert ops.draft_logits(graded, w, head, 1024).requires_grad


def test_threads_and_streams(ops, weight):
    import threading
    xs = [torch.randn(2, 512, device="cuda").to(torch.bfloat16) for _ in range(4)]
    want = [ops.linear(x, weight) for x in xs]
    torch.cuda.synchronize()
    bad = []

    def run(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(50):
                y = ops.linear(xs[i], weight)
        s.synchronize()
        if not torch.equal(y, want[i]):
            bad.append(i)

    ts = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
