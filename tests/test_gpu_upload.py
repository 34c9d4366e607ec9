"""upload() takes what it took before it made marks: memory that is filled later, matrices that only their first use refuses, and a device
without room for marks."""
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


def _encoded(ops, rows=1024, K=2048, R=16):
    src = to_bf16_tensor(o.weights_like(rows, K, rows))
    return src, ops.encode(src, ops.FMT_HUFPAIR, R, False)


@pytest.mark.parametrize("fill", [0, 255, None])
@pytest.mark.parametrize("header", [False, True])
def test_memory_that_is_filled_later(ops, fill, header):
    src, (plane, aux, meta) = _encoded(ops)
    blank = torch.randint(0, 256, aux.shape, dtype=torch.uint8) if fill is None else torch.full_like(aux, fill)
    if header:
        blank[:256] = aux[:256]
    w = ops.upload(torch.empty_like(plane), blank, meta, "cuda")
    torch.cuda.synchronize()
    assert w.marks.numel() == meta.marks_bytes()
    w.plane.copy_(plane)
    w.aux.copy_(aux)
    assert torch.equal(ops.dequant(w).cpu().view(torch.int16), src.view(torch.int16))


def test_marks_are_where_codes_begin(ops):
    """Every part of every lane, walked here code by code."""
    _, (plane, aux, meta) = _encoded(ops, 64, 1024)
    w = ops.upload(plane, aux, meta, "cuda")
    marks = w.marks.view(torch.int16).cpu().view(4, 3, 32)
    a = aux.numpy()
    lut, base = a[meta.off_a:meta.off_a + 16384].view("<u4"), a[meta.off_b:meta.off_b + 16].view("<u4")
    rel = a[meta.off_c:meta.off_c + 256].view("<u2").reshape(4, 32)
    bits = "".join(f"{b:08b}" for word in a[meta.off_d:meta.off_d + (a.size - meta.off_d) // 4 * 4].view("<u4") for b in int(word).to_bytes(4, "big"))
    for u in range(4):
        for lane in range(32):
            start = at = 32 * (int(base[u]) + int(rel[u, lane]))
            for part in range(3):
                for _ in range(64):
                    at += int(lut[int(bits[at:at + 12], 2)]) & 31
                assert int(marks[u, part, lane]) == at - start


def test_refused_at_first_use_only(ops):
    _, (plane, aux, meta) = _encoded(ops)
    x = torch.randn(1, 2048, device="cuda").to(torch.bfloat16)
    for args in ((plane.view(-1)[:-1], aux, meta), (plane, aux[:meta.off_d], meta), (plane.t(), aux, meta), (plane.short(), aux, meta)):
        w = ops.upload(*args, "cuda")
        with pytest.raises(RuntimeError):
            ops.mmv(x, w)


def test_no_room_for_marks(ops, monkeypatch):
    src, enc = _encoded(ops)
    empty = torch.empty

    def full(*a, **k):
        if k.get("dtype") == torch.uint8 and "device" in k:
            raise torch.OutOfMemoryError("no room")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", full)
    w = ops.upload(*enc, "cuda")
    monkeypatch.undo()
    assert w.marks is None and torch.equal(ops.dequant(w).cpu().view(torch.int16), src.view(torch.int16))
