"""Units whose streams are longer than half of a part kernel's buffer (3 bits a weight), alone and between shorter ones, where a block takes
several units in turn: the bits of the product without marks, and no unit left to one warp."""
import numpy as np
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


def _matrix(ops, rows, K, R, long_units):
    """A matrix whose units (by a mask of rows // R) have exponents of one of ten values instead of one of two."""
    g = np.random.default_rng(rows + K)
    bits = o.weights_like(rows, K, rows + K) & 0x807F
    exp = np.where(np.repeat(long_units, R)[:, None], g.integers(100, 110, bits.shape), g.integers(118, 120, bits.shape))
    src = to_bf16_tensor(bits | (exp << 7).astype(np.uint16))
    enc = ops.encode(src, ops.FMT_HUFPAIR, R, False)
    assert enc[2].format == ops.FMT_HUFPAIR
    _, aux, m = enc
    base = aux.numpy()[m.off_b:m.off_b + 4 * (rows // R)].view(np.uint32).astype(np.int64)
    assert ((np.diff(base) * 32 > 3 * R * K) == long_units[:-1]).all()
    return src, ops.upload(*enc, "cuda")


@pytest.mark.parametrize("rows,K,R", [(16 * 1000, 2048, 16), (16 * 2100, 512, 16), (8 * 1100, 2048, 8), (16 * 500, 4096, 16)])
@pytest.mark.parametrize("share", [0.02, 0.5, 1.0])
def test_long_units_among_short_ones(ops, rows, K, R, share):
    units = rows // R
    src, w = _matrix(ops, rows, K, R, np.random.default_rng(units).random(units) < share if share < 1 else np.ones(units, bool))
    plain = ops.Weight(w.plane, w.aux, w.meta)
    good = w.marks.clone()
    ids = torch.arange(0, rows, rows // 100, device="cuda", dtype=torch.int32)
    for marks in (good, torch.zeros_like(good), good.roll(64)):
        for T in (1, 2, 3, 4, 8):
            x = torch.randn(T, K, device="cuda")
            for x in (x, x.to(torch.bfloat16)):
                w.marks = marks.clone()
                assert torch.equal(ops.mmv(x, w), ops.mmv(x, plain)), (T, x.dtype)
        w.marks = marks.clone()
        assert torch.equal(ops.dequant(w).cpu().view(torch.int16), src.view(torch.int16))
        w.marks = marks.clone()
        assert torch.equal(ops.get_rows(ids, w), ops.get_rows(ids, plain))
    assert ops.fault_status() == 0


def _us(call):
    for _ in range(3):
        call()
    took = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(8):
            call()
        b.record()
        b.synchronize()
        took.append(a.elapsed_time(b) * 125)
    return sorted(took)[4]


def test_long_units_are_walked_from_several_places_too(ops):
    """One warp to a unit took 4 to 5 times the calls without marks (667 against 162 us, 446 against 91); now 0.8."""
    rows = 62080
    _, w = _matrix(ops, rows, 2048, 16, np.ones(rows // 16, bool))
    plain = ops.Weight(w.plane, w.aux, w.meta)
    x = torch.randn(8, 2048, device="cuda").to(torch.bfloat16)
    for call in (lambda m: ops.mmv(x, m), ops.dequant):
        assert _us(lambda: call(w)) < 1.5 * _us(lambda: call(plain))
