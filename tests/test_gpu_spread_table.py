"""The code table spread over conflict-free copies (fragment-order products): tables of every number of copies, from a few short codes to
all codes long, at the smallest matrix that takes the staged kernel. The products are the split kernel's of the same rows, bit for bit."""
import numpy as np
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


def _bits(rows, K, tail):
    """Weights whose exponents are one of three values, or, with probability `tail`, one of fifty."""
    g = np.random.default_rng(int(1000 * tail) + K)
    bits = o.weights_like(rows, K, K)
    exp = np.where(g.random(bits.shape) < tail, g.integers(70, 120, bits.shape), g.integers(118, 121, bits.shape)).astype(np.uint16)
    return (bits & 0x807F) | (exp << 7).astype(np.uint16)


def _copies(aux, meta):
    lens = aux.numpy()[meta.off_a:meta.off_a + 16384].view(np.uint32)[::16] & 31
    q = int(np.argmax(lens > 8)) if (lens > 8).any() else 256
    entries = 4096 - 15 * q
    return 32 if entries <= 512 else 16 if entries <= 1024 else 8 if entries <= 2048 else 4


@pytest.mark.parametrize("tail,copies", [(0.0, 32), (0.005, 16), (0.015, 8), (0.05, 4), (0.6, 4)])
@pytest.mark.parametrize("K", [512, 1024])
def test_every_number_of_copies(tail, copies, K):
    from orin_qwen_lossless_b200 import ops
    ops.init()
    sms = ops.sm_count()
    rows = 16 * (6 * sms + 5)
    bits = _bits(rows, K, tail)
    plane, aux, meta = ops.encode(to_bf16_tensor(bits), ops.FMT_HUFPAIR, 16, False, True)
    assert meta.format == ops.FMT_HUFPAIR and _copies(aux, meta) == copies
    w = ops.upload(plane, aux, meta, "cuda")
    few = 16 * (6 * sms - 1)
    part = ops.upload(*ops.encode(to_bf16_tensor(bits[:few]), ops.FMT_HUFPAIR, 16, False, True), "cuda")
    for T in (2, 7, 8):
        x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
        y = ops.mmv(x, w)
        assert torch.equal(y[:, :few], ops.mmv(x, part))
        exact = x.double() @ to_bf16_tensor(bits).cuda().double().t()
        assert ((y.double() - exact).norm() / exact.norm()).item() < 2e-6      # FP32 sums of 512 products and their sum: 4.7e-7 measured
    assert ops.fault_status() == 0
