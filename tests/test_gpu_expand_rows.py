"""Exact reconstruction of pair-Huffman matrices by the ring reader: unit sizes on both sides of its rule (four steps of 512
weights), chunk-major units, one unit, fewer units than SMs, more than a full machine of warps, windows of rows."""
import numpy as np
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, K, R, cm", [
    (16, 512, 16, False), (3, 512, 1, False), (8, 512, 4, False), (6, 1024, 2, False), (5, 2048, 1, False), (34, 2048, 2, False),
    (640, 2048, 16, False), (48, 4096, 16, False), (40, 2048, 8, True), (24, 1024, 4, True), (32768, 512, 4, False),
    (33200, 512, 8, False), (66560, 1024, 16, False), (8320, 1024, 2, False),
])
def test_reconstruction_is_exact(rows, K, R, cm):
    from orin_qwen_lossless_b200 import ops
    ops.init()
    bits = o.weights_like(rows, K, rows + K + R)
    w = ops.upload(*ops.encode(to_bf16_tensor(bits), 3, R, cm), "cuda")
    src = to_bf16_tensor(bits).cuda()
    for r0, n in {(0, rows), (R, rows - R), (rows - R, R)}:
        if n:
            assert torch.equal(ops.dequant(w, r0, n).view(torch.int16), src[r0:r0 + n].view(torch.int16)), (r0, n)
    assert ops.roundtrip_equal(w, src)
    other = src.clone()
    other[rows - 1, K - 1] = 3.0     # the comparison still sees the last weight
    assert not ops.roundtrip_equal(w, other)
