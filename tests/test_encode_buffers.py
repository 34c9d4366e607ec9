"""The tensors that encode() returns are the buffers the encoder wrote: either one stays valid without the other, views keep the
memory alive, and a second call does not touch the first call's result."""
import gc

import numpy as np
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o


def test_results_outlive_each_other():
    from orin_qwen_lossless_b200 import ops
    kept = []
    for seed in range(4):
        bits = o.weights_like(64, 1024, seed)
        plane, aux, _ = ops.encode(to_bf16_tensor(bits), 3, 4, False)
        p0, a0, _ = o.encode(bits, 3, 4)
        kept.append((plane[3:], p0.reshape(64, 1024)[3:]) if seed % 2 else (aux[256:], a0[256:]))
        del plane, aux
        gc.collect()
    torch.full((1 << 20,), 7, dtype=torch.uint8)    # memory that freed buffers would be given to
    for got, want in kept:
        assert np.array_equal(got.numpy(), want)


def test_nibble_bytes_in_a_used_heap():
    """The encoder fills every byte of a NIBBLE tensor: rows with one exponent (tables mostly empty, no escapes), ordinary rows, and
    more escapes than the buffer has room for, in memory that held something else before."""
    from orin_qwen_lossless_b200 import ops
    g = np.random.default_rng(4)
    one = np.full((40, 512), 0x3f80, np.uint16)
    wide = o.f32_to_bf16_bits((g.standard_normal((40, 1024)) * np.exp(9 * g.standard_normal((40, 1024)))).astype(np.float32))
    for bits in (one, wide, o.weights_like(40, 1024, 2), one, wide):
        junk = [torch.full((n,), 0xAB, dtype=torch.uint8) for n in (1 << 12, 1 << 14, 1 << 15, 1 << 16, 1 << 17) for _ in range(8)]
        del junk
        plane, aux, _ = ops.encode(to_bf16_tensor(bits), 1, 0, False)
        p0, a0, _ = o.encode(bits, 1, 0)
        assert np.array_equal(plane.numpy().ravel(), p0.ravel()) and np.array_equal(aux.numpy(), a0)
