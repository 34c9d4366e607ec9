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
