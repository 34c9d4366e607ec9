"""The tensors that encode() returns are the buffers the encoder wrote, in torch's memory: either one stays valid without the other,
views keep the memory alive, a second call does not touch the first call's result, and both can be resized like any tensor."""
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


def test_results_are_ordinary_tensors():
    from orin_qwen_lossless_b200 import ops
    bits = o.weights_like(32, 512, 1)
    for fmt, R in ((1, 0), (2, 4), (3, 4)):
        plane, aux, _ = ops.encode(to_bf16_tensor(bits), fmt, R, False)
        want, n = aux.clone(), aux.numel()
        assert aux.data_ptr() % 16 == 0 and aux.untyped_storage().nbytes() == n
        aux.resize_(n + 4096)
        assert torch.equal(aux[:n], want)
        plane.resize_(64, 512)


def test_no_memory_for_the_result(monkeypatch):
    import pytest
    from orin_qwen_lossless_b200 import ops
    real, calls = torch.empty, []

    def empty(*a, **k):
        calls.append(a)
        if len(calls) == 2:      # the plane is there, the aux buffer is not to be had
            raise MemoryError("no memory")
        return real(*a, **k)

    w = to_bf16_tensor(o.weights_like(32, 512, 1))
    monkeypatch.setattr(ops.torch, "empty", empty)
    with pytest.raises(MemoryError):
        ops.encode(w, 3, 4, False)
    monkeypatch.undo()
    ops.encode(w, 3, 4, False)
