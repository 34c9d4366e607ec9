"""Grouped and single NIBBLE products where rows differ most: rows of 4096 columns beside short ones (the group kernel for wide
rows), rows with none, a few and more than 64 escapes, BF16 and FP32 activations, 1 to 8 columns, row counts that leave warps
without a row. A group's outputs have the bits of the single products, and those are within the FP32 bound of FP64."""
import numpy as np
import pytest
import torch

from conftest import GEMV_REL, to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


def _bits(rows, K, seed):
    g = np.random.default_rng(seed)
    w = (g.standard_normal((rows, K)) * 0.02).astype(np.float32)
    w[::3] *= np.exp(2.0 * g.standard_normal((len(w[::3]), K))).astype(np.float32)   # wide exponents: many escapes
    return o.f32_to_bf16_bits(w)


@pytest.mark.parametrize("shapes", [[(9, 4096), (40, 512)], [(17, 2048), (3, 1024), (64, 512)], [(1, 4096)], [(2048, 512)]])
@pytest.mark.parametrize("T, fp32", [(1, False), (3, True), (8, False)])
def test_group_equals_single_products(shapes, T, fp32):
    from orin_qwen_lossless_b200 import ops
    ops.init()
    ws, xs, refs = [], [], []
    for i, (rows, K) in enumerate(shapes):
        bits = _bits(rows, K, 10 * i + rows)
        ws.append(ops.upload(*ops.encode(to_bf16_tensor(bits), 1, 0, False), "cuda"))
        xb = o.f32_to_bf16_bits(np.random.default_rng(K + T).standard_normal((T, K)).astype(np.float32))
        x = to_bf16_tensor(xb).cuda()
        xs.append(x.float() if fp32 else x)
        w64, x64 = o.bf16_bits_to_f32(bits).astype(np.float64), o.bf16_bits_to_f32(xb).astype(np.float64)
        refs.append((x64 @ w64.T, np.abs(x64) @ np.abs(w64).T))
    for y, w, x, (ref, s) in zip(ops.mmv_group(xs, ws), ws, xs, refs):
        assert torch.equal(y, ops.mmv(x, w))
        assert (np.abs(y.cpu().numpy() - ref) <= GEMV_REL * s).all()


@pytest.mark.parametrize("K", [512, 1024, 2048, 4096])
@pytest.mark.parametrize("T, fp32, rows", [(1, True, 21), (3, False, 21), (3, True, 4001), (4, False, 4001)])   # 4001: more than three rows to a warp
def test_glu(K, T, fp32, rows):
    from orin_qwen_lossless_b200 import ops
    ops.init()
    bits = _bits(2 * rows, K, K)
    w = ops.upload(*ops.encode(to_bf16_tensor(bits), 1, 0, False), "cuda")
    x = torch.from_numpy(np.random.default_rng(K).standard_normal((T, K)).astype(np.float32)).to(torch.bfloat16).cuda()
    x = x.float() if fp32 else x
    both = ops.mmv(x, w).double()
    g, u = both[:, :rows], both[:, rows:]
    want = g / (1 + torch.exp(-g)) * u
    # the same sums; the fast exponential rounds its argument (two roundings of |g| log2 e, 2^-23 each), it and the division
    # add a few roundings of the result
    assert ((ops.mmv_glu(x, w).double() - want).abs() <= (2e-6 + 2.4e-7 * g.abs()) * want.abs() + 1e-30).all()
