"""Two-pass batched product of fragment-order experts (decode into operand tiles in the call's own scratch, then the
tensor-core pass) against FP64 references over the exact weights: scratch for all experts, for ranges of unequal length, for
one at a time and for none (the fused kernel); token counts around the 128-token groups, experts without tokens."""
import numpy as np
import pytest
import torch

from conftest import BF16_REL, to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu
E, TOPK, H, N = 8, 4, 2048, 512
MMA_REL = 2e-6  # FP32 tensor-core accumulation, relative to sum |w x| (as for the other batched kernels)


@pytest.fixture(scope="module")
def layer():
    from orin_qwen_lossless_b200 import ops
    ops.init()
    bits = {"gate": o.weights_like(E * N, H, 31), "up": o.weights_like(E * N, H, 32), "down": o.weights_like(E * H, N, 33)}
    enc = {k: ops.upload(*ops.encode(to_bf16_tensor(v), 3, 16, False, True), "cuda") for k, v in bits.items()}
    yield ops, enc, {k: o.bf16_bits_to_f32(v).astype(np.float64) for k, v in bits.items()}
    torch.cuda.synchronize()
    assert ops.fault_status() == 0


def _act(shape, seed):
    xb = o.f32_to_bf16_bits(np.random.default_rng(seed).standard_normal(shape).astype(np.float32))
    return to_bf16_tensor(xb).cuda(), o.bf16_bits_to_f32(xb).astype(np.float64)


def _with_scratch(ops, monkeypatch, experts, per_expert):
    """moe_mm_ids calls get scratch for that many experts."""
    def scratch(cw, cu, n_experts, T, n_used, device):
        return torch.empty(experts * per_expert + 1024, dtype=torch.uint8, device=device) if experts else None
    monkeypatch.setattr(ops, "_mm_ids_scratch", scratch)


# 2309 tokens: more passes of one expert (ten of 256 tokens) than the tensor-core pass keeps lists for (eight)
@pytest.mark.parametrize("T, experts", [(T, n) for T in (9, 128, 300) for n in (8, 3, 1, 0)] + [(2309, 8)])
def test_against_fp64(layer, monkeypatch, T, experts):
    ops, enc, f64 = layer
    g = np.random.default_rng(T)
    rest = np.array([0, 1, 3, 4, 5, 6])                                  # expert 7 stays empty, expert 2 gets every token
    ids_np = np.stack([np.concatenate([[2], g.permutation(rest)[:TOPK - 1]]) for _ in range(T)])
    ids = torch.from_numpy(ids_np.astype(np.int32)).cuda()
    x, x64 = _act((T, H), T + 1)
    a, a64 = _act((T, TOPK, N), T + 2)

    _with_scratch(ops, monkeypatch, experts, 2 * N * H * 2)
    glu = ops.moe_mm_ids(x, ids, enc["gate"], E, up=enc["up"], out_dtype=torch.float32).cpu().numpy()
    _with_scratch(ops, monkeypatch, experts, H * N * 2)
    down = ops.moe_mm_ids(a, ids, enc["down"], E).cpu().numpy()
    one = ops.moe_mm_ids(x, ids, enc["up"], E, out_dtype=torch.bfloat16).float().cpu().numpy()
    for e in range(E):
        tt, ss = np.nonzero(ids_np == e)
        if tt.size == 0:
            continue
        wg, wu, wd = (f64[k].reshape(E, -1, f64[k].shape[1])[e] for k in ("gate", "up", "down"))
        ug, uu, ud = x64[tt] @ wg.T, x64[tt] @ wu.T, a64[tt, ss] @ wd.T
        sg, su, sd = np.abs(x64[tt]) @ np.abs(wg).T, np.abs(x64[tt]) @ np.abs(wu).T, np.abs(a64[tt, ss]) @ np.abs(wd).T
        assert (np.abs(down[tt, ss] - ud) <= MMA_REL * sd).all(), e
        assert (np.abs(one[tt, ss] - uu) <= MMA_REL * su + BF16_REL * np.abs(uu)).all(), e
        silu = ug / (1.0 + np.exp(-ug))
        # |silu'| <= 1.1, and the fast exponential and division cost a few FP32 roundings of the result
        bound = MMA_REL * (1.1 * sg * np.abs(uu) + su * np.abs(silu)) + 4e-6 * np.abs(silu * uu)
        assert (np.abs(glu[tt, ss] - silu * uu) <= bound).all(), e


def test_scratch_rule():
    """Few tokens per expert and other layouts ask for nothing; the request is whole experts and bounded."""
    from orin_qwen_lossless_b200 import _lib, ops
    import ctypes as C
    plane, aux, meta = ops.encode(to_bf16_tensor(o.weights_like(E * N, H, 31)), 3, 16, False, True)
    w = ops.upload(plane, aux, meta, "cuda").c()
    need = _lib.lib().bf16n_mm_ids_scratch_bytes
    per = 2 * N * H * 2
    assert need(C.byref(w), C.byref(w), E, 9, TOPK) == 0
    assert need(C.byref(w), C.byref(w), E, 4096, TOPK) == E * per
    assert need(C.byref(w), None, E, 4096, TOPK) == E * per // 2
    assert need(C.byref(w), None, 32, 4096, TOPK) == 0     # 128 rows per expert: no whole row block of 256
    lane_major = ops.encode(to_bf16_tensor(o.weights_like(E * N, H, 31)), 3, 8, True)
    assert need(C.byref(ops.upload(*lane_major, "cuda").c()), None, E, 4096, TOPK) == 0
