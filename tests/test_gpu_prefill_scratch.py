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


def _public(ops, K, rows, n, T, used, glu, seed):
    """A product through ops.moe_mm_ids as a program calls it, and what the scratch rule says about it."""
    import ctypes as C
    from orin_qwen_lossless_b200 import _lib
    w, u = (ops.upload(*ops.encode(to_bf16_tensor(o.weights_like(n * rows, K, seed + i)), 3, 16, False, True), "cuda") for i in range(2))
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, K, device="cuda", generator=g).to(torch.bfloat16)
    ids = torch.rand(T, n, device="cuda", generator=g).topk(used, dim=1).indices.to(torch.int32).contiguous()
    cw, cu = w.c(), u.c()
    need = _lib.lib().bf16n_mm_ids_scratch_bytes(C.byref(cw), C.byref(cu) if glu else None, n, T, used)
    return (lambda: ops.moe_mm_ids(x, ids, w, n, up=u if glu else None, out_dtype=torch.bfloat16 if glu else torch.float32)), need


@pytest.mark.parametrize("K, rows, n, T, used, glu", [
    (512, 512, 8, 4000, 8, False), (512, 512, 64, 4096, 8, True), (1024, 256, 8, 4000, 2, True), (1536, 768, 4, 700, 2, False),
    (2048, 512, 1, 1000, 1, True), (3072, 256, 16, 300, 8, True), (4096, 256, 4, 600, 4, False), (4096, 1024, 3, 129, 3, True),
])
def test_both_forms_give_the_same_bits(layer, monkeypatch, K, rows, n, T, used, glu):
    """The public call takes the two-pass form here; without scratch it runs the fused kernel: not a bit differs, so memory and
    capture, which decide between them, do not show in results."""
    ops = layer[0]
    run, need = _public(ops, K, rows, n, T, used, glu, K + n)
    assert need > 0
    taken = []
    real = ops._mm_ids_scratch
    monkeypatch.setattr(ops, "_mm_ids_scratch", lambda *a: taken.append(real(*a)) or taken[-1])
    two = run()
    assert taken[0] is not None and taken[0].numel() >= need
    monkeypatch.setattr(ops, "_mm_ids_scratch", lambda *a: None)
    assert torch.equal(two, run())


def test_capture_and_a_full_device_run_the_fused_kernel(layer, monkeypatch):
    ops = layer[0]
    monkeypatch.setattr(ops, "_scratch_refused", {})
    run, need = _public(ops, 2048, 512, 48, 600, 8, True, 9)
    assert need == 48 * 2 * 512 * 2048 * 2
    want = run()

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        before = torch.cuda.memory_allocated()
        with torch.cuda.graph(g, stream=s):
            got = run()
        assert torch.cuda.memory_allocated() - before < need      # no tiles in the graph's memory
        got.zero_()
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    del g

    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction(min(1.0, (torch.cuda.memory_reserved() + need // 2) / total))
    try:
        assert torch.equal(run(), want)
        assert list(ops._scratch_refused) == [torch.cuda.current_device()]
        with monkeypatch.context() as m:      # not asked again while the refusal is fresh
            m.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
            empty = torch.empty
            m.setattr(ops.torch, "empty", lambda *a, **k: pytest.fail("asked again") if a and a[0] == need + 1024 else empty(*a, **k))
            assert torch.equal(run(), want)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    ops._scratch_refused.clear()
    assert torch.equal(run(), want)
