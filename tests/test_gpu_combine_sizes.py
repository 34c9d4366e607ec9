"""Weighted combine on both sides of its rule (output values, whole 16-byte groups, alignment) against FP64: slot counts that leave
every remainder of the loads in flight, BF16 and FP32 weights and outputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_used", [1, 3, 4, 6, 8, 12, 15])
@pytest.mark.parametrize("T, N", [(3, 510), (3, 516), (640, 510), (640, 516), (64, 4096), (63, 4096)])
def test_combine(n_used, T, N):
    from orin_qwen_lossless_b200 import _lib, ops
    ops.init()
    g = torch.Generator(device="cuda").manual_seed(n_used * T + N)
    ys = torch.randn(T, n_used, N, device="cuda", generator=g)
    for w in (torch.rand(T, n_used, device="cuda", generator=g), torch.rand(T, n_used, device="cuda", generator=g).to(torch.bfloat16)):
        want = (w.double().unsqueeze(2) * ys.double()).sum(1)
        bound = (n_used + 1) * 2.0 ** -24 * (w.double().unsqueeze(2) * ys.double()).abs().sum(1)   # one rounding per slot
        got = ops.moe_combine(ys, w, torch.float32)
        assert ((got.double() - want).abs() <= bound + 1e-30).all()
        assert torch.equal(ops.moe_combine(ys, w), got.to(torch.bfloat16))
        buf = torch.full((T * N + 3,), 7.0, device="cuda")     # an output that is not 16-byte aligned: same bits
        _lib.check(_lib.lib().bf16n_moe_combine(ys.data_ptr(), w.data_ptr(), int(w.dtype == torch.bfloat16), buf.data_ptr() + 4, 0, T, n_used, N,
                                                torch.cuda.current_stream().cuda_stream))
        assert torch.equal(buf[1:-2].view(T, N), got) and buf[0] == 7.0 and (buf[-2:] == 7.0).all()
