"""Candidate selection and re-scoring of a draft step (bf16n_draft_logits) against a stable sort and FP64 products: scores
with ties across the boundary, infinities and NaN, row counts that leave cluster blocks empty and ones whose keys do not
fit shared memory; and the row gather for few rows over unit sizes, which passes over the rows before the wanted one."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import GEMV_REL, to_bf16_tensor
from oracle import cpu_oracle as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from orin_qwen_lossless_b200 import ops as m
    m.init()
    yield m
    assert m.fault_status() == 0


def _scores(kind, T, rows, g):
    s = g.standard_normal((T, rows)).astype(np.float32)
    if kind == "ties":
        s = np.round(s * 2) / 2                     # about a dozen values: nearly every boundary cuts through equal scores
    elif kind == "equal":
        s[:] = -1.5
    elif kind == "special":
        s[:, ::7] = -np.inf
        s[:, 3::11] = np.nan
        s[:, 5::13] = np.inf
        s[:, 1::5] = -0.0
        s[:, 2::5] = 0.0
    return s


@pytest.mark.parametrize("rows, T, n_cand", [(16, 1, 16), (16, 2, 5), (4112, 3, 128), (62080, 2, 128), (393232, 1, 32)])
def test_candidates_and_scores(ops, rows, T, n_cand):
    from orin_qwen_lossless_b200 import _lib
    K = 512
    bits = o.weights_like(rows, K, rows)
    w = ops.upload(*ops.encode(to_bf16_tensor(bits), 3, 16, False), "cuda")
    g = np.random.default_rng(rows)
    x = torch.from_numpy(g.standard_normal((T, K)).astype(np.float32)).to(torch.bfloat16).cuda()
    vocab = rows + 37
    cw = w.c()
    for kind in ("normal", "ties", "equal", "special"):
        s = _scores(kind, T, rows, g)
        sd = torch.from_numpy(s).cuda()
        cand = torch.empty((T, n_cand), dtype=torch.int32, device="cuda")
        buf = torch.empty((T * n_cand, K), dtype=torch.bfloat16, device="cuda")
        out = torch.full((T, vocab), 7.0, device="cuda")
        _lib.check(_lib.lib().bf16n_draft_logits(sd.data_ptr(), T, rows, n_cand, C.byref(cw), x.data_ptr(), cand.data_ptr(), buf.data_ptr(),
                                                 out.data_ptr(), vocab, torch.cuda.current_stream().cuda_stream))
        out = out.cpu().numpy()
        # order of the selection: NaN above everything, +0 above -0 (as torch.topk's radix keys), then the lowest row
        b = s.view(np.uint32)
        key = np.where(np.isnan(s), np.uint32(0xffffffff), np.where(b >> 31, ~b, b | np.uint32(0x80000000))).astype(np.int64)
        for t in range(T):
            want = np.sort(np.argsort(-key[t], kind="stable")[:n_cand])
            assert np.array_equal(np.sort(cand[t].cpu().numpy()), want), (kind, t)
            rest = np.ones(vocab, bool)
            rest[want] = False
            assert np.isneginf(out[t, rest]).all()
            wr = o.bf16_bits_to_f32(bits[want]).astype(np.float64)
            x64 = x[t].double().cpu().numpy()
            assert (np.abs(out[t, want] - wr @ x64) <= GEMV_REL * (np.abs(wr) @ np.abs(x64))).all(), (kind, t)


@pytest.mark.parametrize("K, R", [(512, 1), (512, 16), (1024, 2), (1024, 16), (2048, 4), (2048, 8), (2048, 16), (4096, 16)])
@pytest.mark.parametrize("n", [1, 300])
def test_rows_of_every_position_in_a_unit(ops, K, R, n):
    rows = 16 * 20
    bits = o.weights_like(rows, K, K + R)
    if K == 1024:   # a matrix of many exponents: units with more than three stream bits per weight
        g = np.random.default_rng(3)
        bits = o.f32_to_bf16_bits((g.standard_normal((rows, K)) * np.exp(3 * g.standard_normal((rows, K)))).astype(np.float32))
    w = ops.upload(*ops.encode(to_bf16_tensor(bits), 3, R, False), "cuda")
    src = to_bf16_tensor(bits).cuda()
    ids = torch.from_numpy(np.random.default_rng(n).permutation(rows)[:n].astype(np.int32)).cuda()
    assert torch.equal(ops.get_rows(ids, w).view(torch.int16), src[ids.long()].view(torch.int16))
    assert torch.equal(ops.get_rows(ids.long(), w, torch.float32).view(torch.int32), src[ids.long()].float().view(torch.int32))


def test_derivatives_keep_the_general_form(ops):
    rows, K = 4096, 2048
    bits = o.weights_like(rows, K, 8)
    w = ops.upload(*ops.encode(to_bf16_tensor(bits), 3, 8, False), "cuda")
    head = ops.DraftHead(2, *ops.int2_quantize(to_bf16_tensor(bits).cuda()), 32)
    h = torch.from_numpy(np.random.default_rng(2).standard_normal((2, K)).astype(np.float32)).to(torch.bfloat16).cuda()
    out = ops.draft_logits(h, w, head, rows)
    assert out.grad_fn is None
    hg = h.clone().requires_grad_()
    og = ops.draft_logits(hg, w, head, rows)
    finite = torch.isfinite(out)
    assert torch.equal(torch.isfinite(og), finite) and torch.allclose(og[finite], out[finite], rtol=1e-4, atol=1e-4)
    og[finite].sum().backward()
    picked = finite.float() @ to_bf16_tensor(bits).cuda().float()
    assert torch.allclose(hg.grad.float(), picked, rtol=2e-2, atol=2e-2)   # BF16 gradient of a sum of 32 rows
    assert ops.draft_logits(h, w, head, rows + 100).shape == (2, rows + 100)
