"""As test_gpu_matrix_swap.py, with marks (of the matrix that was there first, later of whichever the kernels saw last): every call that the
parts serve reads the matrix behind a kernel that overwrites it."""
import pytest
import torch

from conftest import to_bf16_tensor
from oracle import cpu_oracle as o
from test_gpu_matrix_swap import _check, _two

pytestmark = pytest.mark.gpu


def _marked(ops, rows, K, R, cm=False):
    w, enc = _two(ops, rows, K, R, cm)
    w.marks = ops.upload(w.plane, w.aux, w.meta, "cuda").marks
    assert w.marks_ptr() is not None
    return w, enc


@pytest.fixture(scope="module")
def ops():
    from orin_qwen_lossless_b200 import ops as m
    m.init()
    return m


@pytest.mark.parametrize("rows,K,R", [(4096, 2048, 16), (8192, 2048, 16), (2048, 4096, 16), (16384, 512, 16)])
def test_products_and_reconstruction(ops, rows, K, R):
    w = _marked(ops, rows, K, R)
    ids = torch.arange(0, rows, 37, device="cuda", dtype=torch.int32)
    _check([w], lambda ws: ops.dequant(ws[0]))
    _check([w], lambda ws: ops.get_rows(ids, ws[0]))
    for T in (1, 2, 4, 8, 20):
        x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
        _check([w], lambda ws: ops.linear(x, ws[0]))
        if T <= 8:
            _check([w], lambda ws: ops.mmv(x.float(), ws[0]))


def test_draft(ops):
    w = _marked(ops, 4096, 2048, 16)
    head = ops.DraftHead(2, *ops.int2_quantize(to_bf16_tensor(o.weights_like(4096, 2048, 3)).cuda()), 32)
    x = torch.randn(2, 2048, device="cuda").to(torch.bfloat16)
    _check([w], lambda ws: ops.draft_logits(x, ws[0], head, 4096))
