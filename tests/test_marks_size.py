"""Marks are hints in what they hold, not in how many there are: a Weight passes on only marks of its own matrix's size."""
import ctypes as C

import pytest
import torch

from orin_qwen_lossless_b200 import _lib, ops


def _meta(rows, K, R, fmt=ops.FMT_HUFPAIR, cm=False, fo=False):
    return ops.Meta(fmt, K, rows, R, cm, fo, 256, 16640, 20000, 30000)


def _weight(meta, marks):
    return ops.Weight(torch.empty(0, dtype=torch.uint8), torch.empty(0, dtype=torch.uint8), meta, marks)


def test_size_is_the_librarys():
    for fmt in (ops.FMT_NIBBLE, ops.FMT_HUFFMAN, ops.FMT_HUFPAIR):
        for K in range(512, 4097, 512):
            for R in (0, 1, 2, 3, 4, 6, 8, 12, 16, 32):
                for fo in (False, True):
                    m = _meta(max(R, 1) * 37, K, R, fmt, fo=fo)
                    w = _lib.Weight(4096, 8192, fmt, R, K, m.rows, 0, int(fo), 256, 16640, 20000, 30000)
                    assert m.marks_bytes() == _lib.lib().bf16n_marks_bytes(C.byref(w)), (fmt, K, R, fo)


def test_marks_of_another_size_are_left_out():
    small, large = _meta(1024, 2048, 16), _meta(62080, 2048, 16)
    n = small.marks_bytes()
    assert n == 64 * 7 * 64
    right = torch.zeros(n, dtype=torch.uint8)
    assert _weight(small, right).marks_ptr() == right.data_ptr()
    assert _weight(small, right.view(torch.int16)).marks_ptr() == right.data_ptr()
    assert _weight(large, right).marks_ptr() is None                                       # another matrix was put in
    assert _weight(_meta(1024, 2048, 32), right).marks_ptr() is None
    assert _weight(_meta(1024, 2048, 8), right).marks_ptr() is None
    for wrong in (right[:-1], right[:-2], torch.zeros(n + 2, dtype=torch.uint8), torch.zeros(0, dtype=torch.uint8), torch.zeros(2 * n, dtype=torch.uint8)[::2],
                  torch.zeros(n + 1, dtype=torch.uint8)[1:]):
        assert _weight(small, wrong).marks_ptr() is None
    assert _weight(_meta(1024, 512, 8), torch.zeros(0, dtype=torch.uint8)).marks_ptr() is None


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 9])
def test_calls_with_marks_of_another_size(T):
    from conftest import to_bf16_tensor
    from oracle import cpu_oracle as o
    ops.init()
    few, many = (ops.upload(*ops.encode(to_bf16_tensor(o.weights_like(rows, 2048, rows)), ops.FMT_HUFPAIR, 16, False), "cuda") for rows in (256, 4096))
    x, ids = torch.randn(T, 2048, device="cuda").to(torch.bfloat16), torch.arange(0, 4096, 61, device="cuda", dtype=torch.int32)
    plain = ops.Weight(many.plane, many.aux, many.meta)
    few.plane, few.aux, few.meta = many.plane, many.aux, many.meta                         # keeps the marks of 256 rows
    odd = torch.zeros(many.marks.numel() + 1, dtype=torch.uint8, device="cuda")[1:]        # right in number, not 2-byte aligned
    for w in (few, ops.Weight(*(getattr(plain, f) for f in ("plane", "aux", "meta")), odd)):
        for call in (lambda w: ops.linear(x, w), lambda w: ops.dequant(w), lambda w: ops.get_rows(ids, w), lambda w: ops.mmv(x[:1], w),
                     lambda w: ops.mmv(x[:1], w, torch.zeros(1, 1, device="cuda", dtype=torch.int32), 4096)):
            assert torch.equal(call(w), call(plain))
