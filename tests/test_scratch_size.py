"""bf16n_mm_ids_scratch_bytes answers 0 for every call that has no use for scratch: an empty matrix, experts that do not split
evenly or are more than a call takes, an up matrix of another shape or layout. Run in a process of its own: a wrong answer here
was once an arithmetic trap."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZES = """
import ctypes as C, sys
from orin_qwen_lossless_b200 import _lib
def w(rows, K=2048, fo=1, R=16, fmt=3):
    return _lib.Weight(4096, 8192, fmt, R, K, rows, 0, fo, 256, 16640, 20000, 30000)
def need(a, up, experts, tok=8192, used=8):
    return _lib.lib().bf16n_mm_ids_scratch_bytes(C.byref(a), C.byref(up) if up is not None else None, experts, tok, used)
print([need(w(0), None, 8), need(w(0), w(0), 1), need(w(100), None, 8), need(w(-4096), None, 8), need(w(8 * 512), w(8 * 256), 8),
       need(w(8 * 512), w(8 * 512, K=512), 8), need(w(8 * 512), w(8 * 512, fo=0), 8), need(w(8 * 512, fo=0), None, 8),
       need(w(2000 * 512), w(2000 * 512), 2000, 1 << 20), need(w(8 * 512), w(8 * 512), 8)])
"""


def test_sizes():
    r = subprocess.run([sys.executable, "-c", SIZES], capture_output=True, text=True, timeout=120, cwd=ROOT)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    *none, some = eval(r.stdout)
    assert none == [0] * 9 and some == 8 * 2 * 512 * 2048 * 2


def test_a_refusal_is_not_repeated_for_every_call(monkeypatch):
    """A device without memory for the tiles is asked once and then left alone for a while."""
    from orin_qwen_lossless_b200 import _lib, ops
    asked, now = [], [100.0]

    def empty(n, **kw):
        asked.append(kw["device"].index)
        raise torch.cuda.OutOfMemoryError

    monkeypatch.setattr(ops, "_scratch_refused", {})
    monkeypatch.setattr(ops.torch, "empty", empty)
    monkeypatch.setattr(ops.torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(ops.time, "monotonic", lambda: now[0])
    w = _lib.Weight(4096, 8192, 3, 16, 2048, 8 * 512, 0, 1, 256, 16640, 20000, 30000)
    for device, t in ((0, 100.0), (0, 100.1), (1, 101.0), (0, 109.0), (0, 111.0)):
        now[0] = t
        assert ops._mm_ids_scratch(w, w, 8, 8192, 8, torch.device("cuda", device)) is None
    assert asked == [0, 1, 0]


@pytest.mark.parametrize("glu, K, rows, experts, pairs, two_pass", [
    (True, 2048, 512, 256, 16, True), (True, 2048, 512, 256, 256, True), (True, 2048, 512, 16, 16, True), (True, 2048, 512, 1, 4096, True),
    (False, 512, 2048, 256, 80, True), (False, 512, 2048, 256, 64, False), (False, 512, 2048, 4, 4096, True),
    (False, 512, 2048, 1, 256, False), (False, 512, 512, 128, 80, False), (True, 512, 512, 64, 16, False),
    (True, 1024, 1024, 16, 32, False), (False, 1024, 256, 1, 1024, False), (True, 3072, 256, 64, 64, True),
])
def test_the_form_that_was_measured_faster(glu, K, rows, experts, pairs, two_pass):
    """Shapes on both sides of the rule between the fused kernel and the two-pass form (which alone asks for scratch)."""
    from orin_qwen_lossless_b200 import _lib
    w = _lib.Weight(4096, 8192, 3, 16, K, experts * rows, 0, 1, 256, 16640, 20000, 30000)
    used = min(8, experts)
    need = _lib.lib().bf16n_mm_ids_scratch_bytes(C.byref(w), C.byref(w) if glu else None, experts, experts * pairs // used, used)
    assert (need > 0) == two_pass


@pytest.mark.parametrize("K, rows, experts", [(512, 2048, 256), (2048, 512, 256), (4096, 1024, 1), (4096, 256, 64), (1536, 768, 8)])
def test_calls_that_are_not_asked_about_would_get_none(K, rows, experts):
    from orin_qwen_lossless_b200 import _lib, ops
    w = _lib.Weight(4096, 8192, 3, 16, K, experts * rows, 0, 1, 256, 16640, 20000, 30000)
    for one, pairs in enumerate(ops._SCRATCH_PAIRS):
        tokens = pairs * experts - 1          # one slot each: just below the line
        assert _lib.lib().bf16n_mm_ids_scratch_bytes(C.byref(w), None if one else C.byref(w), experts, tokens, 1) == 0
