"""The row gather's skip table (codes_in_window in csrc/format.h, compiled here for the host): every entry names one to three codes
that fit 12 bits, whatever the code table holds, so the loop that skips by it always advances; on encoded matrices an entry
is what decoding its window code by code gives."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oracle import cpu_oracle as o

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "orin_qwen_lossless_b200", "csrc")


@pytest.fixture(scope="module")
def skip_table(tmp_path_factory):
    d = tmp_path_factory.mktemp("skip")
    (d / "skip.cpp").write_text('#include "format.h"\nextern "C" void skip_table(const uint32_t * lut, uint32_t * out) {\n'
                                "    for (uint32_t i = 0; i < b16::HP_MAX_PAIRS; i++) { out[i] = b16::codes_in_window(lut, i); }\n}\n")
    so = str(d / "skip.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "skip.cpp"), "-o", so], check=True)
    fn = C.CDLL(so).skip_table

    def table(lut):
        lut = np.ascontiguousarray(lut, dtype=np.uint32)
        out = np.empty(4096, np.uint32)
        fn(C.c_void_p(lut.ctypes.data), C.c_void_p(out.ctypes.data))
        return out & 0xff, out >> 8
    return table


@pytest.mark.parametrize("kind", ["random", "lengths above 12", "all ones", "zero"])
def test_every_entry_advances(skip_table, kind):
    g = np.random.default_rng(1)
    lut = {"random": g.integers(0, 1 << 32, 4096, dtype=np.uint32), "lengths above 12": g.integers(13, 32, 4096, dtype=np.uint32),
           "all ones": np.full(4096, 0xffffffff, np.uint32), "zero": np.zeros(4096, np.uint32)}[kind]
    bits, codes = skip_table(lut)
    assert ((codes >= 1) & (codes <= 3)).all() and (bits <= 12).all()


def test_entries_of_an_encoded_matrix(skip_table):
    from orin_qwen_lossless_b200 import ops
    from conftest import to_bf16_tensor
    _, aux, meta = ops.encode(to_bf16_tensor(o.weights_like(64, 1024, 5)), 3, 4, False)
    lut = aux[meta.off_a:meta.off_a + 4 * 4096].numpy().view(np.uint32)
    bits, codes = skip_table(lut)
    for i in range(4096):
        n = length = 0
        while n < 3:
            step = int(lut[(i << length) & 4095] & 31)
            if length + step > 12:
                break
            length, n = length + step, n + 1
        assert (bits[i], codes[i]) == (length, n)
