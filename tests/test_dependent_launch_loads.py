"""Kernels launched with launch_chained or launch_behind may start before the kernel in front of them has finished: what that kernel writes
(activations, routing) must be read behind the dependency wait with ordered loads, never through the read-only path
(ld.global.nc), which the compiler may move above the wait and which may serve lines fetched before the stores. Checked on the
sources: __ldg and ld_stream16 in such kernels read matrices only, and their read-only pointer parameters are read through
the ordered helpers only."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "orin_qwen_lossless_b200", "csrc")
SOURCES = {f: re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read()) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}
# what a matrix's view gives: code table, unit and lane offsets, row tables, escapes, plane (pl, pw: pointers into it)
MATRIX = re.compile(r"\b(lut|ubase|lrel|row_lut|esc_off|esc|plane|codes|pl|stream|pfirst|nrow)\b")
CHAINED = sorted({k for s in SOURCES.values() for call in re.findall(r"launch_(?:chained|behind)\(([^;]*?)dim3|launch_(?:chained|behind)\(([^;]*?), grid", s)
                  for k in re.findall(r"\bk_\w+", " ".join(call))})


# read-only parameters that are older than the kernel in front, which itself waited for everything before it
OLDER = {("k_combine_f32", "w")}


def _block(s, start):
    depth, i = 0, s.index("{", start)
    for j in range(i, len(s)):
        depth += {"{": 1, "}": -1}.get(s[j], 0)
        if depth == 0:
            return s[i:j + 1]


def _kernel(name):
    for s in SOURCES.values():
        m = re.search(r"__global__[^;{]*?\b" + name + r"\(([^{;]*)\)\s*\{", s)
        if m:
            return m.group(1), _block(s, m.start(1) + len(m.group(1)))
    raise AssertionError(name)


def test_the_list_is_found():
    assert {"k_tile_mm", "k_expand_tiles", "k_expand_tiles_fo", "k_nib_gemv", "k_swiglu", "k_topk", "k_combine_f32", "k_expert_units",
            "k_pair_rows_staged", "k_select", "k_rescore", "k_fo_gemv_split"} <= set(CHAINED)


@pytest.mark.parametrize("name", CHAINED)
def test_ordered_loads(name):
    params, body = _kernel(name)
    for arg in re.findall(r"(?:__ldg|ld_stream16)\(((?:[^()]|\([^()]*\))*)\)", body):
        assert MATRIX.search(arg), f"{name} reads {arg} through the read-only path"
    for p in re.findall(r"const [\w:]+ \*\s*__restrict__ (\w+)", params):
        if (name, p) in OLDER:
            continue
        assert not re.search(rf"\b{p}\s*\[", body), f"{name} reads {p} without an ordered load"
        for alias in re.findall(rf"(\w+) = {p} \+", body):
            assert not re.search(rf"\b{alias}\s*\[", body), f"{name} reads {p} (as {alias}) without an ordered load"


def test_pass_walk_of_the_tile_product():
    s = SOURCES["prefill.cu"]
    assert "__ldg" not in _block(s, s.index("struct TileWalk"))


def test_kernels_that_let_their_successor_start_wait_themselves():
    for f, s in SOURCES.items():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\([^{;]*\)\s*\{", s):
            body = _block(s, m.end() - 1)
            if "grid_launch_dependents()" in body:
                waits = "grid_dependency_wait()" in body or any("grid_dependency_wait()" in _block(s, s.index(h)) for h in ("nib_item_rows(",) if h in body)
                assert waits, f"{m.group(1)} in {f}"
