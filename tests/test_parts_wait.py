"""The kernels that walk units in parts share their loads (parts.cuh): where each of them waits for the kernel in front, and that what they
read through the read-only path belongs to the matrix. Checked on the sources."""
import re

import pytest
from test_dependent_launch_loads import MATRIX, SOURCES, _block, _kernel

WALKERS = sorted(m.group(1) for f, s in SOURCES.items() if f.endswith(".cu") for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\([^{;]*\)\s*\{", s)
                 if "walk_parts<" in _block(s, m.end() - 1))


def test_the_walkers_are_found():
    assert WALKERS == ["k_down_combine", "k_expand_parts", "k_expert_parts", "k_gemv_parts"]


def test_dense_products_wait_before_they_read_the_matrix():
    body = _kernel("k_gemv_parts")[1]
    wait = body.index("grid_dependency_wait()")
    assert wait < min(body.index(read) for read in ("stage_table(", "walk_parts<", "p.w.", "p.marks") if read in body)


@pytest.mark.parametrize("name", WALKERS + ["k_rows_parts"])
def test_they_wait_before_their_successor_starts(name):
    assert "grid_dependency_wait()" in _kernel(name)[1]


def test_what_the_down_kernels_read_above_the_wait():
    """Ids and weights are older than the gate / up launch in front, which waited for them before it let these start; nothing else may be read there."""
    for name, older in (("k_down_combine", {"p.ids", "weights"}), ("k_fo_down_combine", {"ids", "weights"})):
        params, body = _kernel(name)
        above = body[:body.index("grid_dependency_wait()")]
        for p in re.findall(r"(?:const )?(?:float|int32_t) \* (?:__restrict__ )?(\w+)", params):
            assert p in older or not re.search(rf"\b{p}\b", above), (name, p)
        for read in ("p.x", "ldg_x4", "ld_act"):
            assert read not in above, (name, read)
    for f, function, kernel, front in (("moe_decode.cu", "void moe_decode(", "k_down_combine", "launch_units<4, 8, true"), ("moe_decode.cu", "void moe_decode_frag_order(", "fo_down_combine(", "fo_gemv_two(")):
        s = SOURCES[f]
        body = _block(s, s.index(function))
        assert 0 <= body.index(front) < body.index(kernel)
        assert sum(k.count("launch_chained(" + kernel) for k in SOURCES.values()) <= 1


def test_rows_are_gathered_behind_the_callers_kernels():
    assert "k_rows_parts" not in re.findall(r"launch_chained\((\w+)", SOURCES["gemv_parts.cu"])
    launch = SOURCES["gemv_parts.cu"]
    launch = _block(launch, launch.index("void rows_parts("))
    assert re.search(r"launch_behind\(behind_own, kernel", launch) and launch.count("go(k_rows_parts<") == 3 and "<<<" not in launch


@pytest.mark.parametrize("name", ["parts.cuh", "k_rows_parts"])
def test_read_only_loads_are_the_matrix(name):
    body = SOURCES[name] if name in SOURCES else _kernel(name)[1]
    found = re.findall(r"(?:__ldg|ld_stream16)\(((?:[^()]|\([^()]*\))*)\)", body)
    assert found
    for arg in found:
        assert MATRIX.search(arg) or re.search(r"\b(marks|from|cur|next)\b", arg), arg     # from, cur, next: PartPlane's pointers into the plane


def test_an_expired_wait_of_a_gathered_row_is_the_row_gathers():
    assert "g_wait_expired" not in _kernel("k_rows_parts")[1] and "g_row_wait_expired" in _kernel("k_rows_parts")[1]
    s = SOURCES["capi.cu"]
    bits = re.search(r"FAULT_BITS\[FAULT_WORDS\] = \{([^}]*)\}", s).group(1).replace(" ", "").split(",")
    words = dict(re.findall(r"g_fault_words\[(\d)\] = (\w+)\(\)", s))
    of = {words[str(i)]: b.strip() for i, b in enumerate(bits)}
    assert of["rows_parts_fault_word"] == of["row_gather_fault_word"] == "BF16N_FAULT_ROW_GATHER" and of["gemv_parts_fault_word"] == "BF16N_FAULT_GEMV_STAGED"
