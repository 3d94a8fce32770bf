"""Rules of the kernel sources that no run shows reliably."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crit_kernels_b200", "csrc")


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def early_starters():
    """Sources of the kernels that are resident while the previous kernel of the stream still runs."""
    names = [n for n in sorted(os.listdir(CSRC)) if "griddepcontrol.wait" in code(n)]
    assert {"dg_kernel.cuh", "dg_quantize.cu", "dg_swiglu.cu"} <= set(names)
    return names


@pytest.mark.parametrize("name", early_starters())
def test_kernels_that_start_early_read_nothing_through_the_read_only_path(name):
    """Loads through the non-coherent path (ld.global.nc, __ldg, const __restrict__ parameters, which the compiler turns into
    such loads) are for memory nobody writes during a kernel's whole life. The previous kernel may write what these read: its
    outputs are their activations, and scales unless the caller has declared them static. (A batch's launch parameters are
    read before the wait as it is, so they have to be there before the previous kernel starts.)"""
    text = code(name)
    assert not re.findall(r"ld\.global\.nc|\b__ldg\s*\(|\bldg_nc\w*", text)
    restricted = re.findall(r"const\s+(\w+)\s*\*\s*__restrict__\s+(\w+)", text)
    assert set(restricted) <= {("Params", "items")}, restricted


def test_the_plan_is_what_its_description_says_and_the_version_tells_it_from_the_earlier_one():
    """plan[1] used to be the rows per consumer warp; since every consumer warp takes all rows of a tile it is a tile's groups of
    16 rows, under its own name and a library version of its own."""
    from crit_kernels_b200 import cabi
    assert cabi.load().dg_version() >= 103
    for fmt, n, k, row in (("nvfp4", 8192, 8192, 2 * 512 + 16 + 2 * 64 + 16), ("fp8", 28672, 8192, 2 * 512 + 16)):
        p = cabi.plan(fmt, 1, n, k)                  # (resident activations: a stage is rows of weights and scales)
        assert p["row_groups"] == -(-(p["stage_bytes"] // row) // 16) and p["row_groups"] == p["rows_per_warp"]


def test_the_build_description_names_every_source():
    with open(os.path.join(os.path.dirname(CSRC), "build.toml")) as f:
        named = re.findall(r'"csrc/([^"]+)"', f.read())
    assert sorted(named) == sorted(os.listdir(CSRC))


def test_every_kernel_launched_early_waits_and_the_dequantizer_lets_nobody_start_before_it_has_ended():
    """A kernel launched with programmatic dependent launch reads and writes global memory behind its wait only. The dequantizer's
    output is a weight matrix, which a GEMV told of static weights reads before its own wait, so its successor may not start early."""
    launched = {n for n in os.listdir(CSRC) if "ProgrammaticStreamSerialization" in code(n)}
    waiting = {"dg_abi.cu" if n == "dg_kernel.cuh" else n for n in early_starters()}     # (which launches that header's kernels)
    assert {"dg_abi.cu", "dg_dequant.cu"} <= launched == waiting
    text = code("dg_dequant.cu")
    assert "launch_dependents" not in text
    body = text[text.index("dequantize_kernel("):]
    before, behind = body.split("griddepcontrol.wait", 1)
    touched = r"\b(?:codes|scales|factor|out)\)?\s*\["
    assert not re.findall(touched, before) and len(re.findall(touched, behind)) >= 6
