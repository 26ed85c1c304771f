"""Kernels that start beside the end of the kernel before them (programmatic dependent launch) read what it may have written behind
their wait and by ordinary loads, and let the next one in behind it."""
import os
import re

import pytest

from void_b200 import build

WAIT, TRIGGER = re.compile(r"grid_dependency_wait\(\)|griddepcontrol\.wait"), re.compile(r"grid_launch_dependents\(\)|griddepcontrol\.launch")


def _code(name):
    text = open(os.path.join(build.CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def _block(text, at, pair):
    """The text between the bracket at or behind ``at`` and its partner."""
    start = text.index(pair[0], at)
    depth, i = 1, start + 1
    while depth:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        i += 1
    return text[start + 1:i - 1], i


def _kernels():
    for name in sorted(f for f in os.listdir(build.CSRC) if f.endswith((".cu", ".cuh"))):
        text = _code(name)
        for m in re.finditer(r"__global__ void (?:__launch_bounds__)?", text):
            at = m.end()
            if text[m.start():at].endswith("__launch_bounds__"):
                at = _block(text, at, "()")[1]
            kernel = re.compile(r"\s*(\w+)").match(text, at).group(1)
            params, end = _block(text, at, "()")
            yield name, kernel, params, _block(text, end, "{}")[0]


KERNELS = list(_kernels())
WAITING = [k for k in KERNELS if WAIT.search(k[3]) or "pipeline_setup" in k[3]]


def test_the_kernels_are_found():
    names = {k[1] for k in WAITING}
    assert {"tile_index_kernel", "pack_tiles_kernel", "row_order_kernel", "quant_tiles_kernel", "quant_cols_fused_kernel", "column_sum_kernel",
            "copy_rows_kernel", "transpose_kernel", "rank_bitmap_kernel", "skinny_kernel", "group_kernel", "spmm_rowacc_kernel",
            "spmm_drain_kernel"} <= names
    assert "mark_tiles_kernel" not in names and len(KERNELS) > len(WAITING) + 10


@pytest.mark.parametrize("kernel", WAITING, ids=lambda k: k[1])
def test_a_kernel_that_waits_reads_by_ordinary_loads(kernel):
    _, name, params, body = kernel
    assert not re.search(r"const [\w: ]+\* ?(?:const )?__restrict__", params), name
    assert "__ldg(" not in body and "ld.global.nc" not in body, name


def test_nor_does_what_those_kernels_call():
    for name in ("pipeline.cuh", "rowacc.cuh", "epilogue.cuh", "skinny.cu", "spmm.cu", "group.cu", "prep.cu", "ptx.cuh"):
        code = _code(name)
        assert "__ldg(" not in code and "ld.global.nc" not in code, name


@pytest.mark.parametrize("kernel", [k for k in WAITING if TRIGGER.search(k[3])], ids=lambda k: k[1])
def test_the_next_kernel_is_let_in_behind_the_wait(kernel):
    _, name, _, body = kernel
    assert WAIT.search(body).start() < TRIGGER.search(body).start(), name


def test_only_kernels_that_wait_are_launched_beside_the_one_before():
    waiting = {k[1] for k in WAITING}
    for name in sorted(f for f in os.listdir(build.CSRC) if f.endswith((".cu", ".cuh"))):
        for m in re.finditer(r"launch_pdl\((?:kind == \w+ \? )?(\w+_kernel)", _code(name)):
            assert m.group(1) in waiting, (name, m.group(1))
