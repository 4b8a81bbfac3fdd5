"""How the kernels' waits end that something never comes for, and the orders in their sources that no wait may depend on."""

import os
import re

import pytest

from freetoken_b200.kernels import library, ops


def sources():
    for name in sorted(os.listdir(library.CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(library.CSRC, name)) as f:
                yield name, re.sub(r"//[^\n]*", "", f.read())


def test_what_a_warp_does_together_follows_waits_that_end_alike_for_all_its_lanes():
    """Lanes of a warp that give up singly would leave the others at elect.sync and tcgen05 instructions without end: every wait is voted
    on, at once or (issuing warps) at the end of the key tile, with no way out before that."""
    seen = 0
    for name, text in sources():
        if not name.startswith("attention_tc"):
            continue
        for m in re.finditer(r"mbar_wait2?\(", text):
            before = text[max(text.rindex(";", 0, m.start()), text.rindex("{", 0, m.start())):m.start()]
            seen += 1
            if "all_of_warp(" in before or "__all_sync(" in before:
                continue
            rest = text[m.end():text.index("ok = all_of_warp(fine)", m.end())]
            assert "fine = false;" in rest[:600] and not re.search(r"\b(break|return|continue)\b", rest), (name, text[m.start() - 80:m.end() + 60])
        for issue in re.finditer(r"elect_one\(\)\) ([^\n]*)", text):
            assert issue.group(1).startswith("if (fine)")
    assert seen > 25


def test_tensor_memory_is_allocated_before_the_next_kernel_may_start():
    """A kernel that comes in early may hold columns until this one ends: this one must not still be waiting for its own."""
    checked = 0
    for name, text in sources():
        for kernel in re.split(r"__global__", text)[1:]:
            alloc, trigger = re.search(r"\btmem_alloc\(&", kernel), kernel.find("pdl_trigger();")
            if not alloc or trigger < alloc.start():
                continue
            assert "__syncthreads();" in kernel[alloc.start():trigger], (name, kernel[:60])
            checked += 1
    assert checked >= 6


@pytest.mark.gpu
def test_a_lost_wait_ends_within_its_limit():
    ok, seconds = ops.debug_lost_wait(False)
    # 2^31 cycles at 1,965 MHz are 1.09 s, at half of that clock 2.2 s; and one try more
    assert not ok and 1.0 < seconds < 3.0, seconds
    ok, seconds = ops.debug_lost_wait(True)
    assert not ok and 1e-4 <= seconds < 0.01, seconds


@pytest.mark.gpu
@pytest.mark.parametrize("unit,code", [(0, 101), (1, 201), (2, 501), (3, 601), (4, 701)])
def test_every_status_word_is_read_and_cleared(unit, code):
    assert ops.read_status() == 0
    ops.debug_set_status(unit, code)
    with pytest.raises(ops.KernelError, match=f"status {code}"):
        ops.check_status()
    assert ops.read_status() == 0
