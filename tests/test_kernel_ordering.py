"""Orderings between threads that a kernel cannot do without, checked in its source.

A missing barrier or fence seldom shows in results: threads that happen to run
converged hide it.  So these tests read the kernels' text, without a GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "powergrid_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _block(text, start):
    """The braced block that begins at or after `start`."""
    i = text.index("{", text.index(start))
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i + 1:j]
    raise AssertionError("unbalanced braces")


def _spread3d_owner(ox, oy):
    """Cell -> lane of k_spread3d's window at (ox, oy): lane = 8 dx + dy holds
    (ox + dx, oy + dy) and (ox + dx + 4, oy + dy)."""
    return {(ox + dx + 4 * h, oy + dy): 8 * dx + dy for dx in range(4) for dy in range(8) for h in range(2)}


@pytest.mark.parametrize("step", [(1, 0), (0, 1), (1, 1), (2, 0), (0, -3)])
def test_spread3d_orders_a_cells_lanes(step):
    """A warp of the 3-D spread adds its registers to tile cells with plain loads and
    stores.  When the window moves, cells change their lane, so each such
    read-modify-write starts with a warp barrier."""
    a, b = _spread3d_owner(0, 0), _spread3d_owner(*step)
    assert any(a[c] != b[c] for c in a.keys() & b.keys())
    body = _block(_source("pg_nufft.cu").split("void __launch_bounds__(256) k_spread3d(", 1)[1], "auto put = [&]()")
    assert re.match(r"\s*__syncwarp\(\);", body)


def test_tensor_operand_is_rewritten_after_the_product_that_read_it():
    """k_tc_dft overwrites A in tensor memory (tcgen05.st) once the matrix product that
    read it is complete, and then takes D (tcgen05.ld).  Both need
    tcgen05.fence::after_thread_sync behind the wait on the product's mbarrier, at every
    step: the wait and the fence are one function, and nothing waits without it."""
    src = _source("pg_gdft_tc.cu")
    wait = _block(src, "bool product_wait(")
    assert re.search(r"mbar_wait\(bar, parity\);\s*asm volatile\(\"tcgen05\.fence::after_thread_sync;", wait)
    kernel = _block(src.split("k_tc_dft(", 1)[1], ") {")
    assert "mbar_wait(" not in kernel and len(re.findall(r"= product_wait\(", kernel)) == 2
    step = _block(kernel, "if (h == 0 && pending)")
    assert step.index("product_wait(") < step.index("take(") and "tm_store16(" not in step
    assert kernel.index("product_wait(") < kernel.index("tm_store16(tA")
