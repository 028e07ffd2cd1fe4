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
