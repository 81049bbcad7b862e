"""A window's kernels are launched so that each may start while the one before
drains, and each waits for that one only.  So each has to wait whatever the
network: one that ended without waiting would cut the chain, and the kernel after
it could start while the kernel before it still runs.  A race of that kind need
not show on any one machine; the sources are read instead.  In the per-step
kernels and those of the inputs and the delivery the wait stands outside every
branch and loop, or is made up for there; in the cell kernel it stands in its units' routines, once for a
block's first unit (every block has one)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eden_gb300", "csrc")


def _body(text, name):
    """The body of the kernel or device function `name`, comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    m = re.search(r"\b%s\(" % name, text)
    a = text.index("{", m.end())
    depth, k = 1, a + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        k += 1
    return text[a + 1:k - 1]


def _top_level(body):
    """Statements of a body that stand outside its inner braces."""
    out, depth = [], 0
    for ch in body:
        depth += {"{": 1, "}": -1}.get(ch, 0)
        out.append(ch if depth == 0 and ch != "}" else ";" if depth == 0 else " ")
    return [s.strip() for s in "".join(out).split(";")]


def _window():
    return open(os.path.join(CSRC, "eden_window.cuh")).read()


@pytest.mark.parametrize("kernel", ["k_inputs_t", "k_targets_t", "k_hines_t", "k_deliver_t"])
def test_waits_in_every_network(kernel):
    statements = _top_level(_body(_window(), kernel))
    assert "kernel_order()" in statements or "if (!waited) kernel_order()" in statements


@pytest.mark.parametrize("routine", ["forest_window", "izh_window"])
def test_a_unit_of_the_cell_kernel_waits(routine):
    assert "if (first) kernel_order()" in _top_level(_body(_window(), routine))


def test_every_launch_is_one_of_these():
    launches = re.findall(r"launch_order\([^;]*?ctx->(fn_\w+)|launch_order\([^;]*?\(const void \*\)(k_\w+)",
                          open(os.path.join(CSRC, "eden_gpu.cu")).read())
    assert {a or b for a, b in launches} == {"fn_inputs", "fn_cells", "fn_deliver", "k_targets_t", "k_hines_t"}
