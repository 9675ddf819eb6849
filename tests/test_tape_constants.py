"""CPU: the text of a compiled tape does not depend on the values of its constants (they are arguments of the kernel)."""
import re

import pytest

from vernondsl_b200 import ops


def source(c, rows, cols):
    t = ops.Tape(2, row_vectors=[1])
    x, r = t.input(0), t.input(1)
    t.output(t.op("fma", t.op("max", x, t.const(c)), t.const(2 * c), t.op("div", r, t.const(3.0))))
    return ops.tape_source(t, rows, cols)


@pytest.mark.parametrize("rows,cols", [(30, 1001), (30, 1002), (30, 1024), (1, 17)])
def test_the_text_does_not_depend_on_the_constants(rows, cols):
    comments = re.compile(r"//[^\n]*")
    a, b = source(0.5, rows, cols), source(-7.25, rows, cols)
    assert a != b                                           # shown for inspection, as comments
    assert comments.sub("", a) == comments.sub("", b)
    assert "0x3f000000" in a and "0x3f000000" not in comments.sub("", a)
