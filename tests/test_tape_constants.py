"""CPU: the text of a compiled tape does not depend on the values of its constants (they are arguments of the kernel)."""
import ctypes as C
import re

import pytest

from vernondsl_b200 import _lib as L
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


def test_a_tape_that_says_so_has_its_constants_in_the_text():
    """What the execution graph asks for: its constants never change, and multiplications by 1 or 2 fold away."""
    sources = []
    for c in (1.0, 2.0):
        t = ops.Tape(1)
        t.output(t.op("mul", t.input(0), t.const(c)))
        p = t.params(7, 9)
        p.flags |= L.TAPE_FLAG_LITERALS
        out, need = C.create_string_buffer(1 << 16), C.c_uint64()
        L.check(L.lib().vrhi_tape_source(C.byref(p), out, len(out), C.byref(need)))
        sources.append(out.value.decode())
    assert sources[0] != sources[1]
    assert "__int_as_float((int)0x3f800000u)" in sources[0] and "TapeConstants" not in sources[0]
