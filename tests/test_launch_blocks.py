"""CPU: the parameter blocks that ops.py lays out with struct are the ctypes structures, byte for byte."""
import ctypes as C
import random

import pytest

from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops


def test_argument_array():
    args = [(0x7F0000001000 + k, k, 3 * k, k % 5, 0) for k in range(16)]
    for n in range(17):
        arr = (L.Arg * n)()
        for a, (h, off, nbytes, cls, _) in zip(arr, args):
            a.buffer, a.offset, a.bytes, a.arg_class = h, off, nbytes, cls
        assert bytes(arr) == ops._ARGS[n].pack(*[f for a in args[:n] for f in a])


@pytest.mark.parametrize("rows,cols", [(0, 0), (1, 5), (1 << 40, 3), (-1, 7)])
def test_shapes(rows, cols):
    p = L.RowsParams()
    p.size, p.rows, p.cols = C.sizeof(p), rows, cols
    assert bytes(p) == ops._rows(rows, cols)
    p = L.MapParams()
    p.size, p.n = C.sizeof(p), rows
    assert bytes(p) == ops._MAP.pack(16, 0, rows & ops._M64)
    assert bytes(ops._mse(rows, cols, 2.5)) == ops._MSE.pack(32, 0, rows & ops._M64, cols & ops._M64, 2.5)


def test_tapes():
    rng = random.Random(4)
    for trial in range(200):
        n_in = rng.randrange(1, L.TAPE_MAX_INPUTS + 1)
        t = ops.Tape(n_in, row_vectors=[k for k in range(n_in) if rng.random() < 0.3])
        for _ in range(rng.randrange(0, L.TAPE_MAX_INSTR + 1)):
            top = n_in + len(t.instr)
            if rng.random() < 0.2:
                t.const(rng.choice([0.0, -0.0, 1e-45, 3.4e38, 1e39, float("inf"), rng.uniform(-5, 5)]))
            else:
                t.op(rng.choice(sorted(L.T)), *[rng.randrange(top) for _ in range(3)])
        for _ in range(rng.randrange(1, L.TAPE_MAX_OUTPUTS + 1)):
            t.output(rng.randrange(n_in + len(t.instr)), col_sum=rng.random() < 0.3)
        rows, cols = rng.choice([(1, 1), (4, 7), (-2, 5), (1 << 33, 9)])
        for flags in (0, L.TAPE_FLAG_INTERPRET):
            p = t.params(rows, cols)
            p.flags |= flags
            assert bytes(p) == t._block(rows, cols, flags)
    t.instr += [(0, 0, 0, 0, 0.0)] * (L.TAPE_MAX_INSTR + 1)
    with pytest.raises(ValueError):
        t._block(1, 1, 0)
