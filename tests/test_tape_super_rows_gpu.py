"""GPU: compiled tapes over row lengths that are no multiple of 4, which are walked several rows at a time (tape_jit.cpp):
the interpreting kernel's bits for every remainder of rows and columns, and column sums and totals against binary64."""
import numpy as np
import pytest

from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops

SHAPES = [(r, c) for c in (1, 2, 3, 5, 6, 7, 10, 63, 65, 254, 257, 1001, 1022) for r in (1, 2, 3, 4, 5, 6, 7, 8, 131)] + [(2049, 1001), (1081, 1919), (3, 40001), (20001, 3)]


def expression(**shapes):
    """sigmoid(x*a + b) * y + |x| + s"""
    t = ops.Tape(5, **shapes)
    x, y, a, b, s = (t.input(k) for k in range(5))
    return t, t.op("add", t.op("fma", t.op("sigmoid", t.op("fma", x, a, b)), y, t.op("abs", x)), s)


@pytest.mark.gpu
def test_the_interpreters_bits_and_the_sums(dev, stream):
    rng = np.random.default_rng(9)
    for rows, cols in SHAPES:
        for shapes in ({"row_vectors": [2, 3], "scalars": [4]}, {"row_vectors": [2], "col_vectors": [3], "scalars": [4]}):
            host = []
            for k in range(5):
                n = rows * cols if k < 2 else cols if k in shapes["row_vectors"] else 1 if k == 4 else rows
                host.append(rng.standard_normal(n).astype(np.float32))
            ins = [dev.from_numpy(h, L.INPUT) for h in host]
            guard, n = 16, rows * cols
            outs = [dev.from_numpy(np.full(n + guard, 7.0, np.float32), L.OUTPUT) for _ in range(2)]
            t, v = expression(**shapes)
            t.output(v)
            for o, interpret in zip(outs, (False, True)):
                before = ops.tape_jit_stats()["launches"]
                ops.map_tape(stream, t, ins, [o], rows, cols, interpret=interpret)
                compiled = not interpret and rows * cols >= 256      # smaller ones are the interpreter's
                assert ops.tape_jit_stats()["launches"] - before == compiled, (rows, cols)
            stream.check()
            got, want = (o.download() for o in outs)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (rows, cols, shapes)
            assert (got[n:] == 7.0).all()
            # the same value summed by columns, summed whole (mean), and stored, in one kernel
            t, v = expression(**shapes)
            t.output(v, col_sum=True)
            t.output(v)
            t.output(v)
            p = t.params(rows, cols)
            p.flags, p.total_mask = L.TAPE_FLAG_TOTALS, (1 << 2) | (1 << 10)
            cs, st, to = (dev.from_numpy(np.full(k + guard, 7.0, np.float32), L.OUTPUT) for k in (cols, n, 1))
            ops.launch(stream, "map_tape", [b.arg(L.INPUT) for b in ins] + [b.arg(L.OUTPUT) for b in (cs, st, to)], p)
            stream.check()
            full = want[:n].reshape(rows, cols).astype(np.float64)
            assert np.array_equal(st.download(), want)
            c = cs.download()
            # at most rows roundings per column, of partial sums no larger than the sum of magnitudes
            depth = 16 + rows / 16
            assert (np.abs(c[:cols] - full.sum(0)) <= depth * 2.0 ** -24 * np.abs(full).sum(0) + 1e-30).all(), (rows, cols)
            assert (c[cols:] == 7.0).all()
            m = to.download()
            assert abs(m[0] - full.mean()) <= (depth + 16) * 2.0 ** -24 * np.abs(full).mean() and (m[1:] == 7.0).all()
            for b in ins + outs + [cs, st, to]:
                b.close()
