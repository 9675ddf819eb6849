"""GPU: the two forms of a compiled tape (one long array with a tail; rows, several at a time where their length is no
multiple of 4) at the edges of their tiling, against the interpreting kernel (same bits) and, for summed
outputs, binary64 sums of the stored values (1e-5 of the sum of magnitudes, as in test_rows_gpu.py)."""
import numpy as np
import pytest

from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops

pytestmark = pytest.mark.gpu

SHAPES = [(1, 257), (300, 1), (3, 1023), (2, 1024), (129, 255), (77, 256), (31, 257), (1081, 1919), (5000, 33), (5000, 36), (9, 4100), (2, 300001), (1, 1000003)]


def launch(stream, tape, inputs, outputs, rows, cols, flags=0, colsum=0, total=0):
    p = tape.params(rows, cols)
    p.flags |= flags
    p.colsum_mask, p.total_mask = colsum, total
    ops.launch(stream, "map_tape", [b.arg(L.INPUT) for b in inputs] + [b.arg(L.OUTPUT) for b in outputs], p)


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("broadcast", [False, True])
def test_every_form_gives_the_interpreters_bits(dev, stream, rows, cols, broadcast):
    rng = np.random.default_rng(rows * 7 + cols)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    arrays = [f(rows, cols), f(rows, cols)] + ([f(cols), f(rows)] if broadcast else [f(1), f(1)])
    bufs = [dev.from_numpy(a) for a in arrays]
    t = ops.Tape(4, row_vectors=[2] if broadcast else [], col_vectors=[3] if broadcast else [], scalars=[] if broadcast else [2, 3])
    u = t.op("tanh", t.op("fma", t.input(0), t.input(2), t.input(3)))
    t.output(u)
    t.output(t.op("mul", u, t.input(1)))
    got = [dev.empty((rows, cols), np.float32) for _ in range(2)]
    ref = [dev.empty((rows, cols), np.float32) for _ in range(2)]
    for b in got:
        b.fill(0xEE, stream=stream)
    before = ops.tape_jit_stats()["launches"]
    ops.map_tape(stream, t, bufs, got, rows, cols)
    assert ops.tape_jit_stats()["launches"] == before + 1      # not the interpreter against itself
    ops.map_tape(stream, t, bufs, ref, rows, cols, interpret=True)
    assert ops.tape_jit_stats()["launches"] == before + 1
    stream.check()
    stored = [b.download() for b in ref]
    for g, r in zip(got, stored):
        assert np.array_equal(g.download(), r)
    # the same two values, the first as column sums or as one sum, the second as one mean
    scale = np.abs(stored[0]).astype(np.float64)
    sums, mean = dev.empty(cols, np.float32), dev.empty(4, np.float32)
    launch(stream, t, bufs, [sums, mean], rows, cols, L.TAPE_FLAG_TOTALS, colsum=1, total=0x0202)
    total = dev.empty(4, np.float32)
    launch(stream, t, bufs, [total, got[1]], rows, cols, L.TAPE_FLAG_TOTALS, total=0x0001)
    stream.check()
    assert (np.abs(sums.download() - stored[0].astype(np.float64).sum(axis=0)) <= 1e-5 * scale.sum(axis=0) + 1e-30).all()
    want = stored[1].astype(np.float64)
    assert abs(mean.download()[0] - want.mean()) <= 1e-5 * np.abs(want).mean()
    assert abs(total.download()[0] - stored[0].astype(np.float64).sum()) <= 1e-5 * scale.sum()
    assert np.array_equal(got[1].download(), stored[1])
    for b in bufs + got + ref + [sums, mean, total]:
        b.close()
