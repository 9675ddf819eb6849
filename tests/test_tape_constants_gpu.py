"""GPU: constants are arguments of a compiled tape, so tapes that differ in nothing else share a kernel; and what may be
recorded before it has ever run."""
import numpy as np
import pytest

import vernondsl_b200 as vd
import vernondsl_b200.lang as ti
from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops

pytestmark = pytest.mark.gpu


def stats():
    return ops.tape_jit_stats()


@pytest.mark.parametrize("width", [1001, 1026, 1024])
def test_a_moving_uniform_compiles_one_kernel(width):
    ti.init()
    x, o = ti.field(float, (30, width)), ti.field(float, (30, width))
    host = np.random.default_rng(width).standard_normal((30, width)).astype(np.float32)
    x.from_numpy(host)

    @ti.kernel
    def scaled(t: float):
        for i, j in o:
            o[i, j] = ti.max(x[i, j] * t + 1.5, t)

    def want(t):
        t = np.float32(t)
        return np.maximum(host * t + np.float32(1.5), t)

    before = stats()
    uniforms = [0.5, -2.0, 0.0, -0.0, 3.25, np.inf, 1e-40, 7.0]
    for t in uniforms:
        scaled(t)
        assert np.array_equal(o.to_numpy(), want(t), equal_nan=True), t
    after = stats()
    assert after["compiled"] - before["compiled"] <= 1
    assert after["launches"] - before["launches"] == len(uniforms)
    loop = ti.FrameLoop(scaled, o, ring=4)
    loop.record([0.25 * k for k in range(9)])
    loop.play()
    for k in range(5, 9):
        assert np.array_equal(loop.frame(k), want(0.25 * k)), k
    assert stats()["compiled"] == after["compiled"]
    loop.close()


@pytest.mark.parametrize("rows,cols", [(30, 1001), (64, 1028), (1, 1003)])
def test_a_tape_that_has_never_run_is_recorded_with_the_interpreter(rows, cols):
    dev = vd.Device(0)
    st = dev.stream()
    x = np.random.default_rng(cols).standard_normal((rows, cols)).astype(np.float32)
    X, O, W = dev.from_numpy(x), dev.empty((rows, cols), np.float32), dev.empty((rows, cols), np.float32)
    t = ops.Tape(1)
    v = t.input(0)
    for k in range(2 + rows % 5):          # a tape of its own per shape
        v = t.op("fma", v, t.const(1.0 + k), t.op("cos", v))
    t.output(v)
    before = stats()
    with st.record() as seq:
        ops.map_tape(st, t, [X], [O], rows, cols)
    assert stats() == before               # neither compiled nor launched
    seq.launch()
    ops.map_tape(st, t, [X], [W], rows, cols)
    assert stats()["compiled"] == before["compiled"] + 1
    st.check()
    assert np.array_equal(O.download().view(np.uint32), W.download().view(np.uint32))
    seq.close()
    st.close()
