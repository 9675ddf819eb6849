"""GPU: constants are arguments of a compiled tape, so tapes that differ in nothing else share a kernel; and what may be
recorded before it has ever run."""
import numpy as np
import pytest

import vernondsl_b200 as vd
import vernondsl_b200.lang as ti
from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops
from vernondsl_b200.graph import Graph

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


@pytest.mark.parametrize("n", [1001, 1024, 70001])
@pytest.mark.parametrize("shape", [L.SHAPE_ROWVEC, L.SHAPE_COLVEC])
def test_sums_of_vectors_are_recorded_on_a_stream_that_has_never_run_them(n, shape):
    """Without the compiler and without scratch: both belong to a first run that a recording does not have."""
    dev = vd.Device(0)
    rows, cols = (5, n) if shape == L.SHAPE_ROWVEC else (n, 5)
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    X = dev.from_numpy(x)
    outs = [dev.empty(1, np.float32) for _ in range(3)]
    g = Graph(dev, rows, cols)
    v = g.input(X, shape)
    g.output(g.sum(v), outs[0])
    g.output(g.mean(g.unary("cos", v)), outs[1])
    g.output(g.sum(g.square(v) * v), outs[2])
    g.compile()
    x64 = x.astype(np.float64)
    want = [x64.sum(), np.cos(x64).mean(), (x64 ** 3).sum()]
    scale = [np.abs(x64).sum(), np.abs(np.cos(x64)).mean(), np.abs(x64 ** 3).sum()]
    got = []
    for recorded in (True, False):         # on a fresh stream, then plain
        st = dev.stream()
        for o in outs:
            o.fill(0xEE, stream=st)
        st.check()
        if recorded:
            with st.record() as seq:
                g.launch(st)
            seq.launch()
        else:
            g.launch(st)
        st.check()
        got.append([float(o.download()[0]) for o in outs])
        if recorded:
            seq.close()
        st.close()
        # a thread's chain is at most n / 256 groups long, then four components, five lanes' and eight warps' sums
        bound = [(n / 1024 + 24) * 2.0 ** -24 * s for s in scale]
        assert all(abs(a - b) <= e for a, b, e in zip(got[-1], want, bound)), (recorded, got, want)
    g.close()


@pytest.mark.parametrize("rows,cols", [(301, 1003), (64, 1021)])
def test_a_graph_with_sums_is_recorded_before_it_has_run(rows, cols):
    """On a stream that holds scratch (some other operator has run there): the kernels are compiled with the graph."""
    dev = vd.Device(0)
    st = dev.stream()
    x = np.random.default_rng(rows).standard_normal((rows, cols)).astype(np.float32)
    X, total, cols_out = dev.from_numpy(x), dev.empty(1, np.float32), dev.empty(cols, np.float32)
    ops.col_sum(st, X, cols_out, rows, cols)
    g = Graph(dev, rows, cols)
    v = g.input(X)
    g.output(g.mean(g.square(v)), total)
    g.output(g.reduce(L.R_COL_SUM, g.unary("cos", v)), cols_out)
    g.compile()
    with st.record() as seq:
        g.launch(st)
    seq.launch()
    st.check()
    x64 = x.astype(np.float64)
    bound = (rows / 4 + 24) * 2.0 ** -24
    assert abs(float(total.download()[0]) - (x64 ** 2).mean()) <= bound * (x64 ** 2).mean()
    c = np.cos(x64)
    assert (np.abs(cols_out.download() - c.sum(0)) <= bound * np.abs(c).sum(0)).all()
    seq.close()
    g.close()
    st.close()
