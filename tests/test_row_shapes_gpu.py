"""GPU: every row kernel at the edges of its range of row lengths, against binary64."""
import numpy as np
import pytest

from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops

# lengths at which the kernel, the split of a row or the registers per thread change, and their odd neighbours
COLS = [1, 2, 12, 68, 1020, 1012, 8164, 8165, 16357, 32740, 32741, 32764, 131043, 131044, 3, 4, 5, 15, 16, 17, 63, 64, 65, 67, 68, 127, 129, 255, 256, 257, 511, 1001, 1024, 1025, 1028, 2047, 2049, 4096, 4099, 5121, 8192, 8193,
        10007, 10240, 12292, 16384, 16387, 20483, 32768, 32771, 40001, 65536, 65539, 131072, 131075, 131079]
ROWS = [1, 2, 5, 33, 150]


def shapes():
    for c in COLS:
        for r in ROWS:
            if c * r <= 1 << 22:
                yield r, c


@pytest.mark.gpu
def test_sums_maxima_and_softmax_of_every_row_length(dev, stream):
    rng = np.random.default_rng(5)
    for rows, cols in shapes():
        x = rng.standard_normal((rows, cols)).astype(np.float32) * 3
        X = dev.from_numpy(x, L.INPUT)
        guard = 64      # nothing may be written behind an output
        S, M, S2, M2 = (dev.from_numpy(np.full(rows + guard, 7.0, np.float32), L.OUTPUT) for _ in range(4))
        P, Q = (dev.from_numpy(np.full(rows * cols + guard, 7.0, np.float32), L.OUTPUT) for _ in range(2))
        ops.row_sum(stream, X, S, rows, cols)
        ops.row_max(stream, X, M, rows, cols)
        ops.row_softmax(stream, X, P, rows, cols)
        ops.row_stats_softmax(stream, X, S2, M2, Q, rows, cols)
        stream.check()
        x64 = x.astype(np.float64)
        # each sum is a tree of at most 40 roundings deep in every kernel but the streaming ones, whose trips add one more each
        depth = 48 + cols / 4096
        bound = depth * 2.0 ** -24 * np.abs(x64).sum(1)
        for s in (S, S2):
            s = s.download()
            assert (np.abs(s[:rows] - x64.sum(1)) <= bound).all(), (rows, cols)
            assert (s[rows:] == 7.0).all()
        for m in (M, M2):
            m = m.download()
            assert np.array_equal(m[:rows], x.max(1)), (rows, cols)
            assert (m[rows:] == 7.0).all()
        e = np.exp(x64 - x64.max(1, keepdims=True))
        want = e / e.sum(1, keepdims=True)
        for p in (P, Q):
            p = p.download()
            got = p[:rows * cols].reshape(rows, cols)
            # exponential: 2e-6 (k_rows.cu, exp2_approx); normaliser: the depth above; two more roundings
            assert (np.abs(got - want) <= (2e-6 + (depth + 4) * 2.0 ** -24) * want + 1e-38).all(), (rows, cols)
            assert (p[rows * cols:] == 7.0).all(), (rows, cols)
        for b in (X, S, M, S2, M2, P, Q):
            b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cols", [3, 16, 40, 64, 65, 100, 257, 1001, 4096, 4099, 10007, 20000, 50001, 140001])
def test_infinities_nan_and_the_lowest_value(dev, stream, cols):
    f = np.float32
    x = np.random.default_rng(2).standard_normal((7, cols)).astype(f)
    x[0, :] = -np.inf
    x[1, : cols // 2] = -np.inf                 # a whole slice or lane may hold nothing but -inf
    x[2, cols // 3] = np.inf
    x[3, cols - 1] = np.nan
    x[4, :] = np.finfo(f).min
    x[5, :-1] = np.finfo(f).min
    rows = x.shape[0]
    X = dev.from_numpy(x, L.INPUT)
    S, M = dev.empty(rows, f, L.OUTPUT), dev.empty(rows, f, L.OUTPUT)
    P = dev.empty((rows, cols), f, L.OUTPUT)
    ops.row_stats_softmax(stream, X, S, M, P, rows, cols)
    stream.check()
    m, p = M.download(), P.download()
    ops.row_max(stream, X, M, rows, cols)
    stream.check()
    m2 = M.download()
    want = np.fmax.reduce(x, axis=1)
    assert np.array_equal(m, want) and np.array_equal(m2, want)
    assert np.isnan(p[0]).all() and np.isnan(p[3]).all()
    assert np.isnan(p[2]).all()
    assert (p[1, : cols // 2] == 0).all()
    assert abs(float(p[1].astype(np.float64).sum()) - 1) < 1e-5
    if cols % 4 or cols <= 64 or cols > 8192:    # the lengths whose exponential is of x - max
        assert np.allclose(p[4], 1.0 / cols, rtol=1e-5)
    assert p[5, -1] == 1.0 and (p[5, :-1] == 0).all()
    assert abs(float(p[6].astype(np.float64).sum()) - 1) < 1e-5
    for b in (X, S, M, P):
        b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cols", [67, 1001, 10007, 20483, 32741, 40001, 50002, 140003])
@pytest.mark.parametrize("special", [np.nan, np.inf, -np.inf])
def test_special_values_at_the_ends_of_rows_of_every_phase(dev, stream, cols, special):
    """The first and the last element of a row lie in front of and behind its float4 groups, how many of them there are
    depends on where the row starts: eight rows of one length, four with the value first and four with it last."""
    f = np.float32
    x = np.random.default_rng(cols).standard_normal((8, cols)).astype(f)
    x[:4, 0] = special
    x[4:, -1] = special
    rows = x.shape[0]
    X = dev.from_numpy(x, L.INPUT)
    S, M, M2 = (dev.empty(rows, f, L.OUTPUT) for _ in range(3))
    P, Q = (dev.empty((rows, cols), f, L.OUTPUT) for _ in range(2))
    ops.row_stats_softmax(stream, X, S, M, P, rows, cols)
    ops.row_max(stream, X, M2, rows, cols)
    ops.row_softmax(stream, X, Q, rows, cols)
    stream.check()
    want = np.fmax.reduce(x, axis=1)
    assert np.array_equal(M.download(), want) and np.array_equal(M2.download(), want)
    s, p, q = S.download(), P.download(), Q.download()
    if special == -np.inf:
        assert (s == -np.inf).all() and (p[:4, 0] == 0).all() and (p[4:, -1] == 0).all()
        assert (np.abs(p.astype(np.float64).sum(1) - 1) < 1e-5).all()
    else:      # x - max is NaN at the value itself, so the row's normaliser is
        assert (np.isnan(s) if special != special else s == special).all()
        assert np.isnan(p).all()
    assert np.array_equal(p, q, equal_nan=True)
    for b in (X, S, M, M2, P, Q):
        b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cols", [40001, 50002, 140003])
@pytest.mark.parametrize("at", [0, -1])
def test_a_nan_hides_no_maximum_of_its_own_thread(dev, stream, cols, at):
    """Rows long enough for two passes: the thread that holds the element in front of or behind the groups also holds one
    group of the first few hundred behind the 2016th element; the maximum goes through all of them, for every phase."""
    f = np.float32
    x = np.random.default_rng(cols).standard_normal((64, cols)).astype(f)
    x[:, at] = np.nan
    x[np.arange(64), 2016 + np.arange(64)] = 9.0
    X = dev.from_numpy(x, L.INPUT)
    S, M = dev.empty(64, f, L.OUTPUT), dev.empty(64, f, L.OUTPUT)
    P = dev.empty((64, cols), f, L.OUTPUT)
    ops.row_stats_softmax(stream, X, S, M, P, 64, cols)
    stream.check()
    assert (M.download() == 9.0).all()
    for b in (X, S, M, P):
        b.close()
