"""GPU: the vertex stage at the edges of its tiles of 1024 vertices, against binary64."""
import numpy as np
import pytest

from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 85, 86, 255, 256, 257, 341, 1023, 1024, 1025, 1026, 1027, 5000, 700001])
def test_vertices_at_the_edges_of_a_tile(dev, stream, n):
    rng = np.random.default_rng(n)
    pos = rng.standard_normal((n, 3)).astype(np.float32)
    mats = [rng.standard_normal((4, 4)).astype(np.float32) for _ in range(3)]
    P = dev.from_numpy(pos)
    M = [dev.from_numpy(m, L.UNIFORM) for m in mats]
    guard = 32
    out = dev.from_numpy(np.full(4 * n + guard, 7.0, np.float32), L.OUTPUT)
    var = dev.from_numpy(np.full(3 * n + guard, 7.0, np.float32), L.VARYING)
    ops.vertex_transform(stream, P, *M, out, var, n)
    stream.check()
    v = np.concatenate([pos, np.ones((n, 1), np.float32)], 1).astype(np.float64)
    size = np.abs(v)
    for m in mats:
        v, size = v @ m.T.astype(np.float64), size @ np.abs(m.T)
    got = out.download()
    # four roundings per product, three products: 12 * 2^-24 of the sum of magnitudes, to first order
    assert (np.abs(got[:4 * n].reshape(n, 4) - v) <= 13 * 2.0 ** -24 * size).all()
    assert (got[4 * n:] == 7.0).all()
    got = var.download()
    assert np.array_equal(got[:3 * n].reshape(n, 3), pos) and (got[3 * n:] == 7.0).all()
    for buf in [P, out, var] + M:
        buf.close()
