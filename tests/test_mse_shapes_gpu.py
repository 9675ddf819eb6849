"""GPU: the fused loss and its gradients at the edges of its tiles (row lengths with and without float4 groups), against binary64."""
import numpy as np
import pytest

from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops

SHAPES = [(1, 1), (3, 1), (1, 5), (700, 3), (5, 4), (3000, 4), (513, 7), (257, 127), (64, 128), (300, 129), (33, 255), (17, 1001), (2049, 1001), (9, 1024),
          (7, 1028), (5, 4099), (3, 20001)]


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", SHAPES)
def test_loss_and_gradients(dev, stream, rows, cols):
    rng = np.random.default_rng(rows * 7 + cols)
    W, x, t = (rng.standard_normal((rows, cols)).astype(np.float32) for _ in range(3))
    b = rng.standard_normal(cols).astype(np.float32)
    ins = [dev.from_numpy(v, L.INPUT) for v in (W, x, b, t)]
    guard = 32
    DW, DX, DB, LO, LF = (dev.from_numpy(np.full(k + guard, 7.0, np.float32), L.OUTPUT) for k in (rows * cols, rows * cols, cols, 1, 1))
    ops.mse_tanh_bwd(stream, *ins, DW, DX, DB, rows, cols, loss=LO)
    ops.mse_tanh_fwd(stream, *ins, LF, rows, cols)
    stream.check()
    W, x, b, t = (v.astype(np.float64) for v in (W, x, b, t))
    u = W * x + b
    y, sech2 = np.tanh(u), 1 / np.cosh(u) ** 2
    g = 2.0 / (rows * cols) * (y - t) * sech2
    # u carries one rounding, 2^-24 |u|, which moves 1 - tanh^2 by twice that of itself; exponential (two units in the last
    # place), reciprocal, products and sums: under 1.5e-6.  tanh = (1-E)/(1+E) has an absolute error where E is near 1:
    # half of E's 2.4e-7, and three roundings of numbers below 1
    rel = 2.0 ** -23 * np.abs(u) + 1.5e-6
    size = 2.0 / (rows * cols) * (rel * np.abs(y - t) + 3.5e-7) * sech2
    for got, want, scale in ((DW, g * x, size * np.abs(x)), (DX, g * W, size * np.abs(W)), (DB, g.sum(0), size.sum(0))):
        got = got.download()
        n = want.size
        assert (np.abs(got[:n].reshape(want.shape) - want) <= scale + 1e-37).all()
        assert (got[n:] == 7.0).all()
    for lo in (LO, LF):
        lo = lo.download()
        assert lo[0] == pytest.approx(float(((y - t) ** 2).mean()), rel=4e-6)
        assert (lo[1:] == 7.0).all()
    for buf in ins + [DW, DX, DB, LO, LF]:
        buf.close()
