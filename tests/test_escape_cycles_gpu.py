"""GPU: pixels of the regrouping kernel whose orbit repeats a state end there with max_iter (k_escape_pair.cu); the counts are
those of running every step."""
import numpy as np
import pytest

import oracle
from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops

VIEWS = [(-2.5, 1.0, -1.0, 1.0),          # the whole set
         (-0.1, 0.45, -0.3, 0.3),         # inside and around the cusp of the cardioid, where orbits converge slowly
         (-1.3, -0.7, -0.3, 0.3),         # the disc of period 2 and its neighbours
         (-0.2, -0.05, 0.65, 0.8)]        # a bulb of period 3 and the antenna of its branches


@pytest.mark.gpu
@pytest.mark.parametrize("max_iter", [200, 1000, 3001])
@pytest.mark.parametrize("view", VIEWS)
def test_counts_of_converging_orbits(dev, stream, view, max_iter):
    w, h = 1021, 517                      # above 512 Ki pixels: the regrouping kernel
    x0, x1, y0, y1 = view
    dx, dy = ops.grid_steps(x0, x1, y0, y1, w, h)
    img = dev.empty((h, w), np.uint32, L.IMAGE)
    for bound, test, otest in ((4.0, L.TEST_NORM2_GT, oracle.TEST_NORM2_GT), (20.0, L.TEST_NORM_GE, oracle.TEST_NORM_GE)):
        p = ops.escape_params(L.MANDELBROT, w, h, x0, y0, dx, dy, max_iter=max_iter, test=test, bound=bound)
        ops.escape_time(stream, img, p)
        stream.check()
        want, _ = oracle.escape_time(oracle.MANDELBROT, w, h, x0, y0, dx, dy, max_iter=max_iter, test=otest, bound=bound)
        assert (want == max_iter).any()
        assert np.array_equal(img.download(), want)
    p = ops.escape_params(L.MANDELBROT, w, h, x0, y0, dx, dy, max_iter=max_iter, mode=L.FAST)
    ops.escape_time(stream, img, p)
    stream.check()
    want, _ = oracle.escape_time(oracle.MANDELBROT, w, h, x0, y0, dx, dy, max_iter=max_iter, fast=True)
    assert np.array_equal(img.download(), want)
