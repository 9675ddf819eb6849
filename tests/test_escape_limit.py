"""The test `sqrt(a+b) < bound` runs as `a+b <= limit` (k_escape.cu, escape_limit): same counts for every bound."""
import math

import numpy as np
import pytest

import oracle

BOUNDS = [20.0, 2.0, 1.9999999, 3.3, 4.0, 1e-3, 1e-30, 1e30, 3e38, float("inf"), 0.0, -1.0, float("nan"), 0.7071068, 1.8446743e19]


def limit_of(bound):
    """escape_limit restated in binary32 numpy."""
    f = np.float32
    b = f(bound)
    if not b > 0:
        return f(-1.0)
    top = np.finfo(f).max
    with np.errstate(over="ignore", under="ignore"):
        s = b * b
    s = s if s <= top else top
    while s > 0 and not np.sqrt(s) < b:
        s = np.nextafter(s, f(0))
    while s < top and np.sqrt(np.nextafter(s, f(np.inf))) < b:
        s = np.nextafter(s, f(np.inf))
    return s


@pytest.mark.parametrize("bound", BOUNDS + list(np.random.default_rng(3).uniform(0.1, 1e4, 50).astype(np.float32)))
def test_the_limit_separates_the_same_sums(bound):
    f = np.float32
    lim = limit_of(bound)
    near = [f(0), f(1e-45), f(lim) if lim >= 0 else f(0), f(np.inf), f(np.nan), np.finfo(f).max]
    for _ in range(3):
        near += [np.nextafter(near[2], f(np.inf)), np.nextafter(near[2], f(0))]
        near[2] = np.nextafter(near[2], f(np.inf))
    for s in near + list(np.random.default_rng(1).uniform(0, 2, 100).astype(f) * np.maximum(lim, f(1))):
        if math.isinf(s) or math.isnan(s):
            assert not s <= lim
        with np.errstate(invalid="ignore", over="ignore"):
            assert bool(np.sqrt(s) < f(bound)) == bool(s <= lim), (bound, s)


@pytest.mark.gpu
@pytest.mark.parametrize("bound", BOUNDS)
@pytest.mark.parametrize("max_iter", [50, 100])
def test_counts_equal_the_oracle(dev, stream, bound, max_iter):
    from vernondsl_b200 import _lib as L
    from vernondsl_b200 import ops

    w, h = 333, 97
    dx, dy = ops.grid_steps(-2.0, 2.0, -1.0, 1.0, w, h)
    img = dev.empty((h, w), np.uint32, L.IMAGE)
    for kind, okind in ((L.JULIA, oracle.JULIA), (L.MANDELBROT, oracle.MANDELBROT)):
        p = ops.escape_params(kind, w, h, -2.0, -1.0, dx, dy, cr=-0.8, ci=0.156, max_iter=max_iter, test=L.TEST_NORM_GE, bound=bound)
        for _ in range(2):          # the work counter is back at 0 for the second launch
            img.fill(0xFF)
            ops.escape_time(stream, img, p)
            stream.check()
            want, _ = oracle.escape_time(okind, w, h, -2.0, -1.0, dx, dy, -0.8, 0.156, max_iter, test=oracle.TEST_NORM_GE, bound=bound)
            assert np.array_equal(img.download(), want), (kind, bound)
