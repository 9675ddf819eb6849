"""GPU: escape_time around the lines at which the regrouping kernel takes over from the block kernel (launch_escape_time),
against the step-by-step kernel: the same counts on both sides of every line, for both sets."""
import numpy as np
import pytest

from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops

pytestmark = pytest.mark.gpu

SIZES = [(150, 160), (200, 160), (300, 300), (301, 300), (384, 383), (384, 385), (424, 424), (425, 425), (496, 495), (496, 496), (543, 543), (544, 543), (677, 677),
         (678, 678), (1024, 511), (1024, 512)]
STEPS = [191, 192, 255, 256, 511, 512, 1023, 1024, 1100]


@pytest.mark.parametrize("kind", [L.JULIA, L.MANDELBROT])
@pytest.mark.parametrize("w,h", SIZES)
def test_both_sides_of_every_line(dev, stream, w, h, kind):
    dx, dy = ops.grid_steps(-2.0, 1.2, -1.2, 1.2, w, h)
    img, ref = (dev.empty((h, w), np.uint32, L.IMAGE) for _ in range(2))
    for max_iter in STEPS:
        def p(**kw):
            return ops.escape_params(kind, w, h, -2.0, -1.2, dx, dy, cr=-0.123, ci=0.745, max_iter=max_iter, **kw)
        img.fill(0xEE)
        ops.escape_time(stream, img, p())
        ops.escape_time(stream, ref, p(checked_only=True))
        stream.check()
        assert np.array_equal(img.download(), ref.download()), max_iter
    for b in (img, ref):
        b.close()


@pytest.mark.parametrize("max_iter", [600, 1200])
def test_recorded_without_scratch(dev, max_iter):
    """The regrouping kernel's work counter lives in the stream's scratch; a launch recorded on a stream that has none is
    recorded with the block kernel."""
    w, h = 700, 600
    st = dev.stream()
    dx, dy = ops.grid_steps(-2.0, 1.2, -1.2, 1.2, w, h)
    img, ref = (dev.empty((h, w), np.uint32, L.IMAGE) for _ in range(2))
    for kind in (L.JULIA, L.MANDELBROT):
        p = ops.escape_params(kind, w, h, -2.0, -1.2, dx, dy, cr=-0.123, ci=0.745, max_iter=max_iter)
        fresh = dev.stream()
        img.fill(0xEE)
        with fresh.record() as seq:
            ops.escape_time(fresh, img, p)
        assert seq.stats()["kernels"] == 1
        seq.launch()
        fresh.check()
        ops.escape_time(st, ref, p)
        st.check()
        assert np.array_equal(img.download(), ref.download())
        seq.close()
        fresh.close()
    st.close()
