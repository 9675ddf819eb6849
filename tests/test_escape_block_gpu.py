"""The block kernel of escape_time (k_escape_block.cu): its tiles' edges and options against the oracle, and on the CPU the
premise of its unchecked blocks (escape_common.cuh, EscapeDev::c2_unsafe_lo)."""
import numpy as np
import pytest

import oracle

F = np.float32


def step(zr, zi, cr, ci, fast):
    """One update in binary32, as the kernels round it (fma: one rounding, through binary64)."""
    d = np.float64
    if fast:
        nzi = (d(zr + zr) * d(zi) + d(ci)).astype(F)
        return (d(zr) * d(zr) + d((-d(zi) * d(zi) + d(cr)).astype(F))).astype(F), nzi
    t = zr * zi
    return (zr * zr - zi * zi) + cr, (2.0 * d(t) + d(ci)).astype(F)


def norm2(zr, zi, fast):
    d = np.float64
    return (d(zi) * d(zi) + d(zr * zr)).astype(F) if fast else zr * zr + zi * zi


def just_outside(radius, angle, fast, limit):
    """Points whose a+b lies within a few roundings above `limit`, at the given angles."""
    zr, zi = (radius * np.cos(angle)).astype(F), (radius * np.sin(angle)).astype(F)
    ok = norm2(zr, zi, fast) > F(limit)
    return zr[ok], zi[ok]


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("limit", [4.0, 4.02, 4.05, 4.2, 6.0, 400.0, 1e6, 1e30])
def test_escape_is_final_outside_the_unsafe_ring(limit, fast):
    rng = np.random.default_rng(11)
    n = 400000
    root = np.sqrt(limit)
    cmax = min(limit - 1.005 * root, 0.5 * limit)
    angle = rng.uniform(0, 2 * np.pi, n)
    angle[: n // 4] = np.pi * rng.integers(0, 4, n // 4) / 2 + rng.normal(0, 1e-4, n // 4)   # the axes, where c cancels most
    zr, zi = just_outside(root * (1 + rng.exponential(1e-6, n)), angle, fast, limit)
    m = zr.size
    # constants up to the largest one, pointing against z^2
    r = cmax * (1 - rng.exponential(1e-4, m).clip(0, 1))
    away = 2 * np.arctan2(zi.astype(np.float64), zr) + np.pi + rng.normal(0, 1e-2, m)
    cr, ci = (r * np.cos(away)).astype(F), (r * np.sin(away)).astype(F)
    with np.errstate(over="ignore", invalid="ignore"):
        for _ in range(6):
            before = norm2(zr, zi, fast)
            zr, zi = step(zr, zi, cr, ci, fast)
            after = norm2(zr, zi, fast)
            assert not (after <= F(limit)).any()
            finite = np.isfinite(after)
            assert (after[finite] > before[finite]).all()
    if cmax * cmax >= 4.05:
        return
    # the other side of the ring, Mandelbrot: the orbit of 0 never shrinks again
    r = np.sqrt(4.05) * (1 + rng.exponential(0.3, n))
    cr, ci = (r * np.cos(angle)).astype(F), (r * np.sin(angle)).astype(F)
    zr, zi = cr.copy(), ci.copy()
    with np.errstate(over="ignore", invalid="ignore"):
        for _ in range(6):
            before = norm2(zr, zi, fast)
            zr, zi = step(zr, zi, cr, ci, fast)
            after = norm2(zr, zi, fast)
            finite = np.isfinite(after)
            assert (after[finite] > before[finite]).all() and not (after[~finite] <= F(limit)).any()


def test_inside_the_ring_the_premise_fails():
    """c = -2, z = 2 + one rounding: z' comes back to the circle, so such constants take tested blocks."""
    c, z = F(-2.0), np.nextafter(F(2.0), F(3))
    assert norm2(z, F(0), False) > 4
    z = F(2.0)
    assert not norm2(z, F(0), False) > 4 and not norm2(z * z + c, F(0), False) > 4


CASES = [(1, 1), (7, 9), (8, 8), (9, 7), (65, 33), (333, 97), (640, 12)]


@pytest.mark.gpu
@pytest.mark.parametrize("max_iter", [1, 3, 4, 5, 50, 127, 128, 131])
@pytest.mark.parametrize("w,h", CASES)
def test_tiles(dev, stream, w, h, max_iter):
    from vernondsl_b200 import _lib as L
    from vernondsl_b200 import ops

    dx, dy = ops.grid_steps(-2.2, 2.2, -1.5, 1.5, w, h)
    img, img16, col = dev.empty((h, w), np.uint32, L.IMAGE), dev.empty((h, w), np.uint16, L.IMAGE), dev.empty((h, w), np.float32, L.IMAGE)
    wire, plane = dev.empty((h, w), np.uint16, L.IMAGE), dev.empty((h, w), np.uint8, L.IMAGE)
    for kind, okind in ((L.JULIA, oracle.JULIA), (L.MANDELBROT, oracle.MANDELBROT)):
        for mode in (L.EXACT, L.FAST):
            def p(**kw):
                return ops.escape_params(kind, w, h, -2.2, -1.5, dx, dy, cr=-0.8, ci=0.156, max_iter=max_iter, mode=mode, **kw)
            ops.escape_time(stream, img, p(checked_only=True))
            stream.check()
            want = img.download()
            if mode == L.EXACT:
                assert np.array_equal(want, oracle.escape_time(okind, w, h, -2.2, -1.5, dx, dy, -0.8, 0.156, max_iter)[0])
            for b in (img, img16, col, wire, plane):
                b.fill(0xEE)
            ops.escape_time(stream, img, p(), wire, plane)
            ops.escape_time(stream, img16, p(output=L.OUT_COUNT_U16))
            ops.escape_time(stream, col, p(output=L.OUT_COLOR_F32, color_scale=1.0 / 64))
            stream.check()
            assert np.array_equal(img.download(), want) and np.array_equal(wire.download(), want) and np.array_equal(img16.download(), want)
            assert np.array_equal(plane.download(), np.minimum(want, 255))
            assert np.array_equal(col.download(), F(1) - want.astype(F) * F(1.0 / 64))


@pytest.mark.gpu
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("chunk", [None, (3, 0, 2), (3, 1, 2), (8, 1, 3)])
def test_partitions_and_orders(dev, stream, transposed, chunk):
    from vernondsl_b200 import _lib as L
    from vernondsl_b200 import ops

    w, h = 77, 50
    img = dev.empty((h, w), np.uint32, L.IMAGE)
    part, rows = None, np.ones(h, bool)
    if chunk:
        part = L.RowPartition()
        part.chunk_rows, part.chunk_first, part.chunk_step = chunk
        chunks = range(chunk[1], (h + chunk[0] - 1) // chunk[0], chunk[2])
        part.chunk_count = len(chunks)
        rows[:] = False
        for c in chunks:
            rows[c * chunk[0]:(c + 1) * chunk[0]] = True
    for kind in (L.JULIA, L.MANDELBROT):
        def p(**kw):
            return ops.escape_params(kind, w, h, -2.0, -1.0, F(4 / w), F(2 / h), cr=-0.8, ci=0.156, max_iter=50, partition=part, transposed=transposed, **kw)
        got = []
        for checked in (True, False):
            img.fill(0xEE)
            ops.escape_time(stream, img, p(checked_only=checked))
            stream.check()
            got.append(img.download())
        assert np.array_equal(*got)
        assert (got[1][~rows] == 0xEEEEEEEE).all() and (got[1][rows] <= 50).all()


@pytest.mark.gpu
@pytest.mark.parametrize("max_iter,w,h", [(100, 4000, 9), (300, 4000, 9), (300, 4000, 201)])
def test_the_needle_and_the_ring_around_two(dev, stream, max_iter, w, h):
    """A view of the real axis from -2.05 to -1.9: constants on both sides of the ring and in it, to max_iter on the axis itself
    (block kernel below 512 Ki pixels, regrouping kernel above)."""
    from vernondsl_b200 import _lib as L
    from vernondsl_b200 import ops

    img = dev.empty((h, w), np.uint32, L.IMAGE)
    dx, dy = F(0.15 / w), F(2.0 ** -12)
    y0 = F(-(h // 2) * 2.0 ** -12)
    for bound in (4.0, 4.02, 4.1):
        ops.escape_time(stream, img, ops.escape_params(L.MANDELBROT, w, h, -2.05, y0, dx, dy, max_iter=max_iter, bound=bound))
        stream.check()
        want, _ = oracle.escape_time(oracle.MANDELBROT, w, h, -2.05, y0, dx, dy, 0.0, 0.0, max_iter, bound=bound)
        assert (want[h // 2] == max_iter).sum() > 100
        assert np.array_equal(img.download(), want)
    for cr, ci in ((-1.97, 0.0), (-1.9899, 0.0), (-1.995, 0.0), (0.3, 1.95), (-2.0, 0.0)):
        ops.escape_time(stream, img, ops.escape_params(L.JULIA, w, h, -2.05, y0, dx, dy, cr=cr, ci=ci, max_iter=max_iter))
        stream.check()
        want, _ = oracle.escape_time(oracle.JULIA, w, h, -2.05, y0, dx, dy, cr, ci, max_iter)
        assert np.array_equal(img.download(), want), (cr, ci)
