"""CPU: a kernel's kept plan gives the parameter block a fresh walk would, and gives way when anything it rests on changes."""
import ctypes as C
import sys

import numpy as np
import pytest

import vernondsl_b200.lang as ti

SCALE = 0.2
LIMIT = 50
BIAS = np.float32(0.25)


def fields(half):
    with ti.plan_only():
        return ti.field(dtype=float, shape=(2 * half, half))


@ti.func
def csq(w):
    return ti.Vector([w[0] ** 2 - w[1] ** 2, w[1] * w[0] * 2])


def painter(half):
    canvas = fields(half)
    radius = 20

    @ti.kernel
    def draw(phase: float):
        for a, b in canvas:
            k = ti.Vector([-0.8, ti.cos(phase) * SCALE + BIAS])
            w = ti.Vector([a / half - 1, b / half - 0.5]) * 2
            steps = 0
            while w.norm() < radius and steps < LIMIT:
                w = csq(w) + k
                steps += 1
            canvas[a, b] = 1 - steps * 0.02

    def change(**kw):
        nonlocal canvas, half, radius
        canvas, half, radius = kw.get("canvas", canvas), kw.get("half", half), kw.get("radius", radius)

    return draw, change


def lowered(kernel, *args):
    with ti.plan_only():
        kernel(*args)
    return bytes(C.string_at(C.byref(kernel.last_params), C.sizeof(kernel.last_params))), kernel.last_plan


def fresh(kernel, *args):
    """The same call through a walk with nothing kept."""
    again = ti.Kernel(kernel.fn)
    again._plannable = False
    return lowered(again, *args)


def test_other_arguments_give_the_walks_parameters():
    draw, _ = painter(64)
    lowered(draw, 0.1)
    plan = draw._plan
    assert plan is not None
    for x in (0.0, -0.0, 1, 7, 0.3, 1e9, -3.7, np.float32(0.77), np.float64(0.77), 1e-40):
        assert lowered(draw, x) == fresh(draw, x), x
        assert draw._plan is plan
    for bad in (float("nan"), float("inf")):
        with pytest.raises(Exception) as one, np.errstate(invalid="ignore"):
            lowered(draw, bad)
        with pytest.raises(Exception) as two, np.errstate(invalid="ignore"):
            fresh(draw, bad)
        assert type(one.value) is type(two.value)
    with pytest.raises(TypeError):
        lowered(draw)


def test_what_the_walk_read_is_compared_on_every_call(monkeypatch):
    draw, change = painter(64)
    module = sys.modules[__name__]
    lowered(draw, 0.1)
    steps = [lambda: monkeypatch.setattr(module, "SCALE", 0.3), lambda: monkeypatch.setattr(module, "LIMIT", 77),
             lambda: monkeypatch.setattr(module, "BIAS", np.float32(0.5)), lambda: change(half=32), lambda: change(radius=3.0),
             lambda: change(canvas=fields(48)), lambda: monkeypatch.setattr(ti, "cos", ti.sin)]
    before = lowered(draw, 0.4)
    for k, step in enumerate(steps):
        step()
        after = lowered(draw, 0.4)
        assert after == fresh(draw, 0.4), k
        assert after != before, k
        before = after


def test_a_field_of_another_shape_under_the_same_object():
    draw, change = painter(64)
    canvas = fields(40)
    change(canvas=canvas)
    lowered(draw, 0.2)
    canvas.shape = (30, 20)
    assert lowered(draw, 0.2) == fresh(draw, 0.2)
    assert "20x30" in draw.last_plan


def test_arguments_that_reach_more_than_the_constant_are_walked_every_time():
    canvas = fields(32)

    @ti.kernel
    def zoomed(zoom: float):
        for a, b in canvas:
            k = ti.Vector([-0.8, 0.156])
            w = ti.Vector([a / 32 - 1, b / 32 - 0.5]) * zoom
            steps = 0
            while w.norm() < 20 and steps < 50:
                w = csq(w) + k
                steps += 1
            canvas[a, b] = 1 - steps * 0.02

    @ti.kernel
    def deeper(n: int):
        for a, b in canvas:
            k = ti.Vector([-0.8, 0.156])
            w = ti.Vector([a / 32 - 1, b / 32 - 0.5])
            steps = 0
            while w.norm() < 20 and steps < n:
                w = csq(w) + k
                steps += 1
            canvas[a, b] = 1 - steps * 0.02

    for kernel, args in ((zoomed, (2.0, 3.0, 0.5)), (deeper, (50, 60, 70))):
        seen = {lowered(kernel, x) for x in args}
        assert len(seen) == 3 and kernel._plan is None
        for x in args:
            assert lowered(kernel, x) == fresh(kernel, x)


def test_an_error_in_the_body_is_still_the_walks_error():
    canvas = fields(32)

    @ti.kernel
    def wrong(x: float):
        for a, b in canvas:
            k = ti.Vector([x, missing])  # noqa: F821
            w = ti.Vector([a / 32 - 1, b / 32 - 0.5])
            steps = 0
            while w.norm() < 20 and steps < 50:
                w = csq(w) + k
                steps += 1
            canvas[a, b] = 1 - steps * 0.02

    for _ in range(2):
        with pytest.raises(ti.LangError, match="missing"):
            lowered(wrong, 0.5)
