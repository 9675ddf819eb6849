"""The work this package is timed on: what its users have it do, through its public entry points.

Each case is a dict of plain values; ``prepare`` makes what a user's program holds before the call
(arrays on the GPU, a compiled graph, a recorded frame loop), ``run`` is one pass, ``work`` says
what a pass cannot do without and ``tolerance`` how far a correct result may be off.

Operations (``op``) and the real use each stands for:

  escape   an escape-time image (Mandelbrot or Julia) into uint32 / uint16 counts or a float colour
  paint    one call of a Taichi-style kernel per frame: the reference's own program, fractal.py
  frames   the same program's frame loop, recorded once and replayed into a ring of frames
  map      the fused map chain  tanh(a*x + y) * exp(-x*x/2) + sqrt(|y| + 1e-3)
  tape     a user's own fused elementwise expression with per-column parameters
  softmax  row softmax, alone or with the row sums and maxima of the same matrix
  reduce   row sums, row maxima and column sums of one matrix
  mse      loss = mean((tanh(W*x + b) - t)^2): forward, or its gradients together with the loss
  graph    a loss stated in the execution graph, differentiated and fused by it (no hand-written kernel)
  vertex   the vertex stage of color.mlir over an array of vertices
"""
from __future__ import annotations

import math

import numpy as np
import torch

import vernondsl_b200 as vd
import vernondsl_b200.lang as ti
from vernondsl_b200 import _lib as L
from vernondsl_b200 import ops
from vernondsl_b200.graph import Graph


def listed():
    return [
        # the largest image: the whole plane of one Julia set, deep iteration (the benchmark's headline)
        {"name": "julia-16384", "op": "escape", "set": "julia", "width": 16384, "height": 16384, "max_iter": 4096, "out": "u32",
         "mode": "exact", "test": "norm2"},
        # one frame of an interactive Mandelbrot viewer at display size
        {"name": "mandelbrot-1080p", "op": "escape", "set": "mandelbrot", "width": 1920, "height": 1080, "max_iter": 256, "out": "u32",
         "mode": "exact", "test": "norm2"},
        # the reference's own program, one kernel call per frame: the smallest call, latency and host work count
        {"name": "paint-640x320", "op": "paint", "half": 320},
        # the reference's frame loop without its window: 64 frames in one submission
        {"name": "frames-640x320x64", "op": "frames", "half": 320, "frames": 64},
        # a bandwidth-bound map over arrays far larger than any cache
        {"name": "map-2^28", "op": "map", "n": 1 << 28},
        # a user's expression over an image-sized array whose row length is odd (a cropped frame)
        {"name": "tape-1081x1919", "op": "tape", "rows": 1081, "cols": 1919},
        # softmax with row statistics of a large matrix, power-of-two rows
        {"name": "softmax-65536x4096", "op": "softmax", "rows": 65536, "cols": 4096, "stats": True},
        # softmax over long rows of an odd length (a vocabulary or class count that nobody rounded up)
        {"name": "softmax-4099x10007", "op": "softmax", "rows": 4099, "cols": 10007, "stats": False},
        # an ordinary, small table: sums and maxima of its rows, sums of its columns
        {"name": "reduce-1000x1001", "op": "reduce", "rows": 1000, "cols": 1001},
        # a large training step: gradients of W, x and b, and the loss
        {"name": "mse-grad-32768x4096", "op": "mse", "rows": 32768, "cols": 4096, "grad": True},
        # a loss with no hand-written kernel, differentiated by the graph; neither dimension is round
        {"name": "graph-grad-2049x1001", "op": "graph", "rows": 2049, "cols": 1001},
        # the vertex stage over a mesh
        {"name": "vertex-1000003", "op": "vertex", "n": 1000003},
    ]


def _log(rng, lo, hi):
    """An integer spread evenly over the logarithm of lo..hi; every other one is a multiple of 4 (where that fits)."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5 and v >= 8:
        v = v // 4 * 4
    return max(lo, min(hi, v))


def _matrix(rng, rows, cols, most):
    """rows x cols from the two ranges, at most `most` elements."""
    while True:
        r, c = _log(rng, *rows), _log(rng, *cols)
        if r * c <= most:
            return r, c


def draw(rng):
    op = rng.choice(["escape", "escape", "paint", "frames", "map", "tape", "softmax", "reduce", "mse", "graph", "vertex"])
    if op == "escape":
        while True:
            w, h, n = _log(rng, 256, 8192), _log(rng, 256, 8192), _log(rng, 32, 4096)
            if w * h * n <= 1 << 33:      # a third of a Mandelbrot view can run all max_iter steps
                break
        out = rng.choice(["u32", "u32", "u16", "color"])
        return {"op": op, "set": rng.choice(["julia", "mandelbrot"]), "width": w, "height": h, "max_iter": n, "out": out,
                "mode": rng.choice(["exact", "exact", "exact", "fast"]), "test": rng.choice(["norm2", "norm2", "norm"])}
    if op == "paint":
        return {"op": op, "half": _log(rng, 64, 1024)}
    if op == "frames":
        return {"op": op, "half": _log(rng, 64, 640), "frames": rng.randrange(8, 129)}
    if op in ("map", "vertex"):
        return {"op": op, "n": _log(rng, 1000, 1 << 27 if op == "map" else 1 << 24)}
    if op == "tape":
        r, c = _matrix(rng, (1, 8192), (3, 1 << 20), 1 << 25)
    elif op == "softmax":
        r, c = _matrix(rng, (16, 65536), (8, 65536), 1 << 27)
        return {"op": op, "rows": r, "cols": c, "stats": rng.random() < 0.5}
    elif op == "reduce":
        r, c = _matrix(rng, (16, 1 << 20), (4, 65536), 1 << 26)
    elif op == "mse":
        r, c = _matrix(rng, (16, 65536), (4, 16384), 1 << 26)
        return {"op": op, "rows": r, "cols": c, "grad": rng.random() < 0.7}
    else:
        r, c = _matrix(rng, (16, 65536), (4, 16384), 1 << 24)
    return {"op": op, "rows": r, "cols": c}


# ------------------------------------------------------------------------------ what a program holds
class _Program:
    """One device and one stream for the whole process, as a program keeps them."""
    dev = None
    stream = None

    @classmethod
    def get(cls):
        if cls.dev is None:
            cls.dev = vd.Device(0)
            cls.stream = cls.dev.stream()
        return cls.dev, cls.stream


class State:
    """What a pass needs: a function and its outputs.  `owned` (a graph, handles on torch's tensors) is closed when the
    state goes; the outputs are torch tensors, or fields, which live as long as the process."""

    def __init__(self, call, outputs, owned):
        self.call, self.outputs, self.owned = call, outputs, owned

    def __del__(self):
        try:
            torch.cuda.synchronize()
            for o in self.owned:
                o.close()
        except Exception:      # the interpreter or the device is already going down
            pass


def _escape_view(case, r):
    """A view of the set, panned by the seed.  x0, x1, y0, y1, cr, ci."""
    px, py = 0.01 * r.uniform(-1, 1), 0.01 * r.uniform(-1, 1)
    if case["set"] == "julia":
        return -1.6 + px, 1.6 + px, -1.6 + py, 1.6 + py, -0.8, 0.156
    return -2.5 + px, 1.0 + px, -1.0 + py, 1.0 + py, 0.0, 0.0


def _painter(half):
    """fractal.py:8-25: a field of (2n, n) pixels and the kernel that fills it for one phase."""
    canvas = ti.field(dtype=float, shape=(2 * half, half))

    @ti.func
    def csq(w):
        return ti.Vector([w[0] ** 2 - w[1] ** 2, w[1] * w[0] * 2])

    @ti.kernel
    def draw_frame(phase: float):
        for a, b in canvas:
            k = ti.Vector([-0.8, ti.cos(phase) * 0.2])
            w = ti.Vector([a / half - 1, b / half - 0.5]) * 2
            steps = 0
            while w.norm() < 20 and steps < 50:
                w = csq(w) + k
                steps += 1
            canvas[a, b] = 1 - steps * 0.02

    return canvas, draw_frame


def prepare(case, seed):
    dev, st = _Program.get()
    op = case["op"]
    r = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda:0")
    gen.manual_seed(int(r.integers(1 << 62)))
    owned = []

    def randn(*shape, scale=1.0):
        return torch.randn(shape, generator=gen, device="cuda:0").mul_(scale)

    def empty(*shape, dtype=torch.float32):
        return torch.empty(shape, device="cuda:0", dtype=dtype)

    def buf(t, cls):
        b = dev.wrap_tensor(t, cls)
        owned.append(b)
        return b

    def ins(*ts):
        return [buf(t, L.INPUT) for t in ts]

    def outs(*ts):
        return [buf(t, L.OUTPUT) for t in ts]

    if op == "escape":
        w, h = case["width"], case["height"]
        x0, x1, y0, y1, cr, ci = _escape_view(case, r)
        dx, dy = ops.grid_steps(x0, x1, y0, y1, w, h)
        out, dtype = {"u32": (L.OUT_COUNT_U32, torch.int32), "u16": (L.OUT_COUNT_U16, torch.int16),
                      "color": (L.OUT_COLOR_F32, torch.float32)}[case["out"]]
        p = ops.escape_params(L.JULIA if case["set"] == "julia" else L.MANDELBROT, w, h, x0, y0, dx, dy, cr=cr, ci=ci,
                              max_iter=case["max_iter"], mode=L.EXACT if case["mode"] == "exact" else L.FAST,
                              test=L.TEST_NORM2_GT if case["test"] == "norm2" else L.TEST_NORM_GE,
                              bound=4.0 if case["test"] == "norm2" else 20.0, output=out, color_scale=1.0 / case["max_iter"])
        image_t = empty(h, w, dtype=dtype)
        image = buf(image_t, L.IMAGE)
        return State(lambda: ops.escape_time(st, image, p), image_t, owned)
    if op == "paint":
        canvas, draw_frame = _painter(case["half"])
        phase = float(r.uniform(0.0, 6.0))
        return State(lambda: draw_frame(phase), canvas.buffer.as_tensor(), [])
    if op == "frames":
        canvas, draw_frame = _painter(case["half"])
        loop = ti.FrameLoop(draw_frame, canvas, ring=4)
        start = float(r.uniform(0.0, 6.0))
        loop.record([start + 0.03 * k for k in range(case["frames"])])
        ring = [b.as_tensor(np.float32, canvas.shape) for b in loop.ring]
        return State(loop.play, ring, [])
    if op == "map":
        n = case["n"]
        a = torch.rand(n, generator=gen, device="cuda:0").mul_(2).sub_(1)
        out_t = empty(n)
        A, X, Y = ins(a, randn(n), randn(n))
        O, = outs(out_t)
        return State(lambda: ops.fused_map(st, A, X, Y, O, n), out_t, owned)
    if op == "tape":
        # a gated, normalised image: out = sigmoid(x*scale + shift) * y + |x|, scale and shift per column
        rows, cols = case["rows"], case["cols"]
        t = ops.Tape(4, row_vectors=[2, 3])
        x, y, scale, shift = (t.input(k) for k in range(4))
        t.output(t.op("fma", t.op("sigmoid", t.op("fma", x, scale, shift)), y, t.op("abs", x)))
        out_t = empty(rows, cols)
        inputs = ins(randn(rows, cols), randn(rows, cols), randn(cols), randn(cols))
        outputs = outs(out_t)
        return State(lambda: ops.map_tape(st, t, inputs, outputs, rows, cols), out_t, owned)
    rows, cols = case.get("rows", 0), case.get("cols", 0)
    if op == "softmax":
        M, = ins(randn(rows, cols, scale=2.0))
        soft = empty(rows, cols)
        if case["stats"]:
            s, m = empty(rows), empty(rows)
            S, X, F = outs(s, m, soft)
            return State(lambda: ops.row_stats_softmax(st, M, S, X, F, rows, cols), [s, m, soft], owned)
        F, = outs(soft)
        return State(lambda: ops.row_softmax(st, M, F, rows, cols), soft, owned)
    if op == "reduce":
        M, = ins(randn(rows, cols).add_(1.0))
        s, m, c = empty(rows), empty(rows), empty(cols)
        S, X, C = outs(s, m, c)

        def call():
            ops.row_sum(st, M, S, rows, cols)
            ops.row_max(st, M, X, rows, cols)
            ops.col_sum(st, M, C, rows, cols)

        return State(call, [s, m, c], owned)
    if op == "mse":
        W, X, B, T = ins(randn(rows, cols), randn(rows, cols), randn(cols), randn(rows, cols))
        loss = empty(4)[:1].contiguous()
        if not case["grad"]:
            LO, = outs(loss)
            return State(lambda: ops.mse_tanh_fwd(st, W, X, B, T, LO, rows, cols), loss, owned)
        dw, dx, db = empty(rows, cols), empty(rows, cols), empty(cols)
        DW, DX, DB, LO = outs(dw, dx, db, loss)
        return State(lambda: ops.mse_tanh_bwd(st, W, X, B, T, DW, DX, DB, rows, cols, loss=LO), [dw, dx, db, loss], owned)
    if op == "graph":
        # loss = mean((sigmoid(W*x + b) - t)^2): dW, dx, db and the loss
        W, X, B, T = ins(randn(rows, cols), randn(rows, cols), randn(cols), torch.rand((rows, cols), generator=gen, device="cuda:0"))
        dw, dx, db, loss = empty(rows, cols), empty(rows, cols), empty(cols), empty(1)
        g = Graph(dev, rows, cols)
        w, x, t, b = g.input(W), g.input(X), g.input(T), g.input(B, L.SHAPE_ROWVEC)
        value = g.mean(g.square(g.unary("sigmoid", w * x + b) - t))
        grads = g.grad(value, [w, x, b])
        for node, o in zip(grads + [value], outs(dw, dx, db, loss)):
            g.output(node, o)
        g.compile()
        return State(lambda: g.launch(st), [dw, dx, db, loss], [g] + owned)
    if op == "vertex":
        n = case["n"]
        pos, out_pos, varying = randn(n, 3), empty(n, 4), empty(n, 3)
        P, = ins(pos)
        mats = [buf(randn(4, 4), L.UNIFORM) for _ in range(3)]
        G, = outs(out_pos)
        V = buf(varying, L.VARYING)
        return State(lambda: ops.vertex_transform(st, P, *mats, G, V, n), [out_pos, varying], owned)
    raise ValueError(op)


def run(state):
    state.call()
    return state.outputs


# ------------------------------------------------------------------------------ what a pass needs
def _mean_count(case):
    """Mean iteration count of the case's view, from a 160 x 160 sample of it (numpy, binary32)."""
    n = 160
    julia = case["op"] != "escape" or case["set"] == "julia"
    if case["op"] == "escape":
        x0, x1, y0, y1, cr, ci = _escape_view(case, np.random.default_rng(0))
        max_iter, limit = case["max_iter"], np.float32(4.0 if case["test"] == "norm2" else 400.0)
    else:
        x0, x1, y0, y1, cr, ci, max_iter, limit = -2.0, 2.0, -1.0, 1.0, -0.8, 0.1, 50, np.float32(400.0)
    re = (x0 + (np.arange(n) + 0.5) * (x1 - x0) / n).astype(np.float32)[None, :].repeat(n, 0).ravel()
    im = (y0 + (np.arange(n) + 0.5) * (y1 - y0) / n).astype(np.float32)[:, None].repeat(n, 1).ravel()
    zr, zi = (re, im) if julia else (np.zeros_like(re), np.zeros_like(im))
    kr, ki = (np.float32(cr), np.float32(ci)) if julia else (re, im)
    total = 0
    for _ in range(max_iter):
        live = zr * zr + zi * zi <= limit
        zr, zi = zr[live], zi[live]
        if not julia:
            kr, ki = kr[live], ki[live]
        if zr.size == 0:
            break
        zr, zi = zr * zr - zi * zi + kr, 2 * zr * zi + ki
        total += zr.size
    return total / (n * n)


def work(case):
    op = case["op"]
    if op == "escape":
        px = case["width"] * case["height"]
        return {"bytes": px * (2 if case["out"] == "u16" else 4), "flops": 8 * px * _mean_count(case)}
    if op in ("paint", "frames"):
        px = 2 * case["half"] ** 2 * case.get("frames", 1)
        return {"bytes": 4 * px, "flops": 8 * px * _mean_count(case)}
    if op == "map":
        return {"bytes": 16 * case["n"], "flops": 12 * case["n"]}
    if op == "vertex":
        return {"bytes": 40 * case["n"] + 192, "flops": 84 * case["n"]}
    r, c = case["rows"], case["cols"]
    n = r * c
    if op == "tape":
        return {"bytes": 12 * n + 8 * c, "flops": 8 * n}
    if op == "softmax":
        return {"bytes": 8 * n + (8 * r if case["stats"] else 0), "flops": (6 if case["stats"] else 5) * n}
    if op == "reduce":
        return {"bytes": 4 * n + 8 * r + 4 * c, "flops": 3 * n}
    if op == "mse" and not case["grad"]:
        return {"bytes": 12 * n + 4 * c + 4, "flops": 8 * n}
    return {"bytes": 20 * n + 8 * c + 4, "flops": 14 * n}      # mse with gradients, graph


def tolerance(case):
    """Counts and colours are exact.  Floating results: about four times what the path differs by from the same
    computation in binary64 on the same inputs (2-norm, and the largest element)."""
    op = case["op"]
    if op in ("escape", "paint", "frames"):
        return "exact"
    return {"map": {"rel": 2e-7, "max": 1e-6}, "tape": {"rel": 2e-7, "max": 8e-7}, "vertex": {"rel": 4e-7, "max": 3e-6},
            "softmax": {"rel": 5e-7, "max": 2.5e-6}, "reduce": {"rel": 3e-7, "max": 1e-6}, "mse": {"rel": 6e-7, "max": 3e-6},
            "graph": {"rel": 5e-7, "max": 1e-5}}[op]
