"""GPU: column sums at the edges of the kernel's tiling: one column, fewer columns than a warp, one column or
float4 more than a tile, one row, fewer rows than a block takes at a time, and shapes whose partial sums
need the second stage.  Oracle: binary64 sums.  Tolerance: 1e-5 of each column's sum of magnitudes, as in
test_rows_gpu.py (sums of n binary32 values in any order are off by at most n*2^-24 of it, and the tree keeps
chains below 8 + 4096 + 20 terms)."""
import numpy as np
import pytest

import oracle
from vernondsl_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 4), (2, 256), (3, 260), (100000, 1), (70001, 4), (20000, 33), (5003, 127), (5003, 128), (2500, 129),
                                       (999, 255), (15, 256), (17, 257), (4097, 1024), (1000, 1001), (37, 65537), (40, 65540)])
def test_col_sum_at_the_edges_of_its_tiles(dev, stream, rows, cols):
    m = (np.random.default_rng(rows * 31 + cols).standard_normal((rows, cols)) + 0.25).astype(np.float32)
    M, c = dev.from_numpy(m), dev.empty(cols, np.float32)
    got = []
    for _ in range(2):
        c.fill(0xEE, stream=stream)
        ops.col_sum(stream, M, c, rows, cols)
        stream.check()
        got.append(c.download())
    scale = np.abs(m).astype(np.float64).sum(axis=0)
    assert (np.abs(got[0].astype(np.float64) - oracle.col_sum(m)) <= 1e-5 * scale + 1e-30).all()
    assert np.array_equal(got[0], got[1])      # fixed order of additions
    M.close()
    c.close()


def rows_per_thread(rows, cols, sms):
    """How many rows a thread of the first stage adds, and how many threads of a block share a column (k_rows.cu, plan_col_sum)."""
    vec = cols % 4 == 0
    groups = cols // 4 if vec else cols
    gx = -(-groups // (64 if vec else 128))
    W = -(-groups // gx)
    R = 256 // W
    gy = max(1, min(sms * (5 if vec else 8) // gx, -(-rows // (8 * R)), 4096))
    return -(-rows // (gy * R)), R


@pytest.mark.parametrize("rows,cols", [(1024, 65535), (1024, 65536), (4096, 16384), (4097, 16381), (40000, 257), (33, 4)])
def test_rounding_errors_do_not_add_up_along_the_rows(dev, stream, rows, cols):
    """Every element is the same v, chosen so that one addition of v to a sum near the end of a thread's rows drops almost
    half a unit, always to the same side: the error of a chain of n additions is then n/4 units of 2^-24, and only a
    short chain stays inside the bound.  A thread adds whole groups of eight rows as trees (3 roundings, then one to the
    running sum), or, single columns, into four running sums; the up to seven rows left over one by one; a block its R
    sums as a tree.  The rest is binary64.  Equal values grow a running sum evenly: c additions to it lose (c + 1) / 2
    units of the result at most, half the bound for arbitrary values."""
    n, R = rows_per_thread(rows, cols, dev.sm_count)
    unit = 2.0 ** (max(int(n - 1).bit_length(), 2) - 1 - 23)       # of sums in the upper half of a thread's range
    v = np.float32(1 + int(0.49 * unit * 2 ** 23) * 2.0 ** -23)
    m = np.full((rows, cols), v, np.float32)
    M, c = dev.from_numpy(m), dev.empty(cols, np.float32)
    ops.col_sum(stream, M, c, rows, cols)
    stream.check()
    chain = n // 8 if cols % 4 == 0 else n // 8 * 2
    depth = (chain + 1) / 2 + 3 + n % 8 + int(R).bit_length() + 1
    want = rows * float(v)
    assert np.abs(c.download().astype(np.float64) - want).max() <= depth * 2.0 ** -24 * want, (n, R)
    M.close()
    c.close()
