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
