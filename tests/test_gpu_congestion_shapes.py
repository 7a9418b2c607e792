"""Congestion grids on both sides of each limit of the column scan's stripes (256, 512 and 1024 rows;
columns past 4096 stripes of 8 and 16) and of the cells below which a warp's increments are always
matched (4096), against the oracle's counts. The counts are whole numbers; the
overflow is an FP64 sum of f32 terms, within cells x 2^-53 of the exact one in any order."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,rows", [(1, 1), (8, 8), (63, 65), (64, 64), (33, 256), (33, 257), (100, 512), (100, 513),
                                       (70, 1024), (70, 1025), (1184, 256), (1185, 256), (1185, 512),
                                       (1185, 1024), (1184, 1025), (5, 4097), (2050, 1031),
                                       (32768, 600), (32769, 600), (65537, 300), (131072, 3)])
def test_counts_and_overflow(fx, ctx, oracle, cols, rows):
    rng = np.random.default_rng(cols + rows)
    n, side = 1200, 100.0
    c = fx.Circuit.from_nets(np.arange(n).reshape(-1, 3).tolist(), n, side, side)
    # a net's three gates lie close together (the oracle walks every cell of its box)
    near = np.repeat(rng.random((2, n // 3)) * side, 3, axis=1) + rng.normal(0, 0.5, (2, n))
    x, y = near.clip(0, side).astype(np.float32)
    d = fx.Design(ctx, c)
    try:
        first = d.congestion(cols, rows, x, y)
        counts, hpwl, total, most = d.congestion(cols, rows, x, y)  # the scan re-armed the grid
    finally:
        d.close()
    assert np.array_equal(first[0], counts) and first[1:] == (hpwl, total, most)
    h, v = oracle.congestion(c.net_ptr, c.net_gate, x, y, side, side, cols, rows)
    f = counts.astype(np.float32)
    assert np.array_equal(f, h) and np.array_equal(f, v)
    cap = (np.float32(side) / np.float32(cols) + np.float32(side) / np.float32(rows)) * np.float32(0.5)
    over = np.maximum((f + f) - cap, np.float32(0))
    exact = math.fsum(over.reshape(-1).astype(np.float64))
    assert abs(total - exact) <= cols * rows * 2.0 ** -53 * exact
    assert np.float32(most) == over.max()
