"""The refinement loop's total overflow, the reference's sequential f32 running sum
(HAPR_fluxion_v4/src/data/grid.rs:86-91), against the same sum in numpy float32, bit for bit:
around the chunk size (4096 cells), with capacities that make rounding ties common (dyadic)
or absent, all-zero stretches, and sums far past 2^24 units. No tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,rows", [(1, 1), (7, 5), (91, 90), (128, 64), (4097, 1), (8193, 1),
                                       (256, 256), (300, 517)])
@pytest.mark.parametrize("pitch", [1.0, 0.25, 3.1415927, 400.0])
@pytest.mark.parametrize("nets", [60, 30000])
def test_total_is_the_sequential_sum(fx, ctx, cols, rows, pitch, nets):
    rng = np.random.default_rng(cols * 7 + rows + nets)
    n = 2000
    w, h = np.float32(cols * pitch), np.float32(rows * pitch)
    pairs = rng.integers(0, n, (nets, 2))
    pairs[:, 1] = np.where(pairs[:, 0] == pairs[:, 1], (pairs[:, 1] + 1) % n, pairs[:, 1])
    c = fx.Circuit.from_nets(pairs.tolist(), n, float(w), float(h))
    # half the gates in a corner, so that large parts of the grid stay empty with few nets
    x = (rng.random(n) * np.where(np.arange(n) % 2, w, w / 16)).astype(np.float32)
    y = (rng.random(n) * np.where(np.arange(n) % 2, h, h / 16)).astype(np.float32)
    d = fx.Design(ctx, c)
    try:
        st, counts = d.refine(fx.refine_cfg(max_iterations=0, grid_cols=cols, grid_rows=rows),
                              x, y, counts=True)
    finally:
        d.close()
    cap = np.float32((w / np.float32(cols) + h / np.float32(rows)) * np.float32(0.5))
    f = counts.astype(np.float32)
    a = np.maximum((f + f) - cap, np.float32(0.0))
    total = np.cumsum(a, dtype=np.float32)[-1]
    assert np.float32(st.total_overflow) == total
    assert np.float32(st.max_overflow) == a.max()
