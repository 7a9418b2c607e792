"""fx_stage_attraction's outputs where both come back in one copy (up to 8,192 gates) and in two: equal
to the outputs of calls that ask for one of them, bit for bit, and near the FP64 sums."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 100, 8192, 8193])
def test_both_and_each(fx, ctx, oracle, n):
    rng = np.random.default_rng(n)
    c = fx.Circuit.from_nets(rng.integers(0, n, (2 * n, 2)).tolist(), n, 100.0, 100.0)
    x, y = (rng.random((2, n)) * 100).astype(np.float32)
    d = fx.Design(ctx, c)
    try:
        d.set_positions(x, y)
        got = d.attraction(1.5)
        for axis in (0, 1):
            out = np.full(n, np.nan, np.float32)
            p = out.ctypes.data_as(C.POINTER(C.c_float))
            args = (p, None) if axis == 0 else (None, p)
            assert d.lib.fx_stage_attraction(ctx.handle, d.handle, 1.5, *args) == 0
            assert np.array_equal(out, got[axis])
    finally:
        d.close()
    ap, ai = oracle.build_adjacency(n, c.net_ptr, c.net_gate)
    want = oracle.attraction_f64(ap, ai, x, y)
    for g, w in zip(got, want):
        # at most some tens of neighbours, terms up to 100: f32 sums within 1e-5 of the largest
        assert np.abs(g - 1.5 * np.asarray(w)).max() <= 1e-5 * (1.5 * np.abs(w).max() + 1e-30)
