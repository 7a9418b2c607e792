"""FX_BH_FAST with distance floors so small that a point's term to itself, k / min_dist^3, or the
reciprocal root of the floor's square is infinite in single precision: forces are finite and within
the mode's 1e-5 of the exact walk's, and every interaction is counted, as with an ordinary floor."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 3000, 40000])
@pytest.mark.parametrize("min_dist", [1e-12, 1e-13, 1e-18, 2e-19, 1e-21, 1e-30])
def test_forces_are_finite(fx, ctx, n, min_dist):
    rng = np.random.default_rng(n)
    x, y = (rng.random((2, n)) * 100).astype(np.float32)
    d = fx.Design(ctx, fx.Circuit.from_nets([[0, 1]], n, 100.0, 100.0))
    try:
        d.set_positions(x, y)
        got = d.barnes_hut(0.5, 0.5, min_dist, walk=fx.FX_BH_FAST, terms=True)
        want = d.barnes_hut(0.5, 0.5, min_dist, walk=fx.FX_BH_EXACT)
        d.force_iterate(fx.iter_cfg(min_dist=min_dist, density_bins=0, cong_cols=0, cong_rows=0), 1)
        moved = d.get_positions()
    finally:
        d.close()
    g, w = np.stack(got[:2]).astype(np.float64), np.stack(want[:2]).astype(np.float64)
    assert np.isfinite(w).all() and np.isfinite(g).all() and np.isfinite(moved).all()
    assert np.sqrt(((g - w) ** 2).sum() / (w ** 2).sum()) < 1e-5
    assert (got[5] >= 1).all() and (got[5] < n).all()
