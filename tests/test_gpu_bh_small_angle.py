"""The exact walk at opening angles near 0, where most cells are opened: on both sides of the size and of
the angle at which the group walk takes over from the small designs' walk. Forces equal the oracle's bit
for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,theta", [(300, 0.0), (32768, 0.0), (32769, 0.0), (33000, 0.0009),
                                     (33000, 0.002)])
def test_forces(fx, ctx, oracle, n, theta):
    rng = np.random.default_rng(n)
    x, y = (rng.random((2, n)) * 300).astype(np.float32)
    d = fx.Design(ctx, fx.Circuit.from_nets([[0, 1]], n, 300.0, 300.0))
    try:
        d.set_positions(x, y)
        bx, by, keys = d.barnes_hut(0.5, theta, 0.1, walk=fx.FX_BH_EXACT)[:3]
    finally:
        d.close()
    o = oracle.bh_forces(x, y, 0.5, float(np.float32(theta)), float(np.float32(0.1)), threads=8)
    assert np.array_equal(keys, o["keys"])
    assert np.array_equal(bx, o["fx32"]) and np.array_equal(by, o["fy32"])
