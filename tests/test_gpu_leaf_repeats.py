"""Leaf batches that list gates more than once, on both sides of the 8,192 gates up to which the host
looks for repeats and the device does beyond: positions equal the oracle's leaf by leaf placement bit
for bit, in calls that alternate with a batch without repeats and with one that is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [1, 256, 257])
def test_repeated_gates(fx, ctx, oracle, leaves):
    rng = np.random.default_rng(leaves)
    g, n = 32 * leaves, 32 * leaves + 3
    c = fx.Circuit.from_nets(rng.integers(0, n, (2 * n, 2)).tolist(), n, 10.0, 10.0)
    lp = (32 * np.arange(leaves + 1)).astype(np.int32)
    plain = rng.permutation(n)[:g].astype(np.int32)
    twice = plain.copy()
    twice[5] = twice[31]                       # in one leaf
    twice[-1] = twice[3]                       # in the first leaf and in the last
    far = plain.copy()
    far[7] = n
    reg = np.tile(np.array([5.0, 5.0, 4.0, 4.0], np.float32), leaves)
    ap, ai = oracle.build_adjacency(n, c.net_ptr, c.net_gate)
    cfg = fx.leaf_cfg(force_iterations=4, schedule=fx._lib.FX_LEAF_CTA64)
    x0 = np.full(n, 3.25, np.float32)
    d = fx.Design(ctx, c)
    try:
        for gates in (twice, plain, far, twice):
            if gates is far:
                with pytest.raises(fx.FluxionError, match="out of range"):
                    d.place_leaves(lp, gates, reg, cfg)
                continue
            x, y, _ = d.place_leaves(lp, gates, reg, cfg, x0, x0.copy())
            ox, oy = x0.copy(), x0.copy()
            for l in range(leaves):
                oracle.place_leaf(gates[lp[l]:lp[l + 1]], ap, ai, reg[:4], 4, 1.0, 0.5, 0.9, 0.1,
                                  ox, oy)
            assert np.array_equal(x, ox) and np.array_equal(y, oy)
    finally:
        d.close()
