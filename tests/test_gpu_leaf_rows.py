"""In-leaf adjacency rows built on the device (batches that list every gate once): leaves of 0,
1, 31-33 and 512 gates, gates in shuffled order, whole batches and batches that leave gates out
(which keep the caller's positions), nets that reach across leaves. Positions equal the oracle's
place_gates_in_leaf bit for bit (no tolerance); a gate out of range is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[0, 1, 31, 32, 33, 0, 64, 65], [512, 1, 300, 0], [7]])
@pytest.mark.parametrize("spare", [0, 5])
def test_rows(fx, ctx, oracle, sizes, spare):
    rng = np.random.default_rng(sum(sizes) + spare)
    g = sum(sizes)
    n = g + spare
    nets = [list(rng.choice(n, size=min(n, int(rng.integers(2, 6))), replace=False))
            for _ in range(3 * n)]
    c = fx.Circuit.from_nets(nets, n, 10.0, 10.0)
    order = rng.permutation(n)[:g].astype(np.int32)
    lp = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    reg = np.array([[l + 0.5, 0.5, 1.0, 1.0] for l in range(len(sizes))], np.float32)
    x0 = np.full(n, 3.25, np.float32)
    d = fx.Design(ctx, c)
    try:
        x, y, _ = d.place_leaves(lp, order, reg.ravel(),
                                 fx.leaf_cfg(force_iterations=15, schedule=fx._lib.FX_LEAF_CTA64),
                                 x0, x0.copy())
        bad = order.copy()
        bad[-1] = n
        with pytest.raises(fx.FluxionError):
            d.place_leaves(lp, bad, reg.ravel(), fx.leaf_cfg(force_iterations=2))
    finally:
        d.close()
    ap, ai = oracle.build_adjacency(n, c.net_ptr, c.net_gate)
    ox, oy = x0.copy(), x0.copy()
    for l in range(len(sizes)):
        if sizes[l]:
            oracle.place_leaf(order[lp[l]:lp[l + 1]], ap, ai, reg[l], 15, 1.0, 0.5, 0.9, 0.1,
                              ox, oy)
    assert np.array_equal(x, ox) and np.array_equal(y, oy)
