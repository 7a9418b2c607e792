"""In-leaf rows of gates with many neighbours (by one lane up to 64, by the warp beyond): a gate on all
nets, cliques of 60 to 300, spread over leaves, whose rows keep the design's adjacency order: positions
equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,pins", [(66, 66, 0), (65, 33, 0), (2000, 64, 0), (3000, 500, 0),
                                         (1200, 97, 60), (1200, 97, 66), (1500, 512, 300)])
def test_rows(fx, ctx, oracle, n, leaf, pins):
    rng = np.random.default_rng(n + leaf + pins)
    nets = [[0, i] for i in range(1, n)] if not pins else \
        [rng.choice(n, pins, replace=False).tolist() for _ in range(6)]
    nets += [[int(a), int(b)] for a, b in rng.integers(0, n, (n, 2)) if a != b]
    c = fx.Circuit.from_nets(nets, n, 40.0, 40.0)
    gates = rng.permutation(n).astype(np.int32)
    lp = np.append(np.arange(0, n, leaf), n).astype(np.int32)
    reg = np.tile(np.array([20.0, 20.0, 30.0, 30.0], np.float32), len(lp) - 1)
    d = fx.Design(ctx, c)
    try:
        x, y, _ = d.place_leaves(lp, gates, reg, fx.leaf_cfg(force_iterations=5,
                                                             schedule=fx._lib.FX_LEAF_CTA64))
    finally:
        d.close()
    ap, ai = oracle.build_adjacency(n, c.net_ptr, c.net_gate)
    ox, oy = np.zeros(n, np.float32), np.zeros(n, np.float32)
    for l in range(len(lp) - 1):
        oracle.place_leaf(gates[lp[l]:lp[l + 1]], ap, ai, reg[:4], 5, 1.0, 0.5, 0.9, 0.1, ox, oy)
    assert np.array_equal(x, ox) and np.array_equal(y, oy)
