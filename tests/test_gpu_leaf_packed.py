"""FX_LEAF_FAST's per-gate schedules in both forms of the pair term: by packed pairs in batches that
fill the device, by scalar instructions in small ones. Leaves placed in either come out bit for bit the
same, and as the pair-triangle schedule has them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,leaves", [(39, 2500), (54, 1500), (81, 1200), (127, 1300)])
def test_forms_agree(fx, ctx, size, leaves):
    rng = np.random.default_rng(size)
    n = size * leaves
    at = np.arange(n) // size * size
    nets = at[:, None] + rng.integers(0, size, (n, 3))
    c = fx.Circuit(n, (3 * np.arange(n + 1)).astype(np.int32), nets.astype(np.int32).reshape(-1),
                   np.ones(n, np.float32), np.ones(n, np.float32), 100.0, 100.0)
    lp = (size * np.arange(leaves + 1)).astype(np.int32)
    reg = rng.uniform(5, 50, 4 * leaves).astype(np.float32)
    few = 7
    d = fx.Design(ctx, c)

    def place(k, schedule):
        x, y, _ = d.place_leaves(lp[:k + 1], np.arange(lp[k], dtype=np.int32), reg[:4 * k],
                                 fx.leaf_cfg(force_iterations=20, precision=fx.FX_LEAF_FAST,
                                             schedule=schedule))
        return np.stack([x[:lp[k]], y[:lp[k]]])

    try:
        want = place(leaves, fx._lib.FX_LEAF_PAIR128)
        for name in ("WARP", "CTA64", "CTA128", "CTA256"):
            schedule = getattr(fx._lib, "FX_LEAF_" + name)
            assert np.array_equal(place(leaves, schedule), want), name
            assert np.array_equal(place(few, schedule), want[:, :lp[few]]), name
    finally:
        d.close()
