"""Barnes-Hut of designs that one cluster sorts (up to 32,768 points): the edges of its tiles
(512 pairs per block and item, eight blocks, 1 to 8 items), its capacity and one past it,
on uniform points, points on a line, one repeated point and a few repeated ones. Keys, order,
root and forces of the exact walk equal the oracle's bit for bit (no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n, rng):
    if kind == "uniform":
        return rng.random(n) * 500, rng.random(n) * 500
    if kind == "line":
        return rng.random(n) * 500, np.full(n, 77.0)
    if kind == "same":
        return np.full(n, 3.5), np.full(n, 9.25)
    c = rng.integers(0, 9, n)  # repeated points and near neighbours
    return c * 50.0 + rng.integers(0, 3, n) * 1e-3, c * 31.0


@pytest.mark.parametrize("n", [1, 2, 7, 9, 33, 511, 513, 4096, 4097, 8193, 16384, 16385, 32767, 32768,
                               32769, 65537, 131073])
@pytest.mark.parametrize("kind", ["uniform", "line", "few"])
def test_cluster_sort_and_tree(fx, ctx, oracle, n, kind):
    if kind == "few" and n > 8192:
        n = n % 4096 + 512  # crowded buckets are quadratic in the oracle's walk
    rng = np.random.default_rng(n)
    x, y = (v.astype(np.float32) for v in _points(kind, n, rng))
    c = fx.Circuit.from_nets([[0, 1]] if n >= 2 else [], n, 501.0, 501.0)
    d = fx.Design(ctx, c)
    try:
        d.set_positions(x, y)
        bx, by, keys, perm, root = d.barnes_hut(0.5, 0.5, 0.1, walk=fx.FX_BH_EXACT)
        gx, gy = d.barnes_hut(0.5, 0.5, 0.1, walk=fx.FX_BH_FAST)[:2]
    finally:
        d.close()
    o = oracle.bh_forces(x, y, 0.5, 0.5, float(np.float32(0.1)))
    assert np.array_equal(root, o["root"])
    assert np.array_equal(keys, o["keys"]) and np.array_equal(perm, o["perm"])
    assert np.array_equal(bx, o["fx32"]) and np.array_equal(by, o["fy32"])
    ref = np.hypot(o["fx"], o["fy"]).sum()
    assert np.hypot(gx - o["fx"], gy - o["fy"]).sum() <= 1e-5 * ref


@pytest.mark.parametrize("n", [262144, 262145, 524288, 524289, 528385])
def test_many_block_sort(fx, ctx, n):
    """Past the cluster's capacity: the sizes where tiles of keys and of prefix sums change.
    Keys and order against a stable sort in numpy; the deep-key path is not taken (die 501)."""
    rng = np.random.default_rng(n)
    x, y = (v.astype(np.float32) for v in _points("uniform", n, rng))
    x[: n // 3] = x[0]  # crowded digits
    c = fx.Circuit.from_nets([[0, 1]], n, 501.0, 501.0)
    d = fx.Design(ctx, c)
    try:
        d.set_positions(x, y)
        keys, perm, root = d.barnes_hut(0.5, 0.5, 0.1, walk=fx.FX_BH_FAST)[2:]
    finally:
        d.close()

    def cell(v, o):
        t = (v - o) / root[2] * np.float32(32768)
        return np.clip(np.ceil(t).astype(np.int64) - 1, 0, 32767).astype(np.uint32)

    def spread(v):
        for m, k in ((0x00ff00ff, 8), (0x0f0f0f0f, 4), (0x33333333, 2), (0x55555555, 1)):
            v = (v | (v << np.uint32(k))) & np.uint32(m)
        return v

    assert np.array_equal(keys, (spread(cell(x, root[0])) << np.uint32(1)) | spread(cell(y, root[1])))
    assert np.array_equal(perm, np.argsort(keys, kind="stable"))


def test_same_point(fx, ctx):
    n = 3000
    c = fx.Circuit.from_nets([[0, 1]], n, 501.0, 501.0)
    d = fx.Design(ctx, c)
    try:
        d.set_positions(np.full(n, 3.5, np.float32), np.full(n, 9.25, np.float32))
        bx, by, keys, perm, _ = d.barnes_hut(0.5, 0.5, 0.1, walk=fx.FX_BH_EXACT)
    finally:
        d.close()
    assert np.all(keys == keys[0]) and np.array_equal(perm, np.arange(n))
    assert not bx.any() and not by.any()
