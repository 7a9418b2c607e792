"""FX_PART_FP64 with a fixed iteration count where a block's share of a depth holds no cluster:
positions of leaves only (a depth of leaves and clusters), or no position at all (a gate whose row
is longer than a share). The shares are restated on the host to show that these inputs make such
blocks; the orders are whole numbers and have no tolerance."""
import ctypes

import numpy as np
import pytest

from test_gpu_partition_fp64 import _mean_norm, _normed

SMS = 148


def _shares(beg, end, clustered, rows):
    """First positions of the blocks' shares of positions [beg, end): eight per position and one
    per in-cluster neighbour, cut evenly. With `clustered`, which positions lie in a cluster."""
    n = len(rows)
    cum = 8 * np.arange(n + 1, dtype=np.int64) + np.concatenate([[0], np.cumsum(rows)])
    grid = SMS * max(1, -(-int(cum[n]) // (SMS * 7168)))
    cut = np.searchsorted(cum, [int(cum[n]) * b // grid for b in range(grid + 1)])
    return [int(clustered[a:b].sum()) for a, b in zip(cut[:-1], cut[1:])]


def _plain(fx, n):
    return fx.synth_plain(n, n, int(1.2 * n), float(1.2 * np.sqrt(n))).circuit


def _hub(fx, n, fan):
    """A plain design with gate 7 on `fan` more two-pin nets; n = fan + 1: a star alone."""
    rng = np.random.default_rng(n)
    ends = [int(g) for g in rng.permutation(n) if g != 7][:fan]
    nets = [[7, g] for g in ends]
    if n > fan + 1:
        c = _plain(fx, n)
        nets += [c.net_gate[a:b].tolist() for a, b in zip(c.net_ptr[:-1], c.net_ptr[1:])]
    side = float(1.2 * np.sqrt(n))
    return fx.Circuit.from_nets(nets, n, side, side)


def _rows(fx, circuit):
    return np.diff(fx.build_adjacency(circuit)[0]).astype(np.int64)


def test_inputs_make_blocks_without_a_cluster(fx):
    # depth 1 of 8,193 gates: a leaf of 4,096 and a cluster of 4,097, of about ten neighbours
    in_cluster = np.arange(8193) >= 4096
    assert _shares(0, 8193, in_cluster, np.where(in_cluster, 10, 0)).count(0) > 20
    for n, fan in ((6000, 2500), (5001, 5000)):  # depth 0: one cluster
        rows = _rows(fx, _hub(fx, n, fan))
        assert _shares(0, n, np.ones(n, bool), rows).count(0) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("n,leaf", [(8193, 4096), (10001, 5000), (24581, 6145)])
def test_depth_of_leaves_and_clusters(fx, ctx, n, leaf):
    d = fx.Design(ctx, _plain(fx, n))
    try:
        got, want = (d.partition(fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=5, tol=t,
                                             max_leaf_size=leaf))
                     for t in (0.0, 1e-300))
    finally:
        d.close()
    assert np.array_equal(got["leaf_ptr"], want["leaf_ptr"])
    assert np.array_equal(got["leaf_gate"], want["leaf_gate"])


@pytest.mark.gpu
@pytest.mark.parametrize("n,fan,iters", [(6000, 2500, 3), (5001, 5000, 3), (20000, 19999, 2)])
def test_row_longer_than_a_share(fx, ctx, n, fan, iters):
    circuit = _hub(fx, n, fan)
    d = fx.Design(ctx, circuit)
    try:
        got = d.partition(fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=iters, tol=0.0,
                                      max_leaf_size=4096))
    finally:
        d.close()
    ap, ai = fx.build_adjacency(circuit)
    libm = ctypes.CDLL("libm.so.6")
    libm.sinf.restype, libm.sinf.argtypes = ctypes.c_float, [ctypes.c_float]
    sin_tab = np.array([libm.sinf(float(np.float32(i) * np.float32(2.71828)))
                        for i in range(n)], np.float32)

    def build(gates):
        m = len(gates)
        if m <= 4096:
            return gates
        o = _order(gates, ap, ai, sin_tab, iters)
        return build(o[:m // 2]) + build(o[m // 2:])

    assert np.array_equal(got["leaf_gate"], np.array(build(list(range(n)))))


def _order(gates, ap, ai, sin_tab, iters):
    """One bisection in the mode's arithmetic: rows as running f32 differences (cumsum adds in
    order), FP64 sums by chunks."""
    n = len(gates)
    at = {g: i for i, g in enumerate(gates)}
    rows = [[at[j] for j in ai[ap[g]:ap[g + 1]].tolist() if j in at] for g in gates]
    deg = np.array([len(r) for r in rows], np.float32)
    v = _normed(sin_tab[:n], *_mean_norm(sin_tab[:n], False))
    for _ in range(iters):
        lv = deg * v
        for i, r in enumerate(rows):
            if r:
                lv[i] = np.cumsum(np.concatenate([lv[i:i + 1], -v[r]]), dtype=np.float32)[-1]
        v = _normed(lv, *_mean_norm(lv, True))
    return [gates[i] for i in np.argsort(v + np.float32(0), kind="stable")]
