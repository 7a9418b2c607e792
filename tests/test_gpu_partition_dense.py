"""FX_PART_FP64 on dense netlists, where a depth's clusters have too many neighbours for a block each
and, denser still, rows too long for the one-launch form: leaf orders equal a numpy restatement's, with
a fixed iteration count and with the stop rule. Whole numbers: no tolerance."""
import ctypes

import numpy as np
import pytest

from test_gpu_partition_fp64 import _mean_norm, _normed, _sum

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pins,nets,iters,tol,leaf", [
    (1500, 100, 20, 6, 0.0, 64),      # 146k neighbours: above the fixed count's limit, below the other
    (1500, 100, 20, 6, 1e-3, 64),
    (1300, 300, 8, 6, 0.0, 64),       # 480k: above both, a few depths
    (1300, 300, 8, 6, 1e-3, 64),
    (5600, 3000, 4, 2, 0.0, 4096),    # 18M, 3,300 a row
])
def test_matches_restatement(fx, ctx, n, pins, nets, iters, tol, leaf):
    rng = np.random.default_rng(n + pins)
    circuit = fx.Circuit.from_nets([rng.choice(n, pins, replace=False).tolist()
                                    for _ in range(nets)] + [[i, i + 1] for i in range(n - 1)],
                                   n, 100.0, 100.0)
    d = fx.Design(ctx, circuit)
    try:
        got = d.partition(fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=iters, tol=tol,
                                      max_leaf_size=leaf))
    finally:
        d.close()
    ap, ai = fx.build_adjacency(circuit)
    libm = ctypes.CDLL("libm.so.6")
    libm.sinf.restype, libm.sinf.argtypes = ctypes.c_float, [ctypes.c_float]
    sin_tab = np.array([libm.sinf(float(np.float32(i) * np.float32(2.71828)))
                        for i in range(n)], np.float32)

    def order(gates):
        m = len(gates)
        place = np.full(n, -1)
        place[gates] = np.arange(m)
        rows = [r[r >= 0] for r in (place[ai[ap[g]:ap[g + 1]]] for g in gates)]
        deg = np.array([len(r) for r in rows], np.float32)
        v = _normed(sin_tab[:m], *_mean_norm(sin_tab[:m], False))
        lam = 0.0
        for it in range(1, iters + 1):
            lv = deg * v
            for i, r in enumerate(rows):
                if len(r):  # a running f32 difference: cumsum adds in order
                    lv[i] = np.cumsum(np.concatenate([lv[i:i + 1], -v[r]]), dtype=np.float32)[-1]
            prev, lam = lam, _sum(v.astype(np.float64) * lv.astype(np.float64))
            v = _normed(lv, *_mean_norm(lv, True))
            if tol > 0 and it > 1 and abs(lam - prev) <= tol * abs(lam):
                break
        return np.asarray(gates)[np.argsort(v + np.float32(0), kind="stable")]

    def build(gates):
        m = len(gates)
        least = int(np.ceil(np.float32(m) * np.float32(0.4)))
        cut = min(max(m // 2, least), m - least)
        if m <= leaf or m <= 8 or cut <= 0 or cut >= m:
            return list(gates)
        o = order(gates)
        return build(o[:cut]) + build(o[cut:])

    assert np.array_equal(got["leaf_gate"], np.array(build(np.arange(n))))


@pytest.mark.parametrize("tol", [0.0, 1e-6])
def test_last_depth_of_few_clusters(fx, ctx, tol):
    """51,201 gates in leaves of 50 have one depth more than 51,200, of a single cluster of 51 gates:
    one launch, however many neighbours the whole design has."""
    launches = []
    for n in (51200, 51201):
        d = fx.Design(ctx, fx.synth_plain(5, n, int(1.2 * n), float(1.2 * np.sqrt(n))).circuit)
        at = ctx.kernel_launches()
        d.partition(fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=3, tol=tol, max_leaf_size=50))
        launches.append(ctx.kernel_launches() - at)
        d.close()
    assert launches[1] == launches[0] + 1, launches
