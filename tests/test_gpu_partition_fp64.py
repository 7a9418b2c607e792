"""FX_PART_FP64 hierarchies against a numpy restatement of the mode's arithmetic, gate for gate:
designs below one 4096-position chunk, just above it, and of several chunks (whose first depths
run the many-block kernels and the rest a block per cluster), fixed iteration counts and the
Rayleigh-quotient stop. Leaf orders are whole numbers: no tolerance."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _chunk_sum(a):
    """32 strided sequential sums and the shuffle tree, as one chunk is summed."""
    rows = np.zeros((-(-len(a) // 32), 32))
    rows.reshape(-1)[:len(a)] = a
    s = np.zeros(32)
    for r in rows:
        s = s + r
    o = 16
    while o:
        s[:32 - o] = s[:32 - o] + s[o:]
        o //= 2
    return s[0]


def _sum(a):
    t = 0.0
    for k in range(0, len(a), 4096):
        t += _chunk_sum(a[k:k + 4096])
    return t


def _mean_norm(x, deflate):
    a = x.astype(np.float64)
    s1, s2 = _sum(a), _sum(a * a)
    m = s1 / len(x) if deflate else 0.0
    var = max(float(Fraction(s2) - Fraction(s1) * Fraction(m)), 0.0) if deflate else s2
    norm = np.sqrt(var)
    return F(m), (F(norm) if norm > 1e-10 else F(0))


def _normed(x, m, r):
    y = x - m
    return y / r if r > 0 else y


def _order(gates, nbr, sin_tab, iters, tol):
    n = len(gates)
    at = {g: i for i, g in enumerate(gates)}
    rows = [[at[j] for j in nbr[g] if j in at] for g in gates]
    width = max((len(r) for r in rows), default=0)
    col = np.array([r + [n] * (width - len(r)) for r in rows], np.int64).reshape(n, width)
    deg = np.array([len(r) for r in rows], F)
    v = _normed(sin_tab[:n], *_mean_norm(sin_tab[:n], False))
    lam = 0.0
    for it in range(1, iters + 1):
        lv = deg * v
        ext = np.append(v, F(0))
        for k in range(width):
            live = col[:, k] < n
            lv[live] = lv[live] - ext[col[live, k]]
        prev, lam = lam, _sum(v.astype(np.float64) * lv.astype(np.float64))
        v = _normed(lv, *_mean_norm(lv, True))
        if tol > 0 and it > 1 and abs(lam - prev) <= tol * abs(lam):
            break
    return [gates[i] for i in np.argsort(v + F(0), kind="stable")]


@pytest.mark.parametrize("n,iters,tol", [(70, 30, 0.0), (700, 30, 0.0), (4096, 5, 0.0),
                                         (4097, 7, 0.0), (9001, 4, 0.0), (3000, 60, 1e-3),
                                         (65, 0, 0.0)])
def test_matches_restatement(fx, ctx, n, iters, tol):
    s = fx.synth_plain(n, n, int(1.2 * n), float(1.2 * np.sqrt(n)))
    d = fx.Design(ctx, s.circuit)
    try:
        got = d.partition(fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=iters, tol=tol))
    finally:
        d.close()
    ap, ai = fx.build_adjacency(s.circuit)
    nbr = [ai[ap[g]:ap[g + 1]].tolist() for g in range(n)]
    import ctypes
    libm = ctypes.CDLL("libm.so.6")
    libm.sinf.restype, libm.sinf.argtypes = ctypes.c_float, [ctypes.c_float]
    sin_tab = np.array([libm.sinf(float(F(i) * F(2.71828))) for i in range(n)], F)

    def build(gates):
        m = len(gates)
        least = int(np.ceil(F(m) * F(0.4)))
        cut = min(max(m // 2, least), m - least)
        if m <= 64 or m <= 8 or cut <= 0 or cut >= m:
            return gates
        o = _order(gates, nbr, sin_tab, iters, tol)
        return build(o[:cut]) + build(o[cut:])

    assert np.array_equal(got["leaf_gate"], np.array(build(list(range(n)))))
