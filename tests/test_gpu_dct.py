"""The fast-transform DCT Poisson solve (FX_DCT_I8 / FX_DCT_SIMT) on every kind of grid length
it takes: powers of two (radix 8 with 4 or 2 left over), odd factors, and the sizes where a
block's threads and its sequences per block change; on a die that is not square.

Tolerance: the transforms run in FP64 and three grids are rounded to f32 between and after
them (2^-24 relative per element each, independent of G), so potential, field and force are
held to 1e-6 relative L2.
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,prec", [(128, "simt"), (256, "i8"), (384, "simt"), (512, "i8"),
                                    (640, "simt"), (896, "i8"), (1024, "i8"), (1408, "i8"),
                                    (3968, "i8"), (4096, "simt"), (4224, "i8"), (8192, "i8")])
def test_solve_vs_fp64(fx, ctx, G, prec):
    rng = np.random.default_rng(G)
    n = 30_000
    w, h = np.float32(310.0), np.float32(190.0)
    # uniform gates, a dense cluster, and the die's corners
    x = np.concatenate([rng.random(n) * w, 40 + rng.normal(0, 2, 3000), [0, w, 0, w]])
    y = np.concatenate([rng.random(n) * h, 90 + rng.normal(0, 3, 3000), [0, 0, h, h]])
    x, y = x.astype(np.float32), y.astype(np.float32)
    c = fx.Circuit.from_nets([[0, 1]], len(x), float(w), float(h))
    d = fx.Design(ctx, c)
    try:
        d.set_positions(x, y)
        code = fx.FX_DCT_SIMT if prec == "simt" else fx.FX_DCT_I8
        out = d.density(G, 0.7, 1.0, code, grids=True)
        again = d.density(G, 0.7, 1.0, code)
        area = (c.gate_widths * c.gate_heights).astype(np.float64)
        ref = orc.density_forces(x, y, area, c.chip_width, c.chip_height, G, 0.7, 1.0)
        assert np.allclose(out["rho"], ref["rho"], rtol=2e-7, atol=1e-6)

        def err(*names):
            num = sum(np.sum((out[k].astype(np.float64) - ref[k]) ** 2) for k in names)
            return np.sqrt(num / sum(np.sum(ref[k] ** 2) for k in names))

        for names in (("phi",), ("ex", "ey"), ("ex",), ("ey",), ("fx", "fy")):
            assert err(*names) < 1e-6, (names, err(*names))
        assert abs(out["energy"] - ref["energy"]) <= 1e-6 * abs(ref["energy"])
        # the accumulator was re-armed, and the solve is reproducible
        assert np.array_equal(out["fx"], again["fx"]) and np.array_equal(out["fy"], again["fy"])
    finally:
        d.close()
