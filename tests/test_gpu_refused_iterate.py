"""fx_force_iterate refuses a congestion grid that cannot be counted before it launches anything, for
any number of iterations, and the design's next call is as if that one had not been made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [0, 1, 2, 9])
@pytest.mark.parametrize("cols,rows", [(46341, 46341), (131073, 1)])
def test_grid_is_refused(fx, ctx, iters, cols, rows):
    s = fx.synth_plain(8, 3000, 3600, 65.0)
    good = fx.iter_cfg(density_bins=128, cong_cols=64, cong_rows=64)
    bad = fx.iter_cfg(density_bins=128, cong_cols=cols, cong_rows=rows)

    def run(refused):
        d = fx.Design(ctx, s.circuit)
        try:
            d.set_positions(s.placement.gate_x, s.placement.gate_y)
            if refused:
                launched = ctx.kernel_launches()
                with pytest.raises(fx.FluxionError, match="congestion grid"):
                    d.force_iterate(bad, iters)
                assert ctx.kernel_launches() == launched
            st = d.force_iterate(good, 3)
            return (*d.get_positions(), st.hpwl, st.total_overflow, st.density_energy)
        finally:
            d.close()

    got, want = run(True), run(False)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert got[2:] == want[2:]


@pytest.mark.parametrize("die", [65.0, 4000.0])  # 4000: the tree's deep-key buffers too
def test_no_memory_before_the_first_launch(fx, ctx, die):
    """Every allocation of the call precedes its launches, so that one that fails leaves nothing
    running on the second stream, which later calls do not wait for."""
    s = fx.synth_plain(9, 3000, 3600, die)
    cfg = fx.iter_cfg(density_bins=128, cong_cols=64, cong_rows=64)
    fail = fx.load().fx_test_fail_alloc
    try:
        for k in range(1, 200):
            d = fx.Design(ctx, s.circuit)
            d.set_positions(s.placement.gate_x, s.placement.gate_y)
            launched = ctx.kernel_launches()
            fail(k)
            try:
                d.force_iterate(cfg, 2)
                assert fail(0) > 0 and k > 10
                return
            except fx.FluxionError:
                assert fail(0) == 0
                assert ctx.kernel_launches() == launched
            finally:
                d.close()
    finally:
        fail(0)
    raise AssertionError("too many allocations")
