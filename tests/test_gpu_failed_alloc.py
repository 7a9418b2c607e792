"""A call that runs out of device memory part-way leaves nothing behind that a later call takes for
a finished setup: each allocation of the call fails once, and the next good call gives what a fresh
design gives, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def fail_alloc(fx):
    lib = fx.load()
    yield lib.fx_test_fail_alloc
    lib.fx_test_fail_alloc(0)


def _failures(fail_alloc, make, call):
    """A fresh state from make(), call(state) with its k-th allocation failing, for every k."""
    for k in range(1, 200):
        state = make()
        fail_alloc(k)
        try:
            call(state)
        except Exception as e:
            assert "allocation" in str(e), e
            assert fail_alloc(0) == 0
            yield state
            continue
        assert fail_alloc(0) > 0, "a failed allocation went unnoticed"
        assert k > 1, "the call allocated nothing"
        state.close()
        return
    raise AssertionError("too many allocations")


@pytest.mark.parametrize("precision", ["FX_DCT_I8", "FX_DCT_TF32", "FX_DCT_BF16"])
def test_density_of_the_previous_grid(fx, ctx, fail_alloc, precision):
    s = fx.synth_plain(5, 2000, 2400, 54.0)
    prec = getattr(fx, precision)

    def make():
        d = fx.Design(ctx, s.circuit)
        d.set_positions(s.placement.gate_x, s.placement.gate_y)
        return d

    def density(d, bins):
        return d.density(bins, 0.7, 1.0, prec)

    d = make()
    want = density(d, 128)
    d.close()

    def with_grid():
        d = make()
        density(d, 128)
        return d

    for d in _failures(fail_alloc, with_grid, lambda d: density(d, 256)):
        got = density(d, 128)
        assert np.array_equal(got["fx"], want["fx"]) and np.array_equal(got["fy"], want["fy"])
        assert got["energy"] == want["energy"]
        d.close()


@pytest.mark.parametrize("die", [54.0, 4000.0])  # 4000: the tree's deep-key buffers too
def test_iteration(fx, ctx, fail_alloc, die):
    s = fx.synth_plain(6, 2000, 2400, die)
    cfgs = [fx.iter_cfg(density_bins=128, dct_precision=fx.FX_DCT_I8, cong_cols=c, cong_rows=c)
            for c in (64, 100)]

    def make():
        return fx.Design(ctx, s.circuit)

    def iterate(d, cfg):
        x, y = s.placement.gate_x.copy(), s.placement.gate_y.copy()
        d.set_positions(x, y)
        st = d.force_iterate(cfg, 2)
        return (*d.get_positions(), st.hpwl, st.total_overflow, st.density_energy)

    d = make()
    want = iterate(d, cfgs[0])
    d.close()

    def same(got):
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        assert got[2:] == want[2:]

    for d in _failures(fail_alloc, make, lambda d: iterate(d, cfgs[0])):
        same(iterate(d, cfgs[0]))
        d.close()

    def with_grid():
        d = make()
        d.congestion(64, 64, s.placement.gate_x, s.placement.gate_y)
        return d

    def other_grid(d):
        return d.congestion(100, 100, s.placement.gate_x, s.placement.gate_y)

    d = with_grid()
    small = d.congestion(64, 64, s.placement.gate_x, s.placement.gate_y)
    d.close()
    for d in _failures(fail_alloc, with_grid, other_grid):
        got = d.congestion(64, 64, s.placement.gate_x, s.placement.gate_y)
        assert np.array_equal(got[0], small[0]) and got[1:] == small[1:]
        d.close()


def test_saved_state(fx, ctx, fail_alloc):
    s = fx.synth_plain(7, 2000, 2400, 54.0)
    x, y = s.placement.gate_x, s.placement.gate_y

    def make():
        d = fx.Design(ctx, s.circuit)
        d.set_positions(x, y)
        return d

    for d in _failures(fail_alloc, make, lambda d: d.save_state()):
        with pytest.raises(Exception):
            d.restore_state()
        d.save_state()
        d.set_positions(y, x)
        d.restore_state()
        got = d.get_positions()
        assert np.array_equal(got[0], x) and np.array_equal(got[1], y)
        d.close()
