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
