"""A fixed power-iteration count, one launch a depth, against the launch-per-step kernels that the
Rayleigh-quotient stop uses: one position above a chunk, a few chunks, several positions a thread,
more chunks than blocks and more of one cluster than are combined at a time. Both sum in the same
order: leaf orders are equal. Leaves of one chunk, so that no cluster of a few gates has a quotient
that repeats exactly, which stops the stepped kernels at any tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,iters", [(4097, 3), (9001, 30), (9001, 0), (333333, 5), (4300001, 2)])
def test_one_launch_is_the_stepped_kernels(fx, ctx, n, iters):
    d = fx.Design(ctx, fx.synth_plain(n, n, int(1.2 * n), float(1.2 * np.sqrt(n))).circuit)
    try:
        got, want = (d.partition(fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=iters, tol=t,
                                             max_leaf_size=4096))
                     for t in (0.0, 1e-300))
    finally:
        d.close()
    assert np.array_equal(got["leaf_ptr"], want["leaf_ptr"])
    assert np.array_equal(got["leaf_gate"], want["leaf_gate"])
