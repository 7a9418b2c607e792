"""A refinement that stops at its first count (nothing above the threshold) counts twice, as one
iteration does: no second iteration is queued before the first decision is read. One that goes on
ends where it did."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [8, 100])
def test_first_stop_counts_twice(fx, ctx, grid):
    s = fx.synth_plain(3, 3000, 3600, 65.0)
    d = fx.Design(ctx, s.circuit)

    def run(**kw):
        x, y = s.placement.gate_x.copy(), s.placement.gate_y.copy()
        at = ctx.kernel_launches()
        st = d.refine(fx.refine_cfg(grid_cols=grid, grid_rows=grid, **kw), x, y)
        return ctx.kernel_launches() - at, st, x

    try:
        stopped, st, x = run(overflow_threshold=1e12, max_iterations=100)
        one, st1, _ = run(overflow_threshold=0.0, max_iterations=1)
        two, st2, _ = run(overflow_threshold=0.0, max_iterations=2)
    finally:
        d.close()
    assert stopped == one < two
    assert (st.iterations, st.moves) == (0, 0) and np.array_equal(x, s.placement.gate_x)
    assert (st1.iterations, st2.iterations) == (1, 2) and st2.moves >= st1.moves
