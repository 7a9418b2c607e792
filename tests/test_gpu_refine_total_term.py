"""One term of the refinement loop's exact overflow sum: its increment in units of the sum's binade
against the f32 addition itself, for terms up to the limit where two roundings could meet (a numpy
restatement, both parities), and on the GPU a grid whose sum is odd when a cell of all-ones mantissa
just below 2^22 units arrives. Bit for bit."""
import numpy as np
import pytest

F = np.float32
WHOLE = F(4194303.0)


def _increments(t):
    """From even and odd sums, as total_term has them."""
    even = (t + F(12582912.0)).view(np.int32) - 0x4b400000
    odd = (t + F(12582913.0)).view(np.int32) - 0x4b400001
    return int(even), int(odd)


def test_increment_is_the_addition():
    rng = np.random.default_rng(3)
    terms = [F(4194290 + 0.25 * i) for i in range(64)]
    for e in range(-4, 23):
        for m in [*range(0xfffff0, 0x1000000), *range(0x800000, 0x800010),
                  *rng.integers(0x800000, 0x1000000, 100)]:
            terms.append(F(np.ldexp(float(m), e - 24)))
    seen = 0
    for t in terms:
        if not t < WHOLE:
            continue
        inc = _increments(t)
        for s in (1 << 23, (1 << 23) + 1, (1 << 23) + 2, 12345678, 12345679):
            total = F(s) + t
            if s + inc[s & 1] < 1 << 24:
                assert F(s + inc[s & 1]) == total, (float(t), s)
            else:  # the term is added by itself
                assert total >= F(1 << 24), (float(t), s)
            seen += 1
    assert seen > 10000


@pytest.mark.gpu
@pytest.mark.parametrize("late", [[33], [33, 0, 33], [33] * 40])
def test_all_ones_term_on_an_odd_sum(fx, ctx, late):
    # cap = 2 + 2^-18: cells of 5, 30 and 33 nets leave an odd sum in [128, 256), where a cell of
    # 33 nets, 64 - 2^-18, is 4194303.75 units; past the cells that are added one by one
    cols, pitch = 1024, F(2 + 2.0 ** -18)
    cells = np.zeros(cols, np.int64)
    cells[:3] = 5, 30, 33
    cells[600:600 + len(late)] = late
    used = np.flatnonzero(cells)
    nets = [[2 * i, 2 * i + 1] for i, c in enumerate(used) for _ in range(cells[c])]
    x = np.repeat((used.astype(F) + F(0.5)) * pitch, 2).astype(F)
    y = np.full(len(x), pitch / 2, F)
    d = fx.Design(ctx, fx.Circuit.from_nets(nets, len(x), float(F(cols) * pitch), float(pitch)))
    try:
        st, counts = d.refine(fx.refine_cfg(max_iterations=0, grid_cols=cols, grid_rows=1), x, y,
                              counts=True)
    finally:
        d.close()
    assert np.array_equal(counts.reshape(-1), cells)
    f = cells.astype(F)
    over = np.maximum((f + f) - pitch, F(0))
    assert F(st.total_overflow) == np.cumsum(over, dtype=F)[-1]
