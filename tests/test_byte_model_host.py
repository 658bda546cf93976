"""metrics.first_sweep_bytes and metrics.iteration_bytes on columns taken from the
grid (form 4): no kernel reads a column, in the first sweep either."""
import pytest


def slots_read():
    """Slots that the eight phases of a first sweep read, a row of each colour:
    those whose neighbour's colour has been swept, in the order 7, 6, ..., 0."""
    total = 0
    for s, c in enumerate(range(7, -1, -1)):
        swept = set(range(7, c, -1))
        for k in range(27):
            flip = (k % 3 != 1) | (k // 3 % 3 != 1) << 1 | (k // 9 != 1) << 2
            total += (c ^ flip) in swept
    return total


@pytest.mark.parametrize("vb", [8, 4])
def test_first_sweep_reads_no_columns_on_grid_columns(vb):
    from hpcg_b200 import metrics
    per_row = slots_read() / 8
    assert per_row == 13
    rest = vb + 2 * vb + 3.5 * vb  # diagonal, right-hand side and x, the swept colours' x
    assert metrics.first_sweep_bytes(1, vb, 4) == per_row * vb + rest
    for pack in (0, 1, 2, 3):
        assert metrics.first_sweep_bytes(1, vb, pack) == metrics.first_sweep_bytes(1, vb) == per_row * (vb + 4) + rest


@pytest.mark.parametrize("vb", [8, 4])
def test_iteration_on_grid_columns(vb):
    """Against 32-bit columns everywhere: 108 bytes less a row and full phase,
    SpMV and restriction (an eighth of the rows), 52 less a row in the first sweep."""
    from hpcg_b200 import metrics
    n = 64
    rows = [n ** 3 >> 3 * l for l in range(4)]
    full = [7 / 8 + 1 / 8 + 15 / 8] * 3 + [7 / 8]
    less = sum(r * (52 + 108 * f) for r, f in zip(rows, full)) + 108 * rows[0]
    got = [metrics.iteration_bytes(n, n, n, vb, (w,) * 4, rtz_fused=True) for w in (0, 4)]
    assert got[0] - got[1] == pytest.approx(less, rel=1e-12)
