"""The multi-system V-cycle on a hierarchy built from a caller's arrays whose
injected rows are not the all-even points: in one run of another colour, at the
top or below it, or not in one run. Bitwise the single-system V-cycle, which is
bitwise the same on stored columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (40, 24, 56)


def levels_with(oracle, level, offset, swap):
    """The 27-point hierarchy with level `level` injecting the points 2c + offset;
    swap: two coarse points trade theirs for a neighbour's (no run of rows)."""
    ref = oracle.generate(*DIMS)
    levels = [dict(nx=L.nx, ny=L.ny, nz=L.nz, nnz=L.nnz, cols=L.cols, vals=L.vals, f2c=L.f2c) for L in ref.levels]
    L = levels[level]
    cz, cy, cx = np.meshgrid(*(np.arange(L[a] // 2) for a in ("nz", "ny", "nx")), indexing="ij")
    ix, iy, iz = (2 * c + o for c, o in zip((cx, cy, cz), offset))
    f2c = ((iz * L["ny"] + iy) * L["nx"] + ix).astype(np.int32).ravel()
    if swap:
        f2c[3] += 1  # (an even x: its odd neighbour)
    L["f2c"] = f2c
    return levels


@pytest.mark.parametrize("level,offset,swap", [(0, (1, 1, 1), False), (0, (1, 0, 0), False), (1, (1, 1, 1), False),
                                               (0, (0, 0, 0), True), (0, (0, 0, 0), False)])
@pytest.mark.parametrize("nrhs", [2, 8])
def test_multi_injection_bitwise_single(oracle, binding, monkeypatch, level, offset, swap, nrhs):
    levels = levels_with(oracle, level, offset, swap)
    rng = np.random.default_rng(nrhs)
    n = int(np.prod(DIMS))
    r = rng.standard_normal((nrhs, n))
    got = []
    for packed in ("0", ""):
        monkeypatch.setenv("HPCG_B200_PACKED", packed)
        p = binding.Problem.optimize(levels)
        try:
            z = np.zeros_like(r)
            for j in range(nrhs):
                p.ComputeMG(np.ascontiguousarray(r[j]), z[j])
            x = np.zeros_like(r)
            p.ComputeMG_multi(r, x)
            got += [z, x]
        finally:
            p.free()
    for other in got[1:]:
        assert np.array_equal(other, got[0])
