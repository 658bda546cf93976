"""A matrix that lacks a neighbour inside the grid does not take its columns from the
grid: a value set in the missing slot multiplies nothing. (With a zero there, as a
matrix that was only built has it, the neighbour's product would not show.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (24, 16, 8)


@pytest.mark.parametrize("level,slot", [(0, 26), (0, 0), (0, 14), (1, 26)])
def test_missing_neighbour_is_not_read(oracle, binding, monkeypatch, level, slot):
    ref = oracle.generate(*DIMS, nlevels=3)
    levels = [dict(nx=L.nx, ny=L.ny, nz=L.nz, nnz=L.nnz.copy(), cols=L.cols.copy(), vals=L.vals.copy(), f2c=L.f2c)
              for L in ref.levels]
    top = levels[level]
    nx, ny, nz = top["nx"], top["ny"], top["nz"]
    row = (nz // 2 * ny + ny // 2) * nx + nx // 2
    cols, vals = top["cols"].reshape(-1, 27), top["vals"].reshape(-1, 27)
    assert top["nnz"][row] == 27
    top["nnz"][row] = 26
    cols[row, slot:26], vals[row, slot:26] = cols[row, slot + 1:].copy(), vals[row, slot + 1:].copy()
    n, nl = int(np.prod(DIMS)), nx * ny * nz
    rng = np.random.default_rng(slot)
    r, x0 = rng.standard_normal(n), rng.standard_normal(n)
    dense = -1.0 - 0.1 * rng.random((nl, 27))
    dense[:, 13] = 40.0
    bare = dense.copy()
    bare[row, slot] = 0.0

    def use(values):
        p = binding.Problem.optimize(levels)
        try:
            p.set_values(level, values)
            y, z, z32, x = np.zeros(n), np.zeros(n), np.zeros(n), x0.copy()
            p.ComputeSPMV(x0, y)
            p.ComputeMG(r, z)
            p.ComputeMG_f32(r, z32)
            p.ComputeSYMGS(r, x)
            zm = np.zeros((2, n))
            p.ComputeMG_multi(np.stack([r, x0]), zm)
            return [y, z, z32, x, zm]
        finally:
            p.free()

    want = None
    for packed, tail in (("0", "0"), ("", "0"), ("", "1")):
        monkeypatch.setenv("HPCG_B200_PACKED", packed)
        monkeypatch.setenv("HPCG_B200_TAIL", tail)
        got = use(dense), use(bare)
        want = want or got[1]
        for g in got:
            for a, b in zip(g, want):
                assert np.array_equal(a, b), (packed, tail)
