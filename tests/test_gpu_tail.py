"""The small end of the V-cycle in one launch (tail.cuh): the same bits as the
phases launched one by one (HPCG_B200_TAIL=0), for grids whose small levels
end on partial slabs, odd sides, one block and several."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# four levels: one block; slabs of unequal runs of z pairs; odd coarsest sides;
# flat in z; level 0 above the one-launch levels
GRIDS = [(8, 8, 8, 4), (16, 24, 32, 4), (24, 40, 16, 4), (40, 24, 72, 4), (64, 48, 8, 4), (72, 56, 40, 4),
         (13, 7, 9, 1), (33, 31, 29, 1), (5, 3, 1, 1), (2, 1, 33, 1), (1, 1, 1, 1)]


def both(binding, monkeypatch, make, use):
    out = []
    for on in ("0", "1"):
        monkeypatch.setenv("HPCG_B200_TAIL", on)
        p = make()
        try:
            out.append(use(p))
        finally:
            p.free()
    return out


@pytest.mark.parametrize("dims", GRIDS)
def test_small_levels_bitwise_as_phases(binding, monkeypatch, dims):
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(sum(dims))
    r, x0 = rng.standard_normal(n), rng.standard_normal(n)
    vals = -1.0 - 0.1 * rng.random((n, 27))
    vals[:, 13] = 30.0 + rng.random(n)
    diag = 40.0 + rng.random(n)

    def use(p):
        got = []
        for change in (None, lambda: p.set_values(0, vals), lambda: p.set_diagonal(diag)):
            if change:
                change()
            z, z32, x = np.zeros(n), np.zeros(n), x0.copy()
            p.ComputeMG(r, z)
            p.ComputeMG_f32(r, z32)
            p.ComputeSYMGS(r, x)
            got += [z, z32, x]
        return got

    a, b = both(binding, monkeypatch, lambda: binding.Problem.generate(*dims[:3], nlevels=dims[3]), use)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)


def test_small_levels_cg_as_phases(binding, monkeypatch):
    """CG whose V-cycle is one launch, as a graph and after a change of values;
    only the order of the r'z sum differs from the phases' fused partials."""
    n = 32 ** 3
    b = np.random.default_rng(3).uniform(-1, 1, n)

    def use(p):
        got = []
        for scale in (1.0, 1.5):
            if scale != 1.0:
                p.set_diagonal(np.full(n, 26.0 * scale))
            x, y = np.zeros(n), np.zeros(n)
            got += [p.CG(b, x, 12, 0.0), p.CG_mixed(b, y, 12, 0.0), x, y]
        return got

    a, c = both(binding, monkeypatch, lambda: binding.Problem.generate(32), use)
    for u, v in zip(a, c):
        if isinstance(u, tuple):
            assert u[0] == v[0] and abs(u[1] / u[2] - v[1] / v[2]) <= 1e-10
        else:
            assert np.max(np.abs(u - v)) <= 1e-10 * np.max(np.abs(u))


def test_matrix_without_a_neighbour_keeps_the_phases(oracle, binding, monkeypatch):
    """A matrix that lacks a neighbour inside the grid does not qualify: its
    results are those of the phases."""
    ref = oracle.generate(16)
    levels = [dict(nx=L.nx, ny=L.ny, nz=L.nz, nnz=L.nnz.copy(), cols=L.cols.copy(), vals=L.vals.copy(), f2c=L.f2c)
              for L in ref.levels]
    top = levels[0]
    cols, vals = top["cols"].reshape(-1, 27), top["vals"].reshape(-1, 27)
    row = 16 * 16 * 8 + 16 * 8 + 8
    top["nnz"][row] -= 1  # drop the last entry of an interior row
    cols[row, 26], vals[row, 26] = row, 0.0
    top["cols"], top["vals"] = cols.reshape(-1), vals.reshape(-1)
    r = np.random.default_rng(5).standard_normal(16 ** 3)

    def use(p):
        z = np.zeros(r.size)
        p.ComputeMG(r, z)
        return [z]

    a, b = both(binding, monkeypatch, lambda: binding.Problem.optimize(levels), use)
    assert np.array_equal(a[0], b[0])
