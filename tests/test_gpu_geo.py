"""Columns taken from the grid (geo.cuh) against the stored 32-bit columns
(HPCG_B200_PACKED=0): every kernel that has both forms gives the same bits, on
sides that are even, odd and mixed, where tiles of rows straddle colour blocks,
and where a colour block is smaller than a tile or empty."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(64, 32, 16, 4), (104, 24, 40, 4), (24, 16, 8, 4), (33, 31, 29, 1), (75, 6, 13, 1), (17, 1, 9, 1),
         (2, 3, 1, 1), (130, 3, 66, 1)]


# 10: the bulk-copy phases; 11, 12: the first sweep's own kernel (1, 2 rows a thread)
@pytest.mark.parametrize("cfg", ["10", "11", "12"])
@pytest.mark.parametrize("dims", GRIDS)
def test_grid_columns_bitwise_stored_columns(binding, monkeypatch, dims, cfg):
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(sum(dims))
    r, x0 = rng.standard_normal(n), rng.standard_normal(n)
    got = []
    for packed, config in (("0", "1"), ("", cfg)):
        monkeypatch.setenv("HPCG_B200_PACKED", packed)
        monkeypatch.setenv("HPCG_B200_CONFIG", config)
        p = binding.Problem.generate(*dims[:3], nlevels=dims[3])
        try:
            y, z, z32, x = np.zeros(n), np.zeros(n), np.zeros(n), x0.copy()
            p.ComputeSPMV(x0, y)
            for _ in range(2):  # launch by launch, then as one graph
                p.ComputeMG(r, z)
                p.ComputeMG_f32(r, z32)
                x[:] = x0
                p.ComputeSYMGS(r, x)
                got.append((packed, y.copy(), z.copy(), z32.copy(), x.copy()))
        finally:
            p.free()
    for other in got[1:]:
        for a, b in zip(got[0][1:], other[1:]):
            assert np.array_equal(a, b), other[0]


@pytest.mark.parametrize("dims", [(48, 40, 32), (64, 64, 64)])
def test_cg_on_grid_columns(binding, monkeypatch, dims):
    """CG with the fused p'Ap and r'z sums: within rounding of the stored columns'."""
    n = int(np.prod(dims))
    b = np.random.default_rng(1).uniform(-1, 1, n)
    got = []
    for packed in ("0", ""):
        monkeypatch.setenv("HPCG_B200_PACKED", packed)
        p = binding.Problem.generate(*dims)
        try:
            x = np.zeros(n)
            got.append((p.CG(b, x, 10, 0.0), x))
        finally:
            p.free()
    (a, x), (c, y) = got
    assert abs(a[1] / a[2] - c[1] / c[2]) <= 1e-10
    assert np.max(np.abs(x - y)) <= 1e-10 * np.max(np.abs(x))
