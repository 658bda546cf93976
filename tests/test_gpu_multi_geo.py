"""The multi-system V-cycle on grid columns (form 3, the default): bitwise the
single-system V-cycle for every system, on levels in and out of the one-launch
part, ragged colour blocks, and every rounded-up system count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("dims", [(8, 8, 8), (40, 24, 56), (104, 24, 40), (64, 64, 32)])
def test_multi_systems_bitwise_single(binding, dims, nrhs):
    p = binding.Problem.generate(*dims)
    try:
        rng = np.random.default_rng(sum(dims) + nrhs)
        r = rng.standard_normal((nrhs, p.nrow))
        for _ in range(2):  # the second call may reuse captured launches
            x = np.zeros_like(r)
            p.ComputeMG_multi(r, x)
        z = np.zeros(p.nrow)
        for j in range(nrhs):
            p.ComputeMG(np.ascontiguousarray(r[j]), z)
            assert np.array_equal(x[j], z), j
    finally:
        p.free()
