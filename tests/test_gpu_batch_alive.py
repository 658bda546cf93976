"""Batches alive at the same time: one whose small levels take much shared memory,
made before batches whose small levels take little or are launched phase by phase,
solved for the first time after them, in either order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(B):
    bs = [np.random.default_rng(p.nrow).uniform(-1, 1, p.nrow) for p in B.problems]
    xs = [np.zeros(p.nrow) for p in B.problems]
    B.CG_mixed(bs, xs, 4, 0.0)
    return xs


@pytest.mark.parametrize("later", [(16, 16, 16), (128, 128, 128), (656, 656, 16)])
@pytest.mark.parametrize("first", [True, False])
def test_batches_side_by_side(binding, later, first):
    dims = [(96, 96, 96)], [later]
    alone = []
    for d in dims:
        B = binding.Batch(d)
        alone.append(solve(B))
        B.free()
    live = [binding.Batch(d) for d in dims]
    try:
        for i in (0, 1) if first else (1, 0):
            for x, y in zip(solve(live[i]), alone[i]):
                assert np.array_equal(x, y)
    finally:
        for B in live:
            B.free()


def test_batches_one_after_another(binding, monkeypatch):
    """Batches whose matrices (and their tensor maps) take the memory that a freed
    batch of other grids gave back: the register kernels' bits, which use no maps."""
    lists = [[(64, 32, 48), (32, 32, 32)], [(32, 48, 64), (48, 16, 32)], [(16, 16, 16)], [(64, 32, 48), (32, 32, 32)]]
    got = {}
    for bulk in ("0", "1"):
        monkeypatch.setenv("HPCG_B200_BATCH_BULK", bulk)
        got[bulk] = []
        for dims in lists:
            B = binding.Batch(dims)
            try:
                got[bulk].append(solve(B))
            finally:
                B.free()
    for a, b in zip(got["0"], got["1"]):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
