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
