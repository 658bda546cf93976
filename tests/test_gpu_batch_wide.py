"""A batch whose level 3 is launched phase by phase because one member's is too wide
for the one-launch small levels: colours of that level share sectors. Every solve
gives the bits of the register kernels (HPCG_B200_BATCH_BULK=0), whose arithmetic and
order of sums it has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(592, 592, 16), (48, 48, 48), (16, 48, 80)]


def test_launched_level_with_shared_sectors(binding, monkeypatch):
    got = []
    for bulk, repeats in (("0", 1), ("1", 8)):
        monkeypatch.setenv("HPCG_B200_BATCH_BULK", bulk)
        B = binding.Batch(DIMS)
        try:
            bs = [np.random.default_rng(i).uniform(-1, 1, p.nrow) for i, p in enumerate(B.problems)]
            for _ in range(repeats):
                xs = [np.zeros(p.nrow) for p in B.problems]
                res = B.CG_mixed(bs, xs, 5, 0.0)
                got.append((xs, res))
        finally:
            B.free()
    for xs, res in got[1:]:
        for a, b in zip(xs, got[0][0]):
            assert np.array_equal(a, b)
        assert np.array_equal(np.asarray(res), np.asarray(got[0][1]))
