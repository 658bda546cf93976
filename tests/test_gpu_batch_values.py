"""A batch follows its members' matrices: values set on a member between two
batched solves are the values of the next one, FP32 V-cycle included, as in the
member's own solve; members that were left alone keep their bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [0, 1, 3])
def test_batch_after_member_values_change(binding, level):
    B = binding.Batch([(32, 32, 32), (48, 32, 16), (16, 16, 16)])
    try:
        bs = [np.random.default_rng(i).uniform(-1, 1, p.nrow) for i, p in enumerate(B.problems)]
        first = [np.zeros(p.nrow) for p in B.problems]
        B.CG_mixed(bs, first, 6, 0.0)
        for i in (0, 2):
            p = B.problems[i]
            v = np.full((p.nrow // 8**level, 27), -1.0)
            v[:, 13] = 40.0
            p.set_values(level, v)
            if level == 0:
                p.set_diagonal(np.full(p.nrow, 39.0))
        xs = [np.zeros(p.nrow) for p in B.problems]
        B.CG_mixed(bs, xs, 6, 0.0)
        assert np.array_equal(xs[1], first[1])
        for i, p in enumerate(B.problems):
            x1 = np.zeros(p.nrow)
            p.CG_mixed(bs[i], x1, 6, 0.0)
            # as for unchanged members: the same V-cycle bits, dots in another order
            assert np.max(np.abs(xs[i] - x1)) <= 1e-9 * max(np.max(np.abs(x1)), 1.0)
            assert i == 1 or not np.array_equal(xs[i], first[i])
    finally:
        B.free()
