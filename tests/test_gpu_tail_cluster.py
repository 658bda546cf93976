"""The small levels where the GPU holds only small clusters (HPCG_B200_TAIL_CLUSTER):
levels that ask for larger ones are launched phase by phase, single, several systems
and batched, with the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(binding, dims):
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    r, x0 = rng.standard_normal((3, n)), rng.standard_normal(n)
    out = []
    p = binding.Problem.generate(*dims)
    try:
        for _ in range(2):
            z, z32, x, zm = np.zeros(n), np.zeros(n), x0.copy(), np.zeros_like(r)
            p.ComputeMG(r[0], z)
            p.ComputeMG_f32(r[0], z32)
            p.ComputeSYMGS(r[0], x)
            p.ComputeMG_multi(r, zm)
            out += [z, z32, x, zm]
    finally:
        p.free()
    B = binding.Batch([dims, (16, 16, 16)] if all(d % 16 == 0 for d in dims) else [(16, 48, 32)])
    try:
        bs = [np.random.default_rng(i).uniform(-1, 1, q.nrow) for i, q in enumerate(B.problems)]
        xs = [np.zeros(q.nrow) for q in B.problems]
        out += [np.concatenate([np.asarray(v, float) for v in B.CG_mixed(bs, xs, 4, 0.0)])] + xs
    finally:
        B.free()
    return out


@pytest.mark.parametrize("limit", ["1", "4", "8", "0"])
@pytest.mark.parametrize("dims", [(32, 32, 32), (40, 24, 72)])
def test_smaller_clusters_bitwise(binding, monkeypatch, dims, limit):
    want = run(binding, dims)
    monkeypatch.setenv("HPCG_B200_TAIL_CLUSTER", limit)
    for a, b in zip(want, run(binding, dims)):
        assert np.array_equal(a, b)
