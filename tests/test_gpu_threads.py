"""One host thread per problem: threads that make, use and free problems of their own
on one GPU at the same time, each capturing its V-cycles and steps while the others
launch and wait, get the bits that each gets alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def work(binding, dims, repeats):
    import torch
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    r, x0 = (torch.from_numpy(rng.standard_normal(n)).cuda() for _ in range(2))
    out = []
    for _ in range(repeats):
        p = binding.Problem.generate(*dims)
        try:
            for _ in range(3):  # launch by launch, captured, from the graph
                y, z, z32, x = torch.zeros_like(r), torch.zeros_like(r), torch.zeros_like(r), x0.clone()
                p.ComputeSYMGS(r, x)
                p.ComputeMG(r, z)
                p.ComputeMG_f32(r, z32)
                p.ComputeSPMV(x0, y)
                out.append(torch.stack([x, z, z32, y]).cpu().numpy())
        finally:
            p.free()
    return out


def test_threads_with_problems_of_their_own(binding):
    grids = [(64, 48, 32), (16, 16, 16), (40, 24, 56), (48, 32, 24)]
    alone = [work(binding, d, 1)[0] for d in grids]
    got, errors = [None] * len(grids), []

    def run(i):
        try:
            got[i] = work(binding, grids[i], 8)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(grids))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for i, outs in enumerate(got):
        for o in outs:
            assert np.array_equal(o, alone[i]), grids[i]
