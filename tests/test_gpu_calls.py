"""The calls' own kernels on device vectors: SpMV in place on natural-order
vectors, the lone reductions, the gradient values, each against the path host
vectors or stored columns take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cuda(a):
    import torch
    return torch.from_numpy(a).cuda()


@pytest.mark.parametrize("dims", [(16, 16, 16), (33, 31, 29), (75, 6, 13), (1, 1, 1), (2, 3, 1), (257, 3, 2), (64, 64, 64)])
def test_spmv_in_place_bitwise_host_vectors(binding, dims):
    p = binding.Problem.generate(*dims, nlevels=1)
    try:
        rng = np.random.default_rng(sum(dims))
        x = rng.standard_normal(p.nrow)
        p.set_values(0, rng.standard_normal((p.nrow, 27)))
        y = np.zeros(p.nrow)
        p.ComputeSPMV(x, y)
        xd, yd = cuda(x), cuda(np.full(p.nrow, np.nan))
        p.ComputeSPMV(xd, yd)
        assert np.array_equal(yd.cpu().numpy(), y)
        p.ComputeSPMV(xd, xd)  # onto itself: as if from a copy
        assert np.array_equal(xd.cpu().numpy(), y)
    finally:
        p.free()


@pytest.mark.parametrize("n", [1, 31, 255, 257, 4097, 303105, 1000003])
def test_lone_reductions(binding, n):
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(n), rng.standard_normal(n)
    ref = float(np.sum(x.astype(np.longdouble) * y.astype(np.longdouble)))
    bound = 4 * np.finfo(float).eps * float(np.sum(np.abs(x * y))) * np.log2(n + 2)  # a tree of log2 n roundings
    xd, yd = cuda(x), cuda(y)
    for _ in range(3):
        d = binding.ComputeDotProduct(n, xd, yd)
        assert d == binding.ComputeDotProduct(n, x, y) and abs(d - ref) <= bound
        assert binding.ComputeResidual(n, xd, yd) == np.max(np.abs(x - y))


@pytest.mark.parametrize("dims", [(16, 24, 8), (40, 8, 16)])
def test_gradient_values_bitwise_stored_columns(binding, monkeypatch, dims):
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    x, g = rng.standard_normal(n), rng.standard_normal(n)
    got = []
    for packed, dev in (("0", False), ("", False), ("", True)):
        monkeypatch.setenv("HPCG_B200_PACKED", packed)
        monkeypatch.setenv("HPCG_B200_CONFIG", "1")
        p = binding.Problem.generate(*dims)
        try:
            gb, gv = np.zeros(n), np.full(27 * n, np.nan)
            if dev:
                gbd, gvd = cuda(gb), cuda(gv)
                p.adjoint(cuda(x), cuda(g), 3, 0.0, gbd, gvd)
                gb, gv = gbd.cpu().numpy(), gvd.cpu().numpy()
            else:
                p.adjoint(x, g, 3, 0.0, gb, gv)
            got.append((gb, gv))
        finally:
            p.free()
    for gb, gv in got[1:]:
        assert np.max(np.abs(gb - got[0][0])) <= 1e-12 * np.max(np.abs(gb))
        assert np.max(np.abs(gv - got[0][1])) <= 1e-12 * np.max(np.abs(gv))
        assert np.array_equal(gv == 0.0, got[0][1] == 0.0)
