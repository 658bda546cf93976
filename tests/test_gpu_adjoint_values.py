"""The gradient values of the adjoint, bit for bit: -(lambda_i x_j) of the lambda
that the same call returned, 0 where a direction leaves the grid; with the values
written over x or over lambda's own array as they are without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(16, 24, 8), (40, 8, 16)]


def expected(dims, lam, x):
    nx, ny, nz = dims
    pad = np.zeros((nz + 2, ny + 2, nx + 2))
    pad[1:-1, 1:-1, 1:-1] = x.reshape(nz, ny, nx)
    out = np.zeros((nz, ny, nx, 27))
    inside = np.zeros_like(pad, bool)
    inside[1:-1, 1:-1, 1:-1] = True
    for k in range(27):
        cut = tuple(slice(o, o + n) for o, n in ((k // 9, nz), (k // 3 % 3, ny), (k % 3, nx)))
        out[..., k] = np.where(inside[cut], -(lam.reshape(nz, ny, nx) * pad[cut]), 0.0)
    return out.ravel()


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("packed", ["0", ""])
@pytest.mark.parametrize("where", ["host", "device", "over x", "over lambda"])
def test_gradient_values_bits(binding, monkeypatch, dims, packed, where):
    import torch
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    x, g = rng.standard_normal(n), rng.standard_normal(n)
    monkeypatch.setenv("HPCG_B200_PACKED", packed)
    p = binding.Problem.generate(*dims)
    try:
        lam, vals = np.zeros(n), np.full(27 * n, np.nan)
        p.adjoint(x, g, 3, 0.0, lam, vals)  # lambda, from host vectors
        if where != "host":
            gd = torch.from_numpy(g).cuda()
            vd = torch.full((27 * n,), float("nan"), dtype=torch.float64, device="cuda")
            xd, ld = torch.from_numpy(x).cuda(), torch.zeros(n, dtype=torch.float64, device="cuda")
            if where == "over x":
                xd = vd[5 * n + 3:6 * n + 3].copy_(xd)
            elif where == "over lambda":
                ld = vd[11 * n + 1:12 * n + 1]
            p.adjoint(xd, gd, 3, 0.0, ld, vd)
            vals = vd.cpu().numpy()
            if where == "device" or where == "over x":
                assert np.array_equal(ld.cpu().numpy(), lam)
    finally:
        p.free()
    assert np.array_equal(vals, expected(dims, lam, x))
