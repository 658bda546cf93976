"""A lone SpMV on device vectors makes the level's choice of configuration, as its
first use, and runs the configuration that the environment names."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,spmv", [(None, 7), ("1", 1), ("6", 6)])
def test_spmv_call_makes_the_choice(binding, monkeypatch, config, spmv):
    import torch
    if config:
        monkeypatch.setenv("HPCG_B200_CONFIG", config)
    p = binding.Problem.generate(24, 16, 8)
    try:
        assert p.level_config(0)["tuned"] == 0
        x = np.random.default_rng(0).standard_normal(p.nrow)
        xd, yd = torch.from_numpy(x).cuda(), torch.zeros(p.nrow, dtype=torch.float64, device="cuda")
        p.ComputeSPMV(xd, yd)
        c = p.level_config(0)
        assert c["tuned"] == 1 and c["spmv"] == spmv
        y = np.zeros(p.nrow)
        p.ComputeSPMV(x, y)
        assert np.array_equal(yd.cpu().numpy(), y)
    finally:
        p.free()
