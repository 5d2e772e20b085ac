"""Float32 batches on both sides of the line between k_sor_split and k_sor_chain: the
same bits as one launch per pass, and as the frames one by one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,K,T,its,lag", [
    (20, 12, 1, 1200, 8, 5), (20, 12, 2, 2432, 8, 5), (64, 9, 2, 1216, 7, 3), (40, 3, 1, 1216, 6, 1),
    (200, 10, 3, 300, 11, 11), (410, 8, 2, 152, 8, 5), (512, 8, 3, 152, 6, 4), (512, 7, 4, 160, 6, 5),
    (512, 8, 1, 305, 6, 2), (900, 8, 2, 60, 6, 5), (1300, 8, 2, 30, 7, 3), (2040, 7, 1, 28, 6, 11)])
def test_same_bits_on_both_sides(H, W, K, T, its, lag):
    from pyflowreg_gb300 import api

    rng = np.random.default_rng(H + K)
    base = np.kron(rng.random((H // 4 + 2, W // 4 + 2, K)), np.ones((4, 4, 1)))[:H + 1, :W + 1]
    fixed = torch.tensor(base[:H, :W], dtype=torch.float32, device="cuda").contiguous()
    g = torch.Generator(device="cuda").manual_seed(H)
    moving = torch.tensor(base[1:, 1:], dtype=torch.float32, device="cuda")[None] + 0.01 * torch.rand(
        (T, H, W, K), generator=g, device="cuda")
    p = api.make_params(K=K, alpha=(1.5, 1.2), levels=100, eta=0.8, iterations=its, update_lag=lag, a_data=0.45,
                        precision="fp32")
    plan = api.Plan(p, H, W, K, T)
    plan.set_reference(fixed)
    out = {}
    for variant in (2, 1):
        for i in range(len(plan.level_tuning())):
            try:
                plan.set_level_variant(i, variant)
            except ValueError:  # a level narrower than three columns
                pass
        out[variant] = plan.displacement(moving.contiguous()).clone()
        torch.cuda.synchronize()
    plan.close()
    assert bool(torch.isfinite(out[2]).all())
    assert torch.equal(out[1], out[2])
    one = api.Plan(p, H, W, K, 1)
    one.set_reference(fixed)
    for t in (0, T // 2, T - 1):
        assert torch.equal(one.displacement(moving[t:t + 1].contiguous())[0], out[2][t])
    torch.cuda.synchronize()
    one.close()
