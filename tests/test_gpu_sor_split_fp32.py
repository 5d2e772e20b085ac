"""The float32 chained solver (strips of 32 rows, one warp per pipelined iteration)
against the rows-in-registers solver of one launch per pass: the same bits, at sizes
on the edges of strips and clusters, with every channel count, pass lengths from one
iteration to eleven, and batches beside single frames."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,K,T,its,lag", [
    (9, 40, 1, 1, 7, 5), (31, 33, 2, 3, 12, 5), (33, 16, 3, 2, 11, 3), (65, 20, 4, 1, 9, 1), (97, 50, 2, 40, 14, 7),
    (512, 24, 1, 2, 8, 5), (530, 20, 2, 1, 13, 11), (1060, 18, 1, 1, 6, 2), (2040, 12, 2, 1, 5, 5), (2080, 12, 2, 1, 6, 5)])
def test_same_bits_as_one_launch_per_pass(H, W, K, T, its, lag):
    from pyflowreg_gb300 import api

    rng = np.random.default_rng(H + K)
    base = np.kron(rng.random((H // 4 + 2, W // 4 + 2, K)), np.ones((4, 4, 1)))[:H + 1, :W + 1]
    fixed = torch.tensor(base[:H, :W], dtype=torch.float32, device="cuda")
    moving = torch.tensor(base[1:, 1:][None] + 0.01 * rng.random((T, H, W, K)), dtype=torch.float32, device="cuda")
    plan = api.Plan(api.make_params(K=K, alpha=(1.5, 1.2), levels=100, eta=0.8, iterations=its, update_lag=lag,
                                    a_data=0.45, precision="fp32"), H, W, K, T)
    plan.set_reference(fixed.contiguous())
    n = len(plan.level_tuning())
    out = {}
    for variant in (2, 1):
        for i in range(n):
            try:
                plan.set_level_variant(i, variant)
            except ValueError:  # a level narrower than three columns
                pass
        out[variant] = plan.displacement(moving.contiguous()).clone()
        torch.cuda.synchronize()
    assert bool(torch.isfinite(out[2]).all())
    assert torch.equal(out[1], out[2])
    plan.close()
