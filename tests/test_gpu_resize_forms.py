"""The float64 path's horizontal resize in rows of shared memory (batches) against one
output per thread (single frames, and rows too long for shared memory): the same flows,
bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,K,T", [(17, 31, 2, 48), (40, 900, 1, 60), (33, 6399, 1, 54), (16, 6400, 1, 140), (64, 70, 3, 16)])
def test_batch_equals_single_frames(H, W, K, T):
    from pyflowreg_gb300 import api

    g = torch.Generator(device="cuda").manual_seed(W)
    fixed = torch.rand((H, W, K), generator=g, device="cuda")
    moving = (fixed + 0.1 * torch.rand((T, H, W, K), generator=g, device="cuda")).contiguous()
    moving[:, :H // 2] = (moving[:, :H // 2] * 8).round() / 8  # sums that end between two float32s
    p = api.make_params(K=K, alpha=(1.5, 1.5), levels=100, eta=0.8, iterations=2, update_lag=2, a_data=0.45, precision="fp64")
    flows = []
    for n, ts in ((T, [0]), (1, [0, 1, T // 2, T - 1])):
        plan = api.Plan(p, H, W, K, n)
        plan.set_reference(fixed)
        flows.append([plan.displacement(moving[t:t + n].contiguous()).clone() for t in ts])
        torch.cuda.synchronize()
        plan.close()
    for t, f in zip([0, 1, T // 2, T - 1], flows[1]):
        assert torch.equal(flows[0][0][t], f[0])
