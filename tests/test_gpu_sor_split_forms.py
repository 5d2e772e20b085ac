"""The float64 strip kernel's forms against one another: single frames (one CTA per SM),
batches over the SMs (two CTAs per SM, 32 or 64 rows by how the clusters pack), levels
over 512 rows in both their forms, and the strip heights that a caller may ask for.  The
same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _flows(p, H, W, K, fixed, moving, n, rows=0):
    from pyflowreg_gb300 import api

    plan = api.Plan(p, H, W, K, n)
    plan.set_reference(fixed)
    if rows:
        for i in range(len(plan.level_tuning())):
            try:
                plan.set_level_tuning(i, 0, rows)
            except ValueError:  # a level that takes no such height
                pass
    out = torch.cat([plan.displacement(moving[i:i + n].contiguous()).clone() for i in range(0, len(moving), n)])
    torch.cuda.synchronize()
    plan.close()
    return out


@pytest.mark.parametrize("H,W,K,T,its,lag", [
    (200, 12, 1, 40, 8, 3), (330, 12, 2, 40, 7, 5), (330, 9, 4, 25, 6, 5), (500, 10, 3, 24, 6, 2), (610, 10, 2, 20, 6, 5),
    (700, 8, 1, 6, 6, 5), (1100, 9, 2, 3, 5, 5)])
def test_batch_equals_single_frames(H, W, K, T, its, lag):
    from pyflowreg_gb300 import api

    g = torch.Generator(device="cuda").manual_seed(H)
    fixed = torch.rand((H, W, K), generator=g, device="cuda")
    moving = (fixed + 0.1 * torch.rand((T, H, W, K), generator=g, device="cuda")).contiguous()
    p = api.make_params(K=K, alpha=(1.5, 1.5), levels=100, eta=0.8, iterations=its, update_lag=lag, a_data=0.45,
                        precision="fp64")
    one = _flows(p, H, W, K, fixed, moving, 1)
    assert bool(torch.isfinite(one).all())
    assert torch.equal(one, _flows(p, H, W, K, fixed, moving, T))
    for rows in (64, 128, 256):
        assert torch.equal(one[:2], _flows(p, H, W, K, fixed, moving[:2], 2, rows))
