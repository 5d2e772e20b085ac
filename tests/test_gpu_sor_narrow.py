"""Levels of three to seven columns: the shortest rows that the split chained solvers
take, where the fold's lead over the update is the row itself.

Float64 against the oracle: 1e-9 of the field's norm for a level (float64's own
rounding, amplified by the iterations with lagged weights, is below 1e-12), 1e-3 px
for a whole flow.  Float32 against the one-launch-per-pass solver: the same bits."""
import numpy as np
import pytest
import torch

from test_gpu_sor_fixed import _both, _case, _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [3, 4, 5, 6, 7])
@pytest.mark.parametrize("h,K,scale", [(1, 1, 1.0), (33, 2, 1.0), (70, 3, 3e3), (530, 1, 3e3), (1030, 2, 3e3)])
def test_level(oracle, w, h, K, scale):
    got, ref = _both(oracle, _case(h, w, K, h + w, scale), (1.5, 1.2), 15, 5, 0.45)
    _close(got, ref)


def _frames(H, W, K, T, seed):
    rng = np.random.default_rng(seed)
    base = np.kron(rng.random((H // 4 + 2, W // 4 + 2, K)), np.ones((4, 4, 1)))[:H + 1, :W + 1]
    fixed = torch.tensor(base[:H, :W], dtype=torch.float32, device="cuda")
    moving = torch.tensor(base[1:, 1:][None] + 0.01 * rng.random((T, H, W, K)), dtype=torch.float32, device="cuda")
    return fixed.contiguous(), moving.contiguous()


@pytest.mark.parametrize("H,W", [(40, 3), (40, 4), (70, 5), (33, 7)])
def test_flow_fp64(oracle, H, W):
    from pyflowreg_gb300 import api

    fixed, moving = _frames(H, W, 1, 2, H + W)
    kw = dict(alpha=(1.5, 1.5), iterations=20, update_lag=5, levels=100, eta=0.8)
    got = api.get_displacement_device(fixed, moving, precision="fp64", **kw).cpu().numpy()
    for t in range(2):
        ref = oracle.get_displacement(fixed[..., 0].cpu().numpy(), moving[t, ..., 0].cpu().numpy(), **kw)
        assert np.abs(got[t] - ref).max() <= 1e-3


@pytest.mark.parametrize("H,W,K,T", [(40, 3, 1, 3), (70, 4, 2, 2), (33, 5, 3, 2), (530, 7, 2, 1)])
def test_flow_fp32_same_bits(H, W, K, T):
    from pyflowreg_gb300 import api

    fixed, moving = _frames(H, W, K, T, H + W)
    plan = api.Plan(api.make_params(K=K, alpha=(1.5, 1.2), levels=100, eta=0.8, iterations=15, update_lag=5,
                                    a_data=0.45, precision="fp32"), H, W, K, T)
    plan.set_reference(fixed)
    out = {}
    for variant in (2, 1):
        for i in range(len(plan.level_tuning())):
            try:
                plan.set_level_variant(i, variant)
            except ValueError:  # a level narrower than three columns
                pass
        out[variant] = plan.displacement(moving).clone()
        torch.cuda.synchronize()
    plan.close()
    assert bool(torch.isfinite(out[2]).all())
    assert torch.equal(out[1], out[2])


@pytest.mark.parametrize("w", [3, 4, 5, 6])
@pytest.mark.parametrize("lag", [1, 2, 3, 6, 11])
@pytest.mark.parametrize("scale", [1.0, 3e3])
def test_level_short_passes(oracle, w, lag, scale):
    got, ref = _both(oracle, _case(37, w, 2, w + lag, scale), (1.5, 1.2), 23, lag, 0.45)
    _close(got, ref)


@pytest.mark.parametrize("W,lag", [(3, 1), (4, 1), (5, 2)])
def test_flow_short_passes(oracle, W, lag):
    from pyflowreg_gb300 import api

    fixed, moving = _frames(45, W, 1, 1, W + lag)
    kw = dict(alpha=(1.5, 1.5), iterations=20, update_lag=lag, levels=100, eta=0.8)
    got = api.get_displacement_device(fixed, moving, precision="fp64", **kw).cpu().numpy()
    ref = oracle.get_displacement(fixed[..., 0].cpu().numpy(), moving[0, ..., 0].cpu().numpy(), **kw)
    assert np.abs(got[0] - ref).max() <= 1e-3
