"""The differentiable forward with one launch per window, at window lengths on
each side of what a thread's registers take (longer windows run one launch per
half-sweep), frames smaller than a tile, of several tiles and ragged, last
windows shorter than the others, against the differentiable oracle.

Bound 1e-6 px in float64, as for the forward elsewhere (the pyramid amplifies
rounding by about 1e7).  In float32 the two checkpoint modes, which run different
launches around the same windows, give the same bits."""
import numpy as np
import pytest
import torch

from test_gpu_diff import _frames, _oracle_flow, _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,h,w,its,lag", [
    (1, 9, 8, 6, 1), (2, 17, 35, 5, 2), (1, 70, 33, 9, 4), (1, 34, 67, 13, 6),
    (1, 40, 37, 15, 7), (1, 24, 52, 24, 20)])
def test_windows_match_oracle_fp64(K, h, w, its, lag):
    from pyflowreg_gb300.diff import flow

    fixed, moving, _, _ = _frames([3, 4], K, h, w)
    opts = dict(iterations=its, update_lag=lag, pixel_order="gauss_seidel")
    dev = torch.device("cuda")
    alpha = torch.tensor([1.5, 1.2], dtype=torch.float64)
    got = flow(torch.tensor(fixed, device=dev), torch.tensor(moving, device=dev), alpha,
               _plan(h, w, K, 2, torch.float64, **opts)).cpu()
    for f in range(2):
        ref = _oracle_flow(torch.tensor(fixed[f]), torch.tensor(moving[f]), alpha, K, **opts)
        assert float((got[f] - ref).abs().max()) <= 1e-6


@pytest.mark.parametrize("h,w,its,lag", [(8, 70, 7, 3), (33, 64, 12, 5), (100, 41, 50, 5), (65, 90, 9, 8)])
def test_checkpoint_modes_same_bits_fp32(h, w, its, lag):
    from pyflowreg_gb300.diff import flow

    fixed, moving, _, _ = _frames([5, 6], 1, h, w)
    dev = torch.device("cuda")
    out = []
    for ckpt in ("ticks", "sweeps"):
        f, m = (torch.tensor(a, device=dev, dtype=torch.float32, requires_grad=True) for a in (fixed, moving))
        fl = flow(f, m, torch.tensor(1.5, device=dev), _plan(h, w, 1, 2, torch.float32, iterations=its, update_lag=lag, checkpoint=ckpt))
        out.append([fl.detach(), *torch.autograd.grad(fl.square().sum(), (f, m))])
    assert torch.equal(out[0][0], out[1][0])
    assert bool(torch.isfinite(out[0][0]).all())
    for a, b in zip(out[0][1:], out[1][1:]):
        assert float((a - b).abs().max()) <= 1e-4 * float(a.abs().max())
