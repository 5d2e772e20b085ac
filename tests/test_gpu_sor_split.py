"""The float64 level solver's strip kernel against the oracle: sizes at the edges
of its 32-row strips, of its clusters and of its ring, pass lengths, channel
counts and weights.  Displacements of this size lie outside the fixed-point
form's ranges, so the float64 kernel computes them.

Tolerance 1e-9 of the field's norm: float64's own rounding, amplified by the
iterations with lagged weights, moves the result by up to 1e-12."""
import numpy as np
import pytest

from test_gpu_sor_fixed import _both, _case, _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,K,its,lag", [
    (1, 9, 1, 10, 5), (31, 8, 2, 12, 5), (32, 9, 2, 11, 5), (33, 11, 1, 12, 3), (64, 12, 2, 13, 1),
    (65, 16, 3, 14, 7), (97, 33, 4, 21, 11), (200, 17, 8, 7, 2), (513, 20, 2, 9, 4), (1025, 24, 1, 6, 5)])
def test_sizes_and_passes(oracle, h, w, K, its, lag):
    got, ref = _both(oracle, _case(h, w, K, h + w, scale=3e3), (1.5, 1.2), its, lag, 0.45)
    _close(got, ref)


@pytest.mark.parametrize("H,W,K,its,lag", [(9, 70, 2, 8, 3), (70, 9, 1, 8, 5), (40, 33, 3, 9, 1)])
def test_batch_equals_single_frames(H, W, K, its, lag):
    """Strips of one frame and of a batch are split differently; the bits are the same."""
    import torch

    from pyflowreg_gb300 import api

    rng = np.random.default_rng(H + W)
    fr = torch.tensor(rng.random((40, H, W, K)), dtype=torch.float32, device="cuda")
    p = api.make_params(K=K, alpha=(1.5, 1.5), levels=100, eta=0.8, iterations=its, update_lag=lag, a_data=0.45,
                        precision="fp64")
    flows = []
    for n in (1, 40):
        plan = api.Plan(p, H, W, K, n)
        plan.set_reference(fr[0].contiguous())
        flows.append(torch.cat([plan.displacement(fr[i:i + n].contiguous()).clone() for i in range(0, 40, n)]))
        torch.cuda.synchronize()
        plan.close()
    assert torch.equal(flows[0], flows[1])
