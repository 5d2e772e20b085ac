"""The compensation warp's form for 1 to 4 interleaved channels against the
general form (which takes 5 and more): the same bits for every channel, whatever
the tensors' alignment, with displacements out of the frame, infinite and NaN."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _at_offset(a, off):
    buf = torch.empty(a.numel() + 4, dtype=torch.float32, device="cuda")
    view = buf[off:off + a.numel()].view(a.shape)
    view.copy_(a)
    return view


@pytest.mark.parametrize("method", ["cubic", "linear"])
@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("H,W,off", [(1, 1, 0), (3, 33, 0), (9, 31, 1), (40, 64, 2), (17, 70, 3)])
def test_same_bits_as_the_general_form(method, K, H, W, off):
    from pyflowreg_gb300.api import imregister_device

    rng = np.random.default_rng(K * 100 + W)
    T = 3
    fr = torch.tensor(rng.standard_normal((T, H, W, 6)), dtype=torch.float32, device="cuda")
    ref = torch.tensor(rng.standard_normal((H, W, 6)), dtype=torch.float32, device="cuda")
    fl = rng.standard_normal((T, H, W, 2)).astype(np.float32) * 5
    fl.reshape(-1)[::37] = np.round(fl.reshape(-1)[::37])
    fl.reshape(-1)[5::53] = np.nan
    fl.reshape(-1)[7::91] = np.inf
    fl = torch.tensor(fl, device="cuda")
    want = imregister_device(fr, fl, ref, method)[..., :K]
    got = imregister_device(_at_offset(fr[..., :K], off), _at_offset(fl, off), _at_offset(ref[..., :K], off), method,
                            out_t=_at_offset(torch.zeros_like(want), off))
    assert torch.equal(got.contiguous().view(torch.int32), want.contiguous().view(torch.int32))
