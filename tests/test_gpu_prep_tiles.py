"""Preprocessing tiles and the flow statistics at their edges, against the
numpy/scipy restatement: frames smaller than the halo, partial tiles, several
radii and storage types, halos too large for a tile (the two-kernel form);
statistics of flows one to three pixels wide, off 8-byte alignment, with NaN and
infinities."""
import numpy as np
import pytest
import torch

from oracle import prep_oracle as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(1, 1), (2, 40), (33, 3), (32, 64), (31, 65)])
@pytest.mark.parametrize("K,norm,sigma,dtype", [
    (1, "together", ((0.0, 0.0, 0.1),), np.float32),
    (2, "together", ((1.0, 1.0, 0.1),), np.float32),
    (3, "together", ((0.5, 2.0, 0.1), (3.0, 0.0, 0.1), (1.0, 1.5, 0.1)), np.float32),
    (2, "separate", ((1.0, 1.5, 0.1), (2.0, 1.0, 0.1)), np.float32),
    (1, "together", ((1.0, 1.0, 0.1),), np.uint16),
    (1, "together", ((4.0, 12.0, 0.1),), np.float32),
])
def test_tiles_bit_exact(H, W, K, norm, sigma, dtype):
    from pyflowreg_gb300.prep import preprocess_device

    rng = np.random.default_rng(H * W + K)
    raw = rng.gamma(2.0, 300.0, (2, H, W, K))
    raw[0].reshape(-1)[::3] = 512.0  # equal neighbours: sums that end between two float32s
    raw = raw.round().astype(dtype) if dtype == np.uint16 else raw.astype(dtype)
    ref = raw.mean(0)
    if H * W == 1:
        ref = np.concatenate([ref, ref + 3], 0)
    sig = np.asarray(sigma, dtype=np.float64)
    sig = sig[0] if sig.shape[0] == 1 else sig
    want = P.preprocess(raw, ref, sig, norm).astype(np.float32)
    got = preprocess_device(torch.tensor(raw.astype(np.float32), device="cuda"), ref, sig, norm, frames_dtype=raw.dtype)
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("H,W", [(1, 1), (1, 5), (2, 2), (3, 3), (2, 300), (17, 4), (40, 257)])
@pytest.mark.parametrize("special", [None, np.nan, np.inf, -np.inf, 1e-30])
@pytest.mark.parametrize("off", [0, 1])
def test_statistics_at_the_edges(H, W, special, off):
    from pyflowreg_gb300.prep import flow_statistics_device

    rng = np.random.default_rng(H * 7 + W)
    w = (rng.standard_normal((4, H, W, 2)) * 3).astype(np.float32)
    w[1] = np.round(w[1])
    if special is not None:
        for i, q in enumerate((0, w[0].size // 2, w[0].size - 1)):
            w[i].reshape(-1)[q] = special
    buf = torch.empty(w.size + 1, dtype=torch.float32, device="cuda")
    view = buf[off:off + w.size].view(w.shape)
    view.copy_(torch.tensor(w))
    valid, stats = flow_statistics_device(view)
    np.testing.assert_array_equal(valid.cpu().numpy(), P.valid_masks(w))
    with np.errstate(all="ignore"):
        want = P.statistics(w.astype(np.float64)) if min(H, W) > 1 else None
    got = stats.cpu().numpy()
    if want is None:  # np.gradient wants two samples
        mag = np.sqrt((w.astype(np.float64) ** 2).sum(-1)).reshape(4, -1)
        np.testing.assert_allclose(got[:, 0], mag.mean(1), rtol=1e-9, atol=1e-9)
        return
    want = np.asarray(want)
    # the maximum passes NaN over, as the kernel's fmax always has
    cols = [0, 2, 3] if special is not None and np.isnan(special) else [0, 1, 2, 3]
    np.testing.assert_allclose(got[:, cols], want[:, cols], rtol=1e-9, atol=1e-9)
