"""|w| of the flow statistics, element by element: frames of one pixel, whose mean and
largest magnitude are the pixel's own.  u^2 + v^2 is exact but for one rounding in
float64 and the square root is correctly rounded, so numpy's bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _norms(w):
    from pyflowreg_gb300.prep import flow_statistics_device

    out = []
    for i in range(0, len(w), 60000):
        t = torch.tensor(w[i:i + 60000], device="cuda").view(-1, 1, 1, 2)
        out.append(flow_statistics_device(t)[1].cpu().numpy()[:, :2])
    return np.concatenate(out)


@pytest.mark.parametrize("kind", ["flows", "exponents", "squares", "middles", "edges"])
def test_every_magnitude_is_correctly_rounded(kind):
    rng = np.random.default_rng(len(kind))
    n = 240000
    if kind == "flows":
        w = rng.normal(0, 3, (n, 2))
    elif kind == "exponents":
        w = rng.uniform(1, 2, (n, 2)) * 2.0 ** rng.integers(-126, 127, (n, 2))
    elif kind == "squares":
        w = np.stack([rng.integers(1, 1 << 24, n), np.zeros(n)], 1).astype(np.float64)
        m, q = rng.integers(1, 3000, (2, n // 2))
        w[::2] = np.stack([abs(m * m - q * q), 2 * m * q], 1)  # Pythagorean
    elif kind == "middles":
        # roots just beside a power of two and beside the middle between two doubles
        w = np.stack([2.0 ** rng.integers(-40, 40, n), rng.integers(1, 400, n) * 2.0 ** rng.integers(-30, 12, n)], 1)
    else:
        tiny = np.float32(1e-45) * rng.integers(0, 50, (n, 2))
        w = np.where(rng.random((n, 2)) < 0.5, tiny, np.float32(3.4e38) * rng.random((n, 2)))
    w = (w * rng.choice([-1, 1], (n, 2))).astype(np.float32)
    got = _norms(w)
    d = w.astype(np.float64)
    want = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1])
    assert np.array_equal(got[:, 0], want)
    assert np.array_equal(got[:, 1], want)


def test_masks_beyond_the_float32_integers():
    """Columns over 2^24, where x and W - x are no float32s: x + u >= 0 and x + u < W in float64."""
    from pyflowreg_gb300.prep import flow_statistics_device

    n = (1 << 24) + 4099
    x = np.arange(n, dtype=np.float64)
    rng = np.random.default_rng(5)
    w = np.zeros((n, 2), dtype=np.float32)
    # onto the borders and a float32 to either side of them
    u = np.where(rng.random(n) < 0.5, -x, n - x).astype(np.float32)
    step = rng.integers(-1, 2, n)
    w[:, 0] = np.where(step == 0, u, np.nextafter(u, np.where(step < 0, -np.inf, np.inf).astype(np.float32)))
    m = x + w[:, 0].astype(np.float64)
    want = np.where((m >= 0) & (m < n), 255, 0).astype(np.uint8)
    valid = flow_statistics_device(torch.tensor(w, device="cuda").view(1, 1, n, 2))[0]
    assert np.array_equal(valid.cpu().numpy().reshape(-1), want)
