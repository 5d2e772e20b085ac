"""Sums kept as float32 pairs whose products underflow: the float64 sum's result."""
import numpy as np
import pytest
import torch

from oracle import prep_oracle as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.0, 0.5, 1.0, 2.0])
@pytest.mark.parametrize("x", [3e-36, 1.4e-35, 4e-35, 1e-34, -1.4e-35])
def test_preprocessing_of_subnormal_samples(x, sigma):
    """Samples of 0 to 7e-45 after normalising by 1e10: bit-exact with scipy."""
    from pyflowreg_gb300.prep import preprocess_device

    rng = np.random.default_rng(3)
    raw = np.zeros((2, 45, 40, 1), dtype=np.float32)
    raw[0] = x
    raw[1, 10:30, 5:25] = x * rng.integers(0, 5, (20, 20, 1))
    ref = np.zeros((45, 40, 1), dtype=np.float32)
    ref[0, 0] = 1e10
    sig = np.array([sigma, sigma, 0.1])
    want = P.preprocess(raw, ref, sig, "together").astype(np.float32)
    got = preprocess_device(torch.tensor(raw, device="cuda"), ref, sig, "together", frames_dtype=raw.dtype).cpu().numpy()
    assert np.array_equal(got, want)
