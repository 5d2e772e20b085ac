"""The fixed-point form of the float64 level solver against the oracle: sizes at
the edges of its row strips and of its ring, pass lengths, channel counts, both
smoothness weights, and displacements outside its number formats (which the
second launch or the float64 kernel computes).

Tolerance 1e-9 of the field's norm: float64's own rounding, amplified by 50
iterations with lagged weights, moves the result by up to 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(h, w, K, seed, scale=1.0, uv=1.0):
    rng = np.random.default_rng(seed)
    shape = (h + 2, w + 2, K)
    # rank-two positive semidefinite tensors, as gradient constancy gives
    g = rng.standard_normal((2, 2) + shape)
    g /= np.sqrt((g ** 2).sum(1, keepdims=True)) + 0.05 * rng.random((2, 1) + shape)
    t = scale * rng.standard_normal((2,) + shape)
    x, y = g[:, 0], g[:, 1]
    J = [(x * x).sum(0), (y * y).sum(0), (t * t).sum(0), (x * y).sum(0), (x * t).sum(0), (y * t).sum(0)]
    wgt = rng.random(shape) / K
    u, v = uv * rng.standard_normal((2, h + 2, w + 2))
    return J, wgt, u, v


def _both(oracle, case, alpha, its, lag, a_data):
    import pyflowreg_gb300 as G

    J, wgt, u, v = case
    K = wgt.shape[2]
    ad = np.full(K, a_data) if np.isscalar(a_data) else np.asarray(a_data)
    got = G.level_solver(*J, wgt, u, v, alpha, its, lag, 0, ad, 1.0, 1.0, 1.0)
    ref = oracle.compute_flow(*J, wgt, u, v, alpha[0], alpha[1], its, lag, ad, 1.0, 1.0, 1.0)
    return got, (ref[..., 0], ref[..., 1])


def _close(got, ref):
    for g, r in zip(got, ref):
        assert np.linalg.norm(g - r) <= 1e-9 * np.linalg.norm(r)


@pytest.mark.parametrize("h,w,K,its,lag", [
    (1, 9, 1, 10, 5), (31, 8, 2, 12, 5), (32, 9, 2, 12, 5), (33, 11, 1, 12, 3), (64, 12, 2, 23, 1),
    (65, 16, 3, 14, 7), (97, 33, 4, 30, 11), (513, 20, 2, 9, 4), (700, 24, 1, 6, 5)])
def test_sizes_and_passes(oracle, h, w, K, its, lag):
    got, ref = _both(oracle, _case(h, w, K, h + w), (1.5, 1.5), its, lag, 0.45)
    _close(got, ref)


@pytest.mark.parametrize("alpha,a_data", [((2.0, 0.7), 0.45), ((0.05, 0.05), 0.45), ((1.5, 1.5), [1.0, 0.45]),
                                          ((1.5, 1.5), [1.7, 2.5])])
def test_weights_and_exponents(oracle, alpha, a_data):
    got, ref = _both(oracle, _case(40, 37, 2, 5), alpha, 20, 5, a_data)
    _close(got, ref)


@pytest.mark.parametrize("scale,uv", [(0.0, 0.0), (1e-9, 0.0), (1e-3, 0.0), (30.0, 0.0), (3e3, 0.0), (1.0, 1e4)])
def test_displacements_outside_the_formats(oracle, scale, uv):
    got, ref = _both(oracle, _case(45, 50, 2, 9, scale, uv), (1.5, 1.5), 15, 5, 0.45)
    if scale == 0.0:
        assert all(np.array_equal(r, np.zeros_like(r)) for r in ref)
        assert all(np.array_equal(g, r) for g, r in zip(got, ref))
    else:
        _close(got, ref)


def test_not_a_number_reaches_the_result(oracle):
    case = _case(40, 30, 1, 3)
    case[0][4][20, 15, 0] = np.nan
    got, ref = _both(oracle, case, (1.5, 1.5), 10, 5, 0.45)
    for g, r in zip(got, ref):
        assert np.array_equal(np.isnan(g), np.isnan(r))
