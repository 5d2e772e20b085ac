"""The float64 path's resize at row widths on each side of its forms' limits
(32, 16 or 8 rows of shared memory per block, or rows read from memory), and with
planes whose sums end exactly between two float32s, through whole flows against
the oracle.  Bar: max 1e-3 px, mean 1e-4 px, as for every float64 flow."""
import numpy as np
import pytest

import pyflowreg_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(33, 31), (20, 900), (17, 3400), (9, 6700)])
@pytest.mark.parametrize("levels_of_grey", [0, 8])
def test_flow_of_wide_rows(oracle, H, W, levels_of_grey):
    rng = np.random.default_rng(W)
    x = np.arange(W) + 0.6 * np.sin(np.arange(W) / 40.0)
    y = np.arange(H)
    tex = lambda xx: (0.5 + 0.25 * np.sin(xx / 3.1)[None] * np.cos(y / 2.7)[:, None] + 0.2 * np.cos(xx / 11.0)[None])
    fixed, moving = tex(np.arange(W, dtype=float)), tex(x) + 0.002 * rng.standard_normal((H, W))
    if levels_of_grey:
        fixed, moving = (np.round(a * levels_of_grey) / levels_of_grey for a in (fixed, moving))
    fixed, moving = fixed.astype(np.float32), moving.astype(np.float32)
    kw = dict(alpha=(1.5, 1.5), iterations=6, update_lag=3)
    d = G.get_displacement(fixed, moving, precision="fp64", **kw) - oracle.get_displacement(fixed, moving, **kw)
    assert np.abs(d).max() <= 1e-3 and np.sqrt((d ** 2).sum(-1)).mean() <= 1e-4
