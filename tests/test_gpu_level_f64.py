"""frg_level_solve_f64 (a_smooth = 1): as exact as float64 in the reference's order, the
same bits on a captured stream, and a whole pyramid through level_solver."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from test_gpu_sor_fixed import _both, _case

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _extended(J, wgt, u, v, alpha, its, lag, a_data, omega=1.95):
    """compute_flow in extended precision (np.longdouble).  Pixels of an anti-diagonal do not read
    one another, so a diagonal is one vector operation."""
    Q = np.longdouble
    J = [np.asarray(j[1:-1, 1:-1], dtype=Q) for j in J]
    wg = np.asarray(wgt[1:-1, 1:-1], dtype=Q)
    h, w, K = wg.shape
    ax, ay, om = Q(alpha[0]), Q(alpha[1]), Q(omega)

    def lap(a):
        a = np.asarray(a, dtype=Q)
        c = a[1:-1, 1:-1]
        return ax * (a[1:-1, :-2] - c) + ax * (a[1:-1, 2:] - c) + ay * (a[:-2, 1:-1] - c) + ay * (a[2:, 1:-1] - c)

    lu, lv = lap(u), lap(v)
    du, dv = np.zeros((2, h + 2, w + 2), dtype=Q)
    rows = [np.arange(max(0, d - w + 1), min(h, d + 1)) for d in range(h + w - 1)]
    wp = wg
    for it in range(its):
        if (it + 1) % lag == 0:
            a, b = du[1:-1, 1:-1, None], dv[1:-1, 1:-1, None]
            E = J[0] * a * a + J[1] * b * b + J[2] + 2 * (J[3] * a * b + J[4] * a + J[5] * b)
            wp = wg * Q(a_data) * (np.maximum(E, 0) + Q(0.00001)) ** Q(a_data - 1.0)
        A11, A22, A12, A13, A23 = ((wp * J[q]).sum(2) for q in (0, 1, 3, 4, 5))
        for a in (du, dv):
            a[:, 0], a[:, -1] = a[:, 1], a[:, -2]
            a[0], a[-1] = a[1], a[-2]
        for d, r in enumerate(rows):
            c = d - r
            R, C = r + 1, c + 1
            nb = lambda a: ax * (a[R, C - 1] + a[R, C + 1]) + ay * (a[R - 1, C] + a[R + 1, C])  # noqa: E731
            nu = lu[r, c] - A13[r, c] + nb(du) - A12[r, c] * dv[R, C]
            x = (1 - om) * du[R, C] + om * nu / (A11[r, c] + 2 * ax + 2 * ay)
            nv = lv[r, c] - A23[r, c] + nb(dv) - A12[r, c] * x
            du[R, C] = x
            dv[R, C] = (1 - om) * dv[R, C] + om * nv / (A22[r, c] + 2 * ax + 2 * ay)
    return du, dv


@pytest.mark.parametrize("h,w,K", [(40, 37, 2), (66, 21, 1)])
@pytest.mark.parametrize("scale", [1e-6, 1e-4, 1e-2, 1.0, 30.0])
def test_as_exact_as_float64(oracle, h, w, K, scale):
    """Eight times the oracle's own error: both are float64 evaluations of one recurrence that group the
    terms differently, and after 20 iterations their errors differ by a factor of a few either way."""
    case = _case(h, w, K, h + K, scale, uv=0.0)
    got, ref = _both(oracle, case, (1.5, 1.2), 20, 5, 0.45)
    want = _extended(*case, (1.5, 1.2), 20, 5, 0.45)
    for g, r, q in zip(got, ref, want):
        g, r, q = (a[1:-1, 1:-1] for a in (g, r, q))
        own = float(np.linalg.norm((r - q).astype(np.float64)))
        assert float(np.linalg.norm((g - q).astype(np.float64))) <= 8 * own


_CAPTURE = """
import sys, ctypes
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import numpy as np, torch
from pyflowreg_gb300 import _lib
from pyflowreg_gb300.api import _ptr, _stream_ptr
from test_gpu_sor_fixed import _case
J, wgt, u, v = _case(50, 41, 2, 7)
t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (np.stack(J), wgt, u, v)]
ad = (ctypes.c_double * 2)(0.45, 0.45)
lib = _lib.load()
def solve(du, dv):
    _lib.check(lib.frg_level_solve_f64(52, 43, 2, *map(_ptr, t), 1.5, 1.2, 12, 5, ad, 1.0, 1.0, 1.0, 1.95, -1.0, _ptr(du),
                                       _ptr(dv), _stream_ptr()), "frg_level_solve_f64")
a, b = torch.full((2, 2, 52, 43), 7.0, dtype=torch.float64, device="cuda")
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    solve(a[0], a[1])  # the process's first call
g.replay()
solve(b[0], b[1])
torch.cuda.synchronize()
assert torch.equal(a, b) and bool(torch.isfinite(a).all())
print("same")
"""


def test_first_call_under_capture_gives_the_same_bits():
    out = subprocess.run([sys.executable, "-c", _CAPTURE, os.path.dirname(HERE)], capture_output=True, text=True, timeout=300)
    assert out.stdout.strip().endswith("same"), out.stderr[-2000:]


@pytest.mark.parametrize("shape,K", [((96, 110), 1), ((83, 71), 2)])
def test_whole_pyramid_through_the_seam(oracle, shape, K):
    """Every level through level_solver: within the parity bar of the oracle, as the plan's own levels are."""
    import pyflowreg_gb300 as G

    rng = np.random.default_rng(K)
    base = np.kron(rng.random((shape[0] // 4 + 2, shape[1] // 4 + 2, K)), np.ones((4, 4, 1)))
    base = sum(np.roll(base, (i, j), (0, 1)) for i in range(-2, 3) for j in range(-2, 3)) / 25
    fixed = base[:shape[0], :shape[1]].astype(np.float32)
    moving = (base[1:shape[0] + 1, 1:shape[1] + 1] + 0.01 * rng.random(fixed.shape)).astype(np.float32)
    if K == 1:
        fixed, moving = fixed[..., 0], moving[..., 0]
    kw = dict(alpha=(1.5, 1.5), iterations=30, update_lag=5, levels=100, eta=0.8)
    ref = oracle.get_displacement(fixed, moving, **kw)
    got = G.get_displacement(fixed, moving, level_solver_backend=G.level_solver, **kw)
    own = G.get_displacement(fixed, moving, **kw)
    assert np.abs(own - ref).max() <= 1e-3
    assert np.abs(got - ref).max() <= 1e-3


@pytest.mark.parametrize("scale", [1.0, 3e3])
@pytest.mark.parametrize("q,value", [(2, np.nan), (2, -np.nan), (2, np.inf), (2, -np.inf), (0, np.inf), (1, -np.nan), (5, np.inf)])
def test_not_a_number_reaches_the_result(oracle, q, value, scale):
    """A weight psi of a quadratic form that is no number is none either, whatever the NaN's sign."""
    case = _case(40, 30, 2, 3, scale)
    case[0][q][20, 15, 1] = value
    with np.errstate(all="ignore"):
        got, ref = _both(oracle, case, (1.5, 1.5), 12, 5, 0.45)
    for g, r in zip(got, ref):
        assert np.array_equal(np.isnan(g), np.isnan(r))
