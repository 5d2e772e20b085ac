"""The calls this framework is measured on, through its public entry points.

Every case is a whole call as a program that registers microscopy recordings
makes it: one pair of frames with numpy arrays in and out, one or many frames
that already lie on the device, a batch of mixed sizes, the level solver on
its own, the compensation warp, the per-batch preprocessing and statistics,
and a training step through the differentiable flow.  Frames are photon
counts of blob images that move by a rigid shift and a smooth field, then
normalised and blurred, which is what the flow path sees in use.
"""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

import pyflowreg_gb300 as G
from pyflowreg_gb300 import diff
from pyflowreg_gb300.batch import UnevenBatch
from pyflowreg_gb300.prep import flow_statistics_device, preprocess_device

# The options of the video workloads (the benchmark's own).
VIDEO = dict(alpha=(1.5, 1.5), eta=0.8, levels=100, iterations=50, update_lag=5, a_data=0.45, min_level=0)


def listed():
    return [
        # One small region of interest, as a quick preview or a unit of a larger tool registers it:
        # the smallest call, numpy in and out.
        dict(name="pair_64x72x1", kind="pair", H=64, W=72, K=1, const="gc", precision="fp64"),
        # One 256 x 256 pair with the default options of get_displacement.
        dict(name="pair_256x256x1", kind="pair", H=256, W=256, K=1, const="gc", precision="fp64"),
        # The online form: one two-channel frame at a time, already on the device.
        dict(name="frame_512x512x2", kind="frames", T=1, H=512, W=512, K=2, const="gc", precision="fp64"),
        # A recording's batch at the default buffer size (400 frames) in the reference's precision.
        dict(name="batch400_512x512x2", kind="frames", T=400, H=512, W=512, K=2, const="gc", precision="fp64"),
        # A short batch of odd-sized three-channel frames with brightness constancy.
        dict(name="batch24_333x417x3_gray", kind="frames", T=24, H=333, W=417, K=3, const="gray", precision="fp64"),
        # Large frames: levels taller than one thread block's rows.
        dict(name="batch4_2048x2048x2", kind="frames", T=4, H=2048, W=2048, K=2, const="gc", precision="fp64"),
        # Frames of several sizes and channel counts in one call, launch sequences replayed as graphs.
        dict(name="uneven48", kind="uneven", precision="fp64",
             shapes="256x256x1*6,256x256x2*6,512x512x1*6,512x512x2*6,796x512x1*6,796x512x2*6,1024x1024x1*6,1024x1024x2*6"),
        # The float32 option on a lane's worth of video frames.
        dict(name="batch128_512x512x2_fp32", kind="frames", T=128, H=512, W=512, K=2, const="gc", precision="fp32"),
        # The level solver that pyflowreg plugs into its own pyramid: float64 numpy arrays in and out.
        dict(name="level_410x410x2", kind="level", H=410, W=410, K=2, iterations=50, update_lag=5),
        # The compensation warp of a batch's raw frames by its flows.
        dict(name="warp200_512x512x2", kind="warp", T=200, H=512, W=512, K=2, method="cubic"),
        # What surrounds the flow in the batch loop: normalise and blur the raw frames, masks and statistics of the flows.
        dict(name="prep200_512x512x2", kind="prep", T=200, H=512, W=512, K=2, sigma=1.0, norm="together"),
        # A training step: forward and exact backward of the registration loss.
        dict(name="diff16_512x512x1", kind="diff", T=16, H=512, W=512, K=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: kind, sizes and options over the listed cases' ranges."""
    kind = rng.choice(["pair", "frames", "frames", "frames", "uneven", "level", "warp", "prep", "diff"])
    if kind == "pair":
        return dict(kind=kind, H=_log(rng, 40, 320), W=_log(rng, 40, 320), K=rng.randint(1, 2),
                    const=rng.choice(["gc", "gc", "gray"]), precision=rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "frames":
        H, W, K = _log(rng, 128, 2048), _log(rng, 128, 2048), rng.randint(1, 3)
        if max(H, W) > 1024:
            K = min(K, 2)
        # at most half the 400-frame batch's pixels: large frames cost more per pixel
        most = max(1, min(400, 50_000_000 // (H * W * K)))
        if max(H, W) > 1024:
            most = min(most, 3)
        return dict(kind=kind, T=_log(rng, 1, most) if most > 1 else 1, H=H, W=W, K=K,
                    const=rng.choice(["gc", "gc", "gray"]), precision=rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "uneven":
        parts = ["%dx%dx%d*%d" % (_log(rng, 128, 900), _log(rng, 128, 900), rng.randint(1, 2), rng.randint(1, 5))
                 for _ in range(rng.randint(3, 7))]
        return dict(kind=kind, precision=rng.choice(["fp64", "fp64", "fp32"]), shapes=",".join(dict.fromkeys(parts)))
    if kind == "level":
        return dict(kind=kind, H=_log(rng, 20, 450), W=_log(rng, 20, 450), K=rng.randint(1, 3), iterations=50,
                    update_lag=rng.choice([5, 5, 10]))
    T, H, W, K = 0, _log(rng, 100, 1024), _log(rng, 100, 1024), rng.randint(1, 3)
    if kind in ("warp", "prep"):
        T = _log(rng, 1, max(2, min(400, 100_000_000 // (H * W * K))))
        if kind == "warp":
            return dict(kind=kind, T=T, H=H, W=W, K=K, method=rng.choice(["cubic", "cubic", "linear"]))
        return dict(kind=kind, T=T, H=H, W=W, K=K, sigma=rng.choice([0.5, 1.0, 1.0, 2.0]),
                    norm=rng.choice(["together", "separate"]))
    H, W = _log(rng, 64, 512), _log(rng, 64, 512)
    return dict(kind="diff", T=_log(rng, 1, min(32, 4_000_000 // (H * W))), H=H, W=W, K=rng.randint(1, 2))


# --------------------------------------------------------------------------
# Frames
# --------------------------------------------------------------------------
def _gen(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _image(rng, H, W, dev):
    """Gaussian blobs on a background of 0.05 (the exponential separates)."""
    n = max(40, H * W // 6500)
    cy, cx = rng.uniform(0, H, n), rng.uniform(0, W, n)
    s, a = rng.uniform(2.0, 6.0, n), rng.uniform(0.3, 1.0, n)
    gy = a[:, None] * np.exp(-((np.arange(H)[None] - cy[:, None]) ** 2) / (2 * s[:, None] ** 2))
    gx = np.exp(-((np.arange(W)[None] - cx[:, None]) ** 2) / (2 * s[:, None] ** 2))
    gy, gx = (torch.tensor(x, dtype=torch.float32, device=dev) for x in (gy, gx))
    return 0.05 + gy.t() @ gx


def _field(rng, T, H, W, dev, amp=2.0, shift=3.0):
    """(T, H, W, 2) displacements: a rigid shift N(0, shift) per frame and a
    drifting sum of four plane waves of at most `amp` pixels per component."""
    yy = torch.arange(H, dtype=torch.float32, device=dev)[:, None]
    xx = torch.arange(W, dtype=torch.float32, device=dev)[None]
    lam, th, ph = rng.uniform(64, 256, (2, 4)), rng.uniform(0, 2 * np.pi, (2, 4)), rng.uniform(0, 2 * np.pi, (2, 4))
    rigid = rng.normal(0.0, shift, (T, 2))
    out = torch.empty((T, H, W, 2), dtype=torch.float32, device=dev)
    phase = torch.tensor(2 * np.pi * np.arange(T) / 250.0, dtype=torch.float32, device=dev)[:, None, None]
    for c in range(2):
        acc = 0.0
        for k in range(4):
            ky, kx = 2 * np.pi / lam[c, k] * np.cos(th[c, k]), 2 * np.pi / lam[c, k] * np.sin(th[c, k])
            arg = float(ky) * yy + float(kx) * xx + float(ph[c, k])
            acc = acc + torch.sin(arg[None] + phase)
        out[..., c] = acc * (amp / 4) + torch.tensor(rigid[:, c], dtype=torch.float32, device=dev)[:, None, None]
    return out


def _sample(img, flow):
    """img (K, H, W) at x - flow(x): (T, H, W, K)."""
    K, H, W = img.shape
    out = torch.empty(flow.shape[:3] + (K,), dtype=torch.float32, device=img.device)
    yy = torch.arange(H, dtype=torch.float32, device=img.device)[:, None]
    xx = torch.arange(W, dtype=torch.float32, device=img.device)[None]
    for t0 in range(0, flow.shape[0], 32):
        f = flow[t0:t0 + 32]
        grid = torch.stack([(xx - f[..., 0]) * (2.0 / (W - 1)) - 1.0, (yy - f[..., 1]) * (2.0 / (H - 1)) - 1.0], -1)
        s = F.grid_sample(img[None].expand(f.shape[0], K, H, W), grid, mode="bicubic", padding_mode="border",
                          align_corners=True)
        out[t0:t0 + 32] = s.permute(0, 2, 3, 1)
    return out


def _blur(x):
    """Spatial Gaussian, sigma 1, of (T, H, W, K)."""
    g = torch.exp(-0.5 * torch.arange(-4, 5, dtype=torch.float32, device=x.device) ** 2)
    g = g / g.sum()
    T, H, W, K = x.shape
    out = torch.empty_like(x)
    for t0 in range(0, T, 64):
        y = x[t0:t0 + 64].permute(0, 3, 1, 2).reshape(-1, 1, H, W)
        y = F.conv2d(F.pad(y, (4, 4, 0, 0), mode="reflect"), g.view(1, 1, 1, -1))
        y = F.conv2d(F.pad(y, (0, 0, 4, 4), mode="reflect"), g.view(1, 1, -1, 1))
        out[t0:t0 + 64] = y.reshape(-1, K, H, W).permute(0, 2, 3, 1)
    return out


def _counts(seed, T, H, W, K, dev):
    """(reference (H, W, K), frames (T, H, W, K), flows (T, H, W, 2)): photon counts of a moving scene."""
    rng = np.random.default_rng(seed)
    img = torch.stack([_image(rng, H, W, dev) for _ in range(K)])
    flow = _field(rng, T, H, W, dev)
    lam = torch.tensor(np.exp(rng.uniform(np.log(50.0), np.log(2000.0), T)), dtype=torch.float32, device=dev)
    raw = _sample(img, flow).clamp_(min=0).mul_(0.5 * lam[:, None, None, None])
    raw = torch.poisson(raw, generator=_gen(seed + 1, dev))
    ref = torch.poisson((img * (500.0 * 50)).permute(1, 2, 0).contiguous(), generator=_gen(seed + 2, dev)) / 50.0
    return ref, raw, flow


def _frames(seed, T, H, W, K, dev):
    """The same, normalised by the reference's range and blurred."""
    ref, raw, flow = _counts(seed, T, H, W, K, dev)
    lo, hi = ref.min(), ref.max()
    proc = _blur((raw - lo) / (hi - lo))
    return _blur(((ref - lo) / (hi - lo))[None])[0].contiguous(), proc.contiguous(), flow


def _tensor(f1, f2):
    """Gradient-constancy motion tensor of two (K, H, W) float64 images, six
    (H + 2, W + 2, K) arrays with a zero ring, the form the level solver takes."""
    def d(a, ax):
        p = F.pad(a[None], (1, 1, 1, 1), mode="replicate")[0]
        return 0.5 * (p[:, 1:-1, 2:] - p[:, 1:-1, :-2]) if ax else 0.5 * (p[:, 2:, 1:-1] - p[:, :-2, 1:-1])

    def d2(a, ax):
        p = F.pad(a[None], (1, 1, 1, 1), mode="replicate")[0]
        c = p[:, 1:-1, 1:-1]
        return p[:, 1:-1, 2:] - 2 * c + p[:, 1:-1, :-2] if ax else p[:, 2:, 1:-1] - 2 * c + p[:, :-2, 1:-1]

    m, t = 0.5 * (f1 + f2), f2 - f1
    fxx, fyy, fxy, fxt, fyt = d2(m, 1), d2(m, 0), d(d(m, 1), 0), d(t, 1), d(t, 0)
    rx, ry = 1.0 / (fxx ** 2 + fxy ** 2 + 1e-6), 1.0 / (fxy ** 2 + fyy ** 2 + 1e-6)
    J = [rx * fxx ** 2 + ry * fxy ** 2, rx * fxy ** 2 + ry * fyy ** 2, rx * fxt ** 2 + ry * fyt ** 2,
         rx * fxx * fxy + ry * fxy * fyy, rx * fxx * fxt + ry * fxy * fyt, rx * fxy * fxt + ry * fyy * fyt]
    return [F.pad(j, (1, 1, 1, 1)).permute(1, 2, 0).contiguous().cpu().numpy() for j in J]


def _shapes(case):
    for part in case["shapes"].split(","):
        size, n = part.split("*")
        h, w, k = (int(v) for v in size.split("x"))
        yield h, w, k, int(n)


# --------------------------------------------------------------------------
# The four functions of a case
# --------------------------------------------------------------------------
def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind, s = case["kind"], 1000 * int(seed) + 7
    if kind == "uneven":
        refs, groups = {}, []
        for i, (h, w, k, n) in enumerate(_shapes(case)):
            ref, proc, _ = _frames(s + 10 * i, n, h, w, k, dev)
            refs[(h, w, k)] = ref
            groups.append([proc[j].contiguous() for j in range(n)])
        # the frames arrive in mixed order
        frames = [g[j] for j in range(max(len(g) for g in groups)) for g in groups if j < len(g)]
        opts = {k: v for k, v in VIDEO.items() if k != "min_level"}
        return dict(kind=kind, frames=frames, batch=UnevenBatch(refs, graphs=True, precision=case["precision"], **opts))
    T, H, W, K = case.get("T", 1), case["H"], case["W"], case["K"]
    if kind == "pair":
        ref, proc, _ = _frames(s, 1, H, W, K, dev)
        fixed, moving = ref.cpu().numpy(), proc[0].cpu().numpy()
        if K == 1:
            fixed, moving = fixed[..., 0], moving[..., 0]
        return dict(kind=kind, fixed=np.ascontiguousarray(fixed), moving=np.ascontiguousarray(moving),
                    opts=dict(const_assumption=case["const"], precision=case["precision"]))
    if kind == "frames":
        ref, proc, _ = _frames(s, T, H, W, K, dev)
        return dict(kind=kind, fixed=ref, moving=proc,
                    opts=dict(VIDEO, const_assumption=case["const"], precision=case["precision"]))
    if kind == "level":
        ref, proc, _ = _frames(s, 1, H, W, K, dev)
        J = _tensor(ref.permute(2, 0, 1).double(), proc[0].permute(2, 0, 1).double())
        rng = np.random.default_rng(s)
        wgt = np.full((H + 2, W + 2, K), 1.0 / K)
        u, v = (np.pad(f, 1, mode="edge") for f in _field(rng, 1, H, W, dev)[0].double().cpu().numpy().transpose(2, 0, 1))
        return dict(kind=kind, J=J, weight=wgt, u=u, v=v, iterations=case["iterations"], lag=case["update_lag"], K=K)
    if kind == "diff":
        ref, proc, flow = _frames(s, T, H, W, K, dev)
        fixed, moving = ref.permute(2, 0, 1).contiguous(), proc.permute(0, 3, 1, 2).contiguous()
        plan = diff.DiffPlan(H, W, K, T, dtype=torch.float32, checkpoint="sweeps", levels=100, eta=0.8, iterations=50,
                             update_lag=5)
        plan.set_weight([1.0 / K] * K)
        return dict(kind=kind, fixed=fixed, moving=moving, truth=fixed[None].expand_as(moving).contiguous(),
                    w_true=flow.permute(0, 3, 1, 2).contiguous(), alpha=torch.tensor(1.5, device=dev), plan=plan)
    ref, raw, flow = _counts(s, T, H, W, K, dev)
    if kind == "warp":
        return dict(kind=kind, frames=raw, flow=flow, ref=ref, method=case["method"])
    # prep: the raw reference is a host array, as the batch loop holds it
    return dict(kind=kind, frames=raw, flow=flow, ref=ref.cpu().numpy(), sigma=((case["sigma"], case["sigma"], 0.1),),
                norm=case["norm"])


def run(state):
    kind = state["kind"]
    if kind == "pair":
        return G.get_displacement(state["fixed"], state["moving"], **state["opts"])
    if kind == "frames":
        return G.api.get_displacement_device(state["fixed"], state["moving"], **state["opts"])
    if kind == "uneven":
        return state["batch"].register(state["frames"])
    if kind == "level":
        K = state["K"]
        return G.level_solver(*state["J"], state["weight"], state["u"], state["v"], (1.5, 1.5), state["iterations"],
                              state["lag"], 0, np.full(K, 0.45), 1.0, 1.0, 1.0)
    if kind == "warp":
        return G.imregister_device(state["frames"], state["flow"], state["ref"], state["method"])
    if kind == "prep":
        proc = preprocess_device(state["frames"], state["ref"], state["sigma"], state["norm"], frames_dtype=np.uint16)
        mask, stats = flow_statistics_device(state["flow"])
        return [proc, mask, stats]
    fixed, moving, alpha = (state[k].detach().requires_grad_(True) for k in ("fixed", "moving", "alpha"))
    loss = diff.registration_loss(fixed, moving, state["truth"], state["w_true"], alpha, state["plan"])
    return [loss.detach(), *torch.autograd.grad(loss, (fixed, moving, alpha))]


def _level_pixels(H, W, eta=0.8):
    """Pixels of all pyramid levels (ratio eta per side, coarsest about 10 px)."""
    px, h, w = 0.0, float(H), float(W)
    while min(h, w) >= 9.5:
        px += h * w
        h, w = h * eta, w * eta
    return max(px, float(H * W))


def _flow_work(H, W, K, T, es):
    """One frame: each level's 50 sweeps of 28 flops per pixel, ten psi ticks of
    about 60 flops per channel, tensor, warp, resize and median about 350 per
    channel; frames in, flow out."""
    px = _level_pixels(H, W)
    return T * (H * W * K * 4 + H * W * 2 * es) + H * W * K * 4, T * px * (50 * 28 + 10 * 60 * K + 350 * K)


def work(case):
    kind = case["kind"]
    if kind == "uneven":
        es = 8 if case["precision"] == "fp64" else 4
        b = f = 0.0
        for h, w, k, n in _shapes(case):
            x, y = _flow_work(h, w, k, n, es)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    T, H, W, K = case.get("T", 1), case["H"], case["W"], case["K"]
    px = T * H * W
    if kind in ("pair", "frames"):
        b, f = _flow_work(H, W, K, T, 8 if case["precision"] == "fp64" else 4)
        return {"bytes": b, "flops": f}
    if kind == "level":
        n = (H + 2) * (W + 2)
        return {"bytes": n * 8 * (7 * K + 4), "flops": px * (case["iterations"] * 28 + case["iterations"] // case["update_lag"] * 60 * K)}
    if kind == "warp":
        return {"bytes": px * (8 * K + 8) + H * W * K * 4, "flops": px * (32 * K + 30)}
    if kind == "prep":
        taps = 2 * int(4 * case["sigma"] + 0.5) + 1
        return {"bytes": px * (8 * K + 8 + 1), "flops": px * (K * (4 * taps + 3) + 12)}
    # forward and about twice that backward
    b, f = _flow_work(H, W, K, T, 4)
    return {"bytes": b + T * H * W * (K * 12 + 16), "flops": 3 * f}


# --------------------------------------------------------------------------
# The same results in 64 bits
# --------------------------------------------------------------------------
def _exact_level(st):
    """compute_flow: column by column, row by row SOR (omega 1.95) in place.
    Pixels of one anti-diagonal do not read one another, so a diagonal is one
    vector operation; arrays are stored by diagonal."""
    K, its, lag = st["K"], st["iterations"], st["lag"]
    J = [j[1:-1, 1:-1].astype(np.float64) for j in st["J"]]
    wgt = st["weight"][1:-1, 1:-1]
    h, w = J[0].shape[:2]
    ax = 1.5
    idx = [(np.arange(max(0, d - w + 1), min(h, d + 1)), d - np.arange(max(0, d - w + 1), min(h, d + 1)))
           for d in range(h + w - 1)]

    def lap(a):
        c = a[1:-1, 1:-1]
        return ax * (a[1:-1, :-2] - c) + ax * (a[1:-1, 2:] - c) + ax * (a[:-2, 1:-1] - c) + ax * (a[2:, 1:-1] - c)

    lu, lv = lap(st["u"]), lap(st["v"])
    du, dv = np.zeros((h + 2, w + 2)), np.zeros((h + 2, w + 2))
    psi = np.ones((h, w, K))
    om = 1.95
    for it in range(its):
        if (it + 1) % lag == 0:
            a, b = du[1:-1, 1:-1, None], dv[1:-1, 1:-1, None]
            E = J[0] * a * a + J[1] * b * b + J[2] + 2 * J[3] * a * b + 2 * J[4] * a + 2 * J[5] * b
            psi = 0.45 * (np.maximum(E, 0.0) + 0.00001) ** (0.45 - 1.0)
        for a in (du, dv):
            a[:, 0], a[:, -1] = a[:, 1], a[:, -2]
            a[0], a[-1] = a[1], a[-2]
        if it == 0 or (it + 1) % lag == 0:
            wp = wgt * psi
            A11, A22, A12, A13, A23 = ((wp * J[q]).sum(2) for q in (0, 1, 3, 4, 5))
        for r, c in idx:
            R, C = r + 1, c + 1
            nu = lu[r, c] - A13[r, c] + ax * (du[R, C - 1] + du[R, C + 1] + du[R - 1, C] + du[R + 1, C]) - A12[r, c] * dv[R, C]
            x = (1 - om) * du[R, C] + om * nu / (A11[r, c] + 4 * ax)
            nv = lv[r, c] - A23[r, c] + ax * (dv[R, C - 1] + dv[R, C + 1] + dv[R - 1, C] + dv[R + 1, C]) - A12[r, c] * x
            du[R, C] = x
            dv[R, C] = (1 - om) * dv[R, C] + om * nv / (A22[r, c] + 4 * ax)
    return du, dv


def _exact_warp(st):
    """Bicubic (A = -0.75) or bilinear sampling at coordinates rounded to 1/32
    pixel, borders repeated, the reference outside the frame.  Coordinates are
    float32 sums, as the frames' flows are; weights and sums are 64-bit."""
    fr, fl, ref = st["frames"], st["flow"], st["ref"].double()
    T, H, W, K = fr.shape
    dev = fr.device
    yy = torch.arange(H, dtype=torch.float32, device=dev)[:, None]
    xx = torch.arange(W, dtype=torch.float32, device=dev)[None]
    cubic = st["method"] == "cubic"
    taps = 4 if cubic else 2

    def weights(t):
        if not cubic:
            return [1 - t, t]
        A = -0.75
        out = lambda x: ((A * x - 5 * A) * x + 8 * A) * x - 4 * A  # noqa: E731
        inn = lambda x: ((A + 2) * x - (A + 3)) * x * x + 1  # noqa: E731
        return [out(1 + t), inn(t), inn(1 - t), out(2 - t)]

    res = torch.empty((T, H, W, K), dtype=torch.float64, device=dev)
    for t in range(T):
        mx, my = xx + fl[t, ..., 0], yy + fl[t, ..., 1]
        oob = (mx < 0) | (mx >= W) | (my < 0) | (my >= H)
        X = torch.round(mx.clamp(0, W - 1) * 32).long()
        Y = torch.round(my.clamp(0, H - 1) * 32).long()
        wx, wy = weights((X & 31).double() / 32), weights((Y & 31).double() / 32)
        off = 1 if cubic else 0
        acc = 0.0
        src = fr[t].double()
        for i in range(taps):
            yi = ((Y >> 5) - off + i).clamp(0, H - 1)
            for j in range(taps):
                xi = ((X >> 5) - off + j).clamp(0, W - 1)
                acc = acc + (wy[i] * wx[j])[..., None] * src[yi, xi]
        res[t] = torch.where(oob[..., None], ref, acc)
    return res


def _exact_prep(st):
    """(x - min) / (max - min + 1e-8) and a Gaussian per axis with the edge
    sample repeated; per frame mean and largest |w|, mean divergence, |mean w|."""
    fr, ref, s = st["frames"], st["ref"].astype(np.float64), st["sigma"][0][0]
    T, H, W, K = fr.shape
    dev = fr.device
    if st["norm"] == "separate":
        lo, hi = ref.min((0, 1)), ref.max((0, 1))
    else:
        lo, hi = np.full(K, ref.min()), np.full(K, ref.max())
    r = int(4 * s + 0.5)
    g = np.exp(-0.5 / (s * s) * np.arange(-r, r + 1) ** 2)
    g = g / g.sum()

    def taps(n):
        i = np.arange(n)[None] + np.arange(-r, r + 1)[:, None]
        i = np.where(i < 0, -i - 1, i)
        return torch.tensor(np.where(i >= n, 2 * n - 1 - i, i), device=dev)

    iy, ix = taps(H), taps(W)
    lo_t, den = (torch.tensor(a, device=dev) for a in (lo, hi - lo + 1e-8))
    out = torch.empty((T, H, W, K), dtype=torch.float64, device=dev)
    for t in range(T):
        x = (fr[t].double() - lo_t) / den
        x = sum(float(g[k]) * x[iy[k]] for k in range(2 * r + 1))
        out[t] = sum(float(g[k]) * x[:, ix[k]] for k in range(2 * r + 1))
    stats = torch.empty((T, 4), dtype=torch.float64, device=dev)
    for t in range(T):
        w = st["flow"][t].double()
        mag = torch.sqrt(w[..., 0] ** 2 + w[..., 1] ** 2)
        div = torch.gradient(w[..., 0], dim=1)[0] + torch.gradient(w[..., 1], dim=0)[0]
        m = w.mean((0, 1))
        stats[t] = torch.stack([mag.mean(), mag.max(), div.mean(), torch.sqrt(m[0] ** 2 + m[1] ** 2)])
    return [out, None, stats]


def exact(case, seed):
    """None for the whole flow calls and the training step: their 64-bit run
    would be the whole pyramid again, pixel by pixel."""
    if case["kind"] not in ("level", "warp", "prep"):
        return None
    st = prepare(case, seed)
    return {"level": _exact_level, "warp": _exact_warp, "prep": _exact_prep}[case["kind"]](st)
