"""Workloads of the framework as its users run them, for timing and for comparing results.

Frames are seeded synthetic PIV pairs (Gaussian particle images moved by a smooth
divergence-free field, noise, 8 bits), rendered on the GPU.  `listed()` holds one or two
cases of every path a user calls, from one small filter to a mixed batch of uneven pairs;
`draw()` gives further ones over the same ranges: frame sides of 96 to 2048 pixels, odd ones
included, all four methods, both Liu-Shen arithmetics, tensors and host arrays.

`exact()` restates the methods in float64 with torch alone.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "opticalflow-ri_b200"))

import Farneback_PyCL as FB  # noqa: E402
import HornSchunck as HS  # noqa: E402
import PhysicsBasedOpticalFlowLiuShen as LS  # noqa: E402
import denseLucasKanade_PyCL as LK  # noqa: E402
from GenericPyramidalOpticalFlow import genericPyramidalOpticalFlow  # noqa: E402
from gaussian_filter import gaussian_filterPx  # noqa: E402
from ofb200 import batch, warmstart  # noqa: E402

MAX_DISP = 4.0  # pixels


def listed():
    return [
        # the prefilter of one small frame: a single launch, all latency
        {"name": "prefilter_256", "kind": "prefilter", "h": 256, "w": 256, "sigma": 0.48, "taps": 5},
        # the Horn-Schunck calibration on one 256 x 256 pair: 600 sweeps, latency of one solve
        {"name": "hs_256", "kind": "hs", "h": 256, "w": 256, "sweeps": 600},
        # dense Lucas-Kanade, two pyramid levels, the 512 x 512 calibration
        {"name": "lk_512", "kind": "lk", "h": 512, "w": 512, "half_window": 13},
        # one Lucas-Kanade level from a given field on a ragged frame, with the status and
        # error planes that a user masks vectors with, and a window other than the default
        {"name": "lk_status_ragged", "kind": "lk_status", "h": 301, "w": 413, "half_window": 9},
        # Farneback alone on a ragged frame, tensors in and out
        {"name": "farneback_ragged", "kind": "farneback", "h": 719, "w": 1013, "window": 33, "poly": 7},
        # Liu-Shen refinement of the largest frames
        {"name": "liushen_2048", "kind": "liushen", "h": 2048, "w": 2048, "arithmetic": "fast"},
        # the bit-exact Liu-Shen arithmetic on a ragged frame
        {"name": "liushen_exact_ragged", "kind": "liushen", "h": 517, "w": 389, "arithmetic": "exact"},
        # the Farneback + Liu-Shen calibration as a script calls it: one pair, host arrays in and out
        {"name": "fbls_1024_call", "kind": "fbls_call", "h": 1024, "w": 1024},
        # the same calibration over a stack of pairs on the GPU (the throughput path)
        {"name": "fbls_1024_batch8", "kind": "fbls_batch", "h": 1024, "w": 1024, "pairs": 8},
        # the learned warm start over a batch of pairs
        {"name": "learned_1024_batch30", "kind": "learned", "pairs": 30},
        # one training step of its network: forward, loss, backward, Adam
        {"name": "train_128_batch16", "kind": "train", "crop": 128, "pairs": 16},
        # a batch of pairs of uneven sizes and all four methods
        {"name": "mixed_24", "kind": "mixed", "pairs": 24, "largest": 2048},
    ]


def draw(rng):
    def side(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | rng.randint(0, 1))

    kind = rng.choice(["prefilter", "hs", "lk", "lk_status", "farneback", "liushen", "liushen", "fbls_call",
                       "fbls_batch", "learned", "train", "mixed"])
    c = {"kind": kind}
    if kind == "learned":  # the packaged network runs at 1 / 8 of 1024 x 1024 frames
        return {**c, "pairs": rng.randint(1, 30)}
    if kind == "train":
        crop = rng.choice([64, 128, 256])
        return {**c, "crop": crop, "pairs": 2 * rng.randint(1, 8)}
    if kind == "mixed":
        return {**c, "pairs": rng.randint(4, 24), "largest": rng.choice([512, 1024, 2048])}
    hi = {"prefilter": 2048, "hs": 512, "lk": 640, "lk_status": 640, "farneback": 1536, "liushen": 2048,
          "fbls_call": 1536, "fbls_batch": 1024}[kind]
    c.update(h=side(96, hi), w=side(96, hi))
    if kind == "prefilter":
        c.update(sigma=rng.choice([0.48, 2.0, 3.4]), taps=rng.choice([3, 5]))
    elif kind == "hs":
        c.update(sweeps=rng.choice([100, 600]))
    elif kind in ("lk", "lk_status"):
        c.update(half_window=rng.choice([13, 13, 9, 7]))
    elif kind == "farneback":
        c.update(window=rng.choice([33, 33, 21]), poly=rng.choice([7, 7, 5]))
    elif kind == "liushen":
        c.update(arithmetic=rng.choice(["fast", "fast", "exact"]))
    elif kind == "fbls_batch":
        c.update(pairs=rng.randint(2, 12))
    return c


# ------------------------------------------------------------------------------ inputs
def _pair(h, w, seed):
    """Two uint8 frames on the GPU: about 0.05 particles per pixel of 2 to 3 pixels diameter,
    moved by a random divergence-free field of 32 modes, with 2 grey levels of noise.  The
    particle images are summed in fixed point, so the sum does not depend on its order."""
    host = np.random.default_rng(seed)
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    k = host.uniform(1.0, 8.0, 32) * 2 * np.pi / max(h, w)
    ang, phase, amp = host.uniform(0, 2 * np.pi, 32), host.uniform(0, 2 * np.pi, 32), host.normal(0, 1, 32)
    kx, ky, phase, amp = (torch.tensor(a, device=dev) for a in (k * np.cos(ang), k * np.sin(ang), phase, amp / k))
    pad = 12
    n = int(0.05 * (h + 2 * pad) * (w + 2 * pad))
    rnd = lambda lo, hi: lo + (hi - lo) * torch.rand(n, generator=gen, device=dev, dtype=torch.float64)  # noqa: E731
    px, py, peak, diam = rnd(-pad, w + pad), rnd(-pad, h + pad), rnd(128, 255), rnd(2, 3)
    c = amp * torch.cos(px[:, None] * kx + py[:, None] * ky + phase)
    u, v = (c * ky).sum(1), -(c * kx).sum(1)
    s = MAX_DISP / torch.hypot(u, v).max()
    o = torch.arange(-4, 5, device=dev)
    frames = []
    for x, y in ((px, py), (px + s * u, py + s * v)):
        ix, iy = torch.floor(x).long()[:, None, None] + o[None, None, :], torch.floor(y).long()[:, None, None] + o[None, :, None]
        r2 = (ix - x[:, None, None]) ** 2 + (iy - y[:, None, None]) ** 2
        val = (peak[:, None, None] * torch.exp(-8.0 * r2 / diam[:, None, None] ** 2) * 65536.0).round().long()
        keep = (ix >= 0) & (ix < w) & (iy >= 0) & (iy < h)
        img = torch.zeros(h * w, dtype=torch.int64, device=dev)
        img.index_add_(0, (iy * w + ix)[keep], val[keep])
        img = img.reshape(h, w).double() / 65536.0
        img = img + 2.0 * torch.randn(h, w, generator=gen, device=dev, dtype=torch.float64)
        frames.append(img.round().clamp(0, 255).to(torch.uint8))
    return frames


def _field(h, w, seed):
    """A smooth initial flow of up to a pixel or two."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 77)
    coarse = torch.randn(1, 2, 6, 6, generator=gen, device="cuda")
    f = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=True)[0]
    return f[0].contiguous(), f[1].contiguous()


def _manifest(case):
    """Entries of a mixed batch: sizes up to the case's largest, every method, ragged widths
    for every third pair.  The layout depends on the case alone, as a plan's does."""
    sizes = [s for s in batch.CONFIG4_SIZES if s <= case["largest"]]
    rng = np.random.default_rng(case["pairs"] * 7919 + case["largest"])
    out = []
    for i in range(case["pairs"]):
        size = case["largest"] if i == 0 else int(rng.choice(sizes))
        out.append({"size": size, "method": batch.CONFIG4_METHODS[i % 4],
                    "w": size - 1 - 2 * int(rng.integers(0, size // 8)) if i % 3 == 2 else size})
    return out


_plans = {}  # one batch plan per case, as a program that feeds it frame after frame keeps it


def _plan(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _plans:
        kind = case["kind"]
        if kind == "fbls_batch":
            plan = batch.PairBatch([batch.method_spec("ls") for _ in range(case["pairs"])], streams=8)
        elif kind == "learned":
            net, meta = warmstart.load_trained()
            plan = warmstart.LearnedBatch(net, meta, case["pairs"], 1024, streams=8)
        else:
            plan = batch.BatchRunner(_manifest(case), chunk=64, streams=8)
        while len(_plans) >= 3:
            del _plans[next(iter(_plans))]
        _plans[key] = plan
    return _plans[key]


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "fbls_batch":
        st.update(plan=_plan(case), frames=[_pair(case["h"], case["w"], seed * 1000 + i) for i in range(case["pairs"])])
    elif kind == "learned":
        st.update(plan=_plan(case), frames=[_pair(1024, 1024, seed * 1000 + i) for i in range(case["pairs"])])
    elif kind == "mixed":
        st.update(plan=_plan(case),
                  frames=[_pair(e["size"], e["w"], seed * 1000 + i) for i, e in enumerate(_manifest(case))])
    elif kind == "train":
        n, crop = case["pairs"], case["crop"]
        net = warmstart.WarmStartNet(seed=seed)
        st.update(net=net, b=net.buffers(n, crop), g=net.grad_buffers(n, crop), frames=_train_frames(case, seed),
                  label=_train_label(case, seed))
    else:
        a, b = _pair(case["h"], case["w"], seed)
        if kind == "prefilter":
            st["frame"] = a.float()
        elif kind == "fbls_call":
            st.update(a=a.cpu().numpy().astype(np.float32), b=b.cpu().numpy().astype(np.float32))
        else:
            st.update(a=a.float(), b=b.float())
        if kind in ("lk_status", "liushen", "farneback"):
            st["U"], st["V"] = _field(case["h"], case["w"], seed)
    return st


def _train_frames(case, seed):
    return [tuple(f.float() for f in _pair(case["crop"], case["crop"], seed * 1000 + i)) for i in range(case["pairs"])]


def _train_label(case, seed):
    f = [torch.stack(_field(case["crop"], case["crop"], seed * 1000 + i), -1) for i in range(case["pairs"])]
    return torch.stack(f).contiguous()


# ------------------------------------------------------------------------------ one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "prefilter":  # filters in place: the program keeps its frame
        return gaussian_filterPx(st["frame"].clone(), case["sigma"], case["taps"])
    if kind == "hs":
        return genericPyramidalOpticalFlow(st["a"], st["b"], 3.4, HS.HSOpticalFlowAlgoAdapter([21], case["sweeps"]), 1)
    if kind == "lk":
        return genericPyramidalOpticalFlow(st["a"], st["b"], 2.0, LK.denseLucasKanade_PyCl(halfWindow=case["half_window"]), 2)
    if kind == "lk_status":
        return LK.denseLucasKanade_PyCl(halfWindow=case["half_window"]).compute_with_status(st["a"], st["b"], st["U"], st["V"])
    if kind == "farneback":
        fb = FB.Farneback_PyCL(windowSize=case["window"], polyN=case["poly"])
        return fb.compute(st["a"], st["b"], st["U"], st["V"])[:2]
    if kind == "liushen":
        u, v, _ = LS.LiuShenOpticalFlowAlgoAdapter(10, case["arithmetic"]).compute(st["a"], st["b"], st["U"], st["V"])
        return u, v
    if kind == "fbls_call":
        return genericPyramidalOpticalFlow(st["a"], st["b"], 0, FB.Farneback_PyCL(), 2, 1, 0.48,
                                           LS.LiuShenOpticalFlowAlgoAdapter(10))
    if kind == "train":
        net, b, g = st["net"], st["b"], st["g"]
        for i, (a0, a1) in enumerate(st["frames"]):
            net.pack_input(b, i, a0, a1)
        net.forward(b)
        loss = net.loss(b, g, st["label"])
        net.backward(b, g)
        grads = net.grads.clone()
        net.adam(0.0)  # the optimizer and the weight packing at rate 0: a pass can be repeated on the same weights
        return loss, b["out"], grads
    return st["plan"].run(st["frames"])


# ------------------------------------------------------------------------------ work
def _net_flops(pixels):
    scale = {"c0a": 1, "c0b": 1, "c1a": 4, "c1b": 4, "c2a": 16, "c2b": 16, "c3a": 64, "c3b": 64, "d2": 16, "d1": 4,
             "d0": 1, "head": 1}
    return sum(18.0 * ci * co * pixels / scale[name] for name, ci, co in warmstart.LAYERS)


_HS = 45.0         # per pixel and sweep: two 8-term sums, one quotient, two updates
_LS = 75.0         # per pixel and sweep: twelve stencils, two 2 x 2 products
_FB = 5 * 690.0    # per pixel: five iterations of a 33-tap separable blur of 5 planes, solve, matrices
_FB_SETUP = 260.0  # per pixel: two polynomial expansions


def _lk(half_window):  # per pixel: the gradient matrix and two Newton steps over the window
    return (2 * half_window + 1) ** 2 * (6 + 2 * 16.0)


def work(case):
    kind = case["kind"]
    if kind == "learned":
        px = 1024.0 * 1024 * case["pairs"]
        return {"bytes": 10 * px, "flops": px * (_FB / 5 + _FB_SETUP + 4 * _LS) + _net_flops(px / 64)}
    if kind == "train":
        px = float(case["crop"]) ** 2 * case["pairs"]
        return {"bytes": 16 * px + 28.0 * warmstart.n_params(), "flops": 3 * _net_flops(px)}
    if kind == "mixed":
        total = {"bytes": 0.0, "flops": 0.0}
        per = {"hs": 600 * _HS, "lk": 1.25 * _lk(13), "fb": 1.25 * (_FB + _FB_SETUP),
               "ls": 1.25 * (_FB + _FB_SETUP + 60 * _LS)}
        for e in _manifest(case):
            px = float(e["size"]) * e["w"]
            total["bytes"] += 10 * px
            total["flops"] += px * per[e["method"]]
        return total
    px = float(case["h"]) * case["w"]
    if kind == "prefilter":
        return {"bytes": 8 * px, "flops": 4 * case["taps"] * px}
    if kind == "hs":
        return {"bytes": 16 * px, "flops": case["sweeps"] * _HS * px}
    if kind == "lk":
        return {"bytes": 16 * px, "flops": 1.25 * _lk(case["half_window"]) * px}
    if kind == "lk_status":
        return {"bytes": 29 * px, "flops": (_lk(case["half_window"]) + 20 * (2 * case["half_window"] + 1) ** 2) * px}
    if kind == "farneback":
        return {"bytes": 24 * px, "flops": (_FB * case["window"] / 33.0 + _FB_SETUP * case["poly"] / 7.0) * px}
    if kind == "liushen":
        return {"bytes": 24 * px, "flops": 60 * _LS * px}
    n = case.get("pairs", 1)
    return {"bytes": (10 if kind == "fbls_batch" else 16) * px * n, "flops": 1.25 * (_FB + _FB_SETUP + 60 * _LS) * px * n}


# ------------------------------------------------------------------------------ float64
def _pad(t, p, mode):
    """Borders of a (..., h, w) float64 stack; scipy's 'mirror' is reflect, 'nearest' replicate."""
    lead = t.shape[:-2]
    t = t.reshape(1, -1, *t.shape[-2:])
    t = torch.nn.functional.pad(t, (p, p, p, p), mode=mode) if mode != "zero" else torch.nn.functional.pad(t, (p,) * 4)
    return t.reshape(*lead, *t.shape[-2:])


def _sh(t, p, dy, dx):
    """The plane shifted by (dy, dx) out of its padded form."""
    h, w = t.shape[-2] - 2 * p, t.shape[-1] - 2 * p
    return t[..., p + dy:p + dy + h, p + dx:p + dx + w]


def _x_prefilter(img, sigma, taps):
    x = torch.arange(-(taps // 2), taps // 2 + 1, dtype=torch.float64, device=img.device)
    k = torch.exp(-x * x / (2.0 * sigma * sigma))
    k = k / k.sum()
    for _ in range(2):  # rows, then columns through the transpose
        h, n = taps // 2, img.shape[1]
        t = torch.cat([img[:, :h].flip(1), img, img[:, n - h:]], 1)
        img = sum(k[j] * t[:, 2 * h - j:2 * h - j + n] for j in range(taps)).t()
    return img


def _x_hs(a, b, u, v, sweeps, alpha=21.0):
    def corners(f):
        p = _pad(f, 1, "reflect")
        return f, _sh(p, 1, 0, 1), _sh(p, 1, 1, 0), _sh(p, 1, 1, 1)

    fx = fy = 0.0
    for f in (a, b):
        c00, c01, c10, c11 = corners(f)
        fx = fx + 0.25 * (c00 - c01 + c10 - c11)
        fy = fy + 0.25 * (c00 + c01 - c10 - c11)
    ft = 0.25 * (sum(corners(a)) - sum(corners(b)))
    den = alpha ** 2 + fx * fx + fy * fy
    f = torch.stack([u, v])
    for _ in range(sweeps):
        p = _pad(f, 1, "reflect")
        m = (sum(_sh(p, 1, y, x) for y in (-1, 1) for x in (-1, 1)) / 12.0
             + sum(_sh(p, 1, y, x) for y, x in ((-1, 0), (1, 0), (0, -1), (0, 1))) / 6.0)
        d = (fx * m[0] + fy * m[1] + ft) / den
        f = torch.stack([m[0] - fx * d, m[1] - fy * d])
    return f[0], f[1]


def _x_liushen(a, b, U, V, h=10.0, most=60, tol=1e-8):
    i1, i2 = a / a.max(), b / b.max()
    p1, pe = _pad(i1, 1, "replicate"), _pad(i2 - i1, 1, "replicate")
    dy = lambda p: 0.5 * (_sh(p, 1, 1, 0) - _sh(p, 1, -1, 0))  # noqa: E731
    dx = lambda p: 0.5 * (_sh(p, 1, 0, 1) - _sh(p, 1, 0, -1))  # noqa: E731
    mm = lambda p: 0.25 * (_sh(p, 1, -1, -1) - _sh(p, 1, -1, 1) - _sh(p, 1, 1, -1) + _sh(p, 1, 1, 1))  # noqa: E731
    ring = [(y, x) for y in (-1, 0, 1) for x in (-1, 0, 1) if y or x]
    cnt = sum(_sh(_pad(torch.ones_like(i1), 1, "zero"), 1, y, x) for y, x in ring)
    iix, iiy, ii, ixt, iyt = i1 * dy(p1), i1 * dx(p1), i1 * i1, i1 * dy(pe), i1 * dx(pe)
    a11 = i1 * (_sh(p1, 1, -1, 0) - 2 * i1 + _sh(p1, 1, 1, 0) - 2 * i1) - h * cnt
    a22 = i1 * (_sh(p1, 1, 0, -1) - 2 * i1 + _sh(p1, 1, 0, 1) - 2 * i1) - h * cnt
    a12 = i1 * mm(p1)
    det = a11 * a22 - a12 * a12
    b11, b12, b22 = a22 / det, -a12 / det, a11 / det
    u, v = V, U  # row and column components
    for _ in range(most):
        pu, pv = _pad(u, 1, "replicate"), _pad(v, 1, "replicate")
        zu, zv = _pad(u, 1, "zero"), _pad(v, 1, "zero")
        bu = (2 * iix * dy(pu) + iix * dx(pv) + iiy * dy(pv) + ii * (_sh(pu, 1, -1, 0) + _sh(pu, 1, 1, 0)) + ii * mm(pv)
              + h * sum(_sh(zu, 1, y, x) for y, x in ring) + ixt)
        bv = (iiy * dy(pu) + iix * dx(pu) + 2 * iiy * dx(pv) + ii * mm(pu) + ii * (_sh(pv, 1, 0, -1) + _sh(pv, 1, 0, 1))
              + h * sum(_sh(zv, 1, y, x) for y, x in ring) + iyt)
        un, vn = -(b11 * bu + b12 * bv), -(b12 * bu + b22 * bv)
        err = (torch.linalg.norm(un - u) + torch.linalg.norm(vn - v)) / u.numel()
        u, v = un, vn
        if float(err) <= tol:
            break
    return v, u


def _x_bilinear(J, y, x):
    h, w = J.shape[-2:]
    y0, x0 = torch.floor(y), torch.floor(x)
    fy, fx = y - y0, x - x0
    ya, xa = y0.long(), x0.long()
    i = [(t.clamp(0, n - 1)) for t, n in ((ya, h), (ya + 1, h), (xa, w), (xa + 1, w))]
    g = lambda r, c: J[..., r, c]  # noqa: E731
    return ((1 - fy) * ((1 - fx) * g(i[0], i[2]) + fx * g(i[0], i[3])) + fy * ((1 - fx) * g(i[1], i[2]) + fx * g(i[1], i[3])))


def _x_lk(I, J, U, V, hw, steps=5):
    h, w = I.shape
    yy, xx = torch.meshgrid(torch.arange(h, device=I.device), torch.arange(w, device=I.device), indexing="ij")
    at = lambda P, y, x: P[y.clamp(0, h - 1), x.clamp(0, w - 1)]  # noqa: E731
    p = _pad(I, hw + 1, "replicate")
    q = hw + 1
    S = lambda y, x: _sh(p, q, y, x)  # noqa: E731
    offs = [(r, c) for r in range(-hw, hw + 1) for c in range(-hw, hw + 1)]

    def grad(r, c):
        gx = 3 * (S(r - 1, c + 1) + S(r + 1, c + 1) - S(r - 1, c - 1) - S(r + 1, c - 1)) + 10 * (S(r, c + 1) - S(r, c - 1))
        gy = 3 * (S(r + 1, c - 1) + S(r + 1, c + 1) - S(r - 1, c - 1) - S(r - 1, c + 1)) + 10 * (S(r + 1, c) - S(r - 1, c))
        return gx, gy

    a11 = a12 = a22 = torch.zeros_like(I)
    for r, c in offs:
        gx, gy = grad(r, c)
        a11, a12, a22 = a11 + gx * gx, a12 + gx * gy, a22 + gy * gy
    D = a11 * a22 - a12 * a12
    ok = D >= 1.192092896e-07
    D = torch.where(ok, D, torch.ones_like(D))
    px, py = xx + U, yy + V
    live = ok.clone()
    for _ in range(steps):
        live = live & ~((px < 0) | (px - hw >= w) | (py < 0) | (py - hw >= h))
        b1 = b2 = torch.zeros_like(I)
        for r, c in offs:
            gx, gy = grad(r, c)
            d = _x_bilinear(J, py + r, px + c) - S(r, c)
            b1, b2 = b1 + d * gx, b2 + d * gy
        dx, dy = 32 * (a12 * b2 - a22 * b1) / D, 32 * (a12 * b1 - a11 * b2) / D
        px, py = torch.where(live, px + dx, px), torch.where(live, py + dy, py)
        live = live & ~((dx.abs() < 0.01) & (dy.abs() < 0.01))
    return torch.where(ok, px - xx, U), torch.where(ok, py - yy, V)


def _half_kernel(n):
    """The Gaussian window of n taps, sigma = 0.15 n + 0.35 (centre first); 3 taps are 1/4, 1/2, 1/4."""
    if n == 3:
        return [0.5, 0.25]
    s = 0.15 * n + 0.35
    k = [math.exp(-0.5 * (j / s) ** 2) for j in range(n // 2 + 1)]
    t = k[0] + 2 * sum(k[1:])
    return [x / t for x in k]


def _x_blur(f, k):
    r = len(k) - 1
    p = _pad(f, r, "reflect")
    t = k[0] * p[..., r:-r, :] + sum(k[j] * (p[..., r - j:p.shape[-2] - r - j, :] + p[..., r + j:p.shape[-2] - r + j, :])
                                     for j in range(1, r + 1))
    n = p.shape[-1]
    return k[0] * t[..., r:-r] + sum(k[j] * (t[..., r - j:n - r - j] + t[..., r + j:n - r + j]) for j in range(1, r + 1))


def _x_farneback(a, b, U, V, window=33, n=7, sigma=1.5, iters=5):
    h, w = a.shape
    x = np.arange(-n, n + 1)
    g = np.exp(-x * x / (2 * sigma * sigma))
    g = g / g.sum()
    m2, m4, m22 = (g * x * x).sum(), (g * x ** 4).sum(), (g * x * x).sum() ** 2
    G = np.zeros((6, 6))
    G[0, 0], G[1, 1], G[2, 2], G[3, 3], G[4, 4], G[5, 5] = 1.0, m2, m2, m4, m4, m22
    G[0, 3] = G[0, 4] = G[3, 0] = G[4, 0] = m2
    G[3, 4] = G[4, 3] = m22
    iG = np.linalg.inv(G)

    def expand(f):
        p = _pad(_x_blur(f, [0.5, 0.25]), n, "replicate")
        rows = [sum(c * p[n + j:n + j + h, :] for j, c in zip(x, t)) for t in (g, g * x, g * x * x)]
        cols = lambda r, t: sum(c * r[:, n + j:n + j + w] for j, c in zip(x, t))  # noqa: E731
        b1, b2, b3 = cols(rows[0], g), cols(rows[0], g * x), cols(rows[1], g)
        b4, b5, b6 = cols(rows[0], g * x * x), cols(rows[2], g), cols(rows[1], g * x)
        return torch.stack([b3 * iG[1, 1], b2 * iG[1, 1], b1 * iG[0, 3] + b5 * iG[3, 3], b1 * iG[0, 3] + b4 * iG[3, 3],
                            b6 * iG[5, 5]])

    R0, R1 = expand(a), expand(b)
    yy, xx = torch.meshgrid(torch.arange(h, device=a.device), torch.arange(w, device=a.device), indexing="ij")
    bord = torch.tensor([0.14, 0.14, 0.4472, 0.4472, 0.4472, 1.0], dtype=torch.float64, device=a.device)
    edge = (bord[xx.clamp(max=5)] * bord[yy.clamp(max=5)] * bord[(w - 1 - xx).clamp(max=5)] * bord[(h - 1 - yy).clamp(max=5)])
    k = _half_kernel(window)

    def matrices(dx, dy):
        fx, fy = xx + dx, yy + dy
        x1, y1 = torch.floor(fx), torch.floor(fy)
        inside = (x1 >= 0) & (y1 >= 0) & (x1 < w - 1) & (y1 < h - 1)
        r = _x_bilinear(R1, torch.where(inside, fy, yy.double()), torch.where(inside, fx, xx.double()))
        r2, r3 = torch.where(inside, r[0], 0.0), torch.where(inside, r[1], 0.0)
        r4, r5 = (torch.where(inside, 0.5 * (R0[i] + r[i]), R0[i]) for i in (2, 3))
        r6 = torch.where(inside, 0.25 * (R0[4] + r[4]), 0.5 * R0[4])
        r2, r3 = 0.5 * (R0[0] - r2) + r4 * dy + r6 * dx, 0.5 * (R0[1] - r3) + r6 * dy + r5 * dx
        r2, r3, r4, r5, r6 = (t * edge for t in (r2, r3, r4, r5, r6))
        return torch.stack([r4 * r4 + r6 * r6, (r4 + r5) * r6, r5 * r5 + r6 * r6, r4 * r2 + r6 * r3, r6 * r2 + r5 * r3])

    for _ in range(iters):
        g11, g12, g22, h1, h2 = _x_blur(matrices(U, V), k)
        d = 1.0 / (g11 * g22 - g12 * g12 + 1e-3)
        U, V = (g11 * h2 - g12 * h1) * d, (g22 * h1 - g12 * h2) * d
    return U, V


def _x_half(img):
    """Pillow's bicubic resize to half size (sizes rounded to even) through one weight matrix per axis."""
    def weights(n):
        m = int(np.round(n * 0.5))
        s = n / m
        W = np.zeros((m, n))
        for i in range(m):
            c = (i + 0.5) * s
            lo, hi = max(int(c - 2 * s + 0.5), 0), min(int(c + 2 * s + 0.5), n)
            t = np.abs((np.arange(lo, hi) - c + 0.5) / s)
            k = np.where(t < 1, (1.5 * t - 2.5) * t * t + 1, np.where(t < 2, (((t - 5) * t + 8) * t - 4) * -0.5, 0.0))
            W[i, lo:hi] = k / k.sum()
        return torch.tensor(W, device=img.device)
    return weights(img.shape[0]) @ img @ weights(img.shape[1]).t()


def _x_spline(f, h, w):
    """The interpolating not-a-knot cubic spline of f at the h x w grid, one matrix per axis."""
    def matrix(n, N):
        A, B = np.zeros((n, n)), np.zeros((n, n))
        for i in range(1, n - 1):
            A[i, i - 1:i + 2] = 1, 4, 1
            B[i, i - 1:i + 2] = 6, -12, 6
        A[0, :3], A[-1, -3:] = (1, -2, 1), (1, -2, 1)
        M = np.linalg.solve(A, B)
        s = np.clip(np.arange(N) / N * n, 0, n - 1)
        i = np.minimum(np.floor(s).astype(int), n - 2)
        t = (s - i)[:, None]
        u = 1 - t
        E = np.eye(n)
        return torch.tensor(u * E[i] + t * E[i + 1] + ((u ** 3 - u) * M[i] + (t ** 3 - t) * M[i + 1]) / 6, device=f.device)
    return matrix(f.shape[0], h) @ f @ matrix(f.shape[1], w).t()


def _x_pyramid2(a, b, method, hw=13):
    """Two levels without warping: the coarse field, upsampled, starts the fine level, whose
    result is the answer."""
    U = V = None
    for level in (0, 1):
        x, y = (_x_half(a), _x_half(b)) if level == 0 else (a, b)
        h, w = x.shape
        if level == 0:
            U = V = torch.zeros_like(x)
        else:
            # Lucas-Kanade scales the field between intermediate levels only, Farneback at the last one
            sx, sy = (1.0, 1.0) if method == "lk" else (w / U.shape[1], h / U.shape[0])
            U, V = _x_spline(U, h, w) * sx, _x_spline(V, h, w) * sy
        if method == "lk":
            U, V = _x_lk(_x_prefilter(x, 2.0, 3), _x_prefilter(y, 2.0, 3), U, V, hw)
        else:
            U, V = _x_farneback(x, y, U, V)
            U, V = _x_liushen(_x_prefilter(x, 0.48, 5), _x_prefilter(y, 0.48, 5), U, V)
    return U, V


def _x_train(case, seed):
    """Loss, network output and gradients by autograd in float64 (weights rounded to bf16 as
    the tensor cores read them, activations not rounded)."""
    net = warmstart.WarmStartNet(seed=seed)
    host = net.params.double()
    W = {}
    for name, ci, co in warmstart.LAYERS:
        wo, bo, _, _ = net.off[name]
        k = host[wo:bo].reshape(3, 3, co, ci).permute(2, 3, 0, 1).bfloat16().double().contiguous().requires_grad_()
        W[name] = (k, host[bo:bo + co].clone().requires_grad_())
    F = torch.nn.functional
    cv = lambda name, t: F.relu(F.conv2d(t, *W[name], padding=1))  # noqa: E731
    up = lambda t: F.interpolate(t, scale_factor=2, mode="nearest")  # noqa: E731
    x = torch.stack([torch.stack([p.double() / p.double().max() for p in pair]) for pair in _train_frames(case, seed)])
    e0 = cv("c0b", cv("c0a", x.bfloat16().double()))
    e1 = cv("c1b", cv("c1a", F.avg_pool2d(e0, 2)))
    e2 = cv("c2b", cv("c2a", F.avg_pool2d(e1, 2)))
    e3 = cv("c3b", cv("c3a", F.avg_pool2d(e2, 2)))
    d = cv("d2", torch.cat([up(e3), e2], 1))
    d = cv("d1", torch.cat([up(d), e1], 1))
    d = cv("d0", torch.cat([up(d), e0], 1))
    out = F.conv2d(d, *W["head"], padding=1).permute(0, 2, 3, 1)
    loss = ((out - _train_label(case, seed).double()) ** 2).sum() / (2 * out.shape[0] * out.shape[1] * out.shape[2])
    loss.backward()
    grads = torch.cat([t for name, _, _ in warmstart.LAYERS
                       for t in (W[name][0].grad.permute(2, 3, 0, 1).reshape(-1), W[name][1].grad)])
    return loss.detach(), out.detach().contiguous(), grads


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mixed", "learned"):
        return None  # many whole pipelines: each method is compared on its own in the other cases
    if kind == "train":
        return _x_train(case, seed)
    if kind == "fbls_batch":
        if case["pairs"] * case["h"] * case["w"] > 9 << 20:
            return None
        return [_x_pyramid2(*(f.double() for f in _pair(case["h"], case["w"], seed * 1000 + i)), "fbls")
                for i in range(case["pairs"])]
    a, b = (f.double() for f in _pair(case["h"], case["w"], seed))
    if kind == "prefilter":
        return _x_prefilter(a, case["sigma"], case["taps"])
    if kind == "hs":
        z = torch.zeros_like(a)
        return _x_hs(_x_prefilter(a, 3.4, 3), _x_prefilter(b, 3.4, 3), z, z, case["sweeps"])
    if kind == "lk":
        return _x_pyramid2(a, b, "lk", case["half_window"])
    if kind == "fbls_call":
        return tuple(t.cpu().numpy() for t in _x_pyramid2(a, b, "fbls"))
    U, V = (t.double() for t in _field(case["h"], case["w"], seed))
    if kind == "lk_status":
        return (*_x_lk(a, b, U, V, case["half_window"]), None, None)
    if kind == "farneback":
        return _x_farneback(a, b, U, V, case["window"], case["poly"])
    return _x_liushen(a, b, U, V)
