"""The work that users of the prescalers have them do, as measurable cases.

A case is one call of the public interface: ``HookModel.upscale`` on planes in
device memory (one plane, planar colour, or a batch of frames),
``HookModel.upscale_host`` on frames in host memory, or ``prescale_frame`` on
a whole 4:2:0 frame.  Together the cases cover the families (ravu-lite, ravu,
ravu-zoom, ravu-3x, NNEDI3; luma / yuv / rgb; with and without anti-ringing),
both precision forms a player uses (plain FP32 planes, the call's default, and
FP16 planes in the fast form) and frames from a thumbnail to batches of 1080p.

Weights: the hook files' structure (window, key layout, thresholds) with
weights made here -- oriented interpolation kernels that vary smoothly with
the key, as trained RAVU tables do, and centred random neurons for NNEDI3.
Frames: sinusoids, hard edges and noise, made on the GPU from the seed.
"""
import dataclasses
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """The package (its folder's name is no module name), from the working folder."""
    name = "mpv_prescalers_gb300"
    if name not in sys.modules:
        root = os.path.join(os.getcwd(), "mpv-prescalers_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(root, "__init__.py"),
                                                      submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---------------------------------------------------------------- cases ----

def _case(name, model, w, h, frames=1, dtype="fp16", ow=0, oh=0, call="planes"):
    """`dtype`: of the planes; FP32 planes run the plain form (the default of
    the call), FP16 planes the fast form."""
    c = {"model": model, "w": w, "h": h, "frames": frames, "dtype": dtype, "ow": ow, "oh": oh, "call": call}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a thumbnail or a tile of a picture, default precision: the call itself is what costs
        _case("thumb-lite-r3-fp32", "ravu-lite-r3", 160, 90, dtype="fp32"),
        # one standard-definition plane in plain FP32, the parity form's own configuration
        _case("lite-r3-fp32-960x540", "ravu-lite-r3", 960, 540, dtype="fp32"),
        # a batch of 1080p frames with the heaviest 2x luma shader
        _case("lite-ar-r4-8x1080p", "ravu-lite-ar-r4", 1920, 1080, frames=8),
        # a player's 1080p -> 2160p luma frame through the two-pass lattice
        _case("ravu-r3-1080p", "ravu-r3", 1920, 1080),
        # 4:4:4 colour at the largest radius
        _case("ravu-r4-yuv-1080p", "ravu-r4-yuv", 1920, 1080),
        # RGB to an arbitrary window size, with anti-ringing
        _case("zoom-ar-r2-rgb-1080p", "ravu-zoom-ar-r2-rgb", 1920, 1080, ow=2880, oh=1620),
        # a cropped standard-definition plane (odd sizes) to a window of no simple ratio, plain FP32
        _case("zoom-r3-fp32-odd", "ravu-zoom-r3", 853, 479, dtype="fp32", ow=1501, oh=843),
        # 3x of a cropped 720p plane (odd sizes), plain FP32
        _case("3x-r3-fp32-odd", "ravu-3x-r3", 1279, 719, dtype="fp32"),
        # neural doubling of a batch of 720p planes on the tensor cores
        _case("nnedi3-128-8x6-4x720p", "nnedi3-nns128-win8x6", 1280, 720, frames=4),
        # neural doubling of one standard-definition plane with the call's default precision
        _case("nnedi3-64-8x4-fp32-480p", "nnedi3-nns64-win8x4", 854, 480, dtype="fp32"),
        # a software decoder's frames: host memory in, host memory out
        _case("host-lite-ar-r3-4x720p", "ravu-lite-ar-r3", 1280, 720, frames=4, call="host"),
        # a whole 4:2:0 frame: chroma merged, chain, shift corrected
        _case("frame420-ravu-r3-yuv-720p", "ravu-r3-yuv", 1280, 720, call="frame"),
    ]


_DRAWN = (
    ["ravu-lite-r2", "ravu-lite-r3", "ravu-lite-r4", "ravu-lite-ar-r2", "ravu-lite-ar-r3", "ravu-lite-ar-r4"]
    + ["ravu-r%d%s" % (r, s) for r in (2, 3, 4) for s in ("", "-yuv", "-rgb")]
    + ["ravu-3x-r%d%s" % (r, s) for r in (2, 3, 4) for s in ("", "-rgb")]
    + ["ravu-zoom-r2", "ravu-zoom-r3", "ravu-zoom-ar-r2", "ravu-zoom-ar-r2-rgb", "ravu-zoom-r3-yuv"]
    + ["nnedi3-nns%d-win8x%d" % (n, k) for n in (16, 32, 64, 128, 256) for k in (4, 6)]
)


def draw(rng):
    """A model, a size spread over its logarithm (odd ones among them), a
    count of frames and a form; no heavier than the heaviest listed case."""
    most_b = max(work(c)["bytes"] for c in listed())
    most_f = max(work(c)["flops"] for c in listed())
    while True:
        model = rng.choice(_DRAWN)
        w = int(round(math.exp(rng.uniform(math.log(64), math.log(2560)))))
        h = max(36, int(round(w * rng.choice([9 / 16, 3 / 4, 9 / 21, 16 / 9]) * rng.uniform(0.9, 1.1))))
        s = rng.uniform(1.1, 3.0)
        zoom = "zoom" in model
        call = "planes"
        frames = rng.choice([1, 1, 1, 2, 3, 5])
        if rng.random() < 0.15:
            call = "host"
        elif model.startswith("ravu-r") and model.endswith("-yuv") and rng.random() < 0.4:
            call, frames, w, h = "frame", 1, w & ~1, h & ~1
        c = _case(None, model, w, h, frames, rng.choice(["fp16", "fp16", "fp32"]),
                  int(math.ceil(w * s)) if zoom else 0, int(math.ceil(h * s)) if zoom else 0, call)
        k = work(c)
        if k["bytes"] <= most_b and k["flops"] <= most_f:
            return c


# -------------------------------------------------------------- geometry ---

def _info(name):
    if name.startswith("nnedi3"):
        a, b = name.split("-nns")[1].split("-win8x")
        return {"family": "nnedi3", "nns": int(a), "win_h": int(b), "ch": 1, "channels": "luma", "scale": 2}
    fam = next((f for f in ("lite", "zoom", "3x") if "-" + f in name), "ravu")
    channels = name.rsplit("-", 1)[1] if name.endswith(("-yuv", "-rgb")) else "luma"
    r = next(k for k in (2, 3, 4) if "-r%d" % k in name)
    n = 2 * r - 1 if fam in ("lite", "3x") else 2 * r
    strength = {"ravu": ("log2", 2000.0, 8.0), "3x": ("thr", (0.005, 0.02))}.get(fam, ("thr", (0.004, 0.016, 0.05)))
    ns = int(strength[2]) + 1 if strength[0] == "log2" else len(strength[1]) + 1
    return {"family": fam, "r": r, "n": n, "ch": 1 if channels == "luma" else 3, "channels": channels,
            "ar": 0.8 if "-ar" in name else 0.0, "strength": strength, "ns": ns, "rows": 24 * ns * 3,
            "scale": 3 if fam == "3x" else 2}


def _out_size(case):
    i = _info(case["model"])
    if i["family"] == "zoom":
        return case["ow"], case["oh"]
    return i["scale"] * case["w"], i["scale"] * case["h"]


def work(case):
    """Planes read and written once; the arithmetic of the shaders' own steps
    (a fused multiply-add counts 2)."""
    i = _info(case["model"])
    es = 4 if case["dtype"] == "fp32" else 2
    px, (ow, oh) = case["w"] * case["h"] * case["frames"], _out_size(case)
    opx = ow * oh * case["frames"]
    in_ch = 1.5 if case["call"] == "frame" else i["ch"]
    nbytes = es * (in_ch * px + i["ch"] * opx)
    if i["family"] == "nnedi3":
        t = 8 * i["win_h"]
        return {"bytes": nbytes, "flops": 3 * px * (2.0 * t * 2 * i["nns"] + 8 * i["nns"] + 7 * t)}
    s, n, c = i["n"] ** 2, i["n"], i["ch"]
    key = 13 * (s if n <= 4 else (n - 2) ** 2) + 35
    if i["family"] == "lite":
        taps = s if i["r"] == 2 else 13
        fl = px * (key + 8 * s + (48 * taps + 32 if i["ar"] else 0))
    elif i["family"] == "3x":
        fl = px * (key + 16 * s * c)
    elif i["family"] == "ravu":
        fl = 3 * px * (key + 1.5 * s * c)
    else:
        fl = opx * (key + 12 * s + 2 * s * c + (12 * s + 20 * s * c if i["ar"] else 0))
    if case["call"] == "frame":
        fl += 2 * px * 8 + 3 * opx * 40
    return {"bytes": float(nbytes), "flops": float(fl)}


# --------------------------------------------------------------- weights ---

def _grad_weights(i):
    """Gaussian exp(-d^2 / 8) over the gradient points, summing to 1."""
    n = i["n"]
    p = np.arange(n) if n <= 4 else np.arange(1, n - 1)
    q = (p - (n - 1) / 2.0) ** 2
    w = np.exp(-(q[:, None] + q[None, :]) / 8.0).ravel()
    return w / w.sum()


def _kernels(i, dx, dy):
    """[rows][...] values of every key's kernel at positions (dx, dy) from the
    target: a Gaussian drawn out along the key's edge (more so where it is
    coherent) with a negative ring."""
    a, s, c = np.meshgrid(np.arange(24), np.arange(i["ns"]), np.arange(3), indexing="ij")
    th = ((a + 0.5) * np.pi / 24).ravel()
    along = (0.52 + 0.16 * c + 0.08 * s / i["ns"]).ravel()
    sh = (slice(None),) + (None,) * np.ndim(dx)
    u = np.cos(th)[sh] * dx + np.sin(th)[sh] * dy          # across the edge
    v = -np.sin(th)[sh] * dx + np.cos(th)[sh] * dy         # along it
    r2 = dx ** 2 + dy ** 2
    core = np.exp(-u ** 2 / (2 * 0.5 ** 2) - v ** 2 / (2 * along[sh] ** 2))
    return core, core - 0.08 * np.exp(-r2 / (2 * 1.5 ** 2))


def _lut(i):
    """(LUT, anti-ringing LUT or None): float32 [rows][columns][4] as the hook files embed them."""
    n, s, r = i["n"], i["n"] ** 2, i["r"]
    k = np.arange(s)
    lo = 0.0 if i["family"] in ("lite", "3x") else 0.5
    tx, ty = k // n - (r - 1) - lo, k % n - (r - 1) - lo
    if i["family"] in ("lite", "3x"):
        offs = ([(-.25, -.25), (-.25, .25), (.25, -.25), (.25, .25)] if i["family"] == "lite" else
                [(x / 3, y / 3) for x in (-1, 0, 1) for y in (-1, 0, 1) if (x, y) != (0, 0)])
        ox, oy = np.array(offs).T
        w = _kernels(i, tx[:, None] - ox, ty[:, None] - oy)[1]           # [rows][s][outputs]
        w = (w / w.sum(1, keepdims=True))[:, : s // 2 + 1]
        return w.reshape(i["rows"], -1, 4).astype(np.float32), None
    if i["family"] == "ravu":
        w = _kernels(i, tx, ty)[1]
        w = w / w.sum(1, keepdims=True)
        cols = (s // 2 + 3) // 4
        out = np.zeros((i["rows"], 4 * cols))
        out[:, : s // 2] = w[:, : s // 2]
        return out.reshape(i["rows"], cols, 4).astype(np.float32), None
    nb, sub = (s // 2 + 3) // 4, np.arange(9) / 8.0
    px = (tx + 0.5)[None, None, :] - sub[None, :, None]                   # [jy][jx][tap]
    py = (ty + 0.5)[None, None, :] - sub[:, None, None]
    px, py = np.broadcast_arrays(px, py)
    core, w = _kernels(i, px, py)                                         # [rows][9][9][s]
    w = w / w.sum(-1, keepdims=True)

    def texels(x):
        full = np.zeros(x.shape[:3] + (4 * nb,))
        full[..., : s // 2] = x[..., : s // 2]
        full = full.reshape(i["rows"], 9, 9, nb, 4).transpose(0, 1, 3, 2, 4)
        return np.ascontiguousarray(full.reshape(i["rows"] * 9, nb * 9, 4), dtype=np.float32)

    return texels(w), texels(core ** 3) if i["ar"] else None


_WEIGHTS = {}


def _weights(name):
    if name not in _WEIGHTS:
        i = _info(name)
        if i["family"] == "nnedi3":
            rng, t = np.random.default_rng(i["nns"] * 8 + i["win_h"]), 8 * i["win_h"]
            a, b = (rng.normal(0.0, sd, size=(t, i["nns"])) for sd in (0.3, 0.2))
            _WEIGHTS[name] = {"a": (a - a.mean(0)).astype(np.float32), "b": (b - b.mean(0)).astype(np.float32),
                              "ba": rng.normal(0, 1.0, i["nns"]).astype(np.float32),
                              "bb": rng.normal(0, 0.5, i["nns"]).astype(np.float32)}
        else:
            lut, lut_ar = _lut(i)
            _WEIGHTS[name] = {"lut": lut, "lut_ar": lut_ar, "gw": _grad_weights(i)}
    return _WEIGHTS[name]


_MODELS = {}


def _model(name):
    """The loaded model: a program loads its hook file once and keeps it on the device."""
    if name not in _MODELS:
        pkg, w, i = _package(), _weights(name), _info(name)
        from mpv_prescalers_gb300 import synth
        m = synth.synthetic_model(name)
        if i["family"] == "nnedi3":
            m = dataclasses.replace(m, weights_a=w["a"], weights_b=w["b"], bias_a=w["ba"], bias_b=w["bb"])
        else:
            m = dataclasses.replace(m, lut=w["lut"], lut_ar=w["lut_ar"], grad_weights=w["gw"], ar=i["ar"],
                                    strength=i["strength"], coherence=(0.25, 0.5))
        _MODELS[name] = pkg.HookModel(m)
        _MODELS[name].device_handle()
    return _MODELS[name]


# ---------------------------------------------------------------- frames ---

def _plane(h, w, seed, dtype):
    """One [h][w] CUDA plane in [0, 1]: 8 sinusoids, 16 flat ellipses and half
    planes with hard edges, noise of sigma 0.01."""
    rng = np.random.default_rng(seed)
    y = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    x = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    img = torch.full((h, w), 0.5, device="cuda")
    for _ in range(8):
        phi, psi = rng.uniform(0, math.pi), rng.uniform(0, 2 * math.pi)
        k = 2 * math.pi / math.exp(rng.uniform(math.log(4), math.log(64)))
        img += rng.uniform(0.02, 0.1) * torch.sin(k * (x * math.cos(phi) + y * math.sin(phi)) + psi)
    for _ in range(16):
        cx, cy, phi = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(0, math.pi)
        ra, rb = rng.uniform(4, 0.3 * min(w, h), 2)
        u = (x - cx) * math.cos(phi) + (y - cy) * math.sin(phi)
        v = (y - cy) * math.cos(phi) - (x - cx) * math.sin(phi)
        inside = (u / ra) ** 2 + (v / rb) ** 2 < 1
        if rng.random() < 0.3:
            inside &= u > 0
        img = torch.where(inside, torch.full_like(img, rng.uniform(0, 1)), img)
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))
    img += 0.01 * torch.randn((h, w), device="cuda", generator=g)
    return img.clamp_(0, 1).to(torch.float32 if dtype == "fp32" else torch.float16)


def _inputs(case, seed):
    """[frames][channels][h][w], or the three planes of a 4:2:0 frame."""
    w, h, dt, ch = case["w"], case["h"], case["dtype"], _info(case["model"])["ch"]
    if case["call"] == "frame":
        return [_plane(h, w, 10 * seed, dt)] + [_plane(h // 2, w // 2, 10 * seed + k, dt) for k in (1, 2)]
    out = torch.empty((case["frames"], ch, h, w), device="cuda",
                      dtype=torch.float32 if dt == "fp32" else torch.float16)
    for f in range(case["frames"]):
        for c in range(ch):
            out[f, c] = _plane(h, w, 1000 * seed + 10 * f + c, dt)
    return out


def prepare(case, seed):
    m, x = _model(case["model"]), _inputs(case, seed)
    state = {"case": case, "model": m, "precision": "fp32" if case["dtype"] == "fp32" else "fast",
             "out_size": _out_size(case) if _info(case["model"])["family"] == "zoom" else None}
    if case["call"] == "host":
        ow, oh = _out_size(case)
        state["x"] = x.cpu().pin_memory()
        state["out"] = torch.empty(x.shape[:2] + (oh, ow), dtype=x.dtype, pin_memory=True)
    elif case["call"] == "frame":
        state["x"] = _package().Frame(x, "yuv", "left")
    else:   # one plane [H][W], planar colour [C][H][W] or a batch [N][C][H][W]
        state["x"] = x if case["frames"] > 1 else (x[0, 0] if x.shape[1] == 1 else x[0])
    return state


def run(state):
    m, p = state["model"], state["precision"]
    call = state["case"]["call"]
    if call == "host":
        return m.upscale_host(state["x"], out=state["out"], out_size=state["out_size"], precision=p)
    if call == "frame":
        return _package().prescale_frame(m, state["x"], precision=p).planes
    if state["out_size"] is not None:
        return m.upscale(state["x"], out_size=state["out_size"], precision=p)
    return m.upscale(state["x"], precision=p)


# ----------------------------------------------------------------- exact ---
# The shaders' arithmetic in 64 bits, in bands of rows (plain torch).

_EPS = 1.192092896e-7


def _fetch(p, ys, xs):
    return p[..., ys.clamp(0, p.shape[-2] - 1), xs.clamp(0, p.shape[-1] - 1)]


def _deriv(s, n, four, p):
    if p == 0:
        return s(1) - s(0)
    if p == n - 1:
        return s(n - 1) - s(n - 2)
    if four and 2 <= p <= n - 3:
        return (-s(p + 2) + 8.0 * s(p + 1) - 8.0 * s(p - 1) + s(p - 2)) / 12.0
    return (s(p + 1) - s(p - 1)) / 2.0


def _key(lum, i, gw):
    """The table row of each window stack lum[k] (grid (k // n, k % n))."""
    n, four = i["n"], i["family"] in ("ravu", "zoom")
    a = b = d = torch.zeros_like(lum[0])
    pts, k = (range(n) if n <= 4 else range(1, n - 1)), 0
    for px in pts:
        for py in pts:
            gx = _deriv(lambda q: lum[q * n + py], n, four, px)
            gy = _deriv(lambda q: lum[px * n + q], n, four, py)
            a, b, d, k = a + gx * gx * gw[k], b + gx * gy * gw[k], d + gy * gy * gw[k], k + 1
    t = a + d
    delta = (t * t / 4 - (a * d - b * b)).clamp_min(0).sqrt()
    l1, l2 = t / 2 + delta, t / 2 - delta
    r1, r2 = l1.sqrt(), l2.sqrt()
    th = torch.atan2(l1 - a, b) + math.pi
    th = torch.where(b.abs() < _EPS, torch.zeros_like(th), th - math.pi * torch.floor(th / math.pi))
    mu = torch.where(r1 + r2 < _EPS, torch.zeros_like(th), (r1 - r2) / (r1 + r2))
    st = i["strength"]
    if st[0] == "log2":
        strength = torch.floor(torch.log2(r1 * st[1] + _EPS)).clamp(0, st[2])
    else:
        strength = sum((r1 >= v).to(r1.dtype) for v in st[1])
    coh = (mu >= 0.25).to(r1.dtype) + (mu >= 0.5).to(r1.dtype)
    key = (torch.floor(th * 24 / math.pi) * i["ns"] + strength) * 3 + coh
    return key.to(torch.int64)


def _luma(v, i):
    return 0.2126 * v[0] + 0.7152 * v[1] + 0.0722 * v[2] if i["channels"] == "rgb" else v[0]


def _ar_finish(res, sums, strength):
    lo, hi, lo2, hi2 = sums
    c = torch.minimum(torch.maximum(res, 1.1 - lo2 / lo), hi2 / hi - 0.1)
    return res * (1 - strength) + c * strength


def _powers(v):
    return (1.1 - v) ** 32, (0.1 + v) ** 32, (1.1 - v) ** 33, (0.1 + v) ** 33


def _window(x, i, ys, xs):
    n, r = i["n"], i["r"]
    return [_fetch(x, ys + (k % n - (r - 1)), xs + (k // n - (r - 1))) for k in range(n * n)]


def _exact_lite_3x(x, i, w, y0, y1):
    """2x2 (lite) or 3x3 outputs of input rows y0..y1: [C][scale*rows][scale*W]."""
    c, _, width = x.shape
    ys = torch.arange(y0, y1, device=x.device)[:, None]
    xs = torch.arange(width, device=x.device)[None, :]
    vals, s, lut = _window(x, i, ys, xs), i["n"] ** 2, w["lut"]
    row = _key([_luma(v, i) for v in vals], i, w["gw"]).clamp(0, i["rows"] - 1)
    no = 4 if i["family"] == "lite" else 8
    lut = lut.reshape(i["rows"], s // 2 + 1, no)
    res = [0.0] * no
    sums = [[0.0] * 4 for _ in range(no)]
    for t in range(s // 2 + 1):
        wt = lut[:, t][row]
        n, r = i["n"], i["r"]
        ar = i["ar"] and (r == 2 or abs(t // n - (r - 1)) + abs(t % n - (r - 1)) <= 2)
        sides = [(vals[t], list(range(no)))]
        if t < s // 2:
            sides.append((vals[s - 1 - t], list(range(no - 1, -1, -1))))
        for v, order in sides:
            pw = _powers(v) if ar else None
            for k in range(no):
                res[k] = res[k] + v * wt[..., order[k]]
                if ar:
                    g = wt[..., order[k]].clamp_min(0)
                    sums[k] = [q + p * g for q, p in zip(sums[k], pw)]
    out = torch.empty((c, (y1 - y0) * i["scale"], width * i["scale"]), dtype=x.dtype, device=x.device)
    if i["family"] == "lite":
        for k, (dx, dy) in enumerate(((0, 0), (0, 1), (1, 0), (1, 1))):
            out[:, dy::2, dx::2] = _ar_finish(res[k], sums[k], i["ar"]) if i["ar"] else res[k].clamp(0, 1)
    else:
        out[:, 1::3, 1::3] = vals[s // 2]
        for k, (dx, dy) in enumerate([(a, b) for a in range(3) for b in range(3) if (a, b) != (1, 1)]):
            out[:, dy::3, dx::3] = res[k].clamp(0, 1)
    return out


def _ravu_pass(vals, i, w):
    row = _key([_luma(v, i) for v in vals], i, w["gw"]).clamp(0, i["rows"] - 1)
    s, lut = i["n"] ** 2, w["lut"].reshape(i["rows"], -1)
    return sum((vals[k] + vals[s - 1 - k]) * lut[:, k][row] for k in range(s // 2)).clamp(0, 1)


def _exact_ravu(x, i, w):
    """The lattice chain of one frame [C][H][W]: int11, then int10 and int01."""
    c, h, width = x.shape
    xs = torch.arange(width, device=x.device)[None, :]
    bands = [torch.arange(y, min(h, y + 135), device=x.device)[:, None] for y in range(0, h, 135)]
    i11 = torch.cat([_ravu_pass(_window(x, i, ys, xs), i, w) for ys in bands], 1)
    out = torch.empty((c, 2 * h, 2 * width), dtype=x.dtype, device=x.device)
    out[:, 0::2, 0::2], out[:, 1::2, 1::2] = x, i11
    n = i["n"]
    for ys in bands:
        rows = slice(int(ys[0]), int(ys[-1]) + 1)
        for second in (0, 1):
            vals = []
            for k in range(n * n):
                s, d = k // n + k % n - (n - 1), k % n - k // n
                even = s % 2 == 0
                if not second:
                    src, dx, dy = (i11, s // 2, (d - 1) // 2) if even else (x, (s + 1) // 2, d // 2)
                else:
                    src, dx, dy = (x, s // 2, (d + 1) // 2) if even else (i11, (s - 1) // 2, d // 2)
                vals.append(_fetch(src, ys + dy, xs + dx))
            r = _ravu_pass(vals, i, w)
            if second:
                out[:, 1::2, 0::2][:, rows] = r
            else:
                out[:, 0::2, 1::2][:, rows] = r
    return out


def _exact_zoom(x, i, w, ow, oh, y0, y1):
    c, h, width = x.shape

    def pos(k, n_in, n_out):
        num = (2 * k + 1) * n_in - n_out
        q = torch.div(num, 2 * n_out, rounding_mode="floor")
        return q, (num - q * 2 * n_out).to(x.dtype) / (2 * n_out)

    iy, sy = pos(torch.arange(y0, y1, device=x.device)[:, None], h, oh)
    ix, sx = pos(torch.arange(ow, device=x.device)[None, :], width, ow)
    vals, s = _window(x, i, iy, ix), i["n"] ** 2
    key = _key([_luma(v, i) for v in vals], i, w["gw"])

    def bilinear(lut, blk, fx, fy):
        tx, ty = blk * 9 + 8 * fx, key * 9 + 8 * fy
        x0, yy0 = torch.floor(tx), torch.floor(ty)
        ax, ay = (tx - x0)[..., None], (ty - yy0)[..., None]
        rows, cols = lut.shape[:2]
        xa, ya = x0.to(torch.int64).clamp(0, cols - 1), yy0.to(torch.int64).clamp(0, rows - 1)
        xb, yb = (xa + 1).clamp(max=cols - 1), (ya + 1).clamp(max=rows - 1)
        top = lut[ya, xa.expand_as(ya)] * (1 - ax) + lut[ya, xb.expand_as(ya)] * ax
        bot = lut[yb, xa.expand_as(ya)] * (1 - ax) + lut[yb, xb.expand_as(ya)] * ax
        return top * (1 - ay) + bot * ay

    res, sums = 0.0, [0.0] * 4
    for blk in range((s // 2 + 3) // 4):
        ws, wi = bilinear(w["lut"], blk, sx, sy), bilinear(w["lut"], blk, 1 - sx, 1 - sy)
        if i["ar"]:
            gs, gi = bilinear(w["lut_ar"], blk, sx, sy), bilinear(w["lut_ar"], blk, 1 - sx, 1 - sy)
        for j in range(4):
            k = blk * 4 + j
            if k >= s // 2:
                break
            res = res + vals[k] * ws[..., j] + vals[s - 1 - k] * wi[..., j]
            if i["ar"]:
                for v, g in ((vals[k], gs[..., j]), (vals[s - 1 - k], gi[..., j])):
                    sums = [q + p * g for q, p in zip(sums, _powers(v))]
    return _ar_finish(res, sums, i["ar"]) if i["ar"] else res.clamp(0, 1)


def _exact_double(x, i, w, transpose):
    """One NNEDI3 doubling pass of [H][W] along rows (or columns)."""
    p = x.t().contiguous() if transpose else x
    h, width = p.shape
    kh = i["win_h"]
    xs = torch.arange(width, device=x.device)[None, :]
    out = torch.empty((2 * h, width), dtype=x.dtype, device=x.device)
    out[0::2] = p
    rows = max(1, (1 << 19) // width)
    for y in range(0, h, rows):
        ys = torch.arange(y, min(h, y + rows), device=x.device)[:, None]
        win = torch.stack([_fetch(p, ys + dy, xs + dx) for dy in range(-(kh // 2 - 1), kh // 2 + 1)
                           for dx in range(-3, 5)], -1)
        mean = win.mean(-1)
        cent = win - mean[..., None]
        var = (cent * cent).mean(-1)
        inv = torch.where(var >= _EPS, var.clamp_min(1e-300).rsqrt(), torch.zeros_like(var))
        s1 = (win @ w["a"]) * inv[..., None] + w["ba"]
        s2 = (win @ w["b"]) * inv[..., None] + w["bb"]
        e = torch.exp(s1)
        v = (e * s2 / (1 + s2.abs())).sum(-1) / e.sum(-1)
        out[1::2][y:y + rows] = (mean + 5 * v * var * inv).clamp(0, 1)
    return out.t() if transpose else out


def _exact_frame(x, case, i, w):
    """The chain on one frame [C][H][W] (float64)."""
    h = x.shape[1]
    if i["family"] == "nnedi3":
        return _exact_double(_exact_double(x[0], i, w, False), i, w, True)[None]
    if i["family"] == "ravu":
        return _exact_ravu(x, i, w)
    if i["family"] == "zoom":
        return torch.cat([_exact_zoom(x, i, w, case["ow"], case["oh"], y, min(case["oh"], y + 135))
                          for y in range(0, case["oh"], 135)], 1)
    return torch.cat([_exact_lite_3x(x, i, w, y, min(h, y + 135)) for y in range(0, h, 135)], 1)


def _resample(p, ow, oh, sx, ox, sy, oy, cubic):
    """Separable interpolation at (sx * x + ox, sy * y + oy), edges replicated."""
    def axis(p, n_out, s, o, dim):
        u = s * torch.arange(n_out, device=p.device, dtype=p.dtype) + o
        k = torch.floor(u)
        t = u - k
        k = k.to(torch.int64)
        if cubic:
            w = [(-t ** 3 + 2 * t ** 2 - t) / 2, (3 * t ** 3 - 5 * t ** 2 + 2) / 2,
                 (-3 * t ** 3 + 4 * t ** 2 + t) / 2, (t ** 3 - t ** 2) / 2]
        else:
            w = [1 - t, t]
        shape = [1, 1]
        shape[dim] = n_out
        return sum(wt.reshape(shape) * p.index_select(dim, (k + j - (1 if cubic else 0)).clamp(0, p.shape[dim] - 1))
                   for j, wt in enumerate(w))
    return axis(axis(p, oh, sy, oy, 0), ow, sx, ox, 1)


def exact(case, seed):
    i, x = _info(case["model"]), _inputs(case, seed)
    w = {k: None if v is None else torch.as_tensor(v, device="cuda").to(torch.float64)
         for k, v in _weights(case["model"]).items()}
    if case["call"] == "frame":
        width, h = case["w"], case["h"]
        planes = [x[0].double()] + [_resample(c.double(), width, h, 0.5, 0.0, 0.5, -0.25, False) for c in x[1:]]
        up = _exact_frame(torch.stack(planes), case, i, w)
        return [_resample(p, 2 * width, 2 * h, 1.0, -0.5, 1.0, -0.5, True) for p in up]
    out = torch.stack([_exact_frame(f.double(), case, i, w) for f in x])
    if case["call"] == "host" or case["frames"] > 1:
        return out
    return out[0, 0] if out.shape[1] == 1 else out[0]
