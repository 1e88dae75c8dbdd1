"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (images in
host memory, or an engine with the pair's features resident), ``run`` is one pass through the public
entry points of ``zcmir_b200``, ``exact`` the same outputs in float64 by plain torch.

Kinds (``case["kind"]``):

* ``score``     Engine.score of one pose on a resident pair: what an outer optimiser or a viewer
                calls for each pose it tries.
* ``gradient``  Engine.gradient with the Gauss–Newton matrix: one step of an outer optimiser.
* ``refine``    Engine.refine_poses: the batched Gauss–Newton from several seeds (proposals).
* ``map``       Engine.set_images + Engine.shift_map of a new pair with the map read back: the
                translation search of one pair, from host images to the score of every shift.
* ``auto``      the same with uint8 images and every setting at its default (CLAHE, f16 texels, the
                automatic map of at most 512 × 512 shifts): what a first-time user runs.
* ``stack``     Engine.stack_maps along slices of uneven sizes (serial sections, time series).
* ``search``    Engine.set_images + Engine.search: the rotation × scale sweep, its Gauss–Newton
                screen and finalists, from host images to the pose.
* ``propose``   zcmir_b200.cnn.forward: the pose network's logits for a batch of pairs.

Pairs are a smooth blob-and-grating field (modality A) against its inverted nonlinear remap or its
8-level segmentation (modality B), the moving one under a known similarity, with noise, quantised to
16 (``auto``: 8) bits: the value distributions of ``zcmir_b200.synth``, made on the GPU.
"""
import math

import numpy as np
import torch

from zcmir_b200 import Engine, cnn

F64 = torch.float64


def listed():
    return [
        # one pose score of a small pair: launches and latency
        {"name": "score_256", "kind": "score", "mw": 256, "mh": 256, "fw": 256, "fh": 256, "mode": "laplacian"},
        # one optimiser step on an ordinary pair
        {"name": "gradient_512", "kind": "gradient", "mw": 512, "mh": 512, "fw": 512, "fh": 512, "mode": "laplacian"},
        # proposal seeds refined together, ragged sizes
        {"name": "refine_497x377", "kind": "refine", "mw": 497, "mh": 377, "fw": 451, "fh": 389, "mode": "laplacian",
         "poses": 8, "iters": 10},
        # the small translation map (the 256² workload of the tests and the synthetic inputs)
        {"name": "map_256", "kind": "map", "mw": 256, "mh": 256, "fw": 256, "fh": 256, "mode": "laplacian", "cap": 512,
         "calibrated": False, "turn": 0.0, "want_map": True},
        # ragged sizes, three features, a rotated prior: the canvas and its FFT lengths are odd ones
        {"name": "map_487x391_turned", "kind": "map", "mw": 487, "mh": 391, "fw": 531, "fh": 413, "mode": "three",
         "cap": 2048, "calibrated": False, "turn": 4.0, "want_map": True},
        # the headline map: 1024², 2048² shifts, 45 correlations, calibrated; the pose is what is read
        {"name": "map_1024_calibrated", "kind": "map", "mw": 1024, "mh": 1024, "fw": 1024, "fh": 1024,
         "mode": "laplacian", "cap": 2048, "calibrated": True, "turn": 0.0, "want_map": False},
        # an ordinary pair at a rotated prior with the whole map read back
        {"name": "map_611x747_turned", "kind": "map", "mw": 611, "mh": 747, "fw": 683, "fh": 702, "mode": "laplacian",
         "cap": 2048, "calibrated": False, "turn": 2.0, "want_map": True},
        # the largest map: a 2 k × 1.5 k micrograph pair at full resolution
        {"name": "map_2013x1507", "kind": "map", "mw": 2013, "mh": 1507, "fw": 2013, "fh": 1507, "mode": "laplacian",
         "cap": 4096, "calibrated": False, "turn": 0.0, "want_map": False},
        # the default call on 8-bit images
        {"name": "auto_1024x768", "kind": "auto", "mw": 1024, "mh": 768, "fw": 1024, "fh": 768, "turn": 0.0},
        # serial sections of 384 to 1024 px
        {"name": "stack_10", "kind": "stack", "slices": 10, "lo": 384, "hi": 1024, "mode": "laplacian"},
        # the full rotation × scale search (360 rotations × 9 scales) of a 512² pair
        {"name": "search_512_3240", "kind": "search", "mw": 512, "mh": 512, "fw": 512, "fh": 512, "mode": "laplacian",
         "rotations": 360, "scales": 9},
        # the pose network on a batch of pairs
        {"name": "propose_64", "kind": "propose", "pairs": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: sizes log-uniform, odd ones among them."""
    kind = rng.choice(["score", "gradient", "refine", "map", "map", "map", "auto", "stack", "search", "propose"])
    mode = rng.choice(["laplacian", "laplacian", "three", "cubic"])
    if kind == "propose":
        return {"kind": kind, "pairs": _log(rng, 2, 64)}
    if kind == "stack":
        return {"kind": kind, "slices": rng.randint(3, 10), "lo": _log(rng, 128, 384), "hi": _log(rng, 400, 1024), "mode": mode}
    hi = {"score": 1200, "gradient": 1200, "refine": 512, "map": 1400, "auto": 1600, "search": 512}[kind]
    mw = _log(rng, 128, hi)
    aspect = lambda: rng.uniform(0.75, 1.33)
    mh = max(96, min(hi, int(mw * aspect())))
    c = {"kind": kind, "mw": mw, "mh": mh}
    # half the pairs share a size (one camera), half are ragged
    if rng.random() < 0.5:
        c["fw"], c["fh"] = mw, mh
    else:
        c["fw"], c["fh"] = (max(96, min(hi, int(v * rng.uniform(0.85, 1.18)))) for v in (mw, mh))
    if kind != "auto":
        c["mode"] = mode
    if kind in ("map", "auto"):
        c["turn"] = 0.0 if rng.random() < 0.5 else rng.uniform(-8.0, 8.0)
    if kind == "map":
        big = max(c["mw"], c["fw"], c["mh"], c["fh"]) > 640
        c.update(cap=4096 if big else 2048, calibrated=big and rng.random() < 0.5, want_map=not big)
    if kind == "refine":
        c.update(poses=rng.randint(1, 8), iters=rng.randint(4, 10))
    if kind == "search":
        c.update(rotations=rng.choice([36, 90, 180, 360]), scales=rng.choice([3, 5, 9]))
    return c


# ── inputs ───────────────────────────────────────────────────────────────────────────────────

def _mat(rows):
    return np.array(rows, np.float64)


def _similarity(cm, cf, deg, scale, tx, ty):
    """Moving → fixed (1-based): turn and scale about the moving centre, onto the fixed centre, shift."""
    c, s = scale * math.cos(math.radians(deg)), scale * math.sin(math.radians(deg))
    T = lambda x, y: _mat([[1, 0, x], [0, 1, y], [0, 0, 1]])
    return T(cf[0] + tx, cf[1] + ty) @ _mat([[c, -s, 0], [s, c, 0], [0, 0, 1]]) @ T(-cm[0], -cm[1])


def _field(w, h, pad, rng):
    """Blobs and two gratings over the w × h frame with `pad` pixels around it, in [0, 1] (float64, GPU)."""
    W, H = w + 2 * pad, h + 2 * pad
    k = int(64 * W * H / 65536.0) + 8
    x = torch.arange(W, dtype=F64, device="cuda")
    y = torch.arange(H, dtype=F64, device="cuda")
    on = lambda a: torch.as_tensor(a, dtype=F64, device="cuda")
    sg = on(rng.uniform(4, 20, k))[:, None]
    gx = torch.exp(-((x[None] - on(rng.uniform(0, W, k))[:, None]) ** 2) / (2 * sg * sg))
    gy = torch.exp(-((y[None] - on(rng.uniform(0, H, k))[:, None]) ** 2) / (2 * sg * sg))
    f = (gy * on(rng.uniform(-1, 1, k))[:, None]).T @ gx
    for _ in range(2):
        th, period, ph = rng.uniform(0, math.pi), rng.uniform(24, 64), rng.uniform(0, 2 * math.pi)
        f += 0.3 * torch.sin(2 * math.pi * (math.cos(th) * x[None] + math.sin(th) * y[:, None]) / period + ph)
    f -= f.min()
    return f / f.max()


def _look(f, pad, H, w, h):
    """The field at H·(x, y) for the 1-based pixels of a w × h image (bilinear, edge values outside)."""
    M = torch.as_tensor(H, dtype=F64, device="cuda")
    yy, xx = torch.meshgrid(torch.arange(h, dtype=F64, device="cuda") + 1, torch.arange(w, dtype=F64, device="cuda") + 1,
                            indexing="ij")
    px = M[0, 0] * xx + M[0, 1] * yy + M[0, 2] - 1 + pad
    py = M[1, 0] * xx + M[1, 1] * yy + M[1, 2] - 1 + pad
    g = torch.stack([2 * px / (f.shape[1] - 1) - 1, 2 * py / (f.shape[0] - 1) - 1], -1)
    return torch.nn.functional.grid_sample(f[None, None], g[None], mode="bilinear", padding_mode="border", align_corners=True)[0, 0]


def _modality(f, which, rng):
    """0: the field, 1: 1 − field², 2: its 8-level segmentation in shuffled levels; with noise."""
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 30)))
    if which == 1:
        f = 1.0 - f * f
    elif which == 2:
        s = f.flatten()[:: max(1, f.numel() // 65536)].sort().values
        edges = s[[int(s.numel() * q / 8) for q in range(1, 8)]]
        f = torch.as_tensor(rng.permutation(8), dtype=F64, device="cuda")[torch.bucketize(f, edges)] / 7.0
    return f + (0.0, 0.02, 0.03)[which] * torch.randn(f.shape, dtype=F64, device="cuda", generator=g)


def _quant(f, top):
    return (f.clamp(0, 1) * top + 0.5).floor()


def _pinned(a):
    """A host array in page-locked memory, as a program that maps many pairs keeps its buffers."""
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=True)
    t.copy_(a)
    return t.numpy()


def _pair(case, seed, top=65535.0, spread=None, wide=False):
    """(moving, fixed) as float64 GPU images on `top` + 1 levels, the true pose, and the generator."""
    rng = np.random.default_rng(seed)
    mw, mh, fw, fh = case["mw"], case["mh"], case["fw"], case["fh"]
    deg = rng.uniform(0, 360) if wide else case.get("turn", 0.0)
    scale = math.exp(rng.uniform(math.log(0.8), math.log(1.25))) if wide else 1.0
    r = max(8, min(mw, mh, fw, fh) // 8)
    H = _similarity(((mw + 1) / 2, (mh + 1) / 2), ((fw + 1) / 2, (fh + 1) / 2), deg, scale, *(int(v) for v in rng.integers(-r, r + 1, 2)))
    pad = max(mw, mh, fw, fh) // 2 + r
    f = _field(fw, fh, pad, rng)
    fixed = f[pad:pad + fh, pad:pad + fw]
    moving = _modality(_look(f, pad, H, mw, mh), 1 if case["kind"] == "auto" else 2, rng)
    return _quant(moving, top), _quant(fixed, top), H, rng


def _prior(case):
    """The pose a map starts from: centres aligned to whole pixels, turned by the case's angle."""
    mw, mh, fw, fh = case["mw"], case["mh"], case["fw"], case["fh"]
    if case["turn"] == 0.0:
        return _mat([[1, 0, (fw - mw) // 2], [0, 1, (fh - mh) // 2], [0, 0, 1]])
    return _similarity(((mw + 1) / 2, (mh + 1) / 2), ((fw + 1) / 2, (fh + 1) / 2), case["turn"], 1.0, 0, 0)


def _near(case, H, rng, k):
    """k poses within a few pixels and a degree of H."""
    c = ((case["fw"] + 1) / 2, (case["fh"] + 1) / 2)
    return [_similarity(c, c, rng.uniform(-1, 1), math.exp(rng.uniform(-0.01, 0.01)), *rng.uniform(-2, 2, 2)) @ H for _ in range(k)]


def _slices(case, seed):
    """Slices of uneven sizes, each a small drift of the one before, the modalities alternating."""
    rng = np.random.default_rng(seed)
    n, lo, hi = case["slices"], case["lo"], case["hi"]
    side = hi + 128
    f = _field(side, side, 64, rng)
    c, deg, sc, t = (side + 1) / 2, 0.0, 1.0, np.zeros(2)
    out = []
    for k in range(n):
        w, h = (int(v) for v in np.exp(rng.uniform(math.log(lo), math.log(hi), 2)))
        H = _similarity(((w + 1) / 2, (h + 1) / 2), (c, c), deg, sc, *t)
        out.append(_quant(_modality(_look(f, 64, H, w, h), k % 2, rng), 65535.0) / 65535.0)
        deg, sc, t = deg + rng.normal(0, 1.0), sc * math.exp(rng.normal(0, 0.01)), t + np.round(rng.normal(0, 8, 2))
    return out


def _bits(case, seed):
    """Feature stacks [n][128][128][8] as BF16 bits: whitened planes of smooth images, unit variance."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((case["pairs"], 8, 32, 32), device="cuda", generator=g)
    x = torch.nn.functional.interpolate(x, size=(128, 128), mode="bilinear", align_corners=True)
    x = x + 0.3 * torch.randn(x.shape, device="cuda", generator=g)
    return x.permute(0, 2, 3, 1).contiguous().bfloat16()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "propose":
        return {"kind": kind, "params": cnn.shipped_params(), "x": _bits(case, seed).view(torch.int16).cpu().numpy().view(np.uint16)}
    if kind == "stack":
        return {"kind": kind, "eng": Engine(half=False, smi_features=case["mode"]), "slices": [_pinned(s) for s in _slices(case, seed)]}
    if kind == "auto":
        m, f, _, _ = _pair(case, seed, top=255.0)
        return {"kind": kind, "eng": Engine(calibrated=False), "moving": m.to(torch.uint8).cpu().numpy(),
                "fixed": f.to(torch.uint8).cpu().numpy(), "H": _prior(case)}
    m, f, H, rng = _pair(case, seed, wide=kind == "search")
    s = {"kind": kind, "moving": _pinned(m / 65535.0), "fixed": _pinned(f / 65535.0)}
    if kind == "search":
        s["eng"] = Engine(half=False, smi_features=case["mode"], sw_nth=case["rotations"], sw_ns=case["scales"], sw_smin=0.8, sw_smax=1.25)
        return s
    s["eng"] = Engine(half=False, smi_features=case["mode"])
    if kind == "map":
        s.update(H=_prior(case), cap=case["cap"], calibrated=case["calibrated"], want_map=case["want_map"])
        if case["want_map"]:
            s["out"] = torch.empty(case["cap"] ** 2, dtype=torch.float32, pin_memory=True).numpy()
        return s
    # the pose calls work on a resident pair: its images are set once
    s["eng"].set_images(s["moving"], s["fixed"], preprocess=False)
    s["Hs"] = _near(case, H, rng, case.get("poses", 1))
    s["iters"] = case.get("iters", 0)
    return s


# ── one pass ─────────────────────────────────────────────────────────────────────────────────

def _map_out(m):
    out = {"peak": float(m.peak), "zero": float(m.zero), "dx": float(m.dx), "dy": float(m.dy), "index": int(m.peak_index)}
    if m.map is not None:
        out["map"] = m.map
    return out


def run(state):
    kind, eng = state["kind"], state.get("eng")
    if kind == "score":
        r = eng.score(state["Hs"][0])
        return [r.mean, r.fwd, r.inv]
    if kind == "gradient":
        r = eng.gradient(state["Hs"][0], hess=True)
        # the sums behind these are float32 on the device; the call's float64 arrays only carry them
        return {"score": [r.score, r.fwd, r.inv], "n": r.n, "grad": r.grad.astype(np.float32), "hess": r.hess.astype(np.float32)}
    if kind == "refine":
        H, s = eng.refine_poses(state["Hs"], state["iters"])
        return {"H": H.astype(np.float32), "score": s.astype(np.float32)}
    if kind == "map":
        eng.set_images(state["moving"], state["fixed"], preprocess=False)
        return _map_out(eng.shift_map(state["H"], exact=True, calibrated=state["calibrated"], cap=state["cap"],
                                      want_map=state["want_map"], out=state.get("out")))
    if kind == "auto":
        eng.set_images(state["moving"], state["fixed"])
        return _map_out(eng.shift_map(state["H"]))
    if kind == "stack":
        rs, _ = eng.stack_maps(state["slices"])
        col = lambda k: np.array([getattr(r, k) for r in rs], np.float32)
        return {"peak": col("peak"), "zero": col("zero"), "dx": col("dx"), "dy": col("dy"),
                "index": np.array([r.peak_index for r in rs], np.int64)}
    if kind == "search":
        eng.set_images(state["moving"], state["fixed"], preprocess=False)
        eng.pose = np.eye(3)
        r = eng.search()
        return {"H": r.H.astype(np.float32), "score": float(r.score)}
    return {"logits": cnn.forward(state["params"], state["x"])}


# ── what a pass cannot do without ────────────────────────────────────────────────────────────

def _smooth(n):
    while True:
        m = n
        for p in (2, 3):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _frame(H, mw, mh, fw, fh):
    """(ox, oy, w, h): the fixed image and the moving one's corners under H."""
    q = [H @ [x, y, 1.0] for x, y in ((1, 1), (mw, 1), (mw, mh), (1, mh))]
    xs, ys = [v[0] / v[2] - 1 for v in q], [v[1] / v[2] - 1 for v in q]
    ox, oy = int(min(math.floor(min(xs)), 0)), int(min(math.floor(min(ys)), 0))
    return ox, oy, int(max(math.ceil(max(xs)), fw)) - ox, int(max(math.ceil(max(ys)), fh)) - oy


def _plan(w, h, cap):
    """(nx, ny, cw, ch) of a map over a w × h frame; cap 0: the automatic map."""
    if cap:
        top = cap
        s = min(1.0, (top >> 1) / max(w, h))
        while True:
            cw, ch = max(8, math.floor(w * s + 0.5)), max(8, math.floor(h * s + 0.5))
            nx, ny = _smooth(max(2 * cw - 1, 32)), _smooth(max(2 * ch - 1, 32))
            if nx <= top and ny <= top:
                return nx, ny, cw, ch
            s *= 0.85
    g = 1
    while 2 * -(-max(w, h) // g) - 1 > 512:
        g *= 2
    cw, ch = -(-w // g), -(-h // g)
    p2 = lambda n: min(max(1 << (n - 1).bit_length(), 128), 512)
    return p2(2 * cw - 1), p2(2 * ch - 1), cw, ch


def _map_work(w, h, nx, ny, cw, ch, planes, corrs):
    """Both images read, the map written; both sides' forward transforms of the real planes, the
    correlations' products and inverse transforms (real, 2.5 N log2 N each) and the scores."""
    n = nx * ny
    flops = 2 * planes * 2.5 * n * math.log2(n) + corrs * (2.5 * n * math.log2(n) + 3.0 * n) + 300.0 * n
    return {"bytes": 8.0 * w * h + 4.0 * n, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "propose":
        n = case["pairs"]
        macs = 64 * 64 * 72 * 32 + 32 * 32 * 288 * 64 + 16 * 16 * 576 * 64 + 8 * 8 * 576 * 128 + 128 * 216
        return {"bytes": n * (128 * 128 * 8 * 2 + 216 * 4.0) + 4.0 * 160000, "flops": 2.0 * macs * n}
    three = case.get("mode") == "three"
    planes, corrs = (10, 28) if three else (15, 45)
    if kind == "stack":
        s = int(math.sqrt(case["lo"] * case["hi"]))
        one = _map_work(s, s, *_plan(s, s, 1024), planes, corrs)
        return {k: v * (case["slices"] - 1) for k, v in one.items()}
    px = case["fw"] * case["fh"] + case["mw"] * case["mh"]
    if kind in ("score", "gradient"):
        # both directions: every pixel's features of both images once, its taps and 45 (+ 44) sums
        return {"bytes": 16.0 * px, "flops": (190.0 if kind == "score" else 550.0) * px}
    if kind == "refine":
        # per pose and step: the gradient and at least one candidate's score
        return {"bytes": 16.0 * px, "flops": 740.0 * px * case["poses"] * case["iters"]}
    if kind == "search":
        # per candidate a map of the 128-cell canvas (planes of about 192 points a side)
        one = _map_work(0, 0, 192, 192, 96, 96, planes / 2.0, corrs)
        k = case["rotations"] * case["scales"]
        return {"bytes": 4.0 * px + k * one["bytes"], "flops": k * one["flops"]}
    _, _, w, h = _frame(_prior(case), case["mw"], case["mh"], case["fw"], case["fh"])
    w_ = _map_work(0, 0, *_plan(w, h, case.get("cap", 0)), planes, corrs)
    return {"bytes": w_["bytes"] + (1.0 if kind == "auto" else 4.0) * px, "flops": w_["flops"]}


# ── the same outputs in float64 ──────────────────────────────────────────────────────────────

_TRI = [(0, 0), (0, 1), (0, 2), (0, 3), (1, 1), (1, 2), (1, 3), (2, 2), (2, 3), (3, 3)]


def _clahe(a, clip=40.0, bins=64, grid=4):
    """Contrast-limited equalisation of an image in [0, 1] over grid × grid tiles."""
    h, w = a.shape
    hp, wp = (grid - h % grid) % grid, (grid - w % grid) % grid
    refl = lambda n, pad: (torch.arange(n + pad, device="cuda") - pad).abs().clamp(0, n - 1)
    v = a[refl(h, hp)][:, refl(w, wp)].clamp(0, 1)
    th, tw = (h + hp) // grid, (w + wp) // grid
    # the bins of 8-bit levels as their float32 luma places them (63 · (i / 255) meets whole numbers)
    v32 = v.float()
    b = ((v32 * 0.299 + v32 * 0.587 + v32 * 0.114) * (bins - 1)).floor().clamp(0, bins - 1).long()
    yy, xx = torch.meshgrid(torch.arange(h + hp, device="cuda") // th, torch.arange(w + wp, device="cuda") // tw, indexing="ij")
    hist = torch.bincount(((yy * grid + xx) * bins + b).flatten(), minlength=grid * grid * bins).reshape(grid * grid, bins).to(F64)
    limit = max(clip * th * tw / bins, 1.0)
    cut = hist.clamp(max=limit)
    clipped = th * tw - cut.sum(1, keepdim=True)
    rest = (clipped - bins * (clipped / bins).floor()).floor()
    c = cut + (clipped - rest) / bins + (torch.arange(bins, device="cuda")[None] < rest).to(F64)
    cdf = (c.cumsum(1) / (th * tw)).clamp(0, 1)
    gy = (torch.arange(h, dtype=F64, device="cuda") + 0.5) / h * (grid - 1)
    gx = (torch.arange(w, dtype=F64, device="cuda") + 0.5) / w * (grid - 1)
    y0, x0 = gy.floor().long()[:, None], gx.floor().long()[None]
    fy, fx = gy[:, None] - y0, gx[None] - x0
    y1, x1 = (y0 + 1).clamp(max=grid - 1), (x0 + 1).clamp(max=grid - 1)
    bf = a.clamp(0, 1) * (bins - 1)
    b0 = bf.floor().clamp(0, bins - 2).long()
    fb = bf - b0
    look = lambda ty, tx: cdf[ty * grid + tx, b0] * (1 - fb) + cdf[ty * grid + tx, b0 + 1] * fb
    return (look(y0, x0) * (1 - fx) + look(y0, x1) * fx) * (1 - fy) + (look(y1, x0) * (1 - fx) + look(y1, x1) * fx) * fy


def _features(g, mode):
    """The four whitened feature planes of an image (float64)."""
    h, w = g.shape
    mean = g.mean()
    z = (g - mean) / ((g - mean) ** 2).mean().clamp(min=1e-12).sqrt()
    b = ((z + 4) * 32).clamp(0, 255).long()
    hist = torch.bincount(b.flatten(), minlength=256).to(F64)
    r = ((hist.cumsum(0) - 0.5 * hist)[b] / g.numel()) * 2 - 1
    p = torch.nn.functional.pad(r[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    t = lambda dx, dy: p[1 + dy:1 + dy + h, 1 + dx:1 + dx + w]
    gx = t(1, -1) - t(-1, -1) + 2 * (t(1, 0) - t(-1, 0)) + t(1, 1) - t(-1, 1)
    gy = t(-1, 1) - t(-1, -1) + 2 * (t(0, 1) - t(0, -1)) + t(1, 1) - t(1, -1)
    f3 = {"laplacian": t(-1, 0) + t(1, 0) + t(0, -1) + t(0, 1) - 4 * r, "three": torch.zeros_like(r), "cubic": r ** 3}[mode]
    x = torch.stack([r, r * r, (gx * gx + gy * gy).sqrt(), f3]).reshape(4, -1)
    mu = x.mean(1, keepdim=True)
    G = (x - mu) @ (x - mu).T / x.shape[1]
    G = G + torch.eye(4, dtype=F64, device="cuda") * 1e-4 * (G.trace() / 4).clamp(min=1e-12)
    return torch.linalg.solve_triangular(torch.linalg.cholesky(G), x - mu, upper=False).reshape(4, h, w)


def _acf(f):
    """Each plane's autocorrelation at lags of at most 8, over the pairs inside the image, at lag 0 one."""
    _, h, w = f.shape
    out = torch.zeros((17, 17, 4), dtype=F64, device="cuda")
    for dy in range(-8, 9):
        for dx in range(-8, 9):
            a = f[:, max(0, -dy):h - max(0, dy), max(0, -dx):w - max(0, dx)]
            b = f[:, max(0, dy):h + min(0, dy), max(0, dx):w + min(0, dx)]
            out[dy + 8, dx + 8] = (a * b).mean((1, 2))
    return out / out[8, 8].clamp(min=1e-12)


def _warp(s, Hc, W, Hh):
    """The stack s on the W × Hh canvas by the canvas pose: bilinear inside the image, 0 outside."""
    _, h, w = s.shape
    M = np.linalg.inv(Hc)
    yy, xx = torch.meshgrid(torch.arange(Hh, dtype=F64, device="cuda") + 1, torch.arange(W, dtype=F64, device="cuda") + 1, indexing="ij")
    q = [M[i, 0] * xx + M[i, 1] * yy + M[i, 2] for i in range(3)]
    fx, fy = q[0] / q[2] - 1, q[1] / q[2] - 1
    # whole-pixel poses land on the pixels up to the inverse's rounding
    fx, fy = (torch.where((v - v.round()).abs() < 1e-9, v.round(), v) for v in (fx, fy))
    ok = (fx >= 0) & (fy >= 0) & (fx <= w - 1) & (fy <= h - 1)
    x0, y0 = fx.floor().clamp(0, w - 1).long(), fy.floor().clamp(0, h - 1).long()
    x1, y1 = (x0 + 1).clamp(max=w - 1), (y0 + 1).clamp(max=h - 1)
    tx, ty = fx - x0, fy - y0
    return torch.stack([torch.where(ok, (p[y0, x0] * (1 - tx) + p[y0, x1] * tx) * (1 - ty) + (p[y1, x0] * (1 - tx) + p[y1, x1] * tx) * ty,
                                    torch.zeros_like(tx)) for p in s])


def _resample(c, cw, ch):
    """A canvas on the cw × ch grid: the mean of k × k bilinear taps per cell."""
    _, Hh, W = c.shape
    if (W, Hh) == (cw, ch):
        return c
    fx, fy = W / cw, Hh / ch
    kx, ky = (int(min(max(math.ceil(v - 1e-4), 1), 8)) for v in (fx, fy))

    def taps(n, step, k, size):
        R = torch.zeros((n, size), dtype=F64, device="cuda")
        g = torch.arange(n, dtype=F64, device="cuda")
        for i in range(k):
            p = (g + (i + 0.5) / k) * step - 0.5
            a = p.floor()
            for q, v in ((a, 1 - (p - a)), (a + 1, p - a)):
                R.scatter_add_(1, q.clamp(0, size - 1).long()[:, None], (v / k)[:, None])
        return R

    return taps(ch, fy, ky, Hh) @ c @ taps(cw, fx, kx, W).T


def _shift_map(fa, fb, H, cap, mode, calibrated, min_overlap=0.0):
    """The map of a pair of feature stacks at H and its result, as run() lays them out."""
    one = lambda f: torch.cat([torch.ones_like(f[:1]), f])
    mh, mw, fh, fw = *fa.shape[1:], *fb.shape[1:]
    ox, oy, W, Hh = _frame(H, mw, mh, fw, fh)
    ca = _warp(one(fa), _mat([[1, 0, -ox], [0, 1, -oy], [0, 0, 1]]) @ H, W, Hh)
    cb = torch.zeros((5, Hh, W), dtype=F64, device="cuda")
    cb[:, -oy:-oy + fh, -ox:-ox + fw] = one(fb)
    nx, ny, cw, ch = _plan(W, Hh, cap)
    A, B = _resample(ca, cw, ch), _resample(cb, cw, ch)
    nf = 3 if mode == "three" else 4
    tri = [(i, j) for i, j in _TRI if j < nf]
    second = lambda s, i, j: torch.where(s[0] > 1e-6, s[1 + i] * s[1 + j] / s[0].clamp(min=1e-6), torch.zeros_like(s[0]))
    spec = lambda p: torch.fft.rfft2(p, (ny, nx))
    FA, FB = [spec(A[k]) for k in range(1 + nf)], [spec(B[k]) for k in range(1 + nf)]
    corr = lambda a, b: torch.fft.irfft2(a * b.conj(), (ny, nx))
    n = corr(FA[0], FB[0])
    n = torch.where((n - n.round()).abs() < 1e-6, n.round(), n)
    rn = 1.0 / n.clamp(min=1e-8)
    ma = [corr(FA[1 + i], FB[0]) * rn for i in range(nf)]
    mb = [corr(FA[0], FB[1 + i]) * rn for i in range(nf)]
    C = [[corr(FA[1 + i], FB[1 + j]) * rn - ma[i] * mb[j] for j in range(nf)] for i in range(nf)]

    def factor(sums, m):
        """The Cholesky factor of the ridged covariance per shift, and where it exists."""
        G = {ij: sums(*ij) * rn - m[ij[0]] * m[ij[1]] for ij in tri}
        rg = 1e-4 * (sum(G[i, i] for i in range(nf)) * 0.25).clamp(min=1e-12)
        L, ok = {}, torch.ones_like(n, dtype=torch.bool)
        for i in range(nf):
            for j in range(i + 1):
                s = G[j, i] - sum(L[i, k] * L[j, k] for k in range(j)) + (rg if i == j else 0.0)
                if i == j:
                    ok &= s > 0
                    L[i, i] = torch.where(s > 0, s, torch.ones_like(s)).sqrt()
                else:
                    L[i, j] = s / L[j, j]
        return L, ok

    LA, oka = factor(lambda i, j: corr(spec(second(A, i, j)), FB[0]), ma)
    LB, okb = factor(lambda i, j: corr(FA[0], spec(second(B, i, j))), mb)
    for j in range(nf):
        for i in range(nf):
            C[i][j] = (C[i][j] - sum(LA[i, k] * C[k][j] for k in range(i))) / LA[i, i]
    acc = torch.zeros_like(n)
    for r in range(nf):
        y = []
        for i in range(nf):
            y.append((C[r][i] - sum(LB[i, k] * y[k] for k in range(i))) / LB[i, i])
            acc += y[i] * y[i]
    least = max(12.0, math.floor(min_overlap * cw * ch))
    if calibrated:
        cell = W / cw
        area = float((_acf(fa).sum(2) * _acf(fb).sum(2)).sum()) / 16
        neff = n / max(1.0, max(1.0, area) / (cell * cell))
        dead = (n < least) | (neff <= 10)
        v = acc.clamp(max=nf - 1e-4)
        d2 = nf * (neff - nf - 1)
        fv = d2 / nf / nf * v / (nf - v)
        a, b, c = 2 / (9 * nf * nf), 2 / (9 * d2), fv.clamp(min=0) ** (1 / 3)
        score = (((1 - b) * c - (1 - a)) / (b * c * c + a).sqrt()).clamp(min=0)
    else:
        dead = n < max(least, 0.08 * float(n[0, 0]))
        score = n * acc
    m = torch.where(dead | ~oka | ~okb | ~score.isfinite(), torch.zeros_like(score), score)
    k = int(m.argmax())
    ly, lx = divmod(k, nx)
    lx, ly = lx if lx <= nx // 2 else lx - nx, ly if ly <= ny // 2 else ly - ny
    return {"peak": float(m.max()), "zero": float(m[0, 0]), "dx": lx * W / cw, "dy": ly * Hh / ch, "index": None, "map": m}


def _one_way(fa, fb, H):
    """(score, overlap) of the moving stack fa on fb at H, differentiable in H."""
    _, ah, aw = fa.shape
    _, bh, bw = fb.shape
    M = torch.linalg.inv(H)
    yy, xx = torch.meshgrid(torch.arange(bh, dtype=F64, device="cuda") + 1, torch.arange(bw, dtype=F64, device="cuda") + 1, indexing="ij")
    q = [M[i, 0] * xx + M[i, 1] * yy + M[i, 2] for i in range(3)]
    fx, fy = q[0] / q[2] - 1, q[1] / q[2] - 1
    ramp = lambda v, hi: ((v - 2) / 2).clamp(0, 1) * ((hi - v) / 2).clamp(0, 1)
    ok = (fx >= 2) & (fy >= 2) & (fx <= aw - 3) & (fy <= ah - 3)
    wt = (ramp(fx, aw - 3) * ramp(fy, ah - 3) * ok)[ok]
    fx, fy, b = fx[ok], fy[ok], fb[:, ok]
    x0, y0 = fx.detach().floor().long(), fy.detach().floor().long()
    tx, ty = fx - x0, fy - y0
    a = (fa[:, y0, x0] * (1 - tx) + fa[:, y0, x0 + 1] * tx) * (1 - ty) + (fa[:, y0 + 1, x0] * (1 - tx) + fa[:, y0 + 1, x0 + 1] * tx) * ty
    n = wt.sum()
    ma, mb = (wt * a).sum(1) / n, (wt * b).sum(1) / n
    C = (wt * a) @ b.T / n - ma[:, None] * mb[None]
    ridge = lambda G: G + torch.eye(4, dtype=F64, device="cuda") * 1e-4 * (G.trace() / 4).clamp(min=1e-12)
    GA, GB = ridge((wt * a) @ a.T / n - ma[:, None] * ma[None]), ridge((wt * b) @ b.T / n - mb[:, None] * mb[None])
    return n * (torch.linalg.solve(GA, C) * torch.linalg.solve(GB, C.T).T).sum(), n


def _gradient(fa, fb, H0):
    """The symmetric score at H0 and its derivative over the homography's eight coordinates."""
    N = torch.as_tensor(_mat([[2 / fb.shape[2], 0, -(fb.shape[2] + 1) / fb.shape[2]], [0, 2 / fb.shape[1], -(fb.shape[1] + 1) / fb.shape[1]],
                              [0, 0, 1]]), device="cuda")
    z = torch.zeros(8, dtype=F64, device="cuda", requires_grad=True)
    tx, ty, th, sg, al, ga, px, py = z
    K = torch.stack([torch.stack([sg / 3 + al, ga - th, tx]), torch.stack([ga + th, sg / 3 - al, ty]), torch.stack([px, py, -2 * sg / 3])])
    H = torch.linalg.inv(N) @ torch.linalg.matrix_exp(K) @ N @ torch.as_tensor(H0, device="cuda")
    fwd, n = _one_way(fa, fb, H)
    inv, _ = _one_way(fb, fa, torch.linalg.inv(H))
    mean = 0.5 * (fwd + inv)
    g, = torch.autograd.grad(mean, z)
    return [float(mean.detach()), float(fwd.detach()), float(inv.detach())], float(n.detach()), g


def _logits(params, x):
    """The network's logits for BF16 inputs: weights as given, everything else in float64."""
    p = torch.as_tensor(np.asarray(params, np.float32), device="cuda").to(F64)
    a, at = x.to(F64).permute(0, 3, 1, 2), 0
    for cin, cout in ((8, 32), (32, 64), (64, 64), (64, 128)):
        w = p[at:at + cout * 9 * cin].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
        at += cout * 9 * cin
        a = torch.nn.functional.conv2d(a, w, p[at:at + cout], stride=2, padding=1).relu()
        at += cout
    w = p[at:at + 216 * 128].reshape(216, 128)
    return a.mean((2, 3)) @ w.T + p[at + 216 * 128:at + 216 * 129]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("refine", "search"):
        return None  # poses that an accept-or-reject iteration arrives at have no closed value
    if kind == "propose":
        return {"logits": _logits(cnn.shipped_params(), _bits(case, seed))}
    if kind == "stack":
        fs = [_features(s.float().to(F64), case["mode"]) for s in _slices(case, seed)]
        out = {"peak": [], "zero": [], "dx": [], "dy": []}
        for b, a in zip(fs, fs[1:]):
            H = _mat([[1, 0, (b.shape[2] - a.shape[2]) / 2], [0, 1, (b.shape[1] - a.shape[1]) / 2], [0, 0, 1]])
            r = _shift_map(a, b, H, 1024, case["mode"], False)
            for k in out:
                out[k].append(r[k])
        return {**{k: np.array(v) for k, v in out.items()}, "index": None}
    if kind == "auto":
        m, f, _, _ = _pair(case, seed, top=255.0)
        half = lambda v: v.half().to(F64)
        fa, fb = (_features(half(_clahe(v / 255.0)), "laplacian") for v in (m, f))
        return _shift_map(fa, fb, _prior(case), 0, "laplacian", False, 0.05)
    m, f, H, rng = _pair(case, seed)
    fa, fb = (_features((v / 65535.0).float().to(F64), case["mode"]) for v in (m, f))
    if kind == "map":
        r = _shift_map(fa, fb, _prior(case), case["cap"], case["mode"], case["calibrated"])
        if not case["want_map"]:
            del r["map"]
        return r
    s, n, g = _gradient(fa, fb, _near(case, H, rng, 1)[0])
    # the Gauss–Newton matrix is the framework's own construction: no plain value for it
    return s if kind == "score" else {"score": s, "n": n, "grad": g, "hess": None}
