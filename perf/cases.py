"""Timed workloads of the renderer, through its public Python interface.

Flames come from the bundled workloads (refraktor_gb300/workloads/), moved a
little by the seed: same structure, other affines, weights and colours. The
image steps (blur, tonemap, conversion, denoiser) take seeded stand-ins of
rendered histograms made with torch alone: points of a small iterated function
system, smoothed to an expected density, then Poisson counts at the stated
samples per pixel, so empty, sparse and dense pixels occur as in a render.
"""
import json
import math
from pathlib import Path

import numpy as np
import torch
import torch.nn.functional as F

from refraktor_gb300 import denoise as dn
from refraktor_gb300 import librefrakt as lr

WORKLOADS = Path(lr.__file__).resolve().parent / "workloads"
# the launch shape that the library's autotuner picks for the 1080p workload
TUNED = {"block": 256, "chains_per_thread": 8, "flush": 4, "sort": 2, "blocks_per_sm": 4}
DE = (9.0, 0.0, 0.5)  # blur radius 0-9 px scaled by 1 / sqrt(density)
GAMMA, BRIGHTNESS, VIBRANCY = 2.2, 4.0, 1.0
FORMATS = {"half3": lr.HALF3, "half4": lr.HALF4, "float3": lr.FLOAT3, "float4": lr.FLOAT4, "uchar3": lr.UCHAR3,
           "uchar4": lr.UCHAR4}


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # an editor's preview: the 3-xform flame at low quality with default options; latency and launches count
        {"name": "preview_512", "kind": "frame", "genome": "plain", "w": 512, "h": 512, "spp": 32.0, "tmul": 1, "blur": False},
        # one still of the 1080p workload: re-warm, iterate, blur, tonemap
        {"name": "frame_1080p", "kind": "frame", "genome": "hd", "w": 1920, "h": 1080, "spp": 1024.0, "tmul": 1, "blur": True},
        # a motion-blurred frame: four temporal samples per block along a moving spline
        {"name": "motion_720p", "kind": "frame", "genome": "hd", "w": 1280, "h": 720, "spp": 64.0, "tmul": 4, "blur": True},
        # a piece of an animation between keyframes, rendered as one batch and replayed as a graph
        {"name": "anim_720p", "kind": "batch", "genome": "anim", "w": 1280, "h": 720, "spp": 256.0, "units": 16},
        # unrelated flames of many sizes on one union-of-variations kernel
        {"name": "hetero", "kind": "batch", "genome": "hetero", "w": 0, "h": 0, "spp": 0.0, "units": 16},
        # blur of a converged still, and of a sparse draft of odd size (wide radii)
        {"name": "blur_1080p", "kind": "blur", "w": 1920, "h": 1080, "spp": 1024.0},
        {"name": "blur_draft", "kind": "blur", "w": 1367, "h": 769, "spp": 32.0},
        # tonemap to the half4 image a renderer keeps, and the reference-exact variant with its density histogram
        {"name": "tonemap_1080p", "kind": "tonemap", "w": 1920, "h": 1080, "spp": 1024.0, "fmt": "half4", "precise": True},
        {"name": "tonemap_ref", "kind": "tonemap", "w": 1366, "h": 768, "spp": 128.0, "fmt": "float4", "precise": False},
        # a 4K image to the bytes an encoder takes, bottom row first
        {"name": "export_4k", "kind": "convert", "w": 3840, "h": 2160, "src": "half4", "dst": "uchar3", "flip": True,
         "swap": False},
        # the learned denoiser on a 32-spp 1080p render
        {"name": "denoise_1080p", "kind": "denoise", "w": 1920, "h": 1080, "spp": 32.0, "fmt": "half4"},
        # one training step of the denoiser: forward, backward, Adam; late in the learning-rate schedule
        {"name": "train_512", "kind": "train", "n": 16, "w": 512, "h": 512, "spp": 32.0, "lr": 1e-5},
    ]


def _size(rng, lo, hi):
    """A log-spread, mostly odd width and a height of about 9 / 16 to 1 of it."""
    w = int(round(lo * (hi / lo) ** rng.random()))
    return w, max(16, int(w * rng.uniform(9 / 16, 1.0)))


def draw(rng):
    kind = rng.choice(["preview", "still", "motion", "anim", "hetero", "blur", "tonemap", "convert", "denoise", "train"])
    if kind == "preview":
        w, h = _size(rng, 128, 1024)
        return {"kind": "frame", "genome": "plain", "w": w, "h": h, "spp": round(8 * 16 ** rng.random(), 2), "tmul": 1,
                "blur": rng.random() < 0.5}
    if kind == "still":
        w, h = _size(rng, 480, 1920)
        return {"kind": "frame", "genome": "hd", "w": w, "h": min(h, 1080), "spp": round(32 * 32 ** rng.random(), 2), "tmul": 1,
                "blur": rng.random() < 0.75}
    if kind == "motion":
        w, h = _size(rng, 320, 1280)
        return {"kind": "frame", "genome": "hd", "w": w, "h": h, "spp": round(16 * 8 ** rng.random(), 2),
                "tmul": rng.choice([2, 4, 8]), "blur": True}
    if kind == "anim":
        w, h = _size(rng, 480, 1280)
        return {"kind": "batch", "genome": "anim", "w": w, "h": min(h, 720), "spp": float(rng.randint(128, 256)),
                "units": rng.randint(2, 16)}
    if kind == "hetero":
        return {"kind": "batch", "genome": "hetero", "w": 0, "h": 0, "spp": 0.0, "units": rng.randint(5, 15)}
    if kind == "blur":
        w, h = _size(rng, 256, 2048)
        return {"kind": "blur", "w": w, "h": h, "spp": round(8 * 256 ** rng.random(), 2)}
    if kind == "tonemap":
        w, h = _size(rng, 256, 3840)
        return {"kind": "tonemap", "w": w, "h": h, "spp": round(8 * 256 ** rng.random(), 2),
                "fmt": rng.choice(["half3", "half4", "float3", "float4"]), "precise": rng.random() < 0.75}
    if kind == "convert":
        w, h = _size(rng, 256, 3840)
        return {"kind": "convert", "w": w, "h": h, "src": rng.choice(["half3", "half4"]),
                "dst": rng.choice(["uchar3", "uchar4", "float3", "float4"]), "flip": rng.random() < 0.5,
                "swap": rng.random() < 0.5}
    if kind == "denoise":
        w, h = _size(rng, 128, 1920)
        return {"kind": "denoise", "w": w // 8 * 8, "h": max(16, h // 8 * 8), "spp": float(rng.choice([32, 64, 96, 128])),
                "fmt": rng.choice(["half3", "half4"])}
    return {"kind": "train", "n": rng.randint(1, 16), "w": 512, "h": 8 * rng.randint(16, 64), "spp": float(rng.choice([32, 64, 128])),
            "lr": 1e-5}


# ------------------------------------------------------------------ flames --
_KEPT = {}  # the database, workload files and compiled kernels a program keeps while it runs


def _kept(key, make):
    if key not in _KEPT:
        _KEPT[key] = make()
    return _KEPT[key]


def _db():
    return _kept("db", lr.flamedb)


def _workload(name):
    return _kept(name, lambda: json.loads((WORKLOADS / name).read_text()))


def _moved(genome, rng, amount=1.0):
    """The genome with its affines turned and shifted, its weights and hues changed a little."""
    g = json.loads(json.dumps(genome))
    for xf in g["xforms"]:
        xf["weight"] *= 1.0 + 0.1 * amount * rng.uniform(-1, 1)
        for vl in xf["vchain"]:
            a, d, b, e, c, f = vl["transform"]
            t = 0.04 * amount * rng.uniform(-1, 1)
            co, si = math.cos(t), math.sin(t)
            vl["transform"] = [a * co - d * si, a * si + d * co, b * co - e * si, b * si + e * co,
                               c + 0.02 * amount * rng.uniform(-1, 1), f + 0.02 * amount * rng.uniform(-1, 1)]
    turn = 60.0 * amount * rng.uniform(-1, 1)
    g["palette"] = [[(p[0] + turn) % 360.0, p[1], p[2]] for p in g["palette"]]
    return g


def _kernel(name, flame, opts):
    return _kept(("kernel", name), lambda: lr.flame_compiler().get_flame_kernel(_db(), flame, **opts))


def _prepare_frame(case, seed):
    rng = np.random.default_rng(seed)
    w, h = case["w"], case["h"]
    base = _workload("plain_512.json" if case["genome"] == "plain" else "hd_1080p.json")
    base = _moved(base, rng)
    if case["tmul"] > 1:
        flames = [lr.flame.from_json(_db(), _moved(base, np.random.default_rng(seed + 1), 0.5 * i)) for i in range(4)]
    else:
        flames = [lr.flame.from_json(_db(), base)] * 4
    k = _kernel(case["genome"], flames[0], {} if case["genome"] == "plain" else TUNED)
    samples = np.stack([f.pack_sample(w, h) for f in flames])
    bins = torch.zeros((h, w, 4), device="cuda")  # the renderer's own histogram buffer, adopted by the state
    st = k.warmup(samples, bins, seed % 65536 + 1, 20, temporal_multiplier=case["tmul"])
    # with one temporal sample per block the blocks stop together at the shared target: a pass cap just under it makes
    # every run the same passes (with more of them every block has its own share of the target)
    per_pass = k.info["grid"] * k.info["block"] * k.info["chains_per_thread"]
    cap = max(1, int(0.9 * case["spp"] * w * h / per_pass)) if case["tmul"] == 1 else 0
    return {"kind": "frame", "k": k, "st": st, "samples": samples, "seed": seed % 65536 + 1, "w": w, "h": h,
            "limit": lr.bailout_args(iters=cap, millis=0, quality=case["spp"]), "tm": flames[0].tonemap_params(),
            "bins": bins, "map": lr.tonemapper(),
            "blurred": torch.empty((h, w, 4), device="cuda") if case["blur"] else None,
            "image": torch.empty((h, w, 4), device="cuda", dtype=torch.float16)}


def _run_frame(s):
    dims = (s["w"], s["h"])
    s["st"].rewarm(s["samples"], s["seed"], 20)
    s["k"].bin(s["st"], s["limit"])
    bins = s["bins"]
    if s["blurred"] is not None:
        lr.density_blur(bins, s["blurred"], dims, *DE)
        bins = s["blurred"]
    tm = s["tm"]
    s["map"].run(bins, s["image"], dims, s["st"].quality, tm["gamma"], tm["brightness"], tm["vibrancy"], fmt=lr.HALF4)
    return {"image": s["image"], "histogram": s["bins"]}


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    units, samples = [], []
    if case["genome"] == "anim":
        w, h, n = case["w"], case["h"], case["units"]
        keys = [lr.flame.from_json(_db(), _moved(g, rng)) for g in _workload("anim_720p.json")["keyframes"]]
        kf = keys[0]
        ks = [f.pack_sample(w, h) for f in keys]
        samples = np.stack([ks[0], ks[0], ks[1], ks[2], ks[3], ks[3]])
        tp = kf.tonemap_params()
        for i in range(n):
            x = 3.0 * i / (n - 1)
            seg = min(int(x), 2)
            units.append(lr.batch_unit(w, h, case["spp"], segment=seg, t=float(x - seg), gamma=tp["gamma"],
                                       brightness=tp["brightness"], vibrancy=tp["vibrancy"]))
    else:
        every = _workload("hetero_64.json")["flames"]
        fl = _kept("aligned", lambda: [f.serialize() for f in lr.align_flames(
            _db(), [lr.flame.from_json(_db(), e["genome"]) for e in every[:16]])])
        for i, (g, e) in enumerate(list(zip(fl, every))[:case["units"]]):
            f = lr.flame.from_json(_db(), _moved(g, rng))
            kf = f
            tp = f.tonemap_params()
            units.append(lr.batch_unit(e["width"], e["height"], float(e["spp"]), segment=4 * i, t=0.0, gamma=tp["gamma"],
                                       brightness=tp["brightness"], vibrancy=tp["vibrancy"]))
            samples.append(f.pack_samples(4, e["width"], e["height"]).reshape(4, -1))
        samples = np.concatenate(samples)
    k = _kernel(case["genome"], kf, TUNED)
    b = lr.batch(k, units, samples.shape[0], passes_per_item=256, warmup=20, seed=seed % 65536 + 1, de=DE, out_format=lr.HALF4)
    bins = [b.bins(i) for i in range(len(units))]
    for t in bins:
        t.batch = b  # the batch owns the memory that its histograms view
    return {"kind": "batch", "b": b, "samples": samples, "stream": torch.cuda.Stream(), "bins": bins}


def _run_batch(s):
    s["b"].set_samples(s["samples"])
    s["b"].run(use_graph=True, stream=s["stream"])
    s["b"].wait()
    # the queue hands passes to whichever block is free, so every run is another random sample: the histograms converge,
    # while the log-density images still show their few-hit pixels
    return s["bins"]


# -------------------------------------------------------------- histograms --
def _histogram(w, h, spp, seed):
    """A histogram (h, w, 4) of Poisson counts at spp and the expected one."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, nmaps = 1 << 17, 4
    m = rng.uniform(-1, 1, (nmaps, 2, 2))
    m *= np.minimum(1.0, 0.85 / np.linalg.norm(m, 2, axis=(1, 2)))[:, None, None]
    m = torch.tensor(m, device="cuda", dtype=torch.float32)
    t = torch.tensor(rng.uniform(-1, 1, (nmaps, 2)), device="cuda", dtype=torch.float32)
    bend = torch.tensor(rng.uniform(0, 0.6, nmaps), device="cuda", dtype=torch.float32)
    hue = torch.tensor(rng.uniform(0, 1, nmaps), device="cuda", dtype=torch.float32)
    p = torch.rand((n, 2), device="cuda", generator=g) * 2 - 1
    c = torch.rand(n, device="cuda", generator=g)
    counts = torch.zeros(w * h, device="cuda", dtype=torch.float64)
    hues = torch.zeros_like(counts)
    for step in range(52):
        k = torch.randint(0, nmaps, (n,), device="cuda", generator=g)
        q = (m[k] * p[:, None, :]).sum(-1) + t[k]
        p = q + bend[k][:, None] * (torch.sin(2 * q) - q)
        c = 0.5 * (c + hue[k])
        if step == 12:
            mid, half = p.mean(0), 2.2 * p.std(0) + 1e-3
        if step >= 12:
            u = (p - mid) / half
            x, y = ((u[:, 0] + 1) * (0.5 * w)).floor(), ((u[:, 1] + 1) * (0.5 * h)).floor()
            at = torch.where((x >= 0) & (x < w) & (y >= 0) & (y < h), y * w + x, torch.full_like(x, -1)).long()
            ok = at >= 0
            at, cc = at[ok], (c[ok] * 255).floor().double()
            counts += torch.bincount(at, minlength=w * h)
            hues += torch.bincount(at, weights=cc, minlength=w * h)  # sums of whole numbers: the same in any order
    counts, hues = counts.view(1, 1, h, w), hues.view(1, 1, h, w)
    wide = lambda v: 0.7 * v + 0.3 * F.avg_pool2d(v, 5, 1, 2)  # noqa: E731
    lam, col = wide(counts).view(h, w), (wide(hues).view(h, w) / wide(counts).view(h, w).clamp_min(1e-9) / 255.0).float()
    lam = (lam * (spp * w * h / lam.sum())).float()
    rgb = 0.5 + 0.5 * torch.cos(6.2832 * (col[..., None] + torch.tensor([0.0, 0.33, 0.67], device="cuda")))
    density = torch.poisson(lam, generator=g)
    full = lambda d: torch.cat([rgb * d[..., None], d[..., None]], -1).contiguous()  # noqa: E731
    return full(density), full(lam)


def _tonemap64(bins, q, alpha=True):
    """The log-density tonemap of a histogram at quality q, in 64 bits."""
    b = bins.double()
    d = b[..., 3:]
    k2 = 10.0 ** (-math.log10(q) - 0.5)
    lit = d > 0
    ds = torch.where(lit, d, torch.ones_like(d))
    f = 0.5 * BRIGHTNESS * torch.log10(1.0 + ds * k2) / ds
    v = b[..., :3] * f
    grey = (ds * f) ** (1.0 / GAMMA) / (ds * f)
    rgb = ((1.0 - VIBRANCY) * v.clamp_min(0) ** (1.0 / GAMMA) + VIBRANCY * v * grey).clamp(0, 1)
    a = (torch.log(ds) * (4.0 / math.log(2.0)) / 96.0).clamp(0, 1)
    out = torch.cat([rgb, a], -1) if alpha else rgb
    return torch.where(lit, out, torch.zeros_like(out))


def _channels(fmt):
    return int(fmt[-1])


def _dtype(fmt):
    return {"half": torch.float16, "float": torch.float32, "uchar": torch.uint8}[fmt[:-1]]


def _image(case, fmt):
    return torch.empty((case["h"], case["w"], _channels(fmt)), device="cuda", dtype=_dtype(fmt))


# -------------------------------------------------------------- entry points --
def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        return _prepare_frame(case, seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    w, h = case["w"], case["h"]
    s = {"kind": kind, "dims": (w, h)}
    if kind == "train":
        pairs = [_histogram(w, h, case["spp"], seed * 64 + i) for i in range(case["n"])]
        s["bins"] = torch.stack([p[0] for p in pairs])
        s["base"] = torch.stack([_tonemap64(p[0], case["spp"]).float() for p in pairs])
        s["target"] = torch.stack([_tonemap64(p[1], case["spp"]).float() for p in pairs])
        s |= {"net": dn.denoiser(params=_weights()), "spp": case["spp"], "lr": case["lr"]}
        return s
    if kind == "convert":
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["in"] = torch.rand((h, w, _channels(case["src"])), device="cuda", generator=g).half()
        s |= {"out": _image(case, case["dst"]), "conv": lr.converter(), "src": FORMATS[case["src"]], "dst": FORMATS[case["dst"]],
              "flip": case["flip"], "swap": case["swap"]}
        return s
    s["bins"] = _histogram(w, h, case["spp"], seed)[0]
    if kind == "blur":
        s["out"] = torch.empty_like(s["bins"])
        return s
    s |= {"spp": case["spp"], "fmt": FORMATS[case["fmt"]], "out": _image(case, case["fmt"])}
    if kind == "tonemap":
        s |= {"map": lr.tonemapper(), "precise": case["precise"]}
        if not case["precise"]:
            s |= {"hist": torch.zeros(lr.HISTOGRAM_BINS, device="cuda", dtype=torch.int64),
                  "max": torch.zeros(1, device="cuda", dtype=torch.int64)}
    else:
        s |= {"base": _tonemap64(s["bins"], case["spp"]).float(), "net": dn.denoiser(params=_weights())}
    return s


def _weights():
    return _kept("weights", lambda: dn.read_params(WORKLOADS / "denoiser_weights.npz"))


def run(s):
    kind = s["kind"]
    if kind == "frame":
        return _run_frame(s)
    if kind == "batch":
        return _run_batch(s)
    if kind == "blur":
        lr.density_blur(s["bins"], s["out"], s["dims"], *DE)
        return s["out"]
    if kind == "tonemap":
        if s["precise"]:
            s["map"].run(s["bins"], s["out"], s["dims"], s["spp"], GAMMA, BRIGHTNESS, VIBRANCY, fmt=s["fmt"])
            return s["out"]
        s["hist"].zero_()
        s["max"].zero_()
        s["map"].run(s["bins"], s["out"], s["dims"], s["spp"], GAMMA, BRIGHTNESS, VIBRANCY, fmt=s["fmt"], precise=False,
                     histogram=s["hist"], max_density_out=s["max"])
        return {"image": s["out"], "histogram": s["hist"], "max": s["max"]}
    if kind == "convert":
        s["conv"].run(s["in"], s["out"], s["dims"], s["src"], s["dst"], flip_y=s["flip"], swap_channels=s["swap"])
        return s["out"]
    if kind == "denoise":
        s["net"].denoise(s["bins"], s["base"], s["out"], s["spp"], fmt=s["fmt"])
        return s["out"]
    loss = s["net"].train_step(s["bins"], s["base"], s["spp"], s["target"], s["lr"])
    return {"loss": loss, "params": s["net"].params()}


# layers of the denoiser: (input channels, output channels)
NET = [(32, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 256), (256, 256), (384, 128), (128, 128),
       (192, 64), (64, 64), (96, 32), (32, 32), (32, 32)]


def work(case):
    """Bytes: inputs once, outputs once. Flops: about 100 per chain step, 12 per blur tap of the mean support,
    60 per tonemapped pixel, 2 per multiply-add of the network."""
    kind, px = case["kind"], float(case["w"] * case["h"])
    if kind == "frame":
        return {"bytes": px * (16 + 8), "flops": 100.0 * px * case["spp"]}
    if kind == "batch":
        if case["genome"] == "anim":
            return {"bytes": case["units"] * px * 24, "flops": 100.0 * case["units"] * px * case["spp"]}
        fl = _workload("hetero_64.json")["flames"][:case["units"]]
        return {"bytes": 24.0 * sum(e["width"] * e["height"] for e in fl),
                "flops": 100.0 * sum(e["width"] * e["height"] * e["spp"] for e in fl)}
    if kind == "blur":
        r = min(9.0, 9.0 / math.sqrt(max(case["spp"], 1.0)))
        return {"bytes": px * 32, "flops": px * 12.0 * (2 * r + 1) ** 2}
    if kind == "tonemap":
        return {"bytes": px * (16 + _channels(case["fmt"]) * (2 if case["fmt"].startswith("half") else 4)), "flops": 60.0 * px}
    if kind == "convert":
        out = _channels(case["dst"]) * (1 if case["dst"].startswith("uchar") else 4)
        return {"bytes": px * (2 * _channels(case["src"]) + out), "flops": 4.0 * px}
    level = [1, 1, 4, 4, 16, 16, 64, 64, 16, 16, 4, 4, 1, 1, 1]
    macs = sum(9.0 * ci * co / lv for (ci, co), lv in zip(NET, level))
    if kind == "denoise":
        return {"bytes": px * (32 + 2 * _channels(case["fmt"])), "flops": 2.0 * macs * px}
    return {"bytes": case["n"] * px * 48 + 4.0 * 4 * sum(9 * ci * co + co for ci, co in NET), "flops": 6.0 * macs * px * case["n"]}


# ------------------------------------------------------------ in 64 bits --
def _blur64(bins):
    rmax, rmin, curve = DE
    b = bins.double()
    h, w, _ = b.shape
    d = b[..., 3]
    r = torch.where(d > 0, (rmax * d.clamp_min(1e-300) ** -curve).clamp(rmin, rmax), torch.zeros_like(d))
    level = torch.round(r * 4.0)
    r = level / 4.0
    rc = torch.ceil(r)
    z = torch.zeros(64, device="cuda", dtype=torch.float64)
    for lv in range(int(rmax * 4) + 1):
        q, c = lv / 4.0, math.ceil(lv / 4.0)
        z[lv] = sum(max(0.0, 1.0 - (x * x + y * y) / (q + 1.0) ** 2) for x in range(-c, c + 1) for y in range(-c, c + 1))
    scaled = torch.where((d > 0)[..., None], b / z[level.long()][..., None], torch.zeros_like(b))
    inv = 1.0 / (r + 1.0) ** 2
    out = torch.zeros_like(b)
    n = int(rmax)
    for dy in range(-n, n + 1):
        for dx in range(-n, n + 1):
            # the sources that reach (x + dx, y + dy)
            ys, xs = slice(max(0, -dy), h - max(0, dy)), slice(max(0, -dx), w - max(0, dx))
            yd, xd = slice(max(0, dy), h - max(0, -dy)), slice(max(0, dx), w - max(0, -dx))
            k = (1.0 - (dx * dx + dy * dy) * inv[ys, xs]).clamp_min(0.0) * (rc[ys, xs] >= max(abs(dx), abs(dy)))
            out[yd, xd] += scaled[ys, xs] * k[..., None]
    return out


def _denoise64(bins, base, spp):
    flat, at, layers = torch.tensor(_weights(), device="cuda", dtype=torch.float64), 0, []
    for ci, co in NET:
        wt = flat[at:at + 9 * ci * co].view(co, 9, ci).permute(0, 2, 1).reshape(co, ci, 3, 3).contiguous()
        layers.append((wt, flat[at + 9 * ci * co:at + 9 * ci * co + co]))
        at += 9 * ci * co + co
    b, t = bins.double(), base.double()
    d = b[..., 3]
    ds = torch.where(d > 0, d, torch.ones_like(d))
    x = torch.zeros((32,) + d.shape, device="cuda", dtype=torch.float64)
    x[0] = torch.log1p(d.clamp_min(0)) / 8
    for j in range(3):
        x[1 + j] = torch.where(d > 0, b[..., j] / ds, torch.zeros_like(d))
        x[6 + j] = t[..., j]
    x[4] = (torch.log(ds) * (4.0 / math.log(2.0)) / 96.0).clamp(0, 1) * (d >= 1)
    x[5] = math.log(max(spp, 1.0)) / 8

    def conv(i, v):
        wt, bias = layers[i]
        v = F.pad(v, (1, 1, 1, 1))
        hh, ww = v.shape[1] - 2, v.shape[2] - 2
        acc = bias[:, None].expand(-1, hh * ww).clone()
        for dy in range(3):
            for dx in range(3):
                acc.addmm_(wt[:, :, dy, dx], v[:, dy:dy + hh, dx:dx + ww].reshape(v.shape[0], -1))
        acc = acc.view(-1, hh, ww)
        return acc if i == len(NET) - 1 else acc.relu_()

    pool = lambda v: F.avg_pool2d(v[None], 2)[0]  # noqa: E731
    up = lambda v: v.repeat_interleave(2, 1).repeat_interleave(2, 2)  # noqa: E731
    s1 = conv(1, conv(0, x))
    s2 = conv(3, conv(2, pool(s1)))
    s3 = conv(5, conv(4, pool(s2)))
    m = conv(7, conv(6, pool(s3)))
    d3 = conv(9, conv(8, torch.cat([up(m), s3])))
    d2 = conv(11, conv(10, torch.cat([up(d3), s2])))
    o = conv(14, conv(13, conv(12, torch.cat([up(d2), s1]))))
    rgb = (t[..., :3] + o[:3].permute(1, 2, 0)).clamp(0, 1)
    a = torch.where(d > 0, (torch.log(ds) * (4.0 / math.log(2.0)) / 96.0).clamp(0, 1), torch.zeros_like(d))
    return torch.cat([rgb, a[..., None]], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("blur", "tonemap", "convert", "denoise"):
        return None  # a render is a random sample; a training step in 64 bits takes too long
    w, h = case["w"], case["h"]
    if kind == "convert":
        if case["dst"].startswith("uchar"):
            return None
        g = torch.Generator(device="cuda").manual_seed(seed)
        v = torch.rand((h, w, _channels(case["src"])), device="cuda", generator=g).half().double()
        if v.shape[2] == 3:
            v = torch.cat([v, torch.ones_like(v[..., :1])], -1)
        if case["swap"]:
            v = v[..., [2, 1, 0, 3]]
        return (v.flip(0) if case["flip"] else v)[..., :_channels(case["dst"])].contiguous()
    bins = _histogram(w, h, case["spp"], seed)[0]
    if kind == "blur":
        return _blur64(bins)
    if kind == "denoise":
        return _denoise64(bins, _tonemap64(bins, case["spp"]).float(), case["spp"])[..., :_channels(case["fmt"])].contiguous()
    image = _tonemap64(bins, case["spp"])[..., :_channels(case["fmt"])].contiguous()
    return image if case["precise"] else {"image": image, "histogram": None, "max": None}
