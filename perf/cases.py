"""Performance cases: the work that programs on this framework have it do, each
through its public entry points (hipacc_gb300.api), with the same results in
plain 64-bit torch beside it.

A case is a dict of plain values; "kind" says which program it stands for:

  edges      camera frames: Sobel magnitude with its fused sum and maximum, and
             RGBA to gray (0_Point_Operators, 3_Preprocessing/Sobel)
  conv       one local operator over a batch: a Gaussian mask (f32, bf16, f16,
             u8 storage), or erosion / dilation over a Domain
  separable  a separable Gaussian over a large image
  bilateral  the bilateral filter
  pyramid    Laplacian pyramids of images of uneven sizes, and their collapse
  photo      a photograph through the Harris corner and the Unsharp programs
  train      conv -> bilateral -> MSE: loss and gradients of one training step
  grad       one learnable layer, forward and backward: a convolution, a
             separable filter, a bilateral filter or a MIN / MAX operator
  thumbnail  a frame resampled, with its histogram, sum and maximum
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hipacc_gb300 import api

DEV = "cuda"
TYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "u8": torch.uint8}
BYTES = {"f32": 4, "bf16": 2, "f16": 2, "u8": 1}
BOUNDARY = {"clamp": api.CLAMP, "repeat": api.REPEAT, "mirror": api.MIRROR, "constant": api.CONSTANT}
MODES = ("nn", "lf", "b5", "cf", "l3")


def listed():
    return [
        # a preview frame: launches and host time count
        {"name": "edges_640x480", "kind": "edges", "w": 640, "h": 480, "boundary": "clamp"},
        # the largest camera frame, the framework's headline step
        {"name": "edges_4096x4096", "kind": "edges", "w": 4096, "h": 4096, "boundary": "mirror"},
        # Gaussian blur of a batch of float images
        {"name": "conv5_f32_64x1024x1024", "kind": "conv", "op": "gauss", "dtype": "f32", "size": 5, "n": 64,
         "w": 1024, "h": 1024, "boundary": "clamp"},
        # Gaussian blur of byte images whose rows have an odd length (decoded pictures)
        {"name": "conv5_u8_16x1021x767", "kind": "conv", "op": "gauss", "dtype": "u8", "size": 5, "n": 16,
         "w": 1021, "h": 767, "boundary": "mirror"},
        # smoothing one very large image in reduced-precision storage
        {"name": "separable9_bf16_8192x8192", "kind": "separable", "dtype": "bf16", "size": 9, "n": 1, "w": 8192,
         "h": 8192, "boundary": "repeat"},
        # edge-preserving denoising
        {"name": "bilateral13_f32_4096x4096", "kind": "bilateral", "dtype": "f32", "size": 13, "n": 1, "w": 4096,
         "h": 4096, "boundary": "repeat"},
        # detail manipulation over a batch of photographs of uneven sizes
        {"name": "pyramid8_6_images", "kind": "pyramid", "n": 6, "least": 257, "most": 4096, "pick": 4096,
         "levels": 8, "boundary": "mirror"},
        # corner detection and sharpening of a 12-megapixel photograph
        {"name": "photo_4032x3024", "kind": "photo", "w": 4032, "h": 3024, "boundary": "clamp"},
        # one step of learning a mask and a range width
        {"name": "train_16x2048x2048", "kind": "train", "n": 16, "w": 2048, "h": 2048, "boundary": "mirror"},
        # a learnable separable layer
        {"name": "grad_separable9_4x1920x1080", "kind": "grad", "op": "separable", "size": 9, "n": 4, "w": 1920,
         "h": 1080, "boundary": "mirror"},
        # a dilation layer on odd-sized crops
        {"name": "grad_max5_8x509x381", "kind": "grad", "op": "max", "size": 5, "n": 8, "w": 509, "h": 381,
         "boundary": "clamp"},
        # a frame enlarged for display, with its statistics
        {"name": "thumbnail_cf_2048_to_4096", "kind": "thumbnail", "mode": "cf", "w": 2048, "h": 2048, "dw": 4096,
         "dh": 4096, "bins": 256},
    ]


# ---------------------------------------------------------------- drawn cases


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, most_px):
    """Width and height, spread over their logarithm; two in three widths are as
    they come (odd and ragged), the others a multiple of 64."""
    while True:
        w, h = _log(rng, lo, hi), _log(rng, lo, hi)
        if rng.random() < 0.34:
            w = max(64, w // 64 * 64)
        if w * h <= most_px:
            return w, h


def _batch(rng, w, h, most_px, most):
    return _log(rng, 1, max(1, min(most, most_px // (w * h))))


def draw(rng):
    kind = rng.choice(("edges", "conv", "conv", "separable", "bilateral", "pyramid", "photo", "train", "grad", "grad",
                       "thumbnail"))
    b = rng.choice(("clamp", "repeat", "mirror", "constant"))
    if kind in ("edges", "photo"):
        w, h = _size(rng, 240, 4096, 1 << 24)
        return {"kind": kind, "w": w, "h": h, "boundary": b}
    if kind == "conv":
        op = rng.choice(("gauss", "gauss", "erode", "dilate"))
        size = rng.choice((3, 5, 7, 9, 11, 13) if op == "gauss" else (3, 5, 7))
        w, h = _size(rng, 128, 4096, 1 << 24)
        return {"kind": kind, "op": op, "dtype": rng.choice(("f32", "bf16", "f16", "u8")), "size": size,
                "n": _batch(rng, w, h, 1 << 26 if size <= 5 else 1 << 25, 64), "w": w, "h": h, "boundary": b}
    if kind == "separable":
        w, h = _size(rng, 256, 8192, 1 << 26)
        return {"kind": kind, "dtype": rng.choice(("f32", "bf16", "f16")), "size": rng.choice((3, 5, 7, 9, 11, 13, 15)),
                "n": _batch(rng, w, h, 1 << 25, 16), "w": w, "h": h, "boundary": b}
    if kind == "bilateral":
        w, h = _size(rng, 256, 4096, 1 << 24)
        return {"kind": kind, "dtype": rng.choice(("f32", "bf16", "f16")), "size": rng.choice((3, 5, 7, 9, 11, 13)),
                "n": _batch(rng, w, h, 1 << 24, 8), "w": w, "h": h, "boundary": b}
    if kind == "pyramid":
        levels = rng.randint(3, 8)
        return {"kind": kind, "n": _log(rng, 1, 63 // (levels + 1)), "least": 257, "most": _log(rng, 400, 3000),
                "pick": rng.randint(1, 9999), "levels": levels, "boundary": rng.choice(("clamp", "mirror"))}
    if kind == "train":
        w, h = _size(rng, 128, 2048, 1 << 22)
        return {"kind": kind, "n": _batch(rng, w, h, 1 << 24, 16), "w": w, "h": h,
                "boundary": rng.choice(("clamp", "mirror", "constant"))}
    if kind == "grad":
        op = rng.choice(("conv", "separable", "bilateral", "min", "max"))
        size = rng.choice({"conv": (3, 5, 7), "separable": (3, 5, 7, 9, 11, 13), "bilateral": (3, 5, 7, 9),
                           "min": (3, 5, 7), "max": (3, 5, 7)}[op])
        w, h = _size(rng, 128, 4096, 1 << 23)
        return {"kind": kind, "op": op, "size": size, "n": _batch(rng, w, h, 1 << 23, 16), "w": w, "h": h,
                "boundary": b}
    w, h = _size(rng, 240, 4096, 1 << 23)
    f = math.exp(rng.uniform(math.log(0.25), math.log(2.0)))
    return {"kind": "thumbnail", "mode": rng.choice(MODES), "w": w, "h": h, "dw": max(64, int(w * f)),
            "dh": max(64, int(h * f)), "bins": rng.choice((64, 256, 256, 1024))}


# ---------------------------------------------------------------- inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _field(g, n, h, w):
    """Photograph-like values in [0, 1]: a smooth field, shifted per image, and sensor noise."""
    y = torch.arange(h, device=DEV, dtype=torch.float32)[None, :, None]
    x = torch.arange(w, device=DEV, dtype=torch.float32)[None, None, :]
    a = torch.rand((n, 2, 1, 1), device=DEV, generator=g) * (2 * math.pi)
    f = 0.5 + 0.25 * torch.sin(2 * math.pi * x / 512.0 + a[:, 0]) * torch.cos(2 * math.pi * y / 384.0 + a[:, 1])
    f += 0.05 * torch.randn((n, h, w), device=DEV, generator=g)
    return f.clamp_(0.0, 1.0)


def _bytes(g, n, h, w):
    return (_field(g, n, h, w) * 255.0).round_().to(torch.uint8)


def _rgba(g, h, w):
    return torch.stack([_bytes(g, 1, h, w)[0] for _ in range(4)], dim=-1).contiguous()


def _taps(size):
    sigma = 0.3 * ((size - 1) * 0.5 - 1) + 0.8
    a = np.arange(-(size // 2), size // 2 + 1, dtype=np.float64)
    t = np.exp(-a ** 2 / (2 * sigma * sigma))
    return (t / t.sum()).astype(np.float32)


def _gauss(size):
    t = _taps(size).astype(np.float64)
    return np.outer(t, t).astype(np.float32)


def _smask(size):
    a = np.arange(-(size // 2), size // 2 + 1, dtype=np.float64)
    s = size / 4.0
    return np.exp(-(a[None, :] ** 2 + a[:, None] ** 2) / (2 * s * s)).astype(np.float32)


def _element(size):
    """A disc, the usual structuring element."""
    a = np.arange(size) - size // 2
    return (a[None, :] ** 2 + a[:, None] ** 2 <= (size / 2.0) ** 2).astype(np.uint8)


def _learned(size, seed):
    return _gauss(size) + np.random.default_rng(seed).normal(0, 0.02, (size, size)).astype(np.float32)


SIGMA = 0.1
BINOMIAL = np.outer([1, 4, 6, 4, 1], [1, 4, 6, 4, 1]).astype(np.float32) / 256.0


def _pyramid_sizes(c):
    r = np.random.default_rng(c["pick"])
    return r.integers(c["least"], c["most"] + 1, c["n"]), r.integers(c["least"], c["most"] + 1, c["n"])


def prepare(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    s = {"case": c, "boundary": BOUNDARY.get(c.get("boundary"), api.CLAMP)}
    if kind == "edges":
        s["img"], s["rgba"] = _bytes(g, 1, c["h"], c["w"])[0], _rgba(g, c["h"], c["w"])
        s["mag"], s["gray"] = torch.empty_like(s["img"]), torch.empty_like(s["img"])
        s["sum"] = torch.zeros(1, dtype=torch.int64, device=DEV)
        s["max"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    elif kind == "photo":
        s["img"], s["rgba"] = _bytes(g, 1, c["h"], c["w"])[0], _rgba(g, c["h"], c["w"])
        s["corners"], s["sharp"] = torch.empty_like(s["img"]), torch.empty_like(s["rgba"])
    elif kind in ("conv", "separable", "bilateral"):
        if c["dtype"] == "u8":
            s["x"] = _bytes(g, c["n"], c["h"], c["w"])
        else:
            s["x"] = _field(g, c["n"], c["h"], c["w"]).to(TYPES[c["dtype"]])
        s["y"] = torch.empty_like(s["x"])
        if kind == "conv":
            s["mask"] = _gauss(c["size"]) if c["op"] == "gauss" else None
            s["domain"] = None if c["op"] == "gauss" else _element(c["size"])
            s["reduce"] = {"gauss": api.SUM, "erode": api.MIN, "dilate": api.MAX}[c["op"]]
        else:
            s["mask"] = _taps(c["size"]) if kind == "separable" else _smask(c["size"])
    elif kind == "pyramid":
        ws, hs = _pyramid_sizes(c)
        s["plan"] = api.PyramidPlan(ws, hs, c["levels"], BINOMIAL, s["boundary"])
        s["images"] = [_field(g, 1, int(h), int(w))[0] for w, h in zip(ws, hs)]
        s["slots"] = [s["plan"].gauss(i, 0) for i in range(c["n"])]
        s["laps"] = [[s["plan"].lap(i, k) for k in range(c["levels"] - 1)] for i in range(c["n"])]
        s["last"] = [s["plan"].gauss(i, c["levels"] - 1) for i in range(c["n"])]
        for t in s["slots"] + s["last"] + sum(s["laps"], []):
            t.plan = s["plan"]  # the levels lie in the plan's memory: whoever holds one holds the plan
    elif kind == "train":
        s["x"], s["t"] = _field(g, c["n"], c["h"], c["w"]), _field(g, c["n"], c["h"], c["w"])
        s["mask"] = torch.from_numpy(_learned(7, seed)).to(DEV)
        s["sigma"] = torch.full((1,), SIGMA, device=DEV)
        s["smask"] = _smask(9)
    elif kind == "grad":
        s["x"] = _field(g, c["n"], c["h"], c["w"])
        s["dy"] = torch.randn((c["n"], c["h"], c["w"]), device=DEV, generator=g) / math.sqrt(c["h"] * c["w"])
        s["y"] = torch.empty_like(s["x"])
        if c["op"] == "conv":
            s["mask"] = _learned(c["size"], seed)
        elif c["op"] == "separable":
            r = np.random.default_rng(seed)
            s["row"], s["col"] = (_taps(c["size"]) + r.normal(0, 0.02, c["size"]).astype(np.float32) for _ in "rc")
        elif c["op"] == "bilateral":
            s["mask"] = _smask(c["size"])
        else:
            s["domain"], s["reduce"] = _element(c["size"]), api.MIN if c["op"] == "min" else api.MAX
    else:
        s["u8"], s["x"] = _bytes(g, 1, c["h"], c["w"])[0], _field(g, 1, c["h"], c["w"])[0]
        s["y"] = torch.empty((c["dh"], c["dw"]), device=DEV)
        s["bins"] = torch.empty(c["bins"], dtype=torch.int32, device=DEV)
    return s


# ---------------------------------------------------------------- one pass


def run(s):
    c, b = s["case"], s["boundary"]
    kind = c["kind"]
    if kind == "edges":
        api.sobel_mag(s["img"], s["mag"], boundary=b, sum_out=s["sum"], max_out=s["max"])
        api.gray(s["rgba"], s["gray"])
        return s["mag"], s["sum"], s["max"], s["gray"]
    if kind == "photo":
        return api.harris(s["img"], s["corners"], boundary=b), api.unsharp(s["rgba"], s["sharp"], boundary=b)
    if kind == "conv":
        return api.local_op(s["x"], s["y"], mask=s["mask"], domain=s["domain"], reduce=s["reduce"], boundary=b)
    if kind == "separable":
        return api.separable(s["x"], s["y"], s["mask"], s["mask"], boundary=b)
    if kind == "bilateral":
        return api.bilateral(s["x"], s["y"], s["mask"], SIGMA, boundary=b)
    if kind == "pyramid":
        torch._foreach_copy_(s["slots"], s["images"])
        s["plan"].decompose()
        s["plan"].collapse()
        return s["laps"], s["last"], s["slots"]
    if kind == "train":
        return api.conv_bilateral_mse(s["x"], s["t"], s["mask"], s["sigma"], s["smask"], boundary=b)
    if kind == "grad":
        if c["op"] == "conv":
            y = api.local_op(s["x"], s["y"], mask=s["mask"], boundary=b)
            return y, api.local_op_adjoint(s["dy"], s["mask"], boundary=b, inp=s["x"])
        if c["op"] == "separable":
            y = api.separable(s["x"], s["y"], s["row"], s["col"], boundary=b)
            return y, api.separable_adjoint(s["x"], s["dy"], s["row"], s["col"], boundary=b)
        if c["op"] == "bilateral":
            y = api.bilateral(s["x"], s["y"], s["mask"], SIGMA, boundary=b)
            return y, api.bilateral_adjoint(s["x"], s["dy"], s["mask"], SIGMA, boundary=b)
        y = api.local_op(s["x"], s["y"], domain=s["domain"], reduce=s["reduce"], boundary=b)
        return y, api.minmax_adjoint(s["x"], s["dy"], s["reduce"], domain=s["domain"], boundary=b)
    y = api.resample(s["x"], s["y"], c["mode"])
    bins = api.histogram(s["u8"], c["bins"], bins=s["bins"])
    return y, bins, api.reduce(s["u8"], api.SUM), api.reduce(s["x"], api.MAX)


# ---------------------------------------------------------------- work


def work(case):
    c, kind = case, case["kind"]
    px = c.get("n", 1) * c.get("w", 0) * c.get("h", 0)
    if kind == "edges":
        return {"bytes": 7 * px, "flops": 20 * px}
    if kind == "photo":
        return {"bytes": 10 * px, "flops": 130 * px}
    if kind == "conv":
        taps = c["size"] ** 2 if c["op"] == "gauss" else int(_element(c["size"]).sum())
        return {"bytes": 2 * BYTES[c["dtype"]] * px, "flops": (2 if c["op"] == "gauss" else 1) * taps * px}
    if kind == "separable":
        return {"bytes": 2 * BYTES[c["dtype"]] * px, "flops": 4 * c["size"] * px}
    if kind == "bilateral":
        return {"bytes": 2 * BYTES[c["dtype"]] * px, "flops": 8 * c["size"] ** 2 * px}
    if kind == "pyramid":
        ws, hs = _pyramid_sizes(c)
        level = [sum((int(w) >> k) * (int(h) >> k) for w, h in zip(ws, hs)) for k in range(c["levels"])]
        # image in, levels out, levels in, image out
        return {"bytes": 4 * (2 * level[0] + 2 * sum(level[:-1]) + level[-1]),
                "flops": sum(50 * b + 18 * a for a, b in zip(level, level[1:]))}
    if kind == "train":
        return {"bytes": 12 * px, "flops": (3 * 2 * 49 + 81 * 30) * px}
    if kind == "grad":
        k = c["size"]
        flops = {"conv": 6 * k * k, "separable": 12 * k, "bilateral": 30 * k * k}.get(c["op"])
        if flops is None:
            flops = 2 * int(_element(k).sum())
        return {"bytes": 16 * px, "flops": flops * px}
    out, n = c["dw"] * c["dh"], {"nn": 0, "lf": 2, "b5": 4, "cf": 4, "l3": 6}[c["mode"]]
    return {"bytes": 5 * px + 4 * out, "flops": 2 * n * (n + 1) * out + 3 * px}


# ---------------------------------------------------------------- the same in 64 bits


def _reach(n, r, boundary):
    """Where positions -r .. n + r - 1 of an axis are read, and whether they lie inside."""
    i = torch.arange(-r, n + r, device=DEV)
    inside = (i >= 0) & (i < n)
    if boundary == "repeat":
        return i % n, inside | True
    if boundary == "mirror":
        i = i % (2 * n)
        return torch.where(i < n, i, 2 * n - 1 - i), inside | True
    return i.clamp(0, n - 1), inside if boundary == "constant" else inside | True


class _Pad:
    """Images with their boundary around them, and the transpose of that."""

    def __init__(self, h, w, ry, rx, boundary):
        self.iy, oky = _reach(h, ry, boundary)
        self.ix, okx = _reach(w, rx, boundary)
        self.ok = (oky[:, None] & okx[None, :]).double()
        self.h, self.w = h, w

    def __call__(self, x):
        return x[..., self.iy, :][..., self.ix] * self.ok

    def back(self, g):
        g = g * self.ok
        t = torch.zeros(g.shape[:-1] + (self.w,), dtype=g.dtype, device=DEV).index_add_(-1, self.ix, g)
        return torch.zeros(g.shape[:-2] + (self.h, self.w), dtype=g.dtype, device=DEV).index_add_(-2, self.iy, t)


def _correlate(x, mask, boundary):
    kh, kw = mask.shape
    h, w = x.shape[-2:]
    p = _Pad(h, w, kh // 2, kw // 2, boundary)(x)
    y = torch.zeros_like(x)
    for a in range(kh):
        for b in range(kw):
            y.add_(p[..., a:a + h, b:b + w], alpha=float(mask[a, b]))
    return y


def _correlate_back(x, g, mask, boundary):
    """Gradients of _correlate for its input and its mask."""
    kh, kw = mask.shape
    h, w = x.shape[-2:]
    pad = _Pad(h, w, kh // 2, kw // 2, boundary)
    p = pad(x)
    gp, gm = torch.zeros_like(p), torch.zeros((kh, kw), dtype=torch.float64, device=DEV)
    for a in range(kh):
        for b in range(kw):
            gp[..., a:a + h, b:b + w].add_(g, alpha=float(mask[a, b]))
            gm[a, b] = (p[..., a:a + h, b:b + w] * g).sum()
    return pad.back(gp), gm


def _ranked(x, domain, reduce, boundary):
    """MIN / MAX over a Domain, and the tap that gave it (the last of equal ones)."""
    k = domain.shape[0]
    h, w = x.shape[-2:]
    p = _Pad(h, w, k // 2, k // 2, boundary)(x)
    most = reduce == api.MAX
    f = torch.finfo(torch.float32)
    y = torch.full_like(x, f.tiny if most else f.max)
    won = torch.full(x.shape, -1, dtype=torch.int64, device=DEV)
    for a in range(k):
        for b in range(k):
            if domain[a, b]:
                v = p[..., a:a + h, b:b + w]
                new = ~((y > v) if most else (y < v))
                y, won = torch.where(new, v, y), torch.where(new, a * k + b, won)
    return y, won


def _ranked_back(g, won, k, boundary):
    h, w = g.shape[-2:]
    pad = _Pad(h, w, k // 2, k // 2, boundary)
    gp = torch.zeros(g.shape[:-2] + pad.ok.shape, dtype=torch.float64, device=DEV)
    for a in range(k):
        for b in range(k):
            gp[..., a:a + h, b:b + w].add_(torch.where(won == a * k + b, g, 0.0))
    return pad.back(gp)


def _range_filter(x, smask, sigma, boundary):
    """(sum of weights, result) of the bilateral filter."""
    k = smask.shape[0]
    h, w = x.shape[-2:]
    p = _Pad(h, w, k // 2, k // 2, boundary)(x)
    c = 0.5 / (sigma * sigma)
    sw, sv = torch.zeros_like(x), torch.zeros_like(x)
    for a in range(k):
        for b in range(k):
            v = p[..., a:a + h, b:b + w]
            t = torch.exp(-c * (v - x) ** 2) * float(smask[a, b])
            sw += t
            sv += t * v
    return sw, sv / sw


def _range_filter_back(x, g, smask, sigma, boundary):
    """Gradients of the bilateral filter for its input and its range width."""
    k = smask.shape[0]
    h, w = x.shape[-2:]
    pad = _Pad(h, w, k // 2, k // 2, boundary)
    p, c = pad(x), 0.5 / (sigma * sigma)
    sw, y = _range_filter(x, smask, sigma, boundary)
    q = g / sw
    gx, gp, gc = torch.zeros_like(x), torch.zeros_like(p), 0.0
    for a in range(k):
        for b in range(k):
            v = p[..., a:a + h, b:b + w]
            d = v - x
            t = torch.exp(-c * d * d) * float(smask[a, b]) * q
            e = t * (v - y)
            gc = gc - (e * d * d).sum()
            e = e * (-2.0 * c) * d
            gp[..., a:a + h, b:b + w].add_(t + e)
            gx -= e
    return gx + pad.back(gp), gc * (-1.0 / sigma ** 3)


def _positions(n, m):
    """Where the m samples of an axis of n lie, in the accessor's 32 bits."""
    scale = np.float32(n) / np.float32(m)
    # scale / 2 + scale * i, rounded once
    return torch.from_numpy((np.float64(scale) * np.arange(m) + np.float64(scale * np.float32(0.5))).astype(np.float32))


def _weights(mode, d):
    d = d.abs()
    if mode == "b5":
        return torch.where(d < 0.5, 0.75, torch.where(d < 1.0, 0.5, torch.where(d < 1.5, 0.125, 0.0))).double()
    if mode == "cf":
        near = 1.5 * d ** 3 - 2.5 * d ** 2 + 1.0
        far = -0.5 * d ** 3 + 2.5 * d ** 2 - 4.0 * d + 2.0
        return torch.where(d < 1.0, near, torch.where(d < 2.0, far, 0.0))
    s = torch.sinc(d / 3.0) * torch.sinc(d)
    return torch.where(d < 3.0, s, 0.0)


def _axis(mode, n, m):
    """Taps and weights of one axis of the resampling accessor, m x taps each."""
    x = _positions(n, m)
    if mode == "nn":
        return x.long().clamp(0, n - 1)[:, None].to(DEV), torch.ones((m, 1), dtype=torch.float64, device=DEV), None
    x = (x if mode == "b5" else x - 0.5).clamp(min=0.0)
    i = x.long()
    f = (x - i.float()).double()
    if mode == "lf":
        t, wt = torch.stack([i, i + 1], 1), torch.stack([1 - f, f], 1)
        return t.clamp(0, n - 1).to(DEV), wt.to(DEV), None
    j = torch.arange(6 if mode == "l3" else 4)
    if mode == "b5":
        wt = _weights(mode, (f + 1.0)[:, None] - j)
    else:
        wt = _weights(mode, f[:, None] - (2.0 if mode == "l3" else 1.0) + j)
    first = i[:, None] + j - (2 if mode == "l3" else 1)
    return first.clamp(0, n - 1).to(DEV), wt.to(DEV), (i[:, None] + j - 1).clamp(0, n - 1).to(DEV)


def _resample(x, mode, dh, dw):
    h, w = x.shape
    cx, wx, _ = _axis(mode, w, dw)
    cy, wy, rows = _axis(mode, h, dh)
    cy = cy if rows is None else rows
    plain = torch.zeros((h, dw), dtype=torch.float64, device=DEV)
    for j in range(cx.shape[1]):
        plain += x[:, cx[:, j]] * wx[:, j]
    second = plain
    if mode == "l3":  # the accessor weighs the fifth tap of its second row as the sixth
        second = plain + x[:, cx[:, 4]] * (wx[:, 5] - wx[:, 4])
    y = torch.zeros((dh, dw), dtype=torch.float64, device=DEV)
    for k in range(cy.shape[1]):
        y += (second if k == 1 else plain)[cy[:, k]] * wy[:, k, None]
    return y


def _pyramid(x, levels, boundary):
    g, laps = x, []
    for _ in range(levels - 1):
        h, w = g.shape
        iy, ix = _positions(h, h // 2).long().clamp(max=h - 1), _positions(w, w // 2).long().clamp(max=w - 1)
        small = _correlate(g, BINOMIAL, boundary)[iy.to(DEV)][:, ix.to(DEV)]
        laps.append(g - _resample(small, "lf", h, w))
        g = small
    return laps, g


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("edges", "photo") or c.get("dtype") == "u8":
        return None  # bytes and whole numbers
    s, b = prepare(case, seed), c.get("boundary")
    if kind == "pyramid":
        laps, last, back = [], [], []
        for x in s["images"]:
            x = x.double()
            la, g = _pyramid(x, c["levels"], b)
            laps.append(la)
            last.append(g)
            back.append(x)  # the collapse of a decomposition is the image
        return laps, last, back
    if kind == "thumbnail":
        return _resample(s["x"].double(), c["mode"], c["dh"], c["dw"]), None, None, float(s["x"].max())
    if kind == "conv":
        if c["op"] != "gauss":
            return _ranked(s["x"].double(), s["domain"], s["reduce"], b)[0]
        return torch.stack([_correlate(x.double(), s["mask"], b) for x in s["x"]])
    if kind == "separable":
        t = s["mask"]
        return torch.stack([_correlate(_correlate(x.double(), t[None, :], b), t[:, None], b) for x in s["x"]])
    if kind == "bilateral":
        return torch.stack([_range_filter(x.double(), s["mask"], SIGMA, b)[1] for x in s["x"]])
    if kind == "train":
        m = s["mask"].double().cpu().numpy()
        n = float(s["x"].numel())
        sigma = float(s["sigma"])
        loss, gs, gx, gm = 0.0, 0.0, [], torch.zeros((7, 7), dtype=torch.float64, device=DEV)
        for x, t in zip(s["x"].double(), s["t"].double()):
            y1 = _correlate(x, m, b)
            y = _range_filter(y1, s["smask"], sigma, b)[1]
            loss = loss + ((y - t) ** 2).sum() / n
            g1, d = _range_filter_back(y1, 2.0 * (y - t) / n, s["smask"], sigma, b)
            gs = gs + d
            dx, dm = _correlate_back(x, g1, m, b)
            gx.append(dx)
            gm += dm
        return loss.reshape(1), torch.stack(gx), gm, gs.reshape(1)
    ys, gx, ga, gb = [], [], 0.0, 0.0
    for x, g in zip(s["x"].double(), s["dy"].double()):
        if c["op"] == "conv":
            ys.append(_correlate(x, s["mask"], b))
            d, m = _correlate_back(x, g, s["mask"], b)
            ga = ga + m
        elif c["op"] == "separable":
            row, col = s["row"][None, :], s["col"][:, None]
            t = _correlate(x, row, b)
            ys.append(_correlate(t, col, b))
            gt, m = _correlate_back(t, g, col, b)
            gb = gb + m.reshape(-1)
            d, m = _correlate_back(x, gt, row, b)
            ga = ga + m.reshape(-1)
        elif c["op"] == "bilateral":
            ys.append(_range_filter(x, s["mask"], SIGMA, b)[1])
            d, m = _range_filter_back(x, g, s["mask"], SIGMA, b)
            ga = ga + m.reshape(1)
        else:
            y, won = _ranked(x, s["domain"], s["reduce"], b)
            ys.append(y)
            d = _ranked_back(g, won, c["size"], b)
        gx.append(d)
    y, gx = torch.stack(ys), torch.stack(gx)
    return (y, {"conv": (gx, ga), "separable": (gx, ga, gb), "bilateral": (gx, ga)}.get(c["op"], gx))
