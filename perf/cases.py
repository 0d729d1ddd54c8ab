"""What is measured: reconstruction by dilation as programs call it.

A case is a dict of plain values.  `kind` says which public entry point it
goes through, the rest what the images are: smoothed noise with bright discs
as the mask and an h-dome or sparse-seed marker, or the spiral corridor, in
the sizes and value laws of the benchmark configurations
(`iwpp.synth`, config0 ... config4), generated on the GPU.  Every
reconstruction is in place, so a pass first puts the marker back into the
buffer that it is done in, as a program with a stream of frames fills it.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "iwpp-mp_gb300"))

import iwpp  # noqa: E402

BYTES = {"u8": 1, "u16": 2, "i32": 4}
LOW = {"u8": 0, "u16": 0, "i32": -(1 << 31)}
HIGH = {"u8": 255, "u16": 65535, "i32": (1 << 31) - 1}
STEP = {"u8": 1, "u16": 257, "i32": 0xFFFFFFFF // 255}  # one level of 255
TORCH = {"u8": torch.uint8, "u16": torch.int16, "i32": torch.int32}  # u16: raw 16-bit storage
ARM_PITCH = 256  # between two turns of the spiral


def listed():
    return [
        # One small frame or region of interest (the size of the smoke run): latency and launches.
        dict(name="small_u8", kind="call", width=300, height=200, dtype="u8", conn=8, sigma=3.0, marker="hdome", h=30),
        # Configuration 0, the ordinary single image.
        dict(name="image_1024_u8", kind="call", width=1024, height=1024, dtype="u8", conn=8, sigma=4.0,
             marker="hdome", h=40),
        # Configuration 1 through the reference's own entry point (uint8, square, 4-connected, no handle).
        dict(name="reference_entry_4096", kind="reference", width=4096, height=4096, dtype="u8", conn=4, sigma=8.0,
             marker="hdome", h=10),
        # Configuration 1's longest propagation: deep domes, 8-connected.
        dict(name="deep_4096_u8", kind="call", width=4096, height=4096, dtype="u8", conn=8, sigma=8.0,
             marker="hdome", h=100),
        # The unique queue, one of the three that the reference has, on configuration 1.
        dict(name="unique_4096_u8", kind="call", width=4096, height=4096, dtype="u8", conn=4, sigma=8.0,
             marker="hdome", h=40, variant="unique"),
        # 16-bit frames of odd width as they lie in a contiguous tensor: rows off the 4-byte boundary.
        dict(name="odd_u16", kind="call", width=3001, height=1999, dtype="u16", conn=8, sigma=4.0, marker="hdome",
             h=60),
        # int32 (labels, distances, fixed point) of a ragged size, 4-connected.
        dict(name="ragged_i32", kind="call", width=1777, height=2049, dtype="i32", conn=4, sigma=4.0,
             marker="hdome", h=40),
        # Large frames with sparse seeds (the served stream's other marker kind, its largest side).
        dict(name="seeds_8192_u8", kind="call", width=8192, height=8192, dtype="u8", conn=8, sigma=4.0,
             marker="sparse", h=0),
        # Configuration 2: the longest paths, one corridor through the whole image.
        dict(name="spiral_16384_u8", kind="call", width=16384, height=16384, dtype="u8", conn=8, sigma=16.0,
             marker="spiral", h=0),
        # Configuration 3: 64 images of mixed sizes, types and connectivities, one graph-captured plan.
        dict(name="plan_64_mixed", kind="plan", count=64, layout=3, low=512, high=3072),
        # A burst of the served stream (configuration 4's laws, sides up to 4096) from pinned host memory.
        dict(name="served_burst", kind="served", count=32, layout=4, low=256, high=4096),
        # The reference's whole-image raster and anti-raster sweeps, one call each.
        dict(name="sweeps_4096_u8", kind="sweeps", width=4096, height=4096, dtype="u8", conn=8, sigma=8.0,
             marker="hdome", h=40),
    ]


def _side(rng, low, high):
    return int(round(math.exp(math.log(low) + rng.random() * (math.log(high) - math.log(low)))))


def draw(rng):
    kind = rng.choice(["call", "call", "call", "call", "call", "reference", "queue", "spiral", "plan", "served",
                       "sweeps"])
    if kind == "plan":
        return dict(kind="plan", count=rng.randint(2, 48), layout=rng.randrange(1 << 20), low=256, high=3072)
    if kind == "served":
        return dict(kind="served", count=rng.randint(2, 24), layout=rng.randrange(1 << 20), low=256, high=4096)
    if kind == "spiral":  # images of 2^26 pixels and up: shorter paths are in the other kinds
        return dict(kind="call", width=rng.randint(8192, 16384), height=rng.randint(8192, 14000),
                    dtype=rng.choice(["u8", "u8", "u16"]), conn=8, sigma=16.0, marker="spiral", h=0)
    case = dict(kind=kind, width=_side(rng, 128, 6000), height=_side(rng, 128, 6000),
                dtype=rng.choice(["u8", "u8", "u8", "u16", "i32"]), conn=rng.choice([4, 8]),
                sigma=rng.choice([3.0, 4.0, 8.0]), marker=rng.choice(["hdome", "hdome", "sparse"]),
                h=rng.randint(5, 120))
    if kind == "queue":
        case.update(kind="call", variant=rng.choice(["unique", "double", "mutex"]))
    if kind == "reference":
        case.update(width=case["height"], dtype="u8", conn=4)
    if rng.random() < 0.4 and kind not in ("reference", "sweeps"):  # frames of a power-of-two-ish width: aligned rows
        case["width"] = -(-case["width"] // 64) * 64
    if kind == "sweeps":  # the sweeps want aligned rows
        case["width"] = -(-case["width"] // 4) * 4
    return case


# ------------------------------------------------------------------ inputs
def _smooth(noise, sigma):
    """Separable Gaussian by shifted sums: the same bits wherever it runs."""
    r = int(math.ceil(3 * sigma))
    taps = [math.exp(-0.5 * (i / sigma) ** 2) for i in range(-r, r + 1)]
    total = sum(taps)
    for dim in (0, 1):
        n = noise.shape[dim]
        left, right = noise.narrow(dim, 0, 1), noise.narrow(dim, n - 1, 1)
        padded = torch.cat([left.expand(*[r if d == dim else -1 for d in (0, 1)]), noise,
                            right.expand(*[r if d == dim else -1 for d in (0, 1)])], dim)
        noise = torch.zeros_like(noise)
        for i, t in enumerate(taps):
            noise.add_(padded.narrow(dim, i, n), alpha=t / total)
    return noise


def _levels(x, dtype):
    """x in [0, 1] over the type's whole range, as int64 (float64 for int32 alone: the others fit float32)."""
    if dtype == "i32":
        return (x.double() * 4294967295.0 - 2147483648.0).to(torch.int64)
    return (x * (256 if dtype == "u8" else 65536)).to(torch.int32).clamp_(max=HIGH[dtype])


def _store(v, dtype):
    if dtype == "u16":
        v = torch.where(v > 32767, v - 65536, v)
    return v.to(TORCH[dtype])


def _mask(width, height, dtype, sigma, discs, g):
    x = _smooth(torch.rand(height, width, generator=g, device="cuda"), sigma)
    lo, hi = x.min(), x.max()
    x = (x - lo) / (hi - lo).clamp(min=1e-9)
    v = _levels(x, dtype)
    del x
    if discs:  # radius 5 to 40, level 180 to 255 of 255
        cx = torch.randint(0, width, (discs, 1, 1), generator=g, device="cuda")
        cy = torch.randint(0, height, (discs, 1, 1), generator=g, device="cuda")
        rad = torch.randint(5, 41, (discs, 1, 1), generator=g, device="cuda")
        level = torch.randint(180, 256, (discs, 1, 1), generator=g, device="cuda") * STEP[dtype] + LOW[dtype]
        d = torch.arange(-40, 41, device="cuda")
        px, py = cx + d[None, None, :], cy + d[None, :, None]
        inside = (d[None, None, :] ** 2 + d[None, :, None] ** 2 <= rad * rad) & (px >= 0) & (px < width) & (py >= 0) & (py < height)
        at = (py.clamp(0, height - 1) * width + px.clamp(0, width - 1)).reshape(-1)
        vals = torch.where(inside, level, LOW[dtype]).reshape(-1).to(v.dtype)
        v = v.reshape(-1).scatter_reduce(0, at, vals, "amax").reshape(height, width)
    return v


def _corridor(v, high):
    """One-pixel square spiral at the type's maximum, inward from (ARM_PITCH / 2, ARM_PITCH / 2)."""
    h, w = v.shape
    p = ARM_PITCH
    l, r, t, b = p // 2, w - 1 - p // 2, p // 2, h - 1 - p // 2
    x, y = l, t
    while True:
        if r <= x:
            break
        v[y, x:r + 1] = high
        x, t = r, t + p
        if b <= y:
            break
        v[y:b + 1, x] = high
        y, r = b, r - p
        if x <= l:
            break
        v[y, l:x + 1] = high
        x, b = l, b - p
        if y <= t:
            break
        v[t:y + 1, x] = high
        y, l = t, l + p


def _pair(case, seed):
    """(marker, mask) on the GPU, contiguous."""
    w, h, dtype = case["width"], case["height"], case["dtype"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    spiral = case["marker"] == "spiral"
    v = _mask(w, h, dtype, case["sigma"], 0 if spiral else max(1, round(2000 * w * h / 4096 ** 2)), g)
    if spiral:
        _corridor(v, HIGH[dtype])
    if case["marker"] == "hdome":
        m = (v - case["h"] * STEP[dtype]).clamp_(min=LOW[dtype])
    else:
        n = 64 if spiral else max(1, round(1e-4 * w * h))
        at = torch.randint(0, w * h, (n,), generator=g, device="cuda")
        if spiral:
            at[0] = (ARM_PITCH // 2) * w + ARM_PITCH // 2
        m = torch.full_like(v, LOW[dtype])
        m.view(-1)[at] = v.view(-1)[at]
    return _store(m, dtype), _store(v, dtype)


def _images(case):
    """The images of a batch or burst: configuration 3's or 4's laws over the case's own sides."""
    r = random.Random(case["layout"])
    served = case["kind"] == "served"
    got = []
    for _ in range(case["count"]):
        c = dict(width=_side(r, case["low"], case["high"]), height=_side(r, case["low"], case["high"]), sigma=4.0,
                 h=r.randint(5, 120))
        c["dtype"] = "u8" if r.random() < (0.8 if served else 0.5) else "u16"
        c["conn"] = 8 if served or r.random() < 0.5 else 4
        c["marker"] = "sparse" if served and r.random() < 0.5 else "hdome"
        got.append(c)
    return got


def prepare(case, seed):
    s = dict(kind=case["kind"])
    if case["kind"] == "served":
        s["server"] = iwpp.Server(memory_budget=8 << 30)
        s["requests"] = []
        for i, c in enumerate(_images(case)):
            m, k = (t.cpu().pin_memory() for t in _pair(c, seed * 1009 + i))
            o = torch.empty_like(m).pin_memory()
            s["requests"].append([t.numpy().view(np.uint16) if c["dtype"] == "u16" else t.numpy() for t in (m, k, o)]
                                 + [c["conn"], (m, k, o)])
        return s
    s["handle"] = iwpp.Handle()
    if case["kind"] == "plan":
        images = _images(case)
        pairs = [_pair(c, seed * 1009 + i) for i, c in enumerate(images)]
        # markers of all images in one buffer, each on a 512-byte boundary: one copy restores them
        ends, at = [], 0
        for m, _ in pairs:
            ends.append(at)
            at += -(-m.numel() * m.element_size() // 512) * 512
        s["markers"], s["buffer"] = (torch.zeros(at, dtype=torch.uint8, device="cuda") for _ in range(2))

        def views(buffer):
            return [buffer[b:b + m.numel() * m.element_size()].view(m.dtype).view(m.shape)
                    for b, (m, _) in zip(ends, pairs)]

        for v, (m, _) in zip(views(s["markers"]), pairs):
            v.copy_(m)
        s["out"] = views(s["buffer"])
        s["masks"] = [k for _, k in pairs]
        s["plan"] = iwpp.Plan(s["handle"], [(o, k, c["conn"]) for o, k, c in zip(s["out"], s["masks"], images)])
        return s
    s["marker"], s["mask"] = _pair(case, seed)
    s["out"] = torch.empty_like(s["marker"])
    s["conn"] = case["conn"]
    s["variant"] = case.get("variant", "default")
    return s


def run(s):
    if s["kind"] == "served":
        server = s["server"]
        tickets = [server.submit(m, k, conn, out=o) for m, k, o, conn, _ in s["requests"]]
        return [server.wait(t)[0].view(np.int16) if r[2].dtype == np.uint16 else server.wait(t)[0]
                for t, r in zip(tickets, s["requests"])]
    if s["kind"] == "plan":
        s["buffer"].copy_(s["markers"])
        s["plan"].launch()
        s["plan"].sync()
        return s["out"]
    out, mask = s["out"], s["mask"]
    out.copy_(s["marker"])
    if s["kind"] == "reference":
        n = out.shape[0]
        iwpp.MorphologicalReconstruction(out.data_ptr(), mask.data_ptr(), n, n, n)
    elif s["kind"] == "sweeps":
        for direction in range(4):
            iwpp.sweep(out, mask, direction, connectivity=s["conn"])
    else:
        iwpp.reconstruct(out, mask, connectivity=s["conn"], variant=s["variant"], handle=s["handle"])
    return out


def work(case):
    """Both planes read once and the result written once, per reconstruction or sweep."""
    if "width" in case:
        n = case["width"] * case["height"] * BYTES[case["dtype"]]
    else:
        n = sum(c["width"] * c["height"] * BYTES[c["dtype"]] for c in _images(case))
    return {"bytes": 3 * n * (4 if case["kind"] == "sweeps" else 1), "flops": 0}


def exact(case, seed):
    """The definition, iterated to its fixed point; images where that is quick."""
    if case["kind"] not in ("call", "reference") or case["width"] * case["height"] > 1 << 20:
        return None
    m, k = _pair(case, seed)
    if case["dtype"] == "u16":
        m, k = (t.to(torch.int64) & 0xFFFF for t in (m, k))
    m, k = m.to(torch.int64), k.to(torch.int64)
    lowest = -(1 << 40)
    while True:
        p = torch.nn.functional.pad(m, (1, 1, 1, 1), value=lowest)
        n = m
        for dy in range(3):
            for dx in range(3):
                if case["conn"] == 8 or dy == 1 or dx == 1:
                    n = torch.maximum(n, p[dy:dy + m.shape[0], dx:dx + m.shape[1]])
        n = torch.maximum(torch.minimum(n, k), m)
        if torch.equal(n, m):
            return _store(m, case["dtype"])
        m = n
