"""The workloads the engine's speed is watched on: what they are, how one pass
of each is run through the public entry points, and what it returns in 64 bits.

    listed()            the named workloads
    draw(rng)           one more of the same ranges
    prepare(case, seed) the inputs and the engine a program holds before the call
    run(state)          one pass; returns its outputs
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   run()'s outputs in float64, from plain torch operations

Kinds of work:
    transform   the drop-in host call, Transformer(...).getTransform, regular mode
    ortho       the same in orthonormal mode (stretched image, Hermite circus)
    extended    regular and Hermite circus of one image in one host call
    sinograms   rotate + T-functionals of a device-resident image
    circus      P-functionals of a device-resident sinogram stack
    batch       many uneven device-resident images through the batched engine
    grad        circus functions of device images, forward and backward
"""
import math

import numpy as np
import torch

import tracetransform_gb300 as tt
from tracetransform_gb300 import autograd
from tracetransform_gb300.api import transform_extended
from tracetransform_gb300.device import Engine

DEV = "cuda:0"


def listed():
    return [
        # the smallest call a program makes: a thumbnail, 90 angles, host in and out
        {"name": "transform_64", "kind": "transform", "rows": 64, "cols": 64, "step": 4,
         "t": "012345", "p": "123"},
        # an ordinary image through the drop-in call (the single256 workload)
        {"name": "transform_256", "kind": "transform", "rows": 256, "cols": 256, "step": 1,
         "t": "012345", "p": "123"},
        # the reference's orthonormal mode on a camera-like odd-sized image
        {"name": "ortho_300x211", "kind": "ortho", "rows": 300, "cols": 211, "step": 1,
         "t": "0124", "p": "12345"},
        # a large image with both circus kinds (the single1024 workload, whole call)
        {"name": "extended_1024", "kind": "extended", "rows": 1024, "cols": 1024, "angles": 360,
         "t": "01234567", "p": "123", "h": "12345"},
        # an image kept on the device, plain functionals, ragged sides
        {"name": "sinograms_389x640", "kind": "sinograms", "rows": 389, "cols": 640,
         "angles": 360, "t": "012345"},
        # every T-functional of a large device-resident image
        {"name": "sinograms_1024", "kind": "sinograms", "rows": 1024, "cols": 1024,
         "angles": 360, "t": "01234567"},
        # the largest image, half-degree angles (the single4096 workload's sinograms)
        {"name": "sinograms_4096", "kind": "sinograms", "rows": 4096, "cols": 4096,
         "angles": 720, "t": "01234567"},
        # P-functionals alone, over the stack of an ordinary large image
        {"name": "circus_1449", "kind": "circus", "n": 1449, "angles": 360, "stack": 8,
         "p": "123"},
        # the same of the largest image's columns
        {"name": "circus_5793", "kind": "circus", "n": 5793, "angles": 720, "stack": 8,
         "p": "123"},
        # a mixed bag of images per call (the batch512 workload's sizes, a quarter of it)
        {"name": "batch_128", "kind": "batch", "images": 128, "lo": 64, "hi": 512,
         "t": "012345", "p": "123"},
        # a training step over a batch of images (the grad64 workload)
        {"name": "grad_64x256", "kind": "grad", "images": 64, "rows": 256, "cols": 256,
         "angles": 360, "t": "012", "p": "13"},
        # gradients of one large, odd-sized image (reconstruction from circus functions)
        {"name": "grad_1x777x1000", "kind": "grad", "images": 1, "rows": 777, "cols": 1000,
         "angles": 180, "t": "012", "p": "13"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["transform", "ortho", "extended", "sinograms", "circus", "batch", "grad"])
    if kind == "transform":
        return {"kind": kind, "rows": _log(rng, 24, 600), "cols": _log(rng, 24, 600),
                "step": rng.choice([1, 2, 3, 5]), "t": rng.choice(["012345", "0", "01234567"]),
                "p": rng.choice(["123", "12", "3"])}
    if kind == "ortho":
        return {"kind": kind, "rows": _log(rng, 48, 800), "cols": _log(rng, 48, 800),
                "step": rng.choice([1, 2, 3, 5]), "t": rng.choice(["0", "012", "01245"]),
                "p": rng.choice(["123", "12345"])}
    if kind == "extended":
        rows = _log(rng, 128, 1024)
        return {"kind": kind, "rows": rows, "cols": _log(rng, 128, 1024),
                "angles": rng.randrange(60, min(361, rows)), "t": rng.choice(["0124", "01234567"]),
                "p": "123", "h": rng.choice(["123", "12345"])}
    if kind == "sinograms":
        return {"kind": kind, "rows": _log(rng, 40, 2500), "cols": _log(rng, 40, 2500),
                "angles": rng.choice([45, 180, 360, 719]),
                "t": rng.choice(["0", "012", "012345", "01234567", "67"])}
    if kind == "circus":
        return {"kind": kind, "n": _log(rng, 40, 5793), "angles": _log(rng, 45, 720),
                "stack": rng.randrange(1, 9), "p": rng.choice(["123", "13", "2"])}
    if kind == "batch":
        lo = rng.randrange(24, 129)
        return {"kind": kind, "images": _log(rng, 3, 128), "lo": lo,
                "hi": rng.randrange(lo + 20, 513), "t": rng.choice(["012345", "012", "0"]),
                "p": rng.choice(["123", "13"])}
    return {"kind": kind, "images": _log(rng, 1, 32), "rows": _log(rng, 32, 400),
            "cols": _log(rng, 32, 400), "angles": rng.choice([90, 180, 360]),
            "t": rng.choice(["012", "0"]), "p": rng.choice(["13", "1"])}


# ---- inputs -----------------------------------------------------------------------

def _image(rows, cols, seed):
    """Gaussian blobs plus noise as an 8-bit picture scaled to [0, 1] (what
    gray2mat gives), float32 on the device, (rows, cols)."""
    rng = np.random.default_rng(seed)
    side = min(rows, cols)
    k = int(np.clip(side // 32, 4, 64))

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)

    cx, cy = dev(rng.uniform(0, cols, k)), dev(rng.uniform(0, rows, k))
    sg, am = dev(rng.uniform(side / 32, side / 6, k)), dev(rng.uniform(40, 200, k))
    y = torch.arange(rows, device=DEV, dtype=torch.float32)[:, None]
    x = torch.arange(cols, device=DEV, dtype=torch.float32)[:, None]
    gy = torch.exp(-(y - cy) ** 2 / (2 * sg ** 2))
    gx = torch.exp(-(x - cx) ** 2 / (2 * sg ** 2))
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)
    img = torch.zeros((rows, cols), device=DEV)
    for b in range(k):  # rank-one blobs, summed in a fixed order
        img += am[b] * gy[:, b:b + 1] * gx[:, b][None, :]
    img += 16 * torch.rand((rows, cols), generator=g, device=DEV)
    return torch.round(img.clamp(0, 255)) / 255


def _images(case, seed):
    if case["kind"] == "batch":
        rng = np.random.default_rng(case["images"] * 1000003 + case["lo"] * 1009 + case["hi"])
        sizes = rng.integers(case["lo"], case["hi"] + 1, (case["images"], 2))
        steps = [int(s) for s in np.where(rng.random(case["images"]) < 0.5, 1, 2)]
        return [_image(int(r), int(c), seed * 1000 + i) for i, (r, c) in enumerate(sizes)], steps
    if case["kind"] == "grad":
        return torch.stack([_image(case["rows"], case["cols"], seed * 1000 + i)
                            for i in range(case["images"])])
    return _image(case["rows"], case["cols"], seed)


def _stack(case, seed):
    """A sinogram stack (stack, angles, n) of the shape T-functionals give: the
    projections of blobs in a disc on a chord-length floor, with noise; each
    sinogram on its own scale."""
    n, a = case["n"], case["angles"]
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 31 + 7)
    th = torch.arange(a, device=DEV, dtype=torch.float32)[:, None] * (2 * math.pi / a)
    t = (torch.arange(n, device=DEV, dtype=torch.float32) - (n - 1) / 2)[None, :]
    out = torch.empty((case["stack"], a, n), device=DEV)
    chord = torch.sqrt((1 - (t / (0.49 * n)) ** 2).clamp(min=0))
    for s in range(case["stack"]):
        v = 0.03 * n * chord.expand(a, n).clone()
        for _ in range(8):
            r, ph = rng.uniform(0, 0.35 * n), rng.uniform(0, 2 * math.pi)
            sg, am = rng.uniform(n / 40, n / 8), rng.uniform(0.05, 0.3) * n
            v += float(am) * torch.exp(-((t - float(r) * torch.cos(th - float(ph))) ** 2) /
                                       (2 * float(sg) ** 2))
        v *= 1 + 0.02 * (torch.rand((a, n), generator=g, device=DEV) - 0.5)
        out[s] = v * (chord > 0) * float(10.0 ** rng.uniform(-1, 3))
    return out


def _angles(case):
    return (np.arange(case["angles"], dtype=np.float64) * (360.0 / case["angles"])).astype(np.float32)


def _ids(text):
    return [int(c) for c in text]


def _pad(rows, cols):
    """Side of the padded frame and the image's offset in it: the frame holds
    the circle through the image's far corner about its middle pixel."""
    oy, ox = (rows + 1) // 2 - 1, (cols + 1) // 2 - 1
    half = int(math.ceil(math.hypot(cols - 2 - ox, rows - 2 - oy))) + 1
    return 2 * half + 1, half - oy, half - ox


def _grad_weights(case, seed):
    """The gradient that arrives from the loss: normal, on the scale of each
    functional pair's values so that every pair takes part."""
    n = _pad(case["rows"], case["cols"])[0]
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 17 + 5)
    ts, ps = _ids(case["t"]), _ids(case["p"])
    w = torch.randn((case["images"], len(ts), len(ps), case["angles"]), generator=g, device=DEV)
    for i, t in enumerate(ts):
        mag = (0.2 * n, 0.018 * n ** 2, 0.0043 * n ** 3)[t]
        for j, p in enumerate(ps):
            w[:, i, j] /= 2.5 * mag if p == 1 else 0.05 * mag ** 4 / n
    return w


_engine = None


def _shared_engine():
    """One engine for the process, as a program keeps it."""
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


# ---- a pass -----------------------------------------------------------------------

def prepare(case, seed):
    k = case["kind"]
    s = dict(case)
    if k in ("transform", "ortho", "extended"):
        s["image"] = np.asfortranarray(_images(case, seed).cpu().numpy())
    elif k == "sinograms":
        s["engine"] = _shared_engine()
        s["image"] = _images(case, seed).t().contiguous()  # column-major
    elif k == "circus":
        s["engine"] = _shared_engine()
        s["sino"] = _stack(case, seed)
    elif k == "batch":
        imgs, steps = _images(case, seed)
        s["flat"] = torch.cat([im.t().reshape(-1) for im in imgs])
        s["rows"], s["cols"] = [im.shape[0] for im in imgs], [im.shape[1] for im in imgs]
        s["offsets"] = np.concatenate([[0], np.cumsum([im.numel() for im in imgs])[:-1]])
        s["steps"] = steps
        # a program that compares signatures between runs fixes the tile (the
        # one the tuner picks for these sizes): the tuner's choice may differ
        # from run to run, and with it the last bits of the sums
        s["engine"] = Engine(0)
        s["engine"].batch_tile((8, 8, 2))
    elif k == "grad":
        s["images"] = _images(case, seed)
        s["weights"] = _grad_weights(case, seed)
        s["angle_list"] = [float(a) for a in _angles(case)]
    return s


def run(s):
    k = s["kind"]
    if k in ("transform", "ortho"):
        tr = tt.Transformer(s["image"], "image", s["step"], k == "ortho")
        sig = tr.getTransform(list(s["t"]), [("H" if k == "ortho" else "") + p for p in s["p"]],
                              write_data=False)
        return {"circus": tr.circus, "signatures": sig}
    if k == "extended":
        return transform_extended(s["image"], _angles(s), _ids(s["t"]), list(s["p"]),
                                  _ids(s["h"]))
    if k == "sinograms":
        return s["engine"].sinograms(s["image"], s["rows"], s["cols"], _angles(s), _ids(s["t"]))
    if k == "circus":
        return s["engine"].circus(s["sino"], [(p, -1, -1) for p in _ids(s["p"])])
    if k == "batch":
        return s["engine"].transform_batch(s["flat"], s["offsets"], s["rows"], s["cols"],
                                           s["steps"], _ids(s["t"]),
                                           [(p, -1, -1) for p in _ids(s["p"])])
    images = s["images"].detach().requires_grad_(True)
    circ = autograd.circus(images, s["angle_list"], _ids(s["t"]), _ids(s["p"]))
    (grad,) = torch.autograd.grad(circ, images, s["weights"])
    return {"circus": circ.detach(), "grad": grad}


# ---- what a pass cannot do without --------------------------------------------------

def _sino_flops(rows, cols, angles, ts):
    """Per sample inside the image: 6 for the coordinates, 11 for the bilinear
    value, and the functionals' own sums (one for T0; the tail half of the
    samples for the others; a square root and a weighted count for T3-T7)."""
    per = 17.0
    for t in ts:
        per += {0: 1, 1: 2, 2: 2, 3: 3, 4: 3, 5: 3, 6: 4, 7: 4}[t]
    return per * rows * cols * angles


def _p_flops(n, cols, ps):
    per = {1: 2.0 * n, 2: 2.0 * n, 3: 2.5 * n * math.log2(max(n, 2)), 0: 2.0 * n}
    return cols * sum(per[p] for p in ps)


def _nos_flops(m, a):
    # QR, the polar factor of R, and Q applied to it
    return 2.0 * m * a * a + 10.0 * a ** 3 + 2.0 * m * a * a


def work(case):
    k = case["kind"]
    if k in ("transform", "extended", "ortho"):
        ts = _ids(case["t"])
        a = case["angles"] if k == "extended" else 360 // case["step"]
        r, c = case["rows"], case["cols"]
        if k == "ortho":
            r = c = int(math.ceil(a / math.sqrt(2)))
        n = _pad(r, c)[0]
        out = 2 * 4 * len(ts) * a * (len(case["p"]) + len(case.get("h", "")))
        fl = _sino_flops(r, c, a, ts)
        if k != "ortho":
            fl += _p_flops(n, len(ts) * a, _ids(case["p"]))
        if k != "transform":
            fl += len(ts) * (_nos_flops(n, a) + 2.0 * n * a * len(case.get("h", case["p"])))
        return {"bytes": 4 * case["rows"] * case["cols"] + out, "flops": fl}
    if k == "sinograms":
        n = _pad(case["rows"], case["cols"])[0]
        ts = _ids(case["t"])
        return {"bytes": 4 * case["rows"] * case["cols"] + 4 * len(ts) * n * case["angles"],
                "flops": _sino_flops(case["rows"], case["cols"], case["angles"], ts)}
    if k == "circus":
        cols = case["stack"] * case["angles"]
        return {"bytes": 4 * cols * (case["n"] + len(case["p"])),
                "flops": _p_flops(case["n"], cols, _ids(case["p"]))}
    if k == "batch":
        rng = np.random.default_rng(case["images"] * 1000003 + case["lo"] * 1009 + case["hi"])
        sizes = rng.integers(case["lo"], case["hi"] + 1, (case["images"], 2))
        steps = np.where(rng.random(case["images"]) < 0.5, 1, 2)
        ts, ps = _ids(case["t"]), _ids(case["p"])
        by = fl = 0.0
        for (r, c), st in zip(sizes.tolist(), steps.tolist()):
            a = 360 // st
            by += 4 * r * c + 2 * 4 * len(ts) * len(ps) * a
            fl += _sino_flops(r, c, a, ts) + _p_flops(_pad(r, c)[0], len(ts) * a, ps)
        return {"bytes": by, "flops": fl}
    b, r, c, a = case["images"], case["rows"], case["cols"], case["angles"]
    ts, ps = _ids(case["t"]), _ids(case["p"])
    n = _pad(r, c)[0]
    # backward: per sample the line's gradient (4) and its four bilinear shares
    # (6 + 8 + 4), the P-stage twice
    fl = _sino_flops(r, c, a, ts) + 3 * _p_flops(n, len(ts) * a, ps) + 22.0 * r * c * a
    return {"bytes": b * (2 * 4 * r * c + 2 * 4 * len(ts) * len(ps) * a), "flops": b * fl}


# ---- the same in 64 bits --------------------------------------------------------------

def _rotated(img, angles):
    """Rotated samples (A, column, row) of a (rows, cols) float64 image in its frame."""
    rows, cols = img.shape
    n, ro, co = _pad(rows, cols)
    frame = img.new_zeros((n, n))
    frame = torch.cat([img.new_zeros((ro, cols)), img, img.new_zeros((n - ro - rows, cols))], 0)
    frame = torch.cat([img.new_zeros((n, co)), frame, img.new_zeros((n, n - co - cols))], 1)
    th = -angles * (math.pi / 180)
    c, s = torch.cos(th)[:, None, None], torch.sin(th)[:, None, None]
    o = (n - 1) / 2
    g = torch.arange(n, device=img.device, dtype=torch.float64) - o
    X, Y = g[None, :, None], g[None, None, :]
    qx, qy = X * c + Y * s + o, -X * s + Y * c + o
    ok = (qx >= 0) & (qx < n - 1) & (qy >= 0) & (qy < n - 1)
    xi = torch.where(ok, qx, qx.new_zeros(())).floor()
    yi = torch.where(ok, qy, qy.new_zeros(())).floor()
    xf, yf = qx - xi, qy - yi
    at = (yi * n + xi).long()
    f = frame.reshape(-1)
    v = (f[at] * ((1 - xf) * (1 - yf)) + f[at + 1] * (xf * (1 - yf)) +
         f[at + n] * ((1 - xf) * yf) + f[at + n + 1] * (xf * yf))
    return torch.where(ok, v, v.new_zeros(()))


def _median(x):
    cs = x.detach().cumsum(-1)
    hit = 2 * cs >= cs[..., -1:]
    return torch.where(hit.any(-1), hit.to(torch.uint8).argmax(-1),
                       torch.full_like(hit.any(-1), x.shape[-1] - 1, dtype=torch.long))


def _select(keys, weights, valid):
    """The key at the weighted median of the valid entries in key order."""
    k, order = torch.where(valid, keys, torch.inf).sort(-1)
    w = torch.where(valid, weights, 0.0).gather(-1, order)
    cs = w.cumsum(-1)
    cnt = valid.sum(-1, keepdim=True)
    hit = (2 * cs >= cs[..., -1:]) & (torch.arange(k.shape[-1], device=k.device) < cnt)
    i = torch.where(hit.any(-1), hit.to(torch.uint8).argmax(-1), (cnt[..., 0] - 1).clamp(min=0))
    return k.gather(-1, i[..., None])[..., 0]


def _t_functionals(x, ts):
    """(A, nT, column) of the rotated samples x (A, column, row)."""
    n = x.shape[-1]
    j = torch.arange(n, device=x.device)
    out = []
    m1 = _median(x) if set(ts) & {1, 2, 7} else None
    root = x.detach().clamp(min=0).sqrt() if set(ts) & {3, 4, 5, 6, 7} else None
    m2 = _median(root) if set(ts) & {3, 4, 5, 6} else None
    r1 = (j - m1[..., None]) if m1 is not None else None
    r2 = (j - m2[..., None]) if m2 is not None else None
    for t in ts:
        if t == 0:
            out.append(x.sum(-1))
        elif t in (1, 2):
            out.append((x * r1.clamp(min=0).double() ** t).sum(-1))
        elif t in (3, 4, 5):
            r = r2.clamp(min=0).double()
            lr = r.clamp(min=1).log()
            amp, f = {3: (r, 5), 4: ((r > 0).double(), 3), 5: (r.sqrt(), 4)}[t]
            out.append(torch.hypot((x * amp * torch.cos(f * lr)).sum(-1),
                                   (x * amp * torch.sin(f * lr)).sum(-1)))
        elif t == 6:
            out.append(_select(r2.double() * x, root, r2 >= 0))
        else:
            out.append(_select(x, root, r1 >= 0))
    return torch.stack(out, 1)


def _p_functionals(sino, ps):
    """(..., nP) of sinogram columns (..., n)."""
    n = sino.shape[-1]
    out = []
    for p in ps:
        if p == 1:
            out.append((sino[..., 1:] - sino[..., :-1]).abs().sum(-1))
        elif p == 2:
            out.append(_select(sino, sino, torch.ones_like(sino, dtype=torch.bool)))
        else:
            y = (torch.fft.fft(sino).abs() / n) ** 4
            k = torch.arange(n, device=sino.device)
            y = y[..., torch.where(k <= n // 2, k, n - k)]
            out.append((y[..., 1:] + y[..., :-1]).sum(-1) * (1.0 / (n - 1)))
    return torch.stack(out, -1)


def _zscore(v):
    return (v - v.mean(-1, keepdim=True)) / v.std(-1, keepdim=True)


def _sinograms64(img, angles, ts):
    """(nT, A, N) in float64, a few angles at a time."""
    n = _pad(*img.shape)[0]
    step = max(1, int(3e7 // (n * n)))
    a = torch.from_numpy(np.asarray(angles, np.float64)).to(img.device)
    return torch.cat([_t_functionals(_rotated(img, a[i:i + step]), ts)
                      for i in range(0, len(a), step)]).transpose(0, 1)


def _nearest_orthonormal(sino):
    """(aligned rows x A matrix, center) of an (A, N) sinogram."""
    a, n = sino.shape
    center = int(math.floor((n - 1) / 2))
    off = (_median(sino) - center).cpu().numpy()
    m = n + abs(int(off.max())) + abs(int(off.min()))
    al = sino.new_zeros((m, a))
    for i in range(a):
        shift = int(off.max()) - int(off[i])
        al[shift:shift + n, i] = sino[i]
    u, _, vt = torch.linalg.svd(al, full_matrices=False)
    return u @ vt, center + int(off.max())


def _hermite(nos, center, orders):
    """(nH, A) projections on the weighted Hermite basis stretched to +-10."""
    m = nos.shape[0]
    p = torch.arange(m, device=nos.device, dtype=torch.float64)
    z = torch.where(p < center, p * (10.0 / center) - 10, (p - center) * (10.0 / (m - 1 - center)))
    out = []
    for order in orders:
        h0, h1 = torch.ones_like(z), 2 * z
        for k in range(1, order):
            h0, h1 = h1, 2 * z * h1 - 2 * k * h0
        h = h1 if order else h0
        out.append((h * torch.exp(-z * z / 2) /
                    math.sqrt(2.0 ** order * math.factorial(order) * math.sqrt(math.pi))) @ nos)
    return torch.stack(out)


def _resized(img, side):
    """The image stretched to side x side: bilinear at pixel centres, the
    outermost rows and columns left zero."""
    rows, cols = img.shape
    k = torch.arange(side, device=img.device, dtype=torch.float64)
    # x is scaled by the row ratio and y by the column ratio, as the path does
    qx, qy = (k + 0.5) * (rows / side) - 0.5, (k + 0.5) * (cols / side) - 0.5
    okx = (k >= 1) & (k < side - 1) & (qx >= 0) & (qx < cols - 1)
    oky = (k >= 1) & (k < side - 1) & (qy >= 0) & (qy < rows - 1)
    xi, yi = torch.where(okx, qx, 0.0).floor().long(), torch.where(oky, qy, 0.0).floor().long()
    xf, yf = (qx - xi)[None, :], (qy - yi)[:, None]
    v = (img[yi][:, xi] * (1 - xf) * (1 - yf) + img[yi][:, xi + 1] * xf * (1 - yf) +
         img[yi + 1][:, xi] * (1 - xf) * yf + img[yi + 1][:, xi + 1] * xf * yf)
    return torch.where(oky[:, None] & okx[None, :], v, 0.0)


def _circus64(img, angles, ts, ps):
    return _p_functionals(_sinograms64(img, angles, ts), ps).transpose(1, 2)  # (nT, nP, A)


def exact(case, seed):
    k = case["kind"]
    ts = _ids(case["t"]) if "t" in case else []
    ps = _ids(case["p"]) if "p" in case else []
    if k == "circus":
        if case["n"] * case["angles"] * case["stack"] > 6e7:
            return None
        return _p_functionals(_stack(case, seed).double(), ps).transpose(1, 2)
    if k == "batch":
        imgs, steps = _images(case, seed)
        c = [_circus64(im.double(), np.arange(360 // st) * float(st), ts, ps)
             for im, st in zip(imgs, steps)]
        return (torch.cat([v.reshape(-1) for v in c]),
                torch.cat([_zscore(v).reshape(-1) for v in c]))
    if k == "sinograms":
        if float(case["rows"]) * case["cols"] * case["angles"] > 1.5e9:
            return None
        return _sinograms64(_images(case, seed).double(), _angles(case), ts)
    if k == "grad":
        images, w = _images(case, seed).double(), _grad_weights(case, seed).double()
        ang = torch.from_numpy(_angles(case).astype(np.float64)).to(images.device)
        n = _pad(case["rows"], case["cols"])[0]
        step = max(1, int(6e7 // (n * n)))
        circ, grad = torch.zeros_like(w), torch.zeros_like(images)
        for b in range(case["images"]):
            for i in range(0, len(ang), step):
                img = images[b].clone().requires_grad_(True)
                v = _p_functionals(_t_functionals(_rotated(img, ang[i:i + step]), ts), ps)
                v = v.permute(1, 2, 0)
                (g,) = torch.autograd.grad(v, img, w[b, :, :, i:i + step])
                circ[b, :, :, i:i + step] = v.detach()
                grad[b] += g
        return {"circus": circ, "grad": grad}
    img = _images(case, seed).double()
    if k == "transform":
        c = _circus64(img, np.arange(360 // case["step"]) * float(case["step"]), ts, ps)
        return {"circus": c, "signatures": _zscore(c).reshape(-1, c.shape[-1]).t()}
    if k == "ortho":
        a = 360 // case["step"]
        img = _resized(img, int(math.ceil(math.ceil(360.0 / case["step"]) / math.sqrt(2))))
        sino = _sinograms64(img, np.arange(a) * float(case["step"]), ts)
        h = torch.stack([_hermite(*_nearest_orthonormal(s), ps) for s in sino])
        return {"circus": h, "signatures": _zscore(h).reshape(-1, a).t()}
    sino = _sinograms64(img, _angles(case), ts)
    c = _p_functionals(sino, ps).transpose(1, 2)
    h = torch.stack([_hermite(*_nearest_orthonormal(s), _ids(case["h"])) for s in sino])
    return {"circus": c, "signatures": _zscore(c), "hermite_circus": h,
            "hermite_signatures": _zscore(h), "centers": None}
