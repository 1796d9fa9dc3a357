"""Workloads of the separable filtering path, as programs call them.

Each case is one call (or the few calls that belong together) through the
public entry points of `cucim_b200.ndimage`, `cucim_b200.skimage` and
`cucim_b200.batch` on arrays that are already on the device. The listed cases
are the shapes of this repository's own benchmark and tests, from the
smallest images to the largest volumes; `draw` gives others of the same
ranges, odd sizes among them.
"""

import math

import numpy as np
import torch

from cucim_b200 import ndimage as ndi
from cucim_b200.batch import TileBatch
from cucim_b200.skimage import filters

DEVICE = "cuda"


# ------------------------------------------------------------------- cases

def listed():
    return [
        # a thumbnail or one small field of view, smoothed: the call's own
        # latency (one launch, its host work) is what a user waits for
        {"name": "gaussian_small", "kind": "gaussian2d", "h": 256, "w": 256, "sigma": 1.0,
         "mode": "nearest", "dtype": "float32"},
        # edges of an 8-bit camera image with odd sides: skimage's default
        # call (conversion to float, two derivative chains, the magnitude)
        {"name": "sobel_u8_image", "kind": "sobel2d", "h": 1023, "w": 1537, "mode": "reflect"},
        # the plain 2-D gaussian of the benchmark
        {"name": "gaussian_2d", "kind": "gaussian2d", "h": 2048, "w": 2048, "sigma": 4.0,
         "mode": "reflect", "dtype": "float32"},
        # double precision measurement data, ragged sides, the library's
        # default dtype rule (float64 in, float64 arithmetic, float64 out)
        {"name": "gaussian_f64", "kind": "gaussian2d", "h": 2003, "w": 3001, "sigma": 2.0,
         "mode": "mirror", "dtype": "float64"},
        # a large float32 image, a wide gaussian at full float32 exactness
        {"name": "gaussian_wide", "kind": "wide", "h": 8192, "w": 8192, "sigma": 16.0,
         "mode": "nearest", "algorithm": ""},
        # the same filter where the caller opts for the split-precision
        # tensor-core passes
        {"name": "gaussian_wide_tensor", "kind": "wide", "h": 8192, "w": 8192, "sigma": 16.0,
         "mode": "nearest", "algorithm": "tensor"},
        # a 16-bit microscopy stack, anisotropic smoothing to float32
        {"name": "stack_gaussian", "kind": "stack_gaussian", "d": 512, "h": 1024, "w": 1024,
         "sz": 1.0, "sy": 2.0, "sx": 2.0, "mode": "mirror"},
        # its derivatives along the three axes
        {"name": "stack_sobel", "kind": "stack_sobel", "d": 256, "h": 1024, "w": 1024,
         "mode": "reflect"},
        # box smoothing that stays 16-bit, on a stack cropped to odd sides
        {"name": "stack_uniform", "kind": "stack_uniform", "d": 203, "h": 1021, "w": 1015,
         "size": 5, "mode": "reflect"},
        # blob detection on a float32 volume: the sum of Gaussian second
        # derivatives along every axis
        {"name": "volume_log", "kind": "log", "d": 160, "h": 512, "w": 512, "sigma": 2.0,
         "mode": "reflect"},
        # vesselness of a float32 volume over five scales
        {"name": "frangi_volume", "kind": "frangi", "d": 256, "h": 256, "w": 256, "scales": 5,
         "mode": "reflect"},
        # whole-slide tiles of uneven sizes, gray -> gaussian -> edges in one
        # launch; the tables are prepared once, as a tile loader keeps them
        {"name": "slide_tiles", "kind": "tiles", "layout": 3, "tiles": 1024, "lo": 64,
         "hi": 1024, "smin": 0.5, "smax": 8.0},
    ]


_MODES = ("reflect", "mirror", "nearest", "constant", "wrap")


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _volume(rng, lo, hi, most):
    """Three sides in [lo, hi] with at most `most` voxels, the last ones at
    least as long as the first."""
    while True:
        d, h, w = _log(rng, max(8, lo // 4), hi), _log(rng, lo, hi), _log(rng, lo, hi)
        if rng.random() < 0.5:  # half of all crops come in multiples of four
            h, w = h // 4 * 4, w // 4 * 4
        if d * h * w <= most:
            return d, h, w


def draw(rng):
    kind = rng.choice(["gaussian2d", "gaussian2d", "sobel2d", "wide", "stack_gaussian",
                       "stack_sobel", "stack_uniform", "log", "frangi", "tiles"])
    mode = rng.choice(_MODES)
    if kind == "gaussian2d":
        return {"kind": kind, "h": _log(rng, 64, 4096), "w": _log(rng, 64, 4096),
                "sigma": round(rng.uniform(0.6, 6.0), 2), "mode": mode,
                "dtype": rng.choice(["float32", "float32", "float64"])}
    if kind == "sobel2d":
        return {"kind": kind, "h": _log(rng, 128, 4096), "w": _log(rng, 128, 4096),
                "mode": mode}
    if kind == "wide":
        return {"kind": kind, "h": _log(rng, 2048, 8192), "w": _log(rng, 2048, 8192),
                "sigma": round(rng.uniform(8.0, 16.0), 2), "mode": mode,
                "algorithm": rng.choice(["", "tensor"])}
    if kind == "stack_gaussian":
        d, h, w = _volume(rng, 128, 1024, 1 << 28)
        return {"kind": kind, "d": d, "h": h, "w": w, "sz": round(rng.uniform(0.5, 2.0), 2),
                "sy": round(rng.uniform(0.8, 4.0), 2), "sx": round(rng.uniform(0.8, 4.0), 2),
                "mode": mode}
    if kind == "stack_sobel":
        d, h, w = _volume(rng, 128, 1024, 1 << 27)
        return {"kind": kind, "d": d, "h": h, "w": w, "mode": mode}
    if kind == "stack_uniform":
        d, h, w = _volume(rng, 128, 1024, 1 << 27)
        return {"kind": kind, "d": d, "h": h, "w": w, "size": rng.choice([3, 5, 5, 7, 9]),
                "mode": mode}
    if kind == "log":
        d, h, w = _volume(rng, 96, 512, 1 << 25)
        return {"kind": kind, "d": d, "h": h, "w": w, "sigma": round(rng.uniform(1.0, 3.0), 2),
                "mode": mode}
    if kind == "frangi":
        d, h, w = _volume(rng, 64, 256, 1 << 23)
        return {"kind": kind, "d": d, "h": h, "w": w, "scales": rng.choice([2, 3, 4, 5]),
                # the modes vesselness is run with; a mirrored face makes one
                # eigenvalue exactly zero, where the formula is a coin toss
                "mode": rng.choice(["reflect", "nearest"])}
    return {"kind": kind, "layout": rng.randrange(1 << 20), "tiles": _log(rng, 32, 1024), "lo": 64,
            "hi": rng.choice([256, 512, 1024]), "smin": 0.5,
            "smax": round(rng.uniform(2.0, 8.0), 2)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _stack_u16(d, h, w, seed):
    """Smooth structure over [0, 65535] with shot noise, slab by slab."""
    g = _gen(seed)
    coarse = torch.randn((1, 1, d // 6 + 2, h // 6 + 2, w // 6 + 2), device=DEVICE, generator=g)
    out = torch.empty((d, h, w), dtype=torch.uint16, device=DEVICE)
    planes = torch.nn.functional.interpolate(coarse[0], size=(h, w), mode="bilinear",
                                             align_corners=True)[0]
    pos = torch.linspace(0, planes.shape[0] - 1, d, dtype=torch.float64)
    for z in range(d):
        i = min(int(pos[z]), planes.shape[0] - 2)
        t = float(pos[z]) - i
        s = (planes[i] * (1 - t) + planes[i + 1] * t).mul_(9000).add_(32768).clamp_(0, 65535)
        s += torch.randn((h, w), device=DEVICE, generator=g) * s.sqrt()
        out[z] = s.round_().clamp_(0, 65535).to(torch.int32).to(torch.uint16)
    return out


def _rectangles(h, w, seed):
    """i.i.d. uniform [0, 1) plus 64 constant rectangles of 0-10."""
    x = torch.rand((h, w), device=DEVICE, generator=_gen(seed))
    r = np.random.default_rng(seed)
    for _ in range(64):
        y0, y1 = sorted(r.integers(0, h, 2).tolist())
        x0, x1 = sorted(r.integers(0, w, 2).tolist())
        x[y0:y1 + 1, x0:x1 + 1] += float(r.uniform(0, 10))
    return x


def _segments(d, h, w, seed):
    """Bright tubes of radius 1-4 on background noise N(0, 0.05)."""
    g = _gen(seed)
    x = torch.randn((d, h, w), device=DEVICE, generator=g) * 0.05
    r = np.random.default_rng(seed)
    shape = np.array([d, h, w])
    for _ in range(60):
        p = r.uniform(0, 1, 3) * shape
        v = r.normal(size=3)
        v /= np.linalg.norm(v)
        length, rad = r.uniform(20, 120), r.uniform(1, 4)
        q = p + v * length
        lo = np.maximum(np.floor(np.minimum(p, q) - 3 * rad), 0).astype(int)
        hi = np.minimum(np.ceil(np.maximum(p, q) + 3 * rad) + 1, shape).astype(int)
        if np.any(hi <= lo):
            continue
        ax = [torch.arange(int(a), int(b), device=DEVICE, dtype=torch.float32)
              for a, b in zip(lo, hi)]
        rel = [ax[k].reshape([-1 if j == k else 1 for j in range(3)]) - float(p[k])
               for k in range(3)]
        t = sum(rel[k] * float(v[k]) for k in range(3)).clamp(0, float(length))
        dist = sum((rel[k] - t * float(v[k])) ** 2 for k in range(3))
        sl = tuple(slice(int(a), int(b)) for a, b in zip(lo, hi))
        x[sl] = torch.maximum(x[sl], torch.exp(dist / (-2 * rad * rad)))
    return x


def _image(case, seed):
    dt = getattr(torch, case["dtype"])
    return torch.rand((case["h"], case["w"]), device=DEVICE, generator=_gen(seed), dtype=dt)


def _photo_u8(h, w, seed):
    """Smooth shading with pixel noise, 8 bits."""
    g = _gen(seed)
    coarse = torch.rand((1, 1, h // 32 + 2, w // 32 + 2), device=DEVICE, generator=g)
    s = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear",
                                        align_corners=True)[0, 0]
    s = s * 220 + 6 * torch.randn((h, w), device=DEVICE, generator=g) + 16
    return s.clamp_(0, 255).to(torch.uint8)


def _tile_specs(case):
    """The sides and sigmas of a case's tiles (fixed by its layout number)."""
    r = np.random.default_rng(case["layout"])
    n = case["tiles"]
    hs = r.integers(case["lo"], case["hi"] + 1, n)
    ws = r.integers(case["lo"], case["hi"] + 1, n)
    sigmas = r.uniform(case["smin"], case["smax"], n)
    return hs.tolist(), ws.tolist(), sigmas.tolist()


def _tile_pixels(case, seed):
    """RGB tiles from a 3-component Gaussian mixture per channel."""
    hs, ws, sigmas = _tile_specs(case)
    sizes = [h * w * 3 for h, w in zip(hs, ws)]
    g = _gen(seed)
    # one draw for all tiles, cut up: 60, 150 or 220, each with sd 20
    total = sum(sizes)
    flat = torch.empty(total, dtype=torch.uint8, device=DEVICE)
    means = torch.tensor([60.0, 150.0, 220.0], device=DEVICE)
    step = 1 << 26
    for a in range(0, total, step):
        n = min(step, total - a)
        m = means[torch.randint(0, 3, (n,), device=DEVICE, generator=g)]
        m += 20 * torch.randn(n, device=DEVICE, generator=g)
        flat[a:a + n] = m.clamp_(0, 255).to(torch.uint8)
    tiles, at = [], 0
    for h, w, n in zip(hs, ws, sizes):
        # a tile of its own, as a decoder leaves it
        tiles.append(flat[at:at + n].clone().reshape(h, w, 3))
        at += n
    return tiles, sigmas


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gaussian2d":
        return case, _image(case, seed)
    if kind == "sobel2d":
        return case, _photo_u8(case["h"], case["w"], seed)
    if kind == "wide":
        return case, _rectangles(case["h"], case["w"], seed)
    if kind in ("stack_gaussian", "stack_sobel", "stack_uniform"):
        return case, _stack_u16(case["d"], case["h"], case["w"], seed)
    if kind in ("log", "frangi"):
        return case, _segments(case["d"], case["h"], case["w"], seed)
    # the results land side by side in one buffer, as the next stage takes them
    tiles, sigmas = _tile_pixels(case, seed)
    flat = torch.empty(sum(t.shape[0] * t.shape[1] for t in tiles), device=DEVICE)
    outs, at = [], 0
    for t in tiles:
        n = t.shape[0] * t.shape[1]
        outs.append(flat[at:at + n].view(t.shape[0], t.shape[1]))
        at += n
    return case, (TileBatch(tiles, sigmas, outputs=outs), flat)


# -------------------------------------------------------------------- runs

def run(state):
    case, x = state
    kind, mode = case["kind"], case.get("mode")
    if kind == "gaussian2d":
        return filters.gaussian(x, sigma=case["sigma"], mode=mode)
    if kind == "sobel2d":
        return filters.sobel(x, mode=mode)
    if kind == "wide":
        return ndi.gaussian_filter(x, case["sigma"], mode=mode,
                                   algorithm=case["algorithm"] or None)
    if kind == "stack_gaussian":
        return ndi.gaussian_filter(x, (case["sz"], case["sy"], case["sx"]), mode=mode,
                                   output=np.float32)
    if kind == "stack_sobel":
        return [ndi.sobel(x, axis=a, mode=mode, output=np.float32) for a in range(3)]
    if kind == "stack_uniform":
        # the same bits as int16, which more of torch's operators take
        return ndi.uniform_filter(x, case["size"], mode=mode).view(torch.int16)
    if kind == "log":
        return ndi.gaussian_laplace(x, case["sigma"], mode=mode)
    if kind == "frangi":
        return filters.frangi(x, sigmas=range(1, case["scales"] + 1), black_ridges=False,
                              mode=mode)
    batch, flat = x
    batch.run()
    return flat


# ---------------------------------------------------------- what it must do

def _taps(sigma, truncate=4.0):
    return 2 * int(truncate * sigma + 0.5) + 1


def work(case):
    """One pass' unavoidable bytes (inputs once, outputs once) and the
    multiply-adds of its taps, two operations each."""
    kind = case["kind"]
    if kind == "tiles":
        px = taps = 0
        for h, w, s in zip(*_tile_specs(case)):
            px += h * w
            taps += h * w * (2 * _taps(s) + 12)
        return {"bytes": 7 * px, "flops": 2 * taps + 5 * px}
    n = case.get("d", 1) * case["h"] * case["w"]
    if kind == "gaussian2d":
        es = 4 if case["dtype"] == "float32" else 8
        return {"bytes": 2 * es * n, "flops": 4 * n * _taps(case["sigma"])}
    if kind == "sobel2d":  # two chains of 2 + 3 taps, two squares, a sum, a root
        return {"bytes": 5 * n, "flops": 2 * n * 10 + 4 * n}
    if kind == "wide":
        return {"bytes": 8 * n, "flops": 4 * n * _taps(case["sigma"])}
    if kind == "stack_gaussian":
        return {"bytes": 6 * n,
                "flops": 2 * n * (_taps(case["sz"]) + _taps(case["sy"]) + _taps(case["sx"]))}
    if kind == "stack_sobel":
        return {"bytes": 18 * n, "flops": 3 * 2 * n * 8}
    if kind == "stack_uniform":
        return {"bytes": 4 * n, "flops": 6 * n * case["size"]}
    if kind == "log":
        return {"bytes": 8 * n, "flops": 9 * 2 * n * _taps(case["sigma"])}
    # frangi: 6 + 9 + 9 distinct Gaussian-derivative passes per scale (taps
    # that are zero in float32 left out) and about 150 operations for the
    # eigenvalues and the vesselness
    total = 0
    for s in range(1, case["scales"] + 1):
        total += 24 * 2 * len(_float32_taps(s / math.sqrt(2), 1, 8 if s > 1 else 100)) + 150
    return {"bytes": 8 * n, "flops": total * n}


# --------------------------------------------------------------- tolerance

def tolerance(case):
    """About four times the largest distance of the results from the same
    filter in 64 bits, measured over the listed cases and forty drawn ones
    (the largest seen stands beside each)."""
    kind = case["kind"]
    if kind == "stack_uniform":
        return "exact"
    if kind == "gaussian2d" and case["dtype"] == "float64":
        return {"rel": 1e-15}  # the sums of 17 taps in another order: 2e-16
    if kind == "wide":
        return {"rel": 3e-6} if case["algorithm"] else {"rel": 8e-7}  # 7.0e-7, 1.9e-7
    if kind == "frangi":
        return {"rel": 4e-4}  # 1.0e-4: ratios of differences of eigenvalues
    if kind == "tiles":
        return {"rel": 7e-6}  # 1.8e-6: differences of a smoothed image
    if kind == "gaussian2d" or kind == "stack_gaussian":
        return {"rel": 5e-7}  # 1.1e-7
    return {"rel": 1.4e-6}  # sobel 3.3e-7, second derivatives 3.3e-7


# ------------------------------------------------------------------- exact

def _gauss64(sigma, order, truncate):
    r = int(truncate * sigma + 0.5)
    x = np.arange(-r, r + 1)
    p = np.exp(-0.5 / (sigma * sigma) * x ** 2)
    p /= p.sum()
    if order == 1:
        p = p * (x / (sigma * sigma))
    elif order == 2:
        p = p * ((x / (sigma * sigma)) ** 2 - 1 / (sigma * sigma))
    return p


def _float32_taps(sigma, order, truncate):
    w = _gauss64(sigma, order, truncate).astype(np.float32)
    return np.trim_zeros(w) if sigma > 0 else w


def _index(n, r, mode):
    """Source indices of positions -r .. n - 1 + r along an axis of length n;
    -1 where a constant is read."""
    i = np.arange(-r, n + r)
    if mode == "nearest":
        return np.clip(i, 0, n - 1)
    if mode == "wrap":
        return i % n
    if mode == "constant":
        return np.where((i < 0) | (i >= n), -1, i)
    if mode == "reflect":
        i = i % (2 * n)
        return np.minimum(i, 2 * n - 1 - i)
    if n == 1:
        return np.zeros_like(i)
    i = i % (2 * n - 2)
    return np.minimum(i, 2 * n - 2 - i)


def _pass64(x, w, axis, mode):
    """Correlation with the odd-length taps along one axis in float64, in
    pieces along another axis so that the padded copies stay small."""
    n, r = x.shape[axis], len(w) // 2
    nz = np.nonzero(w)[0]
    r_eff = int(max(abs(nz[0] - r), abs(nz[-1] - r))) if len(nz) else 0
    idx = _index(n, r_eff, mode)
    src = torch.as_tensor(np.maximum(idx, 0), device=x.device)
    gaps = np.nonzero(idx < 0)[0]
    other = 0 if axis != 0 else 1
    step = max(1, (1 << 25) * x.shape[other] // max(1, x.numel()))
    out = torch.empty_like(x, dtype=torch.float64)
    for a in range(0, x.shape[other], step):
        m = min(step, x.shape[other] - a)
        pad = x.narrow(other, a, m).to(torch.float64).index_select(axis, src)
        if len(gaps):
            pad.index_fill_(axis, torch.as_tensor(gaps, device=x.device), 0.0)
        acc = torch.zeros_like(pad.narrow(axis, 0, n))
        for k in range(len(w)):
            if w[k] != 0.0:
                acc.add_(pad.narrow(axis, k - r + r_eff, n), alpha=float(w[k]))
        out.narrow(other, a, m).copy_(acc)
    return out


def _gauss_nd(x, sigmas, orders, mode, truncate=4.0):
    y = x
    for axis, (s, o) in enumerate(zip(sigmas, orders)):
        y = _pass64(y, _gauss64(s, o, truncate), axis, mode)
    return y


def _vesselness64(x, scales, mode):
    """The 3-D frangi filter in float64: Gaussian-derivative Hessians, their
    eigenvalues in closed form, ordered by magnitude."""
    x = -x.to(torch.float64)
    best = gamma2 = None
    for sigma in range(1, scales + 1):
        s = sigma / math.sqrt(2)
        trunc = 8 if sigma > 1 else 100
        unit = [[1 if k == a else 0 for k in range(3)] for a in range(3)]
        grads = [_gauss_nd(x, [s] * 3, unit[a], mode, trunc) for a in range(3)]
        h = {}
        for a in range(3):
            for b in range(a, 3):
                h[a, b] = _gauss_nd(grads[a], [s] * 3, unit[b], mode, trunc)
        del grads
        mean = (h[0, 0] + h[1, 1] + h[2, 2]) / 3
        p2 = sum((h[i, i] - mean) ** 2 for i in range(3)) + 2 * (
            h[0, 1] ** 2 + h[0, 2] ** 2 + h[1, 2] ** 2)
        p = torch.sqrt(p2 / 6).clamp_min_(1e-300)
        b = {k: ((v - mean) if k[0] == k[1] else v) / p for k, v in h.items()}
        det = (b[0, 0] * (b[1, 1] * b[2, 2] - b[1, 2] ** 2)
               - b[0, 1] * (b[0, 1] * b[2, 2] - b[1, 2] * b[0, 2])
               + b[0, 2] * (b[0, 1] * b[1, 2] - b[1, 1] * b[0, 2]))
        phi = torch.acos((det / 2).clamp_(-1, 1)) / 3
        e1 = mean + 2 * p * torch.cos(phi)
        e3 = mean + 2 * p * torch.cos(phi + 2 * math.pi / 3)
        ev = torch.stack([e1, 3 * mean - e1 - e3, e3])
        del b, det, phi, p, p2
        order = ev.abs().argsort(dim=0)
        l1, l2, l3 = ev.gather(0, order)
        rg = l1 * l1 + l2 * l2 + l3 * l3
        if gamma2 is None:
            top = float(rg.max())
            gamma2 = 2.0 if top == 0 else max(2 * (math.sqrt(top) / 2) ** 2, 1e-10)
        l2, l3 = l2.clamp_min(1e-10), l3.clamp_min(1e-10)
        v = 1 - torch.exp(-((l2 / l3) ** 2) / 0.5)
        v *= torch.exp(-(l1 * l1 / (l2 * l3)) / 0.5)
        v *= 1 - torch.exp(-rg / gamma2)
        best = v if best is None else torch.maximum(best, v)
    return best


def _sobel_mag64(x, mode):
    edge, smooth = np.array([-1.0, 0.0, 1.0]) / math.sqrt(2), np.array([0.25, 0.5, 0.25])
    d0 = _pass64(_pass64(x, edge, 0, mode), smooth, 1, mode)
    d1 = _pass64(_pass64(x, edge, 1, mode), smooth, 0, mode)
    return torch.sqrt(d0 * d0 + d1 * d1)


def exact(case, seed):
    kind, mode = case["kind"], case.get("mode")
    if kind == "stack_uniform":
        return None  # whole numbers, cut off after every pass
    if kind == "tiles":
        tiles, sigmas = _tile_pixels(case, seed)
        luma = torch.tensor([0.2125, 0.7154, 0.0721], device=DEVICE, dtype=torch.float64)
        outs = []
        for t, s in zip(tiles, sigmas):
            gray = (t.to(torch.float64) / 255 * luma).sum(-1)
            outs.append(_sobel_mag64(_gauss_nd(gray, (s, s), (0, 0), "nearest"),
                                     "reflect").flatten())
        return torch.cat(outs)
    x = prepare(case, seed)[1]
    if kind == "gaussian2d":
        return _gauss_nd(x, [case["sigma"]] * 2, (0, 0), mode)
    if kind == "sobel2d":
        return _sobel_mag64(x.to(torch.float64) / 255, mode)
    if kind == "wide":
        return _gauss_nd(x, [case["sigma"]] * 2, (0, 0), mode)
    if kind == "stack_gaussian":
        return _gauss_nd(x.to(torch.float32), (case["sz"], case["sy"], case["sx"]), (0, 0, 0),
                         mode)
    if kind == "stack_sobel":
        x = x.to(torch.float32)
        outs = []
        for a in range(3):
            y = x
            for b in range(3):
                y = _pass64(y, np.array([-1.0, 0, 1] if a == b else [1.0, 2, 1]), b, mode)
            outs.append(y)
        return outs
    if kind == "log":
        return sum(_gauss_nd(x, [case["sigma"]] * 3, [2 if a == b else 0 for b in range(3)], mode)
                   for a in range(3))
    return _vesselness64(x, case["scales"], mode)
