"""Performance cases of the focal-raster operations: what a program that uses this package has it do.

``listed()`` are twelve calls over the range of real use, ``draw(rng)`` gives more of the same
ranges.  Every case goes through the public functions (``raster_*`` on an ``OwnedRasterArray``,
``TerrainBatch`` for many tiles).  Rasters live on the GPU before the call, as they do between two
steps of a processing chain, and every call allocates its own results, as those functions do.

Results are float32 where the values are formed in float32 (convolution, Gaussian, slope and aspect
of a float32 DEM, the band stacks) and the functions' default float64 where they are exact or formed
in more than float32 (terrain derivatives, focal statistics, integer DEMs).
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch
import torch.nn.functional as F

_PKG = str(Path(__file__).resolve().parents[1] / "vibespatial-raster_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import vsr_gb300 as vsr  # noqa: E402
from vsr_gb300.batch import TerrainBatch  # noqa: E402

ND = -9999.0
_NP = {"u8": np.uint8, "i16": np.int16, "u16": np.uint16, "f32": np.float32}
_TORCH = {"u8": torch.uint8, "i16": torch.int16, "u16": torch.uint16, "f32": torch.float32}
_SIZE = {"u8": 1, "i16": 2, "u16": 2, "f32": 4, "f64": 8}
_OUT = {"f32": np.float32, "f64": np.float64}


def listed() -> list[dict]:
    return [
        # one map tile of a viewer: the smallest call, where host work and the launch count
        {"name": "hillshade_f32_512", "op": "hillshade", "dtype": "f32", "bands": 1, "h": 512, "w": 512,
         "nodata": True},
        # slope, aspect and hillshade of one integer elevation tile with an odd side (float64 results)
        {"name": "terrain_i16_3601", "op": "terrain", "dtype": "i16", "bands": 1, "h": 3601, "w": 3601,
         "nodata": True},
        # the benchmark's headline: all three from one large float32 DEM with disc holes
        {"name": "terrain_f32_16384", "op": "terrain", "dtype": "f32", "bands": 1, "h": 16384, "w": 16384,
         "nodata": True},
        # ruggedness, position index and curvature of a regional DEM, rows not a multiple of 16 bytes
        {"name": "derivatives_f32_9001x7201", "op": "derivatives", "dtype": "f32", "bands": 1, "h": 9001, "w": 7201,
         "nodata": True},
        # an ordinary small smoothing kernel on a scene with holes, odd sides
        {"name": "convolve5_f32_4099x5003", "op": "convolve", "dtype": "f32", "bands": 1, "h": 4099, "w": 5003,
         "k": 5, "nodata": True, "out": "f32"},
        # the benchmark's large dense kernel
        {"name": "convolve31_f32_8192", "op": "convolve", "dtype": "f32", "bands": 1, "h": 8192, "w": 8192,
         "k": 31, "nodata": False, "out": "f32"},
        # smoothing a DEM before terrain analysis: default kernel size of sigma 2
        {"name": "gaussian13_f32_6000", "op": "gaussian", "dtype": "f32", "bands": 1, "h": 6000, "w": 6000,
         "sigma": 2.0, "k": 13, "nodata": True, "out": "f32"},
        # the benchmark's multiband scene, its wide Gaussian
        {"name": "gaussian65_u16_12x10980", "op": "gaussian", "dtype": "u16", "bands": 12, "h": 10980, "w": 10980,
         "sigma": 8.0, "k": 65, "nodata": True, "out": "f32"},
        # the same scene, its focal mean
        {"name": "mean7_u16_12x10980", "op": "mean", "dtype": "u16", "bands": 12, "h": 10980, "w": 10980,
         "r": 3, "nodata": True, "out": "f32"},
        # roughness: standard deviation of a float32 DEM in a 7 x 7 window
        {"name": "std7_f32_4096", "op": "std", "dtype": "f32", "bands": 1, "h": 4096, "w": 4096,
         "r": 3, "nodata": True, "out": "f64"},
        # diversity of a land-cover map: distinct classes in a 5 x 5 window, odd sides
        {"name": "variety5_u8_5001x4999", "op": "variety", "dtype": "u8", "bands": 1, "h": 5001, "w": 4999,
         "r": 2, "nodata": True, "out": "f64"},
        # uneven DEM tiles (sides 256 .. 4096, own cell size and nodata) in one planned launch, replayed
        {"name": "batch_f32_20_tiles", "op": "batch", "tiles": 20, "lo": 256, "hi": 4096, "pattern": 0},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, most) -> tuple[int, int]:
    """Two sides, log-uniform in [lo, hi], at most ``most`` pixels; half of the widths a multiple of 16."""
    h, w = _log(rng, lo, hi), _log(rng, lo, hi)
    if h * w > most:
        f = math.sqrt(most / (h * w))
        h, w = max(lo // 2, int(h * f)), max(lo // 2, int(w * f))
    if rng.random() < 0.5:
        w = max(16, w // 16 * 16)
    return h, w


def draw(rng) -> dict:
    op = rng.choice(["hillshade", "terrain", "terrain", "derivatives", "convolve", "convolve", "gaussian", "gaussian",
                     "mean", "stat", "stat", "variety", "batch"])
    nd = rng.random() < 0.75
    if op == "batch":
        return {"op": "batch", "tiles": _log(rng, 2, 21), "lo": 256, "hi": _log(rng, 1024, 4096),
                "pattern": rng.randrange(1, 1 << 20)}
    c = {"op": op, "nodata": nd, "bands": 1}
    if op == "hillshade":
        c["dtype"] = "f32"
        c["h"], c["w"] = _sides(rng, 200, 2048, 2048 * 2048)
    elif op == "terrain":
        c["dtype"] = rng.choice(["f32", "f32", "i16"])
        c["h"], c["w"] = _sides(rng, 300, 16384, 120_000_000)
    elif op == "derivatives":
        c["dtype"] = rng.choice(["f32", "f32", "i16"])
        c["h"], c["w"] = _sides(rng, 300, 10000, 64_000_000)
    elif op == "convolve":
        c["dtype"] = rng.choice(["f32", "f32", "u16"])
        c["k"] = rng.choice([3, 5, 7, 9, 11, 15, 21, 31])
        c["h"], c["w"] = _sides(rng, 300, 8192, 8192 * 8192 if c["k"] >= 15 else 4096 * 8192)
        c["out"] = "f32"
    elif op == "gaussian":
        c["dtype"] = rng.choice(["f32", "f32", "u16", "i16"])
        c["sigma"] = round(math.exp(rng.uniform(math.log(0.8), math.log(8.0))), 2)
        c["k"] = 2 * math.ceil(3 * c["sigma"]) + 1
        c["bands"] = rng.choice([1, 1, 3])
        c["h"], c["w"] = _sides(rng, 300, 10980, 60_000_000 // c["bands"])
        c["out"] = "f32"
    elif op == "mean":
        c["dtype"] = rng.choice(["u8", "u16", "u16", "i16", "f32"])
        c["r"] = rng.choice([1, 2, 3, 3, 4, 7])
        c["bands"] = rng.choice([1, 3, 4])
        c["h"], c["w"] = _sides(rng, 300, 10980, 120_000_000 // c["bands"])
        c["out"] = rng.choice(["f32", "f64"])
    elif op == "stat":
        c["op"] = rng.choice(["std", "std", "min", "max", "range"])
        c["dtype"] = rng.choice(["f32", "f32", "u16", "i16"])
        c["r"] = rng.choice([1, 2, 3, 4, 5])
        c["h"], c["w"] = _sides(rng, 300, 8192, 25_000_000)
        c["out"] = "f64"
    else:
        c["dtype"] = rng.choice(["u8", "u8", "i16", "u16"])
        c["r"] = rng.choice([1, 2, 3])
        c["h"], c["w"] = _sides(rng, 300, 5001, 25_000_000)
        c["out"] = "f64"
    return c


# ---- inputs -------------------------------------------------------------------------------------


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _fbm(h: int, w: int, g: torch.Generator, lo: float, hi: float) -> torch.Tensor:
    """Fractional-Brownian elevations: octaves of bilinear value noise, Hurst 0.8, in [lo, hi]."""
    acc = torch.zeros((h, w), device="cuda")
    for o in range(8):
        n = 4 * 2**o + 1
        grid = torch.rand((1, 1, n, n), generator=g, device="cuda")
        acc.add_(F.interpolate(grid, size=(h, w), mode="bilinear", align_corners=True)[0, 0], alpha=2.0 ** (-0.8 * o))
    mn, mx = torch.aminmax(acc)
    return acc.sub_(mn).mul_((hi - lo) / (mx - mn)).add_(lo)


def _holes(d: torch.Tensor, g: torch.Generator, value: float) -> None:
    """Nodata as DEMs have it: about 1 % in blobs (a coarse noise field above a threshold) and single pixels."""
    h, w = d.shape
    coarse = torch.rand((1, 1, h // 64 + 2, w // 64 + 2), generator=g, device="cuda")
    blob = F.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=True)[0, 0] > 0.97
    d[blob] = value
    n = max(1, h * w // 5000)
    d.view(-1)[torch.randint(0, h * w, (n,), generator=g, device="cuda")] = value


def _raster(case: dict, seed: int):
    """(B, H, W) or (H, W) device tensor and the nodata value of the case's raster."""
    g = _gen(seed)
    h, w, dt, bands, op = case["h"], case["w"], case["dtype"], case["bands"], case["op"]
    nd = None
    if op == "variety":  # class map: patches of 12 classes and salt noise, 0 = unclassified
        n = 12 if dt == "u8" else 400
        coarse = torch.randint(1, n + 1, (1, 1, h // 6 + 2, w // 6 + 2), generator=g, device="cuda").float()
        d = F.interpolate(coarse, size=(h, w), mode="nearest")[0, 0]
        salt = torch.rand((h, w), generator=g, device="cuda")
        d = torch.where(salt < 0.05, torch.floor(salt * 20.0 * n) + 1.0, d).clamp_(1, n)
        if case["nodata"]:
            nd = 0
            _holes(d, g, 0.0)
        return d.to(torch.int32).to(_TORCH[dt]), nd
    if dt in ("u16", "u8"):  # reflectances: gamma (shape 2) values, 3 % of pixels 0 = nodata
        top, scale = (10000.0, 800.0) if dt == "u16" else (255.0, 30.0)
        out = torch.empty((bands, h, w), dtype=_TORCH[dt], device="cuda")
        for b in range(bands):
            u = torch.rand((h, w), generator=g, device="cuda").clamp_(min=1e-7)
            u.mul_(torch.rand((h, w), generator=g, device="cuda").clamp_(min=1e-7)).log_().mul_(-scale).clamp_(1.0, top)
            if case["nodata"]:
                u[torch.rand((h, w), generator=g, device="cuda") < 0.03] = 0.0
            out[b] = u.to(torch.int32).to(_TORCH[dt])
        return (out[0] if bands == 1 else out), (0 if case["nodata"] else None)
    stack = []
    for _ in range(bands):
        if op == "convolve":  # noise on a linear trend
            d = torch.rand((h, w), generator=g, device="cuda")
            d.add_(torch.linspace(0.0, 100.0, h, device="cuda")[:, None])
        else:
            d = _fbm(h, w, g, 0.0, 4500.0)
        if dt == "i16":
            d = d.round_()
        if case["nodata"]:
            nd = ND if dt == "f32" else int(ND)
            _holes(d, g, ND)
        stack.append(d.to(_TORCH[dt]))
    return (stack[0] if bands == 1 else torch.stack(stack)), nd


def _tile_shapes(case: dict) -> list[tuple[int, int, float, float, float]]:
    """(height, width, cell size, nodata, nodata share) of each tile: the batch's own layout."""
    rng = np.random.default_rng(1000 + case["pattern"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    out = []
    for _ in range(case["tiles"]):
        h, w = (int(round(math.exp(rng.uniform(lo, hi)))) for _ in range(2))
        out.append((h, w, float(rng.uniform(1.0, 90.0)), ND if rng.random() < 0.5 else float("nan"),
                    float(rng.uniform(0.0, 0.05))))
    return out


def _tiles(case: dict, seed: int) -> list[tuple[torch.Tensor, float, tuple]]:
    g = _gen(seed)
    got = []
    for h, w, cell, nd, share in _tile_shapes(case):
        d = _fbm(h, w, g, 0.0, 3000.0)
        d[torch.rand((h, w), generator=g, device="cuda") < share] = nd
        got.append((d, nd, (cell, 0.0, 0.0, 0.0, -cell, 0.0)))
    return got


def _weights(case: dict, seed: int) -> np.ndarray:
    w = np.random.default_rng(seed).random((case["k"], case["k"]))
    return w / w.sum()


_AFFINE = (10.0, 0.0, 600000.0, 0.0, -10.0, 5000000.0)


def prepare(case: dict, seed: int) -> dict:
    if case["op"] == "batch":
        rasters = [vsr.from_device(d, nodata=nd, affine=af) for d, nd, af in _tiles(case, seed)]
        batch = TerrainBatch(rasters, sigma=1.0, kernel_size=5)
        batch.capture()
        return {"case": case, "batch": batch}
    d, nd = _raster(case, seed)
    state = {"case": case, "raster": vsr.from_device(d, nodata=nd, affine=_AFFINE)}
    if case["op"] == "convolve":
        state["weights"] = _weights(case, seed)
    return state


# ---- one pass -----------------------------------------------------------------------------------

_STAT = {"mean": vsr.raster_focal_mean, "std": vsr.raster_focal_std, "min": vsr.raster_focal_min,
         "max": vsr.raster_focal_max, "range": vsr.raster_focal_range, "variety": vsr.raster_focal_variety}


def run(state: dict):
    case = state["case"]
    op = case["op"]
    if op == "batch":
        state["batch"].replay()
        return state["batch"].outputs
    r = state["raster"]
    if op == "hillshade":
        return vsr.raster_hillshade(r).device_data()
    if op == "terrain":
        return {k: v.device_data() for k, v in vsr.raster_terrain(r).items()}
    if op == "derivatives":
        return {k: v.device_data() for k, v in vsr.raster_terrain_derivatives(r).items()}
    if op == "convolve":
        return vsr.raster_convolve(r, state["weights"], out_dtype=_OUT[case["out"]]).device_data()
    if op == "gaussian":
        return vsr.raster_gaussian_filter(r, case["sigma"], kernel_size=case["k"],
                                          out_dtype=_OUT[case["out"]]).device_data()
    return _STAT[op](r, case["r"], out_dtype=_OUT[case["out"]]).device_data()


def work(case: dict) -> dict:
    """Each input read once, each output written once; one multiply-add per tap where the path is a sum over taps."""
    op = case["op"]
    if op == "batch":
        px = sum(h * w for h, w, *_ in _tile_shapes(case))
        return {"bytes": 16 * px, "flops": px * (60 + 2 * 2 * 5 * 2)}
    px, src = case["bands"] * case["h"] * case["w"], _SIZE[case["dtype"]]
    fl = 4 if case["dtype"] == "f32" else 8
    if op == "hillshade":
        return {"bytes": px * (src + 1), "flops": 40 * px}
    if op == "terrain":
        return {"bytes": px * (src + 2 * fl + 1), "flops": 90 * px}
    if op == "derivatives":
        return {"bytes": px * (src + 3 * 8), "flops": 45 * px}
    out = _SIZE[case["out"]]
    if op == "convolve":
        return {"bytes": px * (src + out), "flops": 2 * case["k"] ** 2 * px}
    if op == "gaussian":
        return {"bytes": px * (src + out), "flops": 2 * 2 * case["k"] * px}
    return {"bytes": px * (src + out), "flops": 2 * 2 * (2 * case["r"] + 1) * px}


# ---- the same in 64 bits --------------------------------------------------------------------------


def _shifts(p: torch.Tensor, kh: int, kw: int):
    """The kh x kw shifted views of a padded array."""
    h, w = p.shape[0] - kh + 1, p.shape[1] - kw + 1
    for i in range(kh):
        for j in range(kw):
            yield i, j, p[i:i + h, j:j + w]


def _edge_pad(z: torch.Tensor) -> torch.Tensor:
    z = torch.cat([z[:1], z, z[-1:]], 0)
    return torch.cat([z[:, :1], z, z[:, -1:]], 1)


def _touches(mask: torch.Tensor) -> torch.Tensor:
    out = torch.zeros_like(mask)
    for _, _, v in _shifts(F.pad(mask, (1, 1, 1, 1)), 3, 3):
        out |= v
    return out


def _exact_slope_aspect(d: torch.Tensor, nd, cell: float):
    z = d.double()
    p = [v for _, _, v in _shifts(_edge_pad(z), 3, 3)]
    gx = ((p[2] + 2.0 * p[5] + p[8]) - (p[0] + 2.0 * p[3] + p[6])) / (8.0 * cell)
    gy = ((p[6] + 2.0 * p[7] + p[8]) - (p[0] + 2.0 * p[1] + p[2])) / (8.0 * cell)
    s = torch.rad2deg(torch.atan((gx * gx + gy * gy).sqrt_()))
    a = torch.remainder(90.0 - torch.rad2deg(torch.atan2(-gy, gx)), 360.0)
    if nd is not None and nd == nd:
        ring = _touches(z == nd)
        s[ring] = nd
        a[ring] = nd
    return s, a


def _exact_derivatives(d: torch.Tensor, nd, cell: float) -> dict:
    z = d.double()
    out_nd = float(nd) if nd is not None else ND
    edge = torch.ones_like(z, dtype=torch.bool)
    edge[1:-1, 1:-1] = False
    if nd is not None:
        edge |= _touches(z == nd)
    tri, tot = torch.zeros_like(z), torch.zeros_like(z)
    p = _edge_pad(z)
    for i, j, v in _shifts(p, 3, 3):
        if (i, j) != (1, 1):
            tri += (v - z).abs_()
            tot += v
    h, w = z.shape
    dx = ((p[1:-1, :w] + p[1:-1, 2:]) / 2.0 - z) / (cell * cell)
    dy = ((p[:h, 1:-1] + p[2:, 1:-1]) / 2.0 - z) / (cell * cell)
    got = {"tri": tri / 8.0, "tpi": z - tot / 8.0, "curvature": -200.0 * (dx + dy)}
    for v in got.values():
        v[edge] = out_nd
    return got


def _correlate(z: torch.Tensor, wy, wx) -> torch.Tensor:
    """Zero-padded correlation with the outer product of two weight vectors."""
    ky, kx = len(wy), len(wx)
    h, w = z.shape
    p = F.pad(z, (kx // 2, kx // 2, 0, 0))
    t = torch.zeros_like(z)
    for j in range(kx):
        t.add_(p[:, j:j + w], alpha=float(wx[j]))
    p = F.pad(t, (0, 0, ky // 2, ky // 2))
    out = torch.zeros_like(z)
    for i in range(ky):
        out.add_(p[i:i + h], alpha=float(wy[i]))
    return out


def _weighted(d: torch.Tensor, nd, correlate) -> torch.Tensor:
    """sum w v valid / sum w valid; a nodata centre or an empty window gives nodata (0 without one)."""
    z = d.double()
    valid = ~(z.isnan() if nd is not None and nd != nd else z == nd) if nd is not None else torch.ones_like(z).bool()
    num, den = correlate(z * valid), correlate(valid.double())
    fill = float(nd) if nd is not None else 0.0
    out = torch.where(den > 0.0, num / den, fill)
    out[~valid] = fill
    return out


def _exact_stat(d: torch.Tensor, nd, r: int, op: str) -> torch.Tensor:
    z = d.double()
    valid = z != nd if nd is not None else torch.ones_like(z).bool()
    fill, k = (float(nd) if nd is not None else 0.0), 2 * r + 1
    pad = (r, r, r, r)
    vp = F.pad(valid, pad)
    if op in ("min", "max", "range"):
        lo, hi = torch.full_like(z, math.inf), torch.full_like(z, -math.inf)
        for _, _, v in _shifts(F.pad(torch.where(valid, z, math.inf), pad, value=math.inf), k, k):
            torch.minimum(lo, v, out=lo)
        for _, _, v in _shifts(F.pad(torch.where(valid, z, -math.inf), pad, value=-math.inf), k, k):
            torch.maximum(hi, v, out=hi)
        out = lo if op == "min" else hi if op == "max" else hi - lo
    else:
        zp = F.pad(torch.where(valid, z, 0.0), pad)
        n, s = torch.zeros_like(z), torch.zeros_like(z)
        for (_, _, v), (_, _, m) in zip(_shifts(zp, k, k), _shifts(vp, k, k)):
            s += v
            n += m
        mean = s / n
        s.zero_()
        for (_, _, v), (_, _, m) in zip(_shifts(zp, k, k), _shifts(vp, k, k)):
            s += torch.where(m, v - mean, 0.0).square_()
        out = (s / n).sqrt_()
    out[~valid] = fill
    return out


def _exact_variety(d: torch.Tensor, nd, r: int) -> torch.Tensor:
    z = d.to(torch.int32)
    valid = z != nd if nd is not None else torch.ones_like(z).bool()
    k, pad = 2 * r + 1, (r, r, r, r)
    taps = [(v, m) for (_, _, v), (_, _, m) in
            zip(_shifts(F.pad(z.to(torch.int16), pad), k, k), _shifts(F.pad(valid, pad), k, k))]
    count = torch.zeros_like(z, dtype=torch.float64)
    for i, (v, m) in enumerate(taps):
        new = m.clone()
        for u, mu in taps[:i]:
            new &= ~((u == v) & mu)
        count += new
    count[~valid] = float(nd) if nd is not None else 0.0
    return count


def exact(case: dict, seed: int):
    op = case["op"]
    if op == "batch":
        g = np.exp(-0.5 * np.arange(-2, 3) ** 2.0)
        g /= g.sum()
        out = []
        for d, nd, af in _tiles(case, seed):
            s, a = _exact_slope_aspect(d, nd, af[0])
            out.append((s, a, _weighted(d, nd, lambda z: _correlate(z, g, g))))
        return out
    d, nd = _raster(case, seed)
    cell = abs(_AFFINE[0])
    if op == "hillshade":
        return None
    if op == "terrain":
        s, a = _exact_slope_aspect(d, nd, cell)
        return {"slope": s, "aspect": a, "hillshade": None}
    if op == "derivatives":
        return _exact_derivatives(d, nd, cell)
    if op == "variety":
        return _exact_variety(d, nd, case["r"])
    if op in ("std", "min", "max", "range"):
        return _exact_stat(d, nd, case["r"], op)
    if op == "convolve":
        wt = _weights(case, seed)
        k = case["k"]

        def correlate(z):
            acc = torch.zeros_like(z)
            for i, j, v in _shifts(F.pad(z, (k // 2,) * 4), k, k):
                acc.add_(v, alpha=float(wt[i, j]))
            return acc

        return _weighted(d, nd, correlate)
    if op == "gaussian":
        g = np.exp(-0.5 * ((np.arange(case["k"]) - case["k"] // 2) / case["sigma"]) ** 2)
        g /= g.sum()
    else:
        g = np.ones(2 * case["r"] + 1)
    correlate = lambda z: _correlate(z, g, g)  # noqa: E731
    if d.ndim == 2:
        return _weighted(d, nd, correlate)
    return torch.stack([_weighted(b, nd, correlate) for b in d])
