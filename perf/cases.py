"""Timed cases of the annual irradiance path, through the public entry points.

Each case is one call (or one training step) that a user of this package
makes: the annual run of a device-resident or host-resident scene with either
list format, the re-run of a traced scene with another year's weather, the
annual form, a batch of uneven tiles, Stage 1 alone (lists for a cache, shadow
words of a few voxels), voxelization, and one training step of the visibility
surrogate.  Scenes are seeded synthetic cities with the densities of the
named workloads (solargpu_b200/inputs.py) at a seeded site; sides run from
the 64-cell plain case to the 1024-cell city, odd and non-square ones among
them.  ``exact`` restates the path in plain torch with 64-bit irradiance.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from solargpu_b200 import api, inputs, surrogate

CITY = inputs.CONFIGS["dsm1024"]
HOURS = 8760
DIRECTIONS = 2592
DAYLIGHT = 4320          # daylight hours of a year (4278 to 4337 at the sites used)
NEIGHBORS = 250          # neighbor ids a voxel on these scenes
WEIGHTS = 205            # of them with a nonzero reflection weight


def listed():
    return [
        # the smallest scene of the package: one courtyard, latency of a whole annual run
        {"name": "site_64", "kind": "run", "w": 64, "h": 64, "format": 0, "accumulation": 0, "reflection": 0},
        # a small town with the compressed lists and compensated sums
        {"name": "town_160_barle", "kind": "run", "w": 160, "h": 160, "format": 1, "accumulation": 1, "reflection": 0},
        # the drop-in C entry point on a raster of the size the reference ships (host arrays in and out)
        {"name": "dropin_366x320", "kind": "dropin", "w": 366, "h": 320, "format": 0},
        # a quarter of the city, defaults
        {"name": "city_512", "kind": "run", "w": 512, "h": 512, "format": 0, "accumulation": 0, "reflection": 0},
        # the same area with the compressed lists, odd sides
        {"name": "city_517x489_barle", "kind": "run", "w": 517, "h": 489, "format": 1, "accumulation": 1,
         "reflection": 0},
        # the city: the benchmark's workload (CSR, compensated sums)
        {"name": "city_1024", "kind": "run", "w": 1024, "h": 1024, "format": 0, "accumulation": 1, "reflection": 0},
        # the annual form, for who wants only the year's sum
        {"name": "annual_384", "kind": "run", "w": 384, "h": 384, "format": 0, "accumulation": 0, "reflection": 1},
        # a traced scene again with another year's weather: saved lists in, no tracing
        {"name": "reweather_200", "kind": "relist", "w": 200, "h": 200, "format": 0},
        # Stage 1 for the cache: both list formats and the shadow words, copied to the host
        {"name": "lists_181x143", "kind": "lists", "w": 181, "h": 143},
        # uneven tiles of a larger area in one batch
        {"name": "batch_5_tiles", "kind": "batch", "tiles": 5, "lo": 128, "hi": 400},
        # a heightmap to voxels, before any of the above
        {"name": "voxelize_2000", "kind": "voxelize", "w": 2000, "h": 2000},
        # one training step of the visibility surrogate (labels, images, forward, backward)
        {"name": "surrogate_step_1024", "kind": "train", "batch": 1024},
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["run", "run", "run", "run", "dropin", "relist", "lists", "batch", "voxelize", "train"])
    if kind == "train":
        return {"kind": kind, "batch": 128 * rng.randint(1, 8)}
    if kind == "voxelize":
        return {"kind": kind, "w": side(128, 2000), "h": side(128, 2000)}
    if kind == "batch":
        return {"kind": kind, "tiles": rng.randint(2, 6), "lo": 128, "hi": rng.randint(200, 400)}
    if kind == "lists":
        return {"kind": kind, "w": side(64, 200), "h": side(64, 200)}
    if kind == "relist":
        return {"kind": kind, "w": side(64, 256), "h": side(64, 256), "format": rng.randint(0, 1)}
    if kind == "dropin":
        return {"kind": kind, "w": side(64, 400), "h": side(64, 400), "format": rng.randint(0, 1)}
    return {"kind": kind, "w": side(64, 900), "h": side(64, 900), "format": rng.randint(0, 1),
            "accumulation": rng.randint(0, 2), "reflection": rng.choice([0, 0, 0, 0, 1, 2])}


# ---------------------------------------------------------------- inputs

WALLS = 0.40             # wall voxels a cell (the 1024 city has 0.44 before any is left out)


def _cfg(n, seed):
    area = (n / CITY.size) ** 2
    return inputs.DsmConfig("scene", n, max(2, round(CITY.n_buildings * area)), max(4, round(CITY.n_trees * area)),
                            side_max=min(30, n // 2), seed=seed)


def _heights(w, h, seed):
    """A cut of a seeded synthetic city with the 1024 city's densities."""
    return inputs.make_dsm(_cfg(max(w, h), seed))[:h, :w].copy()


@functools.lru_cache(maxsize=8)
def _sun(lon, lat, tz):
    return inputs.sun_positions(lon, lat, tz)


def _scene(w, h, seed):
    """A scene at a seeded site (latitude 35 to 60, longitude -10 to 30) with
    seeded weather.  Every seed has the same number of voxels: a city with
    too few walls gets more trees, and of too many a random part is left out
    (facades nobody asked for)."""
    rng = np.random.default_rng(seed)
    lat, lon = round(float(rng.uniform(35.0, 60.0)), 3), round(float(rng.uniform(-10.0, 30.0)), 3)
    z, want, top = _heights(w, h, seed), int(WALLS * w * h), w * h
    while True:
        total, _, pp, wz, sl, asp = inputs.voxelize(z, 1.0)
        if total - top >= want:
            break
        y, x = np.mgrid[0:h, 0:w]
        for _ in range(max(1, (want - (total - top)) // 150)):   # a tree brings about 100 wall voxels
            cy, cx = rng.uniform(0, h), rng.uniform(0, w)
            y0, y1, x0, x1 = max(0, int(cy) - 8), int(cy) + 9, max(0, int(cx) - 8), int(cx) + 9
            d2 = (x[y0:y1, x0:x1] + 0.5 - cx) ** 2 + (y[y0:y1, x0:x1] + 0.5 - cy) ** 2
            bump = (1.5 + rng.uniform(5.0, 15.0) * np.exp(-d2 / 8.0)).astype(np.float32)
            z[y0:y1, x0:x1] = np.maximum(z[y0:y1, x0:x1], bump)
    keep = np.concatenate([np.arange(top), top + np.sort(rng.permutation(total - top)[:want])])
    sun = _sun(lon, lat, int(round(lon / 15.0)))
    direct, diffuse = inputs.make_tmy(sun, seed)
    return inputs.Scene("scene", z.ravel(), w, h, top + want, top, pp[keep], wz[keep[top:] - top], float(z.max()), sun,
                        direct, diffuse, sl[keep], asp[keep])


def _to_device(s):
    wz = s.wall_z if s.wall_z.size else np.zeros(1, np.float32)
    return {k: torch.from_numpy(a).cuda() for k, a in
            (("grid", s.grid), ("pixel_parent", s.pixel_parent), ("wall_z", wz), ("slopes", s.slopes),
             ("aspects", s.aspects))}


def _tile_sides(case, seed):
    rng = np.random.default_rng(seed)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    # the same sizes for every seed, so that the work is the case's own
    r = np.random.default_rng(case["tiles"] * 1000 + case["hi"])
    return [int(math.exp(r.uniform(lo, hi))) // 16 * 16 for _ in range(case["tiles"])], \
        [int(x) for x in rng.integers(1, 1 << 30, case["tiles"])]


ACTIVE = 265
CONV = (64, 64, 128, 128)


def _train_weights(seed):
    """Seeded weights of the conv surrogate, as a checkpoint would hold them."""
    g = torch.Generator().manual_seed(seed)
    shapes, cin, real = [], 2, []
    for c in CONV:
        kp = (16 * cin + 127) // 128 * 128
        shapes.append((c, kp))
        real.append(16 * cin)
        cin = c
    for a, o in ((2112, 512), (512, 512), (512, 512), (512, 384)):
        shapes.append((o, a))
        real.append(a)
    W = []
    for (o, k), r in zip(shapes, real):
        w = torch.zeros(o, k)
        w[:, :r] = torch.randn(o, r, generator=g) * math.sqrt(2.0 / r)
        W.append(w)
    return W, [torch.randn(o, generator=g) * 0.05 for o, _ in shapes]


def _train_data(case, seed):
    s = _scene(200, 200, seed)
    rng = np.random.default_rng(seed + 1)
    n = case["batch"]
    vox = rng.integers(0, s.num_total, n, dtype=np.int32)
    words = rng.integers(0, 1 << 32, (s.num_total, (ACTIVE + 31) // 32), dtype=np.uint32)
    share = rng.random(s.num_total).astype(np.float32) * np.float32(0.3)
    return s, vox, words, share


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        s, vox, words, share = _train_data(case, seed)
        model = surrogate.Surrogate(active=ACTIVE, conv=CONV)
        W, b = _train_weights(seed)
        model.W, model.b = [w.cuda() for w in W], [x.cuda() for x in b]
        model.Wb = [w.to(torch.bfloat16) for w in model.W]
        dev = _to_device(s)
        return {"kind": kind, "model": model, "scene": s, "dev": dev, "vox": torch.from_numpy(vox).cuda(),
                "words": torch.from_numpy(words.view(np.int32)).cuda(), "share": torch.from_numpy(share).cuda()}
    if kind == "voxelize":
        z = _heights(case["w"], case["h"], seed)
        cap = 2 * z.size   # a program's own arrays, with room for the walls
        return {"kind": kind, "ctx": api.Context(0), "grid": torch.from_numpy(z.ravel()).cuda(), "w": case["w"],
                "h": case["h"], "cap": cap, "out": {
                    "pixel_parent": torch.zeros(cap, dtype=torch.int32, device="cuda"),
                    **{k: torch.zeros(cap, dtype=torch.float32, device="cuda")
                       for k in ("wall_z", "slopes", "aspects")}}}
    if kind == "batch":
        scenes = [_scene(n, n, k) for n, k in zip(*_tile_sides(case, seed))]
        return {"kind": kind, "ctxs": [api.Context(0) for _ in scenes], "scenes": scenes,
                "devs": [_to_device(s) for s in scenes],
                "outs": [torch.zeros(s.num_total, dtype=torch.float32, device="cuda") for s in scenes]}
    s = _scene(case["w"], case["h"], seed)
    if kind == "dropin":
        return {"kind": kind, "scene": s, "format": case["format"], "out": np.zeros(s.num_total, np.float32)}
    st = {"kind": kind, "ctx": api.Context(0), "scene": s, "dev": _to_device(s),
          "out": torch.zeros(s.num_total, dtype=torch.float32, device="cuda")}
    if kind == "lists":   # page-locked arrays that the program keeps for the lists of a tile
        n = s.num_total
        st["lists"] = {k: torch.zeros(m, dtype=d).pin_memory() for k, m, d in
                       (("csr_off", n + 1, torch.int64), ("csr_ids", 400 * n, torch.int32),
                        ("barle_off", n + 1, torch.int64), ("barle", 600 * n, torch.uint8),
                        ("shadow", 12 * n, torch.int32))}
    elif kind == "relist":
        st["lists"] = st["ctx"].trace(s, st["dev"], neighbor_format=case["format"])
        s.direct, s.diffuse = inputs.make_tmy(s.sun, seed + 99)
    elif kind == "run":
        st["options"] = dict(neighbor_format=case["format"], accumulation=case["accumulation"],
                             reflection=case["reflection"])
    return st


def _check(rc):
    if rc != 0:
        raise RuntimeError(api.lib().solar_gpu_last_error().decode())


def run(st):
    kind = st["kind"]
    if kind == "train":
        m = st["model"]
        y = m.labels(st["words"], (ACTIVE + 31) // 32, st["vox"], st["share"])
        img, nrm = m.inputs(st["scene"], st["dev"], st["vox"])
        loss, dW, db = m.gradients(img, y, nrm)
        return {"loss": loss, "dW": dW, "db": db}
    if kind == "voxelize":
        n, o = ctypes.c_longlong(), st["out"]
        _check(api.lib().solar_gpu_voxelize(st["ctx"].h, st["grid"].data_ptr(), st["w"], st["h"], 1.0, ctypes.byref(n),
                                            *(o[k].data_ptr() for k in ("pixel_parent", "wall_z", "slopes", "aspects")),
                                            st["cap"], None))
        return dict(o, num_total=int(n.value))
    if kind == "batch":
        api.run_batch(st["ctxs"], st["scenes"], st["devs"], st["outs"])
        return st["outs"]
    s = st["scene"]
    if kind == "dropin":
        fn = api.compressed_gpu_irradiance if st["format"] else api.uncompressed_gpu_irradiance
        fn(s.grid, s.width, s.height, s.num_total, s.num_top, s.pixel_parent, s.wall_z, s.max_height, s.sun, s.direct,
           s.diffuse, s.slopes, s.aspects, st["out"])
        return st["out"]
    if kind == "lists":
        st["ctx"].stage1(s, st["dev"], neighbor_format=api.BOTH)
        ids, size, words = ctypes.c_longlong(), ctypes.c_longlong(), ctypes.c_int()
        _check(api.lib().solar_gpu_trace_sizes(st["ctx"].h, ctypes.byref(ids), ctypes.byref(size), ctypes.byref(words),
                                               None, None))
        o = st["lists"]
        if ids.value > o["csr_ids"].numel() or size.value > o["barle"].numel() or words.value > 12:
            raise ValueError("the arrays are too small for this tile")
        _check(api.lib().solar_gpu_trace_copy(st["ctx"].h, *(o[k].data_ptr() for k in (
            "csr_off", "csr_ids", "barle_off", "barle", "shadow"))))
        return o
    if kind == "relist":
        st["ctx"].run_lists(s, st["dev"], st["lists"], st["out"])
        return st["out"]
    st["ctx"].run_device(s, st["dev"], st["out"], **st["options"])
    return st["out"]


# ---------------------------------------------------------------- work

def _voxels(w, h):
    return (1.0 + WALLS) * w * h


def _run_work(w, h, trace, refl):
    """Bytes: the scene in, the year out.  Operations: 6 a DDA step (two
    compares, a min, two sums, one fused product) at the reference's mean of 15.7
    steps a ray, one fused product a nonzero weight and hour (or one a weight
    for the annual form), 20 a voxel and hour for the direct and diffuse term."""
    n = _voxels(w, h)
    f = 20.0 * n * DAYLIGHT
    if trace:
        f += 6.0 * 15.7 * DIRECTIONS * n
    if refl == 0:
        f += 2.0 * WEIGHTS * n * DAYLIGHT
    elif refl == 1:
        f += 2.0 * WEIGHTS * n
    return {"bytes": 4.0 * w * h + 4.0 * 5 * n + 16.0 * HOURS, "flops": f}


def work(case):
    kind = case["kind"]
    if kind == "train":
        mac, side, cin = 0.0, 64, 2
        for c in CONV:
            side //= 2
            mac += side * side * 16 * cin * c
            cin = c
        mac += 2112 * 512 + 2 * 512 * 512 + 512 * 384
        p = 2 * 16 * 64 + 64 * 16 * 64 + 64 * 16 * 128 + 128 * 16 * 128 + 2112 * 512 + 2 * 512 * 512 + 512 * 384
        return {"bytes": case["batch"] * (64 * 64 * 4 + 128 + 36) + 6.0 * p, "flops": 6.0 * mac * case["batch"]}
    w, h = case.get("w", 0), case.get("h", 0)
    if kind == "voxelize":
        n = _voxels(w, h)
        return {"bytes": 4.0 * w * h + 12.0 * n + 4.0 * (n - w * h), "flops": 40.0 * w * h}
    if kind == "batch":
        each = [_run_work(n, n, True, 0) for n in _tile_sides(case, 0)[0]]
        return {k: sum(x[k] for x in each) for k in ("bytes", "flops")}
    if kind == "lists":
        n = _voxels(w, h)
        return {"bytes": 4.0 * w * h + 12.0 * n + n * (NEIGHBORS * 5.5 + 16 + 36),
                "flops": 6.0 * 15.7 * DIRECTIONS * n}
    if kind == "relist":
        r = _run_work(w, h, False, 0)
        per = NEIGHBORS * (1.45 if case["format"] else 4.0) + 8 + 36
        return {"bytes": r["bytes"] + _voxels(w, h) * per, "flops": r["flops"]}
    return _run_work(w, h, True, case.get("reflection", 0))


# ---------------------------------------------------------------- 64-bit restatement

_F = np.array([
    [-0.0083117, 0.1299457, 0.3296958, 0.5682053, 0.8730280, 1.1326077, 1.0601591, 0.6777470],
    [0.5877285, 0.6825954, 0.4868735, 0.1874525, -0.3920403, -1.2367284, -1.5999137, -0.3272588],
    [-0.0620636, -0.1513752, -0.2210958, -0.2951290, -0.3616149, -0.4118494, -0.3589221, -0.2504286],
    [-0.0596012, -0.0189325, 0.0554140, 0.1088631, 0.2255647, 0.2877813, 0.2642124, 0.1561313],
    [0.0721249, 0.0659650, -0.0639588, -0.1519229, -0.4620442, -0.8230357, -1.1272340, -1.3765031],
    [-0.0220216, -0.0288748, -0.0260542, -0.0139754, 0.0012448, 0.0558651, 0.1310694, 0.2506212]],
    np.float32).astype(np.float64)
_EDGES = np.array([1.065, 1.230, 1.500, 1.950, 2.800, 4.500, 6.200], np.float32).astype(np.float64)


def _f(x):
    return float(np.float32(x))


def _sky(sun):
    """(nudged azimuth and altitude, sun bin of every hour or -1, dense index of every bin)."""
    nud = (sun[:HOURS] - np.float32(1e-8)).astype(np.float32)
    az, alt = nud[:, 0], nud[:, 1]
    up = alt >= np.float32(1.0)
    bi, bj = (az / np.float32(5)).astype(np.int64), (alt / np.float32(5)).astype(np.int64)
    ok = up & (bi >= 0) & (bi < 72) & (bj >= 0) & (bj < 18)
    used = np.zeros(72 * 18, bool)
    used[bi[ok] * 18 + bj[ok]] = True
    dense = np.where(used, np.cumsum(used) - 1, -1)
    return nud, up, np.where(ok, dense[np.clip(bi * 18 + bj, 0, 72 * 18 - 1)], -1), dense


def _directions():
    f = np.float32
    i, j = np.meshgrid(np.arange(72), np.arange(36), indexing="ij")
    el = ((np.where(j < 18, j, j - 18).astype(f) + f(0.5)) * f(5)) * f(0.0174532925)
    az = ((i.astype(f) + f(0.5)) * f(5)) * f(0.0174532925)

    # the host's own 32-bit cosine and sine, as the direction set is defined by them
    libm = ctypes.CDLL("libm.so.6")
    libm.cosf.restype = libm.sinf.restype = ctypes.c_float
    libm.cosf.argtypes = libm.sinf.argtypes = [ctypes.c_float]

    def c(x):
        return np.array([libm.cosf(float(v)) for v in x.ravel()], f).reshape(x.shape)

    def s(x):
        return np.array([libm.sinf(float(v)) for v in x.ravel()], f).reshape(x.shape)
    cx, cy, cz = c(el) * s(az), -c(el) * c(az), np.where(j < 18, s(el), -s(el))
    n = np.sqrt(cx * cx + cy * cy + cz * cz)
    return np.stack([cx / n, cy / n, cz / n], -1).reshape(-1, 3)


def _trace(s, chunk=16384):
    """First-hit cells (1-based, 0 = none) of every voxel and direction, in voxel chunks."""
    d = torch.from_numpy(_directions()).cuda()
    upper = (torch.arange(DIRECTIONS, device="cuda") % 36) < 18
    W, H = s.width, s.height
    grid = torch.from_numpy(s.grid).cuda()
    pp = torch.from_numpy(s.pixel_parent).cuda().long()
    base = torch.cat([grid, torch.from_numpy(s.wall_z).cuda()])
    one = torch.ones((), device="cuda")
    A, inv = d.abs().clamp_min(1e-8), 1.0 / d.abs().clamp_min(1e-8)
    for v0 in range(0, s.num_total, chunk):
        v = torch.arange(v0, min(s.num_total, v0 + chunk), device="cuda")
        gx, gy = (pp[v] % W).float()[:, None], torch.div(pp[v], W, rounding_mode="floor").float()[:, None]
        o = [(g + d[:, k] * 2.0).reshape(-1) for k, g in ((0, gx), (1, gy))]
        oz = (base[v][:, None] + d[:, 2] * 2.0).reshape(-1)
        c = [x.floor() for x in o]
        di = torch.arange(DIRECTIONS, device="cuda", dtype=torch.int32).repeat(v.numel())
        tm = []
        for k in (0, 1):
            pos = d[di, k] >= 0
            tm.append(torch.where(pos, c[k] + one - o[k], o[k] - c[k]) / A[di, k])
        ix, iy = c[0].int(), c[1].int()
        hit = torch.zeros(v.numel() * DIRECTIONS, dtype=torch.int32, device="cuda")
        ray = torch.arange(hit.numel(), device="cuda", dtype=torch.int32)
        tx, ty, step = tm[0], tm[1], 0
        while ray.numel():
            dd = di.long()
            xs = tx < ty
            t = torch.where(xs, tx, ty)
            sx = torch.where(d[dd, 0] >= 0, 1, -1).int()
            sy = torch.where(d[dd, 1] >= 0, 1, -1).int()
            ix, iy = torch.where(xs, ix + sx, ix), torch.where(xs, iy, iy + sy)
            tx, ty = torch.where(xs, tx + inv[dd, 0], tx), torch.where(xs, ty, ty + inv[dd, 1])
            inside = (ix >= 0) & (ix < W) & (iy >= 0) & (iy < H)
            zr = (oz.double() + d[dd, 2].double() * t.double()).float()
            inside &= torch.where(upper[dd], ~(zr > s.max_height), ~(zr < 0))
            cell = torch.where(inside, ix + iy * W, 0)
            stop = inside & ((grid[cell.long()] - zr) > 0.01)
            hit[ray[stop].long()] = cell[stop] + 1
            go = inside & ~stop
            ray, di, tx, ty, ix, iy, oz = (x[go] for x in (ray, di, tx, ty, ix, iy, oz))
            step += 1
        yield v, hit.view(v.numel(), DIRECTIONS)


def _hours(s, nud, up, sun_bin):
    """Per daylight hour, in 64 bits: the sun vector, DNI and the diffuse coefficients."""
    k = np.nonzero(up)[0]
    az, alt = nud[k, 0].astype(np.float64), nud[k, 1].astype(np.float64)
    rad, pi = _f(0.0174532925), _f(math.pi)
    cz = np.cos((90.0 - alt) * rad)
    z = np.arccos(cz)
    dn, df = s.direct[k].astype(np.float64), s.diffuse[k].astype(np.float64)
    am = 1.0 / (cz + _f(0.50572) * (_f(96.07995) - z * (180.0 / pi)) ** _f(-1.6364))
    z3 = _f(1.041) * z ** 3
    with np.errstate(all="ignore"):
        eps = ((df + dn / np.cos(z)) / df + z3) / (1.0 + z3)
    eps = np.fmax(1.0, eps)
    B = 2.0 * pi * ((k // 24) / 365.0)
    e0 = 1367.0 * (_f(1.00011) + _f(0.034221) * np.cos(B) + _f(0.00128) * np.sin(B)
                   + _f(0.000719) * np.cos(2 * B) + _f(0.000077) * np.sin(2 * B))
    delta = am * df / e0
    q = np.searchsorted(_EDGES, eps, side="right")
    F1 = np.maximum(0.0, _F[0, q] + _F[1, q] * delta + _F[2, q] * z)
    F2 = _F[3, q] + _F[4, q] * delta + _F[5, q] * z
    sun = np.stack([np.sin(z) * np.sin(az * rad), -np.sin(z) * np.cos(az * rad), cz], -1)
    b = np.maximum(_f(0.08715574), cz)
    cols = [sun[:, 0], sun[:, 1], sun[:, 2], np.maximum(dn, _f(1e-3)), df * (1 - F1) / 2, df * F1 / b, df * F2]
    return torch.from_numpy(np.stack(cols)).cuda(), torch.from_numpy(sun_bin[k]).cuda()


def _annual(s, reflect):
    """The year's irradiance of every voxel in 64 bits."""
    nud, up, sun_bin, dense = _sky(s.sun)
    hc, hbin = _hours(s, nud, up, sun_bin)
    nb = int(dense.max()) + 1 if (dense >= 0).any() else 0
    # the direction that traces each dense bin
    of_bin = torch.zeros(max(1, nb), dtype=torch.long, device="cuda")
    for q in np.nonzero(dense >= 0)[0]:
        of_bin[dense[q]] = int(q // 18) * 36 + int(q % 18)
    sl, asp = (torch.from_numpy(a).cuda().double() for a in (s.slopes, s.aspects))
    n = torch.stack([sl.sin() * asp.sin(), -sl.sin() * asp.cos(), sl.cos(), sl.sin()], -1)
    pp = torch.from_numpy(s.pixel_parent).cuda().long()
    z = torch.from_numpy(np.concatenate([s.grid, s.wall_z])).cuda().double()
    pos = torch.stack([(pp % s.width).double(), torch.div(pp, s.width, rounding_mode="floor").double(), z], -1)
    own = torch.zeros(s.num_total, dtype=torch.float64, device="cuda")
    lists = []
    has = hbin >= 0
    for v, hit in _trace(s):
        sh = hit[:, of_bin] != 0
        for a in range(0, v.numel(), 4096):
            m = n[v[a:a + 4096]]
            cosi = m[:, :3] @ hc[:3]
            lit = has[None, :] & ~sh[a:a + 4096][:, hbin.clamp_min(0)]
            dif = hc[4] * (1 + m[:, 2:3]) + hc[5] * cosi.clamp_min(0) + hc[6] * m[:, 3:4]
            own[v[a:a + 4096]] = (torch.where(lit & (cosi > 0), hc[3] * cosi, 0.0) + dif.clamp_min(0)).sum(1)
        if reflect:
            srt = hit.sort(1)[0]
            first = torch.ones_like(srt, dtype=torch.bool)
            first[:, 1:] = srt[:, 1:] != srt[:, :-1]
            r, c = torch.nonzero(first & (srt > 0), as_tuple=True)
            lists.append((v[0] + r, srt[r, c].long() - 1))
    out = own.clone()
    for me, g in lists:
        for a in range(0, me.numel(), 1 << 24):
            p, q = me[a:a + (1 << 24)], g[a:a + (1 << 24)]
            dv = pos[q] - pos[p]
            d2 = (dv * dv).sum(1)
            dist = d2.sqrt().clamp_min(1e-30)
            recv = (n[p, :3] * dv).sum(1) / dist
            send = (dv[:, 2].abs() / dist).clamp_min(_f(0.1))
            w = torch.where((d2 >= _f(1e-4)) & (recv > 0), _f(0.2) * recv * send / (_f(3.14159265) * d2.clamp_min(1e-30)),
                            0.0)
            out.index_add_(0, p, w * own[q])
    return out


def _train_exact(case, seed):
    s, vox, words, share = _train_data(case, seed)
    bf = lambda t: t.to(torch.bfloat16).double()  # noqa: E731  (the stored precision of inputs and weights)
    W, b = _train_weights(seed)
    W, b = [bf(w.cuda()).requires_grad_() for w in W], [x.cuda().double().requires_grad_() for x in b]
    z = s.grid.reshape(s.height, s.width)
    pp = s.pixel_parent[vox].astype(np.int64)
    gx, gy = pp % s.width, pp // s.width
    base = np.concatenate([s.grid, s.wall_z])[vox]
    hc, wc = (s.height + 7) // 8, (s.width + 7) // 8
    pad = np.full((hc * 8, wc * 8), -np.inf, np.float32)
    pad[:s.height, :s.width] = z
    coarse = pad.reshape(hc, 8, wc, 8).max((1, 3))

    def patch(a, x, y):
        q = np.zeros((a.shape[0] + 64, a.shape[1] + 64), np.float32)
        q[32:-32, 32:-32] = a
        off = np.arange(64)
        return q[(y[:, None] + off)[:, :, None], (x[:, None] + off)[:, None, :]]
    img = np.stack([patch(z, gx, gy), patch(coarse, gx // 8, gy // 8)], 1)
    img = np.clip((img - base[:, None, None, None]) * np.float32(0.02), -2, 2).astype(np.float32)
    x = bf(torch.from_numpy(img).cuda())
    sl, asp = (a[vox].astype(np.float64) * float(np.float32(0.017453292)) for a in (s.slopes, s.aspects))
    nrm = torch.zeros(len(vox), 64, dtype=torch.float64, device="cuda")
    nrm[:, :3] = torch.from_numpy(np.stack([np.sin(sl) * np.sin(asp), -np.sin(sl) * np.cos(asp), np.cos(sl)], 1)).cuda()
    nrm = bf(nrm)
    cin = 2
    for l, c in enumerate(CONV):   # columns (ky, kx, channel)
        k = W[l][:, :16 * cin].reshape(c, 4, 4, cin).permute(0, 3, 1, 2)
        x = torch.relu(torch.nn.functional.conv2d(x, k, b[l], stride=2, padding=1))
        cin = c
    h = torch.cat([x.permute(0, 2, 3, 1).reshape(len(vox), -1), nrm], 1)
    for l in range(4, 8):
        h = h @ W[l].T + b[l]
        if l < 7:
            h = torch.relu(h)
    bits = ((words[vox][:, :, None] >> np.arange(32, dtype=np.uint32)) & 1).reshape(len(vox), -1)[:, :ACTIVE]
    y = torch.cat([torch.from_numpy(bits.astype(np.float64)).cuda(),
                   torch.from_numpy(share[vox]).cuda().double()[:, None].expand(-1, 16)], 1)
    loss = torch.nn.functional.binary_cross_entropy_with_logits(h[:, :ACTIVE + 16], y)
    loss.backward()
    return {"loss": float(loss.detach()), "dW": [w.grad for w in W], "db": [x.grad for x in b]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train_exact(case, seed)
    if kind == "lists":      # whole numbers only
        return None
    if kind == "batch":
        return [_annual(_scene(n, n, k), True) for n, k in zip(*_tile_sides(case, seed))]
    w, h = case["w"], case["h"]
    if kind == "voxelize":
        return _voxelize_exact(_heights(w, h, seed), w, h)
    if w * h > 600 * 600:    # over the time such a check may take
        return None
    s = _scene(w, h, seed)
    if kind == "relist":
        s.direct, s.diffuse = inputs.make_tmy(s.sun, seed + 99)
    out = _annual(s, case.get("reflection", 0) != 2)
    return out.cpu().numpy() if kind == "dropin" else out


def _voxelize_exact(z, w, h):
    """Slopes and aspects in 64 bits; the counts, parents and wall heights
    follow 32-bit rules (whole numbers, and heights exact by them)."""
    g = torch.from_numpy(z).cuda()
    p = torch.nn.functional.pad(g, (1, 1, 1, 1), value=float("-inf"))
    sides = [p[1:-1, 2:], p[1:-1, :-2], p[:-2, 1:-1], p[2:, 1:-1]]
    low = torch.stack([torch.where(a.isinf(), g, a) for a in sides]).amin(0)
    drop = g - low
    n = torch.where(drop > 1.0, drop.floor(), 0.0).long().reshape(-1)
    par = torch.repeat_interleave(torch.arange(w * h, device="cuda"), n)
    k = torch.arange(par.numel(), device="cuda") - torch.repeat_interleave(n.cumsum(0) - n, n)
    zz = (g.reshape(-1)[par] - (k.float() + 0.5)).double()
    o = [(zz - a.reshape(-1)[par].double().clamp_min(-1e30)).clamp_min(0.0) for a in sides]
    two_pi = 2.0 * math.pi

    def angle(y, x):
        a = torch.atan2(y, x)
        return torch.where(a < 0, a + two_pi, a)
    # a side off the grid counts as 1e30 m below: the 32-bit differences keep only it
    wall = angle((o[0].float() - o[1].float()).double(), (o[2].float() - o[3].float()).double())
    gd = g
    x, y = torch.arange(w, device="cuda"), torch.arange(h, device="cuda")
    xr, xl, yd, yu = (x + 1).clamp_max(w - 1), (x - 1).clamp_min(0), (y + 1).clamp_max(h - 1), (y - 1).clamp_min(0)
    dx = (gd[:, xr] - gd[:, xl]).double() / (xr - xl).double()
    dy = (gd[yd] - gd[yu]).double() / (yd - yu).double()[:, None]
    slope = torch.atan2((dx * dx + dy * dy).sqrt(), torch.ones_like(dx))
    cap, n = 2 * w * h, w * h + par.numel()

    def room(*parts):
        a = torch.zeros(cap, dtype=torch.float64, device="cuda")
        a[:sum(p.numel() for p in parts)] = torch.cat([p.reshape(-1).double() for p in parts])
        return a
    return {"pixel_parent": None, "wall_z": room(zz), "slopes": room(slope, torch.full((n - w * h,), math.pi / 2,
                                                                                    device="cuda")),
            "aspects": room(angle(-dx, dy), wall), "num_total": None}
