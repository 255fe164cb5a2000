"""What a program does with the erosion stage, as cases that can be timed and compared.

A case names a call (`kind`), a grid and the options of that call. `prepare` makes the world a program
has in hand, from the seed alone; `run` makes the call through the package's public entry points.
Host calls take and return numpy arrays, as the reference's hosts hold their fields; the `resident`
kind keeps its world on the device, as a program that generates or renders there does.

Worlds have the shape of the workloads the benchmark and the tests use: fBm heights (spectral exponent
2) over [-10000, 6000] m, uplift along great-circle ridges, a lognormal rock factor with sigma 0.5, rain
and cover as smooth fields. They are made on the GPU, in torch, so that a new world is quick.
"""
import ctypes as C
import math

import numpy as np
import torch

from cartogenesis_gb300 import BeltErosion, BeltWindow, ErosionConfig, ErosionStage, GpuErosionAccelerator, abi
from cartogenesis_gb300.api import FlowRouting, Isostasy, SeaLevelStage, StageRounds, ThermalLimits, default_context

EARTH_KM = 40075.0
RELIEF_M = 16000.0   # 6000 m of land over 10000 m of ocean


def listed():
    return [
        # The reference's own device seam, ErosionAccelerator.erode, on its smallest usual world: a
        # preview's 24 sweeps, where the call's latency and launches count.
        {"name": "sweeps_512x256", "kind": "sweeps", "width": 512, "height": 256, "km": EARTH_KM},
        # The same seam on the largest world the reference's published table has (2048 rows, 192 sweeps).
        {"name": "sweeps_4096x2048", "kind": "sweeps", "width": 4096, "height": 2048, "km": EARTH_KM},
        # SeaLevelStage.apply's cut with its enclosure rule, as a map's shoreline is drawn after erosion.
        {"name": "sea_cut_1024x512", "kind": "sea_cut", "width": 1024, "height": 512, "km": EARTH_KM, "sea": 0.71},
        # The routing RiverStage and GlaciationStage run on their cut: fill, directions, area, order.
        {"name": "route_cut_2048x1024", "kind": "route_cut", "width": 2048, "height": 1024, "km": EARTH_KM, "sea": 0.70,
         "seed": 1},
        # Isostasy.Flexure on its own: the plate's bend under one load.
        {"name": "flexure_2048x1024", "kind": "flexure", "width": 2048, "height": 1024, "km": EARTH_KM},
        # BeltErosion.replay over a 40 Myr exposure window, about a hundred short rounds.
        {"name": "belts_1024x512", "kind": "belts", "width": 1024, "height": 512, "km": EARTH_KM, "sea": 0.71,
         "weather": False, "myr": 40.0, "seed": 3},
        # A batch of planets of uneven size in one call, as a gallery of seeds is generated.
        {"name": "batch_12", "kind": "batch", "worlds": 12, "least": 256, "most": 1024, "sea": 0.70, "profile": 0,
         "rounds": 12, "seed": 1},
        # The plain stage on a preview's world with every output read back.
        {"name": "plain_512x256", "kind": "stage", "width": 512, "height": 256, "km": EARTH_KM, "sea": 0.70,
         "profile": 0, "rounds": 12, "weather": False, "outputs": True, "seed": 1},
        # The plain stage at the finest grid, the world resident on the device: the benchmark's workload.
        {"name": "plain_8192x4096", "kind": "resident", "width": 8192, "height": 4096, "km": EARTH_KM, "sea": 0.70,
         "profile": 0, "rounds": 12, "weather": False, "seed": 1},
        # The outlet notch on a 1024-row world that has its weather.
        {"name": "notch_2048x1024", "kind": "stage", "width": 2048, "height": 1024, "km": EARTH_KM, "sea": 0.71,
         "profile": 1, "rounds": 12, "weather": True, "outputs": False, "seed": 7},
        # The reference's default configuration on its 512-row world: belts, weather solved twice,
        # deposition and the plate's flexure, round by round on a resident world.
        {"name": "default_1024x512", "kind": "default", "width": 1024, "height": 512, "km": EARTH_KM, "sea": 0.71,
         "rounds": 12, "myr": 40.0, "seed": 3},
        # Deposition and flexure at the finest grid, in a draft's few rounds.
        {"name": "draft_8192x4096", "kind": "resident", "width": 8192, "height": 4096, "km": EARTH_KM, "sea": 0.70,
         "profile": 3, "rounds": 4, "weather": False, "seed": 1},
    ]


def draw(rng):
    def grid(least, most):
        w = 2 ** rng.randint(int(math.log2(least)), int(math.log2(most)))
        return w, (w if w <= 2048 and rng.random() < 0.25 else w // 2)

    kind = rng.choice(["sweeps", "sea_cut", "route_cut", "flexure", "belts", "batch", "stage", "stage", "resident",
                       "resident", "default"])
    case = {"kind": kind, "km": EARTH_KM * math.exp(rng.uniform(math.log(0.5), math.log(2.0))),
            "sea": rng.uniform(0.55, 0.80), "seed": rng.randint(1, 10**6)}
    if kind in ("sweeps", "flexure"):
        case["width"], case["height"] = grid(256, 8192)
    elif kind in ("sea_cut", "route_cut"):
        case["width"], case["height"] = grid(256, 2048 if kind == "sea_cut" else 4096)
    elif kind == "belts":
        case["width"], case["height"] = grid(256, 2048)
        case.update(weather=rng.random() < 0.5, myr=rng.uniform(10.0, 40.0))
    elif kind == "batch":
        case.update(worlds=rng.randint(1, 16), least=256, most=rng.choice([256, 512, 1024]), rounds=rng.randint(1, 12),
                    profile=rng.choice([0, 0, 1]))
    elif kind == "default":
        case["width"], case["height"] = grid(256, 1024)
        case.update(rounds=rng.randint(2, 12), myr=rng.uniform(10.0, 40.0))
    else:
        case["profile"] = rng.choice([0, 0, 1, 2, 3])
        w, h = case["width"], case["height"] = grid(256, 8192 if kind == "resident" else 2048)
        # Deposition at the finest grids runs in a draft's few rounds.
        most = 12 if case["profile"] < 2 else max(1, min(12, 10**8 // (w * h)))
        case.update(rounds=rng.randint(1, most), weather=rng.random() < 0.5)
        if kind == "stage":
            case["outputs"] = rng.random() < 0.5
    return case


# ---- worlds

def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _fbm(W, H, beta, seed, salt):
    """Zero-mean, unit-variance fBm, periodic in x, cells 2:1 on the ground as the tests' worlds have them."""
    g = _gen(seed, salt)
    ky = torch.fft.fftfreq(H, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(W, device="cuda", dtype=torch.float64)[None, :] * (W / H) * 0.5
    k = (kx * kx + ky * ky).sqrt()
    k[0, 0] = 1.0
    amp = k ** (-beta / 2.0)
    amp[0, 0] = 0.0
    amp = amp * torch.randn(amp.shape, generator=g, device="cuda", dtype=torch.float64)
    phase = 2.0 * math.pi * torch.rand(amp.shape, generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.irfft2(torch.polar(amp, phase), s=(H, W))
    f -= f.mean()
    return f / f.std()


def _heights(W, H, seed):
    f = _fbm(W, H, 2.0, seed, 1)
    return ((f - f.min()) / (f.max() - f.min())).float()


def _rock(W, H, seed):
    return (0.5 * _fbm(W, H, 3.0, seed, 2)).exp().float()


def _weather(W, H, seed):
    """Rain in mm (lognormal about 800) and a cover in [0, 1]."""
    z = _fbm(W, H, 3.0, seed, 3)
    return (800.0 * (0.7 * z).exp()).float(), (0.5 + 0.5 * torch.tanh(z)).float()


def _load(W, H, seed):
    """A column change of a few hundred metres of crust, in pascals."""
    return (300.0 * 2835.0 * 9.81 * _fbm(W, H, 2.5, seed, 5)).float()


def _sphere(W, H):
    lon = (torch.arange(W, device="cuda", dtype=torch.float64) + 0.5) / W * (2.0 * math.pi)
    lat = math.pi / 2 - (torch.arange(H, device="cuda", dtype=torch.float64) + 0.5) / H * math.pi
    c = lat.cos()[:, None]
    return c * lon.cos()[None, :], c * lon.sin()[None, :], lat.sin()[:, None].expand(H, W)


def _ridges(W, H, seed, km):
    """Uplift in mm a year: 15 Gaussian ridges of 50-4000 m/Myr along great-circle arcs."""
    rng = np.random.Generator(np.random.PCG64([int(seed) & 0xFFFFFFFF, 3000]))
    x, y, z = _sphere(W, H)
    up = torch.zeros(H, W, device="cuda", dtype=torch.float64)
    for _ in range(15):
        a, t = rng.standard_normal(3), rng.standard_normal(3)
        a /= np.linalg.norm(a)
        t -= t.dot(a) * a
        t /= np.linalg.norm(t)
        n = np.cross(a, t)
        length, width, rate = rng.uniform(0.05, 0.35) * math.pi, rng.uniform(100.0, 300.0), rng.uniform(0.05, 4.0)

        def dot(v):
            return x * float(v[0]) + y * float(v[1]) + z * float(v[2])

        off = torch.asin(dot(n).clamp(-1.0, 1.0)) * (km / (2.0 * math.pi))
        along = torch.atan2(dot(t), dot(a))
        ridge = rate * torch.exp(-0.5 * (off / (0.5 * width)) ** 2)
        up = torch.maximum(up, torch.where((along >= 0.0) & (along <= length), ridge, 0.0))
    return up.float()


def _bands(W, H, seed, km):
    """Uplift in mm a year in 100-300 km bands along the active boundaries of 12 plates."""
    rng = np.random.Generator(np.random.PCG64([int(seed) & 0xFFFFFFFF, 2000]))
    centres = rng.standard_normal((12, 3))
    centres /= np.linalg.norm(centres, axis=1, keepdims=True)
    x, y, z = _sphere(W, H)
    ang = torch.stack([torch.acos((x * float(c[0]) + y * float(c[1]) + z * float(c[2])).clamp(-1.0, 1.0))
                       for c in centres])
    near, which = torch.topk(ang, 2, dim=0, largest=False)
    gap = (near[1] - near[0]) * (km / (2.0 * math.pi)) * 0.5

    def per_plate(v):
        return torch.as_tensor(v, device="cuda")[which[0]]

    band, peak = per_plate(rng.uniform(100.0, 300.0, 12)), per_plate(rng.uniform(0.5, 3.0, 12))
    active = per_plate(rng.uniform(size=12) < 0.6)
    return torch.where((gap < band) & active, peak * torch.cos(0.5 * math.pi * gap / band) ** 2, 0.0).float()


def _window(W, H, seed, km, myr):
    """The belts' exposure window under the bands: thickening, wear and onset, and the bands' uplift."""
    up = _bands(W, H, seed, km)
    belt = up > 0.05
    wear = 0.2 + 0.3 * (0.5 + 0.5 * torch.tanh(_fbm(W, H, 3.0, seed, 11)))
    start = 0.4 + 0.6 * (0.5 + 0.5 * torch.tanh(_fbm(W, H, 3.0, seed, 12)))
    tect = torch.where(belt, myr * up, 0.0)
    onset = torch.where(belt, myr * start, -1.0)
    return [_host(v.float()) for v in (tect, tect * wear, onset)], up


def _host(t):
    return t.cpu().numpy()


def _cut(h, sea):
    """A cut to route on: the highest cells are land, `sea` of all cells is not; elevations relative to the shore."""
    H, W = h.shape
    v, at = h.reshape(-1).sort()
    first = int(sea * W * H)
    land = torch.zeros(W * H, device="cuda", dtype=torch.uint8)
    land[at[first:]] = 1
    d = h - v[first - 1]
    rel = torch.where(d > 0, d / (6000.0 / RELIEF_M), d / (10000.0 / RELIEF_M)).clamp(-1.0, 1.0)
    return _host(land.reshape(H, W)), _host(rel.float()), W * H - first


# ---- the calls

def _passes(case):
    """ErosionStage.sweepsFor: 1875 km of debris travel in cells."""
    return int(np.rint(np.float32(1875.0 * case["width"] / case["km"])))


def _limits(case):
    """ErosionStage.thermalLimits: 60 m/km per neighbour kind, in field units."""
    per_km = 60.0 / RELIEF_M
    cw, ch = case["km"] / case["width"], 0.5 * case["km"] / case["height"]
    return [float(np.float32(per_km * d)) for d in (cw, ch, math.hypot(cw, ch))]


def _batch_shapes(case, seed):
    """Planets of 0.25-2 Earth radii: 2R x R grids, R the power of two nearest 1024 r, within the case's range."""
    rng = np.random.Generator(np.random.PCG64([case["seed"], 4000]))
    for i in range(case["worlds"]):
        r = float(rng.uniform(0.25, 2.0))
        rows = int(min(max(2 ** int(np.rint(np.log2(1024.0 * r))), case["least"]), case["most"]))
        yield 2 * rows, rows, EARTH_KM * r, seed * 1000 + i


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "batch":
        s["worlds"] = []
        for W, H, km, wseed in _batch_shapes(case, seed):
            cfg = ErosionConfig(W, H, wseed, sea_level=case["sea"], world_width_km=km, profile=case["profile"],
                                hydraulic_rounds=case["rounds"])
            s["worlds"].append((cfg, _host(_heights(W, H, wseed)), _host(_ridges(W, H, wseed, km)),
                                _host(_rock(W, H, wseed))))
        return s
    W, H, km = case["width"], case["height"], case["km"]
    if kind == "sweeps":
        s.update(h=_host(_heights(W, H, seed)), limits=ThermalLimits(*_limits(case)), passes=_passes(case))
        return s
    s["cfg"] = cfg = ErosionConfig(W, H, case.get("seed", 1), world_width_km=km, sea_level=case.get("sea", 0.71),
                                   hydraulic_rounds=case.get("rounds", 12), profile=case.get("profile", 0))
    if kind == "flexure":
        s["load"] = _host(_load(W, H, seed))
        s["flexure"] = Isostasy.Flexure(cfg)
        return s
    h = _heights(W, H, seed)
    if kind == "sea_cut":
        s["h"] = _host(h)
    elif kind == "route_cut":
        s["land"], s["rel"], s["cells"] = _cut(h, case["sea"])
        s["weights"] = _host(_weather(W, H, seed)[0])
    else:
        rock = _rock(W, H, seed)
        rain, veg = _weather(W, H, seed) if kind == "default" or case["weather"] else (None, None)
        if kind in ("belts", "default"):
            window, up = _window(W, H, seed, km, case["myr"])
            s["window"] = BeltWindow(*window, case["myr"])
        else:
            up = _ridges(W, H, seed, km)
        fields = {"h": h, "up": up, "rock": rock, "rain": rain, "veg": veg}
        if kind == "resident":
            s.update(fields, out=torch.empty_like(h), land=C.c_int32())
            s["inputs"] = abi.Inputs(*[None if t is None else t.data_ptr() for t in fields.values()])
        else:
            s.update({k: None if t is None else _host(t) for k, t in fields.items()})
        if kind == "default":
            cfg.params.profile, cfg.params.climate_feed = 3, 1
            later = _weather(W, H, seed + 1)   # the weather the climate solves halfway
            s["rain2"], s["veg2"] = _host(later[0]), _host(later[1])
    torch.cuda.synchronize()
    return s


def _books(r):
    return [r.rounds, r.belt_cells, r.uplifted_cubic_meters, r.cut_cubic_meters, r.exported_to_sea_cubic_meters,
            r.exported_to_land_cubic_meters, r.shed_beside_cubic_meters, r.eroded_meters]


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "sweeps":
        return GpuErosionAccelerator().erode(case["width"], case["height"], s["h"], s["limits"], s["passes"], 0.25)
    if kind == "batch":
        return ErosionStage.apply_batch(s["worlds"])
    cfg = s["cfg"]
    if kind == "sea_cut":
        return list(SeaLevelStage.drained_cut(cfg, s["h"]))
    if kind == "route_cut":
        return list(FlowRouting.route_cut(cfg, s["land"], s["rel"], s["cells"], s["weights"]))
    if kind == "flexure":
        return s["flexure"].deflection_metres(s["load"])
    if kind == "belts":
        h = s["h"].copy()   # replayed in place
        r = BeltErosion.replay(cfg, h, s["window"], s["up"], s["rain"], s["veg"], s["rock"])
        return [h] + _books(r)
    if kind == "stage":
        want = ErosionStage.WANT if case["outputs"] else ("receivers",)
        r = ErosionStage.apply(cfg, s["h"], s["up"], s["rock"], s["rain"], s["veg"], want=want)
        out = [r.height] + [getattr(r, k) for k in want] + [r.basins["count"]]
        if case["outputs"]:   # a world's basins, in arrays of one length for any world
            for k in ("spill", "entry", "level", "floor", "cells"):
                b = r.basins[k]
                out.append(np.zeros(r.height.size // 8, b.dtype))
                out[-1][:b.size] = b[:r.height.size // 8]
        return out
    if kind == "resident":
        ctx = default_context()
        ctx.check(ctx.lib.cg_erode_stage_dev(ctx.handle, C.byref(cfg.params), C.byref(s["inputs"]),
                                             s["out"].data_ptr(), None, C.byref(s["land"])))
        return [s["out"], s["land"].value]
    # The reference's default: the swept world, the belts' replay, and the rounds with the weather the
    # caller solves before round 0 and halfway.
    stage = StageRounds(cfg, s["h"], s["up"], s["rock"])
    swept = stage.height()
    replay = stage.replay_belts(s["window"], s["rain"], s["veg"])
    rounds = case["rounds"]
    stage.rounds(rounds // 2, s["rain"], s["veg"])
    half = stage.height()
    stage.rounds(rounds, s["rain2"], s["veg2"])
    end = stage.finish()
    return [swept, half, end.height, end.receivers] + _books(replay)


# ---- what a pass cannot do without

# Floating operations a cell takes in one sweep (8 neighbours, a give rate and a move) and in the rest of
# a round (the facets' slopes and draw, the incision's update).
SWEEP_FLOPS, ROUND_FLOPS = 90.0, 120.0


def _stage_flops(case, W, H, km):
    n, rounds = float(W) * H, case["rounds"]
    sweeps = 1875.0 * W / km
    flops = n * (SWEEP_FLOPS * (sweeps + rounds * max(1, sweeps // rounds)) + ROUND_FLOPS * rounds)
    if case.get("profile", 3 if case["kind"] == "default" else 0) >= 3:
        flops += rounds * 20.0 * n * math.log2(2.0 * W * H)
    return flops


def work(case):
    """Each input read once and each output written once; the operations of the sweeps, the facets and the
    flexure's transform."""
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for W, H, km, _ in _batch_shapes(case, 0):
            b += 16.0 * W * H
            f += _stage_flops(case, W, H, km)
        return {"bytes": b, "flops": f}
    W, H, km = case["width"], case["height"], case["km"]
    n = float(W) * H
    if kind == "sweeps":
        return {"bytes": 8.0 * n, "flops": SWEEP_FLOPS * n * _passes(case)}
    if kind == "sea_cut":
        return {"bytes": 9.0 * n, "flops": 4.0 * n}
    if kind == "route_cut":
        return {"bytes": (9.0 + 12.0 + 4.0 * (1.0 - case["sea"])) * n, "flops": 100.0 * (1.0 - case["sea"]) * n}
    if kind == "flexure":
        return {"bytes": 8.0 * n, "flops": 20.0 * n * math.log2(2.0 * W * H)}
    weather = 8.0 if kind == "default" or case["weather"] else 0.0
    if kind == "belts":
        return {"bytes": (24.0 + weather + 8.0) * n, "flops": 100.0 * n}
    if kind == "stage":
        return {"bytes": (16.0 + weather + (29.0 if case["outputs"] else 4.0)) * n, "flops": _stage_flops(case, W, H, km)}
    if kind == "resident":
        return {"bytes": (16.0 + weather) * n, "flops": _stage_flops(case, W, H, km)}
    return {"bytes": (24.0 + 2 * weather + 20.0) * n, "flops": _stage_flops(case, W, H, km)}


# ---- the same in 64 bits

def _sweeps64(case, h):
    """Musgrave's sweeps in double: x wraps, y stops at the poles."""
    ew, ns, dg = _limits(case)
    steps = [(1, 0, ew), (-1, 0, ew), (0, 1, ns), (0, -1, ns), (1, 1, dg), (1, -1, dg), (-1, 1, dg), (-1, -1, dg)]
    rate, settled = 0.25, ew * 1e-3
    H = h.shape[0]
    row = torch.arange(H, device="cuda")[:, None]

    def nb(t, dx, dy):
        return torch.roll(t, (-dy, -dx), (0, 1))

    for _ in range(_passes(case)):
        excess, steepest = torch.zeros_like(h), torch.zeros_like(h)
        for dx, dy, lim in steps:
            drop = torch.where((row + dy >= 0) & (row + dy < H), h - nb(h, dx, dy), 0.0)
            steepest = torch.maximum(steepest, drop)
            excess += torch.where(drop > lim, drop - lim, 0.0)
        give = torch.where(excess > settled, torch.minimum(rate * excess, 0.5 * steepest) / excess, 0.0)
        move = torch.zeros_like(h)
        for dx, dy, lim in steps:
            rise = torch.where((row + dy >= 0) & (row + dy < H), nb(h, dx, dy) - h, 0.0)
            move += torch.where(rise > lim, (rise - lim) * nb(give, dx, dy), 0.0)
            move -= torch.where(-rise > lim, (-rise - lim) * give, 0.0)
        h = h + move
    return h


def _flexure64(case, load):
    """The plate's response to the load less its mean, the map mirrored about each pole."""
    H, W = load.shape
    load = load - load.mean()
    f = torch.fft.fft2(torch.cat([load, load.flip(0)]))
    mpk = 1000.0
    rigidity = 70.0e9 * (30.0 * mpk) ** 3 / (12.0 * (1.0 - 0.0625))
    ka = torch.fft.fftfreq(W, 1.0 / W, device="cuda", dtype=torch.float64) * (2.0 * math.pi / (case["km"] * mpk))
    kd = torch.fft.fftfreq(2 * H, 0.5 / H, device="cuda", dtype=torch.float64) * (2.0 * math.pi / (case["km"] * mpk))
    k2 = ka[None, :] ** 2 + kd[:, None] ** 2
    f = f / (3300.0 * float(np.float32(9.81)) + rigidity * k2 * k2)
    f[0, 0] = 0.0
    return torch.fft.ifft2(f).real[:H]


def exact(case, seed):
    """Values for the two calls that are plain arithmetic on their inputs. The others decide in float (which
    cells are land, drain, pond or fill), so their results have no value in 64 bits to be near to."""
    if case["kind"] == "sweeps" and case["width"] * case["height"] * _passes(case) < 4e9:
        return _host(_sweeps64(case, _heights(case["width"], case["height"], seed).double()))
    if case["kind"] == "flexure":
        return _host(_flexure64(case, _load(case["width"], case["height"], seed).double()))
    return None
