"""What this engine is timed on: its public calls, at the sizes they are used at.

A case is a dict of plain values.  `kind` names the call:

    sector   Engine.compute_sector: one sector in place on the caller's surfaces, the
             call the reference's per-sector loop makes (compute.rs:181-203); `rings` is
             "none", "reference" (the reserved layout) or "compact" (the record stream,
             tvs_compute_sectors_rings)
    records  tvs_compute_sectors_rings: the ring records of several sectors
    tvs      Engine.run: a whole total viewshed of 180 sectors, surfaces and heatmap
             total; with `upload` the elevations are replaced first, as a program does
             that walks over many DEMs of one size
    batch    Batch.run of tiles of uneven size

Terrain is made on the GPU from the seed: `fbm` (spectral fractional Brownian surface)
or `ridged` (a ridged multifractal), `sea` of its rows flat at 0 m, and whole metres
where `metres` is set, as in the 16-bit files the reference reads (main.rs:51-56).
"""

import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

SECTORS = 180
OBSERVER = 1.65


def _package():
    name = "total_viewsheds_b200"
    if name not in sys.modules:
        pkg = Path.cwd() / "total-viewsheds_b200"
        spec = importlib.util.spec_from_file_location(name, pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _case(kind, width, precision, **kw):
    c = dict(kind=kind, width=width, height=width, precision=precision, scale=30.0, los=width // 3,
             terrain="fbm", hurst=0.8, top=1500.0, sea=0.0, metres=True, rings_per_km=5.0)
    c.update(kw)
    return c


def listed():
    cases = [
        # One sector of the smallest region, as an embedding loop calls it: launches, copies
        # and waits are what it costs.
        _case("sector", 301, "exact32", name="sector_301", angle=23, rings="none"),
        # The same loop with its ring records in the reference's own layout.
        _case("sector", 601, "exact32", name="sector_601_rings", angle=107, rings="reference",
              rings_per_km=20.0),
        # The smallest whole region (the reference's CPU-sized run).
        _case("tvs", 301, "exact32", name="tvs_301", upload=False),
        # A 90 m region with sea, one after another of the same size: upload, 180 sectors,
        # read back, in the reference's arithmetic.
        _case("tvs", 1201, "exact32", name="tvs_1201_upload", scale=90.0, hurst=0.75, top=2500.0,
              sea=0.15, upload=True),
        # The same region in double precision throughout.
        _case("tvs", 1201, "fp64", name="tvs_1201_fp64", scale=90.0, hurst=0.75, top=2500.0,
              sea=0.15, upload=False),
        # A cut-out of odd, unequal sides.
        _case("tvs", 1543, "mixed64", name="tvs_1543x1027", height=1027, los=341, hurst=0.7,
              top=3000.0, upload=False),
        # One 1-arc-second tile, the headline workload: new elevations in pinned memory, the
        # whole viewshed with FP64 decisions, surfaces back on the host.
        _case("tvs", 3601, "mixed64", name="tvs_3601_mixed64", los=1200, terrain="ridged",
              top=4500.0, sea=0.1, metres=False, upload=True),
        # The same tile in the reference's f32 arithmetic.
        _case("tvs", 3601, "exact32", name="tvs_3601_exact32", los=1200, terrain="ridged",
              top=4500.0, sea=0.1, metres=False, upload=False),
        # The same tile in the plain reciprocal form.
        _case("tvs", 3601, "fp32", name="tvs_3601_fp32", los=1200, terrain="ridged", top=4500.0,
              sea=0.1, metres=False, upload=False),
        # Four tiles as one region with a 72 km line of sight: the largest DEM in use.
        _case("tvs", 7201, "mixed64", name="tvs_7201_mixed64", los=2400, top=6000.0, upload=False),
        # Every band's ring record, six sectors per call, as a program takes them that draws
        # viewsheds from them.
        _case("records", 1201, "mixed64", name="records_1201x6", scale=90.0, hurst=0.75, top=2500.0,
              sea=0.15, angle=42, sectors=6),
        # A dozen tiles of uneven size in one run.
        _case("batch", 1601, "mixed64", name="batch_12", height=1601, smallest=257, tiles=12,
              hurst=0.75, top=3000.0, shapes=1),
    ]
    return cases


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sector", "records", "tvs", "tvs", "tvs", "batch"])
    precision = rng.choice(["exact32", "mixed64", "mixed64", "fp32", "fp64"])
    look = dict(scale=rng.choice([30.0, 90.0]), metres=rng.random() < 0.6,
                terrain=rng.choice(["fbm", "ridged"]), hurst=round(rng.uniform(0.6, 0.9), 2),
                top=float(rng.randrange(500, 6000)), sea=rng.choice([0.0, 0.0, 0.1, 0.15]))
    if kind == "batch":
        largest = _log_uniform(rng, 400, 1601)
        return _case("batch", largest, precision, height=largest, smallest=257,
                     tiles=rng.randrange(2, 17), shapes=rng.randrange(1, 1000), **look)
    top_width = {"sector": 2401, "records": 1201, "tvs": 3601 if precision == "fp64" else 4801}[kind]
    width = _log_uniform(rng, 257, top_width)
    height = width
    if rng.random() < 0.35:
        height = max(257, int(width * rng.uniform(0.55, 1.0)))
    los = int(min(width, height) * rng.uniform(0.30, 0.36))
    c = _case(kind, width, precision, height=height, los=los, **look)
    if kind == "sector":
        c["angle"] = rng.randrange(SECTORS)
        reserved = "reference" if width <= 801 else "compact"
        c["rings"] = rng.choice(["none", "none", reserved, "compact"])
        if c["rings"] == "reference":  # slots for every step of a band
            c["rings_per_km"] = 25.0 if c["scale"] == 30.0 else 8.0
    elif kind == "records":
        c["sectors"] = 1 if precision == "fp64" else rng.randrange(1, 9)
        c["angle"] = rng.randrange(SECTORS - c["sectors"])
    else:
        c["upload"] = rng.random() < 0.5
        if rng.random() < 0.2:  # one rank's rows of a region that several share
            c["shard"] = rng.randrange(4)
    return c


# ---- terrain ----------------------------------------------------------------

def _fbm(h, w, hurst, gen):
    """Spectral synthesis: white noise under an amplitude of k^-(hurst + 1)."""
    n = 1 << (max(h, w) - 1).bit_length()
    noise = torch.randn((n, n), generator=gen, device="cuda")
    f = torch.fft.rfft2(noise)
    ky = torch.fft.fftfreq(n, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(n, device="cuda")[None, :]
    k2 = ky * ky + kx * kx
    k2[0, 0] = 1.0
    f = f * k2.pow(-(hurst + 1.0) / 2.0)
    f[0, 0] = 0.0
    return torch.fft.irfft2(f, s=(n, n))[:h, :w]


def _ridged(h, w, octaves, gen):
    """Musgrave's ridged multifractal over bicubic lattice noise."""
    total = torch.zeros((h, w), device="cuda")
    weight = torch.ones((h, w), device="cuda")
    period = max(h, w) / 4.0
    for o in range(octaves):
        p = max(period / 2.0 ** o, 1.5)
        grid = torch.rand((1, 1, int(h / p) + 2, int(w / p) + 2), generator=gen, device="cuda")
        noise = torch.nn.functional.interpolate(2 * grid - 1, size=(h, w), mode="bicubic",
                                                align_corners=True)[0, 0]
        signal = (1.0 - noise.abs()) ** 2 * weight
        weight = (2.0 * signal).clamp(0.0, 1.0)
        total += signal * 0.5 ** o
    return total


def _heights(case, height, width, seed):
    """f32 [height, width] in pinned host memory."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    z = (_ridged(height, width, 10, gen) if case["terrain"] == "ridged"
         else _fbm(height, width, case["hurst"], gen))
    lo, hi = z.min(), z.max()
    z = (z - lo) * (case["top"] / (hi - lo))
    if case["metres"]:
        z = z.round()
    z[:int(round(case["sea"] * height))] = 0.0
    host = torch.empty((height, width), dtype=torch.float32, pin_memory=True)
    host.copy_(z)
    return host


def _tile_sides(case):
    """(height, width) of a batch's tiles, from the case alone."""
    r = np.random.default_rng(case["shapes"])
    return [(int(a), int(b)) for a, b in
            r.integers(case["smallest"], case["width"] + 1, (case["tiles"], 2))]


# ---- the calls ----------------------------------------------------------------

def _engine_args(case):
    return dict(observer_height=OBSERVER, precision=case["precision"],
                rings_per_km=case["rings_per_km"])


def _rows(case, tvs_height):
    if "shard" not in case:
        return None
    k = case["shard"]
    return k * tvs_height // 4, (k + 1) * tvs_height // 4


def prepare(case, seed):
    pkg = _package()
    if case["kind"] == "batch":
        sides = _tile_sides(case)
        dems = [(_heights(case, h, w, seed * 64 + i).numpy(), case["scale"],
                 int(min(h, w) // 3 * case["scale"])) for i, (h, w) in enumerate(sides)]
        return {"case": case, "batch": pkg.Batch(dems, **_engine_args(case))}
    z = _heights(case, case["height"], case["width"], seed)
    los = int(case["los"] * case["scale"])
    g = pkg.compute_geometry(pkg.make_params(case["width"], case["scale"], los,
                                             height=case["height"]))
    eng = pkg.Engine(z.numpy(), case["width"], case["scale"], los, height=case["height"],
                     rows=_rows(case, g.tvs_height), **_engine_args(case))
    state = {"case": case, "engine": eng, "pinned": z, "z": z.numpy()}
    if case["kind"] in ("sector", "records"):
        state["surfaces"] = np.zeros(eng.count, np.float32)
        if case.get("rings") == "reference":
            state["slots"] = np.zeros(eng.geometry.ring_slots_per_sector, np.uint32)
        elif case["kind"] == "records" or case["rings"] == "compact":
            # the program's own buffers, kept for every call: an offset per band, and room
            # for twice the ids that rough terrain gives
            bands = eng.geometry.total_bands * case.get("sectors", 1)
            state["offsets"] = _pinned(bands + 1, torch.int64).view(np.uint64)
            state["ids"] = _pinned(bands * (12 + _steps(case["los"]) // 6), torch.int32).view(np.uint32)
    return state


def _pinned(n, dtype):
    return torch.zeros(n, dtype=dtype, pin_memory=True).numpy()


def _records(state, first, sectors, surfaces):
    """The compact record stream through the C ABI, into the program's buffers."""
    eng, lib = state["engine"], _package().lib()
    total = ctypes.c_uint64()

    def ptr(a):
        return a.ctypes.data_as(ctypes.c_void_p)

    rc = lib.tvs_compute_sectors_rings(eng.ctx, first, sectors, ptr(surfaces), ctypes.byref(total),
                                       None)
    if rc == 0 and total.value <= state["ids"].size:
        rc = lib.tvs_read_ring_records(eng.ctx, ptr(state["offsets"]), ptr(state["ids"]))
    if rc or total.value > state["ids"].size:
        raise RuntimeError(f"ring records: status {rc}, {total.value} ids")
    return surfaces, state["offsets"], state["ids"]


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.run()
        b.finish()
        return [b.read(i) for i in range(len(b))]
    eng = state["engine"]
    if case["kind"] == "tvs":
        if case["upload"]:
            eng.set_elevations(state["z"])
        cumulative, total, _ = eng.run()
        return cumulative, total
    surfaces = state["surfaces"].copy()
    if case["kind"] == "records":
        return _records(state, case["angle"], case["sectors"], surfaces)
    if case["rings"] == "compact":
        return _records(state, case["angle"], 1, surfaces)
    if case["rings"] == "reference":
        eng.compute_sector(case["angle"], surfaces, state["slots"])
        return surfaces, state["slots"]
    eng.compute_sector(case["angle"], surfaces)
    return (surfaces,)


# ---- what a pass cannot do without ----------------------------------------------

def _tiles(case):
    """(height, width, line of sight in cells) of each DEM of a case."""
    if case["kind"] == "batch":
        return [(h, w, min(h, w) // 3) for h, w in _tile_sides(case)]
    return [(case["height"], case["width"], case["los"])]


def _steps(los):
    """Steps of a band of sight that the shape fills (band_of_sight.rs:95,158)."""
    band = los + 1
    return 2 * band - int(2 * band * math.sqrt(2.0)) // 2


def work(case):
    """The elevations in, the surfaces (and ring slots, or a record of 12 ids per band) out;
    per sample the subtraction, division and curvature of the reference's expression
    (kernel.rs:164-190)."""
    sectors = {"sector": 1, "records": case.get("sectors", 1)}.get(case["kind"], SECTORS)
    nbytes = flops = 0.0
    for h, w, los in _tiles(case):
        points = (h - 2 * los) * (w - 2 * los)
        nbytes += 4.0 * h * w
        if case["kind"] in ("tvs", "batch"):
            nbytes += 8.0 * points
        else:
            nbytes += 8.0 * points
            if case.get("rings") == "reference":
                slots = int(los * case["scale"] / 1000.0 * case["rings_per_km"])
                nbytes += 4.0 * 2 * points * slots
            elif case["kind"] == "records" or case["rings"] == "compact":
                nbytes += 2.0 * points * sectors * (8 + 4 * 12)
        flops += 3.0 * 2 * points * _steps(los) * sectors / (4 if "shard" in case else 1)
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits --------------------------------------------------------

def _keys(d):
    """radsort's order of f32 values (total order, -0 < +0) as int64."""
    bits = d.view(torch.int32).to(torch.int64)
    return torch.where(bits < 0, -bits - 2 ** 31 - 1, bits)


def _projection(xs, ys, angle32):
    """Distances along the axis at `angle32` (axes.rs:154-189), f32."""
    rad = float(angle32) * (math.pi / 180.0)
    right = -ys.double() * math.cos(rad)
    return (xs.double() * math.sin(rad) - right).float()


def _shape(height, width, los, angle):
    """Forward id offsets and f32 distances of a sector's band of sight
    (band_of_sight.rs:95-170) on the central square of the DEM."""
    side = min(height, width)
    x0, y0 = (width - side) // 2, (height - side) // 2
    ids = torch.arange(side * side, device="cuda")
    xs, ys = x0 + ids % side, y0 + ids // side
    dem = ys * width + xs
    sight = np.float32(angle) + np.float32(0.001)
    sector = np.float32(sight + np.float32(90.0))
    samples = int(2 * (los + 1) * math.sqrt(2.0))
    order = torch.sort(_keys(_projection(xs, ys, sector)), stable=True).indices
    lo = side * side // 2 - samples // 2
    window = torch.sort(order[lo:lo + samples]).values  # by id, then stably by sight distance
    along = _projection(xs, ys, sight)
    window = window[torch.sort(_keys(along[window]), stable=True).indices]
    middle = samples // 2
    filled = 2 * (los + 1) - middle
    strip = window[middle:middle + filled + 1]
    offsets = torch.cumsum(dem[strip[:-1]] - dem[strip[1:]], 0)
    distances = (along[side * side // 2] - along[strip[1:]]).abs()
    return offsets.tolist(), distances.tolist()


def _exact_dem(z, los, first, sectors, rows):
    """Cumulative surfaces and heatmap total of sectors first .. in double."""
    h, w = z.shape
    flat = z.to("cuda", torch.float64).reshape(-1)
    th, tw = h - 2 * los, w - 2 * los
    r0, r1 = rows or (0, th)
    base = (los + r0) * w + los

    def grid(off):
        return flat.as_strided((r1 - r0, tw), (w, 1), base + off)

    observer = grid(0) + float(np.float32(OBSERVER))
    cum = torch.zeros((r1 - r0, tw), dtype=torch.float64, device="cuda")
    total = torch.zeros_like(cum)
    for s in range(first, first + sectors):
        offsets, distances = _shape(h, w, los, s)
        for sign in (1, -1):
            top = torch.full_like(cum, -2000.0)
            surface = torch.zeros_like(cum)
            for off, d in zip(offsets, distances):
                angle = (grid(sign * off) - observer).div_(d).sub_(d / 12742000.0)
                surface.add_(angle > top, alpha=d * 0.0174533)
                torch.maximum(top, angle, out=top)
            cum += surface
        total += cum
    out = []
    for v in (cum, total):
        whole = torch.zeros((th, tw), dtype=torch.float64, device="cuda")
        whole[r0:r1] = v
        out.append(whole.reshape(-1).cpu().numpy())
    return out


def exact(case, seed):
    tiles = _tiles(case)
    sectors = {"sector": 1, "records": case.get("sectors", 1)}.get(case["kind"], SECTORS)
    # about 30 us a step of 0.2 M points, and two sorts of the square a sector
    cost = sum(sectors * (_steps(l) * 2 * (3e-5 + 2e-10 * (h - 2 * l) * (w - 2 * l))
                          + 2e-9 * min(h, w) ** 2) for h, w, l in tiles)
    if cost > 12.0:
        return None
    if case["kind"] == "batch":
        return [tuple(_exact_dem(_heights(case, h, w, seed * 64 + i), l, 0, SECTORS, None))
                for i, (h, w, l) in enumerate(tiles)]
    h, w, los = tiles[0]
    z = _heights(case, h, w, seed)
    if case["kind"] == "tvs":
        return tuple(_exact_dem(z, los, 0, SECTORS, _rows(case, h - 2 * los)))
    cumulative = _exact_dem(z, los, case["angle"], sectors, None)[0]
    if case["kind"] == "records" or case["rings"] == "compact":
        return cumulative, None, None
    if case["rings"] == "reference":
        return cumulative, None
    return (cumulative,)
