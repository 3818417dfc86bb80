"""Workloads of the heightfield pipeline through its public entry points, for timing.

Every stage a world generator calls is here, from one 64^2 chunk to a 4096^2 field: the biome layer
chain, the single histogram filter, the multi-biome heights, the hydraulic erosion, the uint16 format
and the splatmap on device buffers, the per-chunk drop-in generator on host arrays, and the batched
pipeline.  Sizes, droplet settings and biome tables are those of the benchmark and the tests.
"""
import ctypes as C
import math

import numpy as np
import torch

import superterrainplus_gb300 as stp

NOISE_OFFSET = 0.2181661565  # the demo's simplex gradient offset; 8 gradients


def listed():
    return [
        # The smallest call in the tests and the smoke run: one low-detail chunk, where launches count.
        dict(name="filter-64", op="filter", side=64, radius=16, biomes=4, cell=32),
        # The production chunk of the benchmark (8 biomes, filter radius 32).
        dict(name="filter-512", op="filter", side=512, radius=32, biomes=8, cell=192),
        # The benchmark's large single field: 32 biomes, radius 64.
        dict(name="filter-4096", op="filter", side=4096, radius=64, biomes=32, cell=512),
        # Heights of the production chunk from its filtered biomes, away from the world's origin.
        dict(name="heights-512", op="heights", side=512, radius=32, biomes=8, cell=192, offset_x=2048, offset_y=-1536),
        # A distant, low-detail chunk eroded with its eight neighbours.
        dict(name="erode-128", op="erode", side=128, neighbours=3, droplets=37684, brush=3, lifetime=30, biomes=8,
             cell=48),
        # The production chunk's erosion: 3x3 chunks of 512^2, 600,000 droplets.
        dict(name="erode-512", op="erode", side=512, neighbours=3, droplets=600000, brush=4, lifetime=50, biomes=8,
             cell=192),
        # The large single field's erosion, its own neighbourhood: 16,000,000 droplets.
        dict(name="erode-4096", op="erode", side=4096, neighbours=1, droplets=16000000, brush=5, lifetime=64,
             biomes=32, cell=512),
        # Fixed-point heights of one eroded 3x3 neighbourhood.
        dict(name="format-1536", op="format", width=1536, height=1536),
        # Biomes of one chunk from the demo's layer chain, as a world pipeline asks for them.
        dict(name="biomemap-512", op="biomemap", width=512, height=512, offset_x=-4096, offset_z=1024),
        # Texture regions of a rendering buffer of 3x3 chunks with the demo's rules.
        dict(name="splat-1536", op="splat", side=512, chunks=3),
        # The per-chunk drop-in on host arrays: biome chunks in, heights out.
        dict(name="generate-512", op="generate", side=512, radius=32, biomes=8, cell=192, offset_x=512, offset_y=0),
        # The benchmark's headline: sixteen production requests in one tuned graph.
        dict(name="batch-16", op="batch", requests=16, side=512, least=512, radius=32, density=2.2888184, brush=4,
             lifetime=50, biomes=8, cell=192),
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def field(side):
        radius = 2 * between(1, min(32, side // 2))
        return dict(radius=radius, biomes=between(1, 32), cell=between(max(16, radius), 512))

    op = rng.choice(["filter", "filter", "heights", "erode", "erode", "format", "biomemap", "splat", "generate",
                     "batch"])
    if op == "filter":
        side = between(24, 2048)
        return dict(op=op, side=side, **field(side))
    if op == "heights":
        side = between(24, 2048)
        return dict(op=op, side=side, offset_x=rng.randint(-4096, 4096), offset_y=rng.randint(-4096, 4096),
                    **field(side))
    if op == "erode":
        neighbours = rng.choice([1, 3, 3])
        side = between(48, 1024 if neighbours == 3 else 3000)
        density = rng.uniform(0.3, 2.3 if neighbours == 3 else 0.95)
        return dict(op=op, side=side, neighbours=neighbours, droplets=int(density * side * side),
                    brush=rng.randint(2, 6), lifetime=rng.randint(20, 64), biomes=between(1, 16),
                    cell=between(32, 512))
    if op == "format":
        return dict(op=op, width=between(32, 6000), height=between(32, 6000))
    if op == "biomemap":
        return dict(op=op, width=between(16, 2560), height=between(16, 2560), offset_x=rng.randint(-10**6, 10**6),
                    offset_z=rng.randint(-10**6, 10**6))
    if op == "splat":
        return dict(op=op, side=between(24, 1024), chunks=rng.choice([1, 2, 3, 5]))
    if op == "generate":
        side = between(24, 1024)
        return dict(op=op, side=side, offset_x=rng.randint(-4096, 4096), offset_y=rng.randint(-4096, 4096),
                    **field(side))
    side = 8 * between(8, 64)
    return dict(op=op, requests=rng.randint(1, 8), side=side, least=8 * between(6, side // 8),
                radius=2 * between(2, 24), density=round(rng.uniform(0.5, 2.3), 3), brush=rng.randint(2, 5),
                lifetime=rng.randint(20, 50), biomes=between(1, 16), cell=between(32, 256))


# ------------------------------------------------------------------- inputs


def biome_table(biomes, seed):
    """Octaves 4-8, scale log-uniform 64-512, amplitude 0.2-1.0."""
    rng = np.random.default_rng(seed)
    t = np.zeros(biomes, stp.BIOME_DTYPE)
    t["Scale"] = np.exp(rng.uniform(np.log(64.0), np.log(512.0), biomes)).astype(np.float32)
    t["Octave"] = rng.integers(4, 9, biomes)
    t["Persistence"] = 0.5
    t["Lacunarity"] = 2.0
    t["Variation"] = rng.uniform(0.2, 1.0, biomes).astype(np.float32)
    return t


def noise_tables(seed):
    """A permutation of 0..255 written twice, and 8 unit gradients."""
    perm = np.random.default_rng(seed + 1).permutation(256).astype(np.uint8)
    angle = NOISE_OFFSET + 2.0 * np.pi * np.arange(8) / 8.0
    return np.concatenate([perm, perm]), np.stack([np.cos(angle), np.sin(angle)], 1).astype(np.float32).ravel()


def simplex(seed):
    return stp.SimplexSetting(seed, 8, NOISE_OFFSET)


def raindrops(count, brush, lifetime, seed):
    return stp.RaindropSetting(
        Seed=seed, RainDropCount=count, Inertia=0.05, SedimentCapacityFactor=4.0, minSedimentCapacity=0.01,
        initWaterVolume=1.0, minWaterVolume=stp.lifetime_min_water_volume(1.0, 0.01, lifetime), Friction=0.1,
        initSpeed=1.0, ErodeSpeed=0.3, DepositSpeed=0.3, EvaporateSpeed=0.01, Gravity=4.0, ErosionBrushRadius=brush)


def biome_map(side, radius, biomes, cell, seed, whole=False):
    """The 3x3 neighbourhood of a `side`^2 chunk at the world's origin as the filter takes it; of the
    neighbours, `whole` or only the border of `radius` that the filter reads."""
    m = torch.zeros((3 * side, 3 * side), dtype=torch.int16, device="cuda")
    w = side + 2 * radius
    if whole:
        stp.DeviceOps().voronoi_biomemap(m, 3 * side, 3 * side, 3 * side, (-side, -side), cell, biomes, seed)
    else:
        stp.DeviceOps().voronoi_biomemap(m[side - radius:, side - radius:], 3 * side, w, w, (-radius, -radius), cell,
                                         biomes, seed)
    return m


def terrain(side, biomes, cell, seed):
    """Multi-biome heights of a `side`^2 map."""
    ops = stp.DeviceOps()
    radius = 2 * min(16, side // 2)
    offsets, bins, status = ops.shf_filter(biome_map(side, radius, biomes, cell, seed), (side, side), (3, 3), radius,
                                           max_items=biomes, bins_capacity=side * side * min(biomes, 8))
    ops.status_check(status)
    h = torch.empty((side, side), device="cuda")
    perm, grad = noise_tables(seed)
    ops.multibiome_heightmap(h, side, offsets, bins, (side, side), (0.0, 0.0), torch.from_numpy(perm).cuda(),
                             torch.from_numpy(grad).cuda(),
                             torch.from_numpy(biome_table(biomes, seed).view(np.float32)).cuda())
    return h


class Buffer:
    """A library-owned device buffer as torch.as_tensor takes it; a tensor made of it keeps `owner`."""

    def __init__(self, owner, address, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(address, False), shape=shape, typestr=typestr, version=3)


def batch_requests(case, seed):
    """`requests` independent neighbourhoods somewhere in the world, their sides spread evenly from
    `least` to `side`."""
    rng = np.random.default_rng(seed)
    out = []
    for n in range(case["requests"]):
        side = case["least"] + 8 * round((case["side"] - case["least"]) / 8 * n / max(case["requests"] - 1, 1))
        out.append(dict(MapSize=side, ChunkX=4 * n, ChunkY=int(rng.integers(-64, 64)),
                        InterpolationRadius=min(case["radius"], side),
                        DropletCount=int(round(case["density"] * side * side)), BrushRadius=case["brush"],
                        Lifetime=case["lifetime"]))
    return out


def prepare(case, seed):
    s = dict(case)
    op = case["op"]
    ops = s["ops"] = stp.DeviceOps()
    if op in ("filter", "heights"):
        side, radius, biomes = case["side"], case["radius"], case["biomes"]
        s["info"] = stp.NNInfo.make((side, side), (3, 3))
        s["map"] = biome_map(side, radius, biomes, case["cell"], seed)
        s["workspace"] = ops.shf_workspace((side, side), (3, 3), radius, biomes)
        s["capacity"] = side * side * min(biomes, 8)
        s["offsets"] = torch.zeros(side * side + 1, dtype=torch.int32, device="cuda")
        s["bins"] = torch.zeros(s["capacity"], dtype=torch.int64, device="cuda")
        s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    if op == "heights":
        filter_chunk(s)
        perm, grad = noise_tables(seed)
        s["perm"], s["grad"] = torch.from_numpy(perm).cuda(), torch.from_numpy(grad).cuda()
        s["table"] = torch.from_numpy(biome_table(biomes, seed).view(np.float32)).cuda()
        s["out"] = torch.empty((side, side), device="cuda")
    elif op == "erode":
        side, nn, count = case["side"], case["neighbours"], case["droplets"]
        s["before"] = terrain(nn * side, case["biomes"], case["cell"], seed)
        s["out"] = torch.empty_like(s["before"])
        s["starts"] = torch.empty(2 * count, device="cuda")
        ops.droplet_starts(s["starts"], count, seed, 0, (side, side), (nn, nn))
        s["setting"] = raindrops(count, case["brush"], case["lifetime"], seed)
        index, weight = stp.erosion_brush(nn * side, case["brush"])
        s["index"], s["weight"] = torch.from_numpy(index).cuda(), torch.from_numpy(weight).cuda()
    elif op == "format":
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["map"] = torch.rand((case["height"], case["width"]), generator=g, device="cuda") * 1.1 - 0.05
        s["out"] = torch.empty((case["height"], case["width"]), dtype=torch.int16, device="cuda")
    elif op == "biomemap":
        s["chain"], s["ids"] = stp.layer_chain_demo()
        s["seed"] = seed
        s["out"] = torch.empty((case["height"], case["width"]), dtype=torch.int16, device="cuda")
    elif op == "splat":
        side, n = case["side"], case["chunks"]
        width = side * n
        pitch = s["pitch"] = (width + 15) // 16 * 16  # texture rows: a multiple of 32 bytes
        altitude, gradient = stp.splat_rules_demo()
        # the demo's rules, written for biomes 0 and 1, repeated for the 8 biomes
        s["generator"] = stp.STPSplatmapGenerator(
            [(2 * k + r.Sample, r.UpperBound, r.RegionIndex) for k in range(4) for r in altitude],
            [(2 * k + r.Sample, r.minGradient, r.maxGradient, r.LowerBound, r.UpperBound, r.RegionIndex)
             for k in range(4) for r in gradient], simplex(seed), (side, side))
        s["biomes"] = torch.zeros((width, pitch), dtype=torch.int16, device="cuda")
        ops.voronoi_biomemap(s["biomes"], pitch, width, width, (0, 0), 192, 8, seed)
        s["heights"] = torch.zeros((width, pitch), dtype=torch.int16, device="cuda")
        fixed = torch.empty((width, width), dtype=torch.int16, device="cuda")
        ops.format_heightmap(terrain(width, 8, 192, seed), fixed, width, width)
        s["heights"][:, :width] = fixed
        s["out"] = torch.zeros((width, width), dtype=torch.uint8, device="cuda")
        s["list"] = [stp.SplatChunk(c % n, c // n, float(c % n * side), float(c // n * side)) for c in range(n * n)]
    elif op == "generate":
        side = case["side"]
        s["generator"] = stp.STPHeightfieldGenerator(
            stp.ChunkSetting((side, side), (3, 3), (3, 3)), raindrops(1000, 2, 30, seed), simplex(seed),
            biome_table(case["biomes"], seed), case["radius"])
        whole = biome_map(side, case["radius"], case["biomes"], case["cell"], seed, whole=True).cpu().numpy()
        whole = whole.view(np.uint16)
        s["chunks"] = [np.ascontiguousarray(whole[y:y + side, x:x + side]) for y in range(0, 3 * side, side)
                       for x in range(0, 3 * side, side)]
        s["out"] = np.zeros((side, side), np.float32)
    elif op == "batch":
        requests = batch_requests(case, seed)
        b = s["batch"] = stp.Batch(requests, raindrops(1000, case["brush"], case["lifetime"], seed), simplex(seed),
                                   biome_table(case["biomes"], seed))
        b.synthesize(case["cell"], seed)
        b.tune()
        s["out"] = [torch.as_tensor(Buffer(b, b.buffers(n)[1], (3 * r["MapSize"], 3 * r["MapSize"]), "<f4"),
                                    device="cuda") for n, r in enumerate(requests)]
    return s


# --------------------------------------------------------------------- passes


def stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def address(t):
    return C.c_void_p(t.data_ptr())


def filter_chunk(s):
    """The filter through the C ABI into buffers that the caller keeps."""
    stp.check(stp.lib().stpgb_shf_filter(
        address(s["map"]), C.byref(s["info"]), s["radius"], s["biomes"], address(s["workspace"]),
        s["workspace"].numel(), address(s["offsets"]), address(s["bins"]), s["capacity"], address(s["status"]),
        stream()))


def run(state):
    s, op, ops = state, state["op"], state["ops"]
    if op == "filter":
        filter_chunk(s)
        # a bin is {uint16 item, float weight}; bins past the chunk's last stay zero
        return {"offsets": s["offsets"], "items": s["bins"].view(torch.int16).view(-1, 4)[:, 0],
                "weights": s["bins"].view(torch.float32).view(-1, 2)[:, 1]}
    if op == "heights":
        side = s["side"]
        ops.multibiome_heightmap(s["out"], side, s["offsets"], s["bins"], (side, side),
                                 (float(s["offset_x"]), float(s["offset_y"])), s["perm"], s["grad"], s["table"])
    elif op == "erode":
        # the map is eroded in place: every pass starts from the same heights
        s["out"].copy_(s["before"])
        side, nn = s["side"], s["neighbours"]
        ops.hydraulic_erosion(s["out"], (side, side), (nn, nn), s["setting"], s["starts"], s["droplets"], s["index"],
                              s["weight"])
    elif op == "format":
        ops.format_heightmap(s["map"], s["out"], s["width"], s["height"])
    elif op == "biomemap":
        ops.layer_biomemap(s["chain"], s["ids"], s["seed"], s["out"], s["width"], s["width"], s["height"],
                           (s["offset_x"], s["offset_z"]))
    elif op == "splat":
        width = s["side"] * s["chunks"]
        s["generator"](s["biomes"], s["heights"], s["pitch"], s["out"], width, width, width, s["list"])
    elif op == "generate":
        s["generator"].generate(s["out"], s["chunks"], (float(s["offset_x"]), float(s["offset_y"])))
    elif op == "batch":
        # the fixed-point maps that the batch writes beside the heights follow from them; droplets race,
        # so the last digits of both differ from run to run
        s["batch"].run(torch.cuda.current_stream().cuda_stream)
    return s["out"]


def work(case):
    """Bytes read and written once; operations of the noise (60 per octave and bin) and of the droplets
    (about 100 per step and 4 per brush point, 0.6 of the steps eroding)."""
    op = case["op"]

    def bins(side):  # bins of a chunk: one per pixel, and more along the biomes' borders
        return side * side * min(case["biomes"], 1.0 + 5.0 * case["radius"] / case["cell"])

    def erosion(side, droplets, brush, lifetime):
        return droplets * lifetime * (100 + 0.6 * 4 * math.pi * brush * brush)

    if op == "filter":
        side, w = case["side"], case["side"] + 2 * case["radius"]
        return {"bytes": 2 * w * w + 4 * (side * side + 1) + 8 * bins(side), "flops": 0}
    if op == "heights":
        side = case["side"]
        return {"bytes": 4 * (2 * side * side + 1) + 8 * bins(side), "flops": bins(side) * 364}
    if op == "erode":
        side = case["side"] * case["neighbours"]
        return {"bytes": 8 * side * side + 8 * case["droplets"],
                "flops": erosion(side, case["droplets"], case["brush"], case["lifetime"])}
    if op == "format":
        return {"bytes": 6 * case["width"] * case["height"], "flops": 0}
    if op == "biomemap":
        return {"bytes": 2 * case["width"] * case["height"], "flops": 0}
    if op == "splat":
        pixels = (case["side"] * case["chunks"])**2
        return {"bytes": 5 * pixels, "flops": 200 * pixels}
    if op == "generate":
        side = case["side"]
        return {"bytes": 2 * 9 * side * side + 4 * side * side, "flops": bins(side) * 364}
    side = (case["side"] + case["least"]) // 2
    droplets = case["density"] * side * side
    return {"bytes": case["requests"] * ((5 * side)**2 * 2 + (3 * side)**2 * 6 + 8 * droplets),
            "flops": case["requests"] * (9 * bins(side) * 364
                                         + erosion(side, droplets, case["brush"], case["lifetime"]))}


# ---------------------------------------------------------------------- exact


def window_sum(x, length, dim):
    """Sums of `length` consecutive entries along `dim`."""
    c = torch.cumsum(x, dim)
    c = torch.cat([torch.zeros_like(c.narrow(dim, 0, 1)), c], dim)
    n = c.shape[dim] - length
    return c.narrow(dim, length, n) - c.narrow(dim, 0, n)


def last_insertion(present, length, dim):
    """Along `dim`, per entry: the latest position up to it that holds an item none of the `length`
    positions before it held (an item leaves a window of `length` after the next one entered)."""
    n = present.shape[dim]
    pad = torch.zeros_like(present.narrow(dim, 0, 1)).repeat_interleave(length, dim)
    before = window_sum(torch.cat([pad, present], dim).int(), length, dim).narrow(dim, 0, n)
    at = torch.arange(n, device=present.device, dtype=torch.int32)
    at = at.view([-1 if d == dim else 1 for d in range(present.dim())])
    return torch.cummax(torch.where(present & (before == 0), at, torch.full_like(at, -1)), dim).values


def histograms(m, side, radius, biomes):
    """Counts [biome, y, x] of the windows of a chunk, and keys that order a pixel's bins as a window
    that slides down every column and then along the rows met them."""
    w, length = side + 2 * radius, 2 * radius + 1
    region = m[side - radius:side - radius + w, side - radius:side - radius + w].int()
    counts, keys = [], []
    for b in range(biomes):
        inside = region == b
        column = window_sum(inside.int(), length, 0)
        entered = last_insertion(inside, length, 0)[length - 1:]
        counts.append(window_sum(column, length, 1))
        latest = last_insertion(column > 0, length, 1)[:, length - 1:]
        keys.append(latest.long() * (w + 1) + torch.gather(entered, 1, latest.clamp(min=0).long()))
    return torch.stack(counts), torch.stack(keys)


def fractal64(perm, grad, x, y, biome):
    """Fractal simplex noise in [0, 1] at (x, y) in 64 bits."""
    skew, unskew = (math.sqrt(3.0) - 1.0) / 2.0, (3.0 - math.sqrt(3.0)) / 6.0
    total, amplitude, frequency, reach = torch.zeros_like(x), 1.0, 1.0, 0.0
    for _ in range(int(biome["Octave"])):
        u, v = x * frequency, y * frequency
        i, j = torch.floor(u + (u + v) * skew), torch.floor(v + (u + v) * skew)
        dx, dy = u - (i - (i + j) * unskew), v - (j - (i + j) * unskew)
        east = dx > dy
        value = torch.zeros_like(x)
        for a, b in ((torch.zeros_like(east), torch.zeros_like(east)), (east, ~east),
                     (torch.ones_like(east), torch.ones_like(east))):
            shift = unskew * (a.double() + b.double())
            cx, cy = dx - a.double() + shift, dy - b.double() + shift
            g = perm[(i.long() & 255) + a.long() + perm[(j.long() & 255) + b.long()]] % (grad.shape[0])
            fall = torch.clamp(0.5 - cx * cx - cy * cy, min=0.0)
            value += fall**4 * (grad[g, 0] * cx + grad[g, 1] * cy)
        total += 70.0 * value * amplitude
        reach += amplitude
        amplitude *= float(biome["Persistence"])
        frequency *= float(biome["Lacunarity"])
    return torch.clamp((total + reach) / (2.0 * reach), 0.0, 1.0)


def voronoi(width, origin, cell, biomes, seed):
    """The seeded Voronoi biome map: of the jittered sites in the 3x3 cells around a pixel, the nearest
    one's hash."""
    word = (1 << 64) - 1

    def mix(z):
        z = (z + 0x9E3779B97F4A7C15) & word
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & word
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & word
        return z ^ (z >> 31)

    first, last = origin // cell - 1, (origin + width - 1) // cell + 1
    n = last - first + 1
    px, py, ids = np.zeros((n, n), np.int64), np.zeros((n, n), np.int64), np.zeros((n, n), np.int64)
    for r in range(n):
        for c in range(n):
            kx, ky = first + c, first + r
            h = mix(seed ^ mix(((kx * 0x9E3779B97F4A7C15) & word) ^ ((ky * 0xC2B2AE3D27D4EB4F) & word)))
            px[r, c], py[r, c], ids[r, c] = kx * cell + h % cell, ky * cell + (h >> 32) % cell, mix(h) % biomes
    px, py, ids = (torch.from_numpy(a).cuda() for a in (px, py, ids))
    g = torch.arange(origin, origin + width, device="cuda")
    at = torch.div(g, cell, rounding_mode="floor") - first
    best = torch.full((width, width), 1 << 62, device="cuda")
    out = torch.zeros((width, width), dtype=torch.int64, device="cuda")
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            r, c = (at + dy)[:, None], (at + dx)[None, :]
            d = (px[r, c] - g[None, :])**2 + (py[r, c] - g[:, None])**2
            nearer = d < best
            best, out = torch.where(nearer, d, best), torch.where(nearer, ids[r, c], out)
    return out


def exact(case, seed):
    """The weights of the filter and the heights of the noise in 64 bits.  Droplets race, so an eroded
    map has no one value; whole numbers have nothing to be off by; the generators' own permutation is
    not restated here."""
    if case["op"] not in ("filter", "heights") or case["side"] > 1024:
        return None
    side, radius, biomes = case["side"], case["radius"], case["biomes"]
    m = torch.zeros((3 * side, 3 * side), dtype=torch.int64, device="cuda")
    w = side + 2 * radius
    m[side - radius:side - radius + w, side - radius:side - radius + w] = voronoi(w, -radius, case["cell"], biomes,
                                                                                seed)
    counts, keys = histograms(m, side, radius, biomes)
    if case["op"] == "filter":
        keys = torch.where(counts > 0, keys, torch.full_like(keys, 1 << 62))
        ordered = torch.gather(counts, 0, torch.argsort(keys, 0)).permute(1, 2, 0).reshape(-1)
        weights = torch.zeros(side * side * min(biomes, 8), dtype=torch.float64, device="cuda")
        found = ordered[ordered > 0].double()[:weights.numel()]
        weights[:found.numel()] = found / (2 * radius + 1)**2
        return {"offsets": None, "items": None, "weights": weights}
    perm, grad = noise_tables(seed)
    perm = torch.from_numpy(perm.astype(np.int64)).cuda()
    grad = torch.from_numpy(grad.astype(np.float64).reshape(-1, 2)).cuda()
    y, x = torch.meshgrid(torch.arange(side, dtype=torch.float64, device="cuda"),
                          torch.arange(side, dtype=torch.float64, device="cuda"), indexing="ij")
    x, y = x - side / 2.0 + case["offset_x"], y - side / 2.0 + case["offset_y"]
    out = torch.zeros_like(x)
    for b, biome in enumerate(biome_table(biomes, seed)):
        scale = float(biome["Scale"])
        out += counts[b] / (2 * radius + 1.0)**2 * (fractal64(perm, grad, x / scale, y / scale, biome)
                                                     * float(biome["Variation"]) + float(biome["Depth"]))
    return out
