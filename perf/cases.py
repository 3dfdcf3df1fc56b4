"""The work a program has this library do, as cases that can be timed and compared.

Every case goes through the package's public entry points on specialised kernels
(`jit_compile`, which a program calls once per tree); seeds and chunk origins come from the
case's seed, so consecutive passes see other inputs.  Trees, sizes and the request mix are
those of the repository's benchmark and tests.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fastnoise2_gb300 as fn

# ---------------------------------------------------------------- trees

def _node(kind, **members):
    n = fn.Node.new(kind)
    for k, v in members.items():
        n.set(k.replace("_", " "), v)
    return n


def _terrain():
    """Domain-warped ridged SuperSimplex faded with CellularDistance, remapped and terraced."""
    ridged = _node("FractalRidged", Source=_node("SuperSimplex"), Octaves=4)
    warp = _node("DomainWarpGradient", Source=ridged, Warp_Amplitude=30.0)
    warped = _node("DomainWarpFractalProgressive", Domain_Warp_Source=warp, Octaves=3)
    cells = _node("CellularDistance", Distance_Function="Euclidean", Distance_Index_0=0, Distance_Index_1=1,
                  Return_Type="Index0Sub1", Grid_Jitter=1.0)
    fade = _node("Fade", A=warped, B=cells)
    remap = _node("Remap", Source=fade, From_Min=-1.0, From_Max=1.0, To_Min=0.0, To_Max=1.0)
    return _node("Terrace", Source=remap, Step_Count=8.0, Smoothness=0.3)


def _surface():
    """A terrain surface for the meshers: vertical gradient plus fractal noise."""
    g = fn.Node.new("Gradient").set("Multiplier", 0.02, 1)
    return _node("Add", LHS=_node("FractalFBm", Source=_node("Simplex", Feature_Scale=60.0), Octaves=4), RHS=g)


TREES = {
    "simplex": lambda: _node("Simplex", Feature_Scale=50.0),
    "fbm_perlin": lambda: _node("FractalFBm", Source=_node("Perlin"), Octaves=5, Gain=0.5, Lacunarity=2.0, Weighted_Strength=0.0),
    "terrain": _terrain,
    "value": lambda: _node("Value"),
    "cellular_value": lambda: _node("CellularValue"),
    "cellular_lookup": lambda: _node("CellularLookup", Lookup=_node("Simplex")),
    "fbm_simplex": lambda: _node("FractalFBm", Source=_node("Simplex"), Octaves=3),
    "blend": lambda: _node("Add", LHS=_node("Simplex"), RHS=_node("Multiply", LHS=_node("Perlin"), RHS=_node("Value"))),
    "surface": _surface,
}
MIX = ["simplex", "fbm_perlin", "terrain", "value", "cellular_value", "cellular_lookup", "fbm_simplex", "blend"]
MIX_SIZES = [(16, 16, 16), (32, 32, 32), (64, 64, 64), (32, 32), (128, 128), (512, 512)]

# Arithmetic steps of one point of each tree in 2D / 3D / 4D, as the noise functions define
# them (every neighbour cell evaluated; one fused multiply-add, hash multiply or select = 1).
OPS = {
    "simplex": (90, 139, 225), "fbm_perlin": (490, 994, 2218), "terrain": (1019, 2734, 7600), "value": (47, 92, 181),
    "cellular_value": (195, 750, 2781), "cellular_lookup": (310, 995, 3409), "fbm_simplex": (293, 442, 702),
    "blend": (228, 422, 841), "surface": (390, 590, 940),
}


# ---------------------------------------------------------------- cases

def listed():
    return [
        # one game chunk of one plain noise: what a call costs when there is next to nothing to compute
        {"name": "grid3d_simplex_16", "kind": "grid", "tree": "simplex", "nx": 16, "ny": 16, "nz": 16, "nw": 0},
        # the benchmark's single-node call
        {"name": "grid3d_simplex_64", "kind": "grid", "tree": "simplex", "nx": 64, "ny": 64, "nz": 64, "nw": 0},
        # the benchmark's large fractal grid: the usual density volume
        {"name": "grid3d_fbm_perlin_256", "kind": "grid", "tree": "fbm_perlin", "nx": 256, "ny": 256, "nz": 256, "nw": 0},
        # the benchmark's composite terrain tree over one large chunk
        {"name": "grid3d_terrain_128", "kind": "grid", "tree": "terrain", "nx": 128, "ny": 128, "nz": 128, "nw": 0},
        # cellular biome lookup over a ragged volume: no extent is a multiple of a warp or of four
        {"name": "grid3d_cell_lookup_odd", "kind": "grid", "tree": "cellular_lookup", "nx": 150, "ny": 97, "nz": 61, "nw": 0},
        # a heightmap of odd extents, as an image or a terrain heightfield
        {"name": "grid2d_fbm_simplex_odd", "kind": "grid", "tree": "fbm_simplex", "nx": 1001, "ny": 733, "nz": 0, "nw": 0},
        # the benchmark's tileable texture (a 4D torus behind a 2D image)
        {"name": "tile_terrain_1024", "kind": "tile", "tree": "terrain", "nx": 1024, "ny": 1024, "nz": 0, "nw": 0},
        # the serving mix's 4D grid (3D volumes over time)
        {"name": "grid4d_fbm_perlin_32", "kind": "grid", "tree": "fbm_perlin", "nx": 32, "ny": 32, "nz": 32, "nw": 32},
        # the serving mix's scattered positions, 1 M points in [-1e4, 1e4]^3 (object placement, particles)
        {"name": "pos3d_blend_1m", "kind": "positions", "tree": "blend", "nx": 1 << 20, "ny": 0, "nz": 0, "nw": 0},
        # the headline: 4096 chunk and heightmap requests of eight trees in one batched launch
        {"name": "batch_mix_4096", "kind": "batch", "tree": "mix", "nx": 4096, "ny": 0, "nz": 0, "nw": 0},
        # the drop-in call of the reference's C interface: host memory in, host memory out
        {"name": "host_grid3d_value_64", "kind": "host", "tree": "value", "nx": 64, "ny": 64, "nz": 64, "nw": 0},
        # dual marching cubes on a row of eight editor chunks of a terrain surface
        {"name": "mesh_dmc_128x8", "kind": "mesh", "tree": "surface", "nx": 128, "ny": 8, "nz": 0, "nw": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "grid", "grid", "batch", "batch", "tile", "positions", "host", "mesh"])
    c = {"kind": kind, "tree": rng.choice(MIX), "nx": 0, "ny": 0, "nz": 0, "nw": 0}
    if kind in ("grid", "host"):
        dim = rng.choice([2, 3, 3, 3, 4]) if kind == "grid" else rng.choice([2, 3])
        top = {2: 2048, 3: 256, 4: 40}[dim] if kind == "grid" else {2: 512, 3: 64}[dim]
        low = {2: 24, 3: 12, 4: 6}[dim]
        for k in ["nx", "ny", "nz", "nw"][:dim]:
            c[k] = _log_int(rng, low, top)
    elif kind == "tile":
        c["nx"], c["ny"] = _log_int(rng, 48, 1400), _log_int(rng, 48, 1400)
    elif kind == "positions":
        c["nx"] = _log_int(rng, 1000, 3_000_000)
    elif kind == "batch":
        c["tree"], c["nx"] = "mix", _log_int(rng, 6, 3000)
    else:
        c["tree"], c["nx"], c["ny"] = "surface", _log_int(rng, 32, 127), rng.randint(1, 8)
    return c


def _counts(case):
    return [int(case[k]) for k in ("nx", "ny", "nz", "nw") if int(case[k]) > 0]


def _mix_sizes(n):
    """The sizes and trees of a mix of n requests: the same for every seed, so that a pass costs the same."""
    rng = np.random.default_rng(20261203)
    return [(MIX_SIZES[int(rng.integers(len(MIX_SIZES)))], int(rng.integers(len(MIX)))) for _ in range(n)]


# ---------------------------------------------------------------- prepare

def _specialised(pairs):
    """A program compiles its trees once, when it starts."""
    todo = [(n, d) for n, d in pairs if not fn.is_specialised(n, d)]
    if todo:
        fn.jit_compile(todo)


def _origin(rng, size, dim):
    """A chunk origin: a multiple of the chunk's extent, up to a few thousand cells out."""
    return [float(s * int(rng.integers(-64, 65))) for s in size[:dim]]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    dev = torch.device("cuda")
    kind, size = case["kind"], _counts(case)
    s = {"kind": kind, "seed": int(rng.integers(-(2**31), 2**31 - 1)), "size": size}
    if kind == "batch":
        nodes = [TREES[t]() for t in MIX]
        _specialised([(n, d) for n in nodes for d in (2, 3)])
        mix = _mix_sizes(size[0])
        points = [math.prod(sz) for sz, _ in mix]
        s["out"] = torch.empty(sum(points), dtype=torch.float32, device=dev)
        reqs, at = [], s["out"].data_ptr()
        for (sz, t), p in zip(mix, points):
            lim = (1 << 20) // sz[0]
            org = [float(sz[0] * int(v)) for v in rng.integers(-lim, lim + 1, len(sz))]
            reqs.append(fn.make_request(nodes[t], fn.KIND_GRID3D if len(sz) == 3 else fn.KIND_GRID2D, at,
                                        int(rng.integers(-(2**31), 2**31 - 1)), sz, org, (1, 1, 1, 1)))
            at += 4 * p
        # min/max of every request into one host array, as a chunk manager keeps them for culling
        s["mm"] = np.zeros((len(mix), 2), np.float32)
        arr = fn.request_array(reqs)
        for k in range(len(mix)):
            arr[k].minMax = s["mm"][k].ctypes.data_as(type(arr[k].minMax))
        s["reqs"], s["keep"] = arr, (nodes, reqs)
        return s
    node = TREES[case["tree"]]()
    s["node"] = node
    if kind == "mesh":
        _specialised([(node, 3)])
        n, chunks = size
        vcap, icap = n * n * n + 4096, 3 * n * n * n + 8192
        s["vertices"] = torch.zeros((chunks, vcap, 4), dtype=torch.float32, device=dev)
        s["indices"] = torch.zeros((chunks, icap), dtype=torch.int32, device=dev)
        s["buffers"] = [(s["vertices"][k].data_ptr(), vcap, s["indices"][k].data_ptr(), icap) for k in range(chunks)]
        z = n * int(rng.integers(-8, 9))
        s["chunks"] = [(n * (k - chunks // 2), -n // 2, z) for k in range(chunks)]
        return s
    dim = 4 if kind == "tile" else 3 if kind == "positions" else len(size)
    _specialised([(node, dim)])
    s["mm"] = torch.empty(2, dtype=torch.float32, device=dev)
    if kind == "tile":
        s["step"] = (1.0, 1.0)
        s["out"] = torch.empty(size[0] * size[1], dtype=torch.float32, device=dev)
    elif kind == "positions":
        g = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 40)))
        s["pos"] = [(torch.rand(size[0], generator=g, device=dev) * 2e4 - 1e4) for _ in range(3)]
        s["out"] = torch.empty(size[0], dtype=torch.float32, device=dev)
    elif kind == "host":
        s["offset"], s["step"] = _origin(rng, size, dim), [1.0] * dim
        s["out"] = np.zeros(math.prod(size), np.float32)
        s["out"] += 1.0                                       # a buffer that the program has used before
    else:
        s["offset"], s["step"] = _origin(rng, size, dim), [1.0] * dim
        s["out"] = torch.empty(math.prod(size), dtype=torch.float32, device=dev)
    return s


# ---------------------------------------------------------------- run

def run(s):
    kind = s["kind"]
    if kind == "host":
        out, mm = s["node"].gen_uniform_grid(s["offset"], s["size"], s["step"], s["seed"], s["out"])
        return {"out": out, "min": mm[0], "max": mm[1]}
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "grid":
        s["node"].gen_uniform_grid_device(s["out"].data_ptr(), s["offset"], s["size"], s["step"], s["seed"], s["mm"].data_ptr(), stream)
    elif kind == "tile":
        s["node"].gen_tileable_2d_device(s["out"].data_ptr(), s["size"], s["step"], s["seed"], s["mm"].data_ptr(), stream)
    elif kind == "positions":
        s["node"].gen_position_array_device(s["out"].data_ptr(), s["size"][0], [p.data_ptr() for p in s["pos"]], (0.0, 0.0, 0.0),
                                            s["seed"], s["mm"].data_ptr(), stream)
    elif kind == "batch":
        fn.gen_batch(s["reqs"], stream, sync=True)            # the min/max of every request is on the host when it returns
    else:
        res = fn.build_chunk_meshes("dmc", s["node"], s["size"][0], s["chunks"], s["seed"], 0.0, False, s["buffers"], stream)
        if not all(r["fits"] for r in res):
            raise RuntimeError("mesh buffers too small")
        return {"vertices": s["vertices"], "indices": s["indices"],
                "counts": np.array([(r["vertexCount"], r["indexCount"]) for r in res], np.int64),
                "heights": np.array([(r["minAirY"], r["maxSolidY"], *r["minMax"]) for r in res], np.float32)}
    return {"out": s["out"], "minmax": s["mm"]}


def work(case):
    size = _counts(case)
    if case["kind"] == "batch":
        mix = _mix_sizes(size[0])
        return {"bytes": sum(4 * math.prod(sz) + 8 for sz, _ in mix),
                "flops": sum(math.prod(sz) * OPS[MIX[t]][len(sz) - 2] for sz, t in mix)}
    if case["kind"] == "mesh":
        # densities of the chunk and its apron once; a surface of about one layer of quads (6 indices, one vertex each)
        n, chunks = size
        return {"bytes": chunks * n * n * (16 + 24), "flops": chunks * (n + 4) ** 3 * OPS[case["tree"]][1]}
    dim = 4 if case["kind"] == "tile" else 3 if case["kind"] == "positions" else len(size)
    points = math.prod(size)
    read = 12 * points if case["kind"] == "positions" else 0
    return {"bytes": 4 * points + 8 + read, "flops": points * OPS[case["tree"]][dim - 2]}


# ---------------------------------------------------------------- the same numbers in 64 bits
# Simplex, Perlin and Value noise and their fractals from their definitions, on float64 tensors
# (hashes on wrapped 32-bit integers).  The terrain tree, the cellular trees and the meshes have no such
# value here: each takes discrete decisions (cells, terraces, cut edges) on 32-bit positions.

_PRIMES = [(p ^ 0x80000000) - 0x80000000 for p in (0xF797C5C7, 0x6C060C89, 0x465FD04F, 0xF7A62279)]
_MULT = (0xB7E0A5F5 ^ 0x80000000) - 0x80000000


def _wrap(v):
    return ((v + 0x80000000) & 0xFFFFFFFF) - 0x80000000


def _hash(seed, cell):
    h = torch.full_like(cell[0], seed)
    for k, c in enumerate(cell):
        h = h ^ _wrap(c * _PRIMES[k])
    return h


def _gradient_index(seed, cell):
    h = _wrap(_hash(seed, cell) * _MULT)
    return (h >> 15) ^ h


def _pick(cond, a, b):
    return torch.where(cond, a, b)


def _dot(h, d):
    """The hash's gradient direction times the offset d."""
    sign = lambda v, bit: _pick((h >> bit) & 1 == 1, -v, v)    # noqa: E731
    if len(d) == 2:
        x, y = sign(d[0], 0), sign(d[1], 1)
        swap = (h >> 2) & 1 == 1
        return (1.0 + math.sqrt(2.0)) * _pick(swap, y, x) + _pick(swap, x, y)
    if len(d) == 3:
        b = h & 13
        u = _pick(b > 7, d[1], d[0])
        v = _pick(b == 12, d[0], _pick(b < 2, d[1], d[2]))
        return sign(u, 0) + sign(v, 1)
    b = h & 24
    return sign(_pick(b > 0, d[0], d[1]), 0) + sign(_pick(b > 15, d[1], d[2]), 1) + sign(_pick(b > 16, d[2], d[3]), 2)


def _lattice(p):
    base = [torch.floor(v) for v in p]
    return [b.to(torch.int64) for b in base], [v - b for v, b in zip(p, base)]


def _interpolate(cell, frac, ease, corner):
    """corner(cell + bits, bits) blended over the 2^D corners of the lattice cell."""
    dim = len(cell)
    t = [ease(f) for f in frac]
    values = [corner([c + ((m >> k) & 1) for k, c in enumerate(cell)], m) for m in range(1 << dim)]
    for k in range(dim):
        values = [values[2 * j] + t[k] * (values[2 * j + 1] - values[2 * j]) for j in range(len(values) // 2)]
    return values[0]


def _perlin(seed, p):
    cell, frac = _lattice(p)
    v = _interpolate(cell, frac, lambda t: t * t * t * (t * (t * 6 - 15) + 10),
                     lambda c, m: _dot(_gradient_index(seed, c), [f - ((m >> k) & 1) for k, f in enumerate(frac)]))
    return v / {2: 1.726796627044677734375, 3: 1.0363424, 4: 1.33858621120452880859375}[len(p)]


def _value(seed, p):
    cell, frac = _lattice(p)

    def corner(c, m):
        h = _hash(seed, c)
        return _wrap(h * _wrap(h * _MULT)).double()

    return _interpolate(cell, frac, lambda t: t * t * (3 - 2 * t), corner) / 2147483648.0


def _simplex(seed, p):
    dim = len(p)
    skew = {2: (math.sqrt(3.0) - 1) / 2, 3: 1.0 / 3.0, 4: (math.sqrt(5.0) - 1) / 4}[dim]
    unskew = {2: -1 / (math.sqrt(3.0) + 3), 3: -0.5, 4: -1 / (math.sqrt(5.0) + 5)}[dim]
    reach = {2: 0.5, 3: 0.6, 4: 0.6}[dim]
    bound = {2: 0.0261208079755306243896484375, 3: 0.030586399137973785400390625, 4: 0.036730043590068817138671875}[dim]
    total = sum(p) * skew
    cell, frac = _lattice([v + total for v in p])
    order = torch.argsort(torch.stack(frac), dim=0, descending=True, stable=True)
    rank = torch.argsort(order, dim=0)                        # 0 = the axis stepped first
    out = torch.zeros_like(p[0])
    for step in range(dim + 1):
        move = [(rank[k] < step).to(torch.int64) for k in range(dim)]
        d = [f - m for f, m in zip(frac, move)]
        shift = sum(d) * unskew
        d = [v + shift for v in d]
        f = (reach - sum(v * v for v in d)).clamp_min(0.0)
        out += f ** 4 * _dot(_gradient_index(seed, [c + m for c, m in zip(cell, move)]), d)
    return out / bound


def _fractal(noise, octaves, gain):
    def gen(seed, p):
        amp, total = 1.0, 0.0
        for k in range(octaves):
            total = total + amp * noise(seed + k, [v * 2.0 ** k for v in p])
            amp *= gain
        return total
    return gen


def _scaled(noise, scale):
    f = float(np.float32(1.0) / np.float32(scale))
    return lambda seed, p: noise(_wrap(seed), [v * f for v in p])


_EXACT = {
    "simplex": _scaled(_simplex, 50.0),
    "value": _scaled(_value, 100.0),
    "fbm_perlin": _fractal(_scaled(_perlin, 100.0), 5, 0.5),
    "fbm_simplex": _fractal(_scaled(_simplex, 100.0), 3, 0.5),
    "blend": lambda seed, p: (_scaled(_simplex, 100.0)(seed, p) + _scaled(_perlin, 100.0)(seed, p) * _scaled(_value, 100.0)(seed, p)),
}


def exact(case, seed):
    gen = _EXACT.get(case["tree"])
    if gen is None or case["kind"] not in ("grid", "host", "positions"):
        return None
    rng = np.random.default_rng(seed)
    size, call_seed = _counts(case), int(rng.integers(-(2**31), 2**31 - 1))
    if case["kind"] == "positions":
        g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 40)))
        p = [(torch.rand(size[0], generator=g, device="cuda") * 2e4 - 1e4).double() for _ in range(3)]
    else:
        org = _origin(rng, size, len(size))
        axes = [torch.arange(n, device="cuda", dtype=torch.float64) + o for n, o in zip(size, org)]
        p = [v.reshape(-1) for v in torch.meshgrid(*reversed(axes), indexing="ij")][::-1]
    parts = []
    for at in range(0, p[0].numel(), 1 << 21):
        parts.append(gen(call_seed, [v[at:at + (1 << 21)] for v in p]))
    v = torch.cat(parts)
    lo, hi = v.min(), v.max()
    if case["kind"] == "host":
        return {"out": v, "min": float(lo), "max": float(hi)}
    return {"out": v, "minmax": torch.stack([lo, hi])}
