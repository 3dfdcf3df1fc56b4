"""Column kernels asked for by name, so that every state's bookkeeping runs whatever the estimate
would choose: units of 1 to 65 steps (a table holds 32), cells that are kept, entered upwards,
downwards, skipped or left for a coordinate without a cell, planes and columns that are no
multiple of a warp, alone, in batches and in a captured graph.  Bit-identical to the oracle, and
the count of column launches shows that the kernel meant is the one that ran."""
import numpy as np
import pytest
import torch

import fastnoise2_gb300 as fn
from oracle.oracle import OracleTree
from oracle.tree import N
from tests import chunkmix, trees
from tests.parity import assert_parity
from tests.test_gpu_column import TREES

pytestmark = pytest.mark.gpu

LATTICE = {"FBmPerlin", "PerlinRange", "Value", "RidgedValue", "ScaledBlend"}     # states in 4D too
LENGTHS = [1, 5, 31, 32, 33, 64, 65]
SHAPES = {2: [(1, 1), (31, 33), (70, 65), (5, 200)], 3: [(1, 1, 1), (5, 3, 2), (33, 1, 31), (11, 6, 97), (9, 5, 140)],
          4: [(1, 1, 1, 1), (4, 4, 4, 33), (5, 1, 7, 70)]}
# along the last axis: kept cells, the next one up and down, skipped ones, none left
STEPS = [(1.0,) * 4, (0.37, 1.1, -0.9, -1.3), (0.2, 0.1, 0.05, 0.06), (1.5, -2.0, 40.0, 75.0), (1.0, 0.0, 0.0, 0.0)]


def states(name, dim):
    return dim < 4 or name in LATTICE


@pytest.fixture(scope="module")
def columns(gpu):
    nodes = {k: trees.to_product(m()) for k, m in TREES.items()}
    for dim in (2, 3, 4):
        gpu.jit_compile([(n, dim) for n in nodes.values()])
    return nodes


@pytest.fixture(autouse=True)
def route(gpu):
    yield
    gpu.set_grid_route(gpu.GRID_ROUTE_AUTO)


@pytest.mark.parametrize("dim", [2, 3, 4])
@pytest.mark.parametrize("name", sorted(TREES))
def test_units_of_every_length(columns, name, dim):
    oracle, off = OracleTree(TREES[name]()), (-7.5, 3.25, -11.0, 2.0)[:dim]
    for shape in SHAPES[dim]:
        for step in STEPS:
            ref, rmm = oracle.grid(off, shape, step[:dim], 77)
            for length in LENGTHS:
                fn.set_grid_route(fn.GRID_ROUTE_COLUMNS, length)
                got, mm = columns[name].gen_uniform_grid(off, shape, step[:dim], 77)
                assert fn.set_grid_route(fn.GRID_ROUTE_AUTO) == states(name, dim)
                assert_parity(got, mm, ref, rmm, label=f"{name} {shape} {step} {length}")


@pytest.mark.parametrize("name", sorted(TREES))
def test_extreme_positions(columns, name):
    """Across and along the columns: past the int32 cells, infinite and NaN, and columns that come
    from there into the range and leave it again."""
    oracle = OracleTree(TREES[name]())
    inf, nan = float("inf"), float("nan")
    cases = [((0.5, -3.0, v), (1.0, 1.0, 1.0)) for v in (2.0**20, 1.7e7, 3e9, -3e9, 1e30, inf, -inf, nan)]
    cases += [((v, 2.0, 1.0), (1.0, 1.0, 1.0)) for v in (1.7e7, 3e9, -3e9, 1e30, inf, nan)]
    cases += [((0.5, v, -9.0), (1.0, 1.0, 0.5)) for v in (-3e9, inf, nan)]
    cases += [((0.5, -3.0, -s * 17.25), (1.0, 1.0, s)) for s in (1.3e8, 1.1e9, 1.7e10, 2e11, 1e37)]
    cases += [((0.5, -3.0, s * 17.25), (1.0, 1.0, -s)) for s in (1.3e8, 1.7e10, 1e38)]
    cases += [((0.5, -3.0, 1.0), (1.0, 1.0, v)) for v in (inf, nan, 3e38)]
    cases += [((-s * 4.0, -3.0, 1.0), (s, 1.0, 0.25)) for s in (1.1e9, 2e11)]          # some lanes in range
    for off, step in cases:
        ref, rmm = oracle.grid(off, (9, 5, 35), step, -5)
        for length in (5, 32, 64):
            fn.set_grid_route(fn.GRID_ROUTE_COLUMNS, length)
            got, mm = columns[name].gen_uniform_grid(off, (9, 5, 35), step, -5)
            assert fn.set_grid_route(fn.GRID_ROUTE_AUTO) == 1
            assert_parity(got, mm, ref, rmm, label=f"{name} {off} {step} {length}")


@pytest.mark.parametrize("length", [0, 5, 33])
@pytest.mark.parametrize("dim", [2, 3, 4])
@pytest.mark.parametrize("name", sorted(TREES))
def test_batches_and_their_minmax(columns, name, dim, length):
    oracle, off = OracleTree(TREES[name]()), (-7.5, 3.25, -11.0, 2.0)[:dim]
    grids = [(shape, step) for shape in SHAPES[dim] for step in STEPS]
    outs = [torch.full((int(np.prod(shape)),), np.nan, device="cuda") for shape, _ in grids]
    mms = [np.zeros(2, np.float32) for _ in grids]
    kind = {2: fn.KIND_GRID2D, 3: fn.KIND_GRID3D, 4: fn.KIND_GRID4D}[dim]
    reqs = [fn.make_request(columns[name], kind, out.data_ptr(), 77, shape, off, step[:dim], minmax=mm)
            for out, mm, (shape, step) in zip(outs, mms, grids)]
    fn.set_grid_route(fn.GRID_ROUTE_COLUMNS, length)
    fn.gen_batch(reqs, sync=True)
    assert fn.set_grid_route(fn.GRID_ROUTE_AUTO) == (len(grids) if states(name, dim) else 0)
    for out, mm, (shape, step) in zip(outs, mms, grids):
        ref, rmm = oracle.grid(off, shape, step[:dim], 77)
        assert_parity(out.cpu().numpy(), (mm[0], mm[1]), ref, rmm, label=f"{name} {shape} {step}")


def test_captured_column_calls(columns):
    count, off = (40, 33, 70), (-7.5, 3.25, -11.0)
    names = ["FBmPerlin", "Terrain", "CellLookup", "Warp"]
    outs = [torch.empty(int(np.prod(count)), device="cuda") for _ in names]
    mm = torch.empty((len(names), 2), device="cuda")
    stream = torch.cuda.Stream()

    def calls():
        for k, name in enumerate(names):
            columns[name].gen_uniform_grid_device(outs[k].data_ptr(), off, count, (1.0,) * 3, k, mm[k].data_ptr(), stream.cuda_stream)

    fn.set_grid_route(fn.GRID_ROUTE_COLUMNS, 20)
    with torch.cuda.stream(stream):
        calls()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        calls()
        graph.capture_end()
    assert fn.set_grid_route(fn.GRID_ROUTE_AUTO) == 2 * len(names)
    for t in (*outs, mm):
        t.zero_()
    torch.cuda.synchronize()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for k, name in enumerate(names):
        ref, rmm = OracleTree(TREES[name]()).grid(off, count, (1.0,) * 3, k)
        assert_parity(outs[k].cpu().numpy(), tuple(mm[k].tolist()), ref, rmm, label=name)


# (tree, grid, step along every axis, requests, walked in columns alone / in a batch of as many): the
# estimate's side of each.  The last are grids that columns take longer over than points: Value states
# that often enter cells, warps with more neighbourhoods than the table holds, 4D super-simplex
# beside a column state, batches too small to gain a column kernel's longer first and last units.
# Small batches of heavy points take columns: their longest tile takes longer than the longest unit.
RULE = [("FBmPerlin", (256, 256, 256), 1.0, 1, 1, 1), ("FBmPerlin", (16, 16, 16), 1.0, 1, 0, 1), ("FBmPerlin", (32, 32, 32), 1.0, 200, 0, 1),
        ("Terrain", (128, 128, 128), 1.0, 4, 1, 1), ("CellValue", (160, 160, 160), 1.0, 2, 1, 1), ("Value", (1024, 1024), 1.0, 12, None, 1),
        ("CellLookup", (97, 90, 101), 1.0, 8, 1, 1),
        ("FBmPerlin", (128, 128, 128), 40.0, 4, 0, 0), ("Terrain", (3, 3, 2000), 1.0, 64, 0, 0), ("FBmPerlin", (2, 50000), 1.0, 16, 0, 0),
        ("FBmValueShort", (1076, 2092), 3.3, 4, 0, 0), ("FBmValueShort", (691, 284), 2.92, 42, 0, 0), ("CellValue", (160, 160, 160), 60.0, 2, 0, 0),
        ("CellValue", (26, 64, 144), 1.4, 1, 0, 1), ("FadeSuper4D", (75, 37, 21, 58), 1.0, 1, 0, None), ("FBmPerlin2", (95, 227), 2.9, 64, 0, 0),
        ("CellLookup", (2, 2, 2), 1.0, 8, 0, 0), ("Terrain", (32, 32, 32), 1.0, 4, None, 1), ("CellValue", (32, 32, 32), 1.0, 4, None, 1),
        ("CellLookup", (9, 10, 15), 0.75, 18, None, 1), ("FBmPerlin", (2, 2000), 1.0, 16, None, 0)]
RULE_TREES = {"FBmValueShort": lambda: N("FractalFBm", Source=N("Value", Feature_Scale=9.0), Octaves=5),
              "FBmPerlin2": lambda: N("FractalFBm", Source=N("Perlin", Feature_Scale=20.0), Octaves=2),
              "FadeSuper4D": lambda: N("Fade", A=N("FractalFBm", Source=N("SuperSimplex", Feature_Scale=30.0), Octaves=2),
                                       B=N("CellularDistance", Feature_Scale=30.0), Fade=N("Perlin", Feature_Scale=50.0))}


@pytest.mark.parametrize("name,count,step,requests,alone,batch", RULE)
def test_the_estimates_route(columns, name, count, step, requests, alone, batch):
    dim = len(count)
    node = columns[name] if name in columns else trees.to_product(RULE_TREES[name]())
    if name not in columns:
        fn.jit_compile([(node, dim)])
    out = torch.empty(int(np.prod(count)), device="cuda")
    fn.set_grid_route(fn.GRID_ROUTE_AUTO)
    node.gen_uniform_grid_device(out.data_ptr(), (0.0,) * dim, count, (step,) * dim, 3)
    walked = fn.set_grid_route(fn.GRID_ROUTE_AUTO)
    assert alone is None or walked == alone
    kind = {2: fn.KIND_GRID2D, 3: fn.KIND_GRID3D, 4: fn.KIND_GRID4D}[dim]
    outs = torch.empty((requests, out.numel()), device="cuda")
    fn.gen_batch([fn.make_request(node, kind, o.data_ptr(), 3, count, (0.0,) * dim, (step,) * dim) for o in outs])
    walked = fn.set_grid_route(fn.GRID_ROUTE_POINTS)
    assert batch is None or walked == batch * requests
    node.gen_uniform_grid_device(out.data_ptr(), (0.0,) * dim, count, (step,) * dim, 3)
    torch.cuda.synchronize()
    assert fn.set_grid_route(fn.GRID_ROUTE_AUTO) == 0


def test_steps_without_an_estimate_do_not_change_the_other_requests(columns):
    """Infinite and NaN steps have no estimate: such requests run as points, the others of their tree
    in columns as without them."""
    inf, nan = float("inf"), float("nan")
    odd = [((1, 5, 9), (inf, 1.0, 1.0)), ((7, 5, 9), (nan, 1.0, 1.0)), ((40, 3, 20), (inf, 1.0, inf)), ((5, 1, 9), (1.0, nan, nan))]
    for name in ("CellValue", "Terrain", "FBmPerlin"):
        grids = [((32, 32, 32), (1.0, 1.0, 1.0))] * 100 + odd
        outs = [torch.empty(int(np.prod(c)), device="cuda") for c, _ in grids]
        fn.set_grid_route(fn.GRID_ROUTE_AUTO)
        fn.gen_batch([fn.make_request(columns[name], fn.KIND_GRID3D, o.data_ptr(), 5, c, (0.0, 2.0, -3.0), s) for o, (c, s) in zip(outs, grids)])
        assert 100 <= fn.set_grid_route(fn.GRID_ROUTE_AUTO) <= 104, name
        oracle = OracleTree(TREES[name]())
        for o, (c, s) in list(zip(outs, grids))[99:]:
            ref, rmm = oracle.grid((0.0, 2.0, -3.0), c, s, 5)
            assert_parity(o.cpu().numpy(), rmm, ref, rmm, label=f"{name} {c} {s}")


def test_every_batch_variant_of_the_point_kernels(columns, tmp_path):
    """Tuned variants serve the requests that are not walked in columns; asked to take points, every
    request of every tree runs each variant."""
    nodes = [trees.to_product(m()) for m in trees.MIX_TREES]
    fn.jit_compile([(n, d) for n in nodes for d in (2, 3)])
    chunks = chunkmix.make_mix(48, seed=21, sizes=[(16, 16, 16), (31, 9, 20), (64, 64), (70, 33)])
    outs = [torch.empty(int(np.prod(c.count)), device="cuda") for c in chunks]
    mms = [np.zeros(2, np.float32) for _ in chunks]
    reqs = [fn.make_request(nodes[c.tree], fn.KIND_GRID3D if len(c.count) == 3 else fn.KIND_GRID2D, o.data_ptr(), c.seed, c.count,
                            c.offset, (1.0,) * len(c.count), minmax=mm) for c, o, mm in zip(chunks, outs, mms)]
    fn.set_grid_route(fn.GRID_ROUTE_POINTS)
    fn.autotune_batch(reqs)
    path = tmp_path / "tune.txt"
    fn.autotune_save(path)
    lines = path.read_text().splitlines()
    refs = [OracleTree(trees.MIX_TREES[c.tree]()).grid(c.offset, c.count, (1.0,) * len(c.count), c.seed) for c in chunks]
    try:
        for variant in range(5):
            path.write_text("\n".join([ln for ln in lines if not ln.startswith("tree ")] +
                                      [f"tree {ln.split()[1]} {variant} 0 0 0 1.0" for ln in lines if ln.startswith("tree ")]) + "\n")
            fn.autotune_load(path)
            for o in outs:
                o.fill_(float("nan"))
            fn.gen_batch(reqs, sync=True)
            for c, o, mm, (ref, rmm) in zip(chunks, outs, mms, refs):
                assert_parity(o.cpu().numpy(), (mm[0], mm[1]), ref, rmm, label=f"variant {variant} {c}")
    finally:
        path.write_text("\n".join(f"tree {ln.split()[1]} 0 0 0 0 1.0" for ln in lines if ln.startswith("tree ")) + "\n")
        fn.autotune_load(path)
    assert fn.set_grid_route(fn.GRID_ROUTE_AUTO) == 0


def test_invalid_routes(gpu):
    for route, steps in ((-1, 0), (3, 0), (0, -1)):
        with pytest.raises(gpu.FastNoiseError):
            gpu.set_grid_route(route, steps)
