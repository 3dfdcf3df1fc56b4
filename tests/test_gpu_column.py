"""Column kernels (grids walked along their last axis): bit-identical to the oracle where they
can go wrong -- planes and columns that are no multiple of a warp, of the 32-step tables or of a
unit, cells entered upwards, downwards, skipped or never left, and positions without a cell."""
import numpy as np
import pytest
import torch

import fastnoise2_gb300 as fn
from oracle.oracle import OracleTree
from oracle.tree import N
from tests import trees
from tests.parity import assert_parity

pytestmark = pytest.mark.gpu

TREES = {
    "FBmPerlin": trees.fbm_perlin_c1,
    "PerlinRange": lambda: N("Perlin", Feature_Scale=3.7, Seed_Offset=9, Output_Min=-0.25, Output_Max=2.0),
    "Value": lambda: N("Value", Feature_Scale=5.3),
    "RidgedValue": lambda: N("FractalRidged", Source=N("Value", Feature_Scale=11.0), Octaves=4, Weighted_Strength=0.4),
    "ScaledBlend": lambda: N("Add", LHS=N("DomainScale", Source=N("Perlin", Feature_Scale=9.0), Scaling=-1.7),
                             RHS=N("Multiply", LHS=N("DomainOffset", Source=N("Value", Feature_Scale=6.0)).set("Offset", 3.25, 0)
                                                .set("Offset", -7.5, 1).set("Offset", 0.125, 2),
                                   RHS=N("Simplex", Feature_Scale=12.0))),
    "CellValue": lambda: N("CellularValue", Feature_Scale=21.0, Seed_Offset=4),
    "CellDistance": lambda: N("CellularDistance", Feature_Scale=34.0, Grid_Jitter=0.7).set("Distance Function", "Euclidean")
                              .set("Return Type", "Index0Sub1"),
    "CellClosest": lambda: N("CellularDistance", Feature_Scale=9.0, Grid_Jitter=-1.4),
    "CellLookup": lambda: N("CellularLookup", Feature_Scale=27.0, Lookup=N("Perlin", Feature_Scale=40.0)),
    "CellTies": lambda: N("CellularValue", Feature_Scale=8.0, Grid_Jitter=0.0),
    "Terrain": trees.terrain_c2,
    "Warp": lambda: N("DomainWarpGradient", Source=N("Value", Feature_Scale=6.0), Warp_Amplitude=5.0, Feature_Scale=23.0, Seed_Offset=2)
                      .set("Amplitude Scaling", 0.5, 0),
    "WarpIndependent": lambda: N("DomainWarpFractalIndependent", Octaves=3, Weighted_Strength=0.3,
                                 Domain_Warp_Source=N("DomainWarpGradient", Source=N("Perlin"), Warp_Amplitude=8.0, Feature_Scale=40.0)),
}
SHAPES = {2: [(1, 1), (31, 33), (33, 64), (70, 65), (5, 200)],
          3: [(1, 1, 1), (5, 3, 2), (33, 1, 31), (7, 9, 33), (16, 16, 16), (11, 6, 97)],
          4: [(1, 1, 1, 1), (3, 2, 5, 7), (4, 4, 4, 33), (5, 1, 7, 40)]}
STEPS = [(1.0,) * 4, (0.37, 1.1, -0.9, -1.3), (1.5, -2.0, 40.0, 75.0), (1.0, 0.0, 0.0, 0.0)]


@pytest.fixture(scope="module")
def columns(gpu):
    nodes = {k: trees.to_product(m()) for k, m in TREES.items()}
    for dim in (2, 3, 4):
        gpu.jit_compile([(n, dim) for n in nodes.values()])
    return nodes


@pytest.mark.parametrize("dim", [2, 3, 4])
@pytest.mark.parametrize("name", sorted(TREES))
def test_columns_match_the_oracle(columns, name, dim):
    oracle = OracleTree(TREES[name]())
    for shape in SHAPES[dim]:
        for step in STEPS:
            off = (-7.5, 3.25, -11.0, 2.0)[:dim]
            got, mm = columns[name].gen_uniform_grid(off, shape, step[:dim], 77)
            ref, rmm = oracle.grid(off, shape, step[:dim], 77)
            assert_parity(got, mm, ref, rmm, label=f"{name} {shape} {step}")


@pytest.mark.parametrize("name", sorted(TREES))
def test_columns_of_extreme_positions(columns, name):
    """Along the column and across it: coordinates where every step or none changes the cell,
    past the int32 cells, infinite and NaN."""
    oracle = OracleTree(TREES[name]())
    for last in (2.0**20, 1.7e7, 3e9, -3e9, 1e30, float("inf"), float("nan")):
        for off in ((0.5, -3.0, last), (last, 2.0, 1.0)):
            got, mm = columns[name].gen_uniform_grid(off, (9, 5, 35), (1.0, 1.0, 1.0), -5)
            ref, rmm = oracle.grid(off, (9, 5, 35), (1.0, 1.0, 1.0), -5)
            assert_parity(got, mm, ref, rmm, label=f"{name} {off}")


@pytest.mark.parametrize("dim", [2, 3, 4])
@pytest.mark.parametrize("name", sorted(TREES))
def test_columns_of_a_batch_match_the_oracle(columns, name, dim):
    """A batch walks grids of every size in columns; a call of its own does so only where that
    is the faster route."""
    oracle = OracleTree(TREES[name]())
    off = (-7.5, 3.25, -11.0, 2.0)[:dim]
    grids = [(shape, step) for shape in SHAPES[dim] for step in STEPS]
    outs = [torch.full((int(np.prod(shape)),), np.nan, device="cuda") for shape, _ in grids]
    kind = {2: fn.KIND_GRID2D, 3: fn.KIND_GRID3D, 4: fn.KIND_GRID4D}[dim]
    fn.gen_batch([fn.make_request(columns[name], kind, out.data_ptr(), 77, shape, off, step[:dim])
                  for out, (shape, step) in zip(outs, grids)])
    for out, (shape, step) in zip(outs, grids):
        ref, rmm = oracle.grid(off, shape, step[:dim], 77)
        assert_parity(out.cpu().numpy(), rmm, ref, rmm, label=f"{name} {shape} {step}")


@pytest.mark.parametrize("name", sorted(TREES))
@pytest.mark.parametrize("shape", [(1003, 1001), (97, 90, 101), (23, 21, 29, 65)])
def test_calls_large_enough_for_columns(columns, name, shape):
    oracle = OracleTree(TREES[name]())
    off, step = (-7.5, 3.25, -11.0, 2.0)[:len(shape)], (1.0, 0.37, -0.9, 1.3)[:len(shape)]
    got, mm = columns[name].gen_uniform_grid(off, shape, step, 5)
    ref, rmm = oracle.grid(off, shape, step, 5)
    assert_parity(got, mm, ref, rmm, label=f"{name} {shape}")
