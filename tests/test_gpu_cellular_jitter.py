"""Cellular noise with jitters up to the largest floats, on grids large enough for a column kernel:
where every cell's distance overflows, the initial result stays, as in the oracle."""
import pytest

from oracle.oracle import OracleTree
from oracle.tree import N
from tests import trees
from tests.parity import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jitter", [1e9, -1.0e9, 2e18, 5e19, -1e25, 3.4e38])
@pytest.mark.parametrize("kind", ["CellularValue", "CellularDistance", "CellularLookup"])
def test_large_jitters_match_the_oracle(gpu, kind, jitter):
    root = N(kind, Feature_Scale=40.0, Grid_Jitter=jitter)
    if kind == "CellularLookup":
        root.set("Lookup", N("Perlin", Feature_Scale=30.0))
    node, oracle = trees.to_product(root), OracleTree(root)
    gpu.jit_compile([(node, d) for d in (2, 3)])
    for count in ((96, 64, 80), (640, 512)):
        off = (-7.5, 3.25, -11.0)[:len(count)]
        got, mm = node.gen_uniform_grid(off, count, (1.0,) * len(count), 77)
        ref, rmm = oracle.grid(off, count, (1.0,) * len(count), 77)
        assert_parity(got, mm, ref, rmm, label=f"{kind} {jitter} {count}")
