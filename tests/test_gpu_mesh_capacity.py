"""Dual marching cubes into buffers of which one is too small: nothing is written, and counts,
heights and min/max are those of a chunk that fits."""
import pytest
import torch

from oracle.tree import N
from tests.trees import to_product

pytestmark = pytest.mark.gpu

SIZE = 16


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("chunks", [1, 3])
def test_one_buffer_too_small(gpu, chunks, sparse):
    fn = gpu
    node = to_product(N("Add", LHS=N("FractalFBm", Source=N("Simplex", Feature_Scale=18.0), Octaves=2),
                        RHS=N("Gradient").set("Multiplier", 0.08, 1)))
    fn.jit_compile([(node, 3)])
    vcap, icap = 4 * (SIZE + 1)**3, 18 * SIZE**3
    positions = [(16 * k, -8, 16) for k in range(chunks)]

    def mesh(vc, ic):
        v = torch.full((chunks, vcap, 4), -7.0, device="cuda")
        i = torch.full((chunks, icap), -7, dtype=torch.int32, device="cuda")
        bufs = [(v[k].data_ptr(), vc, i[k].data_ptr(), ic) for k in range(chunks)]
        if chunks == 1:
            return [fn.build_chunk_mesh_dmc(node, SIZE, positions[0], 7, 0.0, False, *bufs[0])], v, i
        return fn.build_chunk_meshes("dmc", node, SIZE, positions, 7, 0.0, False, bufs), v, i

    before = fn.set_mesh_density_form(fn.MESH_DENSITY_SPARSE if sparse else fn.MESH_DENSITY_ARRAY)
    try:
        whole, v, i = mesh(vcap, icap)
        assert all(r["fits"] and r["vertexCount"] > 0 for r in whole)
        need_v, need_i = max(r["vertexCount"] for r in whole), max(r["indexCount"] for r in whole)
        for vc, ic in ((vcap, 6), (8, icap), (vcap, 0), (0, icap), (need_v, min(r["indexCount"] for r in whole) - 1)):
            res, v, i = mesh(vc, ic)
            for r, ref in zip(res, whole):
                assert not r["fits"]
                assert {k: r[k] for k in r if k != "fits"} == {k: ref[k] for k in ref if k != "fits"}
            assert bool((v == -7.0).all()) and bool((i == -7).all()), (vc, ic)
        res, v, i = mesh(need_v, need_i)
        assert res == whole
    finally:
        fn.set_mesh_density_form(before)
