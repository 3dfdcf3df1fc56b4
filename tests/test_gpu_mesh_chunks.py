"""Dual marching cubes of many chunks in one call: every chunk's mesh is the one of a call of its
own, bit for bit, for chunk counts below, at and above what is meshed together (32 small ones),
sizes around a warp and a scan tile, chunks without a surface and buffers that are too small."""
import pytest
import torch

from oracle.tree import N
from tests.trees import to_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,count", [(1, 3), (2, 33), (7, 32), (31, 5), (33, 9), (13, 70), (96, 21)])
@pytest.mark.parametrize("up_z", [False, True])
def test_many_chunks_equal_single_calls(gpu, size, count, up_z):
    fn = gpu
    node = to_product(N("Add", LHS=N("FractalFBm", Source=N("Simplex", Feature_Scale=19.0), Octaves=2),
                        RHS=N("Gradient").set("Multiplier", 0.03, 1)))
    vcap, icap = size**3 + 512, 3 * size**3 + 1024
    positions = [((k - 3) * size, ((k % 4) - 2) * size // 2 if k % 5 else 40 * size, -k * size // 3) for k in range(count)]
    verts = torch.zeros((count, vcap, 4), device="cuda")
    index = torch.zeros((count, icap), dtype=torch.int32, device="cuda")
    caps = [(0, 0) if k % 7 == 6 else (vcap, icap) for k in range(count)]
    res = fn.build_chunk_meshes("dmc", node, size, positions, 77, 0.0, up_z,
                                [(verts[k].data_ptr(), caps[k][0], index[k].data_ptr(), caps[k][1]) for k in range(count)])
    v1, i1 = torch.zeros((vcap, 4), device="cuda"), torch.zeros(icap, dtype=torch.int32, device="cuda")
    surfaces = 0
    for k, p in enumerate(positions):
        v1.zero_()
        i1.zero_()
        one = fn.build_chunk_mesh_dmc(node, size, p, 77, 0.0, up_z, v1.data_ptr(), caps[k][0], i1.data_ptr(), caps[k][1])
        for key in ("vertexCount", "indexCount", "minAirY", "maxSolidY", "minMax"):
            assert res[k][key] == one[key], (k, key)
        assert torch.equal(verts[k].view(torch.int32), v1.view(torch.int32)), k
        assert torch.equal(index[k], i1), k
        surfaces += one["vertexCount"] > 0
    assert surfaces or size < 7
