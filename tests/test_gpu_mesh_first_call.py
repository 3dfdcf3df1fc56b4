"""Every mesh entry point as the first mesh call of its thread, and after a call that meshes on
the internal lanes: each has to set up the scratch it uses itself."""
import threading

import pytest
import torch

from oracle.tree import N
from tests.trees import to_product

pytestmark = pytest.mark.gpu

SIZE = 12


def _call(fn, kind, node, plane):
    vcap, icap = 24 * SIZE**3, 36 * SIZE**3
    v = [torch.zeros((vcap, 4), device="cuda") for _ in range(2)]
    i = [torch.zeros(icap, dtype=torch.int32, device="cuda") for _ in range(2)]
    bufs = [(v[k].data_ptr(), vcap, i[k].data_ptr(), icap) for k in range(2)]
    if kind == "heightmap":
        res = [fn.build_chunk_mesh_heightmap(plane, SIZE, (32, -16), 11, 40.0, *bufs[0])]
    elif kind in ("dmc", "bloxel"):
        one = fn.build_chunk_mesh_dmc if kind == "dmc" else fn.build_chunk_mesh_bloxel
        res = [one(node, SIZE, (12, -6, 0), 7, 0.0, False, *bufs[0])]
    else:
        res = fn.build_chunk_meshes(kind[:-1], node, SIZE, [(12, -6, 0), (0, -4, 12)], 7, 0.0, False, bufs)
    assert all(r["fits"] and r["vertexCount"] > 0 for r in res)
    return res, torch.cat([t.view(torch.int32).reshape(-1) for t in v + i]).cpu()


@pytest.mark.parametrize("before", [None, "bloxels"])
@pytest.mark.parametrize("kind", ["heightmap", "dmc", "bloxel", "dmcs", "bloxels"])
def test_first_mesh_call_of_a_thread(gpu, kind, before):
    node = to_product(N("Add", LHS=N("FractalFBm", Source=N("Simplex", Feature_Scale=18.0), Octaves=2),
                        RHS=N("Gradient").set("Multiplier", 0.08, 1)))
    plane = to_product(N("FractalFBm", Source=N("Perlin", Feature_Scale=30.0), Octaves=3))
    got = []

    def work():
        if before:
            _call(gpu, before, node, plane)
        got.append(_call(gpu, kind, node, plane))

    thread = threading.Thread(target=work)
    thread.start()
    thread.join()
    assert got, "the call failed in its thread"
    _call(gpu, "bloxel", node, plane)
    _call(gpu, "dmc", node, plane)
    ref, ref_buffers = _call(gpu, kind, node, plane)
    assert got[0][0] == ref
    assert torch.equal(got[0][1], ref_buffers)
