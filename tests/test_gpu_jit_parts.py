"""Specialised modules of several parts (large trees, trees with column kernels): every kernel is found,
right after the compile and in a process that loads the parts from the on-disk cache."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def check(cache, warm):
    import torch

    import fastnoise2_gb300 as fn
    from oracle.oracle import OracleTree
    from tests import trees
    from tests.parity import assert_parity

    fn.jit_set_cache_dir(cache)
    for root, dim in ((trees.fbm_perlin_c1(), 4), (trees.terrain_c2(), 3), (trees.terrain_c2(), 2), (trees.cellular_value_tree(), 3)):
        node, oracle = trees.to_product(root), OracleTree(root)
        before = fn.jit_cache_info()
        fn.jit_compile([(node, dim)])
        after = fn.jit_cache_info()
        assert (after["misses"] - before["misses"], after["hits"] - before["hits"]) == ((2, 0) if warm else (0, 2))
        count, off, step = (13, 6, 9, 11)[:dim], (-3.0, 5.5, 2.0, -7.0)[:dim], (1.0,) * dim
        ref, rmm = oracle.grid(off, count, step, 9)
        kind = {2: fn.KIND_GRID2D, 3: fn.KIND_GRID3D, 4: fn.KIND_GRID4D}[dim]
        for route in (fn.GRID_ROUTE_POINTS, fn.GRID_ROUTE_COLUMNS):
            fn.set_grid_route(route)
            got, mm = node.gen_uniform_grid(off, count, step, 9)
            assert_parity(got, mm, ref, rmm, label=f"{dim} grid {route}")
            out, bmm = torch.empty(ref.size, device="cuda"), np.zeros(2, np.float32)
            fn.gen_batch([fn.make_request(node, kind, out.data_ptr(), 9, count, off, step, minmax=bmm)], sync=True)
            assert_parity(out.cpu().numpy(), (bmm[0], bmm[1]), ref, rmm, label=f"{dim} batch {route}")
            assert fn.batch_info()["specialised"] == 1
            walked = fn.set_grid_route(fn.GRID_ROUTE_AUTO)
            assert walked == (2 if route == fn.GRID_ROUTE_COLUMNS else 0)
        pos = [np.linspace(-9.0, 40.0 + k, 301, dtype=np.float32) for k in range(dim)]
        assert_parity(*node.gen_position_array(pos, off, 9), *oracle.positions(pos, off, 9), label=f"{dim} positions")
        if dim == 4:
            assert_parity(*node.gen_tileable_2d((17, 12), (0.3, 0.2), 9), *oracle.tileable(17, 12, 0.3, 0.2, 9), label="tileable")
        if dim == 3:
            v, i = torch.zeros((30000, 4), device="cuda"), torch.zeros(90000, dtype=torch.int32, device="cuda")
            res = []
            for form in (fn.MESH_DENSITY_SPARSE, fn.MESH_DENSITY_ARRAY):
                old = fn.set_mesh_density_form(form)
                res.append(fn.build_chunk_mesh_dmc(node, 12, (5, -6, 0), 9, 0.3, False, v.data_ptr(), 30000, i.data_ptr(), 90000))
                fn.set_mesh_density_form(old)
            assert res[0] == res[1]


@pytest.mark.gpu
def test_parts_from_the_compiler_and_from_the_cache(gpu, tmp_path):
    for warm in ("1", "0"):
        r = subprocess.run([sys.executable, os.path.abspath(__file__), str(tmp_path), warm], capture_output=True, text=True, timeout=300, cwd=ROOT)
        assert r.returncode == 0, r.stdout + r.stderr
    files = sorted(tmp_path.glob("*.cubin"))
    assert len(files) == 8


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    check(sys.argv[1], sys.argv[2] == "1")
