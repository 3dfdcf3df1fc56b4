"""Tuning a batch that is walked in columns: the point kernels' variants do not run, so none are
built and no choice is made from timing noise.  In a process of its own, since the table of tuned
trees is the process's."""
import os
import subprocess
import sys
import tempfile
from pathlib import Path

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
COUNT = (32, 32, 64)


def _tree_lines(fn, path):
    fn.autotune_save(path)
    return {ln.split()[1]: int(ln.split()[2]) for ln in path.read_text().splitlines() if ln.startswith("tree ")}


def column_trees_keep_their_variant(path):
    import torch

    import fastnoise2_gb300 as fn
    from oracle.tree import N
    from tests.trees import to_product

    nodes = [to_product(N("FractalFBm", Source=N("Perlin", Feature_Scale=71.5), Octaves=3)), to_product(N("CellularValue", Feature_Scale=63.5))]
    fn.jit_compile([(n, 3) for n in nodes])
    outs = [torch.empty(COUNT, device="cuda") for _ in range(64)]
    reqs = [fn.make_request(nodes[k % 2], fn.KIND_GRID3D, o.data_ptr(), k, COUNT, (32.0 * k, 0.0, -7.0)) for k, o in enumerate(outs)]
    torch.cuda.synchronize()
    fn.set_grid_route(fn.GRID_ROUTE_COLUMNS)
    built = fn.jit_cache_info()["misses"]
    fn.autotune_batch(reqs)
    assert fn.jit_cache_info()["misses"] == built            # no variant was compiled
    tuned = _tree_lines(fn, path)
    assert sorted(tuned.values()) == [0, 0]
    # an earlier choice stays
    path.write_text("".join(f"tree {h} 3 0 0 0 1.0\n" for h in tuned))
    fn.autotune_load(path)
    fn.autotune_batch(reqs)
    assert _tree_lines(fn, path) == {h: 3 for h in tuned}
    # a tuned number of CTAs per SM, which goes with tiles of points, does not bind columns
    fn.gen_batch(reqs)
    free = fn.batch_info()["ctas"]
    fn.autotune_save(path)
    signatures = [ln.split() for ln in path.read_text().splitlines() if not ln.startswith("tree ")]
    assert signatures
    for ctas in (1, 0):
        path.write_text("".join(f"{ln[0]} 2048 {ctas} 1.0\n" for ln in signatures))
        fn.autotune_load(path)
        fn.gen_batch(reqs)
        assert fn.batch_info()["ctas"] == free > 0
    # as points they are tuned
    fn.set_grid_route(fn.GRID_ROUTE_POINTS)
    fn.autotune_batch(reqs)
    assert fn.jit_cache_info()["misses"] > built


@pytest.mark.gpu
def test_column_trees_keep_their_variant(gpu):
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    with tempfile.TemporaryDirectory() as d:
        column_trees_keep_their_variant(Path(d) / "tune.txt")
