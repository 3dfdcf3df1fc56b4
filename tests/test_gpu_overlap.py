"""Per-call launches overlap the tail of the stream's previous kernel; what they read and write
must still be ordered after it: positions written just before, one output buffer written by
consecutive calls, the min/max workspace they share, on a stream and in a captured graph."""
import numpy as np
import pytest

from tests import trees

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(gpu):
    torch = pytest.importorskip("torch")
    nodes = {"simplex": trees.to_product(trees.simplex_c0()), "fbm": trees.to_product(trees.fbm_perlin_c1()),
             "cells": trees.to_product(trees.cellular_value_tree())}
    gpu.jit_compile([(n, 3) for n in nodes.values()])
    return torch, nodes


@pytest.mark.parametrize("count", [(5, 4, 3), (32, 32, 32), (96, 80, 70)])
@pytest.mark.parametrize("name", ["simplex", "fbm", "cells"])
def test_consecutive_calls_share_buffers(setup, name, count):
    torch, nodes = setup
    total = int(np.prod(count))
    stream = torch.cuda.Stream()
    out = torch.empty(total, device="cuda")
    rounds = 40
    mm = torch.empty((rounds, 2), device="cuda")
    kept = []
    with torch.cuda.stream(stream):
        for k in range(rounds):
            nodes[name].gen_uniform_grid_device(out.data_ptr(), (0.0, 3.0, -7.0), count, (1.0,) * 3, k, mm[k].data_ptr(), stream.cuda_stream)
            if k % 8 == 7:
                kept.append((k, out.clone()))
    stream.synchronize()
    for k in range(rounds):
        ref, rmm = nodes[name].gen_uniform_grid((0.0, 3.0, -7.0), count, (1.0,) * 3, k)
        assert (float(mm[k, 0]), float(mm[k, 1])) == rmm, k
        for j, got in kept:
            if j == k:
                assert np.array_equal(got.cpu().numpy().view(np.uint32), ref.view(np.uint32)), k


def test_positions_written_just_before(setup):
    torch, nodes = setup
    n = 200_000
    stream = torch.cuda.Stream()
    base = [torch.rand(n, device="cuda") * 100 for _ in range(3)]
    torch.cuda.synchronize()
    outs, pos = [], [torch.empty(n, device="cuda") for _ in range(3)]
    with torch.cuda.stream(stream):
        for k in range(12):
            for p, b in zip(pos, base):
                torch.add(b, float(k), out=p)
            out = torch.empty(n, device="cuda")
            nodes["simplex"].gen_position_array_device(out.data_ptr(), n, [p.data_ptr() for p in pos], (0.0,) * 3, 9, 0, stream.cuda_stream)
            outs.append(out)
    stream.synchronize()
    for k, out in enumerate(outs):
        ref, _ = nodes["simplex"].gen_position_array([(b + float(k)).cpu().numpy() for b in base], (0.0,) * 3, 9)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32)), k


@pytest.mark.parametrize("n", [4096, 30_720, 300_032])
def test_positions_rewritten_by_the_kernel_between(setup, n):
    """A grid call writes the array that the position calls before and after it read."""
    torch, nodes = setup
    stream = torch.cuda.Stream()
    steps = 30
    x, rest = torch.zeros(n, device="cuda"), [torch.rand(n, device="cuda") * 50 for _ in range(2)]
    outs = [torch.empty(n, device="cuda") for _ in range(steps)]
    torch.cuda.synchronize()
    for k in range(steps):
        nodes["fbm"].gen_uniform_grid_device(x.data_ptr(), (0.0,) * 3, (n // 32, 32, 1), (9.0,) * 3, k, 0, stream.cuda_stream)
        nodes["cells"].gen_position_array_device(outs[k].data_ptr(), n, [x.data_ptr(), rest[0].data_ptr(), rest[1].data_ptr()],
                                                 (0.0,) * 3, 9, 0, stream.cuda_stream)
    stream.synchronize()
    for k in range(steps):
        px, _ = nodes["fbm"].gen_uniform_grid((0.0,) * 3, (n // 32, 32, 1), (9.0,) * 3, k)
        ref, _ = nodes["cells"].gen_position_array([px] + [r.cpu().numpy() for r in rest], (0.0,) * 3, 9)
        assert np.array_equal(outs[k].cpu().numpy().view(np.uint32), ref.view(np.uint32)), k


def test_captured_calls_replay(setup):
    torch, nodes = setup
    count = (40, 33, 20)
    total = int(np.prod(count))
    stream = torch.cuda.Stream()
    a, b = torch.empty(total, device="cuda"), torch.empty(total, device="cuda")
    mm = torch.empty((2, 2), device="cuda")

    def calls():
        nodes["fbm"].gen_uniform_grid_device(a.data_ptr(), (0.0,) * 3, count, (1.0,) * 3, 5, mm[0].data_ptr(), stream.cuda_stream)
        b.copy_(a, non_blocking=True)
        nodes["simplex"].gen_uniform_grid_device(a.data_ptr(), (0.0,) * 3, count, (1.0,) * 3, 6, mm[1].data_ptr(), stream.cuda_stream)

    with torch.cuda.stream(stream):
        calls()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        calls()
        graph.capture_end()
    a.zero_(), b.zero_(), mm.zero_()
    torch.cuda.synchronize()
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    for got, m, name, seed in ((b, mm[0], "fbm", 5), (a, mm[1], "simplex", 6)):
        ref, rmm = nodes[name].gen_uniform_grid((0.0,) * 3, count, (1.0,) * 3, seed)
        assert np.array_equal(got.cpu().numpy().view(np.uint32), ref.view(np.uint32)), name
        assert (float(m[0]), float(m[1])) == rmm
