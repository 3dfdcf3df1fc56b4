"""Launches that leave SMs free do not crowd together: back to back, column calls take about as long
as with a full ordering point (a copy of a few bytes) between them, not a multiple of it."""
import pytest
import torch

from tests import trees

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,steps", [((669, 1365), 32), ((669, 1365), 16), ((78, 135, 84), 28)])
def test_column_calls_back_to_back(gpu, count, steps):
    node = trees.to_product(trees.terrain_c2())
    dim = len(count)
    gpu.jit_compile([(node, dim)])
    out = torch.empty(count, device="cuda")
    a, b = torch.zeros(4, device="cuda"), torch.zeros(4, device="cuda")
    stream = torch.cuda.Stream()

    def per_call(between):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(stream):
            for k in range(60):
                if k == 10:
                    start.record()
                node.gen_uniform_grid_device(out.data_ptr(), (0.0,) * dim, count, (1.0,) * dim, k, 0, stream.cuda_stream)
                if between:
                    a.copy_(b, non_blocking=True)
            end.record()
        end.synchronize()
        return start.elapsed_time(end) / 50

    gpu.set_grid_route(gpu.GRID_ROUTE_COLUMNS, steps)
    try:
        ordered, overlapped = (min(per_call(between) for _ in range(5)) for between in (True, False))
    finally:
        gpu.set_grid_route(gpu.GRID_ROUTE_AUTO)
    assert overlapped < 1.4 * ordered, (overlapped, ordered)
