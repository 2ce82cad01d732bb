"""Frames of different modes queued back to back into shared outputs: each mode has a kernel of its own, all launched
as programmatic dependents, and the glossy one stores a pixel's hit record before its later rays are traced."""
import itertools

import numpy as np
import pytest

import woxel_gb300 as wx
from woxel_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", list(itertools.permutations([3, 4, 5])))
def test_modes_share_outputs(cuda_ctx, order):
    import torch

    topo = wx.Topology.sphere((0, 0, 0), 64.0, 3.0)
    grid = cuda_ctx.build_grid(topo, gpu=True)
    grid.set_values(W.sphere_values(topo), 3.0)
    w, h = 328, 244
    states = [wx.state_build(eye=(40.0 * i, 30.0, 190.0), target=(0, 0, 0), aspect=w / h, fovy=60.0, width=float(w), mode=m)
              for i, m in enumerate(order)]

    def frame(st, rgba, hits):
        cuda_ctx.render(grid, st, w, h, rgba, hits, stream=torch.cuda.current_stream().cuda_stream)

    def buf(n):
        return torch.zeros(w * h * n, dtype=torch.uint8, device="cuda")

    alone = []
    for st in states:
        a, b = buf(4), buf(32)
        frame(st, a, b)
        torch.cuda.synchronize()
        alone.append((a.cpu().numpy(), b.cpu().numpy()))
    for last in range(3):
        a, b = buf(4), buf(32)
        for rep in range(8):
            for st in states[: last + 1]:
                frame(st, a, b)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(a.cpu().numpy(), alone[last][0])
        np.testing.assert_array_equal(b.cpu().numpy(), alone[last][1])
    grid.release()
