"""Frames on both sides of the limits at which 2, 4 and 8 warps share a tile (k_pixel's split), in every mode, tile shape
and block size, against the persistent kernel, which never splits (its own parity is tested elsewhere): colours and hit
records byte for byte, pixels outside the dispatched region untouched."""
import numpy as np
import pytest

import woxel_gb300 as wx
from woxel_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SMS = 152
LIMITS = [SMS * 28 >> s for s in (3, 2, 1)]


@pytest.fixture(scope="module")
def grid(cuda_ctx):
    topo = wx.Topology.sphere((0, 0, 0), 64.0, 3.0)
    g = cuda_ctx.build_grid(topo, gpu=True)
    g.set_values(W.sphere_values(topo), 3.0)
    return g


@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("tiles", [1, 3] + [t + d for t in LIMITS for d in (0, 1)])
def test_split_frames(cuda_ctx, grid, mode, tiles):
    import torch

    # 8x4 tiles: `tiles` of them in rows of 19 (and a ragged edge outside the dispatched region)
    per_row = min(tiles, 19)
    rows = -(-tiles // per_row)
    w, h = per_row * 8 + 5, rows * 4 + 3
    st = wx.state_build(eye=(30.0, 40.0, 180.0), target=(5.0, 0, 0), aspect=w / h, fovy=60.0, width=float(w), mode=mode)
    before = cuda_ctx.tuning
    got = []
    try:
        for tune in (dict(kernel=0, tile_width=8, warps_per_block=4), dict(kernel=1, tile_width=8, warps_per_block=4),
                     dict(kernel=1, tile_width=4, warps_per_block=1), dict(kernel=1, tile_width=32, warps_per_block=8)):
            cuda_ctx.set_tuning(**tune)
            a = torch.full((h * w * 4,), 7, dtype=torch.uint8, device="cuda")
            b = torch.full((h * w * 32,), 7, dtype=torch.uint8, device="cuda")
            cuda_ctx.render(grid, st, w, h, a, b, torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            got.append((a.cpu().numpy(), b.cpu().numpy()))
    finally:
        cuda_ctx.set_tuning(**before)
    assert (got[0][0] == 7).any()
    for a, b in got[1:]:
        np.testing.assert_array_equal(a, got[0][0])
        np.testing.assert_array_equal(b, got[0][1])
