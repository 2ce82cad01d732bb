"""The zero-crossing search's cell and leaf reuse against the oracle, bit for bit: rays along and across leaf, N4 and N5
borders, values outside the box of the dense N5 table, active tiles beside leaves, and a voxel-sized step pattern in
which every sample changes its cell."""
import numpy as np
import pytest

import woxel_gb300 as wx
from parity import compare, gpu_render, oracle_render, oracle_view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("corner", [0, 8, 128, 4096, -4096, 4000])
def test_noise_values_at_borders(cuda_ctx, corner):
    rng = np.random.default_rng(abs(corner) + 5)
    ijk = np.stack(np.mgrid[0:26, 0:26, 0:26], -1).reshape(-1, 3) + corner - 13
    topo = wx.Topology.from_voxels(ijk[rng.random(ijk.shape[0]) < 0.15].astype(np.int32))
    if corner == 128:
        m = topo.masks()
        m["vals4"][1] |= np.uint32(1 << 3)
        topo = wx.Topology.from_masks(m)
    values = rng.uniform(-0.6, 3.0, topo.counts[2] * 512).astype(np.float32)
    view = dict(oracle_view(topo), values=values, band=3.0)
    grid = cuda_ctx.build_grid(topo)
    grid.set_values(values, 3.0)
    crossings = 0
    c = np.array([corner] * 3, float)
    for off in ([60.0, 25.0, 40.0], [0.0, 0.0, 70.0], [-50.0, 0.5, 0.25], [1.0, 2.0, 3.0]):
        st = wx.state_build(eye=tuple(c + off), target=tuple(c + [0.5, 0.25, 0.0]), aspect=1.0, fovy=50.0, width=96.0, mode=5)
        rg, hg = gpu_render(cuda_ctx, grid, st, 96, 96)
        ro, ho = oracle_render(view, st, 96, 96)
        compare(rg, hg, ro, ho, label=f"corner {corner} eye {off}")
        np.testing.assert_array_equal(hg["reserved"], ho["reserved"])
        crossings += int((hg["shadow"] & 1).sum())
    assert crossings > 0 or abs(corner) > 4000
