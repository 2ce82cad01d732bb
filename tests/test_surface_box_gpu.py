"""The zero-crossing search across the faces of the box [-4096, 4096)^3, where the dense table of N5 slots ends and the
search takes the root table: against the oracle, bit for bit, with eyes inside the box and crossings in cells that reach beyond it."""
import numpy as np
import pytest

import woxel_gb300 as wx
from parity import compare, gpu_render, oracle_render, oracle_view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("face", [4096, -4096])
@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1, 2)])
def test_crossings_beyond_the_box(cuda_ctx, face, axes):
    sign = 1 if face > 0 else -1
    centre = np.array([face if a in axes else 40 for a in range(3)])
    rng = np.random.default_rng(abs(face) + 7 * len(axes) + axes[0] + sign)
    ijk = np.stack(np.mgrid[0:26, 0:26, 0:26], -1).reshape(-1, 3) - 13 + centre
    topo = wx.Topology.from_voxels(ijk[rng.random(ijk.shape[0]) < 0.15].astype(np.int32))
    values = rng.uniform(-0.3, 3.0, topo.counts[2] * 512).astype(np.float32)
    view = dict(oracle_view(topo), values=values, band=3.0)
    grid = cuda_ctx.build_grid(topo)
    grid.set_values(values, 3.0)
    inward = np.array([-sign if a in axes else 0 for a in range(3)], float)
    crossings = beyond = 0
    for dist, off in ((30.0, (3.0, 1.5, -2.0)), (9.0, (0.5, -4.0, 2.5)), (3.5, (-2.25, 1.0, 0.75))):
        eye = centre + inward * dist + np.where(inward == 0, off, 0.0)
        st = wx.state_build(eye=tuple(eye), target=tuple(centre - 4 * inward + 0.25), up=(0.3, 0.5, 0.7), aspect=1.0, fovy=60.0,
                            width=96.0, mode=5)
        rg, hg = gpu_render(cuda_ctx, grid, st, 96, 96)
        ro, ho = oracle_render(view, st, 96, 96)
        compare(rg, hg, ro, ho, label=f"face {face} axes {axes} distance {dist}")
        np.testing.assert_array_equal(hg["reserved"], ho["reserved"])
        hit = (ho["shadow"] & 1) == 1
        t, ts = ho["t"][hit].astype(np.float64), ho["reserved"][hit]
        ts = (ts if ts.dtype == np.float32 else ts.view(np.float32)).astype(np.float64)
        e = eye.astype(np.float32).astype(np.float64)
        cell = np.floor(e + (ho["p"][hit] - e) * (ts / np.maximum(t, 1e-6))[:, None])  # eye + ts * direction
        out = (cell < -4096) | (cell + 1 >= 4096)
        crossings += int(hit.sum())
        beyond += int(out.any(axis=1).sum())
    assert crossings > 100 and beyond > 20, (crossings, beyond)
