"""Uploaded views with tile distances around 2^24 (which the integer size of the march loop does not cover) and N5 nodes beyond
[-4096, 4096)^3, where a ray ends whatever lies there: every kernel against the oracle, bit for bit."""
import numpy as np
import pytest

import woxel_gb300 as wx
from parity import compare, gpu_render, oracle_render

pytestmark = pytest.mark.gpu

KERNELS = [dict(kernel=1, rays_per_lane=1), dict(kernel=0, rays_per_lane=1), dict(kernel=1, rays_per_lane=2),
           dict(kernel=1, rays_per_lane=4), dict(kernel=1, rays_per_lane=8)]


def far_view(big):
    """Voxels on both sides of x = 4096, and some N5 tiles (of every N5) with the distance `big`."""
    rng = np.random.default_rng(3)
    ijk = np.concatenate([rng.integers(-200, 200, size=(1500, 3)), rng.integers(-60, 60, size=(1500, 3)) + [4150, 0, 0],
                          rng.integers(-40, 40, size=(500, 3)) + [4040, 0, 0]])
    topo = wx.Topology.from_voxels(ijk.astype(np.int32))
    view = topo.view()
    n5 = topo.counts[0]
    side = view["dims"][0][0]
    d = side >> 5
    bits = np.unpackbits(view["kids5"].view(np.uint8), bitorder="little").reshape(n5, -1)
    node, slot = np.nonzero(bits == 0)
    pick = rng.choice(node.size, node.size // 50, replace=False)
    node, slot = node[pick], slot[pick]
    x, y, z = slot >> 10, (slot >> 5) & 31, slot & 31
    a = view["atlas"][0].copy()
    a[((z + (node // (d * d) << 5)) * side + y + (node // d % d << 5)) * side + x + (node % d << 5)] = big
    view["atlas"][0] = a
    return view


@pytest.mark.parametrize("tune", KERNELS, ids=lambda t: f"kernel{t['kernel']}x{t['rays_per_lane']}")
@pytest.mark.parametrize("big", [2 ** 24 - 1, 2 ** 24, 2 ** 31 - 1])
def test_rays_end_at_the_box(cuda_ctx, big, tune):
    view = far_view(big)
    g = cuda_ctx.upload_view(view)
    before = cuda_ctx.tuning
    cuda_ctx.set_tuning(**tune)
    try:
        beyond = 0
        for k, (eye, target) in enumerate((((3900.0, 20.0, 30.0), (4150.0, 0, 0)), ((4020.0, -3.0, 2.0), (4200.0, 5.0, 1.0)),
                                           ((4400.0, 30.0, 20.0), (4100.0, 0, 0)), ((300.0, 200.0, -250.0), (0, 0, 0)))):
            for mode in (0, 2, 3):
                st = wx.state_build(eye=eye, target=target, aspect=1.0, fovy=60.0, width=96.0, mode=mode)
                rg, hg = gpu_render(cuda_ctx, g, st, 96, 96)
                ro, ho = oracle_render(view, st, 96, 96)
                compare(rg, hg, ro, ho, label=f"big {big} eye {k} mode {mode}")
                beyond += int((ho["p"][..., 0] > 4096).sum())
        assert beyond > 1000  # rays that end past the face
    finally:
        cuda_ctx.set_tuning(**before)
