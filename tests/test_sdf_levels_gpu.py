"""The breadth-first distance steps of the GPU build (sdf.cu: k_sdf_levels) against the host sweeps, every pool word:
remainders of three leaves a warp, distances carried over many inactive leaves and across N4 and N5 borders (where the
DFS order of neighbours differs from the order of their coordinates), and distances on both sides of a leaf byte's 255."""
import numpy as np
import pytest

import woxel_gb300 as wx

pytestmark = pytest.mark.gpu


def check(ctx, origins, masks):
    topo = wx.Topology.from_leaves(np.asarray(origins, np.int32), masks)
    a, b = ctx.build_grid(topo), ctx.build_grid(topo, gpu=True)
    pa, pb = a.pools(), b.pools()
    for k in ("slot5", "slot4", "leaf", "ovf"):
        np.testing.assert_array_equal(pa[k], pb[k], err_msg=k)
    assert a.info == b.info
    return pb


@pytest.mark.parametrize("n", [1, 2, 3, 4, 31])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_rows_of_leaves(cuda_ctx, n, axis):
    o = np.zeros((n, 3), int)
    o[:, axis] = 8 * np.arange(n) - 8 * (n // 2)
    m = np.zeros((n, 8), np.uint64)
    m[0, 3] = 1 << 17
    check(cuda_ctx, o, m)


@pytest.mark.parametrize("corner", [0, 128, 4096, -4096])
@pytest.mark.parametrize("keep", [1.0, 0.9])
def test_inactive_blocks_across_borders(cuda_ctx, corner, keep):
    rng = np.random.default_rng(int(abs(corner) * 2 + keep * 10))
    o = np.stack(np.mgrid[0:9, 0:8, 0:7], -1).reshape(-1, 3) * 8 + corner - 32
    o = o[rng.random(o.shape[0]) < keep]
    m = np.zeros((o.shape[0], 8), np.uint64)
    m[rng.integers(o.shape[0], size=3), rng.integers(8, size=3)] = np.uint64(1) << rng.integers(64, size=3).astype(np.uint64)
    check(cuda_ctx, o, m)


def test_distances_around_a_byte(cuda_ctx):
    n = 64  # the centre of the cube is 256 cells from its faces
    o = np.stack(np.mgrid[0:n, 0:n, 0:n], -1).reshape(-1, 3) * 8 - 8 * 31
    p = check(cuda_ctx, o, np.zeros((o.shape[0], 8), np.uint64))
    assert p["leaf"].max() == 255 and set(p["ovf"][:, 1]) == {255, 256} and (p["leaf"] == 254).any()


def test_no_nodes(cuda_ctx):
    check(cuda_ctx, np.zeros((0, 3), int), np.zeros((0, 8), np.uint64))
