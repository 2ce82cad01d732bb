"""The march loop's own rules (wx_device.cuh: hdda) where they can go wrong.

On the CPU: floor((floor(p) + 0.5) * y) for any y within 2 ulp of 1/size is the shader's
floor(p / size) (a correctly rounded FP32 quotient), over the coordinates next to every integer of
the box and the sizes of every level. Exact whole numbers, so no tolerance.

On the GPU, against the oracle, bit for bit: rays that leave the loop or never enter it (eyes on and
beyond the box's faces, coordinates around -2^-64, -0 and 0), missing N5 nodes beside present ones,
N5 nodes outside the box, and tile distances around 2^24.
"""
from fractions import Fraction

import numpy as np
import pytest

import woxel_gb300 as wx
from parity import compare, gpu_render, oracle_render, oracle_view


def _sizes() -> np.ndarray:
    rng = np.random.default_rng(1)
    dist = np.concatenate([np.arange(1, 60), rng.integers(60, 4097, 40), [4095, 4096, 4097, 65535, 2 ** 24 - 1]])
    return np.unique(np.concatenate([dist * s for s in (1, 8, 128)] + [np.array([4096])])).astype(np.float32)


def test_integer_floor_equals_the_rounded_quotient():
    x = np.arange(-4096, 4097, dtype=np.float64)
    f32 = np.float32
    lo = x.astype(f32)
    hi = np.nextafter((x + 1).astype(f32), f32(-np.inf))  # the last float of the voxel
    p = np.concatenate([lo, np.nextafter(lo, f32(np.inf)), hi, (lo + f32(4e-4)).astype(f32), (lo + f32(0.5)).astype(f32)])
    p = p[~((p < 0) & (p > -2.0 ** -64)) & (p <= 4096)]
    xi = np.floor(p.astype(np.float64))
    for size in _sizes():
        want = np.floor(p / size)  # FP32 division, correctly rounded
        y0 = f32(1) / size
        for y in (y0, np.nextafter(y0, f32(0)), np.nextafter(y0, f32(1e9)), np.nextafter(np.nextafter(y0, f32(0)), f32(0))):
            # one FMA: (x + 0.5) * y is exact in FP64 (14 + 24 bits), then rounded once
            got = np.floor(((xi + 0.5) * np.float64(y)).astype(f32))
            bad = np.nonzero(got != want)[0]
            assert bad.size == 0, f"size {size}: p = {p[bad[:3]]!r}: {got[bad[:3]]} vs {want[bad[:3]]}"


def _add_rd(p: np.float32, m: int) -> np.float32:
    """p + m rounded down to FP32, from the exact sum."""
    exact = Fraction(float(p)) + m
    r = np.float32(float(exact))
    while Fraction(float(r)) > exact:
        r = np.nextafter(r, np.float32(-np.inf))
    return r


def test_floor_by_the_adder():
    """RD(p + 12587008) has the bits 0x4B400000 + floor(p) + 4096 for p in the box, and other bits outside it."""
    f32 = np.float32
    x = np.arange(-4098, 4099, dtype=np.float64).astype(f32)
    p = np.concatenate([x, np.nextafter(x, f32(-np.inf)), np.nextafter(x, f32(np.inf)),
                        np.array([-1e-30, 1e-30, -2.0 ** -126, 8192, -8192, 1e9, -1e9, 1.2e7, -1.2e7], f32)])
    s = np.array([_add_rd(v, 12587008) for v in p], f32)
    off = s.view(np.uint32).astype(np.int64) - 0x4B400000
    inside = (p >= -4096) & (p < 4096)
    np.testing.assert_array_equal(off[inside], np.floor(p[inside]).astype(np.int64) + 4096)
    assert not ((off[~inside] >= 0) & (off[~inside] < 8192)).any()


EYES = [(0.0, 0.0, 300.0), (-0.0, 20.0, 300.0), (-1e-30, 30.0, 300.0), (1e-30, -1e-30, -300.0), (-2.0 ** -64, 9.0, 250.0),
        (-(2.0 ** -63), 9.0, 250.0), (4096.0, 10.0, 300.0), (-4096.0, 10.0, 300.0), (4095.9998, 4096.0, 4096.0),
        (-4096.0005, 0.5, 0.5), (5000.0, 10.0, 20.0), (3.5, 4.5, 5.5), (-1e-42, -1e-42, 700.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("grid", ["octants", "one", "beyond"])
def test_rays_at_the_edges_of_the_loop(cuda_ctx, grid, kernel):
    """octants: all eight N5s; one: seven of them missing; beyond: N5s outside the box as well."""
    cube = np.stack(np.mgrid[0:30, 0:30, 0:30], -1).reshape(-1, 3) - 15
    ijk = {"octants": np.concatenate([cube, cube * 9, cube + [200, 0, 100], cube * [1, 1, 4] - [0, 60, 900]]),
           "one": np.concatenate([cube + 40, cube + [300, 200, 100]]),
           "beyond": np.concatenate([cube, cube + [4100, 0, 0], cube + [5000, 10, 20], cube - [4200, 0, 0]])}[grid]
    topo = wx.Topology.from_voxels(ijk.astype(np.int32))
    view, g = oracle_view(topo), cuda_ctx.build_grid(topo)
    before = cuda_ctx.tuning
    cuda_ctx.set_tuning(kernel=kernel)
    try:
        for k, eye in enumerate(EYES):
            for mode, target in ((3, (0.0, 0.0, 0.0)), (2, (30.0, 25.0, -40.0))):
                st = wx.state_build(eye=eye, target=target, aspect=1.0, fovy=50.0, width=64.0, mode=mode)
                rg, hg = gpu_render(cuda_ctx, g, st, 64, 64)
                ro, ho = oracle_render(view, st, 64, 64)
                compare(rg, hg, ro, ho, label=f"{grid} eye {k} mode {mode}")
    finally:
        cuda_ctx.set_tuning(**before)


@pytest.mark.gpu
@pytest.mark.parametrize("far", [-4198400, -12587008, -4198400 - 2 ** 21, -8392704])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_far_eyes(cuda_ctx, far, axis):
    """Eyes so far out along one axis that their floor word's high bits are a part of the box's (or all clear),
    with the other two coordinates in the box: a ray is in the box only if each of its coordinates is."""
    cube = np.stack(np.mgrid[0:30, 0:30, 0:30], -1).reshape(-1, 3) - 15
    for extra in ([0, 0, 0], [5000, 10, 20]):
        topo = wx.Topology.from_voxels(np.concatenate([cube, cube * 9, cube + extra]).astype(np.int32))
        view, g = oracle_view(topo), cuda_ctx.build_grid(topo)
        for dist, mode in ((100.0, 3), (700.0, 2)):
            eye, target = [3.5, 4.5, 5.5], [3.5, 4.5, 5.5]
            eye[axis], target[axis] = far + 4096 - dist, far + 4096 + 1000.0
            st = wx.state_build(eye=tuple(eye), target=tuple(target), up=(0.3, 0.5, 0.7), aspect=1.0, fovy=60.0, width=64.0, mode=mode)
            rg, hg = gpu_render(cuda_ctx, g, st, 64, 64)
            ro, ho = oracle_render(view, st, 64, 64)
            compare(rg, hg, ro, ho, label=f"far {far} axis {axis} mode {mode}")


@pytest.mark.gpu
@pytest.mark.parametrize("big", [2 ** 24 - 1, 2 ** 24, 2 ** 24 + 1, 2 ** 31 - 1])
def test_large_tile_distances(cuda_ctx, big):
    """Tiles of a hand-made view with distances around the limit of the loop's integer size."""
    rng = np.random.default_rng(13)
    topo = wx.Topology.from_voxels(rng.integers(-200, 200, size=(2000, 3)).astype(np.int32))
    view = topo.view()
    n5, n4, _ = topo.counts
    for lvl, (words, log2) in enumerate(((view["kids5"], 5), (view["kids4"], 4))):
        a, side = view["atlas"][lvl].copy(), view["dims"][lvl][0]
        n, d = (n5, n4)[lvl], side >> log2
        bits = np.unpackbits(words.view(np.uint8), bitorder="little").reshape(n, -1)
        node, slot = np.nonzero(bits == 0)
        pick = rng.choice(node.size, node.size // 3, replace=False)
        node, slot, m = node[pick], slot[pick], (1 << log2) - 1
        x, y, z = slot >> (2 * log2), (slot >> log2) & m, slot & m
        x, y, z = x + (node % d << log2), y + (node // d % d << log2), z + (node // (d * d) << log2)
        a[(z * side + y) * side + x] = big
        view["atlas"][lvl] = a
    g = cuda_ctx.upload_view(view)
    for eye, mode in (((260.0, 150.0, -300.0), 2), ((5.0, 3.0, 2.0), 3), ((2500.0, -1500.0, 900.0), 0)):
        st = wx.state_build(eye=eye, target=(0, 0, 0), aspect=1.0, fovy=60.0, width=96.0, mode=mode)
        rg, hg = gpu_render(cuda_ctx, g, st, 96, 96)
        ro, ho = oracle_render(view, st, 96, 96)
        compare(rg, hg, ro, ho, label=f"big {big} mode {mode}")


@pytest.mark.gpu
@pytest.mark.parametrize("target", [(1, 1, 1), (-1, 1, 1), (1, -1, 1), (-1, -1, 1), (1, 1, -1), (-1, 1, -1), (1, -1, -1),
                                    (-1, -1, -1), (0, 1, 0.02), (1, 0, 0.02), (0.02, 0, 1)])
def test_sign_patterns(cuda_ctx, target):
    """A loop per sign pattern of the directions, and tiles whose rays differ in it (views along an axis)."""
    rng = np.random.default_rng(7)
    topo = wx.Topology.from_voxels(rng.integers(-250, 250, size=(4000, 3)).astype(np.int32))
    view, g = oracle_view(topo), cuda_ctx.build_grid(topo)
    for eye, fovy, mode in (((3.0, -5.0, 7.0), 40.0, 3), (tuple(-300.0 * c for c in target), 80.0, 2)):
        st = wx.state_build(eye=eye, target=tuple(e + 100.0 * c for e, c in zip(eye, target)), aspect=1.5, fovy=fovy,
                            up=(0.0, 0.3, 1.0), width=120.0, mode=mode)
        rg, hg = gpu_render(cuda_ctx, g, st, 120, 80)
        ro, ho = oracle_render(view, st, 120, 80)
        compare(rg, hg, ro, ho, label=f"{target} mode {mode}")
