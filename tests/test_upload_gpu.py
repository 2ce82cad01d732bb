"""The drop-in upload's packing (pack.cu) where it can go wrong: node counts that do not fill a row, a layer or a group of
eight leaves, atlases that are not cubes, and one larger than the upload's buffer. The pools must equal those of the
native build of the same topology, word for word; texels outside the nodes hold a value no pool may contain."""
import numpy as np
import pytest

import woxel_gb300 as wx

pytestmark = pytest.mark.gpu
JUNK = 0x00DEAD00


def relayout(view, counts, blocks):
    """The view with level l's nodes in blocks[l] = (columns, rows, layers); the shader takes the node's place from the
    width (N4, leaves) or the height (N5), so rows >= columns there."""
    out = dict(view, atlas=[], dims=[])
    for l, log2 in enumerate((5, 4, 3)):
        D, side = 1 << log2, view["dims"][l][0]
        a = view["atlas"][l].reshape(side, side, side)
        d = side >> log2
        bx, by, bz = blocks[l]
        e = by if l == 0 else bx
        t = np.full((bz * D, by * D, bx * D), JUNK, np.uint32)
        for i in range(counts[l]):
            src = a[i // (d * d) * D:, i // d % d * D:, i % d * D:][:D, :D, :D]
            t[i // (e * e) * D:, i // e % e * D:, i % e * D:][:D, :D, :D] = src
        out["atlas"].append(t.reshape(-1))
        out["dims"].append((bx * D, by * D, bz * D))
    return out


def check(ctx, topo, blocks=None):
    view = topo.view()
    if blocks:
        view = relayout(view, topo.counts, blocks)
    a, b = ctx.build_grid(topo, gpu=True), ctx.upload_view(view)
    pa, pb = a.pools(), b.pools()
    for k in ("slot5", "slot4", "leaf", "ovf"):
        np.testing.assert_array_equal(pa[k], pb[k], err_msg=k)
    assert a.info == b.info
    a.release()
    b.release()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 63, 700])
def test_counts(cuda_ctx, n):
    rng = np.random.default_rng(n)
    o = np.unique(rng.integers(-60, 60, size=(n, 3)), axis=0) * 8
    check(cuda_ctx, wx.Topology.from_leaves(o.astype(np.int32), rng.integers(0, 1 << 63, size=(o.shape[0], 8)).astype(np.uint64)))


@pytest.mark.parametrize("blocks", [((9, 9, 1), (9, 9, 3), (40, 40, 1)), ((2, 2, 3), (5, 7, 9), (3, 3, 90)),
                                    ((8, 3, 1), (4, 4, 12), (11, 30, 9))])
def test_shapes(cuda_ctx, blocks):
    rng = np.random.default_rng(5)
    topo = wx.Topology.from_voxels(rng.integers(-300, 300, size=(790, 3)).astype(np.int32))
    n5, n4, n3 = topo.counts
    need = [(b[1] if l == 0 else b[0]) ** 2 * b[2] for l, b in enumerate(blocks)]
    assert n5 <= need[0] and n4 <= need[1] and n3 <= need[2], (topo.counts, need)
    check(cuda_ctx, topo, blocks)


def test_larger_than_the_buffer(cuda_ctx):
    o = np.stack(np.mgrid[0:41, 0:41, 0:41], -1).reshape(-1, 3) * 8 - 160  # 68,921 leaves, 65,536 a layer of 134 MB
    rng = np.random.default_rng(6)
    topo = wx.Topology.from_leaves(o.astype(np.int32), rng.integers(0, 1 << 63, size=(o.shape[0], 8)).astype(np.uint64))
    n5, n4, n3 = topo.counts
    check(cuda_ctx, topo, ((2, 2, 2), (8, 8, 8), (256, 256, 2)))


def test_refused_views(cuda_ctx):
    topo = wx.Topology.from_voxels(np.array([[1, 2, 3], [100, 30, 2]], np.int32))
    view = topo.view()
    for lvl, bad, status in ((0, 7, 1), (1, 99, 1)):  # child index out of range
        v = dict(view, atlas=[a.copy() for a in view["atlas"]])
        side = v["dims"][lvl][0]
        words = (view["kids5"], view["kids4"])[lvl]
        o = int(np.nonzero(np.unpackbits(words.view(np.uint8), bitorder="little"))[0][0])
        L = 5 - lvl
        x, y, z = o >> (2 * L), (o >> L) & ((1 << L) - 1), o & ((1 << L) - 1)
        v["atlas"][lvl][(z * side + y) * side + x] = bad
        with pytest.raises(wx.WxError) as ei:
            cuda_ctx.upload_view(v)
        assert ei.value.status == status
    v = dict(view, atlas=[a.copy() for a in view["atlas"]])
    v["atlas"][1][v["atlas"][1] == view["atlas"][1].max()] = 1 << 31  # a tile distance of 2^31
    with pytest.raises(wx.WxError) as ei:
        cuda_ctx.upload_view(v)
    assert ei.value.status == 4
