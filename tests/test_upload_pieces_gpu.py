"""The drop-in upload where the device has less memory than its buffer wants beside the grid: it takes a smaller one and packs the
atlases in more pieces (whole layers, then block rows of a layer), down to one block row; the pools stay those of the native
build, word for word. The shortage is injected: the upload's next `short` allocations fail."""
import numpy as np
import pytest

import woxel_gb300 as wx
from test_upload_gpu import relayout

pytestmark = pytest.mark.gpu


def upload(ctx, view, short):
    wx.inject_alloc_failures(short)
    try:
        return ctx.upload_view(view)
    finally:
        wx.inject_alloc_failures(0)


def shrinks(view, counts):
    """How often the buffer can be halved: from the largest level's layers to the longest block row."""
    least = most = 1024
    for l, (log2, mask) in enumerate(((5, 8192), (4, 1024), (3, 64))):
        w, h, _ = view["dims"][l]
        d = (h if l == 0 else w) >> log2
        rows = -(-counts[l] // d)
        row = (w << (2 * log2 + 2)) + min(counts[l], d) * mask
        least, most = max(least, 1024 + row), max(most, 1024 + row * (rows if rows < d else -(-rows // d) * d))
    n = 0
    while most > least:
        most, n = max(least, most // 2), n + 1
    return n


def check(ctx, topo, view):
    a = ctx.build_grid(topo)
    want = a.pools()
    for short in range(shrinks(view, topo.counts) + 1):
        b = upload(ctx, view, short)
        got = b.pools()
        for k in ("slot5", "slot4", "leaf", "ovf"):
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k}, {short} failures")
        assert a.info == b.info
        b.release()
    a.release()


# Columns, rows and layers of each atlas: the N5 in one row; rows that are left over in a layer; layers higher than their rows.
BLOCKS = [((9, 9, 1), (9, 9, 3), (40, 40, 1)), ((2, 2, 3), (5, 7, 9), (7, 9, 40)), ((3, 3, 1), (4, 4, 12), (12, 12, 9)),
          ((8, 3, 1), (3, 9, 20), (30, 90, 2))]


@pytest.mark.parametrize("blocks", BLOCKS)
@pytest.mark.parametrize("level", [0, 1, 2])
def test_smaller_buffers(cuda_ctx, blocks, level):
    rng = np.random.default_rng(level)
    # Many nodes of one level; of the larger ones few, so that the level decides how much a buffer holds.
    ijk = {0: np.stack(np.mgrid[0:2, 0:2, 0:2], -1).reshape(-1, 3) * 4096 - 4000, 1: rng.integers(-400, 400, size=(150, 3)), 2: rng.integers(0, 120, size=(1500, 3))}[level]
    topo = wx.Topology.from_voxels(ijk.astype(np.int32))
    need = [(b[1] if l == 0 else b[0]) ** 2 * b[2] for l, b in enumerate(blocks)]
    assert all(n <= m for n, m in zip(topo.counts, need)), (topo.counts, need)
    view = relayout(topo.view(), topo.counts, blocks)
    check(cuda_ctx, topo, view)


def test_overflow_in_pieces(cuda_ctx):
    """Leaf distances of 255 and more take a second pass over the leaves."""
    topo = wx.Topology.from_leaves((np.stack(np.mgrid[0:9, 0:9, 0:9], -1).reshape(-1, 3) * 8).astype(np.int32),
                                   np.random.default_rng(1).integers(0, 1 << 63, size=(729, 8)).astype(np.uint64))
    view = topo.view()
    full = view["dims"][2][0] >> 3
    a = view["atlas"][2].copy()
    at = np.random.default_rng(2).choice(np.nonzero(a.reshape(-1) == 1)[0], 900, replace=False)
    a[at] = 1000 + np.arange(900)
    view = dict(view, atlas=view["atlas"][:2] + [a])
    g = cuda_ctx.upload_view(view)
    want = g.pools()
    assert full * full < 729 and len(want["ovf"]) > 0 and shrinks(view, topo.counts) > 0
    for short in range(1, shrinks(view, topo.counts) + 1):
        b = upload(cuda_ctx, view, short)
        for k in ("slot5", "slot4", "leaf", "ovf"):
            np.testing.assert_array_equal(b.pools()[k], want[k], err_msg=f"{k}, {short} failures")
        b.release()


def test_no_memory_at_all(cuda_ctx):
    topo = wx.Topology.sphere((0, 0, 0), 40.0, 3.0)
    with pytest.raises(wx.WxError) as ei:
        upload(cuda_ctx, topo.view(), 1000)
    assert ei.value.status == 3  # WX_ERR_OOM
    cuda_ctx.upload_view(topo.view()).release()


def test_sparse_atlas(cuda_ctx):
    """A few nodes in a wide and high texture: only the block rows that hold nodes are read."""
    topo = wx.Topology.from_voxels(np.random.default_rng(8).integers(-30, 30, size=(40, 3)).astype(np.int32))
    view = relayout(topo.view(), topo.counts, ((8, 8, 1), (32, 32, 1), (128, 128, 1)))
    check(cuda_ctx, topo, view)
