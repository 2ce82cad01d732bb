"""Making a grid while another stream works: the host build and the drop-in upload end before that work does."""
import numpy as np
import pytest

import woxel_gb300 as wx

pytestmark = pytest.mark.gpu


def check(cuda_ctx, topo, make, work):
    import torch

    first = make()  # kernels loaded
    want = first.pools()
    first.release()
    stream, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    work(stream)
    done.record(stream)
    g = make()
    waited = done.query()
    stream.synchronize()
    got = g.pools()
    for k in ("slot5", "slot4", "leaf", "ovf"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    g.release()
    assert not waited, "the call ended after the other stream's work"


@pytest.mark.parametrize("how", ["host", "upload"])
def test_beside_a_long_kernel(cuda_ctx, how):
    """One block for about half a second."""
    import torch

    topo = wx.Topology.sphere((0, 0, 0), 64.0, 3.0)
    view = topo.view()

    def work(stream):
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_000_000_000)

    check(cuda_ctx, topo, (lambda: cuda_ctx.build_grid(topo)) if how == "host" else (lambda: cuda_ctx.upload_view(view)), work)


def test_host_build_beside_a_long_batch(cuda_ctx):
    """A batched launch that holds every SM: the host build launches nothing that has to wait for it."""
    import torch

    topo = wx.Topology.sphere((0, 0, 0), 64.0, 3.0)
    busy = cuda_ctx.build_grid(wx.Topology.noise_leaves(-256, 512, 0.1, 0.5, 4))
    st = wx.state_build(eye=(420.0, 300.0, 500.0), target=(0, 0, 0), aspect=16 / 9, fovy=60.0, width=3840.0, mode=3)
    out = torch.zeros(3840 * 2160 * 4, dtype=torch.uint8, device="cuda")  # the same frame each time

    def work(stream):
        cuda_ctx.render_batch([(busy, st, 3840, 2160, out, None)] * 200, stream.cuda_stream)

    check(cuda_ctx, topo, lambda: cuda_ctx.build_grid(topo), work)
    busy.release()


def test_upload_gives_its_memory_back(cuda_ctx):
    """At a synchronisation all but 32 MB, and those with the context."""
    import torch

    topo = wx.Topology.from_leaves((np.stack(np.mgrid[0:40, 0:40, 0:40], -1).reshape(-1, 3) * 8).astype(np.int32),
                                   np.ones((64000, 8), np.uint64))
    view = topo.view()  # 131 MB of leaf texels
    cuda_ctx.upload_view(view).release()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx = wx.Context(0)
    g = ctx.upload_view(view)
    torch.cuda.synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    assert taken < g.info["device_bytes"] + (40 << 20)
    g.release()
    ctx.close()
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < (4 << 20)
