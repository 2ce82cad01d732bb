"""Batched launches over few grids (which the kernel takes from the launch's grid table), exactly as many as the table
holds, and more: every frame equals the frame rendered alone."""
import numpy as np
import pytest

import woxel_gb300 as wx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 64, 65, 90])
@pytest.mark.parametrize("how", ["batch", "plan", "noalloc", "server"])
def test_many_grids(cuda_ctx, count, how):
    import torch

    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(count)
    grids = [cuda_ctx.build_grid(wx.Topology.from_voxels(rng.integers(-25, 25, size=(300, 3)).astype(np.int32)), gpu=True)
             for _ in range(count)]
    w, h = 72, 44
    n = count + 7  # grids used twice, out of order
    order = [int(i) for i in rng.permutation(n) % count]
    states = [wx.state_build(eye=tuple(float(x) for x in e), target=(0, 0, 0), aspect=w / h, fovy=60.0, width=float(w),
                             mode=[0, 3, 4][i % 3]) for i, e in enumerate(wx.orbit_eyes(n, 90.0, count))]

    def buf(b):
        return torch.zeros(w * h * b, dtype=torch.uint8, device="cuda")

    alone = []
    for g, st in zip(order, states):
        a, b = buf(4), buf(32)
        cuda_ctx.render(grids[g], st, w, h, a, b, stream)
        torch.cuda.synchronize()
        alone.append((a.cpu().numpy(), b.cpu().numpy()))
    if how == "server":
        srv = wx.Server(cuda_ctx, budget_bytes=8 << 30)
        ids = [srv.add_grid(g) for g in grids]
        for i, (g, st) in enumerate(zip(order, states)):
            srv.submit(wx.Server.request(ids[g], st, w, h, hits=True, user=i))
        got = {}
        while len(got) < n:
            for r in srv.poll(64, 1000):
                got[r.user] = srv.fetch(r, hits=True)
                srv.release(r.ticket)
        srv.close()
        got = [(got[i][0].reshape(-1), got[i][1].view(np.uint8).reshape(-1)) for i in range(n)]
    else:
        frames = [(grids[g], st, w, h, buf(4), buf(32)) for g, st in zip(order, states)]
        if how == "batch":
            cuda_ctx.render_batch(frames, stream)
        elif how == "noalloc":
            wx.render_batch_noalloc(frames, stream)
        else:
            plan = cuda_ctx.batch(frames)
            plan.launch(stream)
        torch.cuda.synchronize()
        got = [(f[4].cpu().numpy(), f[5].cpu().numpy()) for f in frames]
    for i in range(n):
        np.testing.assert_array_equal(got[i][0], alone[i][0], err_msg=f"frame {i}")
        np.testing.assert_array_equal(got[i][1], alone[i][1], err_msg=f"frame {i}")
    for g in grids:
        g.release()
