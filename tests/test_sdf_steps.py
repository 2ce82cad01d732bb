"""The step control of the GPU SDF build (csrc/sdf_steps.h): which CTAs and levels take part in a step does not depend
on when a CTA starts. On the CPU its code runs with a thread for each CTA, some of which start only after the others have
found the last distance of a level, of all levels, or have returned; on the GPU builds run while renders on another
stream hold the SMs, so that their CTAs start at different times."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import woxel_gb300 as wx

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "woxel_gb300" / "csrc"


@pytest.fixture(scope="module")
def steps(tmp_path_factory):
    exe = tmp_path_factory.mktemp("sdf_steps") / "steps"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(CSRC), str(HERE / "sdf_steps_host.cpp"), "-o", str(exe)],
                   check=True)

    def run(ctas, k0, k1, last, starts, limit=1 << 30):
        args = [ctas, k0, k1, limit, *last, *starts]
        p = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=60)
        assert p.returncode == 0, (args, p.stdout, p.stderr)
        return p.stdout.split()

    return run


@pytest.mark.parametrize("k0", [1, 9, 255])
@pytest.mark.parametrize("last", [(0, 0, 0), (-1, -1, 0), (0, 1, 3), (2, 0, 0), (5, 6, 4)])
@pytest.mark.parametrize("late", [-1, 0, 1, 2, 3, 4])
@pytest.mark.parametrize("many", [False, True])
def test_ctas_that_start_late(steps, k0, last, late, many):
    """last: each level's last step after k0, -1 for a level without cells; late: see sdf_steps_host.cpp."""
    last = [k0 + n for n in last]
    n = 6
    starts = [-1] * n
    starts[1] = late
    if many and late < 4:
        starts[2:] = [late] * (n - 2)
    # A level that had no cell left at the start keeps 0.
    want = [str(k) if k >= k0 else "0" for k in last]
    for _ in range(3):
        assert steps(n, k0, k0 + 7, last, starts) == want


@pytest.mark.parametrize("ctas", [1, 2, 9])
def test_last_step_of_the_launch(steps, ctas):
    """Cells left after k1 are left alone."""
    assert steps(ctas, 1, 3, (7, 2, 5), [-1] * ctas) == ["3", "2", "3"]
    if ctas > 1:
        assert steps(ctas, 1, 3, (7, 2, 5), [-1] * (ctas - 1) + [4]) == ["3", "2", "3"]


def test_wait_limit(steps):
    """The other CTAs give up one after another when a wait meets its limit."""
    for _ in range(20):
        got = steps(4, 1, 200, (200, 200, 200), [-1] * 4, limit=1)
        assert got in (["error"], ["200", "200", "200"])


def _random_leaves(n, keep, seed):
    rng = np.random.default_rng(seed)
    o = np.unique(rng.integers(-90, 90, size=(n, 3)), axis=0) * 8
    m = np.packbits(rng.random((o.shape[0], 512)) < keep, axis=1, bitorder="little").view(np.uint64)
    return wx.Topology.from_leaves(o.astype(np.int32), m)


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [0, 1])
def test_builds_beside_renders(cuda_ctx, kernel):
    """Small grids (CTAs without open cells; leaves that are done after the first step) and one of many steps."""
    import torch

    busy = cuda_ctx.build_grid(wx.Topology.noise_leaves(-256, 512, 0.1, 0.5, 4))
    st = wx.state_build(eye=(420.0, 300.0, 500.0), target=(0, 0, 0), aspect=16 / 9, fovy=60.0, width=1920.0, mode=3)
    outs = [torch.zeros(1920 * 1080 * 4, dtype=torch.uint8, device="cuda") for _ in range(2)]
    block = np.stack(np.mgrid[0:12, 0:12, 0:12], -1).reshape(-1, 3) * 8
    empty = np.zeros((block.shape[0], 8), np.uint64)
    empty[0, 0] = 1
    topos = [_random_leaves(1, 0.5, 1), _random_leaves(40, 0.9, 2), _random_leaves(3000, 0.5, 3), _random_leaves(3000, 0.01, 4),
             wx.Topology.from_leaves(block.astype(np.int32), empty)]
    host = [cuda_ctx.build_grid(t) for t in topos]
    want = [g.pools() for g in host]
    stream = torch.cuda.Stream()
    before = cuda_ctx.tuning
    cuda_ctx.set_tuning(kernel=kernel)
    try:
        for k in range(60):
            for i in range(8):
                cuda_ctx.render(busy, st, 1920, 1080, outs[i & 1], None, stream.cuda_stream)
            g = cuda_ctx.build_grid(topos[k % len(topos)], gpu=True)
            got = g.pools()
            for name, a in want[k % len(topos)].items():
                np.testing.assert_array_equal(got[name], a, err_msg=f"build {k}: {name}")
            g.release()
            stream.synchronize()
    finally:
        cuda_ctx.set_tuning(**before)
        torch.cuda.synchronize()
