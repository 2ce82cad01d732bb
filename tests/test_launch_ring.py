"""How many warps share a tile of a small frame (csrc/launch_ring.h): on the CPU the rule over sequences of launches, on the GPU
frames on both sides of its limits for the device at hand, alone on a stream and among other streams, byte for byte against
the persistent kernel, which never splits."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import woxel_gb300 as wx

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "woxel_gb300" / "csrc"
SMS = 100  # limits of 350, 700 and 1400 tiles
RING = 32


@pytest.fixture(scope="module")
def splits(tmp_path_factory):
    exe = tmp_path_factory.mktemp("ring") / "ring"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), str(HERE / "launch_ring_host.cpp"), "-o", str(exe)], check=True)

    def run(launches):
        text = "\n".join(" ".join(map(str, x)) for x in launches)
        p = subprocess.run([str(exe), str(SMS)], input=text, capture_output=True, text=True, check=True)
        return [int(x) for x in p.stdout.split()]

    return run


@pytest.mark.parametrize("tiles,split", [(0, 3), (1, 3), (350, 3), (351, 2), (700, 2), (701, 1), (1400, 1), (1401, 0), (2 ** 31, 0)])
def test_one_stream(splits, tiles, split):
    assert splits([(0, 7, 0, tiles)] * 70) == [split] * 70


@pytest.mark.parametrize("n", [2, 3, 4, 16, 31, 64])
@pytest.mark.parametrize("tiles", [20, 300])
def test_streams_in_turn(splits, n, tiles):
    """Once every stream has launched, a frame gets what one frame of all their tiles would get."""
    got = splits([(0, 1 + i % n, 0, tiles) for i in range(4 * max(n, RING))])
    seen = min(n, RING) * tiles
    want = 3 if seen <= 350 else 2 if seen <= 700 else 1 if seen <= 1400 else 0
    assert set(got[max(n, RING):]) == {want}
    assert got[0] == 3


def test_only_the_last_launches_count(splits):
    got = splits([(0, i, 0, 300) for i in range(16)] + [(0, 99, 0, 300)] * 40)
    assert got[15] == 0 and got[16] == 0 and got[-1] == 3
    assert got[16 + RING - 1:] == [3] * (len(got) - 16 - RING + 1)  # the last other launch has left the ring


def test_a_stream_counts_with_its_last_launch(splits):
    assert splits([(0, 1, 0, 100000), (0, 1, 0, 10), (0, 2, 0, 300)]) == [0, 3, 3]
    assert splits([(0, 1, 0, 10), (0, 1, 0, 100000), (0, 2, 0, 300)])[-1] == 0


def test_own_stream_and_other_devices_do_not_count(splits):
    assert splits([(0, 5, 0, 100000), (0, 5, 0, 300)]) == [0, 3]
    assert splits([(1, 5, 0, 100000), (1, 6, 0, 100000), (0, 5, 0, 300)]) == [0, 0, 3]


def test_per_thread_streams(splits):
    """cudaStreamPerThread: one handle, a stream in each thread."""
    assert splits([(0, 2, 111, 300), (0, 2, 111, 300)]) == [3, 3]
    assert splits([(0, 2, 100 + i, 300) for i in range(16)])[-1] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("streams", [1, 3])
def test_frames_around_the_limits(cuda_ctx, mode, streams):
    import torch

    topo = wx.Topology.sphere((0, 0, 0), 64.0, 3.0)
    grid = cuda_ctx.build_grid(topo)
    grid.set_values(topo.sphere_values((0, 0, 0), 64.0, 3.0), 3.0)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pool = [torch.cuda.Stream() for _ in range(streams)]
    before = cuda_ctx.tuning

    def frame(tiles, kernel, tile_width, warps, stream, first=0):
        w, h = 19 * 8 + 5, -(-tiles // 19) * 4 + 3  # 8x4 tiles in rows of 19, and a ragged edge
        st = wx.state_build(eye=(30.0, 40.0, 180.0 + first), target=(5.0, 0, 0), aspect=w / h, fovy=60.0, width=float(w), mode=mode)
        cuda_ctx.set_tuning(kernel=kernel, tile_width=tile_width, warps_per_block=warps)
        a = torch.full((h * w * 4,), 7, dtype=torch.uint8, device="cuda")
        b = torch.full((h * w * 32,), 7, dtype=torch.uint8, device="cuda")
        stream.wait_stream(torch.cuda.current_stream())
        cuda_ctx.render(grid, st, w, h, a, b, stream.cuda_stream)
        return a, b

    try:
        for s in (1, 2, 3):
            for tiles in (-(-(sms * 28 >> s) // 19) * 19 // streams + d for d in (-19, 0, 19)):
                ref = [frame(tiles, 0, 8, 4, pool[0], i) for i in range(streams)]
                for i in range(RING):  # the launches before do not count
                    frame(tiles, 1, 8, 4, pool[i % streams])
                for tile_width, warps in ((8, 4), (4, 1), (16, 8)):
                    got = [frame(tiles, 1, tile_width, warps, pool[i], i) for i in range(streams)]
                    torch.cuda.synchronize()
                    for (ra, rb), (a, b) in zip(ref, got):
                        assert torch.equal(ra, a) and torch.equal(rb, b), (tiles, tile_width, warps)
    finally:
        cuda_ctx.set_tuning(**before)
        torch.cuda.synchronize()
        grid.release()
