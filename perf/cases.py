"""What a user of woxel_gb300 has it do, as cases that can be timed and compared.

Each case goes through the package's public entry points only: Context.render, Context.batch /
Batch.launch, Context.render_batch, Server, Context.build_grid and Context.upload_view. The grids
are the benchmark's three kinds at several sizes: one narrow-band sphere (small, cache resident), a
union of narrow-band spheres (a level-set model), sparse noise leaves (divergent rays, a large
tree). Cameras are orbit views, drawn from the seed like the grids.

listed()   the cases by name
draw(rng)  one more of the same ranges
prepare    the resident grid(s), uniforms and output buffers (or the host data to load from)
run        one pass: the pixels and, where asked for, the hit records, whole
work       bytes and operations of a pass that no implementation can do without
exact      none: see there
"""
from __future__ import annotations

import numpy as np
import torch

import woxel_gb300 as wx

BAND = 3.0
RESOLUTIONS = [(256, 256), (640, 480), (1280, 720), (1920, 1080), (3840, 2160)]


def listed() -> list:
    return [
        # A thumbnail or an icon of one small model, the smallest call there is: launch and
        # host latency, few warps.
        {"name": "thumbnail", "kind": "frames", "grid": "sphere", "count": 1, "half": 512, "frames": 1,
         "width": 160, "height": 120, "mode": 0, "hits": False, "tints": False, "out": "device"},
        # The benchmark's small configuration: one 640x480 window of the r=64 sphere, Lambert with
        # shadow rays, into page-locked host memory as a host-side canvas wants it.
        {"name": "window", "kind": "frames", "grid": "sphere", "count": 1, "half": 512, "frames": 1,
         "width": 640, "height": 480, "mode": 3, "hits": False, "tints": False, "out": "pinned"},
        # The default workload: an animation of 1080p Lambert frames around the 2000-sphere model,
        # one call per frame, queued back to back.
        {"name": "orbit_1080p", "kind": "frames", "grid": "spheres", "count": 2000, "half": 1024, "frames": 8,
         "width": 1920, "height": 1080, "mode": 3, "hits": False, "tints": False, "out": "device"},
        # Sparse divergent occupancy at 4K (the largest grid, 2.7 M leaves): first active voxel.
        {"name": "noise_4k", "kind": "frames", "grid": "noise", "count": 0, "half": 2048, "frames": 2,
         "width": 3840, "height": 2160, "mode": 0, "hits": False, "tints": False, "out": "device"},
        # Picking and debugging in a window of odd size: the step-count colours with the node tints
        # and the full hit record of every pixel.
        {"name": "picking", "kind": "frames", "grid": "spheres", "count": 700, "half": 700, "frames": 1,
         "width": 1366, "height": 769, "mode": 2, "hits": True, "tints": True, "out": "device"},
        # The glossy mode: up to six rays per pixel.
        {"name": "glossy_720p", "kind": "frames", "grid": "spheres", "count": 1000, "half": 800, "frames": 1,
         "width": 1280, "height": 720, "mode": 4, "hits": False, "tints": False, "out": "device"},
        # The zero-crossing mode over level-set values.
        {"name": "surface_1080p", "kind": "frames", "grid": "spheres", "count": 1000, "half": 800, "frames": 1,
         "width": 1920, "height": 1080, "mode": 5, "hits": True, "tints": False, "out": "device"},
        # Many cameras of uneven resolution over two resident grids, as a plan that is replayed.
        {"name": "batch_mixed", "kind": "plan", "grid": "spheres", "count": 1000, "half": 1024, "frames": 48,
         "top": 4, "mode": 3, "hits": False},
        # A contact sheet: many small views in one call, another set of views each time.
        {"name": "contact_sheet", "kind": "batch", "grid": "spheres", "count": 500, "half": 512, "frames": 60,
         "top": 0, "mode": 3, "hits": False},
        # A burst of requests to the render server, each result fetched to host memory.
        {"name": "serve_burst", "kind": "serve", "grid": "spheres", "count": 500, "half": 512, "frames": 24,
         "top": 2, "mode": 3, "hits": False},
        # A model is loaded or switched: SDF and pools built on the GPU from the topology, then the
        # first frame with its hit records.
        {"name": "load_model", "kind": "load", "grid": "spheres", "count": 2000, "half": 1024, "frames": 1,
         "width": 1280, "height": 720, "mode": 3, "hits": True},
        # The same through the drop-in upload of the flattened view (masks, origins, atlases).
        {"name": "upload_view", "kind": "upload", "grid": "spheres", "count": 200, "half": 512, "frames": 1,
         "width": 1280, "height": 720, "mode": 3, "hits": True},
    ]


def _log(rng, lo: float, hi: float) -> float:
    return float(np.exp(rng.uniform(np.log(lo), np.log(hi))))


def draw(rng) -> dict:
    kind = rng.choice(["frames", "frames", "frames", "frames", "plan", "batch", "serve", "load", "load", "upload"])
    if kind == "frames":
        grid = rng.choice(["sphere", "spheres", "spheres", "noise"])
        mode = rng.choice([0, 1, 2, 3, 3, 3, 4] + ([5] if grid != "noise" else []))
        w = int(_log(rng, 96, 3840))
        h = max(64, min(2160, int(w * rng.uniform(0.45, 1.0))))
        c = {"kind": kind, "grid": grid, "count": int(_log(rng, 100, 1500)), "half": int(_log(rng, 256, 1024)),
             "frames": rng.randint(1, 4), "width": w, "height": h, "mode": mode, "hits": rng.random() < 0.4,
             "tints": rng.random() < 0.2, "out": rng.choice(["device", "device", "pinned"])}
        if grid == "sphere":
            c["count"] = 1
        if grid == "noise":
            c["count"], c["half"] = 0, 8 * int(_log(rng, 64, 192))
        return c
    c = {"kind": kind, "grid": "spheres", "count": int(_log(rng, 100, 900)), "half": int(_log(rng, 300, 1024)),
         "mode": rng.choice([0, 3, 3, 3]), "hits": rng.random() < 0.5}
    if kind in ("plan", "batch", "serve"):
        c["frames"] = int(_log(rng, 4, 30))
        c["top"] = rng.randint(0, 3 if kind != "serve" else 2)
    else:
        if kind == "upload":
            c["count"] = int(_log(rng, 40, 130))
        c["frames"], c["width"], c["height"] = 1, int(_log(rng, 200, 1600)), int(_log(rng, 150, 900))
    return c


_contexts: dict = {}


def _context() -> wx.Context:
    """A program has one context per device."""
    dev = torch.cuda.current_device()
    if dev not in _contexts:
        _contexts[dev] = wx.Context(dev)
    return _contexts[dev]


def _model(c: dict, rng):
    """Topology, its level-set values (mode 5) and the orbit's centre and radius."""
    seed = int(rng.integers(1, 2 ** 40))
    if c["grid"] == "sphere":
        o = rng.uniform(-0.5, 0.5, 3) * c["half"]
        r = float(rng.uniform(48, 96))
        o = tuple(float(x) for x in o)
        topo = wx.Topology.sphere(o, r, BAND)
        return topo, (lambda: topo.sphere_values(o, r, BAND)), o, 3.2 * r
    if c["grid"] == "spheres":
        a = (c["count"], 4.0, 40.0, -float(c["half"]), float(c["half"]), BAND, seed)
        topo = wx.Topology.spheres(*a)
        return topo, (lambda: topo.spheres_values(*a)), (0.0, 0.0, 0.0), 2.93 * c["half"]
    topo = wx.Topology.noise_leaves(-c["half"], 2 * c["half"], 0.02, 0.5, seed)
    return topo, None, (0.0, 0.0, 0.0), 1.7 * c["half"]


def _states(c: dict, rng, sizes: list, centre, radius: float) -> list:
    eyes = wx.orbit_eyes(len(sizes), radius, int(rng.integers(1, 2 ** 40)))
    tints = (1, 1, 1) if c.get("tints") else (0, 0, 0)
    return [wx.state_build(eye=tuple(float(e) + o for e, o in zip(eye, centre)), target=centre, aspect=w / h, fovy=60.0,
                           width=float(w), mode=c["mode"], show_345=tints) for eye, (w, h) in zip(eyes, sizes)]


def _buffers(w: int, h: int, hits: bool, out: str = "device") -> tuple:
    kw = {"device": "cuda"} if out == "device" else {"pin_memory": True}
    return (torch.zeros(h * w * 4, dtype=torch.uint8, **kw),
            torch.zeros(h * w * 32, dtype=torch.uint8, **kw) if hits else None)


def prepare(case: dict, seed: int) -> dict:
    c = case
    rng = np.random.default_rng([seed, c["count"], c["half"], c["frames"]])
    ctx = _context()
    topo, values, centre, radius = _model(c, rng)
    s = {"case": c, "ctx": ctx}
    if c["kind"] in ("frames", "load", "upload"):
        sizes = [(c["width"], c["height"])] * c["frames"]
        s["states"] = _states(c, rng, sizes, centre, radius)
        s["buffers"] = [_buffers(w, h, c["hits"], c.get("out", "device")) for w, h in sizes]
        s["grid"] = None
        if c["kind"] == "load":
            s["topo"] = topo
        elif c["kind"] == "upload":
            s["view"] = topo.view()
        else:
            s["grid"] = ctx.build_grid(topo, gpu=True)
            if c["mode"] == wx.MODE_SURFACE:
                s["grid"].set_values(values(), BAND)
        return s
    # plan, batch, serve: two resident grids, the model and a single sphere, resolutions drawn from
    # the benchmark's list up to RESOLUTIONS[top]
    small, _, centre1, radius1 = _model({"grid": "sphere", "half": c["half"]}, rng)
    grids = [ctx.build_grid(topo, gpu=True), ctx.build_grid(small, gpu=True)]
    which = [int(x) for x in rng.integers(0, 2, c["frames"])]
    # 2 of 3 in the order of the list, so that every pass has the same mix of resolutions
    sizes = [RESOLUTIONS[(i * 2 // 3) % (c["top"] + 1)] for i in range(c["frames"])]
    both = [_states(c, rng, sizes, centre, radius), _states(c, rng, sizes, centre1, radius1)]
    states = [both[g][i] for i, g in enumerate(which)]
    s["grids"] = grids
    if c["kind"] == "serve":
        s["server"] = wx.Server(ctx, budget_bytes=3 << 30)
        ids = [s["server"].add_grid(g) for g in grids]
        s["requests"] = [wx.Server.request(ids[g], st, w, h, hits=c["hits"], user=i)
                         for i, (g, st, (w, h)) in enumerate(zip(which, states, sizes))]
        return s
    s["buffers"] = [_buffers(w, h, c["hits"]) for w, h in sizes]
    s["list"] = [(grids[g], st, w, h, a, b) for g, st, (w, h), (a, b) in zip(which, states, sizes, s["buffers"])]
    if c["kind"] == "plan":
        s["plan"] = ctx.batch(s["list"])
    return s


def _outputs(s: dict) -> list:
    return [b for pair in s["buffers"] for b in pair if b is not None]


def run(state: dict):
    s, c = state, state["case"]
    ctx, stream = s["ctx"], torch.cuda.current_stream().cuda_stream
    if c["kind"] == "plan":
        s["plan"].launch(stream)
        return _outputs(s)
    if c["kind"] == "batch":
        ctx.render_batch(s["list"], stream)
        return _outputs(s)
    if c["kind"] == "serve":
        srv = s["server"]
        for r in s["requests"]:
            srv.submit(r)
        got: dict = {}
        while len(got) < len(s["requests"]):
            for res in srv.poll(64, 1000):
                got[res.user] = srv.fetch(res, hits=c["hits"])
                srv.release(res.ticket)
        return [a for i in range(len(got)) for a in (got[i][0], got[i][1].view(np.uint8) if c["hits"] else None)
                if a is not None]
    if c["kind"] in ("load", "upload"):  # the model shown so far goes, the new one comes
        if s["grid"] is not None:
            s["grid"].release()
        s["grid"] = ctx.build_grid(s["topo"], gpu=True) if c["kind"] == "load" else ctx.upload_view(s["view"])
    for st, (rgba, hits) in zip(s["states"], s["buffers"]):
        ctx.render(s["grid"], st, c["width"], c["height"], rgba, hits, stream)
    return _outputs(s)


# Mean march steps of a primary ray over orbit views, and FP32 operations of one step (floor of the
# position, three quotients, three distances, their minimum, the new position).
STEPS = {"sphere": 29, "spheres": 42, "noise": 42}
STEP_FLOPS = 47


def work(case: dict) -> dict:
    c = case
    if c["kind"] in ("plan", "batch", "serve"):
        sizes = [RESOLUTIONS[(i * 2 // 3) % (c["top"] + 1)] for i in range(c["frames"])]
        steps = (STEPS["sphere"] + STEPS["spheres"]) / 2
    else:
        sizes = [(c["width"], c["height"])] * c["frames"]
        steps = STEPS[c["grid"]]
    pixels = sum(w * h for w, h in sizes)
    out = pixels * (4 + (32 if c["hits"] else 0))
    nbytes, flops = out + 256 * len(sizes), pixels * steps * STEP_FLOPS
    if c["kind"] in ("load", "upload"):
        # About 240 leaves and 1.5 N4 nodes a sphere. Read: the masks (64 B a leaf, 1 KB an N4, 8 KB
        # an N5) and, for the drop-in, the atlases; written: a byte a voxel, a word a slot.
        n3, n4, n5 = 240 * c["count"], 1.5 * c["count"], 8
        nbytes += n3 * (64 + 512) + n4 * (1024 + 16384) + n5 * (8192 + 131072)
        if c["kind"] == "upload":
            nbytes += 4 * (n3 * 512 + n4 * 4096 + n5 * 32768)
        flops += 26 * (n3 * 512 + n4 * 4096 + n5 * 32768)  # a minimum over 26 neighbours
    return {"bytes": int(nbytes), "flops": int(flops)}


def exact(case: dict, seed: int):
    """None: every output is bytes (RGBA8 texels; hit records as the bytes that a caller reads), held to
    equality. A march in 64 bits takes other steps than the FP32 one where a ray grazes a cell border,
    so there is no 64-bit value of them."""
    return None
