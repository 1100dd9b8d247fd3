"""What a user of this library has it do, as timed cases.

listed() holds the cases; draw(rng) gives more of the same ranges.  A case is
one pass through the public entry points of pycurast (the C ABI): a frame
loop's cr_render, a batch of views, an out-of-core flight, the image pass.
Every context, mesh, plan and output buffer is made in prepare(), which also
renders the case once synchronously, as a program does that wants its queues
sized before it renders frames back to back; run() then issues the work on
torch's current stream and returns the buffers it writes.

Every output is a word or a byte (64-bit depth-and-id pixels, RGBA8 images)
that is a pure function of the inputs: the library's contract is that they are
bit-identical however the work is scheduled, so the tolerance is "exact", and
there is no 64-bit value they approximate.
"""
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.getcwd(), "curast-ooc_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import pycurast as pc  # noqa: E402
import scenes  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # the smallest frame: a viewport thumbnail of a 4,096-triangle mesh, where launches and latency are the time
        dict(name="frame_small_4k", kind="heightfield", nx=64, nz=32, W=320, H=180, display=4),
        # the ordinary frame: one dense mesh whose triangles cover a pixel or so, every stage in use
        dict(name="frame_heightfield_1m", kind="heightfield", nx=1024, nz=512, W=1920, H=1080, display=4),
        # large and near-plane triangles with shuffled vertices (stages 2 and 3), an odd window
        dict(name="frame_soup_60k", kind="soup", tris=60_000, W=1917, H=1083, display=4),
        # a scanned scene of 400M triangles walked through close up: most of it is off screen
        dict(name="frame_planet_400m", kind="planet", tris=400_000_000, orbit=False, W=1920, H=1080, display=4),
        # the same scene seen whole: its geometry has to be read
        dict(name="frame_orbit_400m", kind="planet", tris=400_000_000, orbit=True, W=1920, H=1080, display=4),
        # an instanced scene: one 1M-triangle mesh drawn 3,000 times
        dict(name="frame_instanced_3000x1m", kind="instances", count=3000, tris=1_000_000, W=1920, H=1080, display=4,
             mirror=False),
        # a prop field: a few hundred mirrored and plain copies of a small mesh, the picking display
        dict(name="frame_props_300x5k", kind="instances", count=300, tris=5_121, W=1280, H=720, display=6, mirror=True),
        # a mesh in the compressed format, as a scene is kept when memory is short, with the colorbuffer asked for
        dict(name="frame_compressed_2m", kind="heightfield", nx=1201, nz=833, W=2560, H=1440, display=3, compressed=True,
             colorbuffer=True),
        # the arithmetic of a host built with fast math, drawn for a drop-in comparison
        dict(name="frame_refmath_1m", kind="heightfield", nx=1024, nz=512, W=1920, H=1080, display=4, refmath=True),
        # 64 views of uneven resolution over a 60M-triangle terrain in one captured plan
        dict(name="batch_64v_60m", kind="batch", views=64, quads=5477, scale=1.0, plan=True),
        # a flight over a scene that streams from host memory through a cache of half its size
        dict(name="ooc_flight_38m", kind="ooc", nodes=24, quads=181, budget=0.5, frames=4, W=1920, H=1080),
        # the image pass of a 2x supersampled 1080p window: eye-dome lighting and ambient occlusion
        dict(name="post_2160p_ss2", kind="post", W=3840, H=2160, factor=2, edl=True, ssao=True, fast=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _window(rng):
    h = _log(rng, 120, 1500)
    return max(64, int(h * rng.choice([1.0, 4 / 3, 16 / 9]) + rng.randrange(3))), h


def draw(rng):
    kind = rng.choice(["heightfield", "heightfield", "soup", "planet", "planet", "instances", "instances", "refmath",
                       "batch", "ooc", "post"])
    W, H = _window(rng)
    display = rng.choice([4, 4, 4, 4, 0, 3, 5, 6, 7])
    if kind in ("heightfield", "refmath"):
        nx = _log(rng, 40, 2000)
        c = dict(kind="heightfield", nx=nx, nz=max(8, nx // 2 + rng.randrange(9)), W=W, H=H, display=display)
        if kind == "refmath":
            c["refmath"] = True
        elif rng.random() < 0.3:
            c["compressed"] = True
        if rng.random() < 0.2:
            c["colorbuffer"] = True
        return c
    if kind == "soup":
        return dict(kind="soup", tris=_log(rng, 500, 100_000), W=W, H=H, display=display)
    if kind == "planet":
        return dict(kind="planet", tris=_log(rng, 1_000_000, 300_000_000), orbit=rng.random() < 0.5, W=W, H=H,
                    display=display)
    if kind == "instances":
        count = _log(rng, 2, 3000)
        return dict(kind="instances", count=count, tris=_log(rng, 1000, min(1_000_000, 2_500_000_000 // count)), W=W,
                    H=H, display=display, mirror=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind="batch", views=rng.randrange(2, 49), quads=_log(rng, 300, 4000),
                    scale=rng.choice([0.25, 0.5, 1.0]), plan=rng.random() < 0.5)
    if kind == "ooc":
        return dict(kind="ooc", nodes=rng.randrange(4, 21), quads=rng.randrange(60, 182), budget=rng.choice([0.3, 0.6, 1.0]),
                    frames=rng.randrange(1, 5), W=W, H=H)
    factor = rng.choice([1, 2, 3])
    return dict(kind="post", W=factor * (W // factor), H=factor * (H // factor), factor=factor, edl=True,
                ssao=rng.random() < 0.7, fast=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _stream():
    return torch.cuda.current_stream().cuda_stream


class _Frame:
    """A single view: context, instances, camera and output buffers."""

    def __init__(self, ctx, inst, cam, W, H, display, flags, colorbuffer, keep):
        self.ctx, self.inst, self.cam, self.display, self.flags, self.keep = ctx, inst, cam, display, flags, keep
        self.vis = torch.empty(W * H, dtype=torch.int64, device=DEV)
        self.rgba = torch.empty(W * H, dtype=torch.int32, device=DEV)
        self.cb = torch.empty(W * H, dtype=torch.int64, device=DEV) if colorbuffer else None

    def render(self, flags=0):
        self.ctx.render(self.inst, self.cam, self.vis.data_ptr(), self.rgba.data_ptr(),
                        self.cb.data_ptr() if self.cb is not None else 0, self.display, self.flags | flags, _stream())
        out = {"vis": self.vis, "rgba": self.rgba}
        if self.cb is not None:
            out["colorbuffer"] = self.cb
        return out


def _moved(view, rng, size):
    """The view with its eye moved by up to `size` along each view axis (a walk's next frame)."""
    v = np.array(view, np.float32)
    v[12:15] += rng.uniform(-size, size, 3).astype(np.float32)
    return v


def _device_mesh(ctx, mesh):
    p, i, c = mesh
    return ctx.mesh_from_device(p.data_ptr(), p.shape[0], i.data_ptr(), i.shape[0], c.data_ptr())


def _frame_state(case, seed):
    W, H, kind = case["W"], case["H"], case["kind"]
    rng = np.random.default_rng(seed)
    ctx = pc.Context()
    keep = None
    if kind == "heightfield":
        pos, idx, col = scenes.heightfield(case["nx"], case["nz"], seed=seed)
        view, proj = scenes.heightfield_camera(W, H)
        view = _moved(view, rng, 0.01)
        if case.get("compressed"):
            mesh = ctx.mesh_compressed(pc.compress_mesh(pos, idx), col)
        else:
            mesh = ctx.mesh_from_host(pos, idx, col)
        inst = pc.make_instances([(mesh, scenes.identity())])
    elif kind == "soup":
        pos, idx, col = scenes.triangle_soup(case["tris"], seed=seed)
        view, proj = scenes.identity(), scenes.perspective(60.0, W / H, 0.01, 100.0)
        inst = pc.make_instances([(ctx.mesh_from_host(pos, idx, col), scenes.identity())])
    elif kind == "planet":
        keep = scenes.planet(case["tris"], seed=seed, device=DEV)
        view, proj = scenes.planet_orbit_camera(W, H) if case["orbit"] else scenes.planet_camera(W, H)
        view = _moved(view, rng, 0.001)
        inst = pc.make_instances([(_device_mesh(ctx, keep), scenes.identity())])
    else:
        keep = scenes.asteroid(case["tris"], seed=seed, device=DEV)
        mesh = _device_mesh(ctx, keep)
        if case["mirror"]:
            worlds = [scenes.random_affine(rng, mirror=bool(k & 1)) for k in range(case["count"])]
        else:
            worlds = scenes.instanced_field(case["count"], seed=seed)
        view, proj = scenes.instanced_camera(W, H)
        inst = pc.make_instances([(mesh, w) for w in worlds])
    state = _Frame(ctx, inst, pc.make_camera(view, proj, W, H), W, H, case["display"],
                   pc.CR_RENDER_REF_MATH if case.get("refmath") else 0, case.get("colorbuffer"), keep)
    state.render(pc.CR_RENDER_SYNC)
    return state


def _batch_cameras(case, seed):
    """Seeded cameras over the seed's terrain; the windows' sizes are the case's own."""
    sizes = [(W, H) for _, _, W, H in scenes.batch_cameras(case["views"], scale=case["scale"])]
    return [(view, scenes.perspective(60.0, W / H, 0.001, 10.0), W, H) for (W, H), (view, _, _, _) in
            zip(sizes, scenes.batch_cameras(case["views"], seed=seed, terrain_seed=seed))]


class _Batch:
    """Several views of one terrain, their buffers one after the other in two tensors."""

    def __init__(self, case, seed):
        self.keep = scenes.terrain(case["quads"], seed=seed, device=DEV)
        self.ctx = pc.Context()
        self.inst = pc.make_instances([(_device_mesh(self.ctx, self.keep), scenes.identity())])
        cams = _batch_cameras(case, seed)
        base = np.concatenate([[0], np.cumsum([2 * ((W * H + 1) // 2) for _, _, W, H in cams])])
        # the pad between views of odd size is never written
        self.vis = torch.zeros(int(base[-1]), dtype=torch.int64, device=DEV)
        self.rgba = torch.zeros(int(base[-1]), dtype=torch.int32, device=DEV)
        self.views = [(pc.make_camera(*cam), self.vis.data_ptr() + 8 * int(b), self.rgba.data_ptr() + 4 * int(b), 0)
                      for cam, b in zip(cams, base)]
        if case["plan"]:
            self.plan = pc.BatchPlan(self.ctx, self.inst, self.views)
        else:
            self.plan = None
            self.ctx.render_batch(self.inst, self.views, stream=_stream())

    def run(self):
        if self.plan is not None:
            self.plan.launch(_stream())
        else:
            self.ctx.render_batch(self.inst, self.views, flags=0, stream=_stream())
        return {"vis": self.vis, "rgba": self.rgba}

    def __del__(self):
        if getattr(self, "plan", None) is not None:
            self.plan.close()


class _Flight:
    """A few frames over an out-of-core terrain."""

    def __init__(self, case, seed):
        W, H, n = case["W"], case["H"], case["frames"]
        nodes, self.keep = scenes.ooc_terrain(case["nodes"], case["nodes"], case["quads"], seed=seed, with_colors=True)
        q = case["quads"]
        self.ctx = pc.Context()
        slot = sum(-(-b // 256) * 256 for b in (12 * (q + 1) ** 2, 24 * q * q, 4 * (q + 1) ** 2))
        self.scene = pc.OocScene(self.ctx, nodes, max(1, int(case["budget"] * len(nodes))) * slot)
        self.cams = [pc.make_camera(*cam) for cam in
                     scenes.ooc_cameras(n, seed=seed, terrain_seed=seed, resolutions=((W, H),))]
        self.vis = torch.empty((n, 2 * ((W * H + 1) // 2)), dtype=torch.int64, device=DEV)
        self.rgba = torch.empty((n, W * H), dtype=torch.int32, device=DEV)
        self.pixels = W * H
        self.run(pc.CR_RENDER_SYNC)

    def run(self, flags=0):
        for k, cam in enumerate(self.cams):
            self.scene.render(cam, self.vis[k].data_ptr(), self.rgba[k].data_ptr(), flags=flags, stream=_stream())
        return {"vis": self.vis[:, :self.pixels], "rgba": self.rgba}

    def __del__(self):
        if getattr(self, "scene", None) is not None:
            self.scene.close()


class _Post:
    """The image pass on a colorbuffer that the library rendered."""

    def __init__(self, case, seed):
        W, H, f = case["W"], case["H"], case["factor"]
        scene = dict(kind="heightfield", nx=512, nz=256, W=W, H=H, display=4, colorbuffer=True)
        self.frame = _frame_state(scene, seed)
        self.proj = scenes.heightfield_camera(W, H)[1]
        self.W, self.H, self.out = W, H, (W // f, H // f)
        self.mode = pc.CR_POST_DISPLAY if f > 1 else pc.CR_POST_SCREENSHOT
        self.flags = ((pc.CR_POST_EDL if case["edl"] else 0) | (pc.CR_POST_SSAO if case["ssao"] else 0) |
                      (pc.CR_POST_FAST_MATH if case["fast"] else 0))
        self.image = torch.empty(self.out[0] * self.out[1], dtype=torch.int32, device=DEV)
        self.run()

    def run(self):
        self.frame.ctx.postprocess(self.frame.cb.data_ptr(), self.W, self.H, self.proj, self.image.data_ptr(), self.flags,
                                   mode=self.mode, out_size=self.out, stream=_stream())
        return self.image


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _Batch(case, seed)
    if kind == "ooc":
        return _Flight(case, seed)
    if kind == "post":
        return _Post(case, seed)
    return _frame_state(case, seed)


def run(state):
    return state.render() if isinstance(state, _Frame) else state.run()


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _mesh_bytes(V, T, compressed=False, colors=True):
    if compressed:
        bits = max(1, math.ceil(math.log2(V)))
        return 6 * V + 3 * T * bits // 8 + (4 * V if colors else 0)
    return 12 * V + 12 * T + (4 * V if colors else 0)


def work(case):
    """Each mesh read once and each output written once; 27 operations to
    transform and project a vertex, for every instance and view of it.  (A
    frame may do with less: groups of triangles that it proves invisible need
    not be read.)"""
    kind = case["kind"]
    colors = case.get("display", 4) == 4
    if kind == "post":
        px, out = case["W"] * case["H"], (case["W"] // case["factor"]) * (case["H"] // case["factor"])
        # per pixel 8 depth taps of the eye-dome term, 32 samples of the occlusion
        return {"bytes": 8 * px + 4 * out, "flops": px * ((8 * 6 if case["edl"] else 0) + (32 * 12 if case["ssao"] else 0))}
    if kind == "batch":
        cams = _batch_cameras(case, 1)
        px = sum(W * H for _, _, W, H in cams)
        V, T = (case["quads"] + 1) ** 2, 2 * case["quads"] ** 2
        return {"bytes": _mesh_bytes(V, T) + 12 * px, "flops": 27 * V * case["views"]}
    if kind == "ooc":
        n, q = case["nodes"] ** 2, case["quads"]
        V, T = n * (q + 1) ** 2, n * 2 * q * q
        # a frame sees about a fifth of the terrain
        return {"bytes": case["frames"] * (0.2 * _mesh_bytes(V, T) + 12 * case["W"] * case["H"]),
                "flops": case["frames"] * 0.2 * 27 * V}
    px = case["W"] * case["H"] * (20 if case.get("colorbuffer") else 12)
    if kind == "heightfield":
        V, T, n = (case["nx"] + 1) * (case["nz"] + 1), 2 * case["nx"] * case["nz"], 1
    elif kind == "soup":
        V, T, n = 3 * case["tris"], case["tris"], 1
    elif kind == "planet":
        V, T, n = case["tris"] // 2, case["tris"], 1
    else:
        V, T, n = case["tris"] // 2, case["tris"], case["count"]
    return {"bytes": _mesh_bytes(V, T, case.get("compressed"), colors) + 64 * n + px, "flops": 27 * V * n}


def tolerance(case):
    return "exact"


def exact(case, seed):
    return None  # words and bytes that are exact by definition: nothing they approximate in 64 bits
