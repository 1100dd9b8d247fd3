"""Out-of-core frames of several passes: what a frame draws does not depend on
what the frames before it left in the cache."""
import numpy as np
import pytest

import pycurast as pc
import scenes

pytestmark = pytest.mark.gpu

QUADS, NODES, SLOTS = 16, 20, 10


def grid(x0, x1, y0, y1, z):
    """QUADS x QUADS quads in the plane z, facing the camera at the origin."""
    n = QUADS + 1
    x, y = np.meshgrid(np.linspace(x0, x1, n), np.linspace(y0, y1, n))
    pos = np.stack([x, y, np.full_like(x, z)], -1).reshape(-1, 3).astype(np.float32)
    a = (np.arange(QUADS)[:, None] * n + np.arange(QUADS)[None]).reshape(-1)
    idx = np.concatenate([np.stack([a, a + 1, a + n], -1), np.stack([a + 1, a + n + 1, a + n], -1)])
    return pos, idx.astype(np.uint32)


def node_set():
    """Nodes of equal size; the even ones fill the middle of the screen (every
    triangle goes to stage 2), the odd ones are specks near its edges."""
    import torch

    rng = np.random.default_rng(8)
    nodes, keep = [], []
    for k in range(NODES):
        if k % 2 == 0:
            pos, idx = grid(-0.5, 0.5, -0.4, 0.4, -2.0 - 0.01 * k)
        else:
            y = -0.9 + 0.09 * k
            pos, idx = grid(1.2, 1.22, y, y + 0.02, -2.0)
        col = rng.integers(0, 2**32, len(pos), np.uint64).astype(np.uint32)
        t = [torch.from_numpy(a).pin_memory() for a in (pos, idx.view(np.int32), col.view(np.int32))]
        keep.append(t)
        nodes.append((t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), len(pos), len(idx), pos.min(0), pos.max(0),
                      scenes.identity()))
    return nodes, keep


def slot_bytes():
    nv, nt = (QUADS + 1) ** 2, 2 * QUADS * QUADS
    return sum(-(-b // 256) * 256 for b in (12 * nv, 12 * nt, 4 * nv))


def camera(fov, W, H):
    return pc.make_camera(scenes.identity(), scenes.perspective(fov, W / H, 0.01, 100.0), W, H)


def frame(scene, cam, flags, stream=0):
    import torch

    n = cam.width * cam.height
    vis = torch.full((n,), 7, dtype=torch.int64, device="cuda")
    rgba = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = scene.render(cam, vis.data_ptr(), rgba.data_ptr(), flags=flags, stream=stream)
    torch.cuda.synchronize()
    return vis.cpu().numpy(), rgba.cpu().numpy(), st


def test_queues_that_held_a_frame_hold_it_again(gpu):
    """Rendered once with SYNC, which sizes the queues for the frame's passes, then
    without: between two frames of the whole scene another brings the nodes
    that fill stage 2's queue into the cache together."""
    nodes, keep = node_set()
    whole, middle = camera(60.0, 1024, 768), camera(20.0, 64, 48)
    with pc.Context() as ctx, pc.OocScene(ctx, nodes, 1 << 30) as sc:
        want = [frame(sc, cam, pc.CR_RENDER_SYNC) for cam in (whole, middle)]
        assert want[0][2].passes == 1 and want[1][2].visible_nodes == NODES // 2
    with pc.Context(max_nontrivial=1024) as ctx, pc.OocScene(ctx, nodes, SLOTS * slot_bytes()) as sc:
        for flags in (pc.CR_RENDER_SYNC, 0, 0, 0):
            for k, cam in enumerate((whole, middle)):
                vis, rgba, st = frame(sc, cam, flags)
                assert st.passes == 2 - k
                assert ctx.stats()[0] == pc.CR_OK
                assert np.array_equal(vis, want[k][0]) and np.array_equal(rgba, want[k][1]), (flags, k)
        # the same view again and again uploads no more than the cache cannot hold
        for _ in range(3):
            st = frame(sc, whole, 0)[2]
        assert st.uploaded_nodes == NODES - SLOTS


@pytest.mark.parametrize("resolve", [0, pc.CR_RENDER_NO_RESOLVE])
def test_an_overflow_of_any_pass_is_reported(gpu, resolve):
    """The first pass overflows stage 2's queue, the last has nothing for it."""
    nodes, keep = node_set()
    two = [nodes[0], nodes[1]]
    cam = camera(60.0, 1024, 768)
    with pc.Context(max_nontrivial=64) as ctx, pc.OocScene(ctx, two, slot_bytes()) as sc:
        assert frame(sc, cam, resolve)[2].passes == 2
        st, stats = ctx.stats()
        assert st == pc.CR_ERR_QUEUE_OVERFLOW and stats.overflow & 1 and stats.nontrivial == 0
        frame(sc, cam, pc.CR_RENDER_SYNC)
        assert ctx.stats()[0] == pc.CR_OK
        frame(sc, cam, resolve)  # the queues are large enough now: nothing is left of the word
        st, stats = ctx.stats()
        assert st == pc.CR_OK and stats.overflow == 0


def test_box_culled_contexts_keep_nothing_of_evicted_nodes(gpu):
    """CR_CULL_BOXES on a stream that does not wait for the legacy one: frames of
    several passes, nodes evicted and uploaded to other slots, against AUTO."""
    import torch

    nodes, keep = scenes.ooc_terrain(nodes_x=6, nodes_z=6, quads=20, extent=8.0, with_colors=True)
    node_bytes = nodes[0][3] * 16 + nodes[0][4] * 12
    W, H = 160, 90
    cams = [pc.make_camera(scenes.look_at((4.0, 5.0 - k, 4.01 + k), (4.0, 0.0, 4.0 - k)),
                           scenes.perspective(60.0, W / H, 0.001, 100.0), W, H) for k in range(4)]
    with pc.Context() as ctx, pc.OocScene(ctx, nodes, 1 << 30) as sc:
        want = [frame(sc, cam, pc.CR_RENDER_SYNC) for cam in cams]
    stream = torch.cuda.Stream()
    with pc.Context(cull_records=pc.CR_CULL_BOXES) as ctx, pc.OocScene(ctx, nodes, 7 * (node_bytes + 1024)) as sc:
        evicted = 0
        for _ in range(3):
            for cam, (vis, rgba, _) in zip(cams, want):
                got = frame(sc, cam, 0, stream.cuda_stream)
                evicted += got[2].evicted_nodes
                assert np.array_equal(got[0], vis) and np.array_equal(got[1], rgba)
        assert evicted > 36


def test_a_closed_scene_gives_its_memory_back(gpu):
    """Scenes opened, drawn and closed in a context with a memory budget that
    does not hold 200 times what a scene's nodes could keep beside the cache (4 KB
    of boxes each); then one with a larger cache."""
    nodes, keep = scenes.ooc_terrain(nodes_x=6, nodes_z=6, quads=20, extent=8.0, with_colors=True)
    cam = pc.make_camera(scenes.look_at((4.0, 9.0, 4.01), (4.0, 0.0, 4.0)), scenes.perspective(60.0, 1.0, 0.001, 100.0), 96, 96)
    with pc.Context(cull_records=pc.CR_CULL_BOXES, max_nontrivial=4096, max_huge=4096, memory_budget=44 << 20) as ctx:
        for _ in range(200):
            with pc.OocScene(ctx, nodes, 2 << 20) as sc:
                assert frame(sc, cam, pc.CR_RENDER_SYNC)[2].visible_nodes == 36
        with pc.OocScene(ctx, nodes, 6 << 20) as sc:
            assert frame(sc, cam, pc.CR_RENDER_SYNC)[2].cache_slots > 36


def test_a_caller_cannot_keep_the_overflow_words(gpu):
    """The bit that marks a further pass of a frame is the library's own."""
    import torch

    pos, idx = grid(-0.5, 0.5, -0.4, 0.4, -2.0)
    cam, small = camera(60.0, 1024, 768), camera(20.0, 64, 48)
    vis = torch.empty(1024 * 768, dtype=torch.int64, device="cuda")
    with pc.Context(max_nontrivial=64) as ctx:
        inst = [(ctx.mesh_from_host(pos, idx), scenes.identity())]
        flags = pc.CR_RENDER_NO_RESOLVE | pc.CR_RENDER_NO_CLEAR | 1 << 30
        for c, want in ((cam, pc.CR_ERR_QUEUE_OVERFLOW), (small, pc.CR_OK)):
            ctx.render(inst, c, vis.data_ptr(), flags=flags)
            torch.cuda.synchronize()
            assert ctx.stats()[0] == want
