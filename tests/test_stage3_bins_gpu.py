"""The binned stage 3 (k_stage3_bins): screen-filling, near-plane and sliver
triangles at the edges of its tiles, regions and rounds, against the CPU oracle
and against the unbinned kernel, which a context with a memory budget takes."""
import numpy as np
import pytest

import oracle_lib as ol
import pycurast as pc
import scenes

pytestmark = pytest.mark.gpu


def triangles(n, seed):
    """Triangles of every size stage 3 sees, some with hostile coordinates."""
    rng = np.random.default_rng(seed)
    z = -rng.uniform(0.3, 6.0, n)
    z[: n // 10] = rng.uniform(-0.2, 0.15, n // 10)  # across the camera plane
    centre = np.stack([rng.uniform(-2, 2, n), rng.uniform(-1.2, 1.2, n), z], -1)
    tri = centre[:, None, :] + rng.normal(size=(n, 3, 3)) * np.exp(rng.normal(0.0, 1.0, n))[:, None, None]
    thin = slice(n // 3, n // 2)  # slivers: the third corner close to the first edge
    t = rng.uniform(0, 1, n)[thin, None]
    tri[thin, 2] = tri[thin, 0] * (1 - t) + tri[thin, 1] * t + rng.normal(size=tri[thin, 2].shape) * 1e-3
    tri[5, 1] = tri[5, 0]                            # no area
    tri[6, 0, 0], tri[7, 1, 2], tri[8, 2, 1] = np.nan, np.inf, 1e30
    tri[9] *= 1e-12
    pos = tri.reshape(-1, 3).astype(np.float32)
    return pos, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), rng.integers(0, 2**32, 3 * n, np.uint64).astype(np.uint32)


# one tile and one past it, columns past the right edge that wrap into the next
# row, many rounds of one tile (1500 triangles over 6 tiles), a wide window
@pytest.mark.parametrize("n,W,H", [(60, 64, 64), (60, 65, 129), (1500, 130, 70), (300, 333, 197), (200, 1917, 300)])
def test_bins_match_the_oracle_and_the_unbinned_kernel(gpu, n, W, H):
    import torch

    mesh = triangles(n, 100 + n + W)
    view, proj = scenes.identity(), scenes.perspective(60.0, W / H, 0.01, 100.0)
    got = []
    for budget in (0, 8 << 30):
        with pc.Context(memory_budget=budget) as ctx:
            inst = [(ctx.mesh_from_host(*mesh), scenes.identity())]
            vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
            rgba = torch.empty(W * H, dtype=torch.int32, device="cuda")
            cam = pc.make_camera(view, proj, W, H)
            for _ in range(2):  # the second frame's chains lie over the first's
                ctx.render(inst, cam, vis.data_ptr(), rgba.data_ptr())
            torch.cuda.synchronize()
            st, stats = ctx.stats()
            assert st == pc.CR_OK and stats.huge_tiles > 0
            got.append((vis.cpu().numpy().view(np.uint64), int(stats.huge_tiles)))
    assert got[0][1] == got[1][1]
    assert np.array_equal(got[0][0], got[1][0])
    fb, _ = ol.raster(ol.Frame([(*mesh, scenes.identity())], view), W, H, proj[5])
    assert np.array_equal(got[0][0], fb)


def covering(n, seed):
    """Front-facing triangles over the whole screen, one behind the other and
    slanted; past 600, every eighth leaves a part of it free."""
    rng = np.random.default_rng(seed)
    z = rng.uniform(2.0, 9.0, (n, 1))
    corner = np.array([[-9.0, -7.0], [9.0, -7.0], [0.0, 14.0]]) * (1 + 0.3 * rng.uniform(-1, 1, (n, 3, 2)))
    corner[600::8] += rng.uniform(-6, 6, (len(corner[600::8]), 1, 2))
    depth = z * (1 + 0.2 * rng.uniform(-1, 1, (n, 3)))
    tri = np.concatenate([corner * z[:, :, None], -depth[:, :, None]], -1)
    pos = tri.reshape(-1, 3).astype(np.float32)
    return pos, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), rng.integers(0, 2**32, 3 * n, np.uint64).astype(np.uint32)


# a tile's entries: one past a unit's 512, several units, more than 128 units
# (which then take more than 512 each); one tile and several, whose edge is ragged
@pytest.mark.parametrize("n,W,H", [(513, 72, 64), (1024, 64, 72), (3000, 130, 70), (70000, 72, 64)])
def test_crowded_tiles_are_shared_out(gpu, n, W, H):
    import torch

    tiles = ((W + 63) // 64) * ((H + 63) // 64)
    mesh = covering(n, n)
    view, proj = scenes.identity(), scenes.perspective(60.0, W / H, 0.01, 100.0)
    got = []
    for budget in (0, 8 << 30):
        with pc.Context(memory_budget=budget) as ctx:
            inst = [(ctx.mesh_from_host(*mesh), scenes.identity())]
            vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
            rgba = torch.empty(W * H, dtype=torch.int32, device="cuda")
            ctx.render(inst, pc.make_camera(view, proj, W, H), vis.data_ptr(), rgba.data_ptr())
            torch.cuda.synchronize()
            st, stats = ctx.stats()
            assert st == pc.CR_OK and stats.overflow == 0
            # queued in every tile: the first 600 and at least seven of every further eight
            assert stats.huge_tiles >= tiles * (min(n, 600) + max(n - 600, 0) * 7 // 8)
            got.append(vis.cpu().numpy().view(np.uint64))
    assert np.array_equal(got[0], got[1])
    assert len(np.unique(got[0])) > W * H // 2
    if n <= 3000:
        fb, _ = ol.raster(ol.Frame([(*mesh, scenes.identity())], view), W, H, proj[5])
        assert np.array_equal(got[0], fb)


def test_bins_that_grow_on_a_side_stream(gpu):
    """Windows and a queue that grow from frame to frame, so that the chains are
    laid out anew, on a stream that does not wait for the legacy one."""
    import torch

    mesh = triangles(400, 77)
    sizes = [(64, 64), (200, 130), (640, 360), (65, 129), (1917, 1083)]
    got = []
    for budget in (8 << 30, 0):
        stream = torch.cuda.Stream()
        with pc.Context(memory_budget=budget, max_huge=64) as ctx:
            inst = [(ctx.mesh_from_host(*mesh), scenes.identity())]
            outs = []
            with torch.cuda.stream(stream):
                for W, H in sizes:
                    vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
                    rgba = torch.empty(W * H, dtype=torch.int32, device="cuda")
                    cam = pc.make_camera(scenes.identity(), scenes.perspective(60.0, W / H, 0.01, 100.0), W, H)
                    ctx.render(inst, cam, vis.data_ptr(), rgba.data_ptr(), stream=stream.cuda_stream)
                    outs.append(vis)
            torch.cuda.synchronize()
            st, stats = ctx.stats()
            assert st == pc.CR_OK and stats.huge_tiles > 64
            got.append(outs)
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_frames_without_memory_for_the_bins(gpu):
    """Drawn by the unbinned kernel, and no error is left behind."""
    import torch

    W, H = 333, 197
    mesh = triangles(300, 78)
    cam = pc.make_camera(scenes.identity(), scenes.perspective(60.0, W / H, 0.01, 100.0), W, H)
    got = []
    for debug in (0, pc.CR_DEBUG_REFUSE_STAGE3_BINS):
        with pc.Context(debug_flags=debug) as ctx:
            inst = [(ctx.mesh_from_host(*mesh), scenes.identity())]
            for _ in range(3):
                vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
                rgba = torch.empty(W * H, dtype=torch.int32, device="cuda")
                ctx.render(inst, cam, vis.data_ptr(), rgba.data_ptr())
                got.append((vis, rgba))
            assert ctx.stats()[1].huge_tiles > 0
            if debug:
                assert pc.load().cr_last_error() == b""
    for v, r in got[1:]:
        assert torch.equal(v, got[0][0]) and torch.equal(r, got[0][1])


def huge(n, seed):
    """Triangles with one coordinate so large that the float products of stage 3
    overflow for some of them (a NaN u or v passes the reference's comparisons)."""
    rng = np.random.default_rng(seed)
    tri = rng.uniform(-1, 1, (n, 3, 3))
    tri[..., 2] = -rng.uniform(0.2, 3.0, (n, 3))
    at = (np.arange(n), rng.integers(0, 3, n), rng.integers(0, 3, n))
    tri[at] = rng.choice([3e38, -3e38, 1e38, 1e30, -1e30, 1e25], n)
    pos = tri.reshape(-1, 3).astype(np.float32)
    return pos, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), rng.integers(0, 2**32, 3 * n, np.uint64).astype(np.uint32)


HUGE_VIEW = ((0.1, -0.2, 0.15), (0.4, 0.3, -2.0))  # eye and target: no axis of the view is one of the object's


@pytest.mark.parametrize("seed", range(6))
def test_coordinates_whose_products_overflow(gpu, seed):
    """The binned kernel, the unbinned one (a context with a memory budget) and
    batched views against the oracle."""
    import torch
    from test_batch_gpu import batched

    W = H = 192
    mesh = huge(40, 300 + seed)
    view, proj = scenes.look_at(*HUGE_VIEW), scenes.perspective(60.0, W / H, 0.01, 100.0)
    fb, st = ol.raster(ol.Frame([(*mesh, scenes.identity())], view), W, H, proj[5])
    assert st.huge_tiles > 9 and (fb != pc.CLEAR_PIXEL).any()
    for budget in (0, 8 << 30):
        with pc.Context(memory_budget=budget) as ctx:
            inst = [(ctx.mesh_from_host(*mesh), scenes.identity())]
            vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
            ctx.render(inst, pc.make_camera(view, proj, W, H), vis.data_ptr(), flags=pc.CR_RENDER_SYNC | pc.CR_RENDER_NO_RESOLVE)
            torch.cuda.synchronize()
            assert np.array_equal(vis.cpu().numpy().view(np.uint64), fb), budget
            for v in batched(ctx, inst, [(view, proj, W, H)] * 2)[0]:
                assert np.array_equal(v, fb)


# SHA-1 of the words that a kernel draws which traces every pixel of every tile (the
# build before rows were narrowed in this arithmetic)
UNPRUNED = ["9feb764a075283de", "be7eff0ecfe3ccdc", "0825419f40ee4a45",
            "5f5f26d43c1c0d4c", "53a26ff30a3af861", "c41377cadbfd2a5a"]


@pytest.mark.parametrize("seed", range(6))
def test_overflow_in_the_reference_build_s_arithmetic(gpu, seed):
    import hashlib

    import torch

    W = H = 192
    view, proj = scenes.look_at(*HUGE_VIEW), scenes.perspective(60.0, W / H, 0.01, 100.0)
    with pc.Context() as ctx:
        inst = [(ctx.mesh_from_host(*huge(40, 300 + seed)), scenes.identity())]
        vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
        ctx.render(inst, pc.make_camera(view, proj, W, H), vis.data_ptr(),
                   flags=pc.CR_RENDER_SYNC | pc.CR_RENDER_NO_RESOLVE | pc.CR_RENDER_REF_MATH_NO_FMA)
        torch.cuda.synchronize()
    assert hashlib.sha1(vis.cpu().numpy().tobytes()).hexdigest()[:16] == UNPRUNED[seed]
