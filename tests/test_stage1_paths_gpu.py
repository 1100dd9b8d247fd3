"""Stage 1's paths draw the same frame: every triangle straight through the
per-triangle path (small AUTO frames), boxes of 16 triangles and a test of single
ones ahead of it (large AUTO frames of sub-pixel triangles, CR_CULL_BOXES), and
per-vertex records (CR_CULL_CELLS, CR_CULL_OUTCODES), which the oracle and the
golden frames hold to the reference."""
import numpy as np
import pytest

import pycurast as pc
import scenes

pytestmark = pytest.mark.gpu


def frames(ctx, inst, cams, display=pc.CR_DISPLAY_VERTEX_COLORS):
    import torch

    out = []
    for view, proj, W, H in cams:
        vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
        rgba = torch.empty(W * H, dtype=torch.int32, device="cuda")
        ctx.render(inst, pc.make_camera(view, proj, W, H), vis.data_ptr(), rgba.data_ptr(), 0, display)
        torch.cuda.synchronize()
        st, stats = ctx.stats()
        assert st == pc.CR_OK
        out.append((vis.cpu().numpy().view(np.uint64), rgba.cpu().numpy().view(np.uint32), stats))
    return out


def upload(ctx, mesh, compressed=False):
    p, i, c = mesh
    return ctx.mesh_compressed(pc.compress_mesh(p, i), c) if compressed else ctx.mesh_from_host(p, i, c)


def scene(kind):
    """meshes, [(mesh, world)], compressed."""
    rng = np.random.default_rng(5)
    if kind == "needles":  # narrower than a pixel, many rows high
        return [scenes.heightfield(450, 223, seed=2)], [(0, scenes.identity())], False
    if kind == "packed":
        return [scenes.heightfield(301, 97, seed=3)], [(0, scenes.identity())], True
    if kind == "one":  # fewer triangles than lanes of a warp
        p, i, c = scenes.heightfield(8, 4, seed=4)
        return [(p, i[:7], c)], [(0, scenes.identity())], False
    if kind == "soup":  # near-plane, non-finite and no-area triangles
        p, i, c = scenes.triangle_soup(3001, seed=9)
        p[17], p[40, 1], p[77, 2] = np.nan, np.inf, -np.inf
        i[5, 1] = i[5, 0]
        return [(p, i, c)], [(0, scenes.identity())], False
    # meshes whose ends lie inside a warp's 32 triangles, mirrored and plain, one of zero scale
    meshes = [scenes.heightfield(9, 5, seed=6), scenes.heightfield(40, 17, seed=7)]
    inst = []
    for k in range(70):
        w = np.array(scenes.translate_scale(*(rng.uniform(-1, 1, 3) * (1, 0.3, 1)), 0.3), np.float32)
        if k % 3 == 1:
            w[0:3] *= -1
        inst.append((k & 1, w))
    inst[9] = (0, scenes.translate_scale(0, 0, 0, 0.0))
    return meshes, inst, False


@pytest.mark.parametrize("kind,sizes", [("needles", [(391, 220), (64, 63)]), ("packed", [(201, 57), (1917, 1083)]),
                                        ("one", [(1920, 1080), (33, 9)]), ("soup", [(640, 363), (31, 17)]),
                                        ("many", [(320, 181), (1280, 720)])])
def test_small_frames_match_every_record_mode(gpu, kind, sizes):
    meshes, inst, compressed = scene(kind)
    eye = scenes.identity() if kind == "soup" else scenes.heightfield_camera(*sizes[0])[0]
    cams = [(eye, scenes.perspective(60.0, W / H, 0.01, 100.0), W, H) for W, H in sizes]
    want = None
    for mode in (pc.CR_CULL_OUTCODES, pc.CR_CULL_CELLS, pc.CR_CULL_BOXES, pc.CR_CULL_AUTO):
        with pc.Context(cull_records=mode) as ctx:
            hs = [upload(ctx, m, compressed) for m in meshes]
            got = frames(ctx, [(hs[m], w) for m, w in inst], cams)
        if want is None:
            want = got
            assert all((v != pc.CLEAR_PIXEL).any() for v, _, _ in want)
        for (v, c, _), (wv, wc, _) in zip(got, want):
            assert np.array_equal(v, wv) and np.array_equal(c, wc), mode
    # AUTO took every triangle through the path
    assert all(s.stage1_survivors == s.triangles for _, _, s in got)


# one, the most and more instances than a direct frame shares out 32 triangles at a time;
# meshes whose ends lie inside a warp's 32, one without triangles among them
@pytest.mark.parametrize("count,compressed", [(1, False), (4, False), (4, True), (5, False)])
def test_direct_frames_of_few_instances(gpu, count, compressed):
    W, H = 201, 113
    meshes = [scenes.heightfield(131 + 7 * k, 61 + k, seed=k) for k in range(count)]
    if count > 2 and not compressed:
        p, i, c = meshes[1]
        meshes[1] = (p, i[:0], c)
    cams = [(scenes.heightfield_camera(W, H)[0], scenes.perspective(60.0, W / H, 0.01, 100.0), W, H)]
    got = []
    for mode in (pc.CR_CULL_CELLS, pc.CR_CULL_AUTO):
        with pc.Context(cull_records=mode) as ctx:
            inst = [(upload(ctx, m, compressed), scenes.translate_scale(0.05 * k, 0.03 * k, -0.1 * k))
                    for k, m in enumerate(meshes)]
            got += frames(ctx, inst, cams)
    assert (got[0][0] != pc.CLEAR_PIXEL).any() and got[1][2].stage1_survivors == got[1][2].triangles
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("tris,orbit,W,H", [(2_300_000, False, 319, 181), (6_000_001, True, 640, 360)])
def test_large_sub_pixel_frames_are_box_culled(gpu, tris, orbit, W, H):
    pos, idx, col = keep = scenes.planet(tris, seed=3, device="cuda", width=W, height=H)
    cams = [(*(scenes.planet_orbit_camera(W, H) if o else scenes.planet_camera(W, H)), W, H) for o in (orbit, not orbit)]
    got = []
    for mode in (pc.CR_CULL_CELLS, pc.CR_CULL_AUTO):
        with pc.Context(cull_records=mode) as ctx:
            h = ctx.mesh_from_device(pos.data_ptr(), pos.shape[0], idx.data_ptr(), idx.shape[0], col.data_ptr())
            got.append(frames(ctx, [(h, scenes.identity())], cams))
    del keep
    for (v, c, s), (av, ac, a) in zip(*got):
        assert np.array_equal(v, av) and np.array_equal(c, ac)
        assert s.vertex_chunks > 0
    assert got[1][0][2].vertex_chunks == 0  # no vertex pass


def test_sub_boxes_are_built_once_memory_is_back(gpu):
    """A frame that had no room for the oriented boxes is drawn from records, and
    box-culled some frames after the room is there."""
    import torch

    W, H = 640, 360
    pos, idx, col = scenes.planet(2_300_000, seed=3, device="cuda", width=W, height=H)
    cam = pc.make_camera(*scenes.planet_orbit_camera(W, H), W, H)
    vis = torch.empty(W * H, dtype=torch.int64, device="cuda")
    rgba = torch.empty(W * H, dtype=torch.int32, device="cuda")
    with pc.Context() as ctx:
        h = ctx.mesh_from_device(pos.data_ptr(), pos.shape[0], idx.data_ptr(), idx.shape[0], col.data_ptr())
        inst = [(h, scenes.identity())]
        chunks, seen = [], []
        torch.cuda.empty_cache()
        try:  # leaves less than the gigabyte that the rule wants
            held = torch.empty(torch.cuda.mem_get_info()[0] - (900 << 20), dtype=torch.uint8, device="cuda")
        except torch.OutOfMemoryError:
            pytest.skip("the GPU's free memory cannot be held in one piece")
        for k in range(140):
            if k == 2:
                del held
                torch.cuda.empty_cache()
            ctx.render(inst, cam, vis.data_ptr(), rgba.data_ptr())
            chunks.append(int(ctx.stats()[1].vertex_chunks))
            if k in (0, 139):
                seen.append((vis.clone(), rgba.clone()))
    assert chunks[0] > 0 and chunks[1] > 0 and chunks[-1] == 0  # no vertex pass in the end
    assert torch.equal(seen[0][0], seen[1][0]) and torch.equal(seen[0][1], seen[1][1])


def test_more_survivors_than_the_list_holds(gpu):
    W, H = 2560, 1440
    pos, idx, col = keep = scenes.terrain(1500, seed=3, device="cuda")
    top = (scenes.look_at((0.5, 0.9, 0.501), (0.5, 0.0, 0.5)), scenes.perspective(60.0, W / H, 0.001, 10.0), W, H)
    got = []
    for mode in (pc.CR_CULL_CELLS, pc.CR_CULL_BOXES):
        with pc.Context(cull_records=mode) as ctx:
            h = ctx.mesh_from_device(pos.data_ptr(), pos.shape[0], idx.data_ptr(), idx.shape[0], col.data_ptr())
            two = [(h, scenes.identity()), (h, scenes.translate_scale(0.0, -0.05, 0.0))]
            got += frames(ctx, two, [top])
    del keep
    assert got[1][2].stage1_survivors > 1 << 22  # the list's first size
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


# one window pixel per triangle and more, and far less; views that fill up a group of
# four and do not; few items (parts of the views) and more
@pytest.mark.parametrize("quads,views,scale", [(40, 64, 0.1), (90, 5, 0.25), (700, 3, 0.05), (300, 33, 0.03)])
def test_batched_views_match_single_frames(gpu, quads, views, scale):
    import torch

    pos, idx, col = keep = scenes.terrain(quads, seed=3, device="cuda")
    cams = scenes.batch_cameras(views, seed=7, terrain_seed=3, scale=scale)
    with pc.Context(cull_records=pc.CR_CULL_CELLS) as ctx:
        h = ctx.mesh_from_device(pos.data_ptr(), pos.shape[0], idx.data_ptr(), idx.shape[0], col.data_ptr())
        mirror = np.array(scenes.identity(), np.float32)
        mirror[0] = -1.0
        inst = [(h, scenes.identity()), (h, mirror), (h, scenes.translate_scale(0.0, 0.1, 0.0, 0.5))]
        want = frames(ctx, inst, cams)
        bufs = [(torch.empty(W * H, dtype=torch.int64, device="cuda"), torch.empty(W * H, dtype=torch.int32, device="cuda"))
                for _, _, W, H in cams]
        ctx.render_batch(inst, [(pc.make_camera(*c), v.data_ptr(), r.data_ptr(), 0) for c, (v, r) in zip(cams, bufs)])
        torch.cuda.synchronize()
    del keep
    for (v, r), (wv, wr, _) in zip(bufs, want):
        assert np.array_equal(v.cpu().numpy().view(np.uint64), wv)
        assert np.array_equal(r.cpu().numpy().view(np.uint32), wr)


@pytest.mark.parametrize("nx,nz", [(1024, 64), (20000, 6)])
def test_slices_of_forced_records_are_the_camera_s(gpu, nx, nz):
    """Record-culled frames of few triangles, which AUTO no longer makes."""
    W, H = 320, 180
    mesh = scenes.heightfield(nx, nz, size=(1.0, 0.5), amp=0.02, seed=3)
    proj = scenes.perspective(60.0, W / H, 0.01, 100.0)
    cams = [(scenes.heightfield_camera(W, H)[0], proj, W, H),
            (scenes.look_at((0.2, 0.25, 0.6), (0.6, 0.0, 0.1)), proj, W, H)]
    with pc.Context(cull_records=pc.CR_CULL_CELLS) as ctx:
        both = frames(ctx, [(upload(ctx, mesh), scenes.identity())], cams)
    with pc.Context(cull_records=pc.CR_CULL_CELLS) as ctx:
        fresh = frames(ctx, [(upload(ctx, mesh), scenes.identity())], cams[1:])
    assert not np.array_equal(both[0][0], both[1][0])
    assert np.array_equal(both[1][0], fresh[0][0]) and np.array_equal(both[1][1], fresh[0][1])
    assert 0 < fresh[0][2].vertex_slices_evaluated == both[1][2].vertex_slices_evaluated


@pytest.mark.parametrize("display", [pc.CR_DISPLAY_VERTEX_COLORS, pc.CR_DISPLAY_MESH_ID, pc.CR_DISPLAY_NORMAL])
@pytest.mark.parametrize("slots", [3, 7])
def test_passes_resolve_what_one_pass_would(gpu, display, slots):
    """Out of core, in passes: each pass's resolve draws its own pixels and no others."""
    import torch

    nodes, keep = scenes.ooc_terrain(nodes_x=6, nodes_z=6, quads=20, extent=8.0, with_colors=True)
    node_bytes = nodes[0][3] * 16 + nodes[0][4] * 12
    W, H = 97, 64
    cams = [pc.make_camera(scenes.look_at((4.0, 9.0, 4.01 + k), (4.0, 0.0, 4.0)), scenes.perspective(60.0, W / H, 0.001, 100.0),
                           W, H) for k in range(3)]
    got = []
    with pc.Context() as ctx:
        for budget in (1 << 30, slots * (node_bytes + 1024)):
            with pc.OocScene(ctx, nodes, geometry_budget=budget) as sc:
                for cam in cams:  # from the second on some nodes are resident
                    vis = torch.full((W * H,), 7, dtype=torch.int64, device="cuda")
                    rgba = torch.full((W * H,), 7, dtype=torch.int32, device="cuda")
                    st = sc.render(cam, vis.data_ptr(), rgba.data_ptr(), display)
                    torch.cuda.synchronize()
                    got.append((vis.cpu().numpy(), rgba.cpu().numpy(), st.passes))
    for one, many in zip(got[:3], got[3:]):
        assert one[2] == 1 and many[2] > 1
        assert np.array_equal(one[0], many[0])
        if display != pc.CR_DISPLAY_MESH_ID:
            assert np.array_equal(one[1], many[1])
            continue
        # a node's colour is that of its place in the cache-sized run of the draw order
        drawn = one[0].view(np.uint64) != pc.CLEAR_PIXEL
        place = (one[0].view(np.uint64)[drawn] & np.uint64((1 << 36) - 1)) // np.uint64(nodes[0][4])
        assert len(np.unique(place)) > 2 * slots
        for k in np.unique(place % np.uint64(slots)):
            first = one[1][drawn][place == k]
            assert (many[1][drawn][place % np.uint64(slots) == k] == first[0]).all()
        assert np.array_equal(one[1][~drawn], many[1][~drawn])
