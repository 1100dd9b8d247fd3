"""Soundness of the frame cull's single-precision item proofs (raster_core.cuh
item_back_facing and obb_misses_samples, with the per-instance data of api.cpp
proof_data), restated in numpy with the same float operations: whenever a proof
says an item is culled, every one of its triangles (vertices) meets stage 1's
float test.  The proofs are given tight oriented boxes (obb); that those of
meshprep.cu k_obbs hold their vertices is a test of its own, on a restatement of
that kernel."""
import numpy as np
import pytest
from test_backface_proof_cpu import back_face_data, det3_glm, item_cone, items, look_at, stage1_backface_culled, xform

F = np.float32
U = F(2.0 ** -24)


def fma(a, b, c):
    return F(float(a) * float(b) + float(c))


def dot_pos(r, c):
    return fma(r[0], c[0], fma(r[1], c[1], fma(r[2], c[2], r[3])))


def dot_dir(r, a):
    return fma(r[0], a[0], fma(r[1], a[1], F(r[2]) * F(a[2])))


def instance_proof(M, lo, hi):
    """api.cpp proof_data: eye, |eye|; |det|, |R|_F, rowAbs, tAbs; S per row."""
    e, det, frob, row, t, el = back_face_data(M)
    R = M.reshape(4, 4).T.astype(np.float64)
    S = np.abs(R[:3, :3]) @ np.maximum(np.abs(lo), np.abs(hi)).astype(np.float64) + np.abs(R[:3, 3])
    up = 1 + 1e-6
    return (e.astype(F), F(el * up), F(det * (1 - 1e-6)), F(frob * up), F(row * up), F(t * up),
            (S * up).astype(F))


def proof_back_facing(M, lo, hi, cone, drop_error=False):
    e, el, det, frob, row, tabs, _ = instance_proof(M, lo, hi)
    m, cosT, nMin, edge, sinT, r = [F(x) if np.ndim(x) == 0 else x.astype(F) for x in cone]
    if not (det > 0 and cosT > 0):
        return False
    mid = (F(0.5) * (lo + hi)).astype(F)
    w = (mid - e).astype(F)
    p = np.abs(mid).max() + r
    wl = np.sqrt(fma(w[0], w[0], fma(w[1], w[1], w[2] * w[2])))
    dm = fma(w[0], m[0], fma(w[1], m[1], w[2] * m[2]))
    cx, cy, cz = (fma(w[1], m[2], -(w[2] * m[1])), fma(w[2], m[0], -(w[0] * m[2])), fma(w[0], m[1], -(w[1] * m[0])))
    cr = np.sqrt(fma(cx, cx, fma(cy, cy, cz * cz)))
    G = ((dm * cosT - cr * sinT) - r) - F(3.814697265625e-06) * (wl + r + el + F(2) * p)
    if not G > 0:
        return False
    g2, g3 = F(2.001) * U, F(3.001) * U
    a, L = frob * (wl + r) * F(1.000001), frob * edge
    Delta = F(1.7320509) * g3 * (row * p + tabs)
    eta = F(2.01) * Delta + U * L
    Lp = L + eta
    E = F(2) * ((Delta + a * F(3.4641018) * g2 + g3 * (a + Delta)) * Lp * Lp * F(1.01) +
                a * (F(2) * eta * L + eta * eta))
    if drop_error:
        E = F(0)
    return bool(det * nMin * G * F(0.999) > E * F(1.001) + F(1e-30))


def obb(p):
    """A box of an (n, 3) float32 set along its principal axes, tighter than meshprep.cu's."""
    q = p.astype(np.float64)
    _, _, ax = np.linalg.svd(q - q.mean(0), full_matrices=True)
    x = q @ ax.T
    lo, hi = x.min(0), x.max(0)
    h, c = 0.5 * (hi - lo), (0.5 * (lo + hi)) @ ax
    slack = 2.0 ** -21 * (np.abs(c).max() + h.sum()) + 1e-37
    return c.astype(F), [(ax[j] * (h[j] * (1 + 2.0 ** -20) + slack)).astype(F) for j in range(3)]


def axis_misses(Fa, row, S, Sz, b, D0, gz, iD, W, margin):
    r0 = F(Fa * dot_pos(row, b[0])) / D0
    e = F(0)
    for j in range(3):
        e = e + np.abs(fma(r0, gz[j], Fa * dot_dir(row, b[1][j])))
    ar = np.abs(r0)
    h = F(0.5) * W * ((e + margin * (F(28) * U * (np.abs(Fa) * S + (ar + F(1e-3)) * Sz) + F(1e-30))) * iD) + \
        margin * F(6) * U * W * (ar + F(1))
    s0 = W * (F(0.5) * r0 + F(0.5)) - F(0.5)
    lo, hi = s0 - h, s0 + h
    k = np.floor(lo)
    return bool(lo > k and k >= 0 and hi < k + F(1) and h < F(0.5))


def proof_misses(M, fa, f, W, H, b, S, margin=F(1)):
    rows = M.reshape(4, 4).T.astype(F)
    gz = [dot_dir(rows[2], a) for a in b[1]]
    D0 = -dot_pos(rows[2], b[0])
    Dmin = (D0 - (np.abs(gz[0]) + np.abs(gz[1]) + np.abs(gz[2]))) - margin * (F(32) * U * S[2] + F(1e-30))
    if not (Dmin > F(1e-30) and Dmin < F(1e30)):
        return False
    iD = F(1) / Dmin * F(1.00000095367431640625)
    return axis_misses(fa, rows[0], S[0], S[2], b, D0, gz, iD, W, margin) or \
        axis_misses(f, rows[1], S[1], S[2], b, D0, gz, iD, H, margin)


def stage1_screen(M, p, fa, f, W, H):
    """viewToNDC, ndcToScreen, -0.5 of every vertex (float32, stage 1's order), and its depth."""
    q = xform(M, p)
    d = -q[:, 2]
    x = ((fa * q[:, 0]) / d * F(0.5) + F(0.5)) * W - F(0.5)
    y = ((f * q[:, 1]) / d * F(0.5) + F(0.5)) * H - F(0.5)
    return x, y, d


def missed(x, y, W, H):
    def axis(s, n):
        lo, hi = max(s.min(), F(0)), min(s.max(), F(n - 1))
        return lo > np.floor(lo) and hi < np.floor(lo) + 1

    return axis(x, W) or axis(y, H)


def clusters(rng, n, drop):
    """n proven (or, with the margins dropped, claimed) clusters of vertices that
    end within a few float spacings of a sample line; the share that is wrong."""
    wrong = claimed = 0
    W, H = 1920, 1080
    f = F(1.7320508)
    fa = F(f / F(W / H))
    for _ in range(n):
        size = 10.0 ** rng.uniform(-5, 0)
        off = rng.uniform(-1, 1, 3) * rng.choice([0.0, 1.0, 100.0])
        Rm = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        # a box's corners and points inside: the box is met by its vertices
        corner = np.array([[(c >> j) & 1 for j in range(3)] for c in range(8)]) * 2.0 - 1.0
        p = (np.concatenate([corner, rng.uniform(-1, 1, (8, 3))]) * size * np.array([1.0, 0.3, 0.02])) @ Rm.T + off
        # a fraction of a pixel wide, its edge next to a sample column, across a row
        dist = size * 10.0 ** rng.uniform(3.1, 6.0)
        px, py = rng.integers(1, W - 2), rng.integers(1, H - 2)
        Vr = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        v = p.astype(F).astype(np.float64) @ Vr.T
        t = np.array([0.0, 0.0, -dist]) - v.mean(0)
        v2 = v + t
        sx = (fa * v2[:, 0] / -v2[:, 2] * 0.5 + 0.5) * W - 0.5
        sy = (f * v2[:, 1] / -v2[:, 2] * 0.5 + 0.5) * H - 0.5
        gap = rng.choice([0.0, 3e-5, 1e-4, 1e-2, 0.02, 0.1])
        t[0] += (px + gap - sx.min()) / W * 2 / float(fa) * dist
        t[1] += (py - sy.mean()) / H * 2 / float(f) * dist
        M = np.eye(4)
        M[:3, :3], M[:3, 3] = Vr, t
        M = M.astype(F).T.reshape(16)
        pts = p.astype(F)
        S = instance_proof(M, pts.min(0), pts.max(0))[-1]
        b = obb(pts)
        if drop:
            b = (b[0], [(a / (1 + 2.0 ** -20)).astype(F) for a in b[1]])
        if proof_misses(M, fa, f, F(W), F(H), b, S, F(0) if drop else F(1)):
            claimed += 1
            x, y, d = stage1_screen(M, pts, fa, f, F(W), F(H))
            wrong += not ((d > 0).all() and missed(x, y, W, H))
    return claimed, wrong


def test_sample_miss_proof_is_sound():
    claimed, wrong = clusters(np.random.default_rng(5), 6000, False)
    assert claimed > 800 and wrong == 0, (claimed, wrong)


def test_sample_miss_margins_matter():
    claimed, wrong = clusters(np.random.default_rng(5), 6000, True)
    assert claimed > 800 and wrong > 0, (claimed, wrong)


def proof_quick(M, fa, f, W, H, tri, S, margin=F(1)):
    """raster_core.cuh make_quick and quick_misses (the reciprocal within 2 ulp either way)."""
    rows = M.reshape(4, 4).T.astype(F)
    kx, ky = F(0.5) * W * fa, F(0.5) * H * f
    rx, ry = (rows[0] * kx).astype(F), (rows[1] * ky).astype(F)
    d = np.array([-dot_pos(rows[2], p) for p in tri], F)
    if not (d > margin * (F(16) * U * S[2] + F(1e-30))).all():
        return False
    r = np.array([F(1) / v for v in d], F)
    for _ in range(2):
        r = np.nextafter(r, F(np.inf) * np.where(np.arange(3) % 2, F(1), F(-1)))
    iD = r.max() * F(1.00000095367431640625)
    for rr, c, n, Fa, Sa in ((rx, F(0.5) * W - F(0.5), W, fa, S[0]), (ry, F(0.5) * H - F(0.5), H, f, S[1])):
        x = [fma(dot_pos(rr, p), r[i], c) for i, p in enumerate(tri)]
        m = margin * fma(F(6) * U * n * (np.abs(Fa) * Sa + S[2]), iD, F(8) * U * n)
        lo, hi = min(x) - m, max(x) + m
        k = np.floor(lo)
        if (k >= 0 and hi < k + F(1)) or hi < F(-0.5) or lo > F(2) * c + F(0.5):
            return True
    return False


@pytest.mark.parametrize("margin", [1, 0])
def test_quick_miss_is_sound(margin):
    """Triangles a fraction of a pixel wide whose edge ends next to a sample line."""
    rng = np.random.default_rng(9)
    W, H = F(1920), F(1080)
    f = F(1.7320508)
    fa = F(f / F(W / H))
    claimed = wrong = 0
    for _ in range(6000):
        size = 10.0 ** rng.uniform(-5, 0)
        dist = size * 10.0 ** rng.uniform(3.1, 5.0)
        Vr = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        p = (rng.normal(size=(3, 3)) * size + rng.uniform(-1, 1, 3) * rng.choice([0.0, 1.0, 100.0])).astype(F)
        v = p.astype(np.float64) @ Vr.T
        t = np.array([0.0, 0.0, -dist]) - v.mean(0)
        v2 = v + t
        sx = (fa * v2[:, 0] / -v2[:, 2] * 0.5 + 0.5) * W - 0.5
        sy = (f * v2[:, 1] / -v2[:, 2] * 0.5 + 0.5) * H - 0.5
        gap = rng.choice([0.0, 3e-5, 1e-4, 3e-3, 0.01, 0.1])
        if rng.random() < 0.3:  # just beyond the left or right side
            sxt = -0.5 - gap - sx.max() if rng.random() < 0.5 else 1919.5 + gap - sx.min()
        else:
            sxt = rng.integers(1, 1918) + gap - sx.min()
        t[0] += sxt / W * 2 / float(fa) * dist
        t[1] += (rng.integers(1, 1078) - sy.mean()) / H * 2 / float(f) * dist
        M = np.eye(4)
        M[:3, :3], M[:3, 3] = Vr, t
        M = M.astype(F).T.reshape(16)
        S = instance_proof(M, p.min(0), p.max(0))[-1]
        if proof_quick(M, fa, f, W, H, p, S, F(margin)):
            claimed += 1
            x, y, d = stage1_screen(M, p, fa, f, W, H)
            q = xform(M, p)
            ndc = (fa * q[:, 0]) / d
            wrong += not ((d > 0).all() and (missed(x, y, W, H) or (ndc > 1).all() or (ndc < -1).all()))
    assert claimed > 800
    assert (wrong == 0) if margin else (wrong > 0), (claimed, wrong)


@pytest.mark.parametrize("drop", [False, True])
def test_back_face_proof_is_sound(drop):
    rng = np.random.default_rng(12)
    proved = wrong = 0
    for pa, pb, pc in items(rng):
        cone = item_cone(pa, pb, pc)
        if cone is None:
            continue
        allp = np.concatenate([pa, pb, pc])
        lo, hi = allp.min(0), allp.max(0)
        centre = 0.5 * (lo.astype(np.float64) + hi)
        for _ in range(40):
            m = cone[0] / np.linalg.norm(cone[0])
            dirn = -m + rng.normal(scale=rng.choice([0.01, 0.3, 1.0]), size=3)
            eye = centre + dirn / np.linalg.norm(dirn) * rng.uniform(0.05, 200.0)
            k = int(rng.integers(128))
            a64 = pa[k].astype(np.float64)
            nk = np.cross(pb[k].astype(np.float64) - a64, pc[k].astype(np.float64) - a64)
            if rng.random() < 0.5:  # just behind the plane of one of the item's triangles
                nk /= np.linalg.norm(nk)
                inpl = np.cross(nk, rng.normal(size=3))
                dist = rng.uniform(0.05, 50.0)
                eye = a64 + inpl / np.linalg.norm(inpl) * dist - nk * dist * rng.choice([1e-8, 1e-6, 1e-5, 1e-4, 1e-3])
            Wm = np.eye(4)
            if rng.random() < 0.5:
                Wm[:3, :3] = np.diag(rng.uniform(0.3, 3.0, 3) * rng.choice([-1, 1], 3))
            V = look_at(eye, centre + rng.normal(scale=0.5, size=3))
            M = (V @ Wm).astype(F).T.reshape(16)
            if proof_back_facing(M, lo, hi, cone, drop):
                proved += 1
                wrong += not stage1_backface_culled(M, det3_glm(M) < 0, pa, pb, pc).all()
    assert proved > 100
    assert (wrong > 0) if drop else (wrong == 0), (proved, wrong)


def lanes_sum(v):
    """A warp's butterfly sum over axis 0 in float32: every lane gets the same value."""
    i = np.arange(len(v))
    d = len(v) // 2
    while d:
        v = (v + v[i ^ d]).astype(F)
        d //= 2
    return v[0]


def off_by(rng, x):
    """A float32 function value, up to 2 ulp from the rounded one."""
    x = F(x)
    for _ in range(int(rng.integers(0, 3))):
        x = np.nextafter(x, F(np.inf) if rng.random() < 0.5 else F(-np.inf))
    return F(x)


def kernel_obb(rng, q, lanes, slack=True):
    """meshprep.cu k_obbs: q (lanes, R, 3 corners, 3) float32, NaN where a lane's
    triangle is past the mesh's end.  Every operation rounded to float32 in the
    kernel's order; rsqrtf, atan2f, sinf and cosf within 2 ulp either way."""
    live = ~np.isnan(q[..., 0, 0])
    R = q.shape[1]
    with np.errstate(all="ignore"):
        n = np.zeros((lanes, 3), F)
        for r in range(R):
            u, v = q[:, r, 1] - q[:, r, 0], q[:, r, 2] - q[:, r, 0]
            x = u[:, 1] * v[:, 2] - u[:, 2] * v[:, 1]
            y = u[:, 2] * v[:, 0] - u[:, 0] * v[:, 2]
            z = u[:, 0] * v[:, 1] - u[:, 1] * v[:, 0]
            l2 = (x * x + y * y) + z * z
            for k in range(lanes):
                if live[k, r] and l2[k] > 0 and l2[k] < np.inf:
                    s = off_by(rng, 1.0 / np.sqrt(float(l2[k])))
                    n[k] = n[k] + np.array([x[k] * s, y[k] * s, z[k] * s], F)
        pts = q[live].reshape(-1, 3)
        lo, hi = pts.min(0), pts.max(0)
        m = lanes_sum(n)
        ml2 = (m[0] * m[0] + m[1] * m[1]) + m[2] * m[2]
        if not (ml2 > F(1e-12) and ml2 < np.inf):
            m = np.array([0, 0, 1], F)
        m = (m * (F(1) / np.sqrt((m[0] * m[0] + m[1] * m[1]) + m[2] * m[2]))).astype(F)
        b1 = np.array([0, m[2], -m[1]] if abs(m[0]) < F(0.6) else [-m[2], 0, m[0]], F)
        b1 = (b1 * (F(1) / np.sqrt((b1[0] * b1[0] + b1[1] * b1[1]) + b1[2] * b1[2]))).astype(F)
        b2 = np.array([m[1] * b1[2] - m[2] * b1[1], m[2] * b1[0] - m[0] * b1[2], m[0] * b1[1] - m[1] * b1[0]], F)
        mid = (F(0.5) * (lo + hi)).astype(F)
        scale = F(1) / (max(hi - lo) + F(1e-30))

        def dot(d, a):
            return (d[..., 0] * a[0] + d[..., 1] * a[1]) + d[..., 2] * a[2]

        acc = np.zeros((lanes, 6), F)  # n, sx, sy, xx, xy, yy
        for r in range(R):
            for k in range(3):
                d = q[:, r, k] - mid
                x, y = dot(d, b1) * scale, dot(d, b2) * scale
                add = np.stack([np.ones(lanes, F), x, y, x * x, x * y, y * y], -1)
                acc = np.where(live[:, r, None], acc + add, acc).astype(F)
        cnt, sx, sy, xx, xy, yy = (lanes_sum(acc[:, j]) for j in range(6))
        inv = F(1) / max(cnt, F(1))
        th = F(0.5) * off_by(rng, np.arctan2(F(2) * (xy - sx * sy * inv), (xx - sx * sx * inv) - (yy - sy * sy * inv)))
        if not np.isfinite(th):
            th = F(0)
        ct, sn = off_by(rng, np.cos(float(th))), off_by(rng, np.sin(float(th)))
        ax = np.stack([ct * b1 + sn * b2, ct * b2 - sn * b1, m]).astype(F)
        x = np.stack([dot(pts - mid, a) for a in ax], -1).astype(F)
        pl, ph = x.min(0), x.max(0)
        h, a = (F(0.5) * (ph - pl)).astype(F), (F(0.5) * (hi - lo)).astype(F)
        if (a[0] * a[1] + a[1] * a[2]) + a[2] * a[0] <= (h[0] * h[1] + h[1] * h[2]) + h[2] * h[0]:
            c, h, ax = mid, a, np.eye(3, dtype=F)
        else:
            t = (pl + ph).astype(F)
            c = (mid + F(0.5) * ((t[0] * ax[0] + t[1] * ax[1]) + t[2] * ax[2])).astype(F)
        M = max(np.abs(lo).max(), np.abs(hi).max())
        grow = F(3.814697265625e-06) * ((h[0] + h[1]) + h[2]) + F(9.5367431640625e-07) * M + F(1e-37)
        hj = (h * F(1.0000019073486328125) + grow).astype(F) if slack else h
        return c, (ax * hj[:, None]).astype(F), pts


def outside(c, A, pts):
    """Whether a vertex lies outside the box c + sum t_j A_j, |t_j| <= 1 (solved in float64)."""
    A = A.astype(np.float64)
    ln = np.linalg.norm(A, axis=1)
    d = pts.astype(np.float64) - c.astype(np.float64)
    if not (ln > 0).all():
        return bool((np.abs(d).max(0) > 0).any())
    t = np.linalg.solve((A / ln[:, None]).T, d.T).T / ln
    return bool((np.abs(t) > 1 + 1e-12).any())


@pytest.mark.parametrize("lanes,R", [(16, 1), (32, 4)])
def test_kernel_boxes_hold_their_vertices(lanes, R):
    """Patches, needles, points and lumps, near the origin and far from it, of
    every scale, whole groups and the ends of meshes."""
    rng = np.random.default_rng(lanes)
    bare = 0
    for k in range(400 if lanes == 16 else 120):
        shape = [(1.0, 0.4, 1e-3), (1.0, 1e-4, 1e-5), (1.0, 1.0, 1.0), (0.0, 0.0, 0.0), (1.0, 1e-7, 0.3)][k % 5]
        size = 10.0 ** rng.uniform(-12, 8)
        rot = np.linalg.qr(rng.normal(size=(3, 3)))[0] if k % 3 else np.eye(3)
        p = (rng.uniform(-1, 1, (lanes, R, 3, 3)) * shape * size) @ rot.T
        p += rng.uniform(-1, 1, 3) * size * rng.choice([0.0, 1.0, 1e3, 1e6])
        q = p.astype(F)
        if k % 4 == 1:  # the mesh ends inside the group
            flat = np.arange(lanes * R).reshape(R, lanes).T  # triangle r * lanes + lane
            q[flat >= int(rng.integers(1, lanes * R))] = np.nan
        c, A, pts = kernel_obb(rng, q, lanes)
        assert not outside(c, A, pts), (k, size)
        bare += outside(*kernel_obb(rng, q, lanes, slack=False))
    assert bare > 20  # without the slack many do not
