// stage3_bins.cuh -- stage 3 of single-view frames, binned by screen tile.
//
// k_stage3 (raster_core.cuh) gives each queued (triangle, 64x64 tile) a warp
// that finds the tile's rows' spans in double precision, traces every pixel of
// them and sends every hit to L2 as a 64-bit atomic minimum, whatever already
// lies in front of it.  What bounds that is the work on hidden fragments: in
// a frame of 375K tiles over 510 screen tiles a pixel is traced hundreds of
// times.  Here stage 2 links each queued tile into one of CR_BIN_CHAINS
// chains of its screen tile and starts a unit of work for every CR_BIN_PART of a
// tile's entries; a block takes a unit -- an even share of one screen tile's
// chains, over one quadrant of the tile -- a warp per region of 16x8 pixels:
//   * a region's words live in shared memory, loaded once and merged into the visbuffer by at most one atomic minimum per pixel:
//     the word kept is the minimum of the same candidates;
//   * the pixel's ray (two divisions, a square root) is formed once per pixel
//     instead of once per fragment: it does not depend on the triangle;
//   * a triangle is first tested against the region, 32 triangles at a time (a
//     lane per triangle): dropped where no pixel can pass intersect_mt, or
//     where no word it could write is below the words already there (bin_test);
//   * four triangles that are left find their eight rows' spans at once (a
//     lane per row, bin_row_span, in float), and the spans' pixels are packed
//     across the lanes; where they fill most of the region the warp steps
//     through all its pixels instead (no packing).
// Every fragment left runs the float test of k_stage3 unchanged, so the
// visbuffer is the same bit for bit.
// Measured (B200, stage 3): 60K-triangle soup at 1917x1083 (375K tiles) 4.90 ->
// 0.275 ms; 2M-triangle compressed heightfield at 2560x1440 (348K) 0.85 -> 0.300; 1M
// heightfield at 1080p (26.6K) 0.117 -> 0.054.  One unit per quadrant whatever the
// length of the tile's list left a tail of a few long lists (0.29, 0.40, 0.086: 24 % of
// the warps active, 4.5 warps per issue at a barrier); a unit's four quadrants one
// after the other in one block, its triangles set up once, made short queues serial
// (0.29, 0.46, 0.076; 60 tiles of a planet frame 0.025 instead of 0.010).  The pixels'
// words in registers, without row spans, cost slivers more (0.23, 0.75, 0.156).
#pragma once
#include "raster_core.cuh"

namespace {

constexpr int B3_WARPS = 8;
constexpr int B3_THREADS = B3_WARPS * 32;
constexpr int B3_W = 16, B3_H = 8;  // a warp's pixels
// four triangles whose spans cover more than this many of a region's 128
// pixels each step through all of them
#ifndef B3_MINB
#define B3_MINB 3
#endif
#ifndef B3_DENSE
#define B3_DENSE 80
#endif
constexpr int B3_BATCH = 256;  // triangles set up per round
static_assert(B3_BATCH >= CR_BIN_CHAINS && B3_BATCH <= B3_THREADS, "a link of every chain fits a round, a thread per triangle");

// A pixel column passes intersect_mt for a triangle only if (see S3Prune) with
// d = (rx, ry, -1) the unnormalised ray, s the sign of T = e2 . (tvec x e1),
//     s N1.d >= 0,  s N2.d >= 0,  s Q.d >= 0,  -s K.d >= 0
// up to rounding.  The kernel's T is one float per triangle, formed exactly
// as intersect_mt forms it, so s needs no margin: T = 0 or not finite never
// hits.  Rounding, with u = 2^-24, the 1-norms S1, S2, St of e1, e2 and tvec,
// and Dn >= |d|, |rx|, |ry|, 1/fa, 1/f over the frame's tiles:
//   the float test: 8u S1 S2 for det, 8u St S2 for U, 8u St S1 for V (per
//   unit |dir|), u + v <= 1 adding 6u |det| and both bounds; the ray's
//   components 8u/fa + 2u|rx| and 8u/f + 2u|ry|, times |N| <= 2 S S;
//   this test's own N1, N2, Q, K (3u S S each product pair) and corner sums
//   (4u |N| Dn).
// All of it is below 60u S S Dn; the margin is 2^-16 S S Dn = 256u S S Dn.
// A region [x0, x1] x [y0, y1] of ray components is rejected when the maximum
// of any of the four forms over its corners is below minus its margin.
//
// Depth: a hit's depth is fl(T fl(1/det)) |dir.z| with |det| at most
// (max s N1.d + mD) / |d|, so it is at least |T| / (max s N1.d + mD) up to
// 8 roundings (none near the denormals when it is above 1e-30); zlow takes
// 2^-18 off that.  Its word is above every word of
// the region when the depth bits of zlow are above the region's greatest, and
// then the atomic minimum would not have kept it.
enum : int {
    BT_N1 = 0,   // s N1, s N2, s Q, -s K: three floats each
    BT_N2 = 3,
    BT_Q = 6,
    BT_K = 9,
    BT_MD = 12,  // margins (K's is their sum)
    BT_MU = 13,
    BT_MV = 14,
    BT_T = 15,   // |T| (1 - 2^-18)
    BT_ROWS = 16,
};

// What intersect_mt needs of the triangle (tvec and qvec = tvec x e1 do not
// depend on the pixel), and its id.
struct alignas(16) BinTri {
    float e1x, e1y, e1z, e2x;
    float e2y, e2z, tx, ty;
    float tz, qx, qy, qz;
    float T;
    uint32_t idLo, idHi, pad;
};
static_assert(sizeof(BinTri) == 64, "BinTri layout");

// Largest of n.d over the corners of the region, d.z = -1.
__device__ __forceinline__ float corner_max(const float (*t)[B3_BATCH], int row, int j, float x0, float x1, float y0,
                                            float y1) {
    const float nx = t[row][j], ny = t[row + 1][j], nz = t[row + 2][j];
    return (fmaxf(nx * x0, nx * x1) + fmaxf(ny * y0, ny * y1)) - nz;
}

// Whether triangle j of the round can hit a pixel of the region, and the least
// high half of a word that it can write there (0: no bound): a word's high
// half is (depth bits & ~7) << 1 | four id bits.
__device__ __forceinline__ bool bin_test(const float (*t)[B3_BATCH], int j, float x0, float x1, float y0, float y1,
                                         uint32_t& zlow) {
    const float mD = t[BT_MD][j], mU = t[BT_MU][j], mV = t[BT_MV][j];
    const float D = corner_max(t, BT_N1, j, x0, x1, y0, y1);
    const float U = corner_max(t, BT_N2, j, x0, x1, y0, y1);
    const float V = corner_max(t, BT_Q, j, x0, x1, y0, y1);
    const float K = corner_max(t, BT_K, j, x0, x1, y0, y1);
    const uint32_t low = __float_as_uint(__fdividef(t[BT_T][j], D + mD));
    zlow = low > 0x0da24260u && low <= 0x7f800000u ? (low & 0x7ffffff8u) << 1 : 0u;  // above 1e-30, not NaN
    return !(D < -mD || U < -mU || V < -mV || K < -(mD + mU + mV));
}

// Columns [lo, lo + len) of a region row that can pass: column c of the row
// has the ray x0 + A c (c = 0..15), y.  Per form the bound is where
// n.d = -margin; the margin holds every rounding of the sums (see above), and
// the quotient's own error (2 ulp of at most 16) is inside the 2^-6 column the
// span is widened by.
__device__ __forceinline__ void bin_row_span(const float (*t)[B3_BATCH], int j, float x0, float A, float y, int& xlo,
                                             int& len) {
    const float mD = t[BT_MD][j], mU = t[BT_MU][j], mV = t[BT_MV][j];
    float lo = 0.0f, hi = (float)(B3_W - 1);
    bool empty = false;
    auto keep = [&](int row, float margin) {
        const float nx = t[row][j];
        const float a = nx * A;
        const float b = ((nx * x0 + t[row + 1][j] * y) - t[row + 2][j]) + margin;
        if (fabsf(a) < 1e-30f) {
            empty = empty || b < -1e-28f;
            return;
        }
        const float r = __fdividef(-b, a);
        if (a > 0.0f) lo = fmaxf(lo, r);
        else hi = fminf(hi, r);
    };
    keep(BT_N1, mD);
    keep(BT_N2, mU);
    keep(BT_Q, mV);
    keep(BT_K, mD + mU + mV);
    const float flo = fmaxf(ceilf(lo - 0.015625f), 0.0f), fhi = fminf(floorf(hi + 0.015625f), (float)(B3_W - 1));
    if (empty || flo > fhi) {
        xlo = len = 0;
        return;
    }
    xlo = (int)flo;
    len = (int)(fhi - flo) + 1;
}

// The word the triangle writes at the pixel with ray d / |d| (d.z = -1, inv =
// 1 / |d|), ~0 if its ray misses: intersect_mt with the triangle-only terms
// formed once.
__device__ __forceinline__ uint64_t bin_word(const BinTri& t, float dx, float dy, float inv) {
    const V3 e1 = {t.e1x, t.e1y, t.e1z}, e2 = {t.e2x, t.e2y, t.e2z};
    const V3 tvec = {t.tx, t.ty, t.tz}, qvec = {t.qx, t.qy, t.qz};
    const V3 dir = {dx * inv, dy * inv, -1.0f * inv};
    const V3 pvec = cross3(dir, e2);
    const float det = dot3(e1, pvec);
    const float inv_det = 1.0f / det;
    const float u = dot3(tvec, pvec) * inv_det;
    const float v = dot3(dir, qvec) * inv_det;
    const float tt = t.T * inv_det;
    if ((det > -1e-7f && det < 1e-7f) || u < 0.0f || u > 1.0f || v < 0.0f || u + v > 1.0f || !(tt > 0.0f) ||
        tt == INFINITY)
        return ~0ull;
    const float depth = ((tt * dir.x) * 0.0f + (tt * dir.y) * 0.0f) + (tt * dir.z) * -1.0f;
    return pack_pixel(depth, ((uint64_t)t.idHi << 32) | t.idLo);
}

// Sets up triangle j of a round from its queue entry.
__device__ __forceinline__ void bin_setup(const CrFrameParams& p, const CrTile& e, float Dn, float (*t)[B3_BATCH],
                                          BinTri* f, int j) {
    const uint32_t inst = (uint32_t)e.instance, tri = (uint32_t)e.triangle;
    const CrInstance* I = p.instances + inst;
    const Mat M = load_mat(p.world_view + 4ull * inst);
    const GeomRef g = geom_of(I);
    const V3 av = xform(M, pos_of(g, geom_index(g, 3ull * tri + 0)));
    const V3 bv = xform(M, pos_of(g, geom_index(g, 3ull * tri + 1)));
    const V3 cv = xform(M, pos_of(g, geom_index(g, 3ull * tri + 2)));
    const V3 e1 = sub3(bv, av);
    const V3 e2 = sub3(cv, av);
    const V3 tvec = {-av.x, -av.y, -av.z};
    const V3 q = cross3(tvec, e1);
    const float T = dot3(e2, q);
    const uint64_t id = __ldg(&I->cum) + (uint64_t)tri;
    f[j] = BinTri{e1.x, e1.y, e1.z, e2.x, e2.y, e2.z, tvec.x, tvec.y, tvec.z, q.x, q.y, q.z,
                  T,    (uint32_t)id, (uint32_t)(id >> 32), 0u};
    const float s = T > 0.0f ? 1.0f : -1.0f;
    V3 n1 = cross3(e2, e1), n2 = cross3(e2, tvec);
    V3 k = {n1.x - (n2.x + q.x), n1.y - (n2.y + q.y), n1.z - (n2.z + q.z)};  // -K
    const float S1 = fabsf(e1.x) + fabsf(e1.y) + fabsf(e1.z);
    const float S2 = fabsf(e2.x) + fabsf(e2.y) + fabsf(e2.z);
    const float St = fabsf(tvec.x) + fabsf(tvec.y) + fabsf(tvec.z);
    const float m = 1.52587890625e-05f * Dn;  // 2^-16 Dn
    float mD = m * (S1 * S2), mU = m * (St * S2), mV = m * (St * S1);
    float aT = fabsf(T) * 0.99999618530273438f;  // 1 - 2^-18
    // products that underflow keep an absolute margin; sums that are huge or
    // not finite, or a product of det, U or V that could overflow (its NaN passes
    // the reference's comparisons), reject nothing; a T that never hits rejects everything
    mD += 1e-30f, mU += 1e-30f, mV += 1e-30f;
    const bool never = !(T != 0.0f && fabsf(T) < INFINITY);
    const float sum = (S1 * S2 + (St * S2 + St * S1)) + ((mD + mU) + mV) * Dn + (fabsf(n1.x) + fabsf(n1.y) + fabsf(n1.z)) * Dn +
                      (fabsf(n2.x) + fabsf(n2.y) + fabsf(n2.z)) * Dn + (fabsf(q.x) + fabsf(q.y) + fabsf(q.z)) * Dn +
                      (fabsf(k.x) + fabsf(k.y) + fabsf(k.z)) * Dn;
    if (never || !(sum < 1e36f)) {
        n1 = n2 = k = V3{0.0f, 0.0f, 0.0f};
        mD = mU = mV = never ? -1.0f : INFINITY;
        aT = 0.0f;
        const V3 z = {0.0f, 0.0f, 0.0f};
        t[BT_Q][j] = z.x, t[BT_Q + 1][j] = z.y, t[BT_Q + 2][j] = z.z;
    } else {
        t[BT_Q][j] = s * q.x, t[BT_Q + 1][j] = s * q.y, t[BT_Q + 2][j] = s * q.z;
    }
    t[BT_N1][j] = s * n1.x, t[BT_N1 + 1][j] = s * n1.y, t[BT_N1 + 2][j] = s * n1.z;
    t[BT_N2][j] = s * n2.x, t[BT_N2 + 1][j] = s * n2.y, t[BT_N2 + 2][j] = s * n2.z;
    t[BT_K][j] = s * k.x, t[BT_K + 1][j] = s * k.y, t[BT_K + 2][j] = s * k.z;
    t[BT_MD][j] = mD, t[BT_MU][j] = mU, t[BT_MV][j] = mV;
    t[BT_T][j] = aT;
}

__global__ void __launch_bounds__(B3_THREADS, B3_MINB) k_stage3_bins(const CrFrameParams p) {
    pdl_enter();
    __shared__ float s_t[BT_ROWS][B3_BATCH];
    __shared__ BinTri s_f[B3_BATCH];
    __shared__ int2 s_ent[B3_BATCH];
    __shared__ unsigned long long s_word[B3_WARPS][B3_W * B3_H];
    __shared__ float s_inv[B3_WARPS][B3_W * B3_H];
    __shared__ float s_dx[B3_WARPS][B3_W], s_dy[B3_WARPS][B3_H];
    __shared__ uint8_t s_ring[B3_WARPS][64];
    __shared__ uint32_t s_unit, s_n;
    const uint64_t count = min((uint64_t)p.counters[CR_CTR_HUGE], p.hugeCap);
    const uint64_t units = 4ull * min((uint64_t)p.counters[CR_CTR_BINUNITS], (uint64_t)p.binUnitCap);
    if (units == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const Target tg = target_of(p);
    const float Wf = (float)tg.W, Hf = (float)tg.H;
    const float ifa = 1.0f / tg.fa, iff = 1.0f / tg.f;
    const uint32_t tilesX = p.binTilesX, tilesY = p.binTilesY;
    // bounds |d| and the ray's components over every pixel of the tile grid
    const float um = 2.0f * (float)(tilesX * CR_TILE_SIZE) / Wf + 1.0f;
    const float vm = 2.0f * (float)(tilesY * CR_TILE_SIZE) / Hf + 1.0f;
    const float Dn = 1.0f + fabsf(ifa) * um + fabsf(iff) * vm;
    const float A = 2.0f * ifa / Wf;  // the ray's x step per column
    const int numPixels = tg.W * tg.H;
    unsigned long long* const word = s_word[w];
    uint8_t* const ring = s_ring[w];
    // the reference's per-pixel ray (tv.cu:690-705)
    auto ray_x = [&](int px) { return ifa * (2.0f * ((float)px + 0.5f) / Wf - 1.0f); };
    auto ray_y = [&](int py) { return iff * (2.0f * ((float)py + 0.5f) / Hf - 1.0f); };
    while (true) {
        // taken only when the block is free for it: the units differ widely
        if (tid == 0) s_unit = (uint32_t)atomicAdd(&p.counters[CR_CTR_S3UNIT], 1ull);
        __syncthreads();
        const uint32_t unit = s_unit;
        if (unit >= units) return;
        const uint2 un = p.binUnits[unit >> 2];
        const uint32_t tile = un.x;
        // this unit's chains: those of its number, modulo the tile's units
        const uint32_t parts =
            min((p.binCounts[tile] + CR_BIN_PART - 1) / (uint32_t)CR_BIN_PART, (uint32_t)CR_BIN_CHAINS);
        uint32_t cur = 0xffffffffu;
        if (tid < CR_BIN_CHAINS && un.y < parts && tid % parts == un.y) {
            const unsigned long long h = p.binHeads[(uint64_t)tile * CR_BIN_CHAINS + tid];
            if ((uint32_t)(h >> 32) == p.binStamp) cur = (uint32_t)h;
        }
        // the chain's next entry is loaded ahead of its use
        CrTile ahead = {};
        if (cur < p.hugeCap) ahead = p.hugeList[cur];
        // this warp's region of the quadrant
        const int x0 = (int)(tile % tilesX) * CR_TILE_SIZE + (int)(unit & 1u) * 32 + (w & 1) * B3_W;
        const int y0 = (int)(tile / tilesX) * CR_TILE_SIZE + (int)((unit >> 1) & 1u) * 32 + (w >> 1) * B3_H;
        const float wx0 = ray_x(x0), wx1 = ray_x(x0 + B3_W - 1);
        const float wy0 = ray_y(y0), wy1 = ray_y(y0 + B3_H - 1);
        // pixel lane + 32 m of the region, rows of 16: column lane & 15, row
        // (lane >> 4) + 2 m.  Columns past the right edge wrap into the next row,
        // as the reference's pixel index does; rows past the end are not written
        // (their word 0 is never undercut).
        const int pid0 = x0 + (lane & 15) + tg.W * (y0 + (lane >> 4));
        const float myDx = ray_x(x0 + (lane & 15));
        if (lane < B3_W) s_dx[w][lane] = myDx;
        if (lane < B3_H) s_dy[w][lane] = ray_y(y0 + lane);
        __syncwarp();
        uint32_t zw = 0;  // the greatest high half of the region's words
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const V3 d = {myDx, s_dy[w][(lane >> 4) + 2 * m], -1.0f};
            s_inv[w][lane + 32 * m] = 1.0f / sqrtf(dot3(d, d));
            const int pid = pid0 + 2 * m * tg.W;
            const uint64_t v = pid < numPixels ? p.fb[pid] : 0ull;
            word[lane + 32 * m] = v;
            zw = max(zw, (uint32_t)(v >> 32));
        }
        zw = __reduce_max_sync(FULL, zw);
        __syncwarp();
        const float rowY = s_dy[w][lane & 7];
        bool touched = false;
        // a chain holds each entry once, so no walk is longer than the queue
        for (uint64_t walked = 0; walked <= count; ++walked) {
            if (tid == 0) s_n = 0;
            int live = __syncthreads_count(cur < p.hugeCap);
            if (live == 0) break;
            // links of the live chains, while another of each fits
            for (int n = 0; live > 0 && n + live <= B3_BATCH;) {
                const bool on = cur < p.hugeCap;  // 0xffffffff: the chain's end
                const unsigned mk = __ballot_sync(FULL, on);
                uint32_t b = 0;
                if (lane == 0 && mk) b = atomicAdd(&s_n, (uint32_t)__popc(mk));
                b = __shfl_sync(FULL, b, 0);
                if (on) {
                    s_ent[b + __popc(mk & ((1u << lane) - 1u))] = make_int2(ahead.instance, ahead.triangle);
                    cur = (uint32_t)ahead.tile_x;  // the next entry of the chain
                    if (cur < p.hugeCap) ahead = p.hugeList[cur];
                }
                n += live;
                live = __syncthreads_count(cur < p.hugeCap);
            }
            const int n = (int)s_n;
            if (tid < n) {
                CrTile e;
                e.instance = s_ent[tid].x;
                e.triangle = s_ent[tid].y;
                bin_setup(p, e, Dn, s_t, s_f, tid);
            }
            __syncthreads();
            // triangles the region test leaves, in a ring, four at a time
            uint32_t qh = 0, qt = 0;
            auto four = [&]() {
                const uint32_t i = qh + (uint32_t)(lane >> 3);
                const int j = i < qt ? (int)ring[i & 63u] : 0;
                int xlo = 0, len = 0;
                if (i < qt) bin_row_span(s_t, j, wx0, A, rowY, xlo, len);
                int incl = len;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(FULL, incl, d);
                    if (lane >= d) incl += v;
                }
                const int total = __shfl_sync(FULL, incl, 31);
                const int k4 = (int)min(qt - qh, 4u);
                bool changed = false;
                if (total > k4 * B3_DENSE) {
                    for (int i2 = 0; i2 < k4; ++i2) {
                        const BinTri t = s_f[ring[(qh + i2) & 63u]];
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            const int q = lane + 32 * m;
                            const uint64_t nw = bin_word(t, myDx, s_dy[w][(lane >> 4) + 2 * m], s_inv[w][q]);
                            if (nw < word[q]) {
                                word[q] = nw;
                                changed = true;
                            }
                        }
                    }
                } else {
                    for (int base = 0; base < total; base += 32) {
                        const int k = base + lane;
                        int r = 0;
#pragma unroll
                        for (int step = 16; step >= 1; step >>= 1) {
                            const int c = __shfl_sync(FULL, incl, r + step - 1);
                            if (c <= k) r += step;
                        }
                        const int col = __shfl_sync(FULL, xlo - (incl - len), r) + k;
                        const int jr = __shfl_sync(FULL, j, r);
                        if (k >= total) continue;
                        const int q = (r & 7) * B3_W + col;
                        const uint64_t nw = bin_word(s_f[jr], s_dx[w][col], s_dy[w][r & 7], s_inv[w][q]);
                        if (nw < word[q]) {  // two lanes may hold one pixel
                            atomicMin(&word[q], (unsigned long long)nw);
                            changed = true;
                        }
                    }
                }
                qh += (uint32_t)k4;
                if (__any_sync(FULL, changed)) {
                    touched = true;
                    __syncwarp();
                    uint32_t z = 0;
#pragma unroll
                    for (int m = 0; m < 4; ++m) z = max(z, (uint32_t)(word[lane + 32 * m] >> 32));
                    zw = __reduce_max_sync(FULL, z);
                }
                __syncwarp();
            };
            for (int base = 0; base < n; base += 32) {
                const int j = base + lane;
                uint32_t zlow = 0;
                const bool keep = j < n && bin_test(s_t, j, wx0, wx1, wy0, wy1, zlow) && zlow <= zw;
                const unsigned mask = __ballot_sync(FULL, keep);
                if (keep) ring[(qt + __popc(mask & ((1u << lane) - 1u))) & 63u] = (uint8_t)j;
                qt += (uint32_t)__popc(mask);
                __syncwarp();
                while (qt - qh >= 4u) four();
            }
            if (qt != qh) four();
        }
        if (touched)
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int pid = pid0 + 2 * m * tg.W;
                const uint64_t v = word[lane + 32 * m];
                if (pid < numPixels && v < p.fb[pid]) fb_min(p.fb, (uint32_t)pid, v);
            }
        __syncwarp();
    }
}

}  // namespace
