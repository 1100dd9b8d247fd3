// meshprep.cu -- per-mesh bounding boxes for hierarchical culling, built once
// when a mesh is created.
//
//   item boxes   one per CR_BATCH (128) consecutive triangles: the box of
//                every vertex those triangles reference (a stage-1 work item)
//   oriented     one per item and (box-culled frames) per CR_SUB (16) consecutive
//   boxes        triangles, for the sample-miss proof of obb_misses_samples
//   chunk boxes  one per CR_VCHUNK (1024) consecutive vertices (a vertex-pass
//                chunk)
//   group boxes  one per CR_GROUP (32) consecutive item boxes and one per 32
//                consecutive chunk boxes: their union, classified first by
//                the group cull
//   mesh box     the union of the item boxes, classified per instance on the
//                host
// Per view, a box classified by classify_chunk as wholly behind the camera
// or wholly beyond one frustum side proves that every triangle of the item
// (every vertex of the chunk) meets the reference's own cull for it, so the
// item is skipped without reading its indices and the chunk's cull records
// are written without reading its positions.  A box touching a non-finite
// position is NaN, which classifies as nothing.
#include <cuda_runtime.h>
#include <cstdint>

#include "cr_device.h"
#include "geom.cuh"

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void extend(float* lo, float* hi, bool& bad, const GeomRef& g, uint32_t v) {
    float q[3];
    geom_pos(g, v, q[0], q[1], q[2]);
    for (int j = 0; j < 3; ++j) {
        bad |= !isfinite(q[j]);
        lo[j] = fminf(lo[j], q[j]);
        hi[j] = fmaxf(hi[j], q[j]);
    }
}

__device__ __forceinline__ void warp_write_box(float* lo, float* hi, bool bad, float* out, int lane) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            lo[j] = fminf(lo[j], __shfl_xor_sync(FULL, lo[j], d));
            hi[j] = fmaxf(hi[j], __shfl_xor_sync(FULL, hi[j], d));
        }
    bad = __any_sync(FULL, bad);
    if (lane < 6) out[lane] = bad ? __int_as_float(0x7fffffff) : (lane < 3 ? lo[lane] : hi[lane - 3]);
}

// One warp per item: lane + 32 r, r < 4, are its triangles.
__global__ void __launch_bounds__(256) k_item_boxes(const uint32_t* idx, const float* pos, const CrCodec* codec,
                                                    uint32_t nT, float* boxes) {
    const int lane = threadIdx.x & 31;
    const GeomRef g = geom_from(pos, idx, codec);
    const uint32_t nItems = (nT + CR_BATCH - 1) / CR_BATCH;
    for (uint32_t b = blockIdx.x * 8 + (threadIdx.x >> 5); b < nItems; b += gridDim.x * 8) {
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        bool bad = false;
        for (int r = 0; r < CR_BATCH / 32; ++r) {
            const uint32_t t = b * CR_BATCH + r * 32 + lane;
            if (t >= nT) continue;
            for (int k = 0; k < 3; ++k) {
                extend(lo, hi, bad, g, geom_index(g, 3ull * t + k));
            }
        }
        warp_write_box(lo, hi, bad, boxes + 6ull * b, lane);
    }
}

// One warp per item: the vertex-pass slices its triangles' vertices lie in
// (CrSegment::itemSlices: two windows of 64 slices, or the whole range).
__global__ void __launch_bounds__(256) k_item_slices(const uint32_t* idx, const float* pos, const CrCodec* codec,
                                                     uint32_t nT, uint32_t nSlices, uint4* out) {
    const int lane = threadIdx.x & 31;
    const GeomRef g = geom_from(pos, idx, codec);
    const uint32_t nItems = (nT + CR_BATCH - 1) / CR_BATCH;
    constexpr uint32_t NONE = 0xffffffffu;
    for (uint32_t b = blockIdx.x * 8 + (threadIdx.x >> 5); b < nItems; b += gridDim.x * 8) {
        uint32_t sl[CR_BATCH / 32][3];
        uint32_t lo = NONE, hi = 0;
#pragma unroll
        for (int r = 0; r < CR_BATCH / 32; ++r) {
            const uint32_t t = b * CR_BATCH + r * 32 + lane;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                sl[r][k] = t < nT ? min(geom_index(g, 3ull * t + k) / (uint32_t)CR_VSLICE, nSlices - 1) : NONE;
                if (sl[r][k] != NONE) {
                    lo = min(lo, sl[r][k]);
                    hi = max(hi, sl[r][k]);
                }
            }
        }
        lo = __reduce_min_sync(FULL, lo);
        hi = __reduce_max_sync(FULL, hi);
        // window B starts at the least slice past window A
        uint32_t b0 = NONE;
#pragma unroll
        for (int r = 0; r < CR_BATCH / 32; ++r)
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (sl[r][k] != NONE && sl[r][k] - lo >= 64u) b0 = min(b0, sl[r][k]);
        b0 = __reduce_min_sync(FULL, b0);
        if (b0 == NONE) b0 = lo + 64u;
        uint32_t a0m = 0, a1m = 0, b0m = 0, b1m = 0;
        bool past = false;
#pragma unroll
        for (int r = 0; r < CR_BATCH / 32; ++r)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (sl[r][k] == NONE) continue;
                const uint32_t d = sl[r][k] - lo;
                if (d < 32u) a0m |= 1u << d;
                else if (d < 64u) a1m |= 1u << (d - 32u);
                else {
                    const uint32_t e = sl[r][k] - b0;
                    if (e < 32u) b0m |= 1u << e;
                    else if (e < 64u) b1m |= 1u << (e - 32u);
                    else past = true;
                }
            }
        a0m = __reduce_or_sync(FULL, a0m);
        a1m = __reduce_or_sync(FULL, a1m);
        b0m = __reduce_or_sync(FULL, b0m);
        b1m = __reduce_or_sync(FULL, b1m);
        past = __any_sync(FULL, past);
        if (lane == 0) {
            out[2ull * b] = make_uint4(lo, b0, a0m, a1m);
            out[2ull * b + 1] = make_uint4(b0m, b1m, lo, hi | (past ? 0x80000000u : 0u));
        }
    }
}

// The normal cone of LANES * R consecutive triangles (CR_CONE_FLOATS, see
// cr_device.h; 32 x 4: an item, 16 x 1: a sub-box), computed in double from the float positions.  The axis is the
// sum of the unit normals, normalised and rounded to float; cosT is the least
// cosine between a unit normal and that float axis, lowered by 1e-9 (far
// above the double rounding of the computation) and rounded down to float;
// nMin is rounded down, edge, sinT (from the stored cosT) and r (half the
// diagonal of the box of the item's vertices) up.  A zero-area or non-finite
// triangle, or a cone wider than acos(0.05), gives cosT = -2 (no proof).
template <int LANES, int R>
__global__ void __launch_bounds__(256) k_cones(const uint32_t* idx, const float* pos, const CrCodec* codec,
                                                    uint32_t nT, float* cones) {
    constexpr uint32_t T = LANES * R;
    const int lane = threadIdx.x & (LANES - 1);
    const GeomRef g = geom_from(pos, idx, codec);
    const uint32_t nItems = (nT + T - 1) / T;
    const uint32_t perBlock = 256 / LANES;
    // whole warps loop together: groups past the end hold no triangle
    for (uint32_t b0 = blockIdx.x * perBlock; b0 < nItems; b0 += gridDim.x * perBlock) {
        const uint32_t b = b0 + threadIdx.x / LANES;
        double n[R][3];
        double len[R];
        bool live[R];
        double sx = 0.0, sy = 0.0, sz = 0.0, nMin = INFINITY, edge = 0.0;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        bool bad = false;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint64_t t = (uint64_t)b * T + r * LANES + lane;
            live[r] = t < nT;
            len[r] = 1.0;
            n[r][0] = n[r][1] = n[r][2] = 0.0;
            if (!live[r]) continue;
            float a[3], bq[3], c[3];
            geom_pos(g, geom_index(g, 3ull * t + 0), a[0], a[1], a[2]);
            geom_pos(g, geom_index(g, 3ull * t + 1), bq[0], bq[1], bq[2]);
            geom_pos(g, geom_index(g, 3ull * t + 2), c[0], c[1], c[2]);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                lo[j] = fminf(lo[j], fminf(a[j], fminf(bq[j], c[j])));
                hi[j] = fmaxf(hi[j], fmaxf(a[j], fmaxf(bq[j], c[j])));
            }
            const double u0 = (double)bq[0] - a[0], u1 = (double)bq[1] - a[1], u2 = (double)bq[2] - a[2];
            const double v0 = (double)c[0] - a[0], v1 = (double)c[1] - a[1], v2 = (double)c[2] - a[2];
            n[r][0] = u1 * v2 - u2 * v1;
            n[r][1] = u2 * v0 - u0 * v2;
            n[r][2] = u0 * v1 - u1 * v0;
            len[r] = sqrt(n[r][0] * n[r][0] + n[r][1] * n[r][1] + n[r][2] * n[r][2]);
            edge = fmax(edge, fmax(sqrt(u0 * u0 + u1 * u1 + u2 * u2), sqrt(v0 * v0 + v1 * v1 + v2 * v2)));
            bad |= !(len[r] > 0.0) || !isfinite(len[r]) || !isfinite(edge);
            nMin = fmin(nMin, len[r]);
            if (len[r] > 0.0 && isfinite(len[r])) {
                sx += n[r][0] / len[r];
                sy += n[r][1] / len[r];
                sz += n[r][2] / len[r];
            }
        }
#pragma unroll
        for (int d = LANES / 2; d >= 1; d >>= 1) {
            sx += __shfl_xor_sync(FULL, sx, d);
            sy += __shfl_xor_sync(FULL, sy, d);
            sz += __shfl_xor_sync(FULL, sz, d);
            nMin = fmin(nMin, __shfl_xor_sync(FULL, nMin, d));
            edge = fmax(edge, __shfl_xor_sync(FULL, edge, d));
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                lo[j] = fminf(lo[j], __shfl_xor_sync(FULL, lo[j], d));
                hi[j] = fmaxf(hi[j], __shfl_xor_sync(FULL, hi[j], d));
            }
        }
        const unsigned badM = __ballot_sync(FULL, bad);
        bad = ((badM >> (threadIdx.x & 31 & ~(LANES - 1))) & (LANES == 32 ? FULL : (1u << (LANES & 31)) - 1u)) != 0u;
        // the axis as stored (float, normalised in double first), renormalised
        // in double as the cone's cosine is measured
        const double sl = sqrt(sx * sx + sy * sy + sz * sz);
        const float mx = (float)(sx / sl), my = (float)(sy / sl), mz = (float)(sz / sl);
        const double ml = sqrt((double)mx * mx + (double)my * my + (double)mz * mz);
        double cosT = INFINITY;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (live[r] && len[r] > 0.0)
                cosT = fmin(cosT, (n[r][0] * mx + n[r][1] * my + n[r][2] * mz) / (len[r] * ml));
#pragma unroll
        for (int d = LANES / 2; d >= 1; d >>= 1) cosT = fmin(cosT, __shfl_xor_sync(FULL, cosT, d));
        cosT -= 1e-9;
        if (bad || !(sl > 0.0) || !isfinite(sl) || !(ml > 0.0) || !isfinite(ml) || !(cosT > 0.05)) cosT = -2.0;
        const float cosTf = __double2float_rd(cosT);
        double r2 = 0.0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double h = 0.5 * ((double)hi[j] - (double)lo[j]);
            r2 += h * h;
        }
        if (lane < CR_CONE_FLOATS && b < nItems) {
            float v;
            if (lane == 0) v = mx;
            else if (lane == 1) v = my;
            else if (lane == 2) v = mz;
            else if (lane == 3) v = cosTf;
            else if (lane == 4) v = bad ? 0.0f : __double2float_rd(nMin * (1.0 - 1e-9));
            else if (lane == 5) v = bad ? INFINITY : __double2float_ru(edge * (1.0 + 1e-9));
            else if (lane == 6) v = __double2float_ru(sqrt(fmax(0.0, 1.0 - (double)cosTf * cosTf)) * (1.0 + 1e-12));
            else v = __double2float_ru(sqrt(r2) * (1.0 + 1e-12));
            cones[(uint64_t)CR_CONE_FLOATS * b + lane] = v;
        }
    }
}

// The oriented box (CR_OBB_F4) of the vertices of LANES * R consecutive
// triangles, R per lane: 32 x 4 for an item, 16 x 1 for a sub-box.  Axes: the sum of the unit normals, and the
// principal direction of the vertices across it (mesh items are mostly thin
// strips of a surface, whose object-space boxes are loose: on the 1M-triangle
// displaced sphere 26 % of the items of a random instance survive the
// sample-miss proof with axis-aligned boxes, 17 % with these), or the object's
// axes where that box has the smaller surface.  All in single precision.
//
// Containment.  The axes are orthonormal within 2^-21 and the extents measured
// along them (differences from the middle of the object-space box, 2^-24 of the
// coordinates each, and three products) are off by less than 2^-22 (M + H), M the
// largest coordinate and H the sum of the half extents; solving p = c + sum t_j A_j
// against nearly orthonormal axes and rounding c and A move a point by less than
// 2^-20 H + 2^-23 M.  Each half extent is enlarged by 2^-19 of itself, 2^-18 H and
// 2^-20 M.
template <int LANES, int R>
__global__ void __launch_bounds__(256) k_obbs(const uint32_t* idx, const float* pos, const CrCodec* codec, uint32_t nT,
                                              float4* obbs) {
    constexpr uint32_t T = LANES * R;
    const int lane = threadIdx.x & 31, gl = lane & (LANES - 1);
    const GeomRef g = geom_from(pos, idx, codec);
    const uint32_t nGroups = (nT + T - 1) / T;
    const uint32_t perBlock = 256 / LANES;
    auto sum = [](float v) {
#pragma unroll
        for (int d = LANES / 2; d >= 1; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
        return v;
    };
    auto least = [](float v) {
#pragma unroll
        for (int d = LANES / 2; d >= 1; d >>= 1) v = fminf(v, __shfl_xor_sync(FULL, v, d));
        return v;
    };
    // whole warps loop together: groups past the end hold no triangle
    for (uint32_t b0 = blockIdx.x * perBlock; b0 < nGroups; b0 += gridDim.x * perBlock) {
        const uint32_t b = b0 + threadIdx.x / LANES;
        float q[R][3][3];
        bool live[R];
        bool bad = false;
        float nx = 0.0f, ny = 0.0f, nz = 0.0f;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint64_t t = (uint64_t)b * T + r * LANES + gl;
            live[r] = t < nT;
            if (!live[r]) continue;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                geom_pos(g, geom_index(g, 3ull * t + k), q[r][k][0], q[r][k][1], q[r][k][2]);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    bad |= !isfinite(q[r][k][j]);
                    lo[j] = fminf(lo[j], q[r][k][j]);
                    hi[j] = fmaxf(hi[j], q[r][k][j]);
                }
            }
            const float u0 = q[r][1][0] - q[r][0][0], u1 = q[r][1][1] - q[r][0][1], u2 = q[r][1][2] - q[r][0][2];
            const float v0 = q[r][2][0] - q[r][0][0], v1 = q[r][2][1] - q[r][0][1], v2 = q[r][2][2] - q[r][0][2];
            const float x = u1 * v2 - u2 * v1, y = u2 * v0 - u0 * v2, z = u0 * v1 - u1 * v0;
            const float l2 = x * x + y * y + z * z;
            if (l2 > 0.0f && l2 < INFINITY) {
                const float s = rsqrtf(l2);
                nx += x * s, ny += y * s, nz += z * s;
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            lo[j] = least(lo[j]);
            hi[j] = -least(-hi[j]);
        }
        nx = sum(nx), ny = sum(ny), nz = sum(nz);
        // an orthonormal frame m, b1, b2 (any will do for the containment, a good
        // one for tightness)
        float m[3] = {nx, ny, nz};
        const float ml2 = m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
        if (!(ml2 > 1e-12f && ml2 < INFINITY)) m[0] = m[1] = 0.0f, m[2] = 1.0f;
        const float im = 1.0f / sqrtf(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
        m[0] *= im, m[1] *= im, m[2] *= im;
        float b1[3];
        if (fabsf(m[0]) < 0.6f) b1[0] = 0.0f, b1[1] = m[2], b1[2] = -m[1];
        else b1[0] = -m[2], b1[1] = 0.0f, b1[2] = m[0];
        const float bl = 1.0f / sqrtf(b1[0] * b1[0] + b1[1] * b1[1] + b1[2] * b1[2]);
        b1[0] *= bl, b1[1] *= bl, b1[2] *= bl;
        const float b2[3] = {m[1] * b1[2] - m[2] * b1[1], m[2] * b1[0] - m[0] * b1[2], m[0] * b1[1] - m[1] * b1[0]};
        const float mid[3] = {0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2])};
        const float scale = 1.0f / (fmaxf(hi[0] - lo[0], fmaxf(hi[1] - lo[1], hi[2] - lo[2])) + 1e-30f);
        float n = 0.0f, sx = 0.0f, sy = 0.0f, xx = 0.0f, xy = 0.0f, yy = 0.0f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!live[r]) continue;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float d[3] = {q[r][k][0] - mid[0], q[r][k][1] - mid[1], q[r][k][2] - mid[2]};
                const float x = (d[0] * b1[0] + d[1] * b1[1] + d[2] * b1[2]) * scale;
                const float y = (d[0] * b2[0] + d[1] * b2[1] + d[2] * b2[2]) * scale;
                n += 1.0f, sx += x, sy += y, xx += x * x, xy += x * y, yy += y * y;
            }
        }
        n = sum(n), sx = sum(sx), sy = sum(sy), xx = sum(xx), xy = sum(xy), yy = sum(yy);
        const float in = 1.0f / fmaxf(n, 1.0f);
        float th = 0.5f * atan2f(2.0f * (xy - sx * sy * in), (xx - sx * sx * in) - (yy - sy * sy * in));
        if (!isfinite(th)) th = 0.0f;
        const float ct = cosf(th), sn = sinf(th);
        float ax[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            ax[0][j] = ct * b1[j] + sn * b2[j];
            ax[1][j] = ct * b2[j] - sn * b1[j];
            ax[2][j] = m[j];
        }
        float pl[3] = {INFINITY, INFINITY, INFINITY}, ph[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!live[r]) continue;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float d[3] = {q[r][k][0] - mid[0], q[r][k][1] - mid[1], q[r][k][2] - mid[2]};
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const float x = d[0] * ax[j][0] + d[1] * ax[j][1] + d[2] * ax[j][2];
                    pl[j] = fminf(pl[j], x);
                    ph[j] = fmaxf(ph[j], x);
                }
            }
        }
        float h[3], a[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            pl[j] = least(pl[j]);
            ph[j] = -least(-ph[j]);
            h[j] = 0.5f * (ph[j] - pl[j]);
            a[j] = 0.5f * (hi[j] - lo[j]);
        }
        float c[3];
        if (a[0] * a[1] + a[1] * a[2] + a[2] * a[0] <= h[0] * h[1] + h[1] * h[2] + h[2] * h[0]) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                c[j] = mid[j];
                h[j] = a[j];
#pragma unroll
                for (int k = 0; k < 3; ++k) ax[j][k] = j == k ? 1.0f : 0.0f;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                c[k] = mid[k] +
                       0.5f * ((pl[0] + ph[0]) * ax[0][k] + (pl[1] + ph[1]) * ax[1][k] + (pl[2] + ph[2]) * ax[2][k]);
        }
        const float M = fmaxf(fmaxf(fmaxf(fabsf(lo[0]), fabsf(hi[0])), fmaxf(fabsf(lo[1]), fabsf(hi[1]))),
                              fmaxf(fabsf(lo[2]), fabsf(hi[2])));
        const float slack = 3.814697265625e-06f * (h[0] + h[1] + h[2]) + 9.5367431640625e-07f * M + 1e-37f;
        const unsigned badM = __ballot_sync(FULL, bad);
        const bool anyBad = ((badM >> (lane & ~(LANES - 1))) & (LANES == 32 ? FULL : (1u << (LANES & 31)) - 1u)) != 0u;
        if (gl == 0 && b < nGroups) {
            float o[12];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                o[j] = anyBad || !(M < 1e18f) ? __int_as_float(0x7fffffff) : c[j];  // huge: sums could overflow
                const float hj = h[j] * 1.0000019073486328125f + slack;
#pragma unroll
                for (int k = 0; k < 3; ++k) o[3 + 3 * j + k] = ax[j][k] * hj;
            }
#pragma unroll
            for (int j = 0; j < CR_OBB_F4; ++j)
                obbs[(uint64_t)CR_OBB_F4 * b + j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        }
    }
}

// One warp per chunk of CR_VCHUNK vertices.
__global__ void __launch_bounds__(256) k_chunk_boxes(const float* pos, const CrCodec* codec, uint32_t nV,
                                                     float* boxes) {
    const int lane = threadIdx.x & 31;
    const GeomRef g = geom_from(pos, nullptr, codec);
    const uint32_t nChunks = (nV + CR_VCHUNK - 1) / CR_VCHUNK;
    for (uint32_t c = blockIdx.x * 8 + (threadIdx.x >> 5); c < nChunks; c += gridDim.x * 8) {
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        bool bad = false;
        for (uint32_t v = c * CR_VCHUNK + lane; v < min(nV, (c + 1) * CR_VCHUNK); v += 32)
            extend(lo, hi, bad, g, v);
        warp_write_box(lo, hi, bad, boxes + 6ull * c, lane);
    }
}

// One warp per group: the union of CR_GROUP consecutive boxes (item boxes or
// chunk boxes), NaN if any of them is NaN.  The group cull classifies these
// first, so a group proven culled skips its members' boxes.
__global__ void __launch_bounds__(256) k_group_boxes(const float* boxes, uint32_t n, float* out) {
    static_assert(CR_GROUP == 32, "one lane per member box");
    const int lane = threadIdx.x & 31;
    const uint32_t nGroups = (n + CR_GROUP - 1) / CR_GROUP;
    for (uint32_t gi = blockIdx.x * 8 + (threadIdx.x >> 5); gi < nGroups; gi += gridDim.x * 8) {
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        bool bad = false;
        const uint32_t b = gi * CR_GROUP + lane;
        if (b < n) {
            const float* q = boxes + 6ull * b;
            for (int j = 0; j < 3; ++j) {
                const float l = q[j], h = q[3 + j];
                bad |= !(l <= h);  // NaN boxes
                lo[j] = l;
                hi[j] = h;
            }
        }
        warp_write_box(lo, hi, bad, out + 6ull * gi, lane);
    }
}

// One block: the union of the item boxes (a NaN box makes it NaN).
__global__ void __launch_bounds__(256) k_mesh_box(const float* itemBoxes, uint32_t nItems, float* out) {
    __shared__ float s_lo[3][8], s_hi[3][8];
    __shared__ int s_bad[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool bad = false;
    for (uint32_t b = threadIdx.x; b < nItems; b += 256) {
        const float* q = itemBoxes + 6ull * b;
        for (int j = 0; j < 3; ++j) {
            const float l = __ldg(q + j), h = __ldg(q + 3 + j);
            bad |= !(l <= h);  // NaN boxes
            lo[j] = fminf(lo[j], l);
            hi[j] = fmaxf(hi[j], h);
        }
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            lo[j] = fminf(lo[j], __shfl_xor_sync(FULL, lo[j], d));
            hi[j] = fmaxf(hi[j], __shfl_xor_sync(FULL, hi[j], d));
        }
    bad = __any_sync(FULL, bad);
    if (lane == 0) {
        for (int j = 0; j < 3; ++j) {
            s_lo[j][w] = lo[j];
            s_hi[j][w] = hi[j];
        }
        s_bad[w] = bad;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int j = threadIdx.x % 3;
        float v = threadIdx.x < 3 ? INFINITY : -INFINITY;
        int anyBad = 0;
        for (int k = 0; k < 8; ++k) {
            v = threadIdx.x < 3 ? fminf(v, s_lo[j][k]) : fmaxf(v, s_hi[j][k]);
            anyBad |= s_bad[k];
        }
        out[threadIdx.x] = (anyBad || nItems == 0) ? __int_as_float(0x7fffffff) : v;
    }
}

}  // namespace

int cr_launch_sub_obbs(const uint32_t* indices, const float* positions, const CrCodec* codec, uint32_t numTriangles,
                       float4* subObbs, float* subCones, void* stream) {
    const uint32_t blocks = ((numTriangles + CR_SUB - 1) / CR_SUB + 15) / 16;
    if (!blocks) return 0;
    k_obbs<CR_SUB, 1><<<blocks < 148 * 16 ? blocks : 148 * 16, 256, 0, (cudaStream_t)stream>>>(
        indices, positions, codec, numTriangles, subObbs);
    k_cones<CR_SUB, 1><<<blocks < 148 * 16 ? blocks : 148 * 16, 256, 0, (cudaStream_t)stream>>>(
        indices, positions, codec, numTriangles, subCones);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int cr_launch_mesh_boxes(const uint32_t* indices, const float* positions, const CrCodec* codec,
                         uint32_t numTriangles, uint32_t numVertices, float* itemBoxes, float* chunkBoxes,
                         float* meshBox, float* groupBoxes, float* chunkGroupBoxes, float* itemCones,
                         uint4* itemSlices, float4* itemObbs, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t nItems = (numTriangles + CR_BATCH - 1) / CR_BATCH;
    const uint32_t nChunks = (numVertices + CR_VCHUNK - 1) / CR_VCHUNK;
    if (nItems) k_item_boxes<<<(nItems + 7) / 8 < 148 * 16 ? (nItems + 7) / 8 : 148 * 16, 256, 0, st>>>(
        indices, positions, codec, numTriangles, itemBoxes);
    if (nItems && itemObbs)
        k_obbs<32, 4><<<(nItems + 7) / 8 < 148 * 16 ? (nItems + 7) / 8 : 148 * 16, 256, 0, st>>>(
            indices, positions, codec, numTriangles, itemObbs);
    if (nChunks) k_chunk_boxes<<<(nChunks + 7) / 8 < 148 * 16 ? (nChunks + 7) / 8 : 148 * 16, 256, 0, st>>>(
        positions, codec, numVertices, chunkBoxes);
    const uint32_t nGroups = (nItems + CR_GROUP - 1) / CR_GROUP;
    const uint32_t nCGroups = (nChunks + CR_GROUP - 1) / CR_GROUP;
    if (nGroups && groupBoxes)
        k_group_boxes<<<(nGroups + 7) / 8 < 148 * 16 ? (nGroups + 7) / 8 : 148 * 16, 256, 0, st>>>(itemBoxes, nItems,
                                                                                                 groupBoxes);
    if (nCGroups && chunkGroupBoxes)
        k_group_boxes<<<(nCGroups + 7) / 8 < 148 * 16 ? (nCGroups + 7) / 8 : 148 * 16, 256, 0, st>>>(
            chunkBoxes, nChunks, chunkGroupBoxes);
    if (nItems && itemCones)
        k_cones<32, 4><<<(nItems + 7) / 8 < 148 * 16 ? (nItems + 7) / 8 : 148 * 16, 256, 0, st>>>(
            indices, positions, codec, numTriangles, itemCones);
    const uint32_t nSlices = (numVertices + CR_VSLICE - 1) / CR_VSLICE;
    if (nItems && nSlices && itemSlices)
        k_item_slices<<<(nItems + 7) / 8 < 148 * 16 ? (nItems + 7) / 8 : 148 * 16, 256, 0, st>>>(
            indices, positions, codec, numTriangles, nSlices, itemSlices);
    if (meshBox) k_mesh_box<<<1, 256, 0, st>>>(itemBoxes, nItems, meshBox);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
