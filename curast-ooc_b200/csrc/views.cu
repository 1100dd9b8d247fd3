// views.cu -- batched multi-view kernels for sm_100a: up to 64 views of one
// instance set rendered by one launch per stage.
//
// No counterpart in the reference, which renders one view per CuRast::draw
// (src/CuRast_render.h:356-592).  Every (triangle, view) pair goes through
// exactly the reference's per-view decisions -- the same stage-1 function,
// the same stage-2 setup and fragment loop and the same stage-3 ray tracer as
// the single-view kernels, on the same float values -- so each view's
// visbuffer is bit-identical to a single-view render of that view.  What is
// shared across views is everything that does not depend on the view:
//
//   vertex   positions are read once and one CrViewMasks record per vertex
//            is written (behind / beyond each frustum side, one bit per
//            view).  The bounding box of each warp's 128 consecutive vertices
//            is first classified against each view's frustum with a rigorous
//            float error bound (classify_chunk); only the views the box
//            straddles are evaluated per vertex.
//   stage 1  a work item's 1536-byte index tile is fetched once (bulk TMA
//            copy into a per-warp ring, as the single-view stage 1) and its
//            triangles' records are gathered once; three 64-bit AND/OR
//            chains give each triangle the set of views in which it survives
//            the all-behind / all-beyond-one-side culls.  The warp then
//            visits, view by view, every view in which any of its triangles
//            survives: that view's survivors are packed across the lanes (as
//            the single-view stage 1 packs its survivors) and run the
//            reference's full per-triangle path with the view's target and
//            matrix, which are the same for the whole warp.  Queue entries
//            carry their view (view << 58 | instance << 32 | triangle).
//   stage 2/3  the single-view kernels instantiated with MULTI = true: each
//            queued entry / tile reads its own view's target and matrix.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "raster_core.cuh"

namespace {

constexpr int VV_THREADS = 256;
constexpr int VV_PER_THREAD = CR_VCHUNK / VV_THREADS;  // 4 vertices per thread

// vertex_outcode with the matrix given as its x, y, z rows: the same float
// operations in the same order as xform.
__device__ __forceinline__ uint32_t outcode_rows(const float4 rx, const float4 ry, const float4 rz, V3 p, float fa,
                                                 float f) {
    const float qz = (rz.x * p.x + rz.y * p.y) + (rz.z * p.z + rz.w * 1.0f);
    const float d = -qz;
    if (d <= 0.0f) return CR_OC_BEHIND;
    const float qx = (rx.x * p.x + rx.y * p.y) + (rx.z * p.z + rx.w * 1.0f);
    const float qy = (ry.x * p.x + ry.y * p.y) + (ry.z * p.z + ry.w * 1.0f);
    const float X = fa * qx, Y = f * qy;
    return (ndc_beyond(X, d) ? CR_OC_RIGHT : 0u) | (ndc_beyond(-X, d) ? CR_OC_LEFT : 0u) |
           (ndc_beyond(Y, d) ? CR_OC_TOP : 0u) | (ndc_beyond(-Y, d) ? CR_OC_BOTTOM : 0u);
}

__device__ __forceinline__ unsigned long long valid_views(uint32_t n) {
    return n >= 64 ? ~0ull : ((1ull << n) - 1ull);
}

// One block per 1024-vertex chunk of one instance; each warp owns 128
// consecutive vertices (lane + 32 k), classifies their bounding box against
// every view (two views per lane) and evaluates per vertex only the views the
// box straddles.  Consecutive vertices of a mesh are usually close (a grid
// row, a patch), so a 128-vertex box is small and most views classify it as a
// whole: entirely behind, entirely beyond one side, or entirely inside.
__global__ void __launch_bounds__(VV_THREADS) k_vertex_views(const CrFrameParams p) {
    __shared__ float4 s_rows[CR_MAX_VIEWS][3];
    __shared__ float s_fa[CR_MAX_VIEWS], s_f[CR_MAX_VIEWS];
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const uint32_t nViews = p.numViews;
    const unsigned long long valid = valid_views(nViews);

    // the chunks the frame cull left for per-vertex records (or every chunk)
    const uint64_t nChunks = p.chunkList ? min((uint64_t)p.counters[CR_CTR_CHUNKS], p.numVChunks) : p.numVChunks;
    for (uint64_t k = blockIdx.x; k < nChunks; k += gridDim.x) {
        const uint64_t c = p.chunkList ? (uint64_t)__ldg(p.chunkList + k) : k;
        uint32_t lo = 0, hi = p.numInstances - 1;  // instance holding chunk c
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (__ldg(&p.instances[mid].vchunkBase) <= c) lo = mid;
            else hi = mid - 1;
        }
        const uint32_t inst = lo;
        const CrInstance* I = p.instances + inst;
        const uint32_t nV = __ldg(&I->numVertices);
        const uint32_t vw = (uint32_t)(c - __ldg(&I->vchunkBase)) * CR_VCHUNK + (uint32_t)warp * (32 * VV_PER_THREAD);
        const GeomRef g = geom_of(I);

        // the views' matrix rows of this instance, once per chunk
        if (tid < CR_MAX_VIEWS && (uint32_t)tid < nViews) {
            const Mat M = load_mat(p.world_view + 4ull * ((uint64_t)tid * p.numInstances + inst));
            s_rows[tid][0] = make_float4(M.c0.x, M.c1.x, M.c2.x, M.c3.x);
            s_rows[tid][1] = make_float4(M.c0.y, M.c1.y, M.c2.y, M.c3.y);
            s_rows[tid][2] = make_float4(M.c0.z, M.c1.z, M.c2.z, M.c3.z);
            s_fa[tid] = __ldg(&p.views[tid].fa);
            s_f[tid] = __ldg(&p.views[tid].f);
        }
        // this lane's vertices and the warp's bounding box
        V3 pv[VV_PER_THREAD];
        float bl[3] = {INFINITY, INFINITY, INFINITY}, bh[3] = {-INFINITY, -INFINITY, -INFINITY};
        bool bad = false;
#pragma unroll
        for (int k = 0; k < VV_PER_THREAD; ++k) {
            const uint32_t v = vw + lane + 32 * k;
            pv[k] = v < nV ? pos_of(g, v) : V3{0.0f, 0.0f, 0.0f};
            if (v < nV) {
                bad |= !(isfinite(pv[k].x) && isfinite(pv[k].y) && isfinite(pv[k].z));
                bl[0] = fminf(bl[0], pv[k].x); bh[0] = fmaxf(bh[0], pv[k].x);
                bl[1] = fminf(bl[1], pv[k].y); bh[1] = fmaxf(bh[1], pv[k].y);
                bl[2] = fminf(bl[2], pv[k].z); bh[2] = fmaxf(bh[2], pv[k].z);
            }
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                bl[j] = fminf(bl[j], __shfl_xor_sync(FULL, bl[j], d));
                bh[j] = fmaxf(bh[j], __shfl_xor_sync(FULL, bh[j], d));
            }
        }
        const bool anyBad = __any_sync(FULL, bad);
        __syncthreads();  // s_rows ready

        // classes of the warp's box: lane classifies views lane and lane + 32
        uint32_t cls[2] = {0u, 0u};
        const bool anyVertex = bl[0] <= bh[0];  // false only past the mesh's end
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t v = (uint32_t)lane + 32u * h;
            if (v < nViews && !anyBad && anyVertex)
                cls[h] = classify_chunk(s_rows[v][0], s_rows[v][1], s_rows[v][2], s_fa[v], s_f[v], bl, bh);
        }
        auto cls64 = [&](uint32_t b) -> unsigned long long {
            const unsigned lo32 = __ballot_sync(FULL, cls[0] & b), hi32 = __ballot_sync(FULL, cls[1] & b);
            return (((unsigned long long)hi32 << 32) | lo32) & valid;
        };
        const unsigned long long cB = cls64(CH_BEHIND), cR = cls64(CH_RIGHT), cL = cls64(CH_LEFT),
                                 cT = cls64(CH_TOP), cO = cls64(CH_BOTTOM), cI = cls64(CH_INSIDE);
        unsigned long long mixed = anyVertex ? valid & ~(cB | cR | cL | cT | cO | cI) : 0ull;

        unsigned long long mb[VV_PER_THREAD], mr[VV_PER_THREAD], ml[VV_PER_THREAD], mt[VV_PER_THREAD],
            mo[VV_PER_THREAD];
#pragma unroll
        for (int k = 0; k < VV_PER_THREAD; ++k) {
            mb[k] = cB;
            mr[k] = cR;
            ml[k] = cL;
            mt[k] = cT;
            mo[k] = cO;
        }
        while (mixed) {  // uniform across the warp
            const int v = __ffsll((long long)mixed) - 1;
            mixed &= mixed - 1;
            const float4 rx = s_rows[v][0], ry = s_rows[v][1], rz = s_rows[v][2];
            const float fa = s_fa[v], f = s_f[v];
            const unsigned long long bit = 1ull << v;
#pragma unroll
            for (int k = 0; k < VV_PER_THREAD; ++k) {
                const uint32_t o = outcode_rows(rx, ry, rz, pv[k], fa, f);
                mb[k] |= (o & CR_OC_BEHIND) ? bit : 0ull;
                mr[k] |= (o & CR_OC_RIGHT) ? bit : 0ull;
                ml[k] |= (o & CR_OC_LEFT) ? bit : 0ull;
                mt[k] |= (o & CR_OC_TOP) ? bit : 0ull;
                mo[k] |= (o & CR_OC_BOTTOM) ? bit : 0ull;
            }
        }
        CrViewMasks* out = p.viewMasks + __ldg(&I->outBase);
#pragma unroll
        for (int k = 0; k < VV_PER_THREAD; ++k) {
            const uint32_t v = vw + lane + 32 * k;
            if (v < nV) {
                ulonglong2* r = reinterpret_cast<ulonglong2*>(out + v);
                r[0] = make_ulonglong2(mb[k], mr[k]);
                r[1] = make_ulonglong2(ml[k], mt[k]);
                r[2] = make_ulonglong2(mo[k], 0ull);
            }
        }
        __syncthreads();  // s_rows are rewritten for the next chunk
    }
}

// The record of vertex v of an instance: its chunk's record where the frame
// cull proved the chunk uniform in every view, else the vertex pass's.
__device__ __forceinline__ const ulonglong2* record_of(const CrFrameParams& p, const CrViewMasks* rec,
                                                       uint64_t vchunkBase, uint32_t v) {
    if (p.chunkUniform) {
        const uint64_t c = vchunkBase + v / CR_VCHUNK;
        if (__ldg(p.chunkUniform + c)) return reinterpret_cast<const ulonglong2*>(p.chunkMasks + c);
    }
    return reinterpret_cast<const ulonglong2*>(rec + v);
}

// Views of one triangle that survive the all-behind and all-beyond-one-side
// culls (tv.cu:110-119) given its three vertex records.
__device__ __forceinline__ unsigned long long surviving_views(const CrFrameParams& p, const CrViewMasks* rec,
                                                              uint64_t vchunkBase, uint32_t i0, uint32_t i1,
                                                              uint32_t i2, unsigned long long valid) {
    const ulonglong2* a = record_of(p, rec, vchunkBase, i0);
    const ulonglong2* b = record_of(p, rec, vchunkBase, i1);
    const ulonglong2* c = record_of(p, rec, vchunkBase, i2);
    const ulonglong2 a0 = __ldg(a), a1 = __ldg(a + 1), a2 = __ldg(a + 2);
    const ulonglong2 b0 = __ldg(b), b1 = __ldg(b + 1), b2 = __ldg(b + 2);
    const ulonglong2 c0 = __ldg(c), c1 = __ldg(c + 1), c2 = __ldg(c + 2);
    const unsigned long long allB = a0.x & b0.x & c0.x;
    const unsigned long long anyB = a0.x | b0.x | c0.x;
    const unsigned long long side =
        (a0.y & b0.y & c0.y) | (a1.x & b1.x & c1.x) | (a1.y & b1.y & c1.y) | (a2.x & b2.x & c2.x);
    return valid & ~(allB | (~anyB & side));
}

// MINB: resident blocks per SM the register allocation must allow (a tuning
// knob: more warps to hide latency against fewer registers per thread).
// PACKED: compiled for frames with compressed meshes.
template <int WARPS, int MINB, bool PACKED>
__global__ void __launch_bounds__(WARPS * 32, MINB) k_stage1_views(const CrFrameParams p) {
    __shared__ __align__(128) uint32_t s_idx[WARPS][S1_STAGES][CR_BATCH * 3];
    __shared__ __align__(8) uint64_t s_bar[WARPS][S1_STAGES];
    __shared__ uint8_t s_surv[WARPS][CR_BATCH];
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const uint64_t gw = (uint64_t)blockIdx.x * WARPS + w;
    const uint64_t nw = (uint64_t)gridDim.x * WARPS;
    const unsigned long long valid = valid_views(p.numViews);

    if (lane == 0) {
        for (int s = 0; s < S1_STAGES; ++s) mbar_init(&s_bar[w][s], 1);
        fence_barrier_init();
    }
    __syncwarp();
    // work items: the frame cull's survivors with their views, or every item
    const uint64_t nItems = p.itemViews ? min((uint64_t)p.counters[CR_CTR_ITEMS], p.itemCap) : p.numItems;
    auto item_at = [&](uint64_t k) -> uint64_t { return p.itemViews ? (uint64_t)__ldg(&p.itemViews[k].item) : k; };
    uint32_t pending = 0;  // ring slots with an issued, unconsumed copy
    for (int s = 0; s < S1_STAGES; ++s) {
        const uint64_t pk = gw + (uint64_t)s * nw;
        if (pk >= nItems) break;
        const Item it = decode_item(p, item_at(pk));
        const CrSegment* sg = p.segments + it.seg;
        if (item_uses_tma(sg, it.batch)) {
            pending |= 1u << s;
            if (lane == 0)
                bulk_load(s_idx[w][s], ldg_ptr(&sg->indices) + (uint64_t)it.batch * (CR_BATCH * 3), CR_BATCH * 12,
                          &s_bar[w][s]);
        }
    }
    __syncwarp();

    uint32_t parity = 0;
    uint32_t k = 0;
    for (uint64_t pk = gw; pk < nItems; pk += nw, ++k) {
        const int slot = (int)(k % S1_STAGES);
        const uint32_t bit = 1u << slot;
        const Item it = decode_item(p, item_at(pk));
        // views of the item; records are gathered only for those its box
        // straddles (in the others every vertex is inside the frustum)
        const unsigned long long itemViews = p.itemViews ? __ldg(&p.itemViews[pk].views) & valid : valid;
        const unsigned long long itemStraddle = p.itemViews ? __ldg(&p.itemViews[pk].straddle) & itemViews : valid;
        const unsigned long long itemInside = itemViews & ~itemStraddle;
        const CrSegment* sg = p.segments + it.seg;
        const uint32_t numTri = __ldg(&sg->numTriangles);
        const GeomRef geo = geom_of_t<PACKED>(sg);
        const bool tma = item_uses_tma(sg, it.batch);
        const uint32_t tri0 = it.batch * CR_BATCH;
        if (tma) {
            const bool ok =
                __all_sync(FULL, mbar_wait_bounded(&s_bar[w][slot], (parity & bit) ? 1u : 0u, p.waitTimeoutNs));
            if (!ok) {
                if (lane == 0) atomicOr(&p.counters[CR_CTR_TIMEOUT], 1ull);
                break;
            }
            parity ^= bit;
            pending &= ~bit;
        }
        auto index_of = [&](uint32_t pos, int c) -> uint32_t {
            if (tma) return s_idx[w][slot][3 * pos + c];
            return geom_index(geo, 3ull * (tri0 + pos) + c);
        };

        const uint32_t first = __ldg(&sg->firstInstance);
        const uint32_t count = __ldg(&sg->instanceCount);
        const uint32_t ib = first + it.chunk * CR_INST_CHUNK;
        const uint32_t ie = min(ib + CR_INST_CHUNK, first + count);
        for (uint32_t inst = ib; inst < ie; ++inst) {
            const CrViewMasks* rec = p.viewMasks + __ldg(&p.instances[inst].outBase);
            const uint64_t vcb = __ldg(&p.instances[inst].vchunkBase);
            unsigned long long m[S1_R];
#pragma unroll
            for (int r = 0; r < S1_R; ++r) {
                const uint32_t tp = r * 32 + lane;
                m[r] = 0ull;
                if (tri0 + tp < numTri)
                    m[r] = itemInside | (itemStraddle ? surviving_views(p, rec, vcb, index_of(tp, 0), index_of(tp, 1),
                                                                        index_of(tp, 2), itemStraddle)
                                                      : 0ull);
            }
            // views in which any of the warp's triangles survives, in order;
            // per view the surviving triangles are packed across the lanes
            // and run the reference's per-triangle path with that view's
            // (warp-uniform) target and matrix
            const unsigned long long any = m[0] | m[1] | m[2] | m[3];
            unsigned long long todo = ((unsigned long long)__reduce_or_sync(FULL, (unsigned)(any >> 32)) << 32) |
                                      __reduce_or_sync(FULL, (unsigned)any);
            if (!todo) continue;
            const uint64_t cum = __ldg(&p.instances[inst].cum);
            while (todo) {
                const uint32_t view = (uint32_t)(__ffsll((long long)todo) - 1);
                todo &= todo - 1ull;
                int nsurv = 0;
#pragma unroll
                for (int r = 0; r < S1_R; ++r) {
                    const bool in = (m[r] >> view) & 1ull;
                    const unsigned bm = __ballot_sync(FULL, in);
                    if (in) s_surv[w][nsurv + __popc(bm & ((1u << lane) - 1u))] = (uint8_t)(r * 32 + lane);
                    nsurv += __popc(bm);
                }
                __syncwarp();
                const uint64_t vi = (uint64_t)view * p.numInstances + inst;
                const Target tg = target_of(p, view);
                const Mat M = load_mat(p.world_view + 4ull * vi);
                const uint32_t flip = __ldg(p.flips + vi);
                const uint64_t entryHi = ((uint64_t)view << CR_ENTRY_VIEW_SHIFT) | ((uint64_t)inst << 32);
                for (int base = 0; base < nsurv; base += 32) {
                    const int j = base + lane;
                    int res = S1_CULL;
                    uint32_t tri = 0;
                    if (j < nsurv) {
                        const uint32_t tp = s_surv[w][j];
                        tri = tri0 + tp;
                        const V3 pa = pos_of(geo, index_of(tp, 0));
                        const V3 pb = pos_of(geo, index_of(tp, 1));
                        const V3 pc = pos_of(geo, index_of(tp, 2));
                        res = stage1_triangle(tg, tg.fa, M, flip, pa, pb, pc, cum - tg.idBase + tri);
                    }
                    const unsigned qmask = __ballot_sync(FULL, res == S1_QUEUE);
                    if (qmask) {  // warp-aggregated append, tv.cu:190-197, tagged with the view
                        const int leader = __ffs(qmask) - 1;
                        unsigned long long b = 0;
                        if (lane == leader)
                            b = atomicAdd(&p.counters[CR_CTR_NONTRIVIAL], (unsigned long long)__popc(qmask));
                        b = __shfl_sync(FULL, b, leader);
                        if (res == S1_QUEUE) {
                            const uint64_t q = b + __popc(qmask & ((1u << lane) - 1u));
                            if (q < p.ntCap) p.ntList[q] = entryHi | tri;
                            else atomicOr(&p.counters[CR_CTR_OVERFLOW], 1ull);
                        }
                    }
                }
                __syncwarp();
            }
        }

        __syncwarp();
        {  // every read of this slot is done: refill it with the item S1_STAGES ahead
            const uint64_t nxt = pk + (uint64_t)S1_STAGES * nw;
            if (nxt < nItems) {
                const Item nt = decode_item(p, item_at(nxt));
                const CrSegment* ns = p.segments + nt.seg;
                if (item_uses_tma(ns, nt.batch)) {
                    pending |= bit;
                    if (lane == 0) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        bulk_load(s_idx[w][slot], ldg_ptr(&ns->indices) + (uint64_t)nt.batch * (CR_BATCH * 3),
                                  CR_BATCH * 12, &s_bar[w][slot]);
                    }
                }
            }
        }
    }
    // only after a timeout can copies still be in flight: wait for them
    // (bounded) so none lands in shared memory after the block has exited
    for (int s = 0; s < S1_STAGES; ++s)
        if (pending & (1u << s)) (void)mbar_wait_bounded(&s_bar[w][s], (parity >> s) & 1u, p.waitTimeoutNs);
}

// Classes of one box (warp-uniform) in every view of `which` for one
// instance: lane classifies views lane and lane + 32; the six 64-bit masks
// (behind, right, left, top, bottom, inside) come from ballots.
struct ViewClasses {
    unsigned long long B, R, L, T, O, I;
};

__device__ __forceinline__ ViewClasses classify_views(const CrFrameParams& p, uint32_t inst, const float lo[3],
                                                      const float hi[3], unsigned long long which, int lane) {
    uint32_t cls[2] = {0u, 0u};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t v = (uint32_t)lane + 32u * h;
        if (v < p.numViews && ((which >> v) & 1ull)) {
            const Mat M = load_mat(p.world_view + 4ull * ((uint64_t)v * p.numInstances + inst));
            cls[h] = classify_box(M, __ldg(&p.views[v].fa), __ldg(&p.views[v].f), lo, hi);
        }
    }
    auto m64 = [&](uint32_t b) -> unsigned long long {
        const unsigned lo32 = __ballot_sync(FULL, cls[0] & b), hi32 = __ballot_sync(FULL, cls[1] & b);
        return ((unsigned long long)hi32 << 32) | lo32;
    };
    return ViewClasses{m64(CH_BEHIND), m64(CH_RIGHT), m64(CH_LEFT), m64(CH_TOP), m64(CH_BOTTOM), m64(CH_INSIDE)};
}

// The box of 32 lanes' boxes (lanes without one pass +inf / -inf).
__device__ __forceinline__ void warp_box(float lo[3], float hi[3]) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            lo[j] = fminf(lo[j], __shfl_xor_sync(FULL, lo[j], d));
            hi[j] = fmaxf(hi[j], __shfl_xor_sync(FULL, hi[j], d));
        }
}

__device__ __forceinline__ bool load_box(const float* b, float lo[3], float hi[3]) {
    for (int j = 0; j < 3; ++j) {
        lo[j] = __ldg(b + j);
        hi[j] = __ldg(b + 3 + j);
    }
    return lo[0] <= hi[0] && lo[1] <= hi[1] && lo[2] <= hi[2];  // false for NaN boxes
}

// Batched frame cull, before the vertex pass.  A warp takes 32 consecutive
// vertex chunks (then 32 consecutive work items): it classifies their common
// box against every view first (rigorous float bounds, classify_chunk), and
// each lane then classifies its own box only in the views the common box
// straddles.
//   chunks  a chunk no view straddles gets one record for all its vertices
//           (exact behind bits; side bits of the sides that prove it
//           outside) and no per-vertex pass; the others are listed for the
//           vertex pass.
//   items   an item whose box is wholly behind or beyond one side in a view
//           has every triangle culled there by the reference's own tests
//           (tv.cu:110-119); items are listed with the views left, and items
//           left with none are not visited by stage 1.
__global__ void __launch_bounds__(256) k_cull_views(const CrFrameParams p) {
    const int lane = threadIdx.x & 31;
    const uint64_t gwarp = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const uint64_t nwarps = (uint64_t)gridDim.x * 8;
    const unsigned long long valid = valid_views(p.numViews);
    const float INF = __int_as_float(0x7f800000);

    if (p.chunkList)
        for (uint64_t base = gwarp * 32; base < p.numVChunks; base += nwarps * 32) {
            const uint64_t g = base + lane;
            const bool has = g < p.numVChunks;
            uint32_t inst = 0;
            float lo[3] = {INF, INF, INF}, hi[3] = {-INF, -INF, -INF};
            bool boxOk = false;
            if (has) {
                uint32_t a = 0, b = p.numInstances - 1;  // instance holding chunk g
                while (a < b) {
                    const uint32_t mid = (a + b + 1) >> 1;
                    if (__ldg(&p.instances[mid].vchunkBase) <= g) a = mid;
                    else b = mid - 1;
                }
                inst = a;
                const float* cb = ldg_ptr(&p.instances[inst].chunkBoxes);
                if (cb) boxOk = load_box(cb + 6ull * (g - __ldg(&p.instances[inst].vchunkBase)), lo, hi);
                if (!boxOk) lo[0] = lo[1] = lo[2] = INF, hi[0] = hi[1] = hi[2] = -INF;
            }
            const uint32_t inst0 = __shfl_sync(FULL, inst, 0);
            const bool same = __all_sync(FULL, !has || (boxOk && inst == inst0));
            ViewClasses c{0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
            unsigned long long todo = valid;  // views this lane classifies alone
            if (same) {
                float glo[3] = {lo[0], lo[1], lo[2]}, ghi[3] = {hi[0], hi[1], hi[2]};
                warp_box(glo, ghi);
                c = classify_views(p, inst0, glo, ghi, valid, lane);
                todo = valid & ~(c.B | c.R | c.L | c.T | c.O | c.I);
            }
            if (has && boxOk) {
                while (todo) {
                    const uint32_t v = (uint32_t)(__ffsll((long long)todo) - 1);
                    todo &= todo - 1ull;
                    const Mat M = load_mat(p.world_view + 4ull * ((uint64_t)v * p.numInstances + inst));
                    const uint32_t k = classify_box(M, __ldg(&p.views[v].fa), __ldg(&p.views[v].f), lo, hi);
                    const unsigned long long bit = 1ull << v;
                    if (k & CH_BEHIND) c.B |= bit;
                    if (k & CH_RIGHT) c.R |= bit;
                    if (k & CH_LEFT) c.L |= bit;
                    if (k & CH_TOP) c.T |= bit;
                    if (k & CH_BOTTOM) c.O |= bit;
                    if (k & CH_INSIDE) c.I |= bit;
                }
            }
            const bool uniform = has && boxOk && !(valid & ~(c.B | c.R | c.L | c.T | c.O | c.I));
            if (has) {
                p.chunkUniform[g] = uniform ? 1 : 0;
                if (uniform) {
                    ulonglong2* r = reinterpret_cast<ulonglong2*>(p.chunkMasks + g);
                    r[0] = make_ulonglong2(c.B, c.R);
                    r[1] = make_ulonglong2(c.L, c.T);
                    r[2] = make_ulonglong2(c.O, 0ull);
                }
            }
            const unsigned m = __ballot_sync(FULL, has && !uniform);
            if (m) {
                const int leader = __ffs(m) - 1;
                unsigned long long b = 0;
                if (lane == leader) b = atomicAdd(&p.counters[CR_CTR_CHUNKS], (unsigned long long)__popc(m));
                b = __shfl_sync(FULL, b, leader);
                if (has && !uniform) p.chunkList[b + __popc(m & ((1u << lane) - 1u))] = (uint32_t)g;
            }
        }

    if (!p.itemViews) return;
    for (uint64_t base = gwarp * 32; base < p.numItems; base += nwarps * 32) {
        const uint64_t item = base + lane;
        const bool has = item < p.numItems;
        uint32_t seg = 0, chunk = 0, ib = 0, ie = 0;
        float lo[3] = {INF, INF, INF}, hi[3] = {-INF, -INF, -INF};
        bool boxOk = false;
        if (has) {
            const Item it = decode_item(p, item);
            seg = it.seg;
            chunk = it.chunk;
            const CrSegment* sg = p.segments + it.seg;
            const uint32_t first = __ldg(&sg->firstInstance);
            ib = first + it.chunk * CR_INST_CHUNK;
            ie = min(ib + CR_INST_CHUNK, first + __ldg(&sg->instanceCount));
            const float* boxes = ldg_ptr(&sg->itemBoxes);
            if (boxes) boxOk = load_box(boxes + 6ull * it.batch, lo, hi);
            if (!boxOk) lo[0] = lo[1] = lo[2] = INF, hi[0] = hi[1] = hi[2] = -INF;
        }
        const uint32_t seg0 = __shfl_sync(FULL, seg, 0), chunk0 = __shfl_sync(FULL, chunk, 0);
        const bool same = __all_sync(FULL, !has || (boxOk && seg == seg0 && chunk == chunk0));
        unsigned long long views = 0ull, straddle = 0ull;
        // the item alone in view v: culled, wholly inside, or straddling
        auto classify_item = [&](uint32_t inst, uint32_t v) {
            const unsigned long long bit = 1ull << v;
            if (!boxOk) {
                views |= bit;
                straddle |= bit;
                return;
            }
            const Mat M = load_mat(p.world_view + 4ull * ((uint64_t)v * p.numInstances + inst));
            const uint32_t k = classify_box(M, __ldg(&p.views[v].fa), __ldg(&p.views[v].f), lo, hi);
            if (k & CR_OC_MASK) return;
            views |= bit;
            if (!(k & CH_INSIDE)) straddle |= bit;
        };
        if (same) {
            float glo[3] = {lo[0], lo[1], lo[2]}, ghi[3] = {hi[0], hi[1], hi[2]};
            warp_box(glo, ghi);
            const uint32_t gib = __shfl_sync(FULL, ib, 0), gie = __shfl_sync(FULL, ie, 0);
            for (uint32_t inst = gib; inst < gie; ++inst) {
                const ViewClasses c = classify_views(p, inst, glo, ghi, valid, lane);
                // views where the common box is culled cull every item, where
                // it is inside every item is inside; the items are classified
                // alone in the others
                const unsigned long long culled = c.B | c.R | c.L | c.T | c.O;
                views |= c.I;
                unsigned long long todo = valid & ~culled & ~c.I;
                if (has)
                    while (todo) {
                        const uint32_t v = (uint32_t)(__ffsll((long long)todo) - 1);
                        todo &= todo - 1ull;
                        classify_item(inst, v);
                    }
            }
        } else if (has) {
            for (uint32_t inst = ib; inst < ie; ++inst) {
                unsigned long long todo = valid;
                while (todo) {
                    const uint32_t v = (uint32_t)(__ffsll((long long)todo) - 1);
                    todo &= todo - 1ull;
                    classify_item(inst, v);
                }
            }
        }
        const bool keep = has && views != 0ull;
        const unsigned m = __ballot_sync(FULL, keep);
        if (m) {
            const int leader = __ffs(m) - 1;
            unsigned long long b = 0;
            if (lane == leader) b = atomicAdd(&p.counters[CR_CTR_ITEMS], (unsigned long long)__popc(m));
            b = __shfl_sync(FULL, b, leader);
            if (keep) {
                const uint64_t q = b + __popc(m & ((1u << lane) - 1u));
                if (q < p.itemCap) {
                    CrItemViews e;
                    e.views = views;
                    e.straddle = straddle;
                    e.item = (uint32_t)item;
                    e.pad = 0;
                    p.itemViews[q] = e;
                }
            }
        }
    }
}

// Stage 1 of batched frames from the frame cull's item list alone (no vertex
// pass runs).  Per (instance, view) of an item the warp proves, four views at a time
// (a lane per view and CR_SUB triangles), that an oriented sub-box misses every
// sample or that its triangles all face away, tests the triangles of the other sub-boxes
// one per lane (quick_misses), two sub-boxes at a time, and queues those still left for
// the reference's full path, 32 at a time across its items.  COARSE (views of half a
// pixel and more per triangle): the triangles are not tested ahead of the path, and the
// warp shares its lanes' rasters.
//
// Bound by instruction issue and by dependent arithmetic that 3 blocks of 80 registers
// do not hide (61 % of the slots, 8 views of a 4M terrain).  64 views over the
// 60M-triangle terrain (0.02 pixels per triangle; 33 % of the triangles face away,
// 52 % miss every sample, 13 % are drawn), ms:
// every triangle of an item that is large on screen through the full path, and cell
// records of the distinct vertices of the others, 18.4; quick_misses ahead of the path
// 14.0; indices by plain loads instead of a TMA tile per item, which freed 20 registers
// of spilled state, 13.2.  Where the triangles are larger the test is wasted and one
// lane's needle holds the others up: 33 views, fine / COARSE, ms: 732K triangles at
// 0.9 pixels each 0.578 / 0.500, at 3.5 1.04 / 0.80, 180K at 14 0.69 / 0.42, 2.9M at 0.9
// 1.51 / 1.40; but 732K at 0.22 0.337 / 0.347, 2.9M at 0.05 0.56 / 0.74.
constexpr uint32_t V1_UNITS = 4;   // units of work per warp, at least
template <int WARPS, int MINB, bool PACKED, bool COARSE>
__global__ void __launch_bounds__(WARPS * 32, MINB) k_stage1_views_boxes(const CrFrameParams p) {
    __shared__ uint64_t s_ring[WARPS][S1_RING];
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const uint64_t gw = (uint64_t)blockIdx.x * WARPS + w;
    const uint64_t nw = (uint64_t)gridDim.x * WARPS;
    const unsigned long long valid = valid_views(p.numViews);

    const uint64_t nItems = min((uint64_t)p.counters[CR_CTR_ITEMS], p.itemCap);
    // Some units of work per warp: an item, or its part in `per` consecutive views
    // where there are too few items (a 33-view frame of 180K triangles has 1,407 for
    // 3,552 warps: 0.375 -> 0.287 ms).  The parts of all items in the first views come
    // first: with an item's parts next to one another the views' targets
    // compete for L2 (2.9M triangles at 0.9 pixels 1.49 unsplit, 1.68; so 1.53).
    const uint32_t fours = (p.numViews + 3) / 4;
    const uint64_t parts = max((uint64_t)1, min((uint64_t)fours, (V1_UNITS * nw + nItems) / (nItems + 1)));
    const uint32_t per = 4 * (uint32_t)((fours + parts - 1) / parts);
    const uint32_t split = (p.numViews + per - 1) / per;

    // Triangles no proof culls, as stage-2 queue entries (view, instance,
    // triangle), queued across the warp's items and run through the reference's
    // full path 32 at a time.
    uint64_t* const ring = s_ring[w];
    uint32_t qh = 0, qt = 0;  // ring head / tail (warp-uniform)
    auto drain = [&]() {
        const uint32_t j = qh + lane;
        int res = S1_CULL;
        uint64_t e = 0;
        Target tg = {};
        S1Raster ras;
        uint64_t rid = 0;
        if (j < qt) {
            e = ring[j & (S1_RING - 1)];
            const uint32_t view = (uint32_t)(e >> CR_ENTRY_VIEW_SHIFT);
            const uint32_t inst = (uint32_t)((e >> 32) & CR_ENTRY_INST_MASK), tri = (uint32_t)e;
            const uint64_t vi = (uint64_t)view * p.numInstances + inst;
            tg = target_of(p, view);
            const CrInstance* I = p.instances + inst;
            const GeomRef g = geom_of_t<PACKED>(I);
            const V3 pa = pos_of(g, geom_index(g, 3ull * tri + 0));
            const V3 pb = pos_of(g, geom_index(g, 3ull * tri + 1));
            const V3 pc = pos_of(g, geom_index(g, 3ull * tri + 2));
            rid = __ldg(&I->cum) - tg.idBase + tri;
            res = stage1_triangle<COARSE, true>(tg, tg.fa, load_mat(p.world_view + 4ull * vi), __ldg(p.flips + vi), pa, pb, pc, rid,
                                                 &ras);
        }
        if constexpr (COARSE) s1_raster_lanes<true>(tg, res, ras, rid);
        qh = min(qh + 32u, qt);
        const unsigned qmask = __ballot_sync(FULL, res == S1_QUEUE);
        if (qmask) {  // warp-aggregated append, tv.cu:190-197, tagged with the view
            const int leader = __ffs(qmask) - 1;
            unsigned long long b = 0;
            if (lane == leader) b = atomicAdd(&p.counters[CR_CTR_NONTRIVIAL], (unsigned long long)__popc(qmask));
            b = __shfl_sync(FULL, b, leader);
            if (res == S1_QUEUE) {
                const uint64_t q = b + __popc(qmask & ((1u << lane) - 1u));
                if (q < p.ntCap) p.ntList[q] = e;
                else atomicOr(&p.counters[CR_CTR_OVERFLOW], 1ull);
            }
        }
        __syncwarp();
    };
    uint64_t pk = gw;
    for (uint32_t part = 0; nItems; pk += nw) {
        while (pk >= nItems && part < split) {
            pk -= nItems;
            ++part;
        }
        if (part >= split) break;
        const unsigned long long partViews = (per < 64 ? (1ull << per) - 1ull : ~0ull) << (part * per);
        const unsigned long long itemViews = __ldg(&p.itemViews[pk].views) & valid & partViews;
        if (!itemViews) continue;
        const Item it = decode_item(p, (uint64_t)__ldg(&p.itemViews[pk].item));
        const CrSegment* sg = p.segments + it.seg;
        const uint32_t numTri = __ldg(&sg->numTriangles);
        const GeomRef geo = geom_of_t<PACKED>(sg);
        const uint32_t tri0 = it.batch * CR_BATCH;
        const uint32_t first = __ldg(&sg->firstInstance);
        const uint32_t ib = first + it.chunk * CR_INST_CHUNK;
        const uint32_t ie = min(ib + CR_INST_CHUNK, first + __ldg(&sg->instanceCount));
        // this lane's sub-box (lane & 7); read again for every four views (it
        // stays in L1), so that it holds no registers over the full path
        const float4* obbs = ldg_ptr(&sg->subObbs);
        const float4* cones = ldg_ptr(&sg->subCones);
        const uint64_t sub = (uint64_t)it.batch * (CR_BATCH / CR_SUB) + (lane & 7);
        const bool hasSub = CR_SUB * (uint32_t)(lane & 7) < numTri - tri0;
        V3 itemAbs = {};
        if (obbs && hasSub) itemAbs = obb_max_abs(load_obb(obbs + CR_OBB_F4 * sub));
        // the largest coordinates in the whole item, for quick_misses.  A sub-box with a
        // vertex that is not finite or is huge has a NaN centre and bounds none of its
        // vertices: the item's bound is then infinite, and nothing of it is dropped
        // (fmaxf would lose the NaN).
        if (!(itemAbs.x < INFINITY)) itemAbs = V3{INFINITY, INFINITY, INFINITY};
#pragma unroll
        for (int d = 4; d >= 1; d >>= 1) {
            itemAbs.x = fmaxf(itemAbs.x, __shfl_xor_sync(FULL, itemAbs.x, d));
            itemAbs.y = fmaxf(itemAbs.y, __shfl_xor_sync(FULL, itemAbs.y, d));
            itemAbs.z = fmaxf(itemAbs.z, __shfl_xor_sync(FULL, itemAbs.z, d));
        }
        for (uint32_t inst = ib; inst < ie; ++inst) {
            unsigned long long todo = itemViews;
            while (todo) {
                // the next four views; view (lane >> 3) of them is this lane's
                unsigned long long four = todo;
                uint32_t mine = CR_MAX_VIEWS;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!todo) break;
                    if ((lane >> 3) == i) mine = (uint32_t)(__ffsll((long long)todo) - 1);
                    todo &= todo - 1ull;
                }
                four &= ~todo;
                bool keep = mine < CR_MAX_VIEWS && hasSub;
                if (keep && obbs) {
                    const Target tg = target_of(p, mine);
                    const uint64_t vi = (uint64_t)mine * p.numInstances + inst;
                    const Obb ob = load_obb(obbs + CR_OBB_F4 * sub);
                    Proof P = proof_rows(load_mat(p.world_view + 4ull * vi), obb_max_abs(ob));
                    P.eye = __ldg(p.instProof + 2 * vi);
                    P.det = __ldg(p.instProof + 2 * vi + 1);
                    keep = !item_back_facing(P, __ldg(cones + 2 * sub), __ldg(cones + 2 * sub + 1), ob.c, obb_radius(ob)) &&
                           !obb_misses_samples(P, tg.fa, tg.f, (float)tg.W, (float)tg.H, ob);
                }
                const uint32_t kept = __ballot_sync(FULL, keep);
#pragma unroll 1
                for (int i = 0; i < 4 && four; ++i) {
                    const uint32_t view = (uint32_t)(__ffsll((long long)four) - 1);
                    four &= four - 1ull;
                    uint32_t rest = (kept >> (8 * i)) & 0xffu;
                    if (!rest) continue;
                    const Target tg = target_of(p, view);
                    const Quick Q = make_quick(
                        proof_rows(load_mat(p.world_view + 4ull * ((uint64_t)view * p.numInstances + inst)), itemAbs),
                        tg.fa, tg.f, (float)tg.W, (float)tg.H);
                    const uint64_t entry = ((uint64_t)view << CR_ENTRY_VIEW_SHIFT) | ((uint64_t)inst << 32) | tri0;
                    while (rest) {
                        const uint32_t b0 = (uint32_t)__ffs(rest) - 1;
                        rest &= rest - 1;
                        const uint32_t b1 = rest ? (uint32_t)__ffs(rest) - 1 : 8u;
                        rest &= rest - 1;
                        const uint32_t tp = CR_SUB * (lane < 16 ? b0 : b1) + (uint32_t)(lane & 15);
                        bool left = tp < CR_BATCH && tri0 + tp < numTri;
                        if (!COARSE && left && obbs)
                            left = !quick_misses(Q, pos_of(geo, geom_index(geo, 3ull * (tri0 + tp) + 0)),
                                                 pos_of(geo, geom_index(geo, 3ull * (tri0 + tp) + 1)),
                                                 pos_of(geo, geom_index(geo, 3ull * (tri0 + tp) + 2)));
                        const unsigned m = __ballot_sync(FULL, left);
                        if (left) ring[(qt + __popc(m & ((1u << lane) - 1u))) & (S1_RING - 1)] = entry + tp;
                        qt += __popc(m);
                        __syncwarp();
                        if (qt - qh >= 32u) drain();
                    }
                }
            }
        }
    }
    if (qt > qh) drain();
}

// The back-face proof's data of every (view, instance): proof_data of api.cpp, a
// thread each (64 views of thousands of instances would take the host longer
// than the frame takes).  Two float4 per entry: eye and |eye|; |det|, |R|_F, the largest
// row sum of |R| and |t|.
__global__ void __launch_bounds__(256) k_view_proofs(const float4* wv, uint32_t n, float4* out) {
    const uint32_t k = blockIdx.x * 256 + threadIdx.x;
    if (k >= n) return;
    const Mat M = load_mat(wv + 4ull * k);
    const double r00 = M.c0.x, r01 = M.c1.x, r02 = M.c2.x, r10 = M.c0.y, r11 = M.c1.y, r12 = M.c2.y, r20 = M.c0.z,
                 r21 = M.c1.z, r22 = M.c2.z, t0 = M.c3.x, t1 = M.c3.y, t2 = M.c3.z;
    const double a00 = r11 * r22 - r12 * r21, a01 = r02 * r21 - r01 * r22, a02 = r01 * r12 - r02 * r11,
                 a10 = r12 * r20 - r10 * r22, a11 = r00 * r22 - r02 * r20, a12 = r02 * r10 - r00 * r12,
                 a20 = r10 * r21 - r11 * r20, a21 = r01 * r20 - r00 * r21, a22 = r00 * r11 - r01 * r10;
    const double det = r00 * a00 + r01 * a10 + r02 * a20;
    const double had = (fabs(r00) + fabs(r10) + fabs(r20)) * (fabs(r01) + fabs(r11) + fabs(r21)) *
                       (fabs(r02) + fabs(r12) + fabs(r22));
    const double frob = r00 * r00 + r01 * r01 + r02 * r02 + r10 * r10 + r11 * r11 + r12 * r12 + r20 * r20 + r21 * r21 +
                        r22 * r22;
    const double row = fmax(fabs(r00) + fabs(r01) + fabs(r02),
                            fmax(fabs(r10) + fabs(r11) + fabs(r12), fabs(r20) + fabs(r21) + fabs(r22)));
    const double tAbs = fmax(fabs(t0), fmax(fabs(t1), fabs(t2)));
    const double e0 = -(a00 * t0 + a01 * t1 + a02 * t2) / det, e1 = -(a10 * t0 + a11 * t1 + a12 * t2) / det,
                 e2 = -(a20 * t0 + a21 * t1 + a22 * t2) / det;
    const bool ok = isfinite(det) && fabs(det) > 1e-4 * had && isfinite(e0) && isfinite(e1) && isfinite(e2) &&
                    isfinite(tAbs) && isfinite(frob);
    const double up = 1.0 + 1e-6;  // above the rounding to float
    out[2ull * k] = ok ? make_float4((float)e0, (float)e1, (float)e2, (float)(sqrt(e0 * e0 + e1 * e1 + e2 * e2) * up))
                       : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    out[2ull * k + 1] = make_float4(ok ? (float)(fabs(det) * (1.0 - 1e-6)) : 0.0f, (float)(sqrt(frob) * up),
                                    (float)(row * up), (float)(tAbs * up));
}

// Clears every view's visbuffer (resolve.cu:213-232); blockIdx.y is the view.
__global__ void __launch_bounds__(256) k_clear_views(const CrView* views, unsigned long long* counters) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < CR_CTR_COUNT) counters[threadIdx.x] = 0ull;
    const CrView* v = views + blockIdx.y;
    uint64_t* fb = ldg_ptr(&v->fb);
    const uint64_t n = (uint64_t)__ldg(&v->W) * (uint64_t)__ldg(&v->H);
    const uint64_t clearv = 0xFFFFFFF000000000ull;
    ulonglong2* q = reinterpret_cast<ulonglong2*>(fb);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n / 2; i += stride)
        q[i] = make_ulonglong2(clearv, clearv);
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) fb[n - 1] = clearv;
}

}  // namespace

constexpr int VS1_WARPS_MAX = 8;
// resident blocks per SM of k_stage1_views_boxes
constexpr int V1_MINB = 3;

int cr_query_batch_shape(int device, CrBatchShape* out) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return -1;
    int bv = 0, b1 = 0, b2 = 0, b3 = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bv, k_vertex_views, VV_THREADS, 0) != cudaSuccess) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_stage1_views<8, 2, false>, 256, 0) != cudaSuccess) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, k_stage2<8, true>, 256, 0) != cudaSuccess) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b3, k_stage3<8, true>, 256, 0) != cudaSuccess) return -1;
    out->numSMs = sms;
    out->vertexBlocks = sms * (bv > 0 ? bv : 1);
    out->stage1Blocks = sms * (b1 > 0 ? b1 : 1);
    out->stage2Blocks = sms * (b2 > 0 ? b2 : 1);
    out->stage3Blocks = sms * (b3 > 0 ? b3 : 1);
    out->stage1Warps = 8;
    out->stage2Warps = 8;
    return 0;
}

int cr_launch_clear_views(const CrFrameParams& p, uint64_t maxPixels, void* stream) {
    if (p.numViews == 0) return 0;
    const uint64_t want = (maxPixels / 2 + 255) / 256;
    const unsigned gx = (unsigned)(want < 1 ? 1 : (want > 148 * 4 ? 148 * 4 : want));
    k_clear_views<<<dim3(gx, p.numViews), 256, 0, (cudaStream_t)stream>>>(p.views, p.counters);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int cr_launch_vertex_views(const CrFrameParams& p, const CrBatchShape& s, void* stream) {
    if (p.numVChunks == 0 || p.numViews == 0 || p.cellMode == CR_REC_BOXES) return 0;
    uint64_t blocks = p.numVChunks;
    if (blocks > (uint64_t)s.vertexBlocks) blocks = (uint64_t)s.vertexBlocks;
    k_vertex_views<<<(unsigned)blocks, VV_THREADS, 0, (cudaStream_t)stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int cr_launch_cull_views(const CrFrameParams& p, const CrBatchShape& s, void* stream) {
    if (p.numViews == 0 || (!p.itemViews && !p.chunkList)) return 0;
    const uint64_t work = std::max<uint64_t>(p.numItems, p.chunkList ? p.numVChunks : 0);
    if (work == 0) return 0;
    uint64_t blocks = (work + 255) / 256;
    if (blocks > (uint64_t)s.numSMs * 8) blocks = (uint64_t)s.numSMs * 8;
    k_cull_views<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int cr_launch_stage1_views(const CrFrameParams& p, const CrBatchShape& s, void* stream) {
    if (p.numItems == 0 || p.numViews == 0) return 0;
    const int warps = s.stage1Warps == 4 ? 4 : VS1_WARPS_MAX;
    uint64_t blocks = (p.numItems + warps - 1) / warps;
    if (blocks > (uint64_t)s.stage1Blocks) blocks = (uint64_t)s.stage1Blocks;
    const unsigned b = (unsigned)blocks;
    cudaStream_t st = (cudaStream_t)stream;
    if (p.cellMode == CR_REC_BOXES && p.itemViews) {  // oriented sub-boxes (no vertex pass)
        const uint32_t pairs = p.numViews * p.numInstances;
        k_view_proofs<<<(pairs + 255) / 256, 256, 0, st>>>(p.world_view, pairs, p.viewProof);
        uint64_t lb = (p.numItems * ((p.numViews + 3) / 4) + 7) / 8;
        if (lb > (uint64_t)s.numSMs * V1_MINB) lb = (uint64_t)s.numSMs * V1_MINB;
        const unsigned g = (unsigned)lb;
        if (p.coopRaster) {
            if (p.anyPacked) k_stage1_views_boxes<8, V1_MINB, true, true><<<g, 256, 0, st>>>(p);
            else k_stage1_views_boxes<8, V1_MINB, false, true><<<g, 256, 0, st>>>(p);
        } else if (p.anyPacked) {
            k_stage1_views_boxes<8, V1_MINB, true, false><<<g, 256, 0, st>>>(p);
        } else {
            k_stage1_views_boxes<8, V1_MINB, false, false><<<g, 256, 0, st>>>(p);
        }
        return cudaGetLastError() == cudaSuccess ? 0 : -1;
    }
    // the register-capped variants let more blocks share an SM
    const bool capped = (uint64_t)s.stage1Blocks > (uint64_t)s.numSMs * (warps == 4 ? 4u : 2u);
    if (p.anyPacked) {
        if (warps == 4) {
            if (capped) k_stage1_views<4, 6, true><<<b, 128, 0, st>>>(p);
            else k_stage1_views<4, 4, true><<<b, 128, 0, st>>>(p);
        } else {
            if (capped) k_stage1_views<8, 3, true><<<b, 256, 0, st>>>(p);
            else k_stage1_views<8, 2, true><<<b, 256, 0, st>>>(p);
        }
    } else if (warps == 4) {
        if (capped) k_stage1_views<4, 6, false><<<b, 128, 0, st>>>(p);
        else k_stage1_views<4, 4, false><<<b, 128, 0, st>>>(p);
    } else {
        if (capped) k_stage1_views<8, 3, false><<<b, 256, 0, st>>>(p);
        else k_stage1_views<8, 2, false><<<b, 256, 0, st>>>(p);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int cr_launch_stage2_views(const CrFrameParams& p, const CrBatchShape& s, void* stream) {
    if (s.stage2Warps == 4) k_stage2<4, true><<<(unsigned)s.stage2Blocks, 128, 0, (cudaStream_t)stream>>>(p);
    else k_stage2<8, true><<<(unsigned)s.stage2Blocks, 256, 0, (cudaStream_t)stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int cr_launch_stage3_views(const CrFrameParams& p, const CrBatchShape& s, void* stream) {
    k_stage3<8, true><<<(unsigned)s.stage3Blocks, 256, 0, (cudaStream_t)stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
