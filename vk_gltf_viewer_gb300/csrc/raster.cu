// Visibility-buffer rasterisation: the mesh shader
// (shaders/visbuffer/visbuffer.mesh.glsl:30-104), the fixed-function
// rasteriser with the pipeline state of application.cpp:326-340 / 830-841, and
// the fragment shader's ID write (shaders/visbuffer/visbuffer.frag.glsl:36).
//
// One warp owns one surviving meshlet draw: it transforms the <= 64 meshlet
// vertices into shared memory, then each lane sets up one triangle at a time
// (homogeneous backface determinant, outcode reject, near/far and guard-band
// clipping, 28.8 fixed-point snap, top-left edge functions, depth plane).
// Triangles of a few pixels are rasterised by the lane itself or by its warp;
// larger ones go to a queue, as one rectangle or cut into chunk x chunk pixel
// rectangles, that k_raster_big drains with a warp per rectangle.  Every covered sample performs a
// 64-bit max of (depth bits << 32 | id + 1), which is the order-independent
// form of the GREATER_OR_EQUAL depth test with ties won by the later draw.
#include <atomic>

#include "kernels.cuh"

namespace vkgv {

namespace {

constexpr float kGuard = 256.0f;
enum : int { OC_XLO = 1, OC_XHI = 2, OC_YLO = 4, OC_YHI = 8, OC_ZLO = 16, OC_ZHI = 32 };

__device__ __forceinline__ int outcode(const float4& v) {
    int c = 0;
    if (v.x < -v.w) c |= OC_XLO;
    if (v.x > v.w) c |= OC_XHI;
    if (v.y < -v.w) c |= OC_YLO;
    if (v.y > v.w) c |= OC_YHI;
    if (v.z < 0.0f) c |= OC_ZLO;
    if (v.z > v.w) c |= OC_ZHI;
    return c;
}

__device__ __forceinline__ bool outside_guard(const float4& v) {
    float g = fmul(kGuard, v.w);
    return v.x < -g || v.x > g || v.y < -g || v.y > g;
}

// What a warp's raster needs of its current view (in shared memory: fewer
// live registers), and of the launch (one per CTA).
struct RasterCtx {
    unsigned long long* depth;
    uint32_t w, h;
    float hw, hh;
    uint32_t view;
};

struct RasterQueue {
    BigTri* big;
    uint32_t* big_count;
    uint32_t big_cap;
    uint32_t small_area;
    uint32_t chunk, chunk_log2;  // a power of two
    uint32_t* status;
};

// The depth test: a 64-bit max whose result is not needed.  atomicMax on the
// view's pointer (which could point anywhere) compiles to an atomic with a
// reply; the reduction on global memory sends none (1080p torus grid's frame
// 306.8 -> 296.7 us, 4K 696 -> 673 us).
__device__ __forceinline__ void plot(unsigned long long* p, unsigned long long v) {
    asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(v) : "memory");
}

__device__ void raster_rect(const int32_t* X, const int32_t* Y, const int32_t* bias, float z0, float pa, float pb,
                            uint32_t id, int px0, int py0, int px1, int py1, unsigned long long* depth,
                            uint32_t w) {
    const unsigned long long lo = (unsigned long long)id + 1ull;
    const int32_t sx0 = px0 * 256 + 128, sy0 = py0 * 256 + 128;
    int64_t erow[3], stx[3], sty[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int a = k, b = (k + 1) % 3;
        const int32_t dx = X[b] - X[a], dy = Y[b] - Y[a];
        erow[k] = (int64_t)dx * (sy0 - Y[a]) - (int64_t)dy * (sx0 - X[a]);
        stx[k] = -(int64_t)dy * 256;
        sty[k] = (int64_t)dx * 256;
    }
    for (int py = py0; py <= py1; ++py) {
        int64_t e0 = erow[0], e1 = erow[1], e2 = erow[2];
        const int32_t sy = py * 256 + 128;
        const float zrow = __fmaf_rn(pb, __int2float_rn(sy - Y[0]), z0);
        unsigned long long* row = depth + (size_t)py * w;
        for (int px = px0; px <= px1; ++px) {
            if (e0 >= bias[0] && e1 >= bias[1] && e2 >= bias[2]) {
                const int32_t sx = px * 256 + 128;
                float z = __fmaf_rn(pa, __int2float_rn(sx - X[0]), zrow);
                if (!(z > 0.0f)) z = 0.0f;
                if (z > 1.0f) z = 1.0f;
                plot(row + px, ((unsigned long long)__float_as_uint(z) << 32) | lo);
            }
            e0 += stx[0];
            e1 += stx[1];
            e2 += stx[2];
        }
        erow[0] += sty[0];
        erow[1] += sty[1];
        erow[2] += sty[2];
    }
}

// A large triangle of the slow instance, set up and waiting for its binned
// rectangles to be queued: the lanes of a warp collect their jobs while they
// diverge over clipping and setup, then queue all of them with one atomic
// per warp.  (One atomic per triangle on the shared queue counter
// serialised: 23,700 slow triangles in one single-view frame.)
struct BinJob {
    int32_t x[3], y[3];       // oriented snapped vertices, 28.8
    float z0, pa, pb;         // depth plane
    uint32_t id;
    int32_t px0, py0, px1, py1;  // clamped pixel bounding box
    uint32_t n;               // rectangles of Q.chunk x Q.chunk pixels
};
// A clipped triangle fans into at most 10 triangles.
constexpr uint32_t kMaxJobs = 10;
struct JobList {
    BinJob job[kMaxJobs];
    uint32_t count;
};

// The rectangles of one job, queued at Q.big[at, at + n) (past the queue's
// capacity they are drawn in place and the overflow is reported).
__device__ void queue_job(const BinJob& j, uint32_t at, const RasterCtx& c, const RasterQueue& Q) {
    const int32_t cs = (int32_t)Q.chunk;
    const uint32_t ncx = (uint32_t)(j.px1 - j.px0 + cs) >> Q.chunk_log2;
    uint32_t flags = kBigNarrow;
    int32_t bias[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int32_t dx = j.x[(k + 1) % 3] - j.x[k], dy = j.y[(k + 1) % 3] - j.y[k];
        bias[k] = (dy < 0 || (dy == 0 && dx > 0)) ? 0 : 1;
        flags |= (uint32_t)bias[k] << k;
        if (max(abs(dx), abs(dy)) >= 1 << 15) flags &= ~kBigNarrow;
    }
    uint32_t cx = 0;
    int32_t qx0 = j.px0, qy0 = j.py0;
    for (uint32_t i = 0; i < j.n; ++i, ++at, ++cx, qx0 += cs) {
        if (cx == ncx) cx = 0, qx0 = j.px0, qy0 += cs;
        const int32_t qx1 = min(j.px1, qx0 + cs - 1), qy1 = min(j.py1, qy0 + cs - 1);
        if (at < Q.big_cap) {
            BigTri t;
            t.x[0] = j.x[0], t.x[1] = j.x[1], t.x[2] = j.x[2];
            t.y[0] = j.y[0], t.y[1] = j.y[1], t.y[2] = j.y[2];
            t.z0 = j.z0, t.pa = j.pa, t.pb = j.pb;
            t.id = j.id;
            t.px0 = (uint16_t)qx0, t.py0 = (uint16_t)qy0, t.px1 = (uint16_t)qx1, t.py1 = (uint16_t)qy1;
            t.view = c.view;
            t.flags = flags;
            Q.big[at] = t;
        } else {
            report(Q.status, kStatusQueueOverflow, at);
            raster_rect(j.x, j.y, bias, j.z0, j.pa, j.pb, j.id, qx0, qy0, qx1, qy1, c.depth, c.w);
        }
    }
}

// Queues the jobs of every lane (the whole warp, converged): an exclusive
// scan of the lanes' rectangle counts, one atomic on the queue counter.
__device__ void flush_jobs(JobList& jobs, const RasterCtx& c, const RasterQueue& Q, int lane) {
    uint32_t mine = 0;
    for (uint32_t i = 0; i < jobs.count; ++i) mine += jobs.job[i].n;
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (total == 0) {
        jobs.count = 0;
        return;
    }
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(Q.big_count, total);
    base = __shfl_sync(0xffffffffu, base, 0) + (incl - mine);
    for (uint32_t i = 0; i < jobs.count; ++i) {
        queue_job(jobs.job[i], base, c, Q);
        base += jobs.job[i].n;
    }
    jobs.count = 0;
}

// Triangle setup on snapped vertices and dispatch to inline or binned
// raster; a triangle to bin becomes a job in `jobs` (queued directly when
// the list is full).
__device__ __noinline__ void setup_and_raster(int32_t X0, int32_t Y0, float Z0, int32_t X1, int32_t Y1, float Z1, int32_t X2,
                                 int32_t Y2, float Z2, uint32_t id, const RasterCtx& c, const RasterQueue& Q, JobList& jobs) {
    int64_t A = (int64_t)(X1 - X0) * (Y2 - Y0) - (int64_t)(Y1 - Y0) * (X2 - X0);
    if (A == 0) return;
    if (A < 0) {
        int32_t tx = X1, ty = Y1;
        float tz = Z1;
        X1 = X2, Y1 = Y2, Z1 = Z2;
        X2 = tx, Y2 = ty, Z2 = tz;
        A = -A;
    }
    const int32_t minx = min(X0, min(X1, X2)), maxx = max(X0, max(X1, X2));
    const int32_t miny = min(Y0, min(Y1, Y2)), maxy = max(Y0, max(Y1, Y2));
    // ceil((min - 128) / 256) and floor((max - 128) / 256); >> is floor division.
    int64_t px0 = ((int64_t)minx - 128 + 255) >> 8, px1 = ((int64_t)maxx - 128) >> 8;
    int64_t py0 = ((int64_t)miny - 128 + 255) >> 8, py1 = ((int64_t)maxy - 128) >> 8;
    px0 = px0 < 0 ? 0 : px0;
    py0 = py0 < 0 ? 0 : py0;
    px1 = px1 > (int64_t)c.w - 1 ? (int64_t)c.w - 1 : px1;
    py1 = py1 > (int64_t)c.h - 1 ? (int64_t)c.h - 1 : py1;
    if (px0 > px1 || py0 > py1) return;
    int32_t X[3] = {X0, X1, X2}, Y[3] = {Y0, Y1, Y2};
    int32_t bias[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int a = k, b = (k + 1) % 3;
        const int32_t dx = X[b] - X[a], dy = Y[b] - Y[a];
        bias[k] = (dy < 0 || (dy == 0 && dx > 0)) ? 0 : 1;
    }
    const float dx1 = __int2float_rn(X1 - X0), dy1 = __int2float_rn(Y1 - Y0);
    const float dx2 = __int2float_rn(X2 - X0), dy2 = __int2float_rn(Y2 - Y0);
    const float af = __ll2float_rn(A);
    const float dz1 = fsub(Z1, Z0), dz2 = fsub(Z2, Z0);
    const float ra = __frcp_rn(af);
    const float pa = fmul(fsub(fmul(dz1, dy2), fmul(dz2, dy1)), ra);
    const float pb = fmul(fsub(fmul(dz2, dx1), fmul(dz1, dx2)), ra);
    const int64_t bw = px1 - px0 + 1, bh = py1 - py0 + 1;
    if (bw * bh <= (int64_t)Q.small_area) {
        raster_rect(X, Y, bias, Z0, pa, pb, id, (int)px0, (int)py0, (int)px1, (int)py1, c.depth, c.w);
        return;
    }
    const uint32_t ncx = (uint32_t)(bw + Q.chunk - 1) >> Q.chunk_log2, ncy = (uint32_t)(bh + Q.chunk - 1) >> Q.chunk_log2;
    BinJob j;
    j.x[0] = X0, j.x[1] = X1, j.x[2] = X2;
    j.y[0] = Y0, j.y[1] = Y1, j.y[2] = Y2;
    j.z0 = Z0, j.pa = pa, j.pb = pb;
    j.id = id;
    j.px0 = (int32_t)px0, j.py0 = (int32_t)py0, j.px1 = (int32_t)px1, j.py1 = (int32_t)py1;
    j.n = ncx * ncy;
    if (jobs.count < kMaxJobs) {
        jobs.job[jobs.count++] = j;
    } else {
        queue_job(j, atomicAdd(Q.big_count, j.n), c, Q);
    }
}

// The 28.8 snap of a vertex with w > 0: one correctly rounded reciprocal of w
// and three products.  False when it leaves the snapped range.
__device__ __forceinline__ bool snap_inside(const float4& v, const RasterCtx& c, int32_t& X, int32_t& Y, float& Z) {
    const float rw = __frcp_rn(v.w);
    const float xd = fmul(v.x, rw), yd = fmul(v.y, rw);
    const float xf = fadd(fmul(xd, c.hw), c.hw), yf = fadd(fmul(yd, c.hh), c.hh);
    const float sx = fmul(xf, 256.0f), sy = fmul(yf, 256.0f);
    X = __float2int_rn(sx);
    Y = __float2int_rn(sy);
    Z = fmul(v.z, rw);
    return fabsf(sx) < 1073741824.0f && fabsf(sy) < 1073741824.0f;
}

__device__ __forceinline__ bool snap(const float4& v, const RasterCtx& c, int32_t& X, int32_t& Y, float& Z) {
    int32_t x, y;
    float z;
    if (!(v.w > 0.0f) || !snap_inside(v, c, x, y, z)) return false;
    X = x, Y = y, Z = z;
    return true;
}

__device__ __forceinline__ float plane_dist(const float4& v, int plane) {
    switch (plane) {
        case 0: return fsub(v.w, v.z);
        case 1: return v.z;
        case 2: return fsub(fmul(kGuard, v.w), v.x);
        case 3: return fadd(v.x, fmul(kGuard, v.w));
        case 4: return fsub(fmul(kGuard, v.w), v.y);
        default: return fadd(v.y, fmul(kGuard, v.w));
    }
}

__device__ int clip_poly(const float4* in, int n, float4* out, int plane) {
    int m = 0;
    for (int i = 0; i < n; ++i) {
        const float4 a = in[i];
        const float4 b = in[(i + 1) % n];
        const float da = plane_dist(a, plane), db = plane_dist(b, plane);
        const bool ia = da >= 0.0f, ib = db >= 0.0f;
        if (ia) out[m++] = a;
        if (ia != ib) {
            const float t = fdiv(da, fsub(da, db));
            out[m++] = make_float4(fadd(a.x, fmul(t, fsub(b.x, a.x))), fadd(a.y, fmul(t, fsub(b.y, a.y))),
                                   fadd(a.z, fmul(t, fsub(b.z, a.z))), fadd(a.w, fmul(t, fsub(b.w, a.w))));
        }
    }
    return m;
}

// Slow path: homogeneous clipping (near/far, then guard band) and a fan.
__device__ __noinline__ void raster_clipped(float4 v0, float4 v1, float4 v2, bool clipz, uint32_t id,
                                            const RasterCtx& c, const RasterQueue& Q, JobList& jobs) {
    float4 bufa[12], bufb[12];
    bufa[0] = v0, bufa[1] = v1, bufa[2] = v2;
    float4* cur = bufa;
    float4* nxt = bufb;
    int n = 3;
    if (clipz) {
        for (int plane = 0; plane < 2 && n >= 3; ++plane) {
            n = clip_poly(cur, n, nxt, plane);
            float4* t = cur;
            cur = nxt;
            nxt = t;
        }
    }
    bool guard = false;
    for (int k = 0; k < n; ++k) guard |= outside_guard(cur[k]);
    if (guard) {
        for (int plane = 2; plane < 6 && n >= 3; ++plane) {
            n = clip_poly(cur, n, nxt, plane);
            float4* t = cur;
            cur = nxt;
            nxt = t;
        }
    }
    if (n < 3) return;
    int32_t X[12], Y[12];
    float Z[12];
    for (int k = 0; k < n; ++k)
        if (!snap(cur[k], c, X[k], Y[k], Z[k])) return;
    for (int k = 1; k + 1 < n; ++k)
        setup_and_raster(X[0], Y[0], Z[0], X[k], Y[k], Z[k], X[k + 1], Y[k + 1], Z[k + 1], id, c, Q, jobs);
}

// Items a warp takes at once, at most (256-view torus grid 32.1 ms; 16: 32.4;
// 8: 33.1).
constexpr uint32_t kMaxRun = 32;

// Views per raster launch (the launcher splits larger batches).
constexpr uint32_t kRasterMaxViews = 1024;

// What the per-meshlet header chain resolves for one work item.
struct ItemHeader {
    const uint32_t* vidx;       // the meshlet's vertex indices
    const uint8_t* tri;         // its triangle-index bytes
    const vkgv_vertex* verts;   // the primitive's vertex stream
    uint32_t d;                 // meshlet draw index
    uint32_t v;                 // view (in this launch)
    uint32_t transform;         // node transform index
    uint8_t vc;                 // vertex count
    uint8_t t0, t1;             // the triangles to draw (none: an index out of range, or no work)
    uint8_t flags;              // kDoubleSided, kSplit
};
constexpr uint8_t kDoubleSided = 1, kSplit = 2;
constexpr uint32_t kParts = 4;   // 32-triangle rounds of a meshlet
static_assert(VKGV_MAX_PRIMITIVES <= 32 * kParts, "a meshlet has at most kParts rounds");
// A deferred meshlet's list entry: the draw index, and for a split item its
// round and the split flag above it.
constexpr uint32_t kDeferSplit = 1u << 31;
constexpr uint32_t kDeferPartShift = VKGV_DRAW_INDEX_BITS;
constexpr uint32_t kDrawMask = (1u << VKGV_DRAW_INDEX_BITS) - 1u;

struct RasterParams {
    SceneArgs S;
    const DeviceView* views;  // this launch's views
    uint32_t nviews;          // <= kRasterMaxViews
    uint32_t view_base;       // index of views[0] in the frame's view table
    RasterLists lists;
    BigTri* big;
    uint32_t* big_count;
    uint32_t big_cap;
    uint32_t small_area;
    uint32_t chunk;
    uint32_t split;           // meshlets at the end of the work list drawn by kParts warps each
    uint32_t deferred_cap;    // entries a view's deferred list holds
    uint32_t* status;
    uint32_t* work;           // items taken beyond the warps' first runs: [0] fast, [1] slow instance
};

// The meshlet list a raster instance draws for one view: pass-1 or pass-2
// survivors, the view's deferred meshlets (slow instance), or an explicit
// list; items are list[first, first + count).
template <bool SLOW>
__device__ __forceinline__ void view_work(const RasterParams& P, const DeviceView& V, const uint32_t*& list,
                                          uint32_t& count, uint32_t& first) {
    first = 0;
    if (SLOW) {
        list = V.deferred;
        count = min(V.counters[P.lists.deferred_slot], P.deferred_cap);
    } else if (P.lists.pass == 1) {
        list = V.survivors;
        count = min(V.counters[0], V.survivor_capacity);
    } else if (P.lists.pass == 2) {
        const uint32_t c0 = min(V.counters[0], V.survivor_capacity);
        list = V.survivors + c0;
        count = min(V.counters[2], V.survivor_capacity - c0);
    } else {
        list = P.lists.list;
        const uint32_t n = *P.lists.count;
        first = P.lists.first;
        count = n > first ? n - first : 0u;
    }
}

// Setup record of one small triangle, shared by the warp while it
// rasterises all small triangles of a round cooperatively: 32 bytes, two
// 16-byte words.  Vertices are relative to the corner of the clamped bbox
// (a small triangle's extent keeps them inside int16).
struct __align__(16) TriRec {
    uint32_t v[3];        // oriented (positive area) snapped vertices, 28.8: x | y << 16
    uint32_t bits;        // triangle (7) | edge biases (3) | bbox width (7) | ceil(4096 / width) (13)
    float z0, pa, pb;     // depth plane
    uint32_t origin;      // clamped bbox origin in pixels: x | y << 16
};

constexpr uint8_t kFlagGuard = 1u << 6;
constexpr uint8_t kFlagSnapped = 1u << 7;
// Triangles whose unclamped bbox is below this many 28.8 units on both axes
// keep every edge-function value of their bbox inside int32.
constexpr int32_t kSmallExtent = 1 << 14;

enum TriKind : int { kDrop = 0, kFast = 1, kSlowClip = 2, kSlowSetup = 3 };

#ifndef VKGV_RASTER_WARPS_PER_SM
#define VKGV_RASTER_WARPS_PER_SM 28
#endif

// Meshlets at the end of a launch's work list that are split (see k_raster),
// per SM.  A quarter of the resident warps: 443 meshlets of a 1280x720 view
// 44 -> 20 us (they had one warp each on a chip of 4,256); the 1080p torus grid's
// frame 342 -> 326 us (the last heavy meshlets, up to 30 us each, and pass 2's
// few hundred).  None: 344 us; 14: 327; 28: 329; 56: 341 (every split meshlet
// transforms its vertices four times).
#ifndef VKGV_RASTER_SPLIT_PER_SM
#define VKGV_RASTER_SPLIT_PER_SM 7
#endif

// Small triangles whose clamped bbox has at most this many pixels are
// rasterised by their own lane; larger small ones by the whole warp.
#ifndef VKGV_RASTER_LANE_AREA
#define VKGV_RASTER_LANE_AREA 4
#endif
constexpr uint32_t kLaneArea = VKGV_RASTER_LANE_AREA;
// Small triangles above this bbox area are queued for k_raster_big.
#ifndef VKGV_RASTER_QUEUE_AREA
#define VKGV_RASTER_QUEUE_AREA 16
#endif
constexpr uint32_t kQueueArea = VKGV_RASTER_QUEUE_AREA;

// Whether the fast instance draws a triangle whose clamped bbox is bw x bh
// pixels (and whose extent is below kSmallExtent): itself, or as one rectangle
// of the queue.  The slow instance queues what takes several: with the line at
// small_area it transformed every meshlet of 8-to-32-pixel triangles again
// (a 256^2 sphere's frame 34.9 -> 30.8 us, the 1365x767 torus grid 206.9 ->
// 197.0, 1080p 259.0 -> 253.8, 64 views of 512^2 568.6 -> 561.0).
__device__ __forceinline__ bool fast_size(uint32_t bw, uint32_t bh, const RasterQueue& Q) {
    return bw * bh <= Q.small_area || max(bw, bh) <= Q.chunk;
}

struct TriClass {
    int2 q0, q1, q2;  // snapped vertices
    int2 f0, f1, f2;  // {depth bits, flags}
};

// Sorts one meshlet triangle into drop / fast / slow-clip / slow-setup.  The
// backface test (visbuffer.mesh.glsl:86-101) and the empty-bbox test are
// both pure filters, so the cheap bbox test runs first for triangles that
// need no clipping.  kFast: snapped, inside the guard band, front-facing,
// non-zero area, a pixel centre in its bbox, bbox of a fast_size and edge
// values within int32.
__device__ __forceinline__ int classify(uint32_t i0, uint32_t i1, uint32_t i2, uint32_t vc, const int2* sxy,
                                        const int2* szf, const float4* clip, bool double_sided, float tdet, const RasterCtx& c,
                                        const RasterQueue& Q, TriClass& k) {
    if (i0 >= vc || i1 >= vc || i2 >= vc) return kDrop;  // reported by the fast instance
    k.q0 = sxy[i0], k.f0 = szf[i0];
    k.q1 = sxy[i1], k.f1 = szf[i1];
    k.q2 = sxy[i2], k.f2 = szf[i2];
    const uint32_t f0 = (uint32_t)k.f0.y, f1 = (uint32_t)k.f1.y, f2 = (uint32_t)k.f2.y;
    auto backfacing = [&]() {
        if (double_sided) return false;
        const float4 a = clip[i0], b = clip[i1], cc = clip[i2];
        const float det = det3(a.x, a.y, a.w, b.x, b.y, b.w, cc.x, cc.y, cc.w);
        return tdet < 0.0f ? det < 0.0f : det > 0.0f;
    };
    if (f0 & f1 & f2 & 63) return kDrop;  // outcode reject
    if ((f0 | f1 | f2) & (OC_ZLO | OC_ZHI | kFlagGuard)) return backfacing() ? kDrop : kSlowClip;
    if (!(f0 & f1 & f2 & kFlagSnapped)) return kDrop;
    const int2 &q0 = k.q0, &q1 = k.q1, &q2 = k.q2;
    const int32_t minx = min(q0.x, min(q1.x, q2.x)), maxx = max(q0.x, max(q1.x, q2.x));
    const int32_t miny = min(q0.y, min(q1.y, q2.y)), maxy = max(q0.y, max(q1.y, q2.y));
    const int32_t qx0 = max((minx - 128 + 255) >> 8, 0), qx1 = min((maxx - 128) >> 8, (int32_t)c.w - 1);
    const int32_t qy0 = max((miny - 128 + 255) >> 8, 0), qy1 = min((maxy - 128) >> 8, (int32_t)c.h - 1);
    if (qx0 > qx1 || qy0 > qy1 || backfacing()) return kDrop;
    const int64_t A = (int64_t)(q1.x - q0.x) * (q2.y - q0.y) - (int64_t)(q1.y - q0.y) * (q2.x - q0.x);
    if (A == 0) return kDrop;
    const bool small = maxx - minx < kSmallExtent && maxy - miny < kSmallExtent &&
                       fast_size((uint32_t)(qx1 - qx0 + 1), (uint32_t)(qy1 - qy0 + 1), Q);
    return small ? kFast : kSlowSetup;
}

// First stage of the fast instance, on every triangle: 0 = dropped (an
// index out of range, outcode reject, unsnapped vertex, or no pixel centre
// in its clamped bounding box), 2 = needs the slow instance (a vertex
// outside the near/far planes or the guard band), 1 = a candidate for the
// compacted second stage (raster_small), which applies the backface test
// (visbuffer.mesh.glsl:86-101), the zero-area test and the size limits.
// The tests only filter, so their order does not change what is drawn; the
// cheap ones run here on every triangle, the others only on the candidates.
__device__ __forceinline__ int prefilter(uint32_t i0, uint32_t i1, uint32_t i2, const int2* sxy, const int2* szf,
                                         const RasterCtx& c) {
    const uint32_t f0 = (uint32_t)szf[i0].y, f1 = (uint32_t)szf[i1].y, f2 = (uint32_t)szf[i2].y;
    if (f0 & f1 & f2 & 63) return 0;  // outcode reject
    if ((f0 | f1 | f2) & (OC_ZLO | OC_ZHI | kFlagGuard)) return 2;
    if (!(f0 & f1 & f2 & kFlagSnapped)) return 0;
    const int2 q0 = sxy[i0], q1 = sxy[i1], q2 = sxy[i2];
    const int32_t minx = min(q0.x, min(q1.x, q2.x)), maxx = max(q0.x, max(q1.x, q2.x));
    const int32_t miny = min(q0.y, min(q1.y, q2.y)), maxy = max(q0.y, max(q1.y, q2.y));
    const int32_t qx0 = max((minx - 128 + 255) >> 8, 0), qx1 = min((maxx - 128) >> 8, (int32_t)c.w - 1);
    const int32_t qy0 = max((miny - 128 + 255) >> 8, 0), qy1 = min((maxy - 128) >> 8, (int32_t)c.h - 1);
    return (qx0 > qx1 || qy0 > qy1) ? 0 : 1;
}

// The same for a meshlet whose vertices all lie inside the view volume: no
// flag is set and the view clamps nothing (the snapped coordinates are in
// [0, 256 w] x [0, 256 h]), which leaves the empty-box test.  With u = x - 128
// the pixel centres are the multiples of 256, and [min u, max u] holds none
// exactly when min u - 1 and max u share their quotient by 256.
__device__ __forceinline__ bool covers_centre(int2 q0, int2 q1, int2 q2) {
    const uint32_t x = (uint32_t)(min(q0.x, min(q1.x, q2.x)) - 129) ^ (uint32_t)(max(q0.x, max(q1.x, q2.x)) - 128);
    const uint32_t y = (uint32_t)(min(q0.y, min(q1.y, q2.y)) - 129) ^ (uint32_t)(max(q0.y, max(q1.y, q2.y)) - 128);
    return x > 255u && y > 255u;
}

// A small triangle's edge functions and depth plane at a sample, relative to
// its bbox corner: int32 values (the extent bound of a small triangle keeps
// them exact) with the top-left biases subtracted, so that the sample is
// covered when no sign bit is set.
struct SmallEdges {
    int32_t e0, e1, e2;     // at the current sample
    int32_t ax, ay, bx, by, cx, cy;  // edge vectors
    float fx, fy;           // sample - vertex 0
};

__device__ __forceinline__ void edges_at(SmallEdges& s, int32_t x0, int32_t y0, int32_t x1, int32_t y1, int32_t x2,
                                         int32_t y2, uint32_t bias, int32_t sx, int32_t sy) {
    s.ax = x1 - x0, s.ay = y1 - y0, s.bx = x2 - x1, s.by = y2 - y1, s.cx = x0 - x2, s.cy = y0 - y2;
    s.e0 = s.ax * (sy - y0) - s.ay * (sx - x0) - (int32_t)(bias & 1u);
    s.e1 = s.bx * (sy - y1) - s.by * (sx - x1) - (int32_t)((bias >> 1) & 1u);
    s.e2 = s.cx * (sy - y2) - s.cy * (sx - x2) - (int32_t)((bias >> 2) & 1u);
    s.fx = __int2float_rn(sx - x0), s.fy = __int2float_rn(sy - y0);
}

// Depth of a covered sample, clamped to [0, 1] (NaN and -0 to +0), over id + 1.
__device__ __forceinline__ unsigned long long fragment(float pa, float pb, float z0, float fx, float fy, uint32_t id) {
    const float z = __saturatef(__fmaf_rn(pa, fx, __fmaf_rn(pb, fy, z0)));
    return ((unsigned long long)__float_as_uint(z) << 32) | (unsigned long long)(id + 1u);
}

// The sample of pixel (lx, ly) of a record's bbox.
__device__ __forceinline__ void draw_sample(const TriRec& r, uint32_t lx, uint32_t ly, uint32_t d, const RasterCtx& c) {
    SmallEdges e;
    edges_at(e, (int32_t)(int16_t)(r.v[0] & 0xFFFFu), (int32_t)r.v[0] >> 16, (int32_t)(int16_t)(r.v[1] & 0xFFFFu),
             (int32_t)r.v[1] >> 16, (int32_t)(int16_t)(r.v[2] & 0xFFFFu), (int32_t)r.v[2] >> 16, (r.bits >> 7) & 7u,
             (int32_t)(lx << 8) + 128, (int32_t)(ly << 8) + 128);
    if ((e.e0 | e.e1 | e.e2) >= 0)
        plot(c.depth + (size_t)((r.origin >> 16) + ly) * c.w + (r.origin & 0xFFFFu) + lx,
             fragment(r.pa, r.pb, r.z0, e.fx, e.fy, (d << 7) | (r.bits & 127u)));
}

// Second stage of the fast instance: up to 32 compacted candidates, one
// per lane (ct = meshlet-local triangle index, 0xffffffff = none).  A
// candidate that is back-facing or of zero area is dropped; one that is not of
// a fast_size or whose extent leaves int32 edge values needs
// the slow instance (the return value); the rest are set up and
// rasterised.  A triangle whose
// clamped bbox has at most kLaneArea pixels is rasterised by its own lane;
// the larger ones are spread over the warp by a scan of their bbox areas.
// xyw holds each vertex's clip x, y, w and snapped depth.
__device__ __forceinline__ bool raster_small(uint32_t ct, const uint8_t* sidx8, const int2* sxy, const float4* xyw,
                                             bool double_sided, float tdet, uint32_t d, const RasterCtx& c, const RasterQueue& Q,
                                             TriRec* recs, uint16_t* starts, int lane) {
    uint32_t coop_area = 0;
    bool slow = false;
    TriRec rec;
    if (ct != 0xffffffffu) {
        const uint32_t i0 = sidx8[3 * ct], i1 = sidx8[3 * ct + 1], i2 = sidx8[3 * ct + 2];
        const int2 q0 = sxy[i0], q1 = sxy[i1], q2 = sxy[i2];
        const float4 k0 = xyw[i0], k1 = xyw[i1], k2 = xyw[i2];
        bool back = false;
        if (!double_sided) {
            const float det = det3(k0.x, k0.y, k0.z, k1.x, k1.y, k1.z, k2.x, k2.y, k2.z);
            back = tdet < 0.0f ? det < 0.0f : det > 0.0f;
        }
        const int32_t minx = min(q0.x, min(q1.x, q2.x)), maxx = max(q0.x, max(q1.x, q2.x));
        const int32_t miny = min(q0.y, min(q1.y, q2.y)), maxy = max(q0.y, max(q1.y, q2.y));
        const bool fits = maxx - minx < kSmallExtent && maxy - miny < kSmallExtent;
        // edge values of a triangle of that extent stay inside int32 (the
        // area of a larger one wraps and is not used)
        const int32_t A = (int32_t)((uint32_t)(q1.x - q0.x) * (uint32_t)(q2.y - q0.y) -
                                    (uint32_t)(q1.y - q0.y) * (uint32_t)(q2.x - q0.x));
        const int32_t px0 = max((minx - 128 + 255) >> 8, 0), px1 = min((maxx - 128) >> 8, (int32_t)c.w - 1);
        const int32_t py0 = max((miny - 128 + 255) >> 8, 0), py1 = min((maxy - 128) >> 8, (int32_t)c.h - 1);
        const uint32_t bw = (uint32_t)(px1 - px0 + 1), bh = (uint32_t)(py1 - py0 + 1);
        const bool live = !back && fits && A != 0 && fast_size(bw, bh, Q);
        if (!back && !live) {
            const int64_t A64 = (int64_t)(q1.x - q0.x) * (q2.y - q0.y) - (int64_t)(q1.y - q0.y) * (q2.x - q0.x);
            slow = A64 != 0;
        }
        if (live) {
            const bool flip = A < 0;  // orient to positive area
            const int32_t ox = px0 << 8, oy = py0 << 8;
            const int32_t x0 = q0.x - ox, y0 = q0.y - oy;
            const int32_t x1 = (flip ? q2.x : q1.x) - ox, y1 = (flip ? q2.y : q1.y) - oy;
            const int32_t x2 = (flip ? q1.x : q2.x) - ox, y2 = (flip ? q1.y : q2.y) - oy;
            const float z0 = k0.w, z1 = flip ? k2.w : k1.w, z2 = flip ? k1.w : k2.w;
            const int32_t ax = x1 - x0, ay = y1 - y0, bx = x2 - x1, by = y2 - y1, cx = x0 - x2, cy = y0 - y2;
            // an edge that is not top-left excludes its samples
            const uint32_t bias = ((ay < 0 || (ay == 0 && ax > 0)) ? 0u : 1u) | ((by < 0 || (by == 0 && bx > 0)) ? 0u : 2u) |
                                  ((cy < 0 || (cy == 0 && cx > 0)) ? 0u : 4u);
            const float dx1 = __int2float_rn(ax), dy1 = __int2float_rn(ay);
            const float dx2 = __int2float_rn(-cx), dy2 = __int2float_rn(-cy);
            const float dz1 = fsub(z1, z0), dz2 = fsub(z2, z0);
            const float ra = __frcp_rn(__int2float_rn(flip ? -A : A));
            const float pa = fmul(fsub(fmul(dz1, dy2), fmul(dz2, dy1)), ra);
            const float pb = fmul(fsub(fmul(dz2, dx1), fmul(dz1, dx2)), ra);
            if (bw * bh <= kLaneArea) {
                SmallEdges e;
                edges_at(e, x0, y0, x1, y1, x2, y2, bias, 128, 128);
                const uint32_t id = (d << 7) | ct;
                unsigned long long* row = c.depth + (size_t)(uint32_t)py0 * c.w + (uint32_t)px0;
                for (uint32_t ly = bh;;) {
                    int32_t r0 = e.e0, r1 = e.e1, r2 = e.e2;
                    float fx = e.fx;
                    unsigned long long* p = row;
                    for (uint32_t lx = bw;;) {
                        if ((r0 | r1 | r2) >= 0) plot(p, fragment(pa, pb, z0, fx, e.fy, id));
                        if (--lx == 0) break;
                        r0 -= e.ay << 8, r1 -= e.by << 8, r2 -= e.cy << 8;
                        fx = fadd(fx, 256.0f);  // whole numbers below 2^24: exact
                        ++p;
                    }
                    if (--ly == 0) break;
                    e.e0 += e.ax << 8, e.e1 += e.bx << 8, e.e2 += e.cx << 8;
                    e.fy = fadd(e.fy, 256.0f);
                    row += c.w;
                }
            } else {
                rec.v[0] = ((uint32_t)x0 & 0xFFFFu) | ((uint32_t)y0 << 16);
                rec.v[1] = ((uint32_t)x1 & 0xFFFFu) | ((uint32_t)y1 << 16);
                rec.v[2] = ((uint32_t)x2 & 0xFFFFu) | ((uint32_t)y2 << 16);
                // ceil(4096 / bw): 4096 times the correctly rounded 1 / bw
                // rounded up (whole only for the powers of two, exact there)
                const uint32_t inv = __float2uint_ru(fmul(4096.0f, __frcp_rn((float)bw)));
                rec.bits = ct | (bias << 7) | (bw << 10) | (inv << 17);
                rec.z0 = z0, rec.pa = pa, rec.pb = pb;
                rec.origin = (uint32_t)px0 | ((uint32_t)py0 << 16);
                coop_area = bw * bh;
            }
        }
    }
    unsigned coop = __ballot_sync(0xffffffffu, coop_area != 0);
    if (coop == 0) return slow;
    // Triangles whose bbox exceeds kQueueArea pixels go to the
    // binned-rectangle queue (one rectangle each), drained by k_raster_big
    // with a warp per rectangle: a meshlet of larger triangles then no
    // longer holds one warp for all of its pixels.  The rest, and anything
    // the full queue refuses, take the warp-cooperative raster below.
    const unsigned mm = __ballot_sync(0xffffffffu, coop_area > kQueueArea);
    if (mm) {
        const int leader = __ffs(mm) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(Q.big_count, (uint32_t)__popc(mm));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (coop_area > kQueueArea) {
            const uint32_t slot = base + (uint32_t)__popc(mm & ((1u << lane) - 1u));
            if (slot < Q.big_cap) {
                const uint32_t px0 = rec.origin & 0xFFFFu, py0 = rec.origin >> 16, bw = (rec.bits >> 10) & 127u;
                BigTri t;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    t.x[k] = (int32_t)(int16_t)(rec.v[k] & 0xFFFFu) + (int32_t)(px0 << 8);
                    t.y[k] = ((int32_t)rec.v[k] >> 16) + (int32_t)(py0 << 8);
                }
                t.z0 = rec.z0, t.pa = rec.pa, t.pb = rec.pb;
                t.id = (d << 7) | (rec.bits & 127u);
                t.px0 = (uint16_t)px0, t.py0 = (uint16_t)py0;
                t.px1 = (uint16_t)(px0 + bw - 1u), t.py1 = (uint16_t)(py0 + coop_area / bw - 1u);
                t.view = c.view;
                t.flags = ((rec.bits >> 7) & 7u) | kBigNarrow;
                Q.big[slot] = t;
                coop_area = 0;
            } else {
                report(Q.status, kStatusQueueOverflow, slot);
            }
        }
        // what a full queue refused above small_area, one after another
        unsigned refused = __ballot_sync(0xffffffffu, coop_area > Q.small_area);
        for (; refused; refused &= refused - 1u) {
            const int from = __ffs(refused) - 1;
            if (lane == from) recs[0] = rec;
            const uint32_t area = __shfl_sync(0xffffffffu, coop_area, from);
            if (lane == from) coop_area = 0;
            __syncwarp();
            const TriRec r = recs[0];
            const uint32_t bw = (r.bits >> 10) & 127u;
            for (uint32_t p = lane; p < area; p += 32) draw_sample(r, p % bw, p / bw, d, c);
            __syncwarp();
        }
        coop = __ballot_sync(0xffffffffu, coop_area != 0);
        if (coop == 0) return slow;
    }
    // Warp-cooperative raster: the records compacted in lane order and a scan
    // of their bbox areas spread the pixels evenly over the lanes.  A lane
    // finds its pixel's record by counting the records that start at or before
    // it: those before this step's 32 pixels by a ballot, the others in a mask
    // of the start positions.
    uint32_t incl = coop_area;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t start = coop_area ? incl - coop_area : 0xffffffffu;
    if (coop_area) {
        const uint32_t at = (uint32_t)__popc(coop & ((1u << lane) - 1u));
        recs[at] = rec;
        starts[at] = (uint16_t)start;  // below 32 * 64
    }
    __syncwarp();
    for (uint32_t p0 = 0; p0 < total; p0 += 32) {
        const uint32_t before = (uint32_t)__popc(__ballot_sync(0xffffffffu, start < p0));
        const uint32_t mine = start - p0 < 32u ? 1u << (start - p0) : 0u;
        const uint32_t begins = __reduce_or_sync(0xffffffffu, mine);
        const uint32_t p = p0 + (uint32_t)lane;
        if (p < total) {
            const uint32_t j = before + (uint32_t)__popc(begins & (0xffffffffu >> (31 - lane))) - 1u;
            const TriRec r = recs[j];
            const uint32_t local = p - starts[j], bw = (r.bits >> 10) & 127u;
            const uint32_t ly = (local * (r.bits >> 17)) >> 12, lx = local - ly * bw;
            draw_sample(r, lx, ly, d, c);
        }
    }
    __syncwarp();
    return slow;
}

// A warp's shared memory, in one piece: one base register addresses all of it
// (with an array of each member per CTA the fast instance spilled 34 bytes of
// its 72 registers, with this 30, in colder places: 256 views of the torus grid
// 30.43 -> 29.39 ms, of 128^2 1,380 -> 1,328 us, the 4K frame 515.2 -> 506.3, 1080p
// 252.4 -> 248.6).
struct __align__(16) WarpShared {
    // per vertex: clip {x, y, z, w} (slow instance) or clip {x, y, w} and the
    // snapped depth (fast instance); the snapped {X, Y} (28.8)
    float4 clip[64];
    TriRec tri[32];
    int2 xy[64];
    uint32_t idx[96];           // the meshlet's triangle-index bytes (<= 126 triangles)
    float mvp[16];
    // Per-meshlet headers of the current run, resolved one item per lane so
    // that the dependent loads (list entry -> draw -> primitive -> meshlet
    // record, material) of up to kMaxRun meshlets are in flight together instead
    // of one meshlet after another.
    ItemHeader hdr[kMaxRun];
    RasterCtx ctx;
    float tdet;
    uint16_t start[32];
    uint8_t ring[128];          // the compacted candidate triangle indices (fast instance)
};

// Warp-per-meshlet raster.  The fast instance (SLOW = false) handles every
// triangle that needs no clipping and is of a fast_size, and appends a meshlet that has any other triangle to the view's
// deferred list.  The slow instance (SLOW = true) re-runs those meshlets and
// handles only the remaining triangles (homogeneous clipping, large or
// off-screen-spanning triangles), so the fast instance calls no function.
template <int WARPS, bool SLOW>
__global__ void __launch_bounds__(WARPS * 32, (SLOW ? 16 : VKGV_RASTER_WARPS_PER_SM) / WARPS) k_raster(RasterParams P) {
    pdl_begin();
    __shared__ WarpShared s_warp[WARPS];
    // exclusive prefix of the views' work counts: view v owns the global
    // work items [s_pre[v], s_pre[v + 1])
    // (sized by the launch: 18 KB a CTA leave seven of them in 132 KB and the
    // rest to the L1: the 1080p torus grid's frame 308.0 -> 305.6 us from 25 to
    // 20 KB, 276.3 -> 274.3 us to 18)
    extern __shared__ uint32_t s_pre[];  // nviews + 1
    // The other instance's counter starts its next launch at zero: it is not
    // running, and no CTA has to end with a barrier and an atomic for it (1080p
    // torus grid 263.5 -> 259.0 us a frame, 720p sphere 31.8 -> 31.1).
    if (blockIdx.x == 0 && threadIdx.x == 0) P.work[SLOW ? 0 : 1] = 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nv = P.nviews;
    for (uint32_t v = threadIdx.x; v < nv; v += blockDim.x) {
        const uint32_t* l;
        uint32_t n, f;
        view_work<SLOW>(P, P.views[v], l, n, f);
        s_pre[v + 1] = n;
    }
    __shared__ RasterQueue Q;
    if (threadIdx.x == 0) {
        s_pre[0] = 0;
        Q.big = P.big;
        Q.big_count = P.big_count;
        Q.big_cap = P.big_cap;
        Q.small_area = P.small_area;
        Q.chunk = P.chunk;
        Q.chunk_log2 = 31u - (uint32_t)__clz((int)P.chunk);
        Q.status = P.status;
    }
    __syncthreads();
    if (nv > 1 && warp == 0) {  // (one view: 720p sphere 30.9 -> 29.7 us without)
        // inclusive scan of s_pre[1..nv]: lane-contiguous segments, then a
        // warp scan of the segment sums
        const uint32_t seg = (nv + 31) / 32, b = 1 + lane * seg, e = min(b + seg, nv + 1);
        uint32_t sum = 0;
        for (uint32_t i = b; i < e; ++i) sum += s_pre[i];
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        uint32_t run = incl - sum;
        for (uint32_t i = b; i < e; ++i) {
            run += s_pre[i];
            s_pre[i] = run;
        }
    }
    if (nv > 1) __syncthreads();
    // The last `split` meshlets of the list are drawn by kParts warps each, one
    // 32-triangle round a warp: a launch of few meshlets then fills the chip
    // (and the longest of them takes one round, not four), and at the end of
    // a long one the last warps are not left alone with whole heavy meshlets.
    const uint32_t total = s_pre[nv] + (kParts - 1) * min(s_pre[nv], P.split);
    if (total == 0) return;
    const uint32_t slot = P.lists.deferred_slot;
    const uint32_t defer_cap = P.deferred_cap;
    WarpShared& W = s_warp[warp];
    float4* clip = W.clip;
    int2* sxy = W.xy;
    // {depth bits, flags} of every vertex, which the fast instance reads only
    // for a meshlet that is not entirely inside the view volume, before it
    // writes a record
    static_assert(sizeof(W.tri) >= 64 * sizeof(int2), "vertex flags share the records' memory");
    int2* szf = reinterpret_cast<int2*>(W.tri);
    uint32_t* sidx = W.idx;
    const uint8_t* sidx8 = reinterpret_cast<const uint8_t*>(sidx);
    TriRec* recs = W.tri;
    uint16_t* starts = W.start;
    // Warps take runs of `grab` consecutive work items, their own first and
    // then from one counter, so views are drawn roughly in order (their depth buffers stay in L2) and
    // no warp idles while work is left.
    const uint32_t warps_total = gridDim.x * WARPS;
    const uint32_t grab = max(1u, min(kMaxRun, total / (warps_total * 8u)));
    uint32_t cur_v = 0xffffffffu, cur_t = 0xffffffffu;  // view and node of W.mvp
    const DeviceView* Vp = P.views;
    RasterCtx& c = W.ctx;
    ItemHeader* hdr = W.hdr;
    // the next run is requested while the current one is drawn, so the
    // atomic's round trip is off the critical path
    // The first run of each warp is its own, a warp of every CTA before the
    // second of any: the counter's round trip (2,400 cycles) is not the first
    // thing that a launch of few meshlets waits for (720p sphere 36.7 -> 31.9
    // us a frame, 1080p torus grid, four such launches, 275.4 -> 264.1).
    const uint32_t own = warps_total * grab;
    uint32_t next = ((uint32_t)warp * gridDim.x + blockIdx.x) * grab;
    for (;;) {
        const uint32_t base = __shfl_sync(0xffffffffu, next, 0);
        if (base >= total) break;
        next = 0xffffffffu;
        if (lane == 0 && own < total) next = own + atomicAdd(P.work + (SLOW ? 1 : 0), grab);
        const uint32_t stop = min(base + grab, total);
        {
            uint32_t g = base + (uint32_t)lane;
            ItemHeader h;
            h.d = 0xffffffffu;
            h.v = 0;
            h.t0 = h.t1 = 0;
            if (g < stop) {
                const uint32_t whole = s_pre[nv] - min(s_pre[nv], P.split);
                bool split = g >= whole;
                uint32_t part = 0;
                if (split) {
                    part = (g - whole) % kParts;
                    g = whole + (g - whole) / kParts;
                }
                // the view holding g: the last v with s_pre[v] <= g
                uint32_t v = 0, hi = nv;
                while (v + 1 < hi) {
                    const uint32_t mid = (v + hi) >> 1;
                    if (s_pre[mid] <= g) v = mid;
                    else hi = mid;
                }
                const uint32_t* list;
                uint32_t n, first;
                view_work<SLOW>(P, P.views[v], list, n, first);
                uint32_t d = list[first + (g - s_pre[v])];
                bool skip = false;  // a deferred round that another part of this entry draws
                if (SLOW && (d & kDeferSplit)) {
                    const uint32_t own = (d >> kDeferPartShift) % kParts;
                    skip = split && part != own;
                    split = true;
                    part = own;
                    d &= kDrawMask;
                }
                h.v = v;
                h.d = d;
                bool bad = true;
                if (d < P.S.draw_count) {
                    const vkgv_meshlet_draw dr = P.S.draws[d];
                    const vkgv_primitive* prim = &P.S.prims[dr.primitive_index];
                    if (dr.meshlet_index < prim->meshlet_count) {
                        const vkgv_meshlet* ml =
                            reinterpret_cast<const vkgv_meshlet*>(prim->meshlet_buffer) + dr.meshlet_index;
                        const uint32_t vc = ml->vertex_count, tc = ml->triangle_count;
                        if (vc <= VKGV_MAX_VERTICES && tc <= VKGV_MAX_PRIMITIVES) {
                            h.vidx = reinterpret_cast<const uint32_t*>(prim->vertex_index_buffer) + ml->vertex_offset;
                            h.tri = reinterpret_cast<const uint8_t*>(prim->primitive_index_buffer) + ml->triangle_offset;
                            h.verts = reinterpret_cast<const vkgv_vertex*>(prim->vertex_buffer);
                            h.transform = dr.transform_index;
                            h.vc = (uint8_t)vc;
                            if (!skip) {
                                h.t0 = (uint8_t)(split ? 32u * part : 0u);
                                h.t1 = (uint8_t)(split ? min(tc, 32u * part + 32u) : tc);
                            }
                            h.flags = (uint8_t)((P.S.mats[prim->material_index].double_sided != 0 ? kDoubleSided : 0) |
                                                (split ? kSplit : 0));
                            bad = false;
                        }
                    }
                }
                if (bad) report(P.status, kStatusBadIndex, d);
            }
            __syncwarp();  // every lane is done with the previous run's headers
            if (lane < (int)kMaxRun) hdr[lane] = h;
        }
        __syncwarp();
        for (uint32_t k = 0; k < stop - base; ++k) {
            const ItemHeader& H = hdr[k];
            if (H.t0 >= H.t1) continue;
            const uint32_t v = H.v, d = H.d;
            if (v != cur_v) {
                cur_v = v;
                cur_t = 0xffffffffu;
                Vp = P.views + v;
                __syncwarp();
                if (lane == 0) {
                    c.depth = Vp->depth_id;
                    c.w = Vp->w;
                    c.h = Vp->h;
                    c.hw = 0.5f * (float)Vp->w;
                    c.hh = 0.5f * (float)Vp->h;
                    c.view = P.view_base + v;
                }
                __syncwarp();
            }
            const DeviceView& V = *Vp;
            const uint32_t vc = H.vc, tc = H.t1;
            const uint32_t* vidx = H.vidx;
            const uint8_t* tri = H.tri;
            const vkgv_vertex* verts = H.verts;
            const bool double_sided = (H.flags & kDoubleSided) != 0;
            const uint32_t transform_index = H.transform;
            // mvp = VP * M, one element per lane (lanes 0-15); lane 16 takes the
            // sign source determinant(M) of visbuffer.mesh.glsl:71.
            // Consecutive items of a run mostly come from one node (the draw
            // list is node-major): its matrix and sign are then already here.
            const float* Mg = P.S.transforms + 16 * (size_t)transform_index;
            const bool have_tdet = P.S.tdets != nullptr && transform_index < P.S.transform_count;
            const bool same_node = transform_index == cur_t;
            cur_t = transform_index;
            if (same_node) {
            } else if (lane < 16 && V.mvps && transform_index < P.S.transform_count) {
                W.mvp[lane] = __ldg(V.mvps + 16 * (size_t)transform_index + lane);
            } else if (lane < 16) {
                const int cc = lane >> 2, j = lane & 3;
                const float4 mc = __ldg(reinterpret_cast<const float4*>(Mg) + cc);
                const float* vp = V.cam->view_projection;
                W.mvp[lane] = fadd(fadd(fadd(fmul(vp[0 * 4 + j], mc.x), fmul(vp[1 * 4 + j], mc.y)),
                                              fmul(vp[2 * 4 + j], mc.z)),
                                         fmul(vp[3 * 4 + j], mc.w));
            } else if (lane == 16 && have_tdet) {
                W.tdet = P.S.tdets[transform_index];
            } else if (lane == 16) {
                float M[16];
    #pragma unroll
                for (int q = 0; q < 16; ++q) M[q] = __ldg(Mg + q);
                W.tdet = det4(M);
            }
            if (!same_node) __syncwarp();
            const float tdet = W.tdet;
            const float* mvp = W.mvp;
            // Vertex stage: clip position, outcode, guard flag and the 28.8 snap,
            // each computed once per meshlet vertex (two per lane).  All global
            // loads of the stage, and the triangle-index words (32-bit loads
            // when the block is 4-byte aligned, as meshoptimizer pads each
            // block to 4), are issued before any of the math.
            const uint32_t nbytes = 3 * tc, nwords = (nbytes + 3) / 4;  // <= 95 words
            const bool tri_words = (reinterpret_cast<uintptr_t>(tri) & 3u) == 0;
            uint32_t tw[3] = {0u, 0u, 0u};
            if (tri_words) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (lane + 32u * q < nwords) tw[q] = __ldg(reinterpret_cast<const uint32_t*>(tri) + lane + 32 * q);
            }
            const bool h0 = (uint32_t)lane < vc, h1 = (uint32_t)lane + 32u < vc;
            const vkgv_vertex* vx0 = verts + (h0 ? __ldg(vidx + lane) : 0u);
            const vkgv_vertex* vx1 = verts + (h1 ? __ldg(vidx + lane + 32) : 0u);
            float2 xy0 = make_float2(0.0f, 0.0f), xy1 = xy0;
            float zz0 = 0.0f, zz1 = 0.0f;
            if (h0) {
                xy0 = __ldg(reinterpret_cast<const float2*>(vx0->position));
                zz0 = __ldg(&vx0->position[2]);
            }
            if (h1) {
                xy1 = __ldg(reinterpret_cast<const float2*>(vx1->position));
                zz1 = __ldg(&vx1->position[2]);
            }
            float4 cv[2];
            m4v(mvp, xy0.x, xy0.y, zz0, 1.0f, &cv[0].x);
            m4v(mvp, xy1.x, xy1.y, zz1, 1.0f, &cv[1].x);
            // Inside the view volume no outcode, guard or snap-range test can
            // fire, if w and its reciprocal are finite and not subnormal (an
            // infinite w passes the volume's comparisons, and snaps to no
            // place): a meshlet with all vertices inside skips them here and in
            // the pre-filter (issue-bound: 256 views of 128^2 1,731 -> 1,474 us
            // a frame, the 256-view torus grid 37.0 -> 32.2 ms, with the
            // pre-filter on 8-byte vertices and the relative edge setup).
            // w in [2^-100, 2^100], by the bits: one comparison (two of floats
            // cost the batches 0.5%)
            auto ordinary = [](float w) {
                return __float_as_uint(w) - __float_as_uint(0x1p-100f) <= __float_as_uint(0x1p100f) - __float_as_uint(0x1p-100f);
            };
            auto inside = [&](const float4& q) {
                return fabsf(q.x) <= q.w && fabsf(q.y) <= q.w && q.z >= 0.0f && q.z <= q.w && ordinary(q.w);
            };
            const bool plain = !SLOW && __all_sync(0xffffffffu, (!h0 || inside(cv[0])) && (!h1 || inside(cv[1])));
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (!(q ? h1 : h0)) continue;
                const uint32_t k = (uint32_t)lane + 32u * q;
                const float4 v = cv[q];
                int32_t X = 0, Y = 0;
                float Z = 0.0f;
                if (plain) {
                    snap_inside(v, c, X, Y, Z);
                } else {
                    uint32_t fl = (uint32_t)outcode(v);
                    if (outside_guard(v)) fl |= kFlagGuard;
                    if (snap(v, c, X, Y, Z)) fl |= kFlagSnapped;
                    szf[k] = make_int2(__float_as_int(Z), (int)fl);
                }
                sxy[k] = make_int2(X, Y);
                clip[k] = SLOW ? v : make_float4(v.x, v.y, v.w, Z);
            }
            if (tri_words) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (lane + 32u * q < nwords) sidx[lane + 32 * q] = tw[q];
            } else {
                uint8_t* b = reinterpret_cast<uint8_t*>(sidx);
                for (uint32_t k = lane; k < nbytes; k += 32) b[k] = __ldg(tri + k);
            }
            __syncwarp();
            bool any_slow = false;
            if constexpr (SLOW) {
                // Deferred meshlet: only the triangles the fast instance
                // skipped, 32 per round; the round's binned triangles are
                // queued together when the warp has reconverged.
                JobList jobs;
                jobs.count = 0;
                for (uint32_t tb = H.t0; tb < tc; tb += 32) {
                    const uint32_t t = tb + (uint32_t)lane;
                    if (t < tc) {
                        TriClass k;
                        const uint32_t i0 = sidx8[3 * t], i1 = sidx8[3 * t + 1], i2 = sidx8[3 * t + 2];
                        const int kind = classify(i0, i1, i2, vc, sxy, szf, clip, double_sided, tdet, c, Q, k);
                        if (kind == kSlowClip) {
                            raster_clipped(clip[i0], clip[i1], clip[i2],
                                           ((uint32_t)(k.f0.y | k.f1.y | k.f2.y) & (OC_ZLO | OC_ZHI)) != 0,
                                           (d << 7) | t, c, Q, jobs);
                        } else if (kind == kSlowSetup) {
                            setup_and_raster(k.q0.x, k.q0.y, __int_as_float(k.f0.x), k.q1.x, k.q1.y,
                                             __int_as_float(k.f1.x), k.q2.x, k.q2.y, __int_as_float(k.f2.x),
                                             (d << 7) | t, c, Q, jobs);
                        }
                    }
                    __syncwarp();
                    flush_jobs(jobs, c, Q, lane);
                }
            } else {
                // Pre-filter 32 triangles per round (a pixel centre in the
                // bbox; outcodes and snap flags where a vertex is outside the
                // view volume); the candidates are compacted so that the
                // backface, area and size tests, the setup and the raster run
                // on full warps (at most about a quarter of the triangles of
                // a dense meshlet have a sample in their bbox).
                uint8_t* ring = W.ring;
                uint32_t pending = 0;
                for (uint32_t tbase = H.t0; tbase < tc; tbase += 32) {
                    const uint32_t t = tbase + lane;
                    bool cand = false;
                    if (t < tc) {
                        const uint32_t i0 = sidx8[3 * t], i1 = sidx8[3 * t + 1], i2 = sidx8[3 * t + 2];
                        if (max(i0, max(i1, i2)) >= vc) {
                            report(P.status, kStatusBadIndex, d);
                        } else if (plain) {
                            cand = covers_centre(sxy[i0], sxy[i1], sxy[i2]);
                        } else {
                            const int kind = prefilter(i0, i1, i2, sxy, szf, c);
                            cand = kind == 1;
                            any_slow |= kind == 2;
                        }
                    }
                    const uint32_t fm = __ballot_sync(0xffffffffu, cand);
                    if (cand) ring[pending + __popc(fm & ((1u << lane) - 1u))] = (uint8_t)t;
                    pending += __popc(fm);
                }
                __syncwarp();
                for (uint32_t at = 0; at < pending; at += 32) {
                    const uint32_t ct = at + lane < pending ? ring[at + lane] : 0xffffffffu;
                    any_slow |= raster_small(ct, sidx8, sxy, clip, double_sided, tdet, d, c, Q, recs, starts, lane);
                }
            }
            if (!SLOW && __any_sync(0xffffffffu, any_slow) && lane == 0) {
                const uint32_t k = atomicAdd(&V.counters[slot], 1u);
                if (k < defer_cap)
                    V.deferred[k] = !(H.flags & kSplit) ? d : (d | ((uint32_t)H.t0 / 32u << kDeferPartShift) | kDeferSplit);
                else
                    report(P.status, kStatusListOverflow, d);
            }
            __syncwarp();
        }
    }
}

// A rectangle of a narrow triangle, set up by one lane and drawn by its warp.
struct __align__(16) BigRect {
    int32_t e[3];       // edge values at the rectangle's first pixel centre, clamped, biases subtracted
    uint32_t d[3];      // edge vectors: x | y << 16
    float z0, pa, pb;   // depth plane
    uint32_t id;
    int32_t x, y;       // first pixel centre - vertex 0
    uint32_t width;     // 2^18 / width rounded up (19) | width (7)
    uint32_t area;      // (13) | the view's row pitch in pixels << 16
    unsigned long long* at;
};

// Drains the binned rectangles, each warp up to 32 of them at a time: a lane
// sets up one rectangle (edge values at its corner), then the warp draws them
// one after another, its lanes over a rectangle's pixels in row-major order.
// Issue-bound: set up by all lanes alike, a rectangle of some 34 pixels took
// 160 instructions, most of them setup (119,000 rectangles of the 1080p torus
// grid 34.1 -> 23.5 us).  Runs of neighbouring rectangles instead of every
// warps-th: 31 us.
constexpr int kBigWarps = 8;
__global__ void __launch_bounds__(32 * kBigWarps) k_raster_big(const BigTri* __restrict__ q, const uint32_t* count,
                                                               uint32_t cap, const DeviceView* __restrict__ views) {
    pdl_begin();
    __shared__ BigRect s_rect[kBigWarps][32];
    const uint32_t n = min(*count, cap);
    const uint32_t lane = threadIdx.x & 31u;
    BigRect* rects = s_rect[threadIdx.x >> 5];
    const uint32_t warps = gridDim.x * kBigWarps;
    // Each warp takes every warps-th rectangle (the pieces of one large triangle
    // are neighbours in the queue), 32 of them at a time.
    for (uint32_t first = blockIdx.x * kBigWarps + (threadIdx.x >> 5); first < n; first += 32 * warps) {
        const uint32_t here = min(32u, (n - first + warps - 1) / warps);
        bool wide = false;
        __syncwarp();  // the previous ones are drawn
        if (lane < here) {
            const BigTri t = q[first + lane * warps];
            const DeviceView& V = views[t.view];
            const uint32_t bw = (uint32_t)t.px1 - t.px0 + 1u;
            wide = !(t.flags & kBigNarrow);
            const int32_t cx = ((int32_t)t.px0 << 8) + 128, cy = ((int32_t)t.py0 << 8) + 128;
            BigRect r;
            // Over at most 64 x 64 pixels a narrow triangle's edge value moves
            // by less than 2^30, so the corner's value may be clamped to that
            // without a change of any sign.
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int32_t dx = t.x[(k + 1) % 3] - t.x[k], dy = t.y[(k + 1) % 3] - t.y[k];
                const int64_t c = (int64_t)dx * (cy - t.y[k]) - (int64_t)dy * (cx - t.x[k]) - (int32_t)((t.flags >> k) & 1u);
                constexpr int64_t kLim = 1 << 30;
                r.e[k] = (int32_t)(c < -kLim ? -kLim : (c > kLim ? kLim : c));
                r.d[k] = ((uint32_t)dx & 0xFFFFu) | ((uint32_t)dy << 16);
            }
            r.z0 = t.z0, r.pa = t.pa, r.pb = t.pb;
            r.id = t.id;
            r.x = cx - t.x[0], r.y = cy - t.y[0];
            // floor(i / bw) by a reciprocal rounded up, exact for i < 4096 and
            // bw <= 64: i times its error, below 4096 / 2^18, stays under 1 / bw
            // (whole only for the powers of two, where it is exact)
            r.width = __float2uint_ru(fmul(262144.0f, __frcp_rn((float)bw))) | (bw << 19);
            r.area = (wide ? 0u : bw * ((uint32_t)t.py1 - t.py0 + 1u)) | (V.w << 16);
            r.at = V.depth_id + (size_t)t.py0 * V.w + t.px0;
            rects[lane] = r;
        }
        unsigned wides = __ballot_sync(0xffffffffu, wide);
        for (uint32_t j = 0; j < here; ++j) {
            const BigRect r = rects[j];
            const uint32_t area = r.area & 0xFFFFu, w = r.area >> 16;
            const int32_t dx0 = (int32_t)(int16_t)(r.d[0] & 0xFFFFu), dy0 = (int32_t)r.d[0] >> 16;
            const int32_t dx1 = (int32_t)(int16_t)(r.d[1] & 0xFFFFu), dy1 = (int32_t)r.d[1] >> 16;
            const int32_t dx2 = (int32_t)(int16_t)(r.d[2] & 0xFFFFu), dy2 = (int32_t)r.d[2] >> 16;
            const uint32_t inv = r.width & 0x7FFFFu, bw = r.width >> 19;
            for (uint32_t i = lane; i < area; i += 32) {
                const uint32_t ly = (i * inv) >> 18, lx = i - ly * bw;
                const int32_t sx = (int32_t)(lx << 8), sy = (int32_t)(ly << 8);
                const int32_t a = r.e[0] + sy * dx0 - sx * dy0, b = r.e[1] + sy * dx1 - sx * dy1;
                const int32_t c = r.e[2] + sy * dx2 - sx * dy2;
                if ((a | b | c) >= 0)
                    plot(r.at + (size_t)ly * w + lx,
                         fragment(r.pa, r.pb, r.z0, __int2float_rn(r.x + sx), __int2float_rn(r.y + sy), r.id));
            }
        }
        // triangles of 128 pixels and more: every edge value in 64 bits
        for (; wides; wides &= wides - 1) {
            const BigTri t = q[first + ((uint32_t)__ffs((int)wides) - 1u) * warps];
            const DeviceView& V = views[t.view];
            const uint32_t bw = (uint32_t)t.px1 - t.px0 + 1u, area = bw * ((uint32_t)t.py1 - t.py0 + 1u);
            const uint32_t inv = __float2uint_ru(fmul(262144.0f, __frcp_rn((float)bw)));
            for (uint32_t i = lane; i < area; i += 32) {
                const uint32_t ly = (i * inv) >> 18, px = t.px0 + (i - ly * bw), py = t.py0 + ly;
                const int32_t sx = (int32_t)(px << 8) + 128, sy = (int32_t)(py << 8) + 128;
                bool covered = true;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int64_t ev = (int64_t)(t.x[(k + 1) % 3] - t.x[k]) * (sy - t.y[k]) -
                                       (int64_t)(t.y[(k + 1) % 3] - t.y[k]) * (sx - t.x[k]);
                    covered = covered && ev >= (int64_t)((t.flags >> k) & 1u);
                }
                if (covered)
                    plot(V.depth_id + (size_t)py * V.w + px,
                         fragment(t.pa, t.pb, t.z0, __int2float_rn(sx - t.x[0]), __int2float_rn(sy - t.y[0]), t.id));
            }
        }
    }
}

// Meshlets that a launch splits (see k_raster).
uint32_t raster_split(uint32_t sm_count) { return sm_count * VKGV_RASTER_SPLIT_PER_SM; }

// One wave of CTAs: every warp stays resident and takes work until none is
// left.
template <int WARPS, int SLOW_WARPS = WARPS>
void launch_variant(RasterParams P, uint32_t sm_count, uint32_t blocks_override, cudaStream_t stream) {
    const uint32_t fast = blocks_override ? blocks_override : sm_count * (VKGV_RASTER_WARPS_PER_SM / WARPS);
    const uint32_t slow = blocks_override ? blocks_override : sm_count * (16 / SLOW_WARPS > 0 ? 16 / SLOW_WARPS : 1);
    P.split = raster_split(sm_count);
    const size_t pre = sizeof(uint32_t) * (P.nviews + 1);
    launch_pdl(k_raster<WARPS, false>, dim3(fast), dim3(WARPS * 32), pre, stream, P);
    launch_pdl(k_raster<SLOW_WARPS, true>, dim3(slow), dim3(SLOW_WARPS * 32), pre, stream, P);
}

}  // namespace

uint32_t deferred_capacity(uint32_t draw_count, uint32_t sm_count) {
    // every meshlet once, and the split ones once a round
    const uint32_t split = raster_split(sm_count);
    return draw_count + (kParts - 1) * (draw_count < split ? draw_count : split);
}

void launch_raster(const SceneArgs& S, const DeviceView* views, uint32_t nviews, const RasterLists& lists,
                   const RasterConfig& cfg, BigTri* big, uint32_t* big_count, uint32_t big_capacity,
                   uint32_t* work, uint32_t* status, uint32_t sm_count, cudaStream_t stream, cudaEvent_t between) {
    RasterParams P;
    P.S = S;
    P.lists = lists;
    P.big = big;
    P.big_count = big_count;
    P.big_cap = big_capacity;
    P.small_area = cfg.small_area;
    P.chunk = cfg.chunk;
    P.deferred_cap = deferred_capacity(S.draw_count, sm_count);
    P.status = status;
    P.work = work;
    for (uint32_t v0 = 0; v0 < nviews; v0 += kRasterMaxViews) {
        P.views = views + v0;
        P.nviews = nviews - v0 < kRasterMaxViews ? nviews - v0 : kRasterMaxViews;
        P.view_base = v0;
        // One warp a CTA addresses its shared memory by constants and spills
        // nothing (256 views of the torus grid 29.41 -> 28.77 ms, the 4K frame
        // 506.5 -> 495.1 us, 1080p 248.8 -> 242.6), but a launch of few meshlets
        // waits for its 4,256 CTAs (84 meshlets: 29.2 -> 32.0 us; 1,152: 30.1 ->
        // 30.4; 64 views of 290: 554.8 -> 551.2), and above 512 views their
        // prefixes leave no room for 28 of them on an SM.  The slow instance
        // keeps four (1080p 244.1 with one), also where the caller asks for one,
        // so that a caller who tries one and four tries both forms of the default.
        const bool many = (uint64_t)S.draw_count * P.nviews >= 16384 && P.nviews <= 512;
        switch (cfg.warps_per_cta ? cfg.warps_per_cta : (many ? 1u : 4u)) {
            case 1: launch_variant<1, 4>(P, sm_count, cfg.blocks_per_view, stream); break;
            case 2: launch_variant<2>(P, sm_count, cfg.blocks_per_view, stream); break;
            case 8: launch_variant<8>(P, sm_count, cfg.blocks_per_view, stream); break;
            default: launch_variant<4>(P, sm_count, cfg.blocks_per_view, stream); break;
        }
    }
    if (between) cudaEventRecord(between, stream);
    // Exactly one wave of drain CTAs: its warps stride over the queue
    // statically, so a partial second wave (8 CTAs per SM against 5
    // resident) finished late: single view 36.9 -> 34.8 us, 256 views
    // 0.125 -> 0.111 ms.  (Warps taking rectangles from a counter instead
    // were 1.3-2.9x slower: same-address atomics.)
    static std::atomic<int> resident[64];
    int dev = 0;
    cudaGetDevice(&dev);
    int per_sm = dev >= 0 && dev < 64 ? resident[dev].load(std::memory_order_relaxed) : 0;
    if (per_sm <= 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_raster_big, 32 * kBigWarps, 0) != cudaSuccess || per_sm <= 0)
            per_sm = 4;
        if (dev >= 0 && dev < 64) resident[dev].store(per_sm, std::memory_order_relaxed);
    }
    launch_pdl(k_raster_big, dim3(sm_count * (uint32_t)per_sm), dim3(32 * kBigWarps), 0, stream, (const BigTri*)big,
               (const uint32_t*)big_count, big_capacity, views);
}

}  // namespace vkgv
