// trace_device.cuh -- one-ray-per-thread 3D-DDA traversal (device code of the
// tracer and its single-scene launch helpers, shared by its translation units).
//
// Replaces rtp::UniformGridAccStruct::traceNearestGeometry / traverse3ddda
// (src/rtplugins/UniformGridAccStruct.cpp:30-42, 113-196, 362-378) and the
// reference's GPU tracers (src/rtcuda/RayTracing_kernel.cu:140-275,
// shaders/traversalIntersection_FRAG.glsl:161-263, shaders/shadow_FRAG.glsl:147-245).
//
// The DDA follows the CPU reference exactly -- integer cells, strict-< axis
// choice, exit test x != outX && y != outY && z != outZ, per-cell acceptance
// window [tnear - 1e-4, cellExit + 1e-4] (src/rtcore/RayTriIntersection.cpp:20),
// first cell with a hit ends the walk -- so the visited cells and the tested
// triangles are the reference's.  Each test is Moller-Trumbore, which rejects
// the triangles a ray clearly misses; the candidates it leaves are decided by
// the reference's own projection test on the triangle's TriAccel record, so
// the decisions and the reported t / u / v are the reference's.
//
// Execution: persistent warps.  A warp claims 32 consecutive rays with one
// global atomicAdd, traces them to the end (one ray per lane; consecutive
// camera rays in Morton order stay coherent) and claims the next 32, so no
// warp idles while a block-mate finishes (or, with lane refill, hands new
// rays to its idle lanes as it goes).  Per loop iteration a lane walks up to
// ER empty cells (a tuning parameter), decided from a 4x4x2-brick occupancy
// bitmap whose current word stays in a register, and tests at most one
// non-empty cell (camera rays and coherent arrays: the whole list; other
// arrays: two entries, so that lanes at short lists need not wait for the
// longest), so lanes that reach triangles test them together.  A frame
// (MODE_FRAME) traces each camera ray's shadow ray in the same lane right
// after it.  Rays that meet a long list finish in a group-of-lanes pass,
// those that then meet a dense cluster's list in a block-per-ray pass.
// Launches too small to fill the GPU with one ray a lane (lanes_for) start in
// groups of lanes, which walk consecutive cells of one ray side by side.
#pragma once

#include "common.cuh"
#include "kernels.h"

#include <cuda_fp16.h>

namespace gridrt {

// chunk_alike: how far origins may be apart, in cells, and directions, in lengths
// of the one compared with.  640 x 480 shadow rays of the sphere in Morton order:
// 95 us at 4 and 8 cells, 119 at 2; its 1024^2 ones 128 at a cone of 0.02 to 0.1,
// 162 at 0.01.  Against the first ray (tasks), 640 x 480 camera rays take 192 at
// 0.1 and 235 at 0.05, 64 scenes in one batch 2,514 at 0.1 and 2,539 at 0.15.
static constexpr float kChunkCells = 4.0f;
static constexpr float kChunkCone = 0.1f;
static constexpr unsigned FULL = 0xffffffffu;
static constexpr int32_t kDeferred = -3;    // Lane::id of a ray handed to the group-of-lanes pass
static constexpr int32_t kNoHeavy = 0x7fffffff;
// A ray is also deferred once its tests would pass kHeavyWorkMult x the
// heavy-cell threshold in total (smaller launches: work_mult).
static constexpr int32_t kHeavyWorkMult = 8;


// MODE_FRAME: a camera ray, then in the same lane the shadow ray of its hit
// (any-hit); Lane::tmax is -inf in the camera phase and the shadow ray's
// tmax after.
// MODE_TASK: a batch task's rays, closest hits or occlusion as TraceIO::any
// says (Lane::tmax is -inf for closest hits), one copy of the walk for both.
enum Mode : int { MODE_NEAREST = 0, MODE_ANY = 1, MODE_CAMERA = 2, MODE_FRAME = 3, MODE_TASK = 4 };

struct SParams {
    float bmin[3], bmax[3], cell[3], inv[3];
    int32_t res[3];
    int32_t bx, bxby;
    int32_t failed;
};

__device__ __forceinline__ void fill_sparams(const GridParams* __restrict__ gp, SParams& P) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        P.bmin[d] = gp->bmin[d];
        P.bmax[d] = gp->bmax[d];
        P.cell[d] = gp->cell[d];
        P.inv[d] = gp->inv[d];
        P.res[d] = gp->res[d];
    }
    P.bx = (P.res[0] + 3) >> 2;
    P.bxby = P.bx * ((P.res[1] + 3) >> 2);
    P.failed = build_failed(gp->status) ? 1 : 0;
}

__device__ __forceinline__ void load_sparams(const GridParams* __restrict__ gp, SParams& P) {
    if (threadIdx.x == 0) fill_sparams(gp, P);
    __syncthreads();
}

// Live state of one ray (registers).
struct Lane {
    float ox, oy, oz, dx, dy, dz;
    float ix, iy, iz;
    float tmax, lo;
    float tMx, tMy, tMz, tDx, tDy, tDz;
    int32_t x, y, z;
    int32_t budget;
    int32_t work;        // triangle tests this ray may still make before it is deferred
    int32_t heavy;       // lists longer than this defer it
    float best;
    int32_t id;
    int32_t cw;          // cached occupancy word index
    uint32_t cword;      // its value
    int32_t ray;         // ray index within the launch or task, -1 = none
    int32_t li, le;      // entries of the current cell's list not yet tested (advance_two); li >= le: walking
    bool fast_best;      // best is Moller-Trumbore's t of an accepted entry (test_tri_fast)
};

// Whether the lane's ray looks for occlusion before L.tmax (which may be NaN).
template <int MODE>
__device__ __forceinline__ bool any_hit_phase(const Lane& L) {
    return MODE == MODE_ANY || ((MODE == MODE_FRAME || MODE == MODE_TASK) && L.tmax != -INFINITY);
}

// When the one-lane walk hands the lane's ray on: at a list above `heavy`, or
// once its tests would pass `work` (kNoHeavy: never).
__device__ __forceinline__ void set_deferral(Lane& L, int32_t heavy, int32_t work) {
    L.heavy = heavy;
    L.work = work;
}

inline __host__ __device__ int32_t work_limit(int32_t heavy, int32_t mult) {
    return heavy < kNoHeavy / (mult + 1) ? heavy * mult : kNoHeavy;
}

// Ray::update + AabbIntersection::clipRay + traverse3ddda set-up
// (include/rt/Ray.h:26-37, src/rtcore/AabbIntersection.cpp:37-63,
//  src/rtplugins/UniformGridAccStruct.cpp:122-149).  False if the ray misses
// the grid box.
__device__ __forceinline__ bool setup_ray(const SParams& P, Lane& L, float tnear, float tfar) {
    L.ix = frcp(L.dx);
    L.iy = frcp(L.dy);
    L.iz = frcp(L.dz);
    L.tmax = tfar;
    float rn = tnear, rf = tfar;
    {
        float tn = fmul(fsub(P.bmin[0], L.ox), L.ix), tf = fmul(fsub(P.bmax[0], L.ox), L.ix);
        rn = vmax(rn, vmin(tn, tf));
        rf = vmin(rf, vmax(tn, tf));
        tn = fmul(fsub(P.bmin[1], L.oy), L.iy);
        tf = fmul(fsub(P.bmax[1], L.oy), L.iy);
        rn = vmax(rn, vmin(tn, tf));
        rf = vmin(rf, vmax(tn, tf));
        tn = fmul(fsub(P.bmin[2], L.oz), L.iz);
        tf = fmul(fsub(P.bmax[2], L.oz), L.iz);
        rn = vmax(rn, vmin(tn, tf));
        rf = vmin(rf, vmax(tn, tf));
    }
    if (rn > rf) return false;
    L.lo = fsub(rn, kHitEpsilon);
    const int32_t sx = __float_as_uint(L.dx) >> 31, sy = __float_as_uint(L.dy) >> 31, sz = __float_as_uint(L.dz) >> 31;
    L.x = vclamp(world_to_voxel(fadd(L.ox, fmul(L.dx, rn)), P.bmin[0], P.inv[0]), 0, P.res[0] - 1);
    L.y = vclamp(world_to_voxel(fadd(L.oy, fmul(L.dy, rn)), P.bmin[1], P.inv[1]), 0, P.res[1] - 1);
    L.z = vclamp(world_to_voxel(fadd(L.oz, fmul(L.dz, rn)), P.bmin[2], P.inv[2]), 0, P.res[2] - 1);
    L.tDx = vabs(fmul(P.cell[0], L.ix));
    L.tDy = vabs(fmul(P.cell[1], L.iy));
    L.tDz = vabs(fmul(P.cell[2], L.iz));
    L.tMx = fmul(fsub(voxel_to_world(L.x + (sx ^ 1), P.cell[0], P.bmin[0]), L.ox), L.ix);
    L.tMy = fmul(fsub(voxel_to_world(L.y + (sy ^ 1), P.cell[1], P.bmin[1]), L.oy), L.iy);
    L.tMz = fmul(fsub(voxel_to_world(L.z + (sz ^ 1), P.cell[2], P.bmin[2]), L.oz), L.iz);
    // A walk visits at most nx+ny+nz-2 cells; the bound only guards against a
    // zero direction component (outside the reference's domain) looping.
    L.budget = P.res[0] + P.res[1] + P.res[2] + 3;
    L.best = kFltMax;
    L.id = -1;
    L.cw = -1;
    L.li = L.le = 0;
    return true;
}

#ifndef GRIDRT_EXIT_ALL
#define GRIDRT_EXIT_ALL 0
#endif

// One DDA step (src/rtplugins/UniformGridAccStruct.cpp:179-195): the strict-<
// axis choice and a step of vr::sign(direction).  The reference then exits
// when x == outX (or y, z), with out = -1 for a negative direction sign bit and
// n otherwise (:137-139, :195).  A walk starts inside the grid and moves each
// coordinate only toward its out value, so it reaches out exactly when the
// coordinate leaves [0, n): the test below is the same predicate.  True when
// the walk has left the grid.
__device__ __forceinline__ bool dda_step(const SParams& P, Lane& L) {
    // the other two coordinates did not move and were inside: only the moved
    // one can have left the grid
    bool out;
    if (L.tMx < L.tMy && L.tMx < L.tMz) {
        L.x += L.dx < 0.0f ? -1 : (L.dx > 0.0f ? 1 : 0);
        L.tMx = fadd(L.tMx, L.tDx);
        out = (unsigned)L.x >= (unsigned)P.res[0];
    } else if (L.tMy < L.tMz) {
        L.y += L.dy < 0.0f ? -1 : (L.dy > 0.0f ? 1 : 0);
        L.tMy = fadd(L.tMy, L.tDy);
        out = (unsigned)L.y >= (unsigned)P.res[1];
    } else {
        L.z += L.dz < 0.0f ? -1 : (L.dz > 0.0f ? 1 : 0);
        L.tMz = fadd(L.tMz, L.tDz);
        out = (unsigned)L.z >= (unsigned)P.res[2];
    }
#if GRIDRT_EXIT_ALL
    out = (unsigned)L.x >= (unsigned)P.res[0] || (unsigned)L.y >= (unsigned)P.res[1] ||
          (unsigned)L.z >= (unsigned)P.res[2];
#endif
    return out || --L.budget <= 0;
}

// Triangle test.  Moller-Trumbore on the triangle's {v0, e1, e2} record
// rejects every triangle the ray clearly misses; a triangle that passes it
// within the slacks below -- its barycentrics within kMtBarySlack of the
// triangle, its t within kMtTRelSlack (relative) + 1e-4 of the acceptance
// window and of the best hit so far -- is decided by the reference's own test
// (RayTriIntersection::hitWald, src/rtcore/RayTriIntersection.cpp:12-48) on
// its TriAccel record, in the reference's operation order and rounding.  So
// every accept / reject decision, and the best distance carried from test to
// test, are the reference's: the two float tests round differently near an
// edge or a window bound, but only Wald's decides.  Moller-Trumbore's own
// error stays far inside the slacks (its barycentric error is below 1e-5 for
// the workloads' triangles; a triangle would need a far larger
// distance-to-size ratio for the filter to drop a hit that Wald accepts).
// Returns true when ANY mode found a hit before tmax.
// GRIDRT_MT_EARLY_OUT = 1 lets a lane leave once u (then v) fails.
// GRIDRT_MT_FAST_RCP = 1 takes the filter's 1/det from the hardware's
// approximate reciprocal (rcp.approx), well inside the slacks.
// GRIDRT_DECIDE_WALD = 0 restores plain Moller-Trumbore decisions (ids then
// differ from the reference's at near-ties; the reported values stay Wald's).
#ifndef GRIDRT_MT_EARLY_OUT
#define GRIDRT_MT_EARLY_OUT 1
#endif
#ifndef GRIDRT_MT_FAST_RCP
#define GRIDRT_MT_FAST_RCP 1
#endif
#ifndef GRIDRT_DECIDE_WALD
#define GRIDRT_DECIDE_WALD 1
#endif
static constexpr float kMtBarySlack = GRIDRT_DECIDE_WALD ? 1e-2f : 0.0f;
static constexpr float kMtTRelSlack = 1e-3f;

__device__ __forceinline__ float pick3(float x, float y, float z, uint32_t d) {
    return d == 0 ? x : (d == 1 ? y : z);
}

// hitWald's decision (and f) for triangle `tid` against the lane's ray and
// best distance, window [L.lo, hi].
template <int MODE>
__device__ __forceinline__ bool wald_decide(Lane& L, int32_t tid, float hi, const float4* __restrict__ wald) {
    const float4 a0 = __ldg(wald + 3 * (int64_t)tid);
    const uint32_t k = __float_as_uint(a0.x);
    const uint32_t ku = k == 2 ? 0 : k + 1, kv = k == 0 ? 2 : k - 1;
    const float dk = pick3(L.dx, L.dy, L.dz, k), du = pick3(L.dx, L.dy, L.dz, ku), dv = pick3(L.dx, L.dy, L.dz, kv);
    const float ok = pick3(L.ox, L.oy, L.oz, k), ou = pick3(L.ox, L.oy, L.oz, ku), ov = pick3(L.ox, L.oy, L.oz, kv);
    const float nd = frcp(fadd(fadd(dk, fmul(a0.y, du)), fmul(a0.z, dv)));
    const float f = fmul(nd, fsub(fsub(fsub(a0.w, ok), fmul(a0.y, ou)), fmul(a0.z, ov)));
    if ((f >= L.best) || (f < L.lo) || (f > hi)) return false;
    const float4 a1 = __ldg(wald + 3 * (int64_t)tid + 1);
    const float hu = fadd(ou, fmul(f, du));
    const float hv = fadd(ov, fmul(f, dv));
    const float lambda = fadd(fadd(fmul(hu, a1.x), fmul(hv, a1.y)), a1.z);
    if (lambda < 0.0f) return false;
    const float4 a2 = __ldg(wald + 3 * (int64_t)tid + 2);
    const float mue = fadd(fadd(fmul(hu, a2.x), fmul(hv, a2.y)), a2.z);
    if (mue < 0.0f) return false;
    if (fsub(fsub(1.0f, lambda), mue) < 0.0f) return false;
    L.best = f;
    L.id = tid;
    return (MODE == MODE_ANY || MODE == MODE_FRAME || MODE == MODE_TASK) && f < L.tmax;
}

template <int MODE>
__device__ __forceinline__ bool test_tri(Lane& L, int32_t tid, const float4& A, const float4& B, const float4& C,
                                         float hi, const float4* __restrict__ wald) {
    const float tvx = L.ox - A.x, tvy = L.oy - A.y, tvz = L.oz - A.z;
    const float px = L.dy * C.z - L.dz * C.y;
    const float py = L.dz * C.x - L.dx * C.z;
    const float pz = L.dx * C.y - L.dy * C.x;
    const float det = B.x * px + B.y * py + B.z * pz;
#if GRIDRT_MT_FAST_RCP
    float idet;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(idet) : "f"(det));
#else
    const float idet = frcp(det);
#endif
    const float u = (tvx * px + tvy * py + tvz * pz) * idet;
#if GRIDRT_MT_EARLY_OUT
    // the same predicate, decided in stages: a lane leaves after u
    if (!(u >= -kMtBarySlack)) return false;
#endif
    const float qx = tvy * B.z - tvz * B.y;
    const float qy = tvz * B.x - tvx * B.z;
    const float qz = tvx * B.y - tvy * B.x;
    const float v = (L.dx * qx + L.dy * qy + L.dz * qz) * idet;
#if GRIDRT_MT_EARLY_OUT
    if (!(v >= -kMtBarySlack && (1.0f - u) - v >= -kMtBarySlack)) return false;
#endif
    const float t = (C.x * qx + C.y * qy + C.z * qz) * idet;
#if GRIDRT_DECIDE_WALD
    const float ts = fabsf(t) * kMtTRelSlack + kHitEpsilon;
    if (!((t < L.best + ts) && (t >= L.lo - ts) && (t <= hi + ts) && (u >= -kMtBarySlack) &&
          (v >= -kMtBarySlack) && ((1.0f - u) - v >= -kMtBarySlack)))
        return false;
    return wald_decide<MODE>(L, tid, hi, wald);
#else
    const bool acc = (t < L.best) && (t >= L.lo) && (t <= hi) && (u >= 0.0f) && (v >= 0.0f) &&
                     ((1.0f - u) - v >= 0.0f);
    if (acc) {
        L.best = t;
        L.id = tid;
        if ((MODE == MODE_ANY || MODE == MODE_FRAME || MODE == MODE_TASK) && t < L.tmax) return true;
    }
    return false;
#endif
}

// hitWald's f alone (the exact distance of a hit that test_tri_fast accepted
// without the reference's test, when a later decision compares against it).
__device__ __forceinline__ float wald_f_of(const Lane& L, int32_t tid, const float4* __restrict__ wald) {
    const float4 a0 = __ldg(wald + 3 * (int64_t)tid);
    const uint32_t k = __float_as_uint(a0.x);
    const uint32_t ku = k == 2 ? 0 : k + 1, kv = k == 0 ? 2 : k - 1;
    const float dk = pick3(L.dx, L.dy, L.dz, k), du = pick3(L.dx, L.dy, L.dz, ku), dv = pick3(L.dx, L.dy, L.dz, kv);
    const float ok = pick3(L.ox, L.oy, L.oz, k), ou = pick3(L.ox, L.oy, L.oz, ku), ov = pick3(L.ox, L.oy, L.oz, kv);
    const float nd = frcp(fadd(fadd(dk, fmul(a0.y, du)), fmul(a0.z, dv)));
    return fmul(nd, fsub(fsub(fsub(a0.w, ok), fmul(a0.y, ou)), fmul(a0.z, ov)));
}

// The one-lane walk's test (the same decisions as test_tri).  A candidate
// that Moller-Trumbore puts clearly inside the triangle -- every barycentric
// at least kMtBarySlack inside, t at least the t slack inside the window,
// below the best so far and (any-hit) away from tmax -- is one the
// reference's test accepts too (both tests' errors stay far inside those
// margins), so it is accepted at once with Moller-Trumbore's t as the best
// so far (`fast_best`); only the candidates near an edge or a bound go to the
// reference's test, after the best so far has been replaced by its exact
// value.  The walk ends at the first cell with a hit, so a fast best never
// outlives its cell's list, and the reported values are recomputed exactly
// from the winner's record.
template <int MODE>
__device__ __forceinline__ bool test_tri_fast(Lane& L, int32_t tid, const float4& A, const float4& B,
                                              const float4& C, float hi, const float4* __restrict__ wald,
                                              bool& fast_best) {
#if GRIDRT_DECIDE_WALD
    const float tvx = L.ox - A.x, tvy = L.oy - A.y, tvz = L.oz - A.z;
    const float px = L.dy * C.z - L.dz * C.y;
    const float py = L.dz * C.x - L.dx * C.z;
    const float pz = L.dx * C.y - L.dy * C.x;
    const float det = B.x * px + B.y * py + B.z * pz;
    float idet;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(idet) : "f"(det));
    const float u = (tvx * px + tvy * py + tvz * pz) * idet;
    if (!(u >= -kMtBarySlack)) return false;
    const float qx = tvy * B.z - tvz * B.y;
    const float qy = tvz * B.x - tvx * B.z;
    const float qz = tvx * B.y - tvy * B.x;
    const float v = (L.dx * qx + L.dy * qy + L.dz * qz) * idet;
    const float w = (1.0f - u) - v;
    if (!(v >= -kMtBarySlack && w >= -kMtBarySlack)) return false;
    const float t = (C.x * qx + C.y * qy + C.z * qz) * idet;
    const float ts = fabsf(t) * kMtTRelSlack + kHitEpsilon;
    if (!((t < L.best + ts) && (t >= L.lo - ts) && (t <= hi + ts))) return false;
    const bool any_phase = any_hit_phase<MODE>(L);
    if (u >= kMtBarySlack && v >= kMtBarySlack && w >= kMtBarySlack && t >= L.lo + ts && t <= hi - ts &&
        t < L.best - ts && (!any_phase || t < L.tmax - ts || t > L.tmax + ts)) {
        L.best = t;
        L.id = tid;
        fast_best = true;
        return any_phase && t < L.tmax;
    }
    if (fast_best) {
        L.best = wald_f_of(L, L.id, wald);
        fast_best = false;
    }
    return wald_decide<MODE>(L, tid, hi, wald);
#else
    return test_tri<MODE>(L, tid, A, B, C, hi, wald);
#endif
}

// Tests list entries i and (when i + 1 < e) i + 1, both records loaded before
// either is tested.  True when an any-hit ray is occluded.
template <int MODE>
__device__ __forceinline__ bool test_two(Lane& L, const SceneView& s, int32_t i, int32_t e, float hi) {
    const int32_t i1 = min(i + 1, e - 1);
    int32_t t0 = i, t1 = i1;
    const float4* __restrict__ recs = s.crec;   // in cell-list order: no id indirection
    if (!s.crec) {
        t0 = __ldg(s.ids + i);
        t1 = __ldg(s.ids + i1);
        recs = s.tris;
    }
    const float4 A0 = __ldg(recs + 3 * (int64_t)t0), B0 = __ldg(recs + 3 * (int64_t)t0 + 1),
                 C0 = __ldg(recs + 3 * (int64_t)t0 + 2);
    const float4 A1 = __ldg(recs + 3 * (int64_t)t1), B1 = __ldg(recs + 3 * (int64_t)t1 + 1),
                 C1 = __ldg(recs + 3 * (int64_t)t1 + 2);
    if (test_tri_fast<MODE>(L, __float_as_int(A0.w), A0, B0, C0, hi, s.wald, L.fast_best)) return true;
    return i1 > i && test_tri_fast<MODE>(L, __float_as_int(A1.w), A1, B1, C1, hi, s.wald, L.fast_best);
}

// Walks a lane past up to ER empty cells.  At a non-empty cell sets [L.li, L.le)
// to its list.  True when the ray leaves the grid or is deferred.
template <int ER>
__device__ __forceinline__ bool walk(const SParams& P, Lane& L, const SceneView& s, uint32_t& cells, uint32_t& tests) {
    const int32_t nx = P.res[0], nxy = P.res[0] * P.res[1];
    for (int q = 0; q < ER; ++q) {
        ++cells;
        const int32_t w = (L.x >> 2) + (L.y >> 2) * P.bx + (L.z >> 1) * P.bxby;
        if (w != L.cw) {
            L.cw = w;
            L.cword = __ldg(s.occ + w);
        }
        if (L.cword & occ_bit(L.x, L.y, L.z)) {
            const int32_t c = L.x + L.y * nx + L.z * nxy;
            const int32_t b = __ldg(s.offsets + c), e = __ldg(s.offsets + c + 1);
            if (e - b > min(L.heavy, L.work)) {
                // a long list, or a ray that has made many tests already
                // (grazing a surface): the ray goes to the deferred pass,
                // which resumes the walk at this cell (and counts it)
                --cells;
                L.id = kDeferred;
                return true;
            }
            L.work -= e - b;
            tests += (uint32_t)(e - b);
            L.fast_best = false;
            L.li = b;
            L.le = e;
            return false;
        }
        if (dda_step(P, L)) {
            L.id = -1;
            return true;
        }
    }
    return false;
}

// The end of a cell's list: a hit closer than the best on entry (the
// one-geometry walk starts from FLT_MAX; an instance walk from the instances
// before it) ends the ray -- any-hit: the first cell with a hit decides, here
// not before tmax -- else the ray steps on.  True when the ray is finished.
template <int MODE>
__device__ __forceinline__ bool leave_cell(const SParams& P, Lane& L) {
    if (L.id >= 0) {
        if (any_hit_phase<MODE>(L)) L.id = -1;
        return true;
    }
    if (dda_step(P, L)) {
        L.id = -1;
        return true;
    }
    return false;
}

// One turn of a warp's lanes, each finishing the list it comes to (coherent
// rays: the lanes of a warp meet the same lists).  True for a lane whose ray is
// finished (hit decided, left the grid, or deferred).
template <int MODE, int ER>
__device__ __forceinline__ bool advance(const SParams& P, Lane& L, const SceneView& s, bool active, uint32_t& cells,
                                        uint32_t& tests) {
    bool fin = false;
    if (active) {
        L.li = L.le = 0;
        fin = walk<ER>(P, L, s, cells, tests);
    }
    if (active && !fin && L.li < L.le) {
        const float hi = fadd(vmin(vmin(L.tMx, L.tMy), L.tMz), kHitEpsilon);
        for (; L.li < L.le && !fin; L.li += 2) fin = test_two<MODE>(L, s, L.li, L.le, hi);
        if (!fin) fin = leave_cell<MODE>(P, L);
    }
    return fin;
}

// One turn of a warp's lanes among incoherent rays: lanes between lists walk,
// lanes at a list test two of its entries, so a long list does not hold up the
// warp's other rays.  Whole lists a turn left 7.7 of 32 lanes active on random
// rays; with this turn and refill at 8 idle lanes instead of 16, 4 M closest-hit
// rays went from 2,468 to 2,237 us, 700,001 occlusion segments from 749 to
// 576 us.  Coherent rays do better by whole lists (1024^2 camera rays of the
// sphere given as an array: 246 us, by two entries a turn 349 us).
template <int MODE, int ER>
__device__ __forceinline__ bool advance_two(const SParams& P, Lane& L, const SceneView& s, bool active,
                                            uint32_t& cells, uint32_t& tests) {
    bool fin = false;
    // half the empty cells of a coherent turn: lanes at a list wait for them
    if (active && L.li >= L.le) fin = walk<(ER > 2 ? ER / 2 : ER)>(P, L, s, cells, tests);
    if (active && !fin && L.li < L.le) {
        const float hi = fadd(vmin(vmin(L.tMx, L.tMy), L.tMz), kHitEpsilon);
        fin = test_two<MODE>(L, s, L.li, L.le, hi);
        L.li += 2;
        if (!fin && L.li >= L.le) fin = leave_cell<MODE>(P, L);
    }
    return fin;
}

// Reported hit values of the winning triangle: RayTriIntersection::hitWald
// (src/rtcore/RayTriIntersection.cpp:12-48) on the triangle's TriAccel record
// (written by the build exactly as TriAccel::buildFrom computes it), with the
// reference's operation order and one rounding per operation.  The accept /
// reject decisions of the walk stay Moller-Trumbore's; when the walk's winner
// is the reference's triangle, t (hitWald's f), u (lambda) and v (mue) are the
// reference's bits.
__device__ __forceinline__ int4 wald_hit(const float4* __restrict__ wald, const Lane& L) {
    const float4 a0 = __ldg(wald + 3 * (int64_t)L.id);
    const float4 a1 = __ldg(wald + 3 * (int64_t)L.id + 1);
    const float4 a2 = __ldg(wald + 3 * (int64_t)L.id + 2);
    const uint32_t k = __float_as_uint(a0.x);
    const uint32_t ku = k == 2 ? 0 : k + 1, kv = k == 0 ? 2 : k - 1;
    const float dk = pick3(L.dx, L.dy, L.dz, k), du = pick3(L.dx, L.dy, L.dz, ku), dv = pick3(L.dx, L.dy, L.dz, kv);
    const float ok = pick3(L.ox, L.oy, L.oz, k), ou = pick3(L.ox, L.oy, L.oz, ku), ov = pick3(L.ox, L.oy, L.oz, kv);
    const float nd = frcp(fadd(fadd(dk, fmul(a0.y, du)), fmul(a0.z, dv)));
    const float f = fmul(nd, fsub(fsub(fsub(a0.w, ok), fmul(a0.y, ou)), fmul(a0.z, ov)));
    const float hu = fadd(ou, fmul(f, du));
    const float hv = fadd(ov, fmul(f, dv));
    float lambda = fadd(fadd(fmul(hu, a1.x), fmul(hv, a1.y)), a1.z);
    float mue = fadd(fadd(fmul(hu, a2.x), fmul(hv, a2.y)), a2.z);
    float t = f;
    if (!(isfinite(f) && isfinite(lambda) && isfinite(mue))) {
        // a triangle without a finite projection record (the reference drops
        // such triangles at ingest): keep the walk's t
        t = L.best;
        lambda = 0.0f;
        mue = 0.0f;
    }
    return make_int4(L.id, __float_as_int(t), __float_as_int(lambda), __float_as_int(mue));
}

__device__ __forceinline__ void ray_pixel(int32_t i, const CameraArgs& cam, int32_t& px, int32_t& py) {
    if (cam.order == 1) {
        const int32_t tile = i >> 6;
        const int32_t r = (int32_t)(i & 63);
        const int32_t tiles_x = cam.width >> 3;
        const int32_t tx = (int32_t)(tile % tiles_x), ty = (int32_t)(tile / tiles_x);
        px = tx * 8 + ((r & 1) | ((r >> 1) & 2) | ((r >> 2) & 4));
        py = ty * 8 + (((r >> 1) & 1) | ((r >> 2) & 2) | ((r >> 3) & 4));
    } else {
        px = (int32_t)(i % cam.width);
        py = (int32_t)(i / cam.width);
    }
}

struct TraceIO {
    const float4* rays;       // NEAREST / ANY
    int4* hits;               // NEAREST / CAMERA
    uint8_t* occ;             // ANY
    float4* shadow_rays;      // CAMERA (optional): shadow or diffuse secondary rays
    CameraArgs cam;           // CAMERA
    float3 light;
    int has_light;
    int diffuse;              // CAMERA: secondary = cosine-weighted diffuse ray
    unsigned long long seed;
    long long n;
    unsigned long long* counter;   // [0] ray claims, [1] deferred rays, [2] deferred claims
    TraceCounters* ctr;
    int2* defer;                   // deferred rays {ray index, cell it stopped at} (nullptr: no deferral)
    int32_t defer_cap;
    int32_t heavy;                 // lists longer than this are deferred (kNoHeavy: never)
    int32_t work;                  // and rays with more tests than this
    int32_t defer_base;            // added to a deferred ray's index (a batch task's first)
    int32_t refill;                // > 0: lane refill at this many idle lanes (trace_refill)
    int32_t alike;                 // eighths of a chunk's rays that must be like the ray before them (chunk_alike)
    int any;                       // TASK: occlusion (else closest hits)
    int2* huge;                    // rays at a list above kHugeList, for the block pass (nullptr: none)
    int32_t huge_cap;
};

// Loads ray `r` into the lane; false when the ray ends at once (misses the
// grid, or ANY mode with no shadow ray).
template <int MODE>
__device__ __forceinline__ bool start_ray(const SParams& P, const TraceIO& io, Lane& L, int32_t r) {
    float tnear, tfar;
    if (MODE == MODE_FRAME) L.tmax = -INFINITY;   // the camera phase
    if (MODE == MODE_CAMERA || MODE == MODE_FRAME) {
        int32_t px, py;
        ray_pixel(r, io.cam, px, py);
        const float us = fmul(fadd(__int2float_rn(px), 0.5f), io.cam.inv_w);
        const float vs = fmul(fadd(__int2float_rn(py), 0.5f), io.cam.inv_h);
        L.ox = io.cam.eye[0]; L.oy = io.cam.eye[1]; L.oz = io.cam.eye[2];
        L.dx = fadd(fadd(io.cam.base[0], fmul(io.cam.nu[0], us)), fmul(io.cam.nv[0], vs));
        L.dy = fadd(fadd(io.cam.base[1], fmul(io.cam.nu[1], us)), fmul(io.cam.nv[1], vs));
        L.dz = fadd(fadd(io.cam.base[2], fmul(io.cam.nu[2], us)), fmul(io.cam.nv[2], vs));
        tnear = kRayEpsilon;
        tfar = kFltMax;
    } else {
        const float4 a = __ldg(io.rays + 2 * (int64_t)r), b = __ldg(io.rays + 2 * (int64_t)r + 1);
        L.ox = a.x; L.oy = a.y; L.oz = a.z;
        L.dx = b.x; L.dy = b.y; L.dz = b.z;
        tnear = a.w;
        tfar = b.w;
        if ((MODE == MODE_ANY || (MODE == MODE_TASK && io.any)) && tfar < 0.0f) {   // no shadow ray for this slot
            L.id = -2;
            return false;
        }
    }
    L.id = -1;
    L.best = kFltMax;
    if (P.failed) return false;
    const bool ok = setup_ray(P, L, tnear, tfar);
    if (MODE == MODE_FRAME || (MODE == MODE_TASK && !io.any)) L.tmax = -INFINITY;
    return ok;
}

// splitmix64 finaliser: counter-based random bits for ray index `i`.
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// Cosine-weighted direction about unit normal n (Malley's method: uniform
// disc sample lifted to the hemisphere), 24-bit uniforms from mix64.
__device__ __forceinline__ float3 cosine_dir(float nx, float ny, float nz, unsigned long long bits) {
    const float u1 = (float)(bits >> 40) * (1.0f / 16777216.0f);
    const float u2 = (float)((bits >> 16) & 0xffffffull) * (1.0f / 16777216.0f);
    const float r = sqrtf(u1);
    float sp, cp;
    sincospif(2.0f * u2, &sp, &cp);
    const float lx = r * cp, ly = r * sp, lz = sqrtf(fmaxf(0.0f, 1.0f - u1));
    // orthonormal basis (Frisvad-style, branch on the sign of nz)
    const float sgn = nz >= 0.0f ? 1.0f : -1.0f;
    const float a = -1.0f / (sgn + nz);
    const float b = nx * ny * a;
    const float tx = 1.0f + sgn * nx * nx * a, ty = sgn * b, tz = -sgn * nx;
    const float bx = b, by = sgn + ny * ny * a, bz = -ny;
    return make_float3(lx * tx + ly * bx + lz * nx, lx * ty + ly * by + lz * ny, lx * tz + ly * bz + lz * nz);
}

// Writes the lane's result (when `write`: the lanes of a group or block that
// share a ray all compute it, one writes).  Returns true when the lane goes
// on with a follow-up ray: MODE_FRAME's camera phase sets up the hit's shadow
// ray in the lane, from the same values it writes to the shadow-ray slot.
template <int MODE>
__device__ __forceinline__ bool finish_ray(const TraceIO& io, const SParams& P, const SceneView& sv, Lane& L,
                                           bool write = true) {
    const float4* __restrict__ tris = sv.tris;
    const float4* __restrict__ wald = sv.wald;
    const int64_t r = L.ray;
    if (MODE == MODE_TASK ? io.any != 0 : any_hit_phase<MODE>(L)) {
        if (write) io.occ[r] = L.id == -2 ? 2 : (L.id >= 0 ? 1 : 0);
        return false;
    }
    int4 h = make_int4(-1, 0, 0, 0);
    if (L.id >= 0) h = wald_hit(wald, L);
    if (write) io.hits[r] = h;
    if (MODE == MODE_CAMERA || MODE == MODE_FRAME) {
        float4 sa = make_float4(0.f, 0.f, 0.f, kRayEpsilon), sb = make_float4(0.f, 0.f, 0.f, -1.0f);
        if (L.id >= 0 && io.diffuse) {
            // secondary diffuse ray from the hit point, offset along the
            // normal facing the incoming ray, tnear 2e-4, tfar FLT_MAX
            const float t = __int_as_float(h.y);
            const float4 B = __ldg(tris + 3 * (int64_t)L.id + 1);
            const float4 C = __ldg(tris + 3 * (int64_t)L.id + 2);
            float nx = B.y * C.z - B.z * C.y, ny = B.z * C.x - B.x * C.z, nz = B.x * C.y - B.y * C.x;
            const float rl = rsqrtf(nx * nx + ny * ny + nz * nz);
            nx *= rl; ny *= rl; nz *= rl;
            if (nx * L.dx + ny * L.dy + nz * L.dz > 0.0f) { nx = -nx; ny = -ny; nz = -nz; }
            const float3 w = cosine_dir(nx, ny, nz, mix64(io.seed ^ mix64((unsigned long long)r)));
            sa = make_float4(L.ox + L.dx * t + nx * kRayEpsilon, L.oy + L.dy * t + ny * kRayEpsilon,
                             L.oz + L.dz * t + nz * kRayEpsilon, kRayEpsilon);
            sb = make_float4(w.x, w.y, w.z, kFltMax);
        } else if (L.id >= 0 && io.has_light) {
            // Sample::computeHitPosition, flat normal facing the ray, initLightRay
            // offset and initShadowRay (src/rtcore/Sample.cpp:22-42,177-180,224-236),
            // SimplePointLight::illuminate (src/rtplugins/SimplePointLight.cpp:25-33)
            const float t = __int_as_float(h.y);
            const float4 B = __ldg(tris + 3 * (int64_t)L.id + 1);
            const float4 C = __ldg(tris + 3 * (int64_t)L.id + 2);
            float nx = B.y * C.z - B.z * C.y, ny = B.z * C.x - B.x * C.z, nz = B.x * C.y - B.y * C.x;
            const float rl = rsqrtf(nx * nx + ny * ny + nz * nz);
            nx *= rl; ny *= rl; nz *= rl;
            if (nx * L.dx + ny * L.dy + nz * L.dz > 0.0f) { nx = -nx; ny = -ny; nz = -nz; }
            const float hx = L.ox + L.dx * t + nx * kRayEpsilon;
            const float hy = L.oy + L.dy * t + ny * kRayEpsilon;
            const float hz = L.oz + L.dz * t + nz * kRayEpsilon;
            const float lx = io.light.x - hx, ly = io.light.y - hy, lz = io.light.z - hz;
            if (nx * lx + ny * ly + nz * lz > 0.0f) {
                sa = make_float4(hx, hy, hz, kRayEpsilon);
                sb = make_float4(lx, ly, lz, 1.0f);
            }
        }
        if (io.shadow_rays && write) {
            io.shadow_rays[2 * r] = sa;
            io.shadow_rays[2 * r + 1] = sb;
        }
        if (MODE == MODE_FRAME) {
            // the shadow ray as the any-hit pass would load it from the slot
            if (sb.w < 0.0f) {
                if (write) io.occ[r] = 2;
                return false;
            }
            L.ox = sa.x; L.oy = sa.y; L.oz = sa.z;
            L.dx = sb.x; L.dy = sb.y; L.dz = sb.z;
            L.id = -1;
            L.best = kFltMax;
            if (!setup_ray(P, L, sa.w, sb.w)) {
                if (write) io.occ[r] = 0;
                return false;
            }
            return true;
        }
    }
    return false;
}

// Deferred-queue entry of the lane's ray: its index (plus a batch task's
// first), or -1 - index for a MODE_FRAME shadow ray.
template <int MODE>
__device__ __forceinline__ int32_t defer_tag(const Lane& L, const TraceIO& io) {
    return (MODE == MODE_FRAME && L.tmax > -kFltMax) ? -1 - L.ray : L.ray + io.defer_base;
}

// Hands on the lanes that stopped at a long list, or after many tests: one
// atomicAdd for the warp's.  The walk resumes at the lane's cell in the
// group-of-lanes pass.
template <int MODE>
__device__ __forceinline__ void hand_on(const SParams& P, const TraceIO& io, Lane& L, bool& active, bool& fin) {
    const int lane = threadIdx.x & 31;
    const bool d = fin && L.id == kDeferred;
    const unsigned m = __ballot_sync(FULL, d);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    unsigned long long at = 0;
    if (lane == leader) at = atomicAdd(io.counter + 1, (unsigned long long)__popc(m));
    at = __shfl_sync(FULL, at, leader);
    if (d) {
        const unsigned long long slot = at + __popc(m & ((1u << lane) - 1u));
        if (slot < (unsigned long long)io.defer_cap) {
            io.defer[slot] = make_int2(defer_tag<MODE>(L, io), L.x + L.y * P.res[0] + L.z * P.res[0] * P.res[1]);
            active = false;
        } else {
            set_deferral(L, kNoHeavy, kNoHeavy);   // queue full: the lane tests the cell itself
            L.id = -1;
        }
        fin = false;
    }
}

template <int MODE, int ER>
__device__ __forceinline__ void trace_batch32(const SParams& P, const SceneView& s, const TraceIO& io, Lane& L,
                                              long long base, uint32_t& cells, uint32_t& tests, uint32_t& started) {
    const int lane = threadIdx.x & 31;
    const long long ray = base + lane;
    bool active = ray < io.n;
    L.ray = (int32_t)ray;
    set_deferral(L, io.heavy, io.work);
    if (active) {
        ++started;
        if (!start_ray<MODE>(P, io, L, L.ray)) {
            if (L.id != -2) L.id = -1;
            active = finish_ray<MODE>(io, P, s, L);
        }
    }
    while (__any_sync(FULL, active)) {
        bool fin = advance<MODE, ER>(P, L, s, active, cells, tests);
        if (io.defer) hand_on<MODE>(P, io, L, active, fin);
        if (fin) active = finish_ray<MODE>(io, P, s, L);
    }
}

__device__ __forceinline__ void flush_counters(TraceCounters* ctr, uint32_t started, uint32_t cells, uint32_t tests) {
    unsigned long long r = started, c = cells, t = tests;
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_xor_sync(FULL, r, o);
        c += __shfl_xor_sync(FULL, c, o);
        t += __shfl_xor_sync(FULL, t, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&ctr->rays, r);
        atomicAdd(&ctr->cells, c);
        atomicAdd(&ctr->tests, t);
    }
}

// Eight blocks of 128 threads per SM (64 registers a thread) for camera rays:
// the walk is latency-bound, and resident warps matter more than the few
// spilled words.  Seven for rays given as arrays, whose kernel holds both the
// coherent and the refilled walk: 4 M random closest-hit rays take 2,288 us at
// seven, 2,425 at eight, 2,395 at six.
#ifndef GRIDRT_TRACE_MIN_BLOCKS
#define GRIDRT_TRACE_MIN_BLOCKS 8
#endif
constexpr int trace_min_blocks(int mode, int tpb) {
    return (mode == MODE_NEAREST || mode == MODE_ANY) && tpb <= 128 ? 7 * 128 / tpb : GRIDRT_TRACE_MIN_BLOCKS * 128 / tpb;
}

// Whether the 32 rays from `base` walk alike: of those that follow another ray,
// most start within a few cells of it and go within a narrow cone of its
// direction (camera rays, shadow rays of one surface or two); in a batch's task,
// of the first ray's direction.  Slots without a shadow ray (tfar < 0) are
// neither.  1024^2 shadow rays of the sphere and of plane and debris, scanline,
// 135 and 228 us; every origin against the first slot's, which may hold no ray,
// 178 and 222; pairs within two cells and 0.05 134 and 255 at half of them.
// Directions against the first ray's: camera rays of 540 x 540 pixels, whose rows
// end within a chunk, 100 us for 74 (25,760 triangles: 167 for 141); but 64
// scenes in one batch, images of 50 to 400 pixels a row, 2,514 for 2,565, which
// are the better by refill.  One component at a time: the lanes' walks are live
// around it.
template <bool TASK>
static __device__ __noinline__ bool chunk_alike(float cx, float cy, float cz, const float4* rays, int32_t n, int32_t base,
                                                int32_t eighths) {
    const int32_t r = min(base + (int32_t)(threadIdx.x & 31), n - 1);
    const float* __restrict__ q = reinterpret_cast<const float*>(rays + 2 * (int64_t)r);
    const float cell[3] = {cx, cy, cz};
    const unsigned live = __ballot_sync(FULL, !(__ldg(q + 7) < 0.0f)), pairs = live & (live << 1);
    const int first = live ? __ffs(live) - 1 : 0;
    bool alike = true;
    float off = 0.0f, len = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float o = __ldg(q + a), d = __ldg(q + 4 + a);
        const float o0 = __shfl_up_sync(FULL, o, 1);
        const float d0 = TASK ? __shfl_sync(FULL, d, first) : __shfl_up_sync(FULL, d, 1);
        if (!(fabsf(o - o0) <= kChunkCells * cell[a])) alike = false;
        off += fabsf(d - d0);
        len += fabsf(d0);
    }
    return 8 * __popc(__ballot_sync(FULL, alike && off <= kChunkCone * len) & pairs) >= eighths * __popc(pairs);
}
template <bool TASK>
__device__ __forceinline__ bool chunk_coherent(const SParams& P, const TraceIO& io, int32_t base) {
    return chunk_alike<TASK>(P.cell[0], P.cell[1], P.cell[2], io.rays, (int32_t)io.n, base, io.alike);
}

// Lane refill for incoherent rays: instead of tracing a claimed batch of 32 to
// its end, the warp hands new rays to its idle lanes whenever at least
// io.refill of them are idle (one claim for all of them), keeping the lanes
// busy while long rays finish.  Starts on the 32 rays at `chunk` and goes on to
// the launch's last ray.
template <int MODE, int ER>
__device__ __forceinline__ void trace_refill(const SParams& P, const SceneView& s, const TraceIO& io, Lane& L,
                                             unsigned long long chunk, uint32_t& cells, uint32_t& tests,
                                             uint32_t& started) {
    const int lane = threadIdx.x & 31;
    bool active = false, exhausted = false, first = true;
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !active);
        if (!exhausted && ((int)__popc(idle) >= io.refill || idle == FULL)) {
            const unsigned need = (unsigned)__popc(idle);
            unsigned long long b = chunk;
            if (!first) {
                if (lane == 0) b = atomicAdd(io.counter, (unsigned long long)need);
                b = __shfl_sync(FULL, b, 0);
            }
            first = false;
            if ((long long)(b + need) >= io.n) exhausted = true;
            if (!active) {
                const long long ray = (long long)b + __popc(idle & ((1u << lane) - 1u));
                if (ray < io.n) {
                    L.ray = (int32_t)ray;
                    set_deferral(L, io.heavy, io.work);
                    ++started;
                    if (start_ray<MODE>(P, io, L, L.ray)) {
                        active = true;
                    } else {
                        if (L.id != -2) L.id = -1;
                        active = finish_ray<MODE>(io, P, s, L);
                    }
                }
            }
        }
        if (!__any_sync(FULL, active)) {
            if (exhausted) break;
            continue;
        }
        bool fin = advance_two<MODE, ER>(P, L, s, active, cells, tests);
        if (io.defer) hand_on<MODE>(P, io, L, active, fin);
        if (fin) active = finish_ray<MODE>(io, P, s, L);
    }
}

template <int MODE, bool COUNT, int ER, int TPB>
__global__ void __launch_bounds__(TPB, trace_min_blocks(MODE, TPB)) trace_kernel(SceneView s, TraceIO io) {
    pdl_begin();
    __shared__ SParams P;
    load_sparams(s.params, P);
    const int lane = threadIdx.x & 31;
    Lane L;
    uint32_t cells = 0, tests = 0, started = 0;
    unsigned long long b = 0;
    if (lane == 0) b = atomicAdd(io.counter, 32ull);
    b = __shfl_sync(FULL, b, 0);
    // the warp traces 32 consecutive rays to the end and claims the next 32;
    // with lane refill, from the first 32 that are not alike on, it hands out
    // the launch's rays lane by lane
    constexpr bool kArrays = MODE == MODE_NEAREST || MODE == MODE_ANY;
    while ((long long)b < io.n) {
        if (io.refill > 0 && !(kArrays && chunk_coherent<false>(P, io, (int32_t)b))) {
            trace_refill<MODE, ER>(P, s, io, L, b, cells, tests, started);
            break;
        }
        trace_batch32<MODE, ER>(P, s, io, L, (long long)b, cells, tests, started);
        if (lane == 0) b = atomicAdd(io.counter, 32ull);
        b = __shfl_sync(FULL, b, 0);
    }
    if (COUNT) flush_counters(io.ctr, started, cells, tests);
}

// A deferred ray resumes at the cell where its lane stopped: every coordinate
// moved monotonically from the start cell, one step per crossing of its
// axis, each adding tD to tM, so replaying those additions in order rebuilds
// the walk's exact state there (the earlier cells were tested without a hit).
__device__ __forceinline__ void resume_at(const SParams& P, Lane& L, int32_t cell) {
    const int32_t nx = P.res[0], nxy = P.res[0] * P.res[1];
    const int32_t z = cell / nxy, y = (cell - z * nxy) / nx, x = cell - z * nxy - y * nx;
    const int32_t sx = abs(x - L.x), sy = abs(y - L.y), sz = abs(z - L.z);
    for (int32_t i = 0; i < sx; ++i) L.tMx = fadd(L.tMx, L.tDx);
    for (int32_t i = 0; i < sy; ++i) L.tMy = fadd(L.tMy, L.tDy);
    for (int32_t i = 0; i < sz; ++i) L.tMz = fadd(L.tMz, L.tDz);
    L.x = x;
    L.y = y;
    L.z = z;
    L.budget -= sx + sy + sz;
}

// ---------------------------------------------------------------------------
// Group walk: G lanes trace one ray together, lane j at the j-th next cell of
// its walk.  Used for the rays the one-lane walk defers (a long list, or many
// tests made already) and for every ray of a small launch (lanes_for) or of one
// with RTG_TUNE_LANES 2 or 4.
//
// Bound by latency: a walk is a chain of dependent loads (occupancy word, list
// bounds, ids, records) of ~1 us a non-empty cell, and a launch ends with its
// longest rays.  Lanes that split one cell's list at a time shorten only long
// lists; most of a long ray's cells hold two or three triangles.  So the lanes
// take G consecutive cells at once: each steps the whole DDA itself (the same
// additions in the same order, ten instructions a cell and no loads), their G
// cells' loads are in flight together, and the lists found, end to end, are
// dealt out evenly over the lanes.  The lane that owns an entry's cell gives it
// the list position and the cell's window by shuffle.  A hit in an earlier cell
// beats any in a later one; inside a cell the smaller t wins, then the smaller
// id (ids ascend along a list), which is the one-lane walk's result.
// The pass over deferred rays alone, before -> after: 215 -> 75 us behind 1.5 M
// random rays in 495,000 triangles, 70 -> 46 us behind a 1024^2 frame of the
// 102,400-triangle sphere.
// ---------------------------------------------------------------------------
// What a batch of G cells came to: the ray goes on, is finished (L.id), or
// stopped before a list longer than `thr` (its cell and length).
enum GroupStep : int { GROUP_ON = 0, GROUP_DONE = 1, GROUP_LIST = 2 };
struct GroupOut {
    int step;
    int32_t cell, len, lane;  // GROUP_LIST: the cell, its list's length, the lane that stands on it
    int32_t cells, tests;     // visited and tested by the one-lane walk's count
};

// Direction of a DDA step along each axis (vr::sign of the direction).
__device__ __forceinline__ int3 step_signs(const Lane& L) {
    return make_int3(L.dx < 0.0f ? -1 : (L.dx > 0.0f ? 1 : 0), L.dy < 0.0f ? -1 : (L.dy > 0.0f ? 1 : 0),
                     L.dz < 0.0f ? -1 : (L.dz > 0.0f ? 1 : 0));
}

// Moves every lane `todo` cells on (its place in the group for a new ray, G
// after that, 0 to visit the same cells again) and tests the lists of the
// group's cells, but for those of its first `skip` + 1 lanes.  Called by the
// whole warp; `busy` is the same for a group.
template <int G>
__device__ __forceinline__ GroupOut group_batch(const SParams& P, const SceneView& s, Lane& L, const int3& sg,
                                                bool busy, bool any, int todo, int32_t thr, int skip = -1) {
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), g0 = lane & ~(G - 1);
    constexpr unsigned gm = G == 32 ? FULL : ((1u << G) - 1u);
    // dda_step without its exit test: a coordinate that has left the grid
    // moves on outward, so the batch's end tells whether it ever left
#pragma unroll
    for (int j = 0; j < G; ++j) {
        const bool go = j < todo;
        const bool ax = L.tMx < L.tMy && L.tMx < L.tMz;
        const bool ay = !ax && L.tMy < L.tMz;
        if (go && ax) { L.x += sg.x; L.tMx = fadd(L.tMx, L.tDx); }
        if (go && ay) { L.y += sg.y; L.tMy = fadd(L.tMy, L.tDy); }
        if (go && !ax && !ay) { L.z += sg.z; L.tMz = fadd(L.tMz, L.tDz); }
    }
    L.budget -= todo;
    const bool out = (unsigned)L.x >= (unsigned)P.res[0] || (unsigned)L.y >= (unsigned)P.res[1] ||
                     (unsigned)L.z >= (unsigned)P.res[2] || L.budget <= 0;
    int32_t b = 0, n = 0, c = 0;
    if (busy && !out && gl > skip) {
        const int32_t w = (L.x >> 2) + (L.y >> 2) * P.bx + (L.z >> 1) * P.bxby;
        if (__ldg(s.occ + w) & occ_bit(L.x, L.y, L.z)) {
            c = L.x + P.res[0] * (L.y + L.z * P.res[1]);
            b = __ldg(s.offsets + c);
            n = __ldg(s.offsets + c + 1) - b;
        }
    }
    const unsigned om = (__ballot_sync(FULL, busy && out) >> g0) & gm;   // lanes past the grid
    int hj = G;                                                          // cell of this lane's hit
    int fh = G;                                                          // first cell with a list above thr
    int32_t limit = 0, incl = n;
    if (__any_sync(FULL, n > 0)) {
        const float hi = fadd(vmin(vmin(L.tMx, L.tMy), L.tMz), kHitEpsilon);
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const int32_t y = __shfl_up_sync(FULL, incl, o, G);
            if (gl >= o) incl += y;
        }
        const int32_t excl = incl - n, first = b - excl;
        const unsigned hm = (__ballot_sync(FULL, n > thr) >> g0) & gm;
        if (hm) fh = __ffs(hm) - 1;
        limit = __shfl_sync(FULL, hm ? excl : incl, hm ? fh : G - 1, G);   // hm is the same for the group
        for (int32_t base = 0; __any_sync(FULL, base < limit); base += G) {
            const int32_t q = base + gl;
            int j = 0;                               // the lane whose list holds entry q
#pragma unroll
            for (int w = G >> 1; w > 0; w >>= 1)
                if (__shfl_sync(FULL, incl, j + w - 1, G) <= q) j += w;
            const int32_t at = __shfl_sync(FULL, first, j, G) + q;
            const float hij = __shfl_sync(FULL, hi, j, G);
            if (q < limit && j <= hj) {
                int32_t t;
                float4 A, B, C;
                if (s.crec) {
                    A = __ldg(s.crec + 3 * (int64_t)at);
                    B = __ldg(s.crec + 3 * (int64_t)at + 1);
                    C = __ldg(s.crec + 3 * (int64_t)at + 2);
                    t = __float_as_int(A.w);
                } else {
                    t = __ldg(s.ids + at);
                    A = __ldg(s.tris + 3 * (int64_t)t);
                    B = __ldg(s.tris + 3 * (int64_t)t + 1);
                    C = __ldg(s.tris + 3 * (int64_t)t + 2);
                }
                const int32_t was = L.id;
                test_tri<MODE_NEAREST>(L, t, A, B, C, hij, s.wald);
                if (L.id != was) hj = j;
            }
            if (__any_sync(FULL, hj < G)) {          // nothing after a hit's cell is needed
                int m = hj;
#pragma unroll
                for (int o = G >> 1; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(FULL, m, o));
                const int32_t end = __shfl_sync(FULL, incl, m & (G - 1), G);
                if (m < G) limit = min(limit, end);
            }
        }
    }
    if (__any_sync(FULL, hj < G)) {
#pragma unroll
        for (int o = G >> 1; o > 0; o >>= 1) {
            const int oj = __shfl_xor_sync(FULL, hj, o);
            const float ot = __shfl_xor_sync(FULL, L.best, o);
            const int32_t oid = __shfl_xor_sync(FULL, L.id, o);
            if (oj < hj || (oj == hj && (ot < L.best || (ot == L.best && (uint32_t)oid < (uint32_t)L.id)))) {
                hj = oj;
                L.best = ot;
                L.id = oid;
            }
        }
    }
    // the last shuffles of the batch: the groups part ways below
    const int32_t hit_tests = __shfl_sync(FULL, incl, hj & (G - 1), G);
    GroupOut r;
    r.cell = __shfl_sync(FULL, c, fh & (G - 1), G);
    r.len = __shfl_sync(FULL, n, fh & (G - 1), G);
    r.lane = fh;
    r.tests = limit;
    if (hj < G) {
        r.step = GROUP_DONE;
        r.cells = hj + 1;
        r.tests = hit_tests;
        if (any && !(L.best < L.tmax)) L.id = -1;   // any-hit: the first cell with a hit decides
    } else if (fh < G) {
        r.step = GROUP_LIST;
        r.cells = fh;
    } else if (om) {
        r.step = GROUP_DONE;
        r.cells = __ffs(om) - 1;
        L.id = -1;
    } else {
        r.step = GROUP_ON;
        r.cells = G;
    }
    r.cells -= skip + 1;
    return r;
}

// A lane without a ray, defined so that the warp can step it idly.
__device__ __forceinline__ Lane idle_lane() {
    Lane L;
    L.ox = L.oy = L.oz = L.dx = L.dy = L.dz = 0.0f;
    L.tMx = L.tMy = L.tMz = L.tDx = L.tDy = L.tDz = 0.0f;
    L.x = L.y = L.z = 0;
    L.budget = 0;
    L.tmax = L.lo = 0.0f;
    L.best = kFltMax;
    L.id = -1;
    L.ray = 0;
    return L;
}

// The next rays for a warp's idle groups: `want` of them claimed with one
// atomicAdd on *counter, handed out in group order.  Sets `exhausted` once the
// claims pass `total`.
template <int G>
__device__ __forceinline__ unsigned long long claim_groups(unsigned idle, unsigned long long* counter,
                                                           unsigned long long total, bool& exhausted) {
    const int lane = threadIdx.x & 31;
    const unsigned want = (unsigned)__popc(idle) / G;
    unsigned long long r = 0;
    if (lane == 0) r = atomicAdd(counter, (unsigned long long)want);
    r = __shfl_sync(FULL, r, 0);
    if (r + want >= total) exhausted = true;
    return r + (unsigned)__popc(idle & ((1u << (lane & ~(G - 1))) - 1u)) / G;
}

// Eight blocks of 128 threads per SM: six (80 registers) made the group walk
// of 4 M random rays 9% slower.
#ifndef GRIDRT_GROUP_MIN_BLOCKS
#define GRIDRT_GROUP_MIN_BLOCKS 8
#endif

// QUEUE: the rays another pass deferred, from the cell it stopped at; else the
// launch's rays from their start.  Idle groups take new rays once half of the
// warp's groups are idle.  A ray that comes to a long list is handed on, while
// there is room, to the pass that resumes it there (and counts that cell): from
// the start (io.defer set) lists above io.heavy to the deferred pass, else
// lists above kHugeList to the block-per-ray pass.
template <int MODE, bool COUNT, int G, bool QUEUE>
__global__ void __launch_bounds__(128, GRIDRT_GROUP_MIN_BLOCKS) trace_group_kernel(SceneView s, TraceIO io) {
    pdl_begin();
    __shared__ SParams P;
    load_sparams(s.params, P);
    const int gl = threadIdx.x & (G - 1);
    constexpr int kWant = G < 32 ? 16 / G : 1;
    unsigned long long total = (unsigned long long)io.n;
    if (QUEUE) {
        total = io.counter[1];
        if (total > (unsigned long long)io.defer_cap) total = (unsigned long long)io.defer_cap;
    }
    const bool to_defer = !QUEUE && io.defer;
    const int32_t thr0 = to_defer ? io.heavy : (io.huge ? kHugeList : kNoHeavy);
    uint32_t cells = 0, tests = 0, started = 0;
    bool busy = false, exhausted = false;
    int todo = 0;
    int32_t thr = thr0;
    int3 sg = make_int3(0, 0, 0);
    Lane L = idle_lane();
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !busy);
        if (!exhausted && __popc(idle) >= kWant * G) {
            const unsigned long long r = claim_groups<G>(idle, io.counter + (QUEUE ? 2 : 0), total, exhausted);
            if (!busy && r < total) {
                const int2 d = QUEUE ? __ldg(io.defer + r) : make_int2((int32_t)r, -1);
                const bool shadow = MODE == MODE_FRAME && d.x < 0;   // a frame's shadow ray (its slot holds it)
                L.ray = shadow ? -1 - d.x : d.x;
                busy = shadow ? start_ray<MODE_ANY>(P, io, L, L.ray) : start_ray<MODE>(P, io, L, L.ray);
                if (!QUEUE && gl == 0) ++started;
                if (busy) {
                    if (QUEUE) resume_at(P, L, d.y);
                } else {
                    if (L.id != -2) L.id = -1;
                    busy = finish_ray<MODE>(io, P, s, L, gl == 0);
                }
                todo = gl;
                thr = thr0;
                sg = step_signs(L);
            }
        }
        if (!__any_sync(FULL, busy)) {
            if (exhausted) break;
            continue;
        }
        const bool any = any_hit_phase<MODE>(L);
        GroupOut r = group_batch<G>(P, s, L, sg, busy, any, busy ? todo : 0, thr);
        todo = G;
        const bool hand = busy && r.step == GROUP_LIST;
        if (__any_sync(FULL, hand)) {
            unsigned long long at = 0;
            if (hand && gl == 0) at = atomicAdd(io.counter + (to_defer ? 1 : 3), 1ull);
            at = __shfl_sync(FULL, at, 0, G);
            if (hand && at < (unsigned long long)(to_defer ? io.defer_cap : io.huge_cap)) {
                if (to_defer) {
                    if (gl == 0) io.defer[at] = make_int2(defer_tag<MODE>(L, io), r.cell);
                } else if (gl == 0) {
                    // longest first: lists of kHugeLong+ entries fill the
                    // queue from its back (counter word 5 of them), the rest
                    // from its front (word 6); together they number the
                    // reservations that fit, so the two never meet
                    const bool longl = r.len >= kHugeLong;
                    const unsigned long long pos = atomicAdd(io.counter + (longl ? 5 : 6), 1ull);
                    io.huge[longl ? (unsigned long long)io.huge_cap - 1 - pos : pos] =
                        make_int2(defer_tag<MODE>(L, io), r.cell);
                }
                busy = false;
            } else if (hand) {
                thr = kNoHeavy;   // the queue is full: the group visits its cells again and tests the list
                todo = 0;
                r.cells = r.tests = 0;
            }
        }
        if (COUNT && gl == 0 && (busy || hand)) {
            cells += (uint32_t)r.cells;
            tests += (uint32_t)r.tests;
        }
        if (busy && r.step == GROUP_DONE) {
            // a camera ray's group goes on with its hit's shadow ray: every
            // lane sets it up from the hit (one writes the results)
            busy = finish_ray<MODE>(io, P, s, L, gl == 0);
            todo = gl;
            thr = thr0;
            sg = step_signs(L);
        }
    }
    if (COUNT) flush_counters(io.ctr, started, cells, tests);
}

// Block-per-ray pass over the rays the group pass met at a list above
// kHugeList (a dense cluster: tens of thousands of triangles in one cell).  The
// block's first warp walks the ray as the group pass does; each long list is
// split over the block (thread j tests entries j, j + blockDim, ...), each
// thread keeping the first minimum of its share, and a block reduction takes
// the minimum t, ties to the earlier entry -- the one-lane walk's result, as
// in the group pass.  Bound by the longest rays, one block each (several
// hundred thousand entries), and by their walks between crowded cells.  Lists
// above kSplitRefs are read as 16-byte bounding spheres: 1,048,576 triangles of
// skewed density, the passes behind 1024^2 camera rays and their secondaries
// 420 and 489 -> 240..290 and 270 us, the spheres 25 us of the build's sort.
#ifndef GRIDRT_HUGE_THREADS
#define GRIDRT_HUGE_THREADS 256
#endif
static constexpr int kHugeThreads = GRIDRT_HUGE_THREADS;
#ifndef GRIDRT_HUGE_MIN_BLOCKS
#define GRIDRT_HUGE_MIN_BLOCKS 3
#endif
static_assert(kHugeThreads % 32 == 0 && kHugeThreads <= 1024, "block-per-ray pass: whole warps, one block");

// Crowded lists staged in shared memory.  With cell-ordered records a list
// is one contiguous run of 48-byte records, so the bulk-copy engine
// (cp.async.bulk, completion counted on an mbarrier per buffer) copies it
// into a ring of kStageDepth shared-memory buffers of kStageEntries records:
// while the block tests one chunk the next kStageDepth - 1 are in flight,
// and no thread waits on its own global loads.  A chunk costs a block
// barrier and a wait, so chunks are large: 768 records (36 KB), two
// buffers, 72 KB a block and three blocks an SM (smaller chunks or deeper
// rings measured slower).  Lists shorter than kStageMin keep the direct
// loads.  Every wait is bounded: a copy that has not landed after
// kStageWaitLimit polls sets bit 0 of the launch's counter word 7, the rest
// of the list is tested from global memory and the block stops staging.
#ifndef GRIDRT_STAGE
#define GRIDRT_STAGE 1
#endif
#ifndef GRIDRT_STAGE_ENTRIES
#define GRIDRT_STAGE_ENTRIES 768
#endif
#ifndef GRIDRT_STAGE_DEPTH
#define GRIDRT_STAGE_DEPTH 2
#endif
static constexpr int kStageEntries = GRIDRT_STAGE_ENTRIES;
static constexpr int kStageDepth = GRIDRT_STAGE_DEPTH;
static constexpr size_t kStageBytes = GRIDRT_STAGE ? (size_t)kStageDepth * 3 * kStageEntries * sizeof(float4) : 0;
static_assert(kStageDepth >= 2 && kStageDepth <= 16, "stage ring depth");
static constexpr int32_t kStageMin = 2 * kHugeThreads;
static constexpr uint32_t kStageWaitLimit = 1u << 24;
static_assert(kStageEntries % kHugeThreads == 0 || kHugeThreads % kStageEntries == 0, "stage chunk");

static constexpr int kCand = 512;
struct Stage {
    float4* buf;          // shared: kStageDepth x kStageEntries x 3 float4
    uint64_t* bar;        // shared: one mbarrier per buffer
    int* off;             // shared: 1 once a wait has run out
    int32_t* cand;        // shared: candidates of a list's spheres, kCand at most
    int* cand_n;          // shared: how many there were
    const float4* spheres;   // of the lists above kSplitRefs (GridParams::spheres), or nullptr
    uint32_t phase;       // bit q: the parity of buffer q's next completion
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Thread 0: buffer `dst` <- `bytes` of global memory at `src`, completion
// on `bar` (which expects those bytes and thread 0's arrival).
__device__ __forceinline__ void stage_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Bounded wait for the completion of `bar`'s phase of parity `parity`.
__device__ __forceinline__ bool stage_wait(uint64_t* bar, uint32_t parity) {
    for (uint32_t it = 0; it < kStageWaitLimit; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Whether the ray's line meets a list entry's bounding sphere (build.cu
// hit_sphere; `grow`: 256u (|origin|_1 + 2 |x|_1) of the ray and the cell, dd:
// |d|^2 and a margin).  19 instructions on 16 bytes: nearly all of a dense
// cluster's triangles end here.
__device__ __forceinline__ bool near_sphere(const Lane& L, const float4& q, float grow, float dd) {
    const float2 rw = __half22float2(*reinterpret_cast<const __half2*>(&q.w));
    const float r = rw.x + rw.y * grow;
    const float x = q.x - L.ox, y = q.y - L.oy, z = q.z - L.oz;
    const float cx = y * L.dz - z * L.dy, cy = z * L.dx - x * L.dz, cz = x * L.dy - y * L.dx;
    return !(cx * cx + cy * cy + cz * cz > r * r * dd);
}

// The largest |x|_1 in a cell (and a margin).
__device__ __forceinline__ float cell_l1(const SParams& P, int32_t cell) {
    float m = 0.0f;
    const int32_t nxy = P.res[0] * P.res[1], z = cell / nxy, y = (cell - z * nxy) / P.res[0];
    const int32_t c[3] = {cell - z * nxy - y * P.res[0], y, z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float lo = P.bmin[a] + P.cell[a] * (float)(c[a] - 1), hi = P.bmin[a] + P.cell[a] * (float)(c[a] + 2);
        m += fmaxf(fabsf(lo), fabsf(hi));
    }
    return m;
}

// The next larger float (of a finite distance).
__device__ __forceinline__ float float_above(float x) {
    const int32_t i = __float_as_int(x);
    return x == 0.0f ? __int_as_float(1) : __int_as_float(x > 0.0f ? i + 1 : i - 1);
}

// List entry i from global memory, in any order within the thread's share: of
// two equal distances the smaller id stays.
__device__ __forceinline__ void test_listed(Lane& T, const SceneView& s, int32_t i, float hi) {
    const int32_t t = __ldg(s.ids + i);
    const float4* __restrict__ r = s.crec ? s.crec + 3 * (int64_t)i : s.tris + 3 * (int64_t)t;
    const float best = T.best;
    const int32_t id = T.id;
    if (id >= 0) T.best = float_above(best);
    test_tri<MODE_NEAREST>(T, t, __ldg(r), __ldg(r + 1), __ldg(r + 2), hi, s.wald);
    if (id >= 0 && (T.id == id || (T.best == best && t > id))) {
        T.best = best;
        T.id = id;
    }
}

// What the block's first warp found next along the ray, for its other threads.
struct BlockStep {
    int32_t step, cell, id;
    float best, hi;
};
// Lists longer than this are tested by the whole block.
static constexpr int32_t kBlockList = kHugeThreads;

// The block's ray walked to its end (the same ray on every thread).  The first
// warp walks it 32 cells at a time (group_batch) up to the next list above
// kBlockList; that list is split over the block.  Block-wide steps cell by cell
// made the rays' walks between crowded cells, each with its own barriers and
// chain of loads, the pass's time.
__device__ __forceinline__ void block_walk(const SParams& P, const SceneView& s, Lane& L, bool done, bool any,
                                           uint32_t& cells, uint32_t& tests, float* red_t, int32_t* red_id,
                                           BlockStep* bs, Stage* st = nullptr, unsigned long long* err = nullptr) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (done) return;
    const float o1 = fabsf(L.ox) + fabsf(L.oy) + fabsf(L.oz);
    const float dd = 1.0001f * (L.dx * L.dx + L.dy * L.dy + L.dz * L.dz);
    const int3 sg = step_signs(L);
    int todo = lane, skip = -1;
    for (;;) {
        if (wid == 0) {
            GroupOut r;
            for (;;) {
                r = group_batch<32>(P, s, L, sg, true, any, todo, kBlockList, skip);
                if (lane == 0) {
                    cells += (uint32_t)r.cells;
                    tests += (uint32_t)r.tests;
                }
                if (r.step != GROUP_ON) break;
                todo = 32;
                skip = -1;
            }
            const float hi = __shfl_sync(FULL, fadd(vmin(vmin(L.tMx, L.tMy), L.tMz), kHitEpsilon), r.lane & 31);
            if (lane == 0) *bs = BlockStep{r.step, r.cell, L.id, L.best, hi};
            todo = 0;         // go on from the cells the lanes stand on, behind this list's
            skip = r.lane;
        }
        __syncthreads();
        if (bs->step == GROUP_DONE) {
            L.id = bs->id;
            L.best = bs->best;
            __syncthreads();
            return;
        }
        {
            const int32_t c = bs->cell;
            const int32_t b = __ldg(s.offsets + c), e = __ldg(s.offsets + c + 1);
            const float hi = bs->hi;
            if (threadIdx.x == 0) {
                ++cells;
                tests += (uint32_t)(e - b);
            }
            Lane T = L;
            T.id = -1;
            // a crowded list's entries by their bounding spheres first, when
            // the scene has them: the candidates (one in 3,000 in a dense
            // cluster) are queued in shared memory and tested together behind
            // the list's last chunk -- a warp that tested its own at once
            // waited for their loads at every step
            const bool sph = st && st->spheres && e - b > kSplitRefs;
            // (directions below 1e-10, whose squared distances round to too few
            // bits, meet every sphere)
            const float grow = !sph ? 0.0f : (dd >= 1e-20f ? 256.0f * kRound * (o1 + 2.0f * cell_l1(P, c)) : INFINITY);
            if (GRIDRT_STAGE && st && (sph || (s.crec && e - b >= kStageMin)) && !*st->off) {
                // staged: chunk ch in buffer ch % kStageDepth, the next
                // kStageDepth - 1 chunks in flight
                const float4* __restrict__ src = sph ? st->spheres : s.crec;
                const int32_t quads = sph ? 1 : 3, per = sph ? 3 * kStageEntries : kStageEntries;
                const int32_t nch = (e - b + per - 1) / per;
                if (sph) {
                    if (threadIdx.x == 0) *st->cand_n = 0;
                    __syncthreads();
                }
                if (threadIdx.x == 0) {
                    for (int32_t ch = 0; ch < nch && ch < kStageDepth; ++ch) {
                        const int32_t cb = b + ch * per;
                        const int32_t cn = e - cb < per ? e - cb : per;
                        stage_copy(st->buf + ch * 3 * kStageEntries, src + quads * (int64_t)cb,
                                   (uint32_t)(cn * quads) * 16u, st->bar + ch);
                    }
                }
                for (int32_t ch = 0; ch < nch; ++ch) {
                    const int q = ch % kStageDepth;
                    const int32_t cb = b + ch * per;
                    const int32_t cn = e - cb < per ? e - cb : per;
                    const bool ok = stage_wait(st->bar + q, (st->phase >> q) & 1u);
                    st->phase ^= 1u << q;
                    if (ok) {
                        const float4* sb = st->buf + q * 3 * kStageEntries;
                        if (sph) {
#pragma unroll 3
                            for (int32_t j = (int32_t)threadIdx.x; j < cn; j += kHugeThreads)
                                if (near_sphere(L, sb[j], grow, dd)) {
                                    const int at = atomicAdd(st->cand_n, 1);
                                    if (at < kCand) st->cand[at] = cb + j;
                                    else test_listed(T, s, cb + j, hi);
                                }
                        } else {
                            for (int32_t j = (int32_t)threadIdx.x; j < cn; j += kHugeThreads) {
                                const float4 A = sb[3 * j], B = sb[3 * j + 1], C = sb[3 * j + 2];
                                test_tri<MODE_NEAREST>(T, __float_as_int(A.w), A, B, C, hi, s.wald);
                            }
                        }
                    }
                    // every thread is done with buffer q before chunk
                    // ch + kStageDepth is copied into it
                    if (__syncthreads_or(!ok)) {
                        // a copy has not landed: wait once more (bounded) for
                        // it and the copies in flight behind it, test the rest
                        // of the list from global memory, stop staging
                        if (!ok) stage_wait(st->bar + q, ((st->phase >> q) & 1u) ^ 1u);
                        for (int32_t k = ch + 1; k < nch && k < ch + kStageDepth; ++k) {
                            const int qk = k % kStageDepth;
                            stage_wait(st->bar + qk, (st->phase >> qk) & 1u);
                        }
                        if (threadIdx.x == 0) {
                            *st->off = 1;
                            if (err) atomicOr(err, 1ull);
                        }
                        for (int32_t i = (ok ? cb + cn : cb) + (int32_t)threadIdx.x; i < e; i += kHugeThreads)
                            test_listed(T, s, i, hi);
                        __syncthreads();
                        break;
                    }
                    if (threadIdx.x == 0 && ch + kStageDepth < nch) {
                        const int32_t nb = cb + kStageDepth * per;
                        const int32_t nn = e - nb < per ? e - nb : per;
                        stage_copy(st->buf + q * 3 * kStageEntries, src + quads * (int64_t)nb,
                                   (uint32_t)(nn * quads) * 16u, st->bar + q);
                    }
                }
                if (sph) {
                    // (every chunk ended with a barrier)
                    const int nc = min(*st->cand_n, kCand);
                    for (int k = (int)threadIdx.x; k < nc; k += kHugeThreads) test_listed(T, s, st->cand[k], hi);
                }
            } else if (s.crec) {
                // two entries a thread per step, both loaded before either is
                // tested (the same entries in the same order as one a step)
                for (int32_t i = b + (int32_t)threadIdx.x; i < e; i += 2 * kHugeThreads) {
                    const int32_t i2 = i + kHugeThreads;
                    const float4 A = __ldg(s.crec + 3 * (int64_t)i), B = __ldg(s.crec + 3 * (int64_t)i + 1),
                                 C = __ldg(s.crec + 3 * (int64_t)i + 2);
                    float4 A2 = A, B2 = B, C2 = C;
                    if (i2 < e) {
                        A2 = __ldg(s.crec + 3 * (int64_t)i2);
                        B2 = __ldg(s.crec + 3 * (int64_t)i2 + 1);
                        C2 = __ldg(s.crec + 3 * (int64_t)i2 + 2);
                    }
                    test_tri<MODE_NEAREST>(T, __float_as_int(A.w), A, B, C, hi, s.wald);
                    if (i2 < e) test_tri<MODE_NEAREST>(T, __float_as_int(A2.w), A2, B2, C2, hi, s.wald);
                }
            } else {
                for (int32_t i = b + (int32_t)threadIdx.x; i < e; i += 2 * kHugeThreads) {
                    const int32_t i2 = i + kHugeThreads;
                    const int32_t t = __ldg(s.ids + i), t2 = i2 < e ? __ldg(s.ids + i2) : t;
                    const float4 A = __ldg(s.tris + 3 * (int64_t)t), B = __ldg(s.tris + 3 * (int64_t)t + 1),
                                 C = __ldg(s.tris + 3 * (int64_t)t + 2);
                    const float4 A2 = __ldg(s.tris + 3 * (int64_t)t2), B2 = __ldg(s.tris + 3 * (int64_t)t2 + 1),
                                 C2 = __ldg(s.tris + 3 * (int64_t)t2 + 2);
                    test_tri<MODE_NEAREST>(T, t, A, B, C, hi, s.wald);
                    if (i2 < e) test_tri<MODE_NEAREST>(T, t2, A2, B2, C2, hi, s.wald);
                }
            }
            // ids ascend along a list: the smaller id is the earlier entry
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ot = __shfl_xor_sync(FULL, T.best, o);
                const int32_t oid = __shfl_xor_sync(FULL, T.id, o);
                if (ot < T.best || (ot == T.best && (uint32_t)oid < (uint32_t)T.id)) {
                    T.best = ot;
                    T.id = oid;
                }
            }
            if (lane == 0) {
                red_t[wid] = T.best;
                red_id[wid] = T.id;
            }
            __syncthreads();
            float bt = red_t[0];
            int32_t bid = red_id[0];
            for (int i = 1; i < kHugeThreads / 32; ++i)
                if (red_t[i] < bt || (red_t[i] == bt && (uint32_t)red_id[i] < (uint32_t)bid)) {
                    bt = red_t[i];
                    bid = red_id[i];
                }
            __syncthreads();
            if (bid >= 0) {
                // the first cell with a hit ends the walk; any-hit:
                // occluded only below tmax
                L.best = bt;
                L.id = (any && !(bt < L.tmax)) ? -1 : bid;
                return;
            }
        }
    }
}

template <int MODE, bool COUNT>
__global__ void __launch_bounds__(kHugeThreads, GRIDRT_HUGE_MIN_BLOCKS) trace_huge_kernel(SceneView s, TraceIO io) {
    pdl_begin();
    __shared__ SParams P;
    __shared__ float red_t[kHugeThreads / 32];
    __shared__ int32_t red_id[kHugeThreads / 32];
    __shared__ unsigned long long claim;
    extern __shared__ __align__(128) float4 stage_buf[];   // kStageBytes (dynamic)
    __shared__ __align__(8) uint64_t stage_bar[kStageDepth];
    __shared__ int stage_off;
    __shared__ int32_t cand[kCand];
    __shared__ int cand_n;
    __shared__ BlockStep step;
    if (threadIdx.x == 0) {
        for (int q = 0; q < kStageDepth; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(stage_bar + q)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        stage_off = 0;
    }
    Stage stage{stage_buf, stage_bar, &stage_off, cand, &cand_n, s.params->spheres, 0u};
    load_sparams(s.params, P);
    unsigned long long nh = io.counter[3];
    if (nh > (unsigned long long)io.huge_cap) nh = (unsigned long long)io.huge_cap;
    // the rays at the longest lists (the queue's back) are claimed first, so
    // they do not start last and run on alone at the end of the pass
    const unsigned long long nb = io.counter[5];
    uint32_t cells = 0, tests = 0;
    for (;;) {
        if (threadIdx.x == 0) claim = atomicAdd(io.counter + 4, 1ull);
        __syncthreads();
        const unsigned long long j = claim;
        __syncthreads();
        if (j >= nh) break;
        const int2 d = __ldg(io.huge + (j < nb ? (unsigned long long)io.huge_cap - 1 - j : j - nb));
        const bool shadow = MODE == MODE_FRAME && d.x < 0;   // MODE_FRAME: a shadow ray (in its slot)
        Lane L;
        L.ray = shadow ? -1 - d.x : d.x;
        // the same on every thread
        bool done = shadow ? !start_ray<MODE_ANY>(P, io, L, L.ray) : !start_ray<MODE>(P, io, L, L.ray);
        if (done) {
            if (L.id != -2) L.id = -1;
        } else {
            resume_at(P, L, d.y);
        }
        // one walk, or for a MODE_FRAME camera ray two: its own, then from
        // its start the shadow ray every thread sets up from the hit
        for (int phase = 0; phase < 2; ++phase) {
            block_walk(P, s, L, done, any_hit_phase<MODE>(L), cells, tests,
                       red_t, red_id, &step, &stage, io.counter + 7);
            if (!finish_ray<MODE>(io, P, s, L, threadIdx.x == 0)) break;
            done = false;
        }
    }
    if (COUNT) {
        if (threadIdx.x != 0) cells = tests = 0;
        flush_counters(io.ctr, 0, cells, tests);
    }
}

// Blocks of TPB threads (the RTG_TUNE_BLOCK choice; counter launches use
// 128).  Persistent: as many blocks as fit on the device at once, warps loop
// over ray batches.  One-shot: one batch per warp, blocks scheduled by the
// hardware.
template <int MODE, bool COUNT, int ER, int TPB>
inline void launch_tpb(const SceneView& s, const TraceIO& io, const TraceTuning& tune, int num_sms, cudaStream_t st) {
    static int per_sm = 0;
    if (per_sm == 0) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, trace_kernel<MODE, COUNT, ER, TPB>, TPB, 0);
        per_sm = b > 0 ? b : 1;
    }
    long long blocks = (io.n + TPB - 1) / TPB;
    if (tune.persistent) blocks = blocks < (long long)per_sm * num_sms ? blocks : (long long)per_sm * num_sms;
    if (blocks < 1) blocks = 1;
    if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
    launch_k(trace_kernel<MODE, COUNT, ER, TPB>, (unsigned)blocks, TPB, 0, st, s, io);
}

template <int MODE, bool COUNT, int ER>
inline void launch_er(const SceneView& s, const TraceIO& io, const TraceTuning& tune, int num_sms, cudaStream_t st) {
    if (COUNT || tune.block == 128) launch_tpb<MODE, COUNT, ER, 128>(s, io, tune, num_sms, st);
    else if (tune.block == 64) launch_tpb<MODE, COUNT, ER, COUNT ? 128 : 64>(s, io, tune, num_sms, st);
    else launch_tpb<MODE, COUNT, ER, COUNT ? 128 : 256>(s, io, tune, num_sms, st);
}

template <int MODE, bool COUNT>
inline void launch_count(const SceneView& s, const TraceIO& io, const TraceTuning& tune, int num_sms,
                         cudaStream_t st) {
    if (tune.empty_run <= 2) launch_er<MODE, COUNT, 2>(s, io, tune, num_sms, st);
    else if (tune.empty_run <= 4) launch_er<MODE, COUNT, 4>(s, io, tune, num_sms, st);
    else if (tune.empty_run <= 8) launch_er<MODE, COUNT, 8>(s, io, tune, num_sms, st);
    else launch_er<MODE, COUNT, 16>(s, io, tune, num_sms, st);
}

// The group pass: as many blocks as fit on the device, or as the launch's rays
// need.
template <int MODE, bool COUNT, int G, bool QUEUE>
inline void launch_group(const SceneView& s, const TraceIO& io, int num_sms, cudaStream_t st) {
    static int per_sm = 0;
    if (per_sm == 0) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, trace_group_kernel<MODE, COUNT, G, QUEUE>, 128, 0);
        per_sm = b > 0 ? b : 1;
    }
    const long long full = (long long)per_sm * num_sms, need = (io.n + 128 / G - 1) / (128 / G);
    launch_k(trace_group_kernel<MODE, COUNT, G, QUEUE>, (unsigned)(need < full ? need : full), 128, 0, st, s, io);
}

template <int MODE, bool COUNT>
inline void launch_deferred(const SceneView& s, const TraceIO& io, const TraceTuning& tune, int num_sms,
                            cudaStream_t st) {
    if (tune.heavy_lanes <= 4) launch_group<MODE, COUNT, 4, true>(s, io, num_sms, st);
    else if (tune.heavy_lanes <= 8) launch_group<MODE, COUNT, 8, true>(s, io, num_sms, st);
    else if (tune.heavy_lanes <= 16) launch_group<MODE, COUNT, 16, true>(s, io, num_sms, st);
    else launch_group<MODE, COUNT, 32, true>(s, io, num_sms, st);
}

// As many blocks as fit on the GPU claim the queued rays: each ray's lists
// are long latency chains, so the pass runs as many rays side by side as it
// can hold.
template <int MODE, bool COUNT>
inline void launch_huge(const SceneView& s, const TraceIO& io, int num_sms, cudaStream_t st) {
    static int per_sm = 0;
    if (per_sm == 0) {
        // the staging ring is dynamic shared memory (above the 48 KB of a
        // static allocation for deep rings)
        cudaFuncSetAttribute(trace_huge_kernel<MODE, COUNT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kStageBytes);
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, trace_huge_kernel<MODE, COUNT>, kHugeThreads, kStageBytes);
        per_sm = b > 0 ? b : 1;
    }
    launch_k(trace_huge_kernel<MODE, COUNT>, (unsigned)(per_sm * num_sms), kHugeThreads, kStageBytes, st, s, io);
}

// The eighths of a chunk's rays that must be like the ray before them for the
// chunk to walk by whole lists: half in launches of a few chunks a warp, which
// end with their longest rays, 7 beyond.  Shadow rays of 512^2 images given as
// an array, us at 7 and at 4: plane and debris of 2,000 triangles 52 and 46, of
// 5,000 70 and 58; of 1024^2 images: 100,000 triangles 227 and 258.
inline int32_t alike_eighths(long long n, int sms) { return n <= 2048LL * sms ? 4 : 7; }

// Whether rays through the scene make some 256 tests and more (references a cell,
// over half the cells along the axes: a soup of triangles as large as its box's
// cells makes 1,500, plane and debris of 100,000 triangles 110 to 160).  Not those
// whose references lie in a few crowded cells (a step of the skewed scene would
// take 1,676 us for 1,646).
inline bool dense_scene(const GridParams* g) {
    return g && g->ncells > 0 && g->max_list <= (uint32_t)kHugeList &&
           0.5 * (double)g->nrefs * ((double)g->res[0] + g->res[1] + g->res[2]) > 256.0 * (double)g->ncells;
}

// The tests after which a ray (a frame's with its shadow ray) is handed to a group
// of lanes, in heavy-cell thresholds: the fewer the shorter the tail of a launch,
// but its queue is fixed, so larger launches hand on fewer of their rays.
// Frames of the sphere / of plane and debris, us at 8 -> here: 518,400 pixels
// 166 -> 133 / 398 -> 367 (4), 1,048,576 207 -> 186 / 526 -> 530 (5).  Arrays come
// to 8 at four times the resident lanes (4 M random rays 2,254 us, at 4 2,321);
// 262,144 random rays in plane and debris of 2,000 / 65,536 triangles 132 -> 114 /
// 299 -> 284, segments 166 -> 146 / 369 -> 352 (4).
// Camera and frame launches stay at 8 in dense scenes, where every ray is one of
// those: 640 x 640 camera rays / frames of a soup of 20,000 triangles 206 -> 186 /
// 392 -> 329, of 5,000 800 x 800 192 / 400 -> 291.
inline int32_t work_mult(long long n, int sms, bool camera, const GridParams* grid) {
    if (camera && dense_scene(grid)) return kHeavyWorkMult;
    const long long m = camera ? 2 + n / (2048LL * sms) : 2 * n / (1024LL * sms);
    return (int32_t)(m < 4 ? 4 : (m > kHeavyWorkMult ? kHeavyWorkMult : m));
}

// Lanes per ray of a camera or frame launch that lanes_for gives 8.  Beyond the
// resident lanes that pays while enough of the rays miss the scene's box or walk
// far in it.  A small mesh that fills the image does better by one ray a lane as
// soon as more rays than the resident lanes can meet its box, the smallest ones
// (walks of a few cells) at four fifths; their camera launches, which end with
// the hit, by 6/4 and 5/4 of the lanes at the latest.  us at 8 lanes and at one,
// frames: 229 x 915, the sphere filling the image, 2,352 triangles 97 and 87,
// 9,312 130 and 109; 256 x 1,024, 25,760 triangles 197 and 134; 260 x 1,040,
// plane and debris of 2,000 triangles 111 and 98, of 20,000 (127,000 rays at the
// box) 178 and 238; 200 x 800 (105,000 at the sphere's) 81 and 86.  Camera
// launches, plane and debris of 2,000 triangles: 224 x 896 69 and 65, 256 x 1,024
// 87 and 69; of 5,000: 224 x 896 76 and 79, 256 x 1,024 95 and 81.  In dense
// scenes a lane a ray keeps the GPU busy beyond the resident lanes: 512 x 512
// frames of soups of 20,000 / 60,000 triangles 273 and 238 / 431 and 393, of
// 440 x 440 pixels 215 and 206 / 333 and 318.
static constexpr int64_t kFewTris = 32768, kFewestTris = 4096;
inline int image_lanes(const TraceIO& io, const TraceSlot& slot, bool frame, int num_sms) {
    const long long resident = 1024LL * num_sms;
    if (io.n > resident && dense_scene(slot.grid)) return 1;
    if (!slot.grid || slot.grid->ntris > kFewTris) return 8;
    const bool fewest = slot.grid->ntris <= kFewestTris;
    if (!frame && 4 * io.n > (fewest ? 5 : 6) * resident) return 1;
    const double meet = (double)io.n * image_share(io.cam, slot.grid->bmin, slot.grid->bmax);
    return meet > (fewest ? 0.8 : 1.0) * (double)resident ? 1 : 8;
}

template <int MODE>
inline void launch_mode(const SceneView& s, TraceIO io, const TraceSlot& slot, const TraceTuning& tune, int num_sms,
                        cudaStream_t st) {
    const bool defer = tune.heavy_cell > 0 && slot.defer && slot.defer_cap > 0;
    io.counter = slot.ctr;
    io.defer = defer ? slot.defer : nullptr;
    io.defer_cap = defer ? slot.defer_cap : 0;
    io.heavy = defer ? tune.heavy_cell : kNoHeavy;
    constexpr int camera = MODE == MODE_CAMERA || MODE == MODE_FRAME;
    io.refill = refill_for(tune, camera);
    io.huge = defer ? slot.huge : nullptr;
    io.huge_cap = io.huge ? slot.huge_cap : 0;
    cudaMemsetAsync(slot.ctr, 0, 8 * sizeof(unsigned long long), st);
    io.alike = alike_eighths(io.n, num_sms);
    io.work = work_limit(io.heavy, kHeavyWorkMult);
    if (io.heavy != kNoHeavy) {   // below 128 tests only where the caller's threshold says so
        const int32_t few = io.work < 128 ? io.work : 128, less = work_limit(io.heavy, work_mult(io.n, num_sms, camera, slot.grid));
        io.work = less > few ? less : few;
    }
    int lanes = io.ctr ? 1 : (tune.lanes ? tune.lanes : lanes_for(io.n, num_sms, camera ? 7 : MODE == MODE_ANY ? 3 : 4));
    if (camera && lanes == 8 && io.n > 1024LL * num_sms / 2) lanes = image_lanes(io, slot, MODE == MODE_FRAME, num_sms);
    if (lanes > 1) {
        // every ray walked by a group of lanes from its start.  Groups of 16
        // and 32 deal any list out themselves, as do groups of 8 when no list
        // of the scene would take them more than heavy_cell / 2 turns.  Where
        // there are longer ones, 8 lanes hand on the lists above heavy_cell,
        // as one lane does; 2 and 4 lanes (set by the caller) those of more
        // than heavy_cell / 2 turns.  A 512^2 frame of the sphere with crowded
        // poles (102,720 triangles, k = 4), 8 lanes: 198 us with several frames
        // in flight and 261 alone; handing on above heavy_cell * 4, 233 and
        // 296; one lane a ray, 215 and 281.
        const bool known = io.heavy < kNoHeavy / 64;
        const int32_t deal = known ? io.heavy * lanes / 2 : io.heavy;
        if (lanes >= 16 || (!tune.lanes && slot.longest <= deal)) {
            io.defer = nullptr;
            io.defer_cap = 0;
        }
        if (tune.lanes) io.heavy = deal;
    }
    count_launches(1 + (io.defer ? 1 : 0) + (io.huge ? 1 : 0));
    switch (lanes) {
        case 2: launch_group<MODE, false, 2, false>(s, io, num_sms, st); break;
        case 4: launch_group<MODE, false, 4, false>(s, io, num_sms, st); break;
        case 8: launch_group<MODE, false, 8, false>(s, io, num_sms, st); break;
        case 16: launch_group<MODE, false, 16, false>(s, io, num_sms, st); break;
        case 32: launch_group<MODE, false, 32, false>(s, io, num_sms, st); break;
        default:
            if (io.ctr) launch_count<MODE, true>(s, io, tune, num_sms, st);
            else launch_count<MODE, false>(s, io, tune, num_sms, st);
    }
    if (io.defer) {
        if (io.ctr) launch_deferred<MODE, true>(s, io, tune, num_sms, st);
        else launch_deferred<MODE, false>(s, io, tune, num_sms, st);
    }
    if (io.huge) {
        if (io.ctr) launch_huge<MODE, true>(s, io, num_sms, st);
        else launch_huge<MODE, false>(s, io, num_sms, st);
    }
}

}  // namespace gridrt
