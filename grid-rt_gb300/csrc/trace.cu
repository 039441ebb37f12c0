// trace.cu -- launch counting, the batched tracer (many scenes, one persistent
// launch), two-level instancing and the device-side mesh deformation.
// The single-scene kernels are in trace_device.cuh and trace_{nearest,any,
// camera,frame}.cu.
#include "trace_device.cuh"

namespace gridrt {

static unsigned long long g_launches = 0;
void count_launches(int n) { __atomic_add_fetch(&g_launches, (unsigned long long)n, __ATOMIC_RELAXED); }
unsigned long long launches_so_far() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

// Task t owning flattened ray index f: the last task with first <= f.
__device__ __forceinline__ int find_task(const BatchTask* __restrict__ tasks, int ntasks, long long f) {
    int lo = 0, hi = ntasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].first <= f) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Lane refill inside one batch task: the warp draws 32-ray chunks from the
// flattened counter and hands their rays to idle lanes while the chunks belong
// to its task, so scene and mode stay warp-uniform; starts on the task's chunk
// at `base`, and returns the first chunk past the task once its rays are
// finished.
template <int ER>
__device__ __forceinline__ unsigned long long trace_task_refill(const SParams& P, const SceneView& s,
                                                                const TraceIO& io, Lane& L, long long first,
                                                                int32_t base, uint32_t& cells, uint32_t& tests,
                                                                uint32_t& started) {
    const int lane = threadIdx.x & 31;
    const int32_t n = (int32_t)io.n;
    int32_t at = base, left = min(32, n - base);   // the chunk's next ray, and how many it still has
    unsigned long long next = ~0ull;               // a claimed chunk past this task
    bool active = false;
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !active);
        const int nidle = __popc(idle);
        const bool room = nidle >= io.refill || idle == FULL;
        if (left == 0 && next == ~0ull && room) {
            unsigned long long b = 0;
            if (lane == 0) b = atomicAdd(io.counter, 32ull);
            b = __shfl_sync(FULL, b, 0);
            if ((long long)b - first < (long long)n) {
                at = (int32_t)((long long)b - first);
                left = min(32, n - at);
            } else {
                next = b;
            }
        }
        if (left > 0 && room) {
            const int take = min(nidle, left);
            if (!active) {
                const int rank = __popc(idle & ((1u << lane) - 1u));
                if (rank < take) {
                    L.ray = at + rank;
                    set_deferral(L, io.heavy, io.work);
                    ++started;
                    if (start_ray<MODE_TASK>(P, io, L, L.ray)) {
                        active = true;
                    } else {
                        if (L.id != -2) L.id = -1;
                        finish_ray<MODE_TASK>(io, P, s, L);
                    }
                }
            }
            at += take;
            left -= take;
        }
        if (!__any_sync(FULL, active)) {
            if (left == 0 && next != ~0ull) return next;
            continue;
        }
        bool fin = advance_two<MODE_TASK, ER>(P, L, s, active, cells, tests);
        if (io.defer) hand_on<MODE_TASK>(P, io, L, active, fin);
        if (fin) {
            finish_ray<MODE_TASK>(io, P, s, L);
            active = false;
        }
    }
}

// Six blocks of 128 threads per SM for the batch's group pass: a group keeps
// its own scene's pointers in registers.
#ifndef GRIDRT_GROUP_BATCH_MIN_BLOCKS
#define GRIDRT_GROUP_BATCH_MIN_BLOCKS 6
#endif

// Many (scene, ray batch) tasks in one persistent launch.  Task t owns the
// 32-aligned index range [first, first + n) of one flattened ray space, so a
// 32-ray claim always falls inside one task: scene and mode are warp-uniform.
template <int ER>
__global__ void __launch_bounds__(128, GRIDRT_TRACE_MIN_BLOCKS)
    trace_batch_kernel(const BatchScene* __restrict__ scenes, int nscenes, const BatchTask* __restrict__ tasks,
                       int ntasks, long long total, unsigned long long* counter, int2* defer, int32_t defer_cap,
                       int32_t heavy, int32_t refill) {
    pdl_begin();
    __shared__ SParams P[kMaxBatchScenes];
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x) fill_sparams(scenes[i].view.params, P[i]);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    Lane L;
    uint32_t cells = 0, tests = 0, started = 0;
    unsigned long long b = 0;
    if (lane == 0) b = atomicAdd(counter, 32ull);
    b = __shfl_sync(FULL, b, 0);
    while ((long long)b < total) {
        const BatchTask T = tasks[find_task(tasks, ntasks, (long long)b)];
        const SceneView V = scenes[T.scene].view;
        TraceIO io{};
        io.rays = T.rays;
        io.n = T.n;
        io.counter = counter;
        io.defer = defer;
        io.defer_cap = defer_cap;
        io.heavy = defer ? heavy : kNoHeavy;
        io.work = work_limit(io.heavy, kHeavyWorkMult);
        io.defer_base = (int32_t)T.first;
        io.refill = refill;
        io.alike = 7;
        io.any = T.mode == MODE_ANY;
        io.occ = static_cast<uint8_t*>(T.out);
        io.hits = static_cast<int4*>(T.out);
        const int32_t base = (int32_t)((long long)b - T.first);
        if (refill > 0 && !chunk_coherent<true>(P[T.scene], io, base)) {
            b = trace_task_refill<ER>(P[T.scene], V, io, L, T.first, base, cells, tests, started);
        } else {
            trace_batch32<MODE_TASK, ER>(P[T.scene], V, io, L, base, cells, tests, started);
            if (lane == 0) b = atomicAdd(counter, 32ull);
            b = __shfl_sync(FULL, b, 0);
        }
    }
}

// Group walk over a batch's rays (flattened indices): those its launch deferred
// (QUEUE), or all of a small batch's from their start; each group resolves its
// own task, scene and mode.
template <int G, bool QUEUE>
__global__ void __launch_bounds__(128, GRIDRT_GROUP_BATCH_MIN_BLOCKS)
    trace_group_batch_kernel(const BatchScene* __restrict__ scenes, int nscenes, const BatchTask* __restrict__ tasks,
                             int ntasks, long long rays, unsigned long long* counter, const int2* __restrict__ defer,
                             int32_t defer_cap) {
    pdl_begin();
    __shared__ SParams P[kMaxBatchScenes];
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x) fill_sparams(scenes[i].view.params, P[i]);
    __syncthreads();
    const int gl = threadIdx.x & (G - 1);
    constexpr int kWant = G < 32 ? 16 / G : 1;
    unsigned long long total = (unsigned long long)rays;
    if (QUEUE) {
        total = counter[1];
        if (total > (unsigned long long)defer_cap) total = (unsigned long long)defer_cap;
    }
    bool busy = false, exhausted = false, any = false;
    int todo = 0, scene = 0;
    int3 sg = make_int3(0, 0, 0);
    Lane L = idle_lane();
    TraceIO io{};
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !busy);
        if (!exhausted && __popc(idle) >= kWant * G) {
            const unsigned long long r = claim_groups<G>(idle, counter + (QUEUE ? 2 : 0), total, exhausted);
            if (!busy && r < total) {
                const int2 d = QUEUE ? __ldg(defer + r) : make_int2((int32_t)r, -1);
                const BatchTask T = tasks[find_task(tasks, ntasks, (long long)d.x)];
                scene = T.scene;
                any = T.mode == MODE_ANY;
                io.rays = T.rays;
                io.occ = static_cast<uint8_t*>(T.out);
                io.hits = static_cast<int4*>(T.out);
                L.ray = (int32_t)((long long)d.x - T.first);
                const bool pad = !QUEUE && L.ray >= T.n;   // a task's rays are padded to a multiple of 32
                if (!pad) busy = any ? start_ray<MODE_ANY>(P[scene], io, L, L.ray) : start_ray<MODE_NEAREST>(P[scene], io, L, L.ray);
                if (busy) {
                    if (QUEUE) resume_at(P[scene], L, d.y);
                } else if (!pad) {
                    if (L.id != -2) L.id = -1;
                    if (any) finish_ray<MODE_ANY>(io, P[scene], scenes[scene].view, L, gl == 0);
                    else finish_ray<MODE_NEAREST>(io, P[scene], scenes[scene].view, L, gl == 0);
                }
                todo = gl;
                sg = step_signs(L);
            }
        }
        if (!__any_sync(FULL, busy)) {
            if (exhausted) break;
            continue;
        }
        const SceneView V = scenes[scene].view;
        const GroupOut r = group_batch<G>(P[scene], V, L, sg, busy, any, busy ? todo : 0, kNoHeavy);
        todo = G;
        if (busy && r.step == GROUP_DONE) {
            if (any) finish_ray<MODE_ANY>(io, P[scene], V, L, gl == 0);
            else finish_ray<MODE_NEAREST>(io, P[scene], V, L, gl == 0);
            busy = false;
        }
    }
}

// ---------------------------------------------------------------------------
// two-level instancing: IAccStruct::traceNearestInstance
// (src/rtcore/IAccStruct.cpp:26-72).  The ray is clipped against the scene
// box (union of the instances' world boxes); then, instance by instance in
// order, the ray taken to the instance's local space (same tnear / tfar,
// direction not renormalised, so t is the same in both spaces) walks that
// instance's grid starting from the best distance so far: a later instance
// wins only with a strictly closer hit.  Matrix rows are applied as
// x' = ((m0 x + m1 y) + m2 z) + m3, one rounding per operation.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void xf_point(const float* m, float x, float y, float z, float& ox, float& oy, float& oz) {
    ox = fadd(fadd(fadd(fmul(m[0], x), fmul(m[1], y)), fmul(m[2], z)), m[3]);
    oy = fadd(fadd(fadd(fmul(m[4], x), fmul(m[5], y)), fmul(m[6], z)), m[7]);
    oz = fadd(fadd(fadd(fmul(m[8], x), fmul(m[9], y)), fmul(m[10], z)), m[11]);
}

__device__ __forceinline__ void xf_dir(const float* m, float x, float y, float z, float& ox, float& oy, float& oz) {
    ox = fadd(fadd(fmul(m[0], x), fmul(m[1], y)), fmul(m[2], z));
    oy = fadd(fadd(fmul(m[4], x), fmul(m[5], y)), fmul(m[6], z));
    oz = fadd(fadd(fmul(m[8], x), fmul(m[9], y)), fmul(m[10], z));
}

// A world-space sphere that holds what an instance's local rays can hit: the
// preimage of its grid box under local_from_world, {centre, radius} and the
// growth of the radius per unit of the ray's |origin|_1.  `radius` is 1% above
// the box's and holds the rounding of the local ray: its origin and direction
// are products of three terms, off by less than 16 x 2^-24 of the operands'
// size, times the matrix's condition when taken back to world space.  A
// singular matrix gives an infinite or NaN radius, which culls nothing.
struct InstanceSphere {
    float cx, cy, cz, r, grow, pad[3];
};

__device__ __forceinline__ InstanceSphere instance_sphere(const SParams& P, const float* __restrict__ m) {
    double A[3][3], c[3], h[3];
    for (int i = 0; i < 3; ++i) {
        for (int j = 0; j < 3; ++j) A[i][j] = m[4 * i + j];
        c[i] = 0.5 * ((double)P.bmin[i] + P.bmax[i]) - m[4 * i + 3];
        h[i] = 0.5 * ((double)P.bmax[i] - P.bmin[i]);
    }
    double I[3][3], det = 0.0, na = 0.0, ni = 0.0;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const int a = (j + 1) % 3, b = (j + 2) % 3, e = (i + 1) % 3, f = (i + 2) % 3;
            I[i][j] = A[a][e] * A[b][f] - A[a][f] * A[b][e];
        }
    for (int j = 0; j < 3; ++j) det += A[0][j] * I[j][0];
    double w[3], r = 0.0, lc = 0.0;
    for (int i = 0; i < 3; ++i) {
        w[i] = 0.0;
        for (int j = 0; j < 3; ++j) {
            I[i][j] /= det;
            w[i] += I[i][j] * c[j];
            na += A[i][j] * A[i][j];
            ni += I[i][j] * I[i][j];
        }
        lc += fabs((double)P.bmin[i]) + fabs((double)P.bmax[i]);
    }
    for (int k = 0; k < 4; ++k) {            // the box's four diagonals in world space
        const double hy = k & 1 ? -h[1] : h[1], hz = k & 2 ? -h[2] : h[2];
        double d = 0.0;
        for (int i = 0; i < 3; ++i) {
            const double v = I[i][0] * h[0] + I[i][1] * hy + I[i][2] * hz;
            d += v * v;
        }
        r = d > r || !(d == d) ? d : r;
    }
    const double u = 16.0 / 16777216.0, cond = sqrt(na * ni);
    InstanceSphere S{};
    S.cx = (float)w[0];
    S.cy = (float)w[1];
    S.cz = (float)w[2];
    S.r = (float)(1.01 * sqrt(r) + u * (cond * (fabs(w[0]) + fabs(w[1]) + fabs(w[2])) + sqrt(ni) * lc));
    S.grow = (float)(2.0 * u * cond);
    return S;
}

__global__ void instances_prep_kernel(const InstanceRec* __restrict__ recs, int ninst, SParams* __restrict__ sp,
                                      InstanceSphere* __restrict__ spheres) {
    pdl_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ninst; i += gridDim.x * blockDim.x) {
        SParams P;
        fill_sparams(recs[i].view.params, P);
        sp[i] = P;
        spheres[i] = instance_sphere(P, recs[i].xf);
    }
}

// Bound by the walks' latency and by the per-instance work of rays that miss:
// 16 instances of three meshes, 1024^2 camera rays, 1,073 -> 664 us with the
// sphere test, three sets of instances in turn (997 -> 735 on another machine;
// 1,442 -> 947 us one launch at a time).  Six blocks of 128 an SM: 736 / 673 /
// 660 / 644 us at 4 / 5 / 6 / 7, alone 986 / 939 / 947 / 969.
#ifndef GRIDRT_INST_MIN_BLOCKS
#define GRIDRT_INST_MIN_BLOCKS 6
#endif
template <int MODE, int ER>
__global__ void __launch_bounds__(128, GRIDRT_INST_MIN_BLOCKS) trace_instances_kernel(const InstanceRec* __restrict__ recs,
                                                              const SParams* __restrict__ sp,
                                                              const InstanceSphere* __restrict__ spheres, int ninst,
                                                              InstanceBox box, TraceIO io, int32_t* inst_out) {
    pdl_begin();
    __shared__ SParams Pw[4];
    const int lane = threadIdx.x & 31;
    SParams& P = Pw[threadIdx.x >> 5];
    uint32_t cells = 0, tests = 0, started = 0;
    for (;;) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(io.counter, 32ull);
        b = __shfl_sync(FULL, b, 0);
        if ((long long)b >= io.n) break;
        const long long r = (long long)b + lane;
        bool alive = r < io.n, noray = false;
        float wo[3] = {0.f, 0.f, 0.f}, wd[3] = {1.f, 1.f, 1.f};
        float tn = 0.f, tf = 0.f, tmax = 0.f;
        if (alive) {
            ++started;
            const float4 a = __ldg(io.rays + 2 * r), c = __ldg(io.rays + 2 * r + 1);
            wo[0] = a.x; wo[1] = a.y; wo[2] = a.z;
            wd[0] = c.x; wd[1] = c.y; wd[2] = c.z;
            tn = a.w;
            tf = tmax = c.w;
            if (MODE == MODE_ANY && tf < 0.0f) {
                noray = true;
                alive = false;
            } else {
                // Ray::update + AabbIntersection::clipRay on the scene box
                float rn = tn, rf = tf;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const float inv = frcp(wd[d]);
                    const float t0 = fmul(fsub(box.bmin[d], wo[d]), inv), t1 = fmul(fsub(box.bmax[d], wo[d]), inv);
                    rn = vmax(rn, vmin(t0, t1));
                    rf = vmin(rf, vmax(t0, t1));
                }
                if (rn > rf) alive = false;
                tn = rn;
                tf = rf;
            }
        }
        float gbest = kFltMax;
        int32_t gid = -1, ginst = -1;
        const float dd = wd[0] * wd[0] + wd[1] * wd[1] + wd[2] * wd[2];
        const float o1 = fabsf(wo[0]) + fabsf(wo[1]) + fabsf(wo[2]);
        for (int i = 0; i < ninst; ++i) {
            if (!__any_sync(FULL, alive)) break;
            // the ray passes the instance's sphere, or meets it only behind
            // its start or beyond its best hit: the instance cannot change the
            // ray's result.  The warp takes on an instance that none of its
            // rays passes up; taking one to local space and to its box costs
            // five times the test.
            const float4 s0 = __ldg(reinterpret_cast<const float4*>(spheres + i));
            const float R = s0.w + __ldg(&spheres[i].grow) * o1;
            const float qx = s0.x - wo[0], qy = s0.y - wo[1], qz = s0.z - wo[2];
            const float xx = qy * wd[2] - qz * wd[1], xy = qz * wd[0] - qx * wd[2], xz = qx * wd[1] - qy * wd[0];
            const float q2 = qx * qx + qy * qy + qz * qz, along = qx * wd[0] + qy * wd[1] + qz * wd[2];
            const float R2 = 1.02f * (R * R) + 1e-9f * q2, lim = R2 * dd;
            const float past = along - 1.001f * fminf(gbest, tf) * dd;     // beyond the best hit and the far clip
            // (products below the normal floats round to too few bits to tell)
            const bool tell = dd >= 1e-20f && R2 >= 1e-18f;
            const bool cull = tell && (xx * xx + xy * xy + xz * xz > lim || (tn >= 0.0f && along < 0.0f && q2 > R2) ||
                                       (tn >= 0.0f && past > 0.0f && past * past > lim));
            if (!__any_sync(FULL, alive && !cull)) continue;
            __syncwarp();
            {
                const uint32_t* src = reinterpret_cast<const uint32_t*>(sp + i);
                uint32_t* dst = reinterpret_cast<uint32_t*>(&P);
                for (int w = lane; w < (int)(sizeof(SParams) / 4); w += 32) dst[w] = __ldg(src + w);
            }
            __syncwarp();
            const InstanceRec* rec = recs + i;
            Lane L;
            bool active = alive && !cull && !P.failed && !__ldg(&rec->skip);
            if (active) {
                float m[12];
#pragma unroll
                for (int k = 0; k < 12; ++k) m[k] = __ldg(&rec->xf[k]);
                xf_point(m, wo[0], wo[1], wo[2], L.ox, L.oy, L.oz);
                xf_dir(m, wd[0], wd[1], wd[2], L.dx, L.dy, L.dz);
                active = setup_ray(P, L, tn, tf);
                L.tmax = tmax;
                set_deferral(L, kNoHeavy, kNoHeavy);
                if (MODE == MODE_NEAREST) L.best = gbest;
            }
            const SceneView V = rec->view;
            while (__any_sync(FULL, active)) {
                if (advance<MODE, ER>(P, L, V, active, cells, tests)) {
                    active = false;
                    if (L.id >= 0) {
                        // the next instance compares against the exact
                        // distance (the walk may have accepted its hit on
                        // Moller-Trumbore's t)
                        gbest = wald_f_of(L, L.id, V.wald);
                        gid = L.id;
                        ginst = i;
                        if (MODE == MODE_ANY) alive = false;   // occluded
                    }
                }
            }
        }
        if (r < io.n) {
            if (MODE == MODE_ANY) {
                io.occ[r] = noray ? 2 : (gid >= 0 ? 1 : 0);
            } else {
                int4 h = make_int4(-1, 0, 0, 0);
                if (gid >= 0) {
                    // reported values in the winning instance's space
                    const InstanceRec* R = recs + ginst;
                    float m[12];
#pragma unroll
                    for (int k = 0; k < 12; ++k) m[k] = __ldg(&R->xf[k]);
                    Lane L;
                    xf_point(m, wo[0], wo[1], wo[2], L.ox, L.oy, L.oz);
                    xf_dir(m, wd[0], wd[1], wd[2], L.dx, L.dy, L.dz);
                    L.id = gid;
                    L.best = gbest;
                    h = wald_hit(R->view.wald, L);
                }
                io.hits[r] = h;
                if (inst_out) inst_out[r] = ginst;
            }
        }
    }
    if (io.ctr) flush_counters(io.ctr, started, cells, tests);
}

template <int MODE, int ER>
static void launch_instances_er(const InstanceRec* recs, const SParams* sp, const InstanceSphere* spheres, int ninst,
                                const InstanceBox& box,
                                const TraceIO& io, int32_t* inst_out, const TraceTuning& tune, int num_sms,
                                cudaStream_t st) {
    static int per_sm = 0;
    if (per_sm == 0) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, trace_instances_kernel<MODE, ER>, 128, 0);
        per_sm = b > 0 ? b : 1;
    }
    long long blocks = (io.n + 127) / 128;
    if (tune.persistent) blocks = blocks < (long long)per_sm * num_sms ? blocks : (long long)per_sm * num_sms;
    if (blocks < 1) blocks = 1;
    if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
    trace_instances_kernel<MODE, ER><<<(int)blocks, 128, 0, st>>>(recs, sp, spheres, ninst, box, io, inst_out);
}

size_t instance_params_bytes(int ninst) {
    return (sizeof(InstanceSphere) + sizeof(SParams)) * (size_t)(ninst > 0 ? ninst : 1);
}

void launch_trace_instances(const InstanceRec* recs, void* d_params, int ninst, const InstanceBox& box,
                            const float4* rays, int64_t n, int4* hits, int32_t* inst_out, uint8_t* occ, int mode,
                            TraceCounters* ctr, unsigned long long* counter, const TraceTuning& tune, int num_sms,
                            cudaStream_t st) {
    if (n <= 0 || ninst <= 0) return;
    count_launches(2);
    InstanceSphere* spheres = static_cast<InstanceSphere*>(d_params);
    SParams* sp = reinterpret_cast<SParams*>(spheres + ninst);
    instances_prep_kernel<<<(ninst + 127) / 128, 128, 0, st>>>(recs, ninst, sp, spheres);
    cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);
    TraceIO io{};
    io.rays = rays;
    io.hits = hits;
    io.occ = occ;
    io.n = n;
    io.counter = counter;
    io.ctr = ctr;
    io.heavy = kNoHeavy;
    io.work = kNoHeavy;
    const int er = tune.empty_run;
    if (mode == MODE_ANY) {
        if (er <= 2) launch_instances_er<MODE_ANY, 2>(recs, sp, spheres, ninst, box, io, inst_out, tune, num_sms, st);
        else if (er <= 4) launch_instances_er<MODE_ANY, 4>(recs, sp, spheres, ninst, box, io, inst_out, tune, num_sms, st);
        else launch_instances_er<MODE_ANY, 8>(recs, sp, spheres, ninst, box, io, inst_out, tune, num_sms, st);
    } else {
        if (er <= 2) launch_instances_er<MODE_NEAREST, 2>(recs, sp, spheres, ninst, box, io, inst_out, tune, num_sms, st);
        else if (er <= 4) launch_instances_er<MODE_NEAREST, 4>(recs, sp, spheres, ninst, box, io, inst_out, tune, num_sms, st);
        else launch_instances_er<MODE_NEAREST, 8>(recs, sp, spheres, ninst, box, io, inst_out, tune, num_sms, st);
    }
}

__global__ void deform_kernel(const float* __restrict__ base, const float* __restrict__ nrm, float* __restrict__ out,
                              int64_t nverts, float amp, float freq, float phase) {
    pdl_begin();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nverts; i += stride) {
        const float px = base[3 * i], py = base[3 * i + 1], pz = base[3 * i + 2];
        const float s = amp * sinf(freq * px + phase);
        out[3 * i] = px + s * nrm[3 * i];
        out[3 * i + 1] = py + s * nrm[3 * i + 1];
        out[3 * i + 2] = pz + s * nrm[3 * i + 2];
    }
}

template <int ER>
static void launch_batch_er(const BatchScene* scenes, int nscenes, const BatchTask* tasks, int ntasks, long long total,
                            const TraceSlot& slot, int32_t heavy, int32_t refill, int num_sms, cudaStream_t st) {
    static int per_sm = 0;
    if (per_sm == 0) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, trace_batch_kernel<ER>, 128, 0);
        per_sm = b > 0 ? b : 1;
    }
    long long blocks = (total + 127) / 128;
    blocks = blocks < (long long)per_sm * num_sms ? blocks : (long long)per_sm * num_sms;
    if (blocks < 1) blocks = 1;
    launch_k(trace_batch_kernel<ER>, (unsigned)blocks, 128, 0, st, scenes, nscenes, tasks, ntasks, total, slot.ctr,
             heavy > 0 ? slot.defer : nullptr, slot.defer_cap, heavy, refill);
}

template <int G, bool QUEUE>
static void launch_group_batch(const BatchScene* scenes, int nscenes, const BatchTask* tasks, int ntasks,
                               long long total, const TraceSlot& slot, int num_sms, cudaStream_t st) {
    static int per_sm = 0;
    if (per_sm == 0) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, trace_group_batch_kernel<G, QUEUE>, 128, 0);
        per_sm = b > 0 ? b : 1;
    }
    const long long full = (long long)per_sm * num_sms, need = (total + 128 / G - 1) / (128 / G);
    launch_k(trace_group_batch_kernel<G, QUEUE>, (unsigned)(need < full ? need : full), 128, 0, st, scenes, nscenes,
             tasks, ntasks, total, slot.ctr, slot.defer, slot.defer_cap);
}

void launch_trace_batch(const BatchScene* scenes, int nscenes, const BatchTask* tasks, int ntasks, long long total,
                        const TraceSlot& slot, const TraceTuning& tune, int num_sms, cudaStream_t st) {
    if (total <= 0 || ntasks <= 0) return;
    // deferred entries are int32 flattened indices
    const int lanes = tune.lanes || total > 0x7fffffffLL ? 1 : lanes_for(total, num_sms, 4);
    if (lanes > 1) {
        // a small batch: every ray by a group of lanes, long lists dealt out
        // over it
        count_launches(1);
        cudaMemsetAsync(slot.ctr, 0, 3 * sizeof(unsigned long long), st);
        if (lanes == 32) launch_group_batch<32, false>(scenes, nscenes, tasks, ntasks, total, slot, num_sms, st);
        else if (lanes == 16) launch_group_batch<16, false>(scenes, nscenes, tasks, ntasks, total, slot, num_sms, st);
        else launch_group_batch<8, false>(scenes, nscenes, tasks, ntasks, total, slot, num_sms, st);
        return;
    }
    const bool defer = tune.heavy_cell > 0 && slot.defer && slot.defer_cap > 0 && total <= 0x7fffffffLL;
    const int32_t heavy = defer ? tune.heavy_cell : 0;
    count_launches(defer ? 2 : 1);
    cudaMemsetAsync(slot.ctr, 0, 3 * sizeof(unsigned long long), st);
    if (tune.empty_run <= 2) launch_batch_er<2>(scenes, nscenes, tasks, ntasks, total, slot, heavy, refill_for(tune, 0), num_sms, st);
    else if (tune.empty_run <= 4) launch_batch_er<4>(scenes, nscenes, tasks, ntasks, total, slot, heavy, refill_for(tune, 0), num_sms, st);
    else if (tune.empty_run <= 8) launch_batch_er<8>(scenes, nscenes, tasks, ntasks, total, slot, heavy, refill_for(tune, 0), num_sms, st);
    else launch_batch_er<16>(scenes, nscenes, tasks, ntasks, total, slot, heavy, refill_for(tune, 0), num_sms, st);
    if (defer) {
        if (tune.heavy_lanes <= 4) launch_group_batch<4, true>(scenes, nscenes, tasks, ntasks, total, slot, num_sms, st);
        else if (tune.heavy_lanes <= 8) launch_group_batch<8, true>(scenes, nscenes, tasks, ntasks, total, slot, num_sms, st);
        else if (tune.heavy_lanes <= 16) launch_group_batch<16, true>(scenes, nscenes, tasks, ntasks, total, slot, num_sms, st);
        else launch_group_batch<32, true>(scenes, nscenes, tasks, ntasks, total, slot, num_sms, st);
    }
}

void launch_deform(const float* base, const float* normals, float* out, int64_t nverts, float amp, float freq,
                   float phase, cudaStream_t st) {
    if (nverts <= 0) return;
    count_launches(1);
    int64_t blocks = (nverts + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    launch_k(deform_kernel, (unsigned)blocks, 256, 0, st, base, normals, out, nverts, amp, freq, phase);
}

}  // namespace gridrt
