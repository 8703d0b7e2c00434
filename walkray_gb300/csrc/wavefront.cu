// wavefront.cu — kernels and driver of the wavefront renderer (see
// wavefront.h for the stage structure).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>
#include <map>

#include "wavefront.h"
#include "wr_warp_trace.cuh"

namespace wr {

constexpr uint32_t WF_MAX_JOBS = 256;
constexpr uint32_t WF_MAX_SCENES = 64;
constexpr int WF_FINISH_BLOCK = 128;

uint32_t wf_max_jobs() { return WF_MAX_JOBS; }

// ---------------------------------------------------------------------------
// state load / store
// ---------------------------------------------------------------------------
struct WfPath {
    PRay cur;
    f3 color, prev_d;
    uint32_t depth;
    InsideStack st;
    uint32_t pixel, sample, dim;
    int job;
    float mis_pdf;  // density of the current ray's scatter (WR_RENDER_NEE_MIS)
    f3 acc;         // light connections counted so far (WR_RENDER_NEE_MIS)
};

__device__ __forceinline__ int4 as_i4(float4 v) {
    return make_int4(__float_as_int(v.x), __float_as_int(v.y), __float_as_int(v.z), __float_as_int(v.w));
}
__device__ __forceinline__ float4 as_f4(int4 v) {
    return make_float4(__int_as_float(v.x), __int_as_float(v.y), __int_as_float(v.z), __int_as_float(v.w));
}

// Field f of record i lies in the record's 16-byte chunk f ^ (i & 7): lanes that
// read or write one field of neighbouring records then use all banks of the L1
// cache instead of one group of four (a 128-byte stride takes 0.99 cycles a
// piece on an SM, spread 0.34).
__device__ __forceinline__ uint32_t wf_swizzle(uint64_t i) { return (uint32_t)i & 7u; }

__device__ __forceinline__ void wf_load(const WfSide& X, uint32_t i, WfPath& p) {
    const float4* r = X.rec + (size_t)WF_REC * i;
    const uint32_t x = wf_swizzle(i);
    const float4 a0 = r[WF_O ^ x], a1 = r[WF_D ^ x], a2 = r[WF_RAD ^ x], a3 = r[WF_COL ^ x];
    const int4 ids = as_i4(r[WF_IDS ^ x]), misc = as_i4(r[WF_MISC ^ x]), stk = as_i4(r[WF_STK ^ x]);
    p.cur = ray_default();
    p.cur.o = mk(a0.x, a0.y, a0.z);
    p.cur.oP = a0.w;
    p.cur.d = mk(a1.x, a1.y, a1.z);
    p.cur.dP = a1.w;
    p.cur.rad = mk(a2.x, a2.y, a2.z);
    p.cur.cnorm = mk(a2.w, a3.w, __int_as_float(misc.w));
    p.color = mk(a3.x, a3.y, a3.z);
    p.cur.inside = ids.x;
    p.cur.contact = ids.y;
    p.job = ids.z;
    p.pixel = (uint32_t)ids.w;
    p.sample = (uint32_t)misc.x;
    p.dim = (uint32_t)misc.y;
    p.depth = (uint32_t)misc.z & 0xffffu;
    p.st.n = (int)((uint32_t)misc.z >> 16);
    p.st.v0 = stk.x;
    p.st.v1 = stk.y;
    p.st.v2 = stk.z;
    p.st.v3 = stk.w;
    const float4 a4 = r[WF_PREV ^ x];
    p.prev_d = mk(a4.x, a4.y, a4.z);
    p.mis_pdf = a4.w;
    p.acc = mk(0, 0, 0);
}

__device__ __forceinline__ void wf_load_acc(const WfSide& X, uint32_t i, WfPath& p) {
    const float4 a5 = X.a5[i];
    p.acc = mk(a5.x, a5.y, a5.z);
}

// a path as record number i (its swizzle), its chunks at r
__device__ __forceinline__ void wf_store_at(float4* r, uint32_t i, const WfPath& p) {
    const uint32_t x = wf_swizzle(i);
    r[WF_O ^ x] = make_float4(p.cur.o.x, p.cur.o.y, p.cur.o.z, p.cur.oP);
    r[WF_D ^ x] = make_float4(p.cur.d.x, p.cur.d.y, p.cur.d.z, p.cur.dP);
    r[WF_IDS ^ x] = as_f4(make_int4(p.cur.inside, p.cur.contact, p.job, (int)p.pixel));
    r[WF_MISC ^ x] = as_f4(make_int4((int)p.sample, (int)p.dim, (int)(p.depth | ((uint32_t)p.st.n << 16)),
                                     __float_as_int(p.cur.cnorm.z)));
    r[WF_RAD ^ x] = make_float4(p.cur.rad.x, p.cur.rad.y, p.cur.rad.z, p.cur.cnorm.x);
    r[WF_COL ^ x] = make_float4(p.color.x, p.color.y, p.color.z, p.cur.cnorm.y);
    r[WF_STK ^ x] = as_f4(make_int4(p.st.v0, p.st.v1, p.st.v2, p.st.v3));
    r[WF_PREV ^ x] = make_float4(p.prev_d.x, p.prev_d.y, p.prev_d.z, p.mis_pdf);
}
__device__ __forceinline__ void wf_store(const WfSide& Y, uint32_t j, const WfPath& p) {
    wf_store_at(Y.rec + (size_t)WF_REC * j, j, p);
}

__device__ __forceinline__ void wf_store_acc(const WfSide& Y, uint32_t j, const WfPath& p) {
    Y.a5[j] = make_float4(p.acc.x, p.acc.y, p.acc.z, 0.f);
}

// warp-aggregated append: returns this lane's position (valid if `want`)
__device__ __forceinline__ uint32_t warp_append(unsigned int* counter, bool want, uint32_t offset) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned m = __ballot_sync(0xffffffffu, want);
    uint32_t base = 0;
    if (m) {
        const int leader = __ffs(m) - 1;
        if ((int)lane == leader) base = atomicAdd(counter, (unsigned)__popc(m));
        base = __shfl_sync(0xffffffffu, base, leader);
    }
    return offset + base + __popc(m & ((1u << lane) - 1u));
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__global__ void k_wf_reset(WfSide Y, unsigned long long* work, unsigned int* shadow_count, WfSort B) {
    Y.counts[0] = 0;
    Y.counts[1] = 0;
    work[0] = 0;  // the extend stage's ray counter
    work[1] = 0;  // the shadow stage's
    work[2] = 0;  // the track stage's
    *shadow_count = 0;
    for (int k = 0; k < WF_SORT_KEYS + WF_FLIGHT_KEYS; k++) B.counts[k] = 0;
}

// sort: bucket the queue by shading material.  A block counts a tile of
// WF_SORT_TILE paths in shared memory and adds to the buckets' counters once for
// it: with an addition per warp and key they queued up for the counters' sector
// (mixed-material 1024^2 x 32 spp 30.85 ms,
// 28.85 this way; twice the blocks or tiles of 512 and 2048: within 1 %).
constexpr int WF_SORT_BLOCK = 256, WF_SORT_EACH = 4, WF_SORT_TILE = WF_SORT_BLOCK * WF_SORT_EACH;
__global__ void __launch_bounds__(WF_SORT_BLOCK) k_wf_sort(const RenderScene* __restrict__ scenes,
                                                   const WfJob* __restrict__ jobs, WfSide X,
                                                   const int2* __restrict__ hits, WfSort B, uint32_t capacity) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ uint32_t s_count[WF_SORT_KEYS], s_base[WF_SORT_KEYS];
    const uint32_t n = X.counts[0] + X.counts[1];
    const uint32_t tiles = n / WF_SORT_TILE + (n % WF_SORT_TILE != 0);
    const unsigned lane = threadIdx.x & 31u;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        if (threadIdx.x < WF_SORT_KEYS) s_count[threadIdx.x] = 0;
        __syncthreads();
        int key[WF_SORT_EACH];
        uint32_t rank[WF_SORT_EACH];
#pragma unroll
        for (int t = 0; t < WF_SORT_EACH; t++) {
            const uint32_t i = tile * WF_SORT_TILE + t * WF_SORT_BLOCK + threadIdx.x;
            key[t] = -1;
            if (i < n) {
                key[t] = 0;
                const int slot = hits[i].x;
                const int4 ids = as_i4(X.rec[(size_t)WF_REC * i + (WF_IDS ^ wf_swizzle(i))]);
                if (slot >= 0 || ids.x >= 0) {
                    const RenderScene& S = scenes[jobs[ids.z].scene];
                    const int self = ids.x >= 0 ? ids.x : (int)__float_as_uint(__ldg(&S.tree.tris[slot].v1.w));
                    key[t] = min(1 + (int)obj_type(S, self), WF_SORT_KEYS - 1);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < WF_SORT_EACH; t++) {
            const unsigned peers = __match_any_sync(FULL, key[t]);
            const int leader = __ffs(peers) - 1;
            uint32_t at = 0;
            if (key[t] >= 0 && (int)lane == leader) at = atomicAdd(&s_count[key[t]], (uint32_t)__popc(peers));
            rank[t] = __shfl_sync(FULL, at, leader) + __popc(peers & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (threadIdx.x < WF_SORT_KEYS && s_count[threadIdx.x])
            s_base[threadIdx.x] = atomicAdd(&B.counts[threadIdx.x], s_count[threadIdx.x]);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < WF_SORT_EACH; t++)
            if (key[t] >= 0)
                B.idx[(size_t)key[t] * capacity + s_base[key[t]] + rank[t]] =
                    tile * WF_SORT_TILE + t * WF_SORT_BLOCK + threadIdx.x;
    }
}

// Entry `at` of the list of a flight outcome.  It lies behind material list
// 1 + outcome: the lists together hold at most `capacity` paths, so each has
// room for all paths of the medium's.
__device__ __forceinline__ uint32_t* wf_flight_list(const WfSort& B, uint32_t capacity, int outcome, uint32_t at) {
    return B.idx + (size_t)(1 + outcome) * capacity + B.counts[1 + outcome] + at;
}

// track: the flights of the paths inside heterogeneous media (the bucket of
// that material), delta tracking with lanes that take the next path when
// theirs ends.  A step waits for eight grid reads and a logarithm; in the shade
// stage the longest flight of 32 held the others up, at half of this kernel's
// warps and behind an instruction cache full of materials (media scene
// 18.8 ms, 17.4 this way).  Launched only while a scene has such a medium.
// Refilled at 8 idle lanes, runs of at most 256 paths and a quarter of a warp's
// share, so that the last warps end together.  The ended flights are bucketed
// by what shade has to do for them (WF_FLIGHT_KEYS): in one bucket a warp ran
// the collision, the boundary and every surface's scatter one after the other
// (shade of the media
// scene's second bounce 1.24 ms with 13.6 lanes at work, 0.46 with 23.7).
constexpr int WF_TRACK_BLOCK = 128;
__global__ void __launch_bounds__(WF_TRACK_BLOCK, 7)
    k_wf_track(const RenderScene* __restrict__ scenes, const WfJob* __restrict__ jobs, WfSide X,
               const int2* __restrict__ hits, WfSort B, uint32_t capacity, Flight* __restrict__ flights,
               unsigned int* __restrict__ counter) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int KEY = 1 + WR_MAT_HETEROGENEOUS;
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t n = B.counts[KEY];
    const uint32_t warps = gridDim.x * (WF_TRACK_BLOCK / 32);
    const uint32_t run = min(256u, max(1u, n / (warps * 4u)));
    const uint32_t* __restrict__ idx = B.idx + (size_t)KEY * capacity;
    uint32_t next = 0, end = 0;
    bool dry = false, active = false;
    uint32_t i = 0;
    int steps = 0, outcome = -1, end_key = 0;  // outcome: the ended path's bucket, until it is in its list
    f3 o = mk(0, 0, 0), d = mk(0, 0, 0);
    float far = 0.f, scale = 0.f, mu = 0.f, sgt = 0.f;
    GridDev G{};
    PathRng g;
    g.init(0, 0, 0);
    Flight f{0.f, 0.f, 0, 0u};
    // Ended paths wait in shared memory, 32 of an outcome go to its list at once:
    // the warps' additions to the four counters queue up for their sector (one
    // for each refill 0.39 ms a launch, this way 0.35).
    __shared__ uint32_t s_ended[WF_TRACK_BLOCK / 32][WF_FLIGHT_KEYS][64];
    uint32_t(*ended)[64] = s_ended[threadIdx.x >> 5];
    uint32_t waiting[WF_FLIGHT_KEYS] = {};
    auto flush = [&](int key, uint32_t count) {
        __syncwarp();
        unsigned int at = 0;
        if (lane == 0) at = atomicAdd(&B.counts[WF_SORT_KEYS + key], count);
        at = __shfl_sync(FULL, at, 0);
        waiting[key] -= count;
        if (lane < count) *wf_flight_list(B, capacity, key, at + lane) = ended[key][waiting[key] + lane];
        __syncwarp();
    };
    auto append = [&]() {  // the idle lanes' paths (all lanes call it)
#pragma unroll
        for (int key = 0; key < WF_FLIGHT_KEYS; key++) {
            const unsigned m = __ballot_sync(FULL, outcome == key);
            if (outcome == key) ended[key][waiting[key] + __popc(m & ((1u << lane) - 1u))] = i;
            waiting[key] += __popc(m);
            if (waiting[key] >= 32u) flush(key, 32u);
        }
        outcome = -1;
    };
    for (;;) {
        unsigned idle = __ballot_sync(FULL, !active);
        if (idle == FULL || (!dry && __popc(idle) >= 8)) {
            append();
            while (!dry && (idle == FULL || __popc(idle) >= 8)) {
                if (next == end) {
                    uint32_t b = 0;
                    if (lane == 0) b = atomicAdd(counter, run);
                    next = __shfl_sync(FULL, b, 0);
                    if (next >= n) {
                        dry = true;
                        break;
                    }
                    end = min(next + run, n);
                }
                const uint32_t k = next + __popc(idle & ((1u << lane) - 1u));
                if (!active && k < end) {
                    i = idx[k];
                    const float4* r = X.rec + (size_t)WF_REC * i;
                    const uint32_t x = wf_swizzle(i);
                    const int4 ids = as_i4(r[WF_IDS ^ x]);
                    if (ids.x < 0) {  // the path enters the medium
                        outcome = WF_FLIGHT_BOUNDARY;
                    } else {
                        const float4 a0 = r[WF_O ^ x], a1 = r[WF_D ^ x];
                        const int4 misc = as_i4(r[WF_MISC ^ x]);
                        const WfJob& J = jobs[ids.z];
                        const RenderScene& S = scenes[J.scene];
                        const wr_object_desc* m = &S.objs[ids.x];
                        G = S.grids[__ldg(&m->grid_index)];
                        scale = __ldg(&m->density_scale);
                        sgt = __ldg(&m->sigma_s[0]) + __ldg(&m->sigma_a[0]);
                        mu = G.majorant * scale * sgt;
                        o = mk(a0.x, a0.y, a0.z);
                        d = mk(a1.x, a1.y, a1.z);
                        const int2 hv = hits[i];
                        far = hv.x < 0 ? -1.f : __int_as_float(hv.y);  // as set_hit has it
                        end_key = WF_FLIGHT_OTHER;
                        if (hv.x >= 0) {
                            const int obj = (int)__float_as_uint(__ldg(&S.tree.tris[hv.x].v1.w));
                            if (obj == ids.x) end_key = WF_FLIGHT_BOUNDARY;
                            else if (obj_type(S, obj) == WR_MAT_DIFFUSE) end_key = WF_FLIGHT_DIFFUSE;
                        }
                        g.init(J.seed, (uint32_t)ids.w, (uint32_t)misc.x, (uint32_t)misc.y);
                        f = Flight{0.f, 0.f, 0, 0u};
                        steps = mu > 0.f ? 0 : TRACK_STEPS;
                        active = true;
                    }
                }
                next = min(next + (uint32_t)__popc(idle), end);
                append();
                idle = __ballot_sync(FULL, !active);
            }
            if (idle == FULL) break;
        }
        if (active) {
            bool done = steps >= TRACK_STEPS;
            if (!done) {
                done = track_step(G, scale, mu, sgt, o, d, far, g, f);
                steps++;
            }
            if (done) {
                f.dim = g.dim;
                flights[i] = f;
                active = false;
                outcome = f.collided ? WF_FLIGHT_COLLIDED : end_key;
            }
        }
    }
#pragma unroll
    for (int key = 0; key < WF_FLIGHT_KEYS; key++)
        if (waiting[key]) flush(key, waiting[key]);
}

// film update of a finished path: isLegalColor, fixVignetting, FP32 atomics
__device__ __forceinline__ void film_add(const WfJob& J, uint32_t pixel, f3 result) {
    if (!legal(result)) result = mk(0, 0, 0);
    const f3 c = fix_vignetting(J.cam, result, pixel);
    float* f = J.film + 3 * (size_t)pixel;
    atomicAdd(f + 0, c.x);
    atomicAdd(f + 1, c.y);
    atomicAdd(f + 2, c.z);
    if (J.film2) {
        float* f2 = J.film2 + 3 * (size_t)pixel;
        atomicAdd(f2 + 0, c.x * c.x);
        atomicAdd(f2 + 1, c.y * c.y);
        atomicAdd(f2 + 2, c.z * c.z);
    }
}

// shadow stage, second half: with the closest hit of every NEE connection
// and light connection (WF_SHADOW_*) from k_wf_shadow_trace, the visible
// contributions go to the film or to their path
__global__ void __launch_bounds__(128) k_wf_shadow(const RenderScene* __restrict__ scenes,
                                                     const WfJob* __restrict__ jobs, WfShadow Q,
                                                     const int2* __restrict__ hits, WfSide Y) {
    const uint32_t n = *Q.count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 o = Q.o[i], d = Q.d[i], c = Q.c[i];
        const int4 ids = Q.ids[i];
        const WfJob& J = jobs[ids.z];
        const RenderScene& S = scenes[J.scene];
        const int2 hv = hits[i];
        Hit h;
        h.slot = hv.x;
        h.t = __int_as_float(hv.y);
        const int kind = __float_as_int(c.w);
        const f3 contrib = mk(c.x, c.y, c.z);
        if (kind == WF_SHADOW_NEE) {
            if (nee_visible(h, o.w)) film_add(J, (uint32_t)ids.w, contrib);
            continue;
        }
        LightReq lr;
        lr.dist = o.w;
        lr.light = __float_as_int(d.w);
        const bool vis = light_req_visible(S, h, lr);
        const float4 r = Q.r[i];
        if (kind == WF_SHADOW_MIS_KEEP) {
            if (vis) {
                const int t = __float_as_int(r.w);
                float4 a = Y.a5[t];
                a.x += contrib.x;
                a.y += contrib.y;
                a.z += contrib.z;
                Y.a5[t] = a;
            }
        } else {
            f3 tot = mk(r.x, r.y, r.z);
            if (vis) tot = tot + contrib;
            if (tot.x != 0.f || tot.y != 0.f || tot.z != 0.f) film_add(J, (uint32_t)ids.w, tot);
        }
    }
}

// extend: closest hit of every queued ray; the eye ray (contact == camera)
// without a filter, all others with NoSelfCondition.  Rays of different jobs
// (and scenes) share the queue; each lane follows its own ray's tree.
struct ExtendSrc {
    const RenderScene* __restrict__ scenes;
    const WfJob* __restrict__ jobs;
    WfSide X;
    int2* __restrict__ hits;
    TraceWork work;  // this thread's counts of the exact walk (profiling launches)

    __device__ __forceinline__ void fetch(uint64_t id, TraceRay& a) const {
        const float4* r = X.rec + (size_t)WF_REC * id;
        const uint32_t x = wf_swizzle(id);
        const float4 a0 = r[WF_O ^ x], a1 = r[WF_D ^ x];
        const int4 ids = as_i4(r[WF_IDS ^ x]);
        const WfJob& J = jobs[ids.z];
        a.T = &scenes[J.scene].tree;
        a.o = mk(a0.x, a0.y, a0.z);
        a.d = mk(a1.x, a1.y, a1.z);
        a.pf = prune_factor(J.flags);
        a.filt = ids.y != CAMERA_OBJ;
        a.inside = ids.x;
        a.contact = ids.y;
    }
    __device__ __forceinline__ void put(uint64_t id, const TraceRay&, const Hit& h) const {
        hits[id] = make_int2(h.slot, __float_as_int(h.t));
    }
    // rays of several scenes share the queue
    __device__ __forceinline__ const TriRec* tris_of(const RayInShared& rays, int from) const {
        return rays.tris_of(from);
    }
    __device__ __forceinline__ void load(uint64_t id, TraceLane& L, uint32_t* stack, int stride) const {
        TraceRay a;
        fetch(id, a);
        load_lane(a, L, stack, stride);
    }
    __device__ __forceinline__ void store(uint64_t id, const TraceLane& L) {
        hits[id] = make_int2(L.h.slot, __float_as_int(L.h.t));
        work.rays += 1;
        work.boxes += L.n_box;
        work.tris += L.n_tri;
    }
};

// adds the warp's sum of v to *dst (one atomic per warp)
__device__ __forceinline__ void warp_add(unsigned long long* dst, unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31u) == 0 && v) atomicAdd(dst, v);
}

// MINB > 0: compiled for at least MINB resident CTAs of 128 threads per SM
// (a register cap), chosen by the configuration's ctas_per_sm
#define WR_EXTEND_BOUNDS(MINB) __launch_bounds__(128, (MINB) > 0 ? (MINB) : 1)

// WALK: the reference's own tree (launched while a job with
// WR_RENDER_EXACT_TRAVERSAL, whose counts are the reference's, or a scene
// without a four-wide tree is in the table)
template <bool STATS, bool WALK, int MINB>
__global__ void WR_EXTEND_BOUNDS(MINB) k_wf_extend(const RenderScene* __restrict__ scenes,
                                                     const WfJob* __restrict__ jobs, WfSide X, int2* __restrict__ hits,
                                                     unsigned long long* __restrict__ work, int stack_cap,
                                                     TraceTune tune, unsigned int* __restrict__ err,
                                                     unsigned long long* __restrict__ stats) {
    extern __shared__ __align__(16) uint32_t s_stack[];
    const uint64_t n = (uint64_t)X.counts[0] + X.counts[1];
    if (n == 0) return;
    ExtendSrc src{scenes, jobs, X, hits, TraceWork{0ull, 0ull, 0ull}};
    if (WALK)
        warp_trace<true, STATS>(src, n, work, tune, s_stack + threadIdx.x, blockDim.x, stack_cap, err);
    else
        quad_trace<STATS>(src, (uint32_t)n, reinterpret_cast<unsigned int*>(work), tune, s_stack + threadIdx.x, blockDim.x, stack_cap,
                          warp_queues(s_stack, stack_cap), src.work);
    if (STATS) {
        warp_add(stats + 0, src.work.rays);
        warp_add(stats + 1, src.work.boxes);
        warp_add(stats + 2, src.work.tris);
    }
}

using ExtendKernel = void (*)(const RenderScene*, const WfJob*, WfSide, int2*, unsigned long long*, int, TraceTune,
                              unsigned int*, unsigned long long*);

// shadow stage, first half: the closest hit of every connection in the
// shadow queue, through the same warp-persistent loop as extend (filtered by
// the connection's inside / contact objects).  WALK: the reference's own tree
// (launched while a scene without a four-wide tree is in the table)
struct ShadowSrc {
    const RenderScene* __restrict__ scenes;
    const WfJob* __restrict__ jobs;
    WfShadow Q;
    int2* __restrict__ hits;

    __device__ __forceinline__ void fetch(uint64_t id, TraceRay& a) const {
        const float4 o = Q.o[id], d = Q.d[id];
        const int4 ids = Q.ids[id];
        const WfJob& J = jobs[ids.z];
        a.T = &scenes[J.scene].tree;
        a.o = mk(o.x, o.y, o.z);
        a.d = mk(d.x, d.y, d.z);
        a.pf = prune_factor(J.flags);
        a.filt = true;
        a.inside = ids.x;
        a.contact = ids.y;
        a.enough = enough_before(o.w);
    }
    __device__ __forceinline__ void put(uint64_t id, const TraceRay&, const Hit& h) const {
        hits[id] = make_int2(h.slot, __float_as_int(h.t));
    }
    // rays of several scenes share the queue
    __device__ __forceinline__ const TriRec* tris_of(const RayInShared& rays, int from) const {
        return rays.tris_of(from);
    }
    __device__ __forceinline__ void load(uint64_t id, TraceLane& L, uint32_t* stack, int stride) const {
        TraceRay a;
        fetch(id, a);
        load_lane(a, L, stack, stride);
    }
    __device__ __forceinline__ void store(uint64_t id, const TraceLane& L) const {
        hits[id] = make_int2(L.h.slot, __float_as_int(L.h.t));
    }
};

template <bool WALK, int MINB>
__global__ void WR_EXTEND_BOUNDS(MINB)
    k_wf_shadow_trace(const RenderScene* __restrict__ scenes, const WfJob* __restrict__ jobs, WfShadow Q,
                      int2* __restrict__ hits, unsigned long long* __restrict__ work, int stack_cap, TraceTune tune,
                      unsigned int* __restrict__ err) {
    extern __shared__ __align__(16) uint32_t s_stack[];
    const uint64_t n = *Q.count;
    if (n == 0) return;
    ShadowSrc src{scenes, jobs, Q, hits};
    TraceWork none;
    if (WALK)
        warp_trace<true, false>(src, n, work, tune, s_stack + threadIdx.x, blockDim.x, stack_cap, err);
    else
        quad_trace<false>(src, (uint32_t)n, reinterpret_cast<unsigned int*>(work), tune, s_stack + threadIdx.x, blockDim.x, stack_cap,
                          warp_queues(s_stack, stack_cap), none);
}

using ShadowTraceKernel = void (*)(const RenderScene*, const WfJob*, WfShadow, int2*, unsigned long long*, int,
                                   TraceTune, unsigned int*);

// the shadow traversal for a configuration: the extend stage's register cap
static ShadowTraceKernel shadow_trace_kernel(int ctas_per_sm, bool walk) {
    if (walk) return k_wf_shadow_trace<true, 6>;
    if (ctas_per_sm == 0) ctas_per_sm = 6;
    if (ctas_per_sm >= 8) return k_wf_shadow_trace<false, 8>;
    if (ctas_per_sm >= 7) return k_wf_shadow_trace<false, 7>;
    if (ctas_per_sm >= 6) return k_wf_shadow_trace<false, 6>;
    return k_wf_shadow_trace<false, 0>;
}

// the extend kernel for a configuration: register cap from ctas_per_sm
// (0 = the 6-CTA variant: mixed-material scene 1024^2 x 16 spp 15.3 ms, 16.2 with 7, 16.9 with 5, 17.1 with 8)
static ExtendKernel extend_kernel(int ctas_per_sm, bool stats, bool walk) {
    if (walk) return stats ? k_wf_extend<true, true, 6> : k_wf_extend<false, true, 6>;
    if (ctas_per_sm == 0) ctas_per_sm = 6;
    if (ctas_per_sm >= 8) return stats ? k_wf_extend<true, false, 8> : k_wf_extend<false, false, 8>;
    if (ctas_per_sm >= 7) return stats ? k_wf_extend<true, false, 7> : k_wf_extend<false, false, 7>;
    if (ctas_per_sm >= 6) return stats ? k_wf_extend<true, false, 6> : k_wf_extend<false, false, 6>;
    return stats ? k_wf_extend<true, false, 0> : k_wf_extend<false, false, 0>;
}

// shade: one bounce per path; survivors compacted into Y, finished paths to
// the film.  MIS: compiled with the WR_RENDER_NEE_MIS code (launched while a
// job with that flag is in the table).  MED: MED_FLIGHT behind k_wf_track, else
// MED_TRACK while a scene with participating media is (paths of a cancelled job
// may still be inside a heterogeneous medium then), else MED_NONE.
template <bool MIS, int MED>
__global__ void __launch_bounds__(128, 4) k_wf_shade(const RenderScene* __restrict__ scenes,
                                                    const WfJob* __restrict__ jobs,
                                                    WfJobCounters* __restrict__ counters, WfSide X,
                                                    const int2* __restrict__ hits, WfSide Y, WfShadow Q, WfSort B,
                                                    uint32_t capacity, const Flight* __restrict__ flights) {
    // the flights' buckets stand in for the medium's (k_wf_track)
    constexpr int KEYS = MED == MED_FLIGHT ? WF_SORT_KEYS + WF_FLIGHT_KEYS : WF_SORT_KEYS;
    __shared__ uint32_t s_first[KEYS + 1];  // first queue position of each bucket
    if (threadIdx.x == 0) {
        uint32_t a = 0;
        for (int k = 0; k < KEYS; k++) {
            s_first[k] = a;
            if (MED != MED_FLIGHT || k != 1 + WR_MAT_HETEROGENEOUS) a += B.counts[k];
        }
        s_first[KEYS] = a;
    }
    __syncthreads();
    const uint32_t n = s_first[KEYS];
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += step) {  // warp-uniform trip count
        const uint32_t j = base + threadIdx.x;
        const bool valid = j < n;
        uint32_t i = 0;
        if (valid) {  // the j-th path in bucket order
            int k = 0;
#pragma unroll
            for (int kk = 1; kk < KEYS; kk++) k = j >= s_first[kk] ? kk : k;
            const uint32_t at = j - s_first[k];
            i = k < WF_SORT_KEYS ? B.idx[(size_t)k * capacity + at]
                                 : *wf_flight_list(B, capacity, k - WF_SORT_KEYS, at);
        }
        WfPath p;
        bool keep = false, done = false, shadow = false, has_lr = false, mis = false;
        f3 result = mk(0, 0, 0);
        ShadowReq sr;
        LightReq lr;
        if (valid) {
            wf_load(X, i, p);
            const WfJob& J = jobs[p.job];
            const RenderScene& S = scenes[J.scene];
            mis = MIS && (J.flags & WR_RENDER_NEE_MIS) != 0;
            if (mis) wf_load_acc(X, i, p);
            const int2 hv = hits[i];
            Hit h;
            h.slot = hv.x;
            h.t = __int_as_float(hv.y);
            const bool nee = (J.flags & WR_RENDER_NEE) != 0;
            bool nee_here = false;
            PathRng g;
            g.init(J.seed, p.pixel, p.sample, p.dim);
            if (h.slot < 0 && p.cur.contact != CAMERA_OBJ) {
                done = true;  // a scattered ray that escapes ends with zero radiance
                nee_here = nee;
            } else {
                set_hit(S, p.cur, h);
                done = path_advance<MIS, MED>(S, p.cur, p.color, p.prev_d, p.depth, p.st, g, J.max_path_len, J.flags,
                                              result, nee_here, p.mis_pdf, lr, has_lr, flights + i);
            }
            if (nee_here) shadow = nee_prepare(S, p.cur, p.prev_d, p.color, g, sr);
            p.dim = g.dim;
            keep = !done;
            if (done) {
                if (!legal(result)) result = mk(0, 0, 0);
                result = result + p.acc;  // light connections of earlier vertices
                if (!shadow && !has_lr && (result.x != 0.f || result.y != 0.f || result.z != 0.f))
                    film_add(J, p.pixel, result);
            }
        }
        // survivors, compacted into Y
        const uint32_t out = warp_append(&Y.counts[0], keep, 0);
        if (keep) {
            wf_store(Y, out, p);
            if (mis) wf_store_acc(Y, out, p);
        }
        // connections whose visibility the shadow stage decides
        {
            const bool any = shadow || has_lr;
            const uint32_t k = warp_append(Q.count, any, 0);
            if (shadow) {
                Q.o[k] = make_float4(sr.o.x, sr.o.y, sr.o.z, sr.dist);
                Q.d[k] = make_float4(sr.d.x, sr.d.y, sr.d.z, 0.f);
                Q.c[k] = make_float4(sr.contrib.x, sr.contrib.y, sr.contrib.z, __int_as_float(WF_SHADOW_NEE));
                Q.ids[k] = make_int4(sr.inside, sr.contact, p.job, (int)p.pixel);
            } else if (has_lr) {
                Q.o[k] = make_float4(lr.o.x, lr.o.y, lr.o.z, lr.dist);
                Q.d[k] = make_float4(lr.d.x, lr.d.y, lr.d.z, __int_as_float(lr.light));
                Q.c[k] = make_float4(lr.contrib.x, lr.contrib.y, lr.contrib.z,
                                     __int_as_float(keep ? WF_SHADOW_MIS_KEEP : WF_SHADOW_MIS_DONE));
                Q.r[k] = make_float4(result.x, result.y, result.z, __int_as_float((int)out));
                Q.ids[k] = make_int4(lr.inside, lr.contact, p.job, (int)p.pixel);
            }
        }
        // finished-path counts per job, aggregated over the lanes sharing a job
        {
            const unsigned dm = __ballot_sync(0xffffffffu, done);
            if (done) {
                const unsigned same = __match_any_sync(dm, p.job);
                if ((threadIdx.x & 31u) == (unsigned)(__ffs(same) - 1))
                    atomicAdd(&counters[p.job].finished, (unsigned long long)__popc(same));
            }
        }
    }
}

static auto shade_kernel(bool mis, bool media, bool hetero) {
    if (hetero) return mis ? k_wf_shade<true, MED_FLIGHT> : k_wf_shade<false, MED_FLIGHT>;
    if (media) return mis ? k_wf_shade<true, MED_TRACK> : k_wf_shade<false, MED_TRACK>;
    return mis ? k_wf_shade<true, MED_NONE> : k_wf_shade<false, MED_NONE>;
}

// finish: the paths waiting in X run to their ends without returning to the
// bounce loop, one path to a lane, the lanes of a warp together (search_warp).
// Once nothing is left to generate, each iteration of the loop costs the
// latency of its slowest ray and of seven launches however few paths remain;
// here the paths go on side by side.  Same paths, draws and film additions as
// the loop.  MIS: compiled with the WR_RENDER_NEE_MIS code.
// Bound by latency: a warp's turn lasts as long as its slowest ray's search.
// Few paths are therefore spread over all warps, a few lanes to each.
template <bool MIS, int MED>
__global__ void __launch_bounds__(WF_FINISH_BLOCK, MIS ? 3 : 4)
    k_wf_finish(const RenderScene* __restrict__ scenes, const WfJob* __restrict__ jobs,
                WfJobCounters* __restrict__ counters, WfSide X, unsigned int* __restrict__ next, int stack_cap) {
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) uint32_t s_stack[];
    __shared__ WarpLeaves s_leaves[WF_FINISH_BLOCK / 32];
    uint32_t* stack = s_stack + threadIdx.x;
    WarpLeaves& leaves = s_leaves[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t n = X.counts[0] + X.counts[1];
    const uint32_t warps = gridDim.x * (WF_FINISH_BLOCK / 32);
    const uint32_t lanes = min(32u, n / warps + (n % warps != 0));
    bool active = false, dry = lane >= lanes;
    WfPath p;
    p.cur = ray_default();
    p.job = 0;
    PathRng g;
    g.init(0, 0, 0);
    for (;;) {
        const unsigned need = __ballot_sync(FULL, !active && !dry);
        if (need) {
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(next, (unsigned)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (need >> lane & 1u) {
                const uint32_t i = base + __popc(need & ((1u << lane) - 1u));
                if (i < n) {
                    wf_load(X, i, p);
                    const WfJob& J = jobs[p.job];
                    if (MIS && (J.flags & WR_RENDER_NEE_MIS)) wf_load_acc(X, i, p);
                    g.init(J.seed, p.pixel, p.sample, p.dim);
                    active = true;
                } else {
                    dry = true;
                }
            }
        }
        if (!__any_sync(FULL, active)) break;
        const WfJob& J = jobs[p.job];
        const RenderScene& S = scenes[J.scene];
        const float pf = prune_factor(J.flags);
        const bool filtered = p.cur.contact != CAMERA_OBJ;
        const Hit h = search_warp<false>(S.tree, active, p.cur.o, p.cur.d, pf, filtered, p.cur.inside, p.cur.contact,
                                         stack, WF_FINISH_BLOCK, stack_cap, leaves);
        bool done = false, nee_here = false, has_lr = false;
        f3 result = mk(0, 0, 0);
        LightReq lr;
        if (active) {
            if (h.slot < 0 && filtered) {  // a scattered ray that escapes ends with zero radiance
                done = true;
                nee_here = (J.flags & WR_RENDER_NEE) != 0;
            } else {
                set_hit(S, p.cur, h);
                done = path_advance<MIS, MED>(S, p.cur, p.color, p.prev_d, p.depth, p.st, g, J.max_path_len, J.flags,
                                         result, nee_here, p.mis_pdf, lr, has_lr);
            }
        }
        if (MIS && __any_sync(FULL, has_lr)) {  // the light connection of WR_RENDER_NEE_MIS
            const Hit lh = search_warp<false>(S.tree, has_lr, lr.o, lr.d, pf, true, lr.inside, lr.contact, stack,
                                              WF_FINISH_BLOCK, stack_cap, leaves, enough_before(lr.dist));
            if (has_lr && light_req_visible(S, lh, lr)) p.acc = p.acc + lr.contrib;
        }
        if (__any_sync(FULL, nee_here)) {  // the connection of the NEE branch
            ShadowReq sr;
            const bool conn = nee_here && nee_prepare(S, p.cur, p.prev_d, p.color, g, sr);
            const Hit sh = search_warp<false>(S.tree, conn, sr.o, sr.d, pf, true, sr.inside, sr.contact, stack,
                                              WF_FINISH_BLOCK, stack_cap, leaves, enough_before(sr.dist));
            if (nee_here) result = conn && nee_visible(sh, sr.dist) ? sr.contrib : mk(0, 0, 0);
        }
        if (done) {
            if (!legal(result)) result = mk(0, 0, 0);
            result = result + p.acc;
            if (result.x != 0.f || result.y != 0.f || result.z != 0.f) film_add(J, p.pixel, result);
            active = false;
        }
        const unsigned dm = __ballot_sync(FULL, done);
        if (done) {
            const unsigned same = __match_any_sync(dm, p.job);
            if ((int)lane == __ffs(same) - 1) atomicAdd(&counters[p.job].finished, (unsigned long long)__popc(same));
        }
    }
}

// plan: how the free slots of Y are shared out among the jobs this turn.
// One block, one thread per listed job (`order`: admission order).  Each job
// with paths left gets an equal share of the free slots (processor sharing:
// a small request admitted behind a large one starts at once), capped by what
// it has left; slots nobody's share used go to the jobs in admission order.
// With `equal_share` off, every slot goes in admission order (first come,
// first served).  The queue is filled up to *live_cap paths (at most its
// capacity): a word in device memory, so that the serving loop can shorten
// the queue without recapturing the bounce loop.  The plan reserves each job's index range [first, first +
// quota) by advancing its claim counter; the generate kernel then maps queue
// position t to a job and a path index without atomics.  Which paths a job
// renders does not depend on the plan, only when.
__device__ __forceinline__ unsigned long long block_excl_scan(unsigned long long v, unsigned long long* buf) {
    const int k = threadIdx.x;
    buf[k] = v;
    __syncthreads();
    for (int d = 1; d < (int)blockDim.x; d <<= 1) {
        const unsigned long long add = k >= d ? buf[k - d] : 0ull;
        __syncthreads();
        buf[k] += add;
        __syncthreads();
    }
    const unsigned long long incl = buf[k];
    __syncthreads();
    return incl - v;
}

__global__ void __launch_bounds__(WF_MAX_JOBS) k_wf_plan(const WfJob* __restrict__ jobs, const int* __restrict__ order,
                                                          WfJobCounters* __restrict__ counters, WfSide Y,
                                                          uint32_t capacity, const uint32_t* __restrict__ live_cap,
                                                          int equal_share, WfPlan P, volatile WfStatus* status) {
    __shared__ unsigned long long buf[WF_MAX_JOBS];
    __shared__ unsigned long long s_total_q;
    const int n = order[0];
    const int k = threadIdx.x;
    const uint32_t survivors = Y.counts[0];
    const uint32_t cap = min(capacity, *live_cap);
    const unsigned long long free_slots = cap > survivors ? cap - survivors : 0u;
    int j = -1;
    unsigned long long rem = 0, claimed = 0;
    if (k < n) {
        j = order[1 + k];
        const WfJob& J = jobs[j];
        claimed = counters[j].claimed;
        rem = (J.active && claimed < J.total) ? J.total - claimed : 0ull;
    }
    const int active = __syncthreads_count(rem > 0);
    const unsigned long long share = (equal_share && active) ? free_slots / (unsigned long long)active : 0ull;
    const unsigned long long q = rem < share ? rem : share;
    const unsigned long long q_before = block_excl_scan(q, buf);
    if (k == (int)blockDim.x - 1) s_total_q = q_before + q;
    __syncthreads();
    const unsigned long long leftover = free_slots - s_total_q;
    unsigned long long need = rem - q;
    need = need < free_slots ? need : free_slots;
    const unsigned long long need_before = block_excl_scan(need, buf);
    unsigned long long extra = leftover > need_before ? leftover - need_before : 0ull;
    extra = extra < need ? extra : need;
    const unsigned long long quota = q + extra;
    const unsigned long long off = block_excl_scan(quota, buf);
    if (k < n) {
        P.slot[k] = j;
        P.first[k] = claimed;
        P.off[k] = (uint32_t)off;
        if (quota) counters[j].claimed = claimed + quota;
        if (k == 0) {  // what the host waits for, written to its memory
            status->claimed = claimed + quota;
            status->finished = counters[j].finished;
        }
    }
    if (k == n - 1 || (n == 0 && k == 0)) {
        const uint32_t total = n ? (uint32_t)(off + quota) : 0u;
        P.off[n] = total;
        *P.n = n;
        Y.counts[1] = total;
        status->waiting = survivors + total;
        __threadfence_system();
    }
}

// Pixel of the k-th camera path of a sample when paths are generated tile by
// tile: bands of `tile` rows, each cut into tiles of `tile` columns (the last
// band and the last tile of a band may be smaller), rows within a tile.  A
// bijection of [0, W*H); tile 0 is row order.  Neighbouring queue entries
// then hold neighbouring pixels, whose first bounces visit the same nodes.
__device__ __forceinline__ uint32_t tile_pixel(uint32_t k, uint32_t W, uint32_t H, uint32_t tile) {
    if (tile == 0 || tile >= W) return k;
    const uint32_t band = k / (W * tile);
    const uint32_t y0 = band * tile;
    const uint32_t bh = min(tile, H - y0);  // rows in this band
    const uint32_t r = k - band * W * tile;
    const uint32_t tc = r / (tile * bh);     // tile column (the last one may be narrower)
    const uint32_t x0 = tc * tile;
    const uint32_t tw = min(tile, W - x0);
    const uint32_t q = r - tc * tile * bh;
    return (y0 + q / tw) * W + x0 + q % tw;
}

// generate: new camera paths into the free slots of Y as the plan shares
// them out: queue position survivors + t belongs to the job whose planned
// range holds t; the list lives in device memory so the captured graph does
// not change when jobs come and go
// Each block builds WF_GEN_ROWS consecutive records at a time in a
// shared-memory tile and one thread writes the tile with a bulk tensor store
// (cp.async.bulk.tensor through `tmap`, the side's records as a 2-D tensor of
// 32 floats x capacity rows): full 128-byte lines instead of eight 16-byte
// pieces per record from every thread.  The tile's rows past the last new
// path hold stale data and land past the queue's end, which nothing reads;
// the tensor's bounds clip rows past the capacity.
constexpr uint32_t WF_GEN_ROWS = 128;  // = the generate kernel's block size

__global__ void __launch_bounds__(WF_GEN_ROWS) k_wf_generate(const WfJob* __restrict__ jobs, WfPlan P, WfSide Y,
                                                             const __grid_constant__ CUtensorMap tmap) {
    __shared__ __align__(1024) float4 s_tile[WF_GEN_ROWS * WF_REC];  // 16 KiB
    __shared__ uint32_t s_off[WF_MAX_JOBS + 1];
    __shared__ int s_slot[WF_MAX_JOBS];
    __shared__ unsigned long long s_first[WF_MAX_JOBS];
    const int n = *P.n;
    for (int k = threadIdx.x; k <= n; k += blockDim.x) {
        s_off[k] = P.off[k];
        if (k < n) {
            s_slot[k] = P.slot[k];
            s_first[k] = P.first[k];
        }
    }
    __syncthreads();
    const uint32_t total = s_off[n];
    const uint32_t survivors = Y.counts[0];
    const uint32_t tile_addr = (uint32_t)__cvta_generic_to_shared(s_tile);
    for (uint32_t base = blockIdx.x * WF_GEN_ROWS; base < total; base += gridDim.x * WF_GEN_ROWS) {  // block-uniform
        const uint32_t t = base + threadIdx.x;
        if (t < total) {
            int lo = 0, hi = n - 1;  // the last k with s_off[k] <= t (its range is not empty)
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (s_off[mid] <= t) lo = mid;
                else hi = mid - 1;
            }
            const int jid = s_slot[lo];
            const unsigned long long idx = s_first[lo] + (t - s_off[lo]);
            const WfJob& J = jobs[jid];
            WfPath p;
            p.job = jid;
            p.pixel = tile_pixel((uint32_t)(idx % J.npix), J.cam.width, J.cam.height, J.tile);
            p.sample = J.s0 + (uint32_t)(idx / J.npix);
            PathRng g;
            g.init(J.seed, p.pixel, p.sample);
            p.cur = camera_ray(J.cam, p.pixel, g);
            p.dim = g.dim;
            p.color = mk(1, 1, 1);
            p.prev_d = mk(0, 0, 0);
            p.depth = 0;
            p.st.reset(p.cur.inside);
            p.mis_pdf = 0.f;
            p.acc = mk(0, 0, 0);
            wf_store_at(s_tile + WF_REC * threadIdx.x, survivors + t, p);
            if (J.flags & WR_RENDER_NEE_MIS) wf_store_acc(Y, survivors + t, p);
        }
        // the tile's generic-proxy writes before the tensor unit reads it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            // row survivors + base, column 0: a 16-byte-aligned start (x = 0)
            asm volatile(
                "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];\n\t"
                "cp.async.bulk.commit_group;\n\t"
                "cp.async.bulk.wait_group.read 0;"
                :
                : "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(0), "r"((int)(survivors + base)), "r"(tile_addr)
                : "memory");
        }
        __syncthreads();  // the tile may be written again
    }
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------------------
// engine
// ---------------------------------------------------------------------------
struct WfEngine {
    WfConfig cfg;
    DeviceBuffer side_mem[2], hits, flights, scenes, jobs, order, counters, work, err_word, shadow_mem, sort_mem, plan_mem;
    WfSide side[2];
    CUtensorMap rec_map[2];  // each side's records as a 2-D tensor (k_wf_generate's bulk stores)
    WfPlan plan{};
    int equal_share = 1;  // the plan's policy (captured into the graph)
    DeviceBuffer live_cap;     // uint32: paths the plan fills the queue up to
    uint32_t live_cap_host = 0;
    WfShadow shadow{};
    WfSort sort{};
    int grid_sort = 0, grid_track = 0;
    int grid_shadow = 0;
    std::vector<const RenderData*> scene_of;  // host mirror of the scene table
    std::vector<RenderScene> scene_tab;
    std::vector<WfJob> job_tab;               // host mirror of the job slots
    std::vector<int> order_host;               // [n, slot...]
    int stack_cap = 0;       // the reference walk's stack (tree depth + 3)
    int quad_cap = 0;        // the search's stack
    int grid_extend = 0, grid_walk = 0, grid_shade = 0, grid_gen = 0;
    size_t smem_extend = 0, smem_walk = 0;
    // The bounce loop captured for each set of kernels that the jobs so far have
    // asked for (kind), so that a program that alternates between scenes does
    // not capture anew on each call (8x8 calls with and without media in turn
    // 398 and 502 us, 243 and 334 this way, as alone); dropped when the stacks grow.
    std::map<uint32_t, cudaGraphExec_t> graphs;
    int graph_caps = -1;
    bool mis_any = false;  // a job in the table has WR_RENDER_NEE_MIS: the shade stage with that code
    bool hetero_any = false;  // a job's scene has a heterogeneous medium: the track stage
    bool media_any = false;  // a job's scene has participating media: the shading kernels with that code
    bool bare_any = false;   // a job's scene has no four-wide tree: the walk of the reference's in both stages
    bool walk_any = false;   // or a job has WR_RENDER_EXACT_TRAVERSAL: in the extend stage
    bool conn_any = true;  // a job in the table connects to lights (NEE or MIS): the shadow stage is in the loop
    uint32_t kind() const {
        return (uint32_t)mis_any | (uint32_t)conn_any << 1 | (uint32_t)walk_any << 2 | (uint32_t)bare_any << 3 |
               (uint32_t)media_any << 4 | (uint32_t)hetero_any << 5 | (uint32_t)(equal_share != 0) << 6;
    }
    void drop_graphs() {
        for (auto& g : graphs) cudaGraphExecDestroy(g.second);
        graphs.clear();
    }
    int launches_per_iteration() const { return (conn_any ? 8 : 6) + (hetero_any ? 1 : 0); }
    WfJobCounters* host_counters = nullptr;  // pinned
    WfStatus* status = nullptr;              // pinned and mapped: written by k_wf_plan
    cudaEvent_t turn[2] = {};                // the end of the last two graph replays of a render
    int grid_finish[4] = {};                 // k_wf_finish without and with the light connections, then with media
    ~WfEngine() {
        drop_graphs();
        if (host_counters) cudaFreeHost(host_counters);
        if (status) cudaFreeHost(status);
        for (cudaEvent_t e : turn)
            if (e) cudaEventDestroy(e);
    }
};

const WfConfig& wf_config(const WfEngine* E) { return E->cfg; }

// side k's records as a tensor of 32 floats x capacity rows (128-byte rows),
// written in WF_GEN_ROWS x 32 boxes from shared memory
static PFN_cuTensorMapEncodeTiled_v12000 lookup_encode_tiled() {
    cudaDriverEntryPointQueryResult q{};
    void* fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
        return nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
}

static int map_side(wr_ctx* ctx, WfEngine* E, int k) {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = lookup_encode_tiled();  // once, thread-safe
    if (!encode) return set_error(ctx, WR_ERR_UNSUPPORTED, "the driver has no cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {4 * WF_REC, E->cfg.capacity};
    const cuuint64_t strides[1] = {sizeof(float4) * WF_REC};
    const cuuint32_t box[2] = {4 * WF_REC, WF_GEN_ROWS};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode(&E->rec_map[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, E->side[k].rec, dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(ctx, WR_ERR_INTERNAL, "cuTensorMapEncodeTiled failed for the path records");
    return WR_OK;
}

static int alloc_side(wr_ctx* ctx, WfEngine* E, int k) {
    const size_t Q = E->cfg.capacity;
    const size_t bytes = Q * (WF_REC + 1) * sizeof(float4) + 256;
    WR_CUDA(ctx, E->side_mem[k].reserve(bytes));
    char* p = E->side_mem[k].as<char>();
    WfSide& S = E->side[k];
    S.rec = reinterpret_cast<float4*>(p);
    S.a5 = S.rec + (size_t)WF_REC * Q;
    S.counts = reinterpret_cast<unsigned int*>(S.a5 + Q);
    WR_CUDA(ctx, cudaMemset(S.counts, 0, 2 * sizeof(unsigned int)));
    return WR_OK;
}

int wf_engine_get(wr_ctx* ctx, const WfConfig& cfg, WfEngine** out) {
    // one engine per context, rebuilt when the configuration changes
    WfEngine* cur = static_cast<WfEngine*>(ctx->wavefront.get());
    if (cur && cur->cfg.capacity == cfg.capacity && cur->cfg.extend_block == cfg.extend_block &&
        cur->cfg.shade_block == cfg.shade_block && cur->cfg.ctas_per_sm == cfg.ctas_per_sm &&
        cur->cfg.iters_per_graph == cfg.iters_per_graph && cur->cfg.trace.refill_min == cfg.trace.refill_min &&
        cur->cfg.trace.steps == cfg.trace.steps &&
        cur->cfg.trace.leaf_min == cfg.trace.leaf_min) {
        cur->cfg.drain_paths = cfg.drain_paths;  // host-side only
        cur->cfg.pixel_tile = cfg.pixel_tile;    // a job field, set when jobs are written
        *out = cur;
        return WR_OK;
    }
    if (cur) {
        WR_CUDA(ctx, cudaDeviceSynchronize());
        ctx->wavefront.reset();
    }
    auto E = std::make_shared<WfEngine>();
    E->cfg = cfg;
    for (int k = 0; k < 2; k++) {
        int rc = alloc_side(ctx, E.get(), k);
        if (rc == WR_OK) rc = map_side(ctx, E.get(), k);
        if (rc != WR_OK) return rc;
    }
    WR_CUDA(ctx, E->hits.reserve(sizeof(int2) * (size_t)cfg.capacity));
    WR_CUDA(ctx, E->sort_mem.reserve(sizeof(uint32_t) * ((size_t)WF_SORT_KEYS * cfg.capacity + 64)));
    E->sort.counts = E->sort_mem.as<unsigned int>();
    E->sort.idx = E->sort.counts + 64;
    WR_CUDA(ctx, cudaMemset(E->sort.counts, 0, sizeof(unsigned int) * (WF_SORT_KEYS + WF_FLIGHT_KEYS)));
    E->grid_sort = ctx->num_sms * 4;
    E->grid_track = ctx->num_sms * 7;
    {
        const size_t Q = cfg.capacity;
        WR_CUDA(ctx, E->shadow_mem.reserve(Q * (4 * sizeof(float4) + sizeof(int4)) + 256));
        char* p = E->shadow_mem.as<char>();
        E->shadow.o = reinterpret_cast<float4*>(p);
        E->shadow.d = E->shadow.o + Q;
        E->shadow.c = E->shadow.d + Q;
        E->shadow.r = E->shadow.c + Q;
        E->shadow.ids = reinterpret_cast<int4*>(E->shadow.r + Q);
        E->shadow.count = reinterpret_cast<unsigned int*>(E->shadow.ids + Q);
        WR_CUDA(ctx, cudaMemset(E->shadow.count, 0, sizeof(unsigned int)));
    }
    WR_CUDA(ctx, E->scenes.reserve(sizeof(RenderScene) * WF_MAX_SCENES));
    WR_CUDA(ctx, E->jobs.reserve(sizeof(WfJob) * WF_MAX_JOBS));
    WR_CUDA(ctx, cudaMemset(E->jobs.p, 0, sizeof(WfJob) * WF_MAX_JOBS));
    WR_CUDA(ctx, E->order.reserve(sizeof(int) * (WF_MAX_JOBS + 1)));
    WR_CUDA(ctx, cudaMemset(E->order.p, 0, sizeof(int) * (WF_MAX_JOBS + 1)));
    WR_CUDA(ctx, E->plan_mem.reserve(sizeof(unsigned long long) * WF_MAX_JOBS + sizeof(int) * WF_MAX_JOBS +
                                     sizeof(uint32_t) * (WF_MAX_JOBS + 1) + 64));
    E->plan.first = E->plan_mem.as<unsigned long long>();
    E->plan.slot = reinterpret_cast<int*>(E->plan.first + WF_MAX_JOBS);
    E->plan.off = reinterpret_cast<uint32_t*>(E->plan.slot + WF_MAX_JOBS);
    E->plan.n = reinterpret_cast<int*>(E->plan.off + WF_MAX_JOBS + 1);
    WR_CUDA(ctx, E->counters.reserve(sizeof(WfJobCounters) * WF_MAX_JOBS));
    WR_CUDA(ctx, cudaMemset(E->counters.p, 0, sizeof(WfJobCounters) * WF_MAX_JOBS));
    WR_CUDA(ctx, E->work.reserve(3 * sizeof(unsigned long long)));
    WR_CUDA(ctx, E->err_word.reserve(sizeof(unsigned int)));
    WR_CUDA(ctx, E->live_cap.reserve(sizeof(uint32_t)));
    E->live_cap_host = cfg.capacity;
    WR_CUDA(ctx, cudaMemcpy(E->live_cap.p, &E->live_cap_host, sizeof(uint32_t), cudaMemcpyHostToDevice));
    WR_CUDA(ctx, cudaMemset(E->err_word.p, 0, sizeof(unsigned int)));
    // the job counters, then one extra record for the queue counts of side 0
    WR_CUDA(ctx, cudaMallocHost(&E->host_counters, sizeof(WfJobCounters) * (WF_MAX_JOBS + 1)));
    WR_CUDA(ctx, cudaHostAlloc(&E->status, sizeof(WfStatus), cudaHostAllocMapped));
    *E->status = WfStatus{};
    for (cudaEvent_t& e : E->turn) WR_CUDA(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    E->job_tab.assign(WF_MAX_JOBS, WfJob{});
    E->order_host.assign(1, 0);
    // persistent grids from the occupancy calculator
    int per_sm = 0;
    WR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shade_kernel(false, true, true), cfg.shade_block, 0));
    if (cfg.ctas_per_sm > 0) per_sm = std::min(per_sm, cfg.ctas_per_sm);
    E->grid_shade = ctx->num_sms * std::max(1, per_sm);
    WR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_wf_generate, WF_GEN_ROWS, 0));
    E->grid_gen = ctx->num_sms * std::max(1, per_sm);
    *out = E.get();
    ctx->wavefront = E;
    return WR_OK;
}

int wf_reserve_flights(wr_ctx* ctx, WfEngine* E) {
    WR_CUDA(ctx, E->flights.reserve(sizeof(Flight) * (size_t)E->cfg.capacity));
    return WR_OK;
}

int wf_set_config(wr_ctx* ctx, const WfConfig& cfg) {
    WfEngine* E = nullptr;
    return wf_engine_get(ctx, cfg, &E);
}

// slot of a scene in the device scene table (nullptr entries are free)
static int scene_slot(wr_ctx* ctx, WfEngine* E, const RenderData* rd, int* slot) {
    for (size_t k = 0; k < E->scene_of.size(); k++)
        if (E->scene_of[k] == rd) {
            *slot = (int)k;
            return WR_OK;
        }
    for (size_t k = 0; k < E->scene_of.size(); k++)
        if (!E->scene_of[k]) {
            E->scene_of[k] = rd;
            *slot = (int)k;
            return WR_OK;
        }
    if (E->scene_of.size() >= WF_MAX_SCENES) return set_error(ctx, WR_ERR_BUSY, "too many scenes in flight");
    E->scene_of.push_back(rd);
    *slot = (int)E->scene_of.size() - 1;
    return WR_OK;
}

// a released scene must not stay in the table: a later scene could be
// allocated at the same host address and match the stale device entry
void wf_forget_scene(wr_ctx* ctx, const RenderData* rd) {
    WfEngine* E = static_cast<WfEngine*>(ctx->wavefront.get());
    if (!E || !rd) return;
    for (auto& p : E->scene_of)
        if (p == rd) p = nullptr;
}

int wf_update_jobs(wr_ctx* ctx, WfEngine* E, const std::vector<WfSlotUpdate>& updates, const std::vector<int>& order,
                   cudaStream_t s) {
    if (order.size() > WF_MAX_JOBS) return set_error(ctx, WR_ERR_BUSY, "too many jobs in flight");
    bool scenes_changed = false;
    for (const WfSlotUpdate& u : updates) {
        if (u.slot < 0 || u.slot >= (int)WF_MAX_JOBS) return set_error(ctx, WR_ERR_INTERNAL, "bad job slot");
        WfJob j = u.jh.job;
        j.tile = (uint32_t)std::max(0, E->cfg.pixel_tile);
        if (u.jh.rd) {
            int rc = scene_slot(ctx, E, u.jh.rd, &j.scene);
            if (rc != WR_OK) return rc;
            scenes_changed = true;  // (re)copy the entry: its RenderData may be new at a reused address
        } else {
            j.scene = E->job_tab[u.slot].scene;
        }
        E->job_tab[u.slot] = j;
        WR_CUDA(ctx, cudaMemcpyAsync(E->jobs.as<WfJob>() + u.slot, &E->job_tab[u.slot], sizeof(WfJob),
                                     cudaMemcpyHostToDevice, s));
        if (u.reset_counters)
            WR_CUDA(ctx, cudaMemsetAsync(E->counters.as<WfJobCounters>() + u.slot, 0, sizeof(WfJobCounters), s));
    }
    if (scenes_changed) {
        E->scene_tab.resize(E->scene_of.size());
        int cap = 8, quad_cap = 8;
        for (size_t k = 0; k < E->scene_of.size(); k++) {
            if (!E->scene_of[k]) {
                std::memset(&E->scene_tab[k], 0, sizeof(RenderScene));
                continue;
            }
            E->scene_tab[k] = RenderDataView::scene(E->scene_of[k]);
            cap = std::max(cap, (int)E->scene_tab[k].tree.max_depth + 3);
            quad_cap = std::max(quad_cap, quad_stack_cap(E->scene_tab[k].tree));
        }
        WR_CUDA(ctx, cudaMemcpyAsync(E->scenes.p, E->scene_tab.data(), sizeof(RenderScene) * E->scene_tab.size(),
                                     cudaMemcpyHostToDevice, s));
        if (cap > E->stack_cap || quad_cap > E->quad_cap) {
            const int block = E->cfg.extend_block;
            E->stack_cap = std::max(cap, E->stack_cap);
            E->quad_cap = std::max(quad_cap, E->quad_cap);
            E->smem_walk = (size_t)E->stack_cap * block * sizeof(uint32_t);
            E->smem_extend = quad_smem(E->quad_cap, block);
            if (E->smem_walk > 200 * 1024) return set_error(ctx, WR_ERR_UNSUPPORTED, "tree too deep for the stack");
            if (E->smem_walk > 48 * 1024) {
                WR_CUDA(ctx, cudaFuncSetAttribute(shadow_trace_kernel(E->cfg.ctas_per_sm, true),
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)E->smem_walk));
                for (bool st : {false, true})
                    WR_CUDA(ctx, cudaFuncSetAttribute(extend_kernel(E->cfg.ctas_per_sm, st, true),
                                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      (int)E->smem_walk));
            }
            int per_sm = 0;
            WR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                             &per_sm, extend_kernel(E->cfg.ctas_per_sm, false, false), block, E->smem_extend));
            if (E->cfg.ctas_per_sm > 0) per_sm = std::min(per_sm, E->cfg.ctas_per_sm);
            E->grid_extend = ctx->num_sms * std::max(1, per_sm);
            WR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                             &per_sm, extend_kernel(E->cfg.ctas_per_sm, false, true), block, E->smem_walk));
            if (E->cfg.ctas_per_sm > 0) per_sm = std::min(per_sm, E->cfg.ctas_per_sm);
            E->grid_walk = ctx->num_sms * std::max(1, per_sm);
            WR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_wf_shadow, 128, 0));
            E->grid_shadow = ctx->num_sms * std::max(1, per_sm);
        }
    }
    // the shade stage compiled with the light-connection code only while a job needs it
    // and the shadow stage only while a job can queue a connection
    bool mis_any = false, conn_any = false, walk_any = false, bare_any = false, media_any = false, hetero_any = false;
    for (int slot : order) {
        if (!E->job_tab[slot].active) continue;
        if (E->job_tab[slot].flags & WR_RENDER_NEE_MIS) mis_any = true;
        if (E->job_tab[slot].flags & WR_RENDER_EXACT_TRAVERSAL) walk_any = true;
        if (const RenderData* rd = E->scene_of[E->job_tab[slot].scene]) {
            if (!RenderDataView::scene(rd).tree.quads) walk_any = bare_any = true;
            media_any |= RenderDataView::media(rd);
            hetero_any |= RenderDataView::hetero(rd);
        }
        if (E->job_tab[slot].flags & (WR_RENDER_NEE | WR_RENDER_NEE_MIS)) conn_any = true;
    }
    if (hetero_any) {  // before the loop with the track stage is captured
        const int rc = wf_reserve_flights(ctx, E);
        if (rc != WR_OK) return rc;
    }
    E->hetero_any = hetero_any;
    E->walk_any = walk_any;
    E->bare_any = bare_any;
    E->media_any = media_any;
    E->mis_any = mis_any;
    E->conn_any = conn_any;
    E->order_host.assign(1, (int)order.size());
    E->order_host.insert(E->order_host.end(), order.begin(), order.end());
    WR_CUDA(ctx, cudaMemcpyAsync(E->order.p, E->order_host.data(), sizeof(int) * E->order_host.size(),
                                 cudaMemcpyHostToDevice, s));
    // (copies from pageable memory: the calls have read the host mirrors when they return)
    return WR_OK;
}

// one bounce iteration; `ev` (5 events, profiling only) brackets the stages
static void enqueue_iteration(WfEngine* E, int x, cudaStream_t s, cudaEvent_t* ev = nullptr,
                              unsigned long long* stats = nullptr) {
    const int y = 1 - x;
    const RenderScene* scenes = E->scenes.as<RenderScene>();
    const WfJob* jobs = E->jobs.as<WfJob>();
    WfJobCounters* cnt = E->counters.as<WfJobCounters>();
    k_wf_reset<<<1, 1, 0, s>>>(E->side[y], E->work.as<unsigned long long>(), E->shadow.count, E->sort);
    if (ev) cudaEventRecord(ev[0], s);
    extend_kernel(E->cfg.ctas_per_sm, stats != nullptr, E->walk_any)
        <<<E->walk_any ? E->grid_walk : E->grid_extend, E->cfg.extend_block,
           E->walk_any ? E->smem_walk : E->smem_extend, s>>>(
            scenes, jobs, E->side[x], E->hits.as<int2>(), E->work.as<unsigned long long>(),
            E->walk_any ? E->stack_cap : E->quad_cap, E->cfg.trace, E->err_word.as<unsigned int>(), stats);
    if (ev) cudaEventRecord(ev[1], s);
    k_wf_sort<<<E->grid_sort, WF_SORT_BLOCK, 0, s>>>(scenes, jobs, E->side[x], E->hits.as<int2>(), E->sort, E->cfg.capacity);
    if (E->hetero_any)
        k_wf_track<<<E->grid_track, WF_TRACK_BLOCK, 0, s>>>(scenes, jobs, E->side[x], E->hits.as<int2>(), E->sort,
                                                            E->cfg.capacity, E->flights.as<Flight>(),
                                                            E->work.as<unsigned int>() + 4);
    shade_kernel(E->mis_any, E->media_any, E->hetero_any)<<<E->grid_shade, E->cfg.shade_block, 0, s>>>(scenes, jobs, cnt, E->side[x], E->hits.as<int2>(),
                                                            E->side[y], E->shadow, E->sort, E->cfg.capacity,
                                                            E->flights.as<Flight>());
    if (ev) cudaEventRecord(ev[2], s);
    if (E->conn_any) {  // the connections' closest hits go into E->hits, which shade has read
        shadow_trace_kernel(E->cfg.ctas_per_sm, E->bare_any)
            <<<E->bare_any ? E->grid_walk : E->grid_extend, E->cfg.extend_block,
               E->bare_any ? E->smem_walk : E->smem_extend, s>>>(
                scenes, jobs, E->shadow, E->hits.as<int2>(), E->work.as<unsigned long long>() + 1,
                E->bare_any ? E->stack_cap : E->quad_cap, E->cfg.trace, E->err_word.as<unsigned int>());
        k_wf_shadow<<<E->grid_shadow, 128, 0, s>>>(scenes, jobs, E->shadow, E->hits.as<int2>(), E->side[y]);
    }
    if (ev) cudaEventRecord(ev[3], s);
    k_wf_plan<<<1, WF_MAX_JOBS, 0, s>>>(jobs, E->order.as<int>(), cnt, E->side[y], E->cfg.capacity,
                                        E->live_cap.as<uint32_t>(), E->equal_share,
                                        E->plan, E->status);
    k_wf_generate<<<E->grid_gen, WF_GEN_ROWS, 0, s>>>(jobs, E->plan, E->side[y], E->rec_map[y]);
    if (ev) cudaEventRecord(ev[4], s);
}

// the first camera paths of a render into the empty side 0
static void enqueue_first(WfEngine* E, cudaStream_t s) {
    k_wf_reset<<<1, 1, 0, s>>>(E->side[0], E->work.as<unsigned long long>(), E->shadow.count, E->sort);
    k_wf_plan<<<1, WF_MAX_JOBS, 0, s>>>(E->jobs.as<WfJob>(), E->order.as<int>(), E->counters.as<WfJobCounters>(),
                                        E->side[0], E->cfg.capacity, E->live_cap.as<uint32_t>(), E->equal_share,
                                        E->plan, E->status);
    k_wf_generate<<<E->grid_gen, WF_GEN_ROWS, 0, s>>>(E->jobs.as<WfJob>(), E->plan, E->side[0], E->rec_map[0]);
}

// wr_profile_render: the render of render_wavefront with eager launches
int profile_wavefront(wr_ctx* ctx, RenderData& rd, const RenderParams& P, uint32_t spp_offset, uint32_t spp,
                      float* film, wr_render_profile* out) {
    if (ctx->serving) return set_error(ctx, WR_ERR_BUSY, "the serving loop owns the wavefront queues");
    WfEngine* E = nullptr;
    int rc = wf_engine_get(ctx, wf_tuned_config(ctx), &E);
    if (rc != WR_OK) return rc;
    cudaStream_t s = ctx->stream;
    if ((rc = wf_set_live_cap(ctx, E, wf_config(E).capacity, s)) != WR_OK) return rc;
    const RenderScene& S = RenderDataView::scene(&rd);
    WfSlotUpdate u;
    u.slot = 0;
    u.jh.rd = &rd;
    u.jh.job = make_job(S, S.cam, P.seed, spp_offset, spp, P.max_path_len, P.flags, film, nullptr);
    u.reset_counters = true;
    if ((rc = wf_update_jobs(ctx, E, {u}, {0}, s)) != WR_OK) return rc;
    if ((rc = wf_reset_queues(ctx, E, s)) != WR_OK) return rc;
    DeviceBuffer st;
    WR_CUDA(ctx, st.reserve(4 * sizeof(unsigned long long)));
    WR_CUDA(ctx, cudaMemsetAsync(st.p, 0, 4 * sizeof(unsigned long long), s));
    cudaEvent_t ev[5], t0, t1;
    for (auto& e : ev) WR_CUDA(ctx, cudaEventCreate(&e));
    WR_CUDA(ctx, cudaEventCreate(&t0));
    WR_CUDA(ctx, cudaEventCreate(&t1));
    std::memset(out, 0, sizeof *out);
    std::vector<WfJobCounters> c;
    const unsigned long long total = u.jh.job.total;
    cudaEventRecord(t0, s);
    int x = 0;
    uint32_t queued = 0;  // rays waiting in side x
    for (uint64_t it = 0;; it++) {
        enqueue_iteration(E, x, s, ev, st.as<unsigned long long>());
        ctx->kernel_launches += E->launches_per_iteration();
        x = 1 - x;
        WR_CUDA(ctx, cudaEventSynchronize(ev[4]));
        float a = 0, b = 0, cc = 0, d = 0;
        cudaEventElapsedTime(&a, ev[0], ev[1]);
        cudaEventElapsedTime(&b, ev[1], ev[2]);
        cudaEventElapsedTime(&cc, ev[2], ev[3]);
        cudaEventElapsedTime(&d, ev[3], ev[4]);
        out->ms_extend += a;
        out->ms_shade += b;
        out->ms_shadow += cc;
        out->ms_generate += d;
        if (it < 32) {
            out->iter_rays[it] = queued;
            out->iter_extend_ms[it] = a;
            out->iter_shade_ms[it] = b;
        }
        out->iterations++;
        uint32_t waiting = 0;
        if ((rc = wf_read_counters(ctx, E, c, s, &waiting, x)) != WR_OK) break;
        queued = waiting;
        if (c[0].finished >= total) break;
        if (c[0].claimed >= total && waiting <= E->cfg.drain_threshold(RenderDataView::hetero(&rd))) {
            cudaEventRecord(ev[0], s);
            if ((rc = wf_finish(ctx, E, x, s)) != WR_OK) break;
            cudaEventRecord(ev[1], s);
            WR_CUDA(ctx, cudaEventSynchronize(ev[1]));
            float dm = 0;
            cudaEventElapsedTime(&dm, ev[0], ev[1]);
            out->ms_drain = dm;
            out->drained_paths = waiting;
            if ((rc = wf_read_counters(ctx, E, c, s)) != WR_OK) break;
            if (c[0].finished < total) rc = set_error(ctx, WR_ERR_INTERNAL, "wavefront drain left paths");
            break;
        }
        if (it > 100000) {
            rc = set_error(ctx, WR_ERR_TIMEOUT, "wavefront did not drain");
            break;
        }
    }
    cudaEventRecord(t1, s);
    cudaEventSynchronize(t1);
    float tot = 0;
    cudaEventElapsedTime(&tot, t0, t1);
    out->ms_total = tot;
    unsigned long long h[4] = {0, 0, 0, 0};
    cudaMemcpy(h, st.p, sizeof h, cudaMemcpyDeviceToHost);
    out->rays = h[0];
    out->box_tests = h[1];
    out->tri_tests = h[2];
    out->paths = total;
    for (auto& e : ev) cudaEventDestroy(e);
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    u.jh.job.active = 0;
    u.reset_counters = false;
    if (rc == WR_OK) rc = wf_update_jobs(ctx, E, {u}, {}, s);
    return rc;
}

int wf_launch(wr_ctx* ctx, WfEngine* E, cudaStream_t s) {
    if (E->stack_cap == 0) return set_error(ctx, WR_ERR_INTERNAL, "wavefront launched without a scene");
    const int caps = E->stack_cap << 8 | E->quad_cap;
    if (E->graph_caps != caps) {
        if (!E->graphs.empty()) WR_CUDA(ctx, cudaStreamSynchronize(s));  // a replay may still run
        E->drop_graphs();
        E->graph_caps = caps;
    }
    cudaGraphExec_t& graph = E->graphs[E->kind()];
    if (!graph) {
        cudaStream_t cap;
        WR_CUDA(ctx, cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            for (int it = 0; it < E->cfg.iters_per_graph; it++) {
                enqueue_iteration(E, 0, cap);
                enqueue_iteration(E, 1, cap);
            }
            e = cudaStreamEndCapture(cap, &g);
        }
        cudaStreamDestroy(cap);
        if (e != cudaSuccess) return cuda_error(ctx, e, "capturing the bounce loop");
        e = cudaGraphInstantiate(&graph, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            graph = nullptr;
            return cuda_error(ctx, e, "instantiating the bounce loop");
        }
    }
    WR_CUDA(ctx, cudaGraphLaunch(graph, s));
    // reset, extend, sort, [track,] shade, [shadow trace, shadow,] plan, generate
    ctx->kernel_launches += (uint64_t)E->launches_per_iteration() * 2 * E->cfg.iters_per_graph;
    return WR_OK;
}

int wf_read_counters(wr_ctx* ctx, WfEngine* E, std::vector<WfJobCounters>& out, cudaStream_t s, uint32_t* waiting,
                     int side) {
    out.resize(WF_MAX_JOBS);
    WR_CUDA(ctx, cudaMemcpyAsync(E->host_counters, E->counters.p, sizeof(WfJobCounters) * WF_MAX_JOBS,
                                 cudaMemcpyDeviceToHost, s));
    unsigned int* q = reinterpret_cast<unsigned int*>(E->host_counters + WF_MAX_JOBS);
    if (waiting)
        WR_CUDA(ctx, cudaMemcpyAsync(q, E->side[side].counts, 2 * sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    WR_CUDA(ctx, cudaStreamSynchronize(s));
    std::memcpy(out.data(), E->host_counters, sizeof(WfJobCounters) * WF_MAX_JOBS);
    if (waiting) *waiting = q[0] + q[1];
    return WR_OK;
}

int wf_finish(wr_ctx* ctx, WfEngine* E, int side, cudaStream_t s) {
    const auto kern = E->media_any ? (E->mis_any ? k_wf_finish<true, MED_TRACK> : k_wf_finish<false, MED_TRACK>)
                                   : (E->mis_any ? k_wf_finish<true, MED_NONE> : k_wf_finish<false, MED_NONE>);
    const size_t smem = (size_t)E->quad_cap * WF_FINISH_BLOCK * sizeof(uint32_t);
    int& grid = E->grid_finish[E->mis_any + 2 * E->media_any];
    if (!grid) {
        int per_sm = 0;
        WR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WF_FINISH_BLOCK, smem));
        grid = ctx->num_sms * std::max(1, per_sm);
    }
    WR_CUDA(ctx, cudaMemsetAsync(E->work.p, 0, sizeof(unsigned long long), s));
    kern<<<grid, WF_FINISH_BLOCK, smem, s>>>(E->scenes.as<RenderScene>(), E->jobs.as<WfJob>(),
                                             E->counters.as<WfJobCounters>(), E->side[side],
                                             E->work.as<unsigned int>(), E->quad_cap);
    WR_CUDA(ctx, cudaGetLastError());
    ctx->kernel_launches++;
    return WR_OK;
}

int wf_error_word(wr_ctx* ctx, WfEngine* E, unsigned int* herr, cudaStream_t s) {
    WR_CUDA(ctx, cudaMemcpyAsync(herr, E->err_word.p, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    WR_CUDA(ctx, cudaStreamSynchronize(s));
    return WR_OK;
}

int wf_set_equal_share(wr_ctx* ctx, WfEngine* E, bool on) {
    (void)ctx;
    E->equal_share = on;  // a kernel argument of the captured loop: part of kind()
    return WR_OK;
}

int wf_set_live_cap(wr_ctx* ctx, WfEngine* E, uint32_t paths, cudaStream_t s) {
    paths = std::max<uint32_t>(1, std::min(paths, E->cfg.capacity));
    if (paths == E->live_cap_host) return WR_OK;
    E->live_cap_host = paths;
    // from pageable memory: the call has read `paths` when it returns
    WR_CUDA(ctx, cudaMemcpyAsync(E->live_cap.p, &paths, sizeof(uint32_t), cudaMemcpyHostToDevice, s));
    return WR_OK;
}

uint32_t wf_live_cap(const WfEngine* E) { return E->live_cap_host; }

int wf_reset_queues(wr_ctx* ctx, WfEngine* E, cudaStream_t s) {
    for (int k = 0; k < 2; k++) WR_CUDA(ctx, cudaMemsetAsync(E->side[k].counts, 0, 2 * sizeof(unsigned int), s));
    return WR_OK;
}

WfJob make_job(const RenderScene& S, const CamParams& cam, uint64_t seed, uint32_t s0, uint32_t spp,
               uint32_t max_path_len, uint32_t flags, float* film, float* film2) {
    WfJob j;
    std::memset(&j, 0, sizeof j);
    (void)S;
    j.active = 1;
    j.cam = cam;
    j.seed = seed;
    j.s0 = s0;
    j.spp = spp;
    j.max_path_len = max_path_len;
    j.flags = flags;
    j.npix = cam.width * cam.height;
    j.total = (unsigned long long)j.npix * spp;
    j.film = film;
    j.film2 = film2;
    return j;
}

int render_wavefront(wr_ctx* ctx, RenderData& rd, const RenderParams& P, uint32_t spp_offset, uint32_t spp,
                     float* film, float* film2, cudaStream_t s) {
    if (ctx->serving) return set_error(ctx, WR_ERR_BUSY, "the serving loop owns the wavefront queues");
    WfEngine* E = nullptr;
    int rc = wf_engine_get(ctx, wf_tuned_config(ctx), &E);
    if (rc != WR_OK) return rc;
    if ((rc = wf_set_live_cap(ctx, E, wf_config(E).capacity, s)) != WR_OK) return rc;  // the whole queue
    const RenderScene& S = RenderDataView::scene(&rd);
    WfSlotUpdate u;
    u.slot = 0;
    u.jh.rd = &rd;
    u.jh.job = make_job(S, S.cam, P.seed, spp_offset, spp, P.max_path_len, P.flags, film, film2);
    u.reset_counters = true;
    rc = wf_update_jobs(ctx, E, {u}, {0}, s);
    if (rc != WR_OK) return rc;
    if ((rc = wf_reset_queues(ctx, E, s)) != WR_OK) return rc;
    const unsigned long long total = u.jh.job.total;
    const uint32_t few = E->cfg.drain_threshold(RenderDataView::hetero(&rd));
    volatile WfStatus* st = E->status;
    st->claimed = st->finished = 0;
    st->waiting = 0;
    enqueue_first(E, s);
    ctx->kernel_launches += 3;
    bool finished = false;
    if (total <= few && total <= E->cfg.capacity) {  // every path is in the queue
        if ((rc = wf_finish(ctx, E, 0, s)) != WR_OK) return rc;
    } else {
        // Replay the captured bounce loop until every path of the job has
        // reached the film, or few enough remain.  While camera paths are left
        // to generate, or many wait, the next replay is queued before the last
        // one's counts are read.
        const uint64_t max_launches =
            1 + (total / std::max<uint32_t>(1, E->cfg.capacity) + 4) * (uint64_t)(P.max_path_len + 4) * 4;
        uint64_t queued = 0, seen = 0;
        const auto loop = [&]() -> int {
            for (;;) {
                while (queued == seen || (queued == seen + 1 && (st->claimed < total || st->waiting / 4 > few))) {
                    const int r = wf_launch(ctx, E, s);
                    if (r != WR_OK) return r;
                    WR_CUDA(ctx, cudaEventRecord(E->turn[queued & 1], s));
                    queued++;
                }
                WR_CUDA(ctx, cudaEventSynchronize(E->turn[seen & 1]));
                seen++;
                if (st->finished >= total) {
                    finished = true;
                    return WR_OK;
                }
                if (queued == seen && st->claimed >= total && st->waiting <= few) return wf_finish(ctx, E, 0, s);
                if (seen > max_launches) return set_error(ctx, WR_ERR_TIMEOUT, "wavefront did not drain");
            }
        };
        if ((rc = loop()) != WR_OK) {
            cudaStreamSynchronize(s);  // a queued replay may still write the caller's film
            return rc;
        }
    }
    // the job's counters and the error word
    unsigned int* herr = reinterpret_cast<unsigned int*>(E->host_counters + 1);
    WR_CUDA(ctx, cudaMemcpyAsync(E->host_counters, E->counters.p, sizeof(WfJobCounters), cudaMemcpyDeviceToHost, s));
    WR_CUDA(ctx, cudaMemcpyAsync(herr, E->err_word.p, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    WR_CUDA(ctx, cudaStreamSynchronize(s));
    // retired on the host: nothing launches without a new job table
    E->job_tab[0].active = 0;
    if (!finished && E->host_counters[0].finished < total)
        return set_error(ctx, WR_ERR_INTERNAL, "wavefront finish left paths");
    if (*herr) return set_error(ctx, WR_ERR_INTERNAL, "traversal stack overflow");
    return WR_OK;
}

}  // namespace wr
