// wr_quad_trace.cuh — the warp-persistent closest-hit loop of the batch kernel
// (k_trace_closest) and the wavefront's extend and shadow stages: the search of
// wr_quad.cuh for many rays at once.
//
// How a warp's 32 lanes are kept busy:
//  * a lane walks nodes until it reaches a leaf; the leaf is postponed and the
//    walk goes on to the next leaf, where the lane waits.  Once `leaf_min` lanes
//    wait (or none is walking) the warp tests the postponed leaves together;
//  * lanes whose ray is finished take new rays once `refill_min` of them are
//    idle.  A warp draws ray ids from the global counter in runs, so that the
//    counter is not what the launch waits for;
//  * a finished ray that hit something is put into the warp's queue in shared
//    memory; 32 of them are checked against the reference's boxes
//    (reference_reaches) and written by all lanes at once.
//
// A source class supplies the rays:
//   fetch(id, ray)   fills a TraceRay
//   put(id, ray, h)  writes the closest hit (h.slot < 0: none)
//   tris_of(rays, l) triangles of lane l's ray (RayInShared)
#pragma once

#include "wr_quad.cuh"

namespace wr {

struct TraceRay {
    const DevTree* T;
    f3 o, d;
    float pf;  // pruning factor
    bool filt;
    int inside, contact;  // NoSelfCondition object ids (used when filt)
    float enough = -1.f;  // a hit below this distance ends the search (enough_before; used when filt)
};

// A warp's queues: rays that meet the scene's box and wait for a lane, and
// finished rays with a hit (or for reference_search: slot SLOT_REFERENCE).
// Each holds at most 31 entries when 32 more come.
struct WarpQueues {
    uint32_t in[64];
    uint32_t id[64];
    int slot[64];
    float t[64];
    float ray[RAY_WORDS * 32];  // the lanes' rays (RayInShared)
    WarpLeaves leaves;
};
// this thread's work counts (profiling launches)
struct TraceWork {
    unsigned long long rays, boxes, tris;
};

// dynamic shared memory of a CTA: the threads' stacks, then the warps' queues
inline size_t quad_smem(int cap, int block) {
    return (size_t)cap * block * sizeof(uint32_t) + (size_t)(block / 32) * sizeof(WarpQueues);
}
__device__ __forceinline__ WarpQueues& warp_queues(uint32_t* smem, int cap) {
    return reinterpret_cast<WarpQueues*>(smem + (size_t)cap * blockDim.x)[threadIdx.x >> 5];
}

// the scene's box, grown as all others (a ray for reference_search meets it)
__device__ __forceinline__ bool meets_scene(const TraceRay& a) {
    const DevTree& T = *a.T;
    QuadRay r;
    if (!make_quad_ray(a.o, a.d, T.finite_mag, box_margin(a.o, T.finite_mag), r)) return true;
    const bool px = r.inv.x > 0.f, py = r.inv.y > 0.f, pz = r.inv.z > 0.f;
    return quad_entry(r, px ? T.root_lo[0] : T.root_hi[0], py ? T.root_lo[1] : T.root_hi[1],
                      pz ? T.root_lo[2] : T.root_hi[2], px ? T.root_hi[0] : T.root_lo[0],
                      py ? T.root_hi[1] : T.root_lo[1], pz ? T.root_hi[2] : T.root_lo[2], INFINITY) < INFINITY;
}

// checks a finished ray against the reference's boxes and writes its hit
template <class Src>
__device__ __forceinline__ void finish_ray(Src& src, uint32_t id, Hit h) {
    TraceRay r;
    src.fetch(id, r);
    h = settle(*r.T, h, r.o, r.d, r.pf, r.filt, r.inside, r.contact);
    src.put(id, r, h);
}

// Traces rays [0, n) of `src`, handing out ray ids from *counter (which
// starts at 0).  Every lane of the warp must call it.  `stack`: this thread's
// entries at stack[k * stride], k < cap; `Q`: the warp's queues.
template <bool STATS, class Src>
__device__ __forceinline__ void quad_trace(Src& src, uint32_t n, unsigned int* counter, TraceTune tune,
                                           uint32_t* stack, int stride, int cap, WarpQueues& Q, TraceWork& work) {
    constexpr unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    // ids are drawn in runs: long enough that the counter is quiet, short
    // enough that the warps end together.  Fewer rays than lanes are shared
    // out evenly, a few to a warp: its leaf phases then end sooner.
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t share = max(1u, n / warps + (n % warps != 0));
    const uint32_t lanes = min(32u, share);
    const uint32_t run = share >= 512u ? min(256u, share / 8u & ~31u) : lanes;
    uint32_t next = 0, end = 0;  // the warp's run
    bool dry = false;            // no more runs
    const int top = (cap - 4) * stride;
    uint32_t nin = 0, nfin = 0;  // entries of the queues

    uint32_t id = 0;
    bool active = false;
    SearchLane<RayInShared> L;
    L.ray = RayInShared{Q.ray + lane, 32};
    L.clear();

    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !active);
        if (idle == FULL || __popc(idle) >= (int)(32u - lanes) + tune.refill_min) {
            // intake: 32 rays at a time against the scene's box; those that
            // meet it are queued
            const uint32_t busy = 32u - (uint32_t)__popc(idle);
            const uint32_t want = lanes > busy ? lanes - busy : 0u;
            while (nin < want && !dry) {
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
                const uint32_t i = next + lane;
                bool keep = false;
                if (i < end) {
                    TraceRay a;
                    src.fetch(i, a);
                    keep = meets_scene(a);
                    if (STATS) {
                        work.rays++;
                        work.boxes++;
                    }
                    if (!keep) src.put(i, a, Hit{INFINITY, -1});
                }
                const unsigned km = __ballot_sync(FULL, keep);
                if (keep) Q.in[nin + __popc(km & lt_mask)] = i;
                nin += __popc(km);
                next = min(next + 32u, end);
                __syncwarp();
            }
            const uint32_t k = (uint32_t)__popc(idle & lt_mask);
            if (!active && k < want && k < nin) {
                id = Q.in[nin - 1u - k];
                TraceRay a;
                src.fetch(id, a);
                L.begin(*a.T, a.o, a.d, a.pf, a.filt, a.inside, a.contact, a.enough);
                active = true;
            }
            nin -= min(want, nin);
            __syncwarp();
        }
        const bool walking = active && L.walking();
        const unsigned wm = __ballot_sync(FULL, walking), lm = __ballot_sync(FULL, active && L.at_leaf());
        if (lm && (wm == 0 || __popc(lm) >= tune.leaf_min)) {
            // every postponed leaf, those of lanes still walking too
            const uint32_t tested =
                warp_leaves<3>(L, active && L.pend != NO_WORD, Q.leaves, stack, stride,
                            [&](int from) { return src.tris_of(L.ray, from); });
            if (STATS) work.tris += tested;
        } else if (walking) {
            for (int k = 0; k < tune.steps && L.walking(); k++) {
                L.visit(stack, stride, top);
                if (STATS) work.boxes += 4;
            }
        }
        // finished rays: misses at once, hits through the queue
        const bool done = active && L.finished();
        const unsigned dm = __ballot_sync(FULL, done);
        if (dm) {
            const bool queue = done && L.h.slot != -1;
            if (done && !queue) {
                TraceRay a;
                src.put(id, a, Hit{INFINITY, -1});
            }
            const unsigned qm = __ballot_sync(FULL, queue);
            if (queue) {
                const uint32_t at = nfin + __popc(qm & lt_mask);
                Q.id[at] = id;
                Q.slot[at] = L.h.slot;
                Q.t[at] = L.h.t;
            }
            nfin += __popc(qm);
            if (done) active = false;
            if (nfin >= 32) {
                __syncwarp();
                nfin -= 32;
                finish_ray(src, Q.id[nfin + lane], Hit{Q.t[nfin + lane], Q.slot[nfin + lane]});
                __syncwarp();
            }
            if (dm == FULL || !__ballot_sync(FULL, active)) {
                if (dry && nin == 0) break;
            }
        } else if (!(wm | lm)) {
            if (dry && nin == 0 && idle == FULL) break;
        }
    }
    __syncwarp();
    if (lane < nfin) finish_ray(src, Q.id[lane], Hit{Q.t[lane], Q.slot[lane]});
}

}  // namespace wr
