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
//   tris_of(tris, l) triangles of lane l's ray (`tris`: of this lane's, which
//                    may never have had one); every lane calls it
#pragma once

#include "wr_quad.cuh"

namespace wr {

struct TraceRay {
    const DevTree* T;
    f3 o, d;
    float pf;  // pruning factor
    bool filt;
    int inside, contact;  // NoSelfCondition object ids (used when filt)
};

// A warp's queues: rays that meet the scene's box and wait for a lane, and
// finished rays with a hit (or for reference_search: slot SLOT_REFERENCE).
// Each holds at most 31 entries when 32 more come.
struct WarpQueues {
    uint32_t in[64];
    uint32_t id[64];
    int slot[64];
    float t[64];
    uint8_t item[224];  // the leaf phase's triangles: lane | index in its leaf << 5
};
constexpr int SLOT_REFERENCE = -2;

constexpr uint32_t NO_WORD = QUAD_HOLE;

// this thread's work counts (profiling launches)
struct TraceWork {
    unsigned long long rays, boxes, tris;
};

// stack entries a thread is given: what the deepest walk can need, but at most
// 28.  (Measured on the 1.3 M-triangle icosphere and the mixed-material scene:
// no ray holds more than 17 at once, where the bound from the tree is 39; a ray
// that would need more is left to reference_search.)
inline int quad_stack_cap(const DevTree& T) { return (int)(T.quad_stack + 4 < 28 ? T.quad_stack + 4 : 28); }

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
    if (!make_quad_ray(a.o, a.d, T.scene_mag, box_margin(a.o, T.scene_mag), r)) return true;
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
    if (h.slot < 0 || !reference_reaches(*r.T, h.slot, r.o, r.d))
        h = reference_search(*r.T, r.o, r.d, r.pf, r.filt, r.inside, r.contact);
    src.put(id, r, h);
}

__device__ __forceinline__ const TriRec* shfl_ptr(const TriRec* p, int from) {
    return reinterpret_cast<const TriRec*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), from));
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
    // enough that the warps end together
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t run = min(256u, max(32u, n / (warps * 8u) & ~31u));
    uint32_t next = 0, end = 0;  // the warp's run
    bool dry = false;            // no more runs
    const int top = (cap - 4) * stride;
    uint32_t nin = 0, nfin = 0;  // entries of the queues

    uint32_t id = 0;
    const QuadNode* quads = nullptr;
    const TriRec* tris = nullptr;
    f3 o = mk(0, 0, 0), d = mk(0, 0, 0);
    QuadRay r;
    float M = 0.f, lim = 0.f;
    bool filt = false, active = false;
    int inside = -1, contact = -1, sp = 0;
    uint32_t cur = NO_WORD, pend = NO_WORD;  // the node or leaf to visit; the postponed leaf
    Hit h;
    h.t = 0.f;
    h.slot = -1;

    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !active);
        if (idle == FULL || __popc(idle) >= tune.refill_min) {
            // intake: 32 rays at a time against the scene's box; those that
            // meet it are queued
            const uint32_t want = (uint32_t)__popc(idle);
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
            if (!active && k < nin) {
                id = Q.in[nin - 1u - k];
                TraceRay a;
                src.fetch(id, a);
                o = a.o;
                d = a.d;
                quads = a.T->quads;
                tris = a.T->tris;
                filt = a.filt;
                inside = a.inside;
                contact = a.contact;
                M = box_margin(o, a.T->scene_mag);
                h.t = lim = INFINITY;
                sp = 0;
                pend = NO_WORD;
                active = true;
                const bool ok = make_quad_ray(o, d, a.T->scene_mag, M, r) && quads;
                if (!(a.pf < INFINITY)) M = INFINITY;  // no pruning: `lim` stays infinite
                h.slot = ok ? -1 : SLOT_REFERENCE;
                cur = ok ? 0u : NO_WORD;
            }
            nin -= min(want, nin);
            __syncwarp();
        }
        const bool walking = active && !(cur & QUAD_LEAF);
        const bool waiting = active && pend != NO_WORD && (cur & QUAD_LEAF);
        const unsigned wm = __ballot_sync(FULL, walking), lm = __ballot_sync(FULL, waiting);
        if (lm && (wm == 0 || __popc(lm) >= tune.leaf_min)) {
            // every postponed leaf, those of lanes still walking too: their
            // triangles are dealt out over all lanes, one each
            const bool has = active && pend != NO_WORD;
            const uint32_t first = has ? pend & ((1u << QUAD_COUNT_AT) - 1u) : 0u;
            const uint32_t count = has ? pend >> QUAD_COUNT_AT & 7u : 0u;
            if (STATS) work.tris += count;
            const unsigned c0 = __ballot_sync(FULL, count & 1u), c1 = __ballot_sync(FULL, count & 2u),
                           c2 = __ballot_sync(FULL, count & 4u);
            const uint32_t before =
                __popc(c0 & lt_mask) + 2u * __popc(c1 & lt_mask) + 4u * __popc(c2 & lt_mask);
            const uint32_t total = __popc(c0) + 2u * __popc(c1) + 4u * __popc(c2);
            for (uint32_t k = 0; k < count; k++) Q.item[before + k] = (uint8_t)(lane | k << 5);
            __syncwarp();
            for (uint32_t base = 0; base < total; base += 32u) {
                const bool on = base + lane < total;
                const uint32_t it = on ? Q.item[base + lane] : lane;
                const int own = (int)(it & 31u);
                const f3 ro = mk(__shfl_sync(FULL, o.x, own), __shfl_sync(FULL, o.y, own), __shfl_sync(FULL, o.z, own));
                const f3 rd = mk(__shfl_sync(FULL, d.x, own), __shfl_sync(FULL, d.y, own), __shfl_sync(FULL, d.z, own));
                const int slot = (int)(__shfl_sync(FULL, first, own) + (it >> 5));
                const float best = __shfl_sync(FULL, h.t, own);
                const TriRec* rt = src.tris_of(tris, own);
                float t = -1.f, dd = 0.f;
                if (on) t = tri_slot_test(rt, slot, ro, rd, &dd);
                bool cand = t >= 0.f && t <= best;
                unsigned cm = __ballot_sync(FULL, cand);
                if (cm) {
                    const bool rf = __shfl_sync(FULL, (int)filt, own) != 0;
                    const int ri = __shfl_sync(FULL, inside, own), rc = __shfl_sync(FULL, contact, own);
                    if (cand && rf) cand = noself_slot(rt, slot, rd, ri, rc);
                    // the candidates go back to their rays one by one
                    for (cm = __ballot_sync(FULL, cand); cm; cm &= cm - 1u) {
                        const int b = __ffs(cm) - 1;
                        const int bo = __shfl_sync(FULL, own, b), bs = __shfl_sync(FULL, slot, b);
                        const float bt = __shfl_sync(FULL, t, b), bd = __shfl_sync(FULL, dd, b);
                        if ((int)lane == bo && (bt < h.t || (bt == h.t && bs > h.slot))) {
                            // a near-grazing hit turns pruning off for good (graze_check)
                            const bool off = fabsf(bd) < GRAZE_COS * length(d) || (h.slot >= 0 && !(lim < INFINITY));
                            lim = off ? INFINITY : bt * 1.001f + M;
                            h.t = bt;
                            h.slot = bs;
                        }
                    }
                }
            }
            if (has) {
                pend = NO_WORD;
                if ((cur & QUAD_LEAF) && cur != NO_WORD) {
                    pend = cur;
                    cur = NO_WORD;
                    if (sp > 0) {
                        sp -= stride;
                        cur = stack[sp];
                    }
                }
            }
            __syncwarp();
        } else if (walking) {
            for (int k = 0; k < tune.steps; k++) {
                float4 t;
                uint4 w;
                quad_children(quads + cur, r, lim, t, w);
                if (STATS) work.boxes += 4;
                if (t.w < INFINITY) {
                    stack[sp] = w.w;
                    sp += stride;
                }
                if (t.z < INFINITY) {
                    stack[sp] = w.z;
                    sp += stride;
                }
                if (t.y < INFINITY) {
                    stack[sp] = w.y;
                    sp += stride;
                }
                cur = w.x;
                if (!(t.x < INFINITY)) {
                    cur = NO_WORD;
                    if (sp > 0) {
                        sp -= stride;
                        cur = stack[sp];
                    }
                } else if (sp > top) {  // deeper than the stack: the reference's own walk needs none
                    sp = 0;
                    cur = pend = NO_WORD;
                    h.slot = SLOT_REFERENCE;
                }
                if ((cur & QUAD_LEAF) && cur != NO_WORD && pend == NO_WORD) {  // postpone it and walk on
                    pend = cur;
                    cur = NO_WORD;
                    if (sp > 0) {
                        sp -= stride;
                        cur = stack[sp];
                    }
                }
                if (cur & QUAD_LEAF) break;
            }
        }
        // finished rays: misses at once, hits through the queue
        const bool done = active && cur == NO_WORD && pend == NO_WORD;
        const unsigned dm = __ballot_sync(FULL, done);
        if (dm) {
            const bool queue = done && h.slot != -1;
            if (done && !queue) {
                TraceRay a;
                src.put(id, a, Hit{INFINITY, -1});
            }
            const unsigned qm = __ballot_sync(FULL, queue);
            if (queue) {
                const uint32_t at = nfin + __popc(qm & lt_mask);
                Q.id[at] = id;
                Q.slot[at] = h.slot;
                Q.t[at] = h.t;
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
