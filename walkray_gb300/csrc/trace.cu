// trace.cu — k_trace_closest: closest hits for a batch of rays
// (KDTree::intersect / Scene::intersect, kdtree.cpp:349-353, scene.cpp:102-113).
//
// Persistent warps (the loop of wr_quad_trace.cuh): the grid is sized to fill
// every SM once; warps take rays from a global counter.  Per-thread stacks live
// in shared memory, column-major (entry k of thread t at k * blockDim.x + t) so
// a warp's pushes hit 32 distinct banks.
//
// Bound by the L1 cache's load pipe and the latency behind it: on 4.2 M
// incoherent rays (1,310,720-triangle icosphere) the pipe is 56 % busy, issue
// 46 %, 75 warp instructions a ray (174 when it walked the reference's tree with
// two slab tests a box).  2^24 rays: 3.38 -> 2.05 to 2.2 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/walkray.h"
#include "trace_launch.h"
#include "wr_warp_trace.cuh"

namespace wr {

// rays from a (n x 6) array, hits to wr_hit records
struct BatchSrc {
    const DevTree& T;
    const float* __restrict__ rays;
    const int32_t* __restrict__ inside;
    const int32_t* __restrict__ contact;
    wr_hit* __restrict__ hits;
    bool filtered;

    __device__ __forceinline__ void fetch(uint64_t id, TraceRay& a) const {
        const float* r = rays + 6 * id;
        a.T = &T;
        a.o = mk(r[0], r[1], r[2]);
        a.d = mk(r[3], r[4], r[5]);
        a.pf = 1.001f;
        a.filt = filtered;
        a.inside = filtered ? inside[id] : -1;
        a.contact = filtered ? contact[id] : -1;
    }
    __device__ __forceinline__ void put(uint64_t id, const TraceRay& a, const Hit& h) const {
        uint4 out = make_uint4(WR_NO_HIT, __float_as_uint(-1.f), 0u, 0u);
        if (h.slot >= 0) {
            float u1, u2;
            uint32_t gid;
            hit_barycentrics(T, h.slot, a.o, a.d, h.t, &u1, &u2, &gid);
            out = make_uint4(gid, __float_as_uint(h.t), __float_as_uint(u1), __float_as_uint(u2));
        }
        reinterpret_cast<uint4*>(hits)[id] = out;
    }
    __device__ __forceinline__ const TriRec* tris_of(const RayInShared&, int) const { return T.tris; }
    // the same for the walk that visits every box the reference visits (warp_trace)
    __device__ __forceinline__ void load(uint64_t id, TraceLane& L, uint32_t* stack, int stride) const {
        TraceRay a;
        fetch(id, a);
        load_lane(a, L, stack, stride);
    }
    __device__ __forceinline__ void store(uint64_t id, const TraceLane& L) const {
        TraceRay a;
        a.o = L.q.o;
        a.d = L.q.d;
        put(id, a, L.h);
    }
};

// MINB > 0: compiled for at least MINB resident CTAs per SM (a register cap)
template <int MINB>
__global__ void __launch_bounds__(128, MINB > 0 ? MINB : 1)
    k_trace_closest(const __grid_constant__ DevTree T, const float* __restrict__ rays, uint64_t n,
                    const int32_t* __restrict__ inside, const int32_t* __restrict__ contact,
                    wr_hit* __restrict__ hits, unsigned long long* __restrict__ counter, int stack_cap,
                    TraceTune tune) {
    extern __shared__ __align__(16) uint32_t s_stack[];
    BatchSrc src{T, rays, inside, contact, hits, inside != nullptr};
    TraceWork work;
    quad_trace<false>(src, (uint32_t)n, reinterpret_cast<unsigned int*>(counter), tune, s_stack + threadIdx.x, blockDim.x, stack_cap,
                      warp_queues(s_stack, stack_cap), work);
}

// The walk of the reference's own tree: without pruning by distance
// (WR_CTX_EXACT_TRAVERSAL), or with it where a scene has no four-wide tree
// (more than QUAD_MAX_SLOTS triangles: ray by ray through reference_search a
// batch takes some four times the walk's time).
template <bool PRUNE>
__global__ void __launch_bounds__(128, 7)
    k_trace_closest_walk(const __grid_constant__ DevTree T, const float* __restrict__ rays, uint64_t n,
                          const int32_t* __restrict__ inside, const int32_t* __restrict__ contact,
                          wr_hit* __restrict__ hits, unsigned long long* __restrict__ counter, int stack_cap,
                          TraceTune tune, unsigned int* __restrict__ err) {
    extern __shared__ __align__(16) uint32_t s_stack[];
    BatchSrc src{T, rays, inside, contact, hits, inside != nullptr};
    warp_trace<PRUNE, false>(src, n, counter, tune, s_stack + threadIdx.x, blockDim.x, stack_cap, err);
}

cudaError_t launch_trace_closest(const DevTree& T, const float* d_rays, uint64_t n, const int32_t* d_inside,
                                 const int32_t* d_contact, wr_hit* d_hits, unsigned long long* d_counter,
                                 unsigned int* d_err, int num_sms, bool prune, cudaStream_t stream,
                                 int* launched_blocks, const TraceTune* tune, int ctas_per_sm) {
    constexpr uint64_t MOST = 1ull << 31;  // rays of a launch (32-bit ray ids)
    for (; n > MOST; n -= MOST) {
        const cudaError_t e = launch_trace_closest(T, d_rays, MOST, d_inside, d_contact, d_hits, d_counter, d_err,
                                                   num_sms, prune, stream, launched_blocks, tune, ctas_per_sm);
        if (e != cudaSuccess) return e;
        d_rays += 6 * MOST;
        d_hits += MOST;
        if (d_inside) d_inside += MOST, d_contact += MOST;
    }
    const int block = 128;
    const int ref_cap = (int)T.max_depth + 3;  // stack of the reference's own walk
    if ((size_t)ref_cap * block * sizeof(uint32_t) > 200 * 1024) return cudaErrorInvalidValue;
    const bool search = !trace_walks(T, prune);
    const int stack_cap = search ? quad_stack_cap(T) : ref_cap;
    const size_t smem = search ? quad_smem(stack_cap, block) : (size_t)stack_cap * block * sizeof(uint32_t);
    cudaError_t e = cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return e;
    // blocks per SM from the occupancy calculator for this stack size
    int per_sm = 1;
    // 0: the 6-CTA variant (80 registers; 2^24 rays: 2.22 ms, 2.36 with 7, 2.50 with 8, 2.52 with 5)
    const int variant = ctas_per_sm ? ctas_per_sm : 6;
    const auto kern = variant >= 8   ? k_trace_closest<8>
                      : variant >= 7 ? k_trace_closest<7>
                      : variant >= 6 ? k_trace_closest<6>
                                     : k_trace_closest<0>;
    const auto walk = prune ? k_trace_closest_walk<true> : k_trace_closest_walk<false>;
    const void* fn = search ? reinterpret_cast<const void*>(kern) : reinterpret_cast<const void*>(walk);
    if (smem > 48 * 1024) {
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, smem);
    if (e != cudaSuccess) return e;
    if (ctas_per_sm > 0) per_sm = std::min(per_sm, ctas_per_sm);
    if (per_sm < 1) per_sm = 1;
    // few rays: a warp for each, as far as the grid goes
    uint64_t need_blocks = search ? (n + block / 32 - 1) / (block / 32) : (n + block - 1) / block;
    int grid = num_sms * per_sm;
    if ((uint64_t)grid > need_blocks) grid = (int)(need_blocks ? need_blocks : 1);
    if (launched_blocks) *launched_blocks = grid;
    const TraceTune tt = tune ? *tune : default_trace_tune();
    if (search)
        kern<<<grid, block, smem, stream>>>(T, d_rays, n, d_inside, d_contact, d_hits, d_counter, stack_cap, tt);
    else
        walk<<<grid, block, smem, stream>>>(T, d_rays, n, d_inside, d_contact, d_hits, d_counter, stack_cap, tt, d_err);
    return cudaGetLastError();
}

}  // namespace wr
