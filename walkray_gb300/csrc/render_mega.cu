// render_mega.cu — k_megakernel: the plain form of the renderer.  One thread
// per pixel runs whole paths (PathTracer::renderPixels inner loop,
// pathTracer.cpp:21-70: camera ray, samplePath bounce loop, throughput,
// isLegalColor, fixVignetting) for a range of samples and adds the results
// to an FP32 film (sum and optional sum of squares per channel).
#include <type_traits>

#include "render_launch.h"
#include "wr_shade.cuh"

namespace wr {

constexpr int MEGA_BLOCK = 128;

// The lanes of a warp stay together: each takes one ray of its own path per
// turn (search_warp) and goes on to its pixel's next sample as soon as a path
// ends, so that a warp waits for the lane with the most rays in all, not for
// the longest path of every sample.
template <bool STATS, bool MIS, int MED>
__global__ void __launch_bounds__(MEGA_BLOCK) k_megakernel(RenderScene S, RenderParams P, float* __restrict__ film,
                                                           float* __restrict__ film2) {
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ uint32_t s_stack[];
    __shared__ WarpLeaves s_leaves[MEGA_BLOCK / 32];
    uint32_t* stack = s_stack + threadIdx.x;
    WarpLeaves& leaves = s_leaves[threadIdx.x >> 5];
    const int stride = MEGA_BLOCK;
    const uint32_t npix = S.cam.width * S.cam.height;
    const uint32_t pixel = blockIdx.x * MEGA_BLOCK + threadIdx.x;
    f3 acc = mk(0, 0, 0), acc2 = mk(0, 0, 0);
    const float pf = prune_factor(P.flags);
    const bool nee = (P.flags & WR_RENDER_NEE) != 0;
    uint32_t s = pixel < npix ? P.s0 : P.s1;  // the sample this lane is at
    bool start = true;                        // it begins with this turn
    PathRng g;
    g.init(P.seed, pixel, s);
    PRay cur = ray_default();
    InsideStack st;
    st.reset(-1);
    f3 color = mk(1, 1, 1), result = mk(0, 0, 0), prev_d = mk(0, 0, 0), lit = mk(0, 0, 0);
    uint32_t depth = 0;
    float mis_pdf = 0.f;
    while (__any_sync(FULL, s < P.s1)) {
        const bool on = s < P.s1;
        const bool filtered = !start;  // the eye ray is traced without a condition (camera.cpp:52)
        if (on && start) {
            g.init(P.seed, pixel, s);
            cur = camera_ray(S.cam, pixel, g);
            st.reset(cur.inside);
            color = mk(1, 1, 1);
            result = prev_d = lit = mk(0, 0, 0);
            depth = 0;
            mis_pdf = 0.f;
            start = false;
        }
        const Hit h = search_warp(S.tree, on, cur.o, cur.d, pf, filtered, cur.inside, cur.contact, stack, stride,
                                  P.stack_cap, leaves);
        bool done = false, nee_here = false, has_lr = false;
        LightReq lr;
        if (on) {
            if (h.slot < 0 && filtered) {  // a scattered ray that escapes ends with zero radiance
                nee_here = nee;
                done = true;
            } else {
                set_hit(S, cur, h);
                done = path_advance<MIS, MED>(S, cur, color, prev_d, depth, st, g, P.max_path_len, P.flags, result,
                                         nee_here, mis_pdf, lr, has_lr);
            }
        }
        if (MIS && __any_sync(FULL, has_lr)) {  // the light connection of WR_RENDER_NEE_MIS
            const Hit lh = search_warp(S.tree, has_lr, lr.o, lr.d, pf, true, lr.inside, lr.contact, stack, stride,
                                       P.stack_cap, leaves, enough_before(lr.dist));
            if (has_lr && light_req_visible(S, lh, lr)) lit = lit + lr.contrib;
        }
        if (__any_sync(FULL, nee_here)) {  // the connection of the NEE branch
            ShadowReq sr;
            const bool conn = nee_here && nee_prepare(S, cur, prev_d, color, g, sr);
            const Hit sh = search_warp(S.tree, conn, sr.o, sr.d, pf, true, sr.inside, sr.contact, stack, stride,
                                       P.stack_cap, leaves, enough_before(sr.dist));
            if (conn && nee_visible(sh, sr.dist)) result = sr.contrib;
        }
        if (done) {
            if (!legal(result)) result = mk(0, 0, 0);
            result = result + lit;
            const f3 c = fix_vignetting(S.cam, result, pixel);
            acc = acc + c;
            if (STATS) acc2 = acc2 + vmul(c, c);
            s++;
            start = true;
        }
    }
    if (pixel >= npix) return;
    float* f = film + 3 * (size_t)pixel;
    f[0] += acc.x;
    f[1] += acc.y;
    f[2] += acc.z;
    if (STATS) {
        float* f2 = film2 + 3 * (size_t)pixel;
        f2[0] += acc2.x;
        f2[1] += acc2.y;
        f2[2] += acc2.z;
    }
}

cudaError_t launch_megakernel(const RenderScene& S, const RenderParams& P, float* film, float* film2,
                              bool media, cudaStream_t stream) {
    const int block = MEGA_BLOCK;
    const size_t smem = (size_t)P.stack_cap * block * sizeof(uint32_t);
    const uint32_t npix = S.cam.width * S.cam.height;
    const int grid = (int)((npix + block - 1) / block);
    const bool mis = (P.flags & WR_RENDER_NEE_MIS) != 0;
    auto pick = [&](auto med) {
        constexpr int M = decltype(med)::value;
        return film2 ? (mis ? k_megakernel<true, true, M> : k_megakernel<true, false, M>)
                     : (mis ? k_megakernel<false, true, M> : k_megakernel<false, false, M>);
    };
    auto kern = media ? pick(std::integral_constant<int, MED_TRACK>{}) : pick(std::integral_constant<int, MED_NONE>{});
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    kern<<<grid, block, smem, stream>>>(S, P, film, film2);
    return cudaGetLastError();
}

}  // namespace wr
