// wr_quad.cuh — closest-hit search on the four-wide tree (quad_build.cpp).
//
// Result contract: that of wr_traverse.cuh, the reference's triangle id and t
// bit for bit.  The search is split in two:
//
//  * Candidates.  The tree's leaves are the reference's leaves with their own
//    boxes and a node's box contains its leaves' boxes.  A child is visited
//    unless the ray misses its box grown by the margin M of wr_traverse.cuh,
//    one slab test of one FMA per plane.  Whatever the reference's predicate
//    passes, this test passes: the reference needs a point on a face plane
//    within 4.1 eps (B + |o|) of the box (eps = 2^-24, B the largest
//    coordinate), while the slab test here is off by at most 6 eps (B + |o|)
//    -- half an ulp each of 1/d (one ulp), of o/d and of the FMA -- and M is
//    33 eps (B + |o|).  It is monotone in the box, so a node passes when a leaf
//    below it does.  Every triangle the reference tests is therefore tested,
//    with the same triangle test, and usually a few more.
//  * The winner's way.  Smallest t, then largest slot, among a superset of the
//    reference's candidates is the reference's answer if the reference
//    reaches it: reference_reaches() runs the reference's own predicate on
//    the boxes above the winner's leaf, once per ray that hits something.  When one of
//    them fails (a ray through a box's edge within rounding) the ray is
//    searched again by reference_search(), which descends exactly where the
//    reference does.
//
// Pruning by distance is the rule of wr_traverse.cuh (q.pf, graze_check).
//
// Directions need not be of unit length: distances are in units of |d|, the
// pruning rule's margin too.  Rays that are left to reference_search() alone:
// |d| outside [1e-15, 1e14], where squares of d leave the float range or
// distances may be subnormal (half an ulp of one is 7e-46, times |d| far below
// the 1e-30 in M); coordinates beyond 1e15 |d|, where the slabs' products could
// overflow; values that are not finite.  (B leaves out a scene's coordinates
// that are not finite: boxes with such a plane are always visited, see
// build_quads.)  A direction component below 1e-18 of the direction's length is
// taken as that small: over the scene's extent the ray moves by less than M
// along that axis either way.
// (With bounds of 1e-6 and 1e6 on |d| and 1e9 on coordinates 2^20 rays of length
// 1e7 took 2.97 ms, of unit length 0.18.)
//
// On the mixed-material scene a bounce ray tests 70 boxes in 17 nodes here,
// 104 in 52 node pairs on the reference's tree.
#pragma once

#include "wr_traverse.cuh"

namespace wr {

struct QuadRay {
    f3 inv;              // 1/d
    f3 nb, fb;           // plane * inv + nb (fb): distance to a near (far) plane moved out by M
};

// the margin M (wr_traverse.cuh)
__device__ __forceinline__ float box_margin(f3 o, float scene_mag) {
    return 2e-6f * (scene_mag + fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z)))) + 1e-30f;
}

// false: this ray is for reference_search()
__device__ __forceinline__ bool make_quad_ray(f3 o, f3 d, float scene_mag, float M, QuadRay& r) {
    const float on = fabsf(o.x) + fabsf(o.y) + fabsf(o.z), dn = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    const float least = 1e-18f * dn;
    const float dx = fabsf(d.x) < least ? copysignf(least, d.x) : d.x;
    const float dy = fabsf(d.y) < least ? copysignf(least, d.y) : d.y;
    const float dz = fabsf(d.z) < least ? copysignf(least, d.z) : d.z;
    r.inv = mk(__fdividef(1.f, dx), __fdividef(1.f, dy), __fdividef(1.f, dz));
    r.nb = mk(__fmaf_rn(-o.x, r.inv.x, -M * fabsf(r.inv.x)), __fmaf_rn(-o.y, r.inv.y, -M * fabsf(r.inv.y)),
              __fmaf_rn(-o.z, r.inv.z, -M * fabsf(r.inv.z)));
    r.fb = mk(__fmaf_rn(-o.x, r.inv.x, M * fabsf(r.inv.x)), __fmaf_rn(-o.y, r.inv.y, M * fabsf(r.inv.y)),
              __fmaf_rn(-o.z, r.inv.z, M * fabsf(r.inv.z)));
    return on + scene_mag <= 1e15f * dn && dn >= 1e-15f && dn <= 1e14f;  // false for a NaN
}

// of three at once (a NaN is dropped, as by fmaxf and fminf)
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// entry distance of one child, +inf when the ray misses it or enters it beyond `lim`
__device__ __forceinline__ float quad_entry(const QuadRay& r, float nx, float ny, float nz, float fx, float fy,
                                            float fz, float lim) {
    const float t0 = fmaxf(max3(__fmaf_rn(nx, r.inv.x, r.nb.x), __fmaf_rn(ny, r.inv.y, r.nb.y),
                                __fmaf_rn(nz, r.inv.z, r.nb.z)), 0.f);
    const float t1 = fminf(min3(__fmaf_rn(fx, r.inv.x, r.fb.x), __fmaf_rn(fy, r.inv.y, r.fb.y),
                                __fmaf_rn(fz, r.inv.z, r.fb.z)), lim);
    return t0 <= t1 ? t0 : __int_as_float(0x7f800000);
}

// orders two (distance, word) pairs
__device__ __forceinline__ void quad_order(float& ta, uint32_t& a, float& tb, uint32_t& b) {
    const bool s = tb < ta;
    const float t = s ? tb : ta;
    const uint32_t w = s ? b : a;
    tb = s ? ta : tb;
    b = s ? a : b;
    ta = t;
    a = w;
}

// The four children of a node, the nearest first (ordering the others too saves
// 1 % of the visits); t = +inf: not to be visited.
__device__ __forceinline__ void quad_children(const QuadNode* q, const QuadRay& r, float lim, float4& t, uint4& w) {
    const char* p = reinterpret_cast<const char*>(q);
    // 48 bytes on where the near plane is the upper one (the hi rows)
    const int ox = __float_as_int(r.inv.x) >> 31 & 48, oy = __float_as_int(r.inv.y) >> 31 & 48,
              oz = __float_as_int(r.inv.z) >> 31 & 48;
    const float4 nx = ldg4(reinterpret_cast<const float4*>(p + ox));
    const float4 ny = ldg4(reinterpret_cast<const float4*>(p + oy + 16));
    const float4 nz = ldg4(reinterpret_cast<const float4*>(p + oz + 32));
    const float4 fx = ldg4(reinterpret_cast<const float4*>(p - ox + 48));
    const float4 fy = ldg4(reinterpret_cast<const float4*>(p - oy + 64));
    const float4 fz = ldg4(reinterpret_cast<const float4*>(p - oz + 80));
    w = ldg4u(reinterpret_cast<const uint4*>(p + 96));
    t.x = quad_entry(r, nx.x, ny.x, nz.x, fx.x, fy.x, fz.x, lim);
    t.y = quad_entry(r, nx.y, ny.y, nz.y, fx.y, fy.y, fz.y, lim);
    t.z = quad_entry(r, nx.z, ny.z, nz.z, fx.z, fy.z, fz.z, lim);
    t.w = quad_entry(r, nx.w, ny.w, nz.w, fx.w, fy.w, fz.w, lim);
    quad_order(t.x, w.x, t.y, w.y);
    quad_order(t.x, w.x, t.z, w.z);
    quad_order(t.x, w.x, t.w, w.w);
}

// the reference's triangle test on one record
__device__ __forceinline__ float tri_slot_test(const TriRec* tris, int slot, f3 o, f3 d, float* dd) {
    const TriRec* tr = tris + slot;
    const float4 a = ldg4(&tr->v0), b = ldg4(&tr->v1), c = ldg4(&tr->v2);
    RayQ q;
    q.o = o;
    q.d = d;
    return tri_test(xyz(a), xyz(b), xyz(c), q, dd);
}

// its first half: false where the ray passes outside an edge
__device__ __forceinline__ bool tri_slot_inside(const TriRec* tris, int slot, f3 o, f3 d) {
    const TriRec* tr = tris + slot;
    const float4 a = ldg4(&tr->v0), b = ldg4(&tr->v1), c = ldg4(&tr->v2);
    RayQ q;
    q.o = o;
    q.d = d;
    return tri_inside(xyz(a), xyz(b), xyz(c), q);
}

// its second half
__device__ __forceinline__ float tri_slot_distance(const TriRec* tris, int slot, f3 o, f3 d, float* dd) {
    const TriRec* tr = tris + slot;
    const float4 a = ldg4(&tr->v0), b = ldg4(&tr->v1), c = ldg4(&tr->v2);
    RayQ q;
    q.o = o;
    q.d = d;
    return tri_distance(xyz(a), xyz(b), xyz(c), q, dd);
}

// NoSelfCondition on one record
__device__ __forceinline__ bool noself_slot(const TriRec* tris, int slot, f3 d, int inside, int contact) {
    const TriRec* tr = tris + slot;
    const float4 a = ldg4(&tr->v0), b = ldg4(&tr->v1), c = ldg4(&tr->v2);
    return noself_legal(inside, contact, (int)__float_as_uint(b.w), d, face_normal(xyz(a), xyz(b), xyz(c)));
}

// ---------------------------------------------------------------------------
// the reference's own descent
// ---------------------------------------------------------------------------
// box and topology words of one child (at = pair << 1 | side)
__device__ __forceinline__ Box child_box(const DevTree& T, uint32_t at) {
    const bool right = at & 1u;
    const float4* p = &T.pairs[at >> 1].a + (right ? 1 : 0);
    const float4 a = ldg4(p), b = ldg4(p + 1);  // two 16-byte pieces hold either box
    return right ? Box{a.z, a.w, b.x, b.y, b.z, b.w} : Box{a.x, a.y, a.z, a.w, b.x, b.y};
}

// the reference's face tests on a box
static __device__ __noinline__ bool box_faces(Box b, f3 o, f3 d, float scene_mag) {
    return box_exact(b, make_rayq(o, d, scene_mag));
}

// Does the reference's predicate pass on a box?  Usually told by one far face:
// with the distances to its plane moved in (s) and out (g) by M, the face's
// plane point lies at least M inside the box on another axis when that axis's
// near plane moved in comes before s and its far plane moved in after g.  If
// so on both other axes, and s is in front of the origin, the reference's test
// of this face passes.  (A flat box passes by the face of its thin axis.)
// Anything else -- an edge within M, a NaN -- runs the face tests.  With
// QuadRay's constants the planes moved in are fb for a near and nb for a far
// one.
__device__ __forceinline__ bool reference_passes(const Box& b, const QuadRay& r, f3 o, f3 d, float scene_mag) {
    const bool px = r.inv.x > 0.f, py = r.inv.y > 0.f, pz = r.inv.z > 0.f;
    const float fx = px ? b.hx : b.lx, fy = py ? b.hy : b.ly, fz = pz ? b.hz : b.lz;
    const float nx = __fmaf_rn(px ? b.lx : b.hx, r.inv.x, r.fb.x), ny = __fmaf_rn(py ? b.ly : b.hy, r.inv.y, r.fb.y),
                nz = __fmaf_rn(pz ? b.lz : b.hz, r.inv.z, r.fb.z);
    const float sx = __fmaf_rn(fx, r.inv.x, r.nb.x), sy = __fmaf_rn(fy, r.inv.y, r.nb.y),
                sz = __fmaf_rn(fz, r.inv.z, r.nb.z);
    const float gx = __fmaf_rn(fx, r.inv.x, r.fb.x), gy = __fmaf_rn(fy, r.inv.y, r.fb.y),
                gz = __fmaf_rn(fz, r.inv.z, r.fb.z);
    const bool by_x = (ny <= sx) & (nz <= sx) & (sy >= gx) & (sz >= gx) & (sx >= 0.f);
    const bool by_y = (nx <= sy) & (nz <= sy) & (sx >= gy) & (sz >= gy) & (sy >= 0.f);
    const bool by_z = (nx <= sz) & (ny <= sz) & (sx >= gz) & (sy >= gz) & (sz >= 0.f);
    return (by_x | by_y | by_z) || box_faces(b, o, d, scene_mag);
}

// Does the reference's predicate pass on every box above `slot`'s triangle?
// Each pair knows its next four ancestors, so the loads of a way of 22 boxes
// are 6 deep instead of 22.  Out of line: inlined, its registers made the
// search spill (mixed-material scene 1024^2 x 32 spp 34.7 ms, 34.0 this way).
static __device__ __noinline__ bool reference_reaches(const DevTree& T, int slot, f3 o, f3 d) {
    QuadRay r;
    // (in a scene with an infinite coordinate M is infinite here and no box is
    // told by its planes: on an infinite plane the reference's point is infinite
    // or a NaN, so the face tests decide)
    make_quad_ray(o, d, T.scene_mag, box_margin(o, T.scene_mag), r);
    for (uint32_t at = __ldg(T.leaf_up + slot); at != UP_ROOT;) {
        const uint4 up = ldg4u(T.pair_up + (at >> 1));
        const uint32_t a[4] = {at, up.x, up.y, up.z};
        at = up.w;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (a[k] != UP_ROOT && !reference_passes(child_box(T, a[k]), r, o, d, T.scene_mag)) return false;
    }
    return reference_passes(root_box(T), r, o, d, T.scene_mag);
}

// Closest hit where the reference's predicate decides every descent, without
// a stack: children left to right, back up by the parent links.  Rare (see
// the header), so out of line.
static __device__ __noinline__ Hit reference_search(const DevTree& T, f3 o, f3 d, float pf, bool filt, int inside,
                                                    int contact) {
    RayQ q = make_rayq(o, d, T.scene_mag);
    q.pf = pf;
    Hit h;
    h.t = __int_as_float(0x7f800000);
    h.slot = -1;
    float tn;
    if (!box_pred(root_box(T), q, &tn)) return h;
    if (T.root_w1 & LEAF_FLAG) {
        leaf_test_dyn<true>(T.tris, T.root_w0, T.root_w1 & ~LEAF_FLAG, q, filt, inside, contact, h);
        return h;
    }
    for (uint32_t at = T.root_w0 << 1;;) {
        if (box_pred(child_box(T, at), q, &tn) && !(tn > h.t * q.pf + q.M)) {
            const uint2 w = __ldg(reinterpret_cast<const uint2*>(&T.pairs[at >> 1].t) + (at & 1u));
            if (!(w.y & LEAF_FLAG)) {
                at = w.x << 1;
                continue;
            }
            leaf_test_dyn<true>(T.tris, w.x, w.y & ~LEAF_FLAG, q, filt, inside, contact, h);
        }
        while (at & 1u) {
            at = __ldg(&T.pair_up[at >> 1].x);
            if (at == UP_ROOT) return h;
        }
        at |= 1u;
    }
}

// ---------------------------------------------------------------------------
// one ray per lane
// ---------------------------------------------------------------------------
constexpr uint32_t NO_WORD = QUAD_HOLE;  // neither node nor leaf
constexpr int SLOT_REFERENCE = -2;  // Hit::slot of a ray that is left to reference_search

// Stack entries a thread is given: what the deepest walk can need, but at most
// 20.  (On the 1.3 M-triangle icosphere and the mixed-material scene no ray
// holds more than 17 at once, where the bound from the tree is 39; a ray that
// would need more is left to reference_search.  28 entries leave the L1 cache
// 20 to 30 KB less: mixed-material scene 37.6 ms, with 20 37.0.)
__host__ __device__ inline int quad_stack_cap(const DevTree& T) {
    return (int)(T.quad_stack + 4 < 20 ? T.quad_stack + 4 : 20);
}

// A connection's ray asks whether something is hit before `dist` (nee_visible,
// light_req_visible: up to max(1e-5, 1e-4 dist) short of it counts as reached).
// One such hit answers it: the closest is no farther.  Below this distance its
// search ends with the first hit that the reference reaches (low-variance
// 641x479 x 16 spp 8.70 -> 8.40 ms, bidirectional Cornell box 8.85 -> 8.70).
__device__ __forceinline__ float enough_before(float dist) { return dist - 2.f * fmaxf(1e-5f, 1e-4f * dist); }

// What a search reads only at leaves: the ray, the pruning rule's margin in
// units of |d| (infinite: no pruning), NoSelfCondition's object ids (used when filt) and the
// distance below which any hit ends it (filtered rays only; at most 0: none).
// That distance and filt share a word: 0 is no filter.
__device__ __forceinline__ float filter_word(bool filt, float enough) { return !filt ? 0.f : enough == 0.f ? -1.f : enough; }
// In registers:
struct RayInRegs {
    const TriRec* tt;
    f3 ro, rd;
    float rm;
    float fw;
    int in, co;
    __device__ __forceinline__ void set(const DevTree* T, f3 o, f3 d, float M, bool filt, int inside, int contact,
                                        float enough) {
        tt = T ? T->tris : nullptr;
        ro = o;
        rd = d;
        rm = M;
        fw = filter_word(filt, enough);
        in = inside;
        co = contact;
    }
    __device__ __forceinline__ float margin() const { return rm; }
    __device__ __forceinline__ float enough() const { return fw; }
    __device__ __forceinline__ float length_d() const { return length(rd); }
    // lane l's (every lane of the warp calls these)
    __device__ __forceinline__ void ray_of(int l, f3& o, f3& d) const {
        constexpr unsigned FULL = 0xffffffffu;
        o = mk(__shfl_sync(FULL, ro.x, l), __shfl_sync(FULL, ro.y, l), __shfl_sync(FULL, ro.z, l));
        d = mk(__shfl_sync(FULL, rd.x, l), __shfl_sync(FULL, rd.y, l), __shfl_sync(FULL, rd.z, l));
    }
    __device__ __forceinline__ const TriRec* tris_of(int l) const {
        return reinterpret_cast<const TriRec*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(tt), l));
    }
    __device__ __forceinline__ void ids_of(int l, bool& filt, int& inside, int& contact) const {
        constexpr unsigned FULL = 0xffffffffu;
        filt = __shfl_sync(FULL, fw, l) != 0.f;
        inside = __shfl_sync(FULL, in, l);
        contact = __shfl_sync(FULL, co, l);
    }
};
// or in shared memory, word k of thread t at p[k * stride] of its own p: in
// registers the persistent loop spills at 6 CTAs (2^24 rays 2.30 ms, 2.16 this
// way)
constexpr int RAY_WORDS = 12;
struct RayInShared {
    float* p;
    int stride;
    __device__ __forceinline__ void put_ptr(int k, const void* v) const {
        const unsigned long long x = reinterpret_cast<unsigned long long>(v);
        p[k * stride] = __uint_as_float((uint32_t)x);
        p[(k + 1) * stride] = __uint_as_float((uint32_t)(x >> 32));
    }
    __device__ __forceinline__ static unsigned long long get_ptr(const float* q, int k, int stride) {
        return __float_as_uint(q[k * stride]) | (unsigned long long)__float_as_uint(q[(k + 1) * stride]) << 32;
    }
    __device__ __forceinline__ void set(const DevTree* T, f3 o, f3 d, float M, bool filt, int inside, int contact,
                                        float enough) {
        put_ptr(10, T ? T->tris : nullptr);
        p[0] = o.x;
        p[stride] = o.y;
        p[2 * stride] = o.z;
        p[3 * stride] = d.x;
        p[4 * stride] = d.y;
        p[5 * stride] = d.z;
        p[6 * stride] = M;
        p[7 * stride] = filter_word(filt, enough);
        p[8 * stride] = __int_as_float(inside);
        p[9 * stride] = __int_as_float(contact);
    }
    __device__ __forceinline__ const TriRec* tris_of(int l) const {
        return reinterpret_cast<const TriRec*>(get_ptr(p + (l - (int)(threadIdx.x & 31u)), 10, stride));
    }
    __device__ __forceinline__ float margin() const { return p[6 * stride]; }
    __device__ __forceinline__ float enough() const { return p[7 * stride]; }
    __device__ __forceinline__ float length_d() const { return length(mk(p[3 * stride], p[4 * stride], p[5 * stride])); }
    __device__ __forceinline__ void ray_of(int l, f3& o, f3& d) const {
        const float* q = p + (l - (int)(threadIdx.x & 31u));
        o = mk(q[0], q[stride], q[2 * stride]);
        d = mk(q[3 * stride], q[4 * stride], q[5 * stride]);
    }
    __device__ __forceinline__ void ids_of(int l, bool& filt, int& inside, int& contact) const {
        const float* q = p + (l - (int)(threadIdx.x & 31u));
        filt = q[7 * stride] != 0.f;
        inside = __float_as_int(q[8 * stride]);
        contact = __float_as_int(q[9 * stride]);
    }
};

template <class Ray>
struct SearchLane {
    Ray ray;
    const QuadNode* quads;
    QuadRay r;
    float lim;             // boxes entered beyond it are skipped
    Hit h;
    uint32_t cur, pend;    // the node or leaf to visit; the postponed leaf
    int sp;                // stack[0], stack[stride], ... below it are waiting

    __device__ __forceinline__ bool walking() const { return !(cur & QUAD_LEAF); }
    __device__ __forceinline__ bool at_leaf() const { return pend != NO_WORD && (cur & QUAD_LEAF); }
    __device__ __forceinline__ bool finished() const { return cur == NO_WORD && pend == NO_WORD; }
    __device__ __forceinline__ void clear() {
        quads = nullptr;
        ray.set(nullptr, mk(0, 0, 0), mk(0, 0, 0), 0.f, false, -1, -1, -1.f);
        r = QuadRay{mk(0, 0, 0), mk(0, 0, 0), mk(0, 0, 0)};
        lim = 0.f;
        h = Hit{0.f, -1};
        cur = pend = NO_WORD;
        sp = 0;
    }
    // starts at the root
    __device__ __forceinline__ void begin(const DevTree& T, f3 o, f3 d, float pf, bool filt, int inside,
                                          int contact, float enough = -1.f) {
        quads = T.quads;
        lim = INFINITY;
        sp = 0;
        pend = NO_WORD;
        const float M = box_margin(o, T.finite_mag);
        const bool ok = make_quad_ray(o, d, T.finite_mag, M, r) && quads;
        const float unit = min3(fabsf(r.inv.x), fabsf(r.inv.y), fabsf(r.inv.z));  // 1 / |d| to 1.7 / |d|
        ray.set(&T, o, d, pf < INFINITY ? M * unit : INFINITY, filt, inside, contact, enough);
        h = Hit{INFINITY, ok ? -1 : SLOT_REFERENCE};
        cur = ok ? 0u : NO_WORD;
    }
    __device__ __forceinline__ void pop(const uint32_t* stack, int stride) {
        cur = NO_WORD;
        if (sp > 0) {
            sp -= stride;
            cur = stack[sp];
        }
    }
    // the postponed leaf's triangles
    __device__ __forceinline__ uint32_t leaf(uint32_t& first) const {
        first = pend & ((1u << QUAD_COUNT_AT) - 1u);
        return pend >> QUAD_COUNT_AT & 7u;
    }
    // visits the node `cur`; `top`: the last `sp` with room for four more
    __device__ __forceinline__ void visit(uint32_t* stack, int stride, int top) {
        float4 t;
        uint4 w;
        quad_children(quads + cur, r, lim, t, w);
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
            pop(stack, stride);
        } else if (sp > top) {  // deeper than the stack: the reference's own walk needs none
            sp = 0;
            cur = pend = NO_WORD;
            h.slot = SLOT_REFERENCE;
        }
        if ((cur & QUAD_LEAF) && cur != NO_WORD && pend == NO_WORD) {  // postpone it and walk on
            pend = cur;
            pop(stack, stride);
        }
    }
    // a triangle hit that NoSelfCondition allows
    __device__ __forceinline__ void take(float t, int slot, float dd) {
        if (!(t < h.t || (t == h.t && slot > h.slot))) return;
        // a near-grazing hit turns pruning off for good (graze_check)
        const bool off = fabsf(dd) < GRAZE_COS * ray.length_d() || (h.slot >= 0 && !(lim < INFINITY));
        lim = off ? INFINITY : t * 1.001f + ray.margin();
        h = Hit{t, slot};
        if (t < ray.enough()) cur = pend = NO_WORD;
    }
    // the postponed leaf is done: the next one, if the walk stands at it
    __device__ __forceinline__ void leaf_done(const uint32_t* stack, int stride) {
        pend = NO_WORD;
        if ((cur & QUAD_LEAF) && cur != NO_WORD) {
            pend = cur;
            pop(stack, stride);
        }
    }
};

// the winner checked against the reference's boxes
__device__ __forceinline__ Hit settle(const DevTree& T, const Hit& h, f3 o, f3 d, float pf, bool filt, int inside,
                                      int contact) {
    if (h.slot == -1 || (h.slot >= 0 && reference_reaches(T, h.slot, o, d))) return h;
    return reference_search(T, o, d, pf, filt, inside, contact);
}

// Closest hit of this thread's ray on its own (any subset of a warp may call
// it).  Its stack: entries at stack[k * stride], k < cap.
__device__ __forceinline__ Hit search_closest(const DevTree& T, f3 o, f3 d, float pf, bool filt, int inside,
                                              int contact, uint32_t* stack, int stride, int cap) {
    SearchLane<RayInRegs> L;
    L.begin(T, o, d, pf, filt, inside, contact);
    const int top = (cap - 4) * stride;
    while (!L.finished()) {
        while (L.walking()) L.visit(stack, stride, top);
        if (L.pend == NO_WORD) break;
        uint32_t first;
        const uint32_t count = L.leaf(first);
        for (uint32_t k = 0; k < count; k++) {
            const int slot = (int)(first + k);
            float dd = 0.f;
            const float t = tri_slot_test(T.tris, slot, o, d, &dd);
            if (t >= 0.f && t <= L.h.t && (!filt || noself_slot(T.tris, slot, d, inside, contact))) L.take(t, slot, dd);
        }
        L.leaf_done(stack, stride);
    }
    return settle(T, L.h, o, d, pf, filt, inside, contact);
}

// a warp's scratch of a leaf phase, in shared memory
struct WarpLeaves {
    float t[32], dd[32];
    int slot[32];                       // a lane's closest candidate (-1: none)
    uint8_t item[32 * QUAD_LEAF_MAX];   // triangles: lane | index in its leaf << 5
};

// Tests the postponed leaves of a warp's lanes (`has`): their triangles are
// dealt out over all 32 lanes, one each, so that leaves of different lengths do
// not leave lanes idle (the test in each lane's own loop kept 7 to 14 lanes
// busy, this 24 to 29; the batch of 2^24 rays 2.69 -> 2.31 ms).  The distance
// half of the test runs once for the triangles whose edges the rays pass
// inside, about one in ten.  Every lane of the warp calls it.
// tris_of(tris, l): the triangles of lane l's tree.  Returns this lane's count.
// FEW: a pass's candidates, up to so many, are handed back to their rays one by
// one (25 instructions each), more by groups (60): 3 in the persistent loop
// (Cornell box 3.95 -> 3.55 ms); where a warp waits for its own rays the groups'
// longer chain costs more than it saves (megakernel 4.92 -> 5.11 ms).
template <int FEW, class Ray, class TrisOf>
__device__ __forceinline__ uint32_t warp_leaves(SearchLane<Ray>& L, bool has, WarpLeaves& W, const uint32_t* stack,
                                                int stride, TrisOf tris_of) {
    constexpr unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    uint32_t first = 0u, count = 0u;
    if (has) count = L.leaf(first);
    const unsigned c0 = __ballot_sync(FULL, count & 1u), c1 = __ballot_sync(FULL, count & 2u),
                   c2 = __ballot_sync(FULL, count & 4u);
    const uint32_t before = __popc(c0 & lt_mask) + 2u * __popc(c1 & lt_mask) + 4u * __popc(c2 & lt_mask);
    const uint32_t total = __popc(c0) + 2u * __popc(c1) + 4u * __popc(c2);
    for (uint32_t k = 0; k < count; k++) W.item[before + k] = (uint8_t)(lane | k << 5);
    __syncwarp();
    // the edge tests of all; those inside stay in the list
    uint32_t left = 0;
    for (uint32_t base = 0; base < total; base += 32u) {
        const bool on = base + lane < total;
        const uint32_t it = on ? W.item[base + lane] : lane;
        const int own = (int)(it & 31u);
        f3 ro, rd;
        L.ray.ray_of(own, ro, rd);
        const int slot = (int)(__shfl_sync(FULL, first, own) + (it >> 5));
        const TriRec* rt = tris_of(own);
        const bool in = on && tri_slot_inside(rt, slot, ro, rd);
        const unsigned im = __ballot_sync(FULL, in);
        if (in) W.item[left + __popc(im & lt_mask)] = (uint8_t)it;
        left += __popc(im);
        __syncwarp();
    }
    // the distances of the few that are left
    for (uint32_t base = 0; base < left; base += 32u) {
        const bool on = base + lane < left;
        const uint32_t it = on ? W.item[base + lane] : lane;
        const int own = (int)(it & 31u);
        f3 ro, rd;
        L.ray.ray_of(own, ro, rd);
        const int slot = (int)(__shfl_sync(FULL, first, own) + (it >> 5));
        const float best = __shfl_sync(FULL, L.h.t, own);
        const TriRec* rt = tris_of(own);
        float t = -1.f, dd = 0.f;
        if (on) t = tri_slot_distance(rt, slot, ro, rd, &dd);
        bool cand = t >= 0.f && t <= best;
        if (__any_sync(FULL, cand)) {
            bool rf;
            int ri, rc;
            L.ray.ids_of(own, rf, ri, rc);
            if (cand && rf) cand = noself_slot(rt, slot, rd, ri, rc);
            unsigned cm = __ballot_sync(FULL, cand);
            if (__popc(cm) <= FEW) {
                for (; cm; cm &= cm - 1u) {
                    const int b = __ffs(cm) - 1;
                    const int bo = __shfl_sync(FULL, own, b), bs = __shfl_sync(FULL, slot, b);
                    const float bt = __shfl_sync(FULL, t, b), bd = __shfl_sync(FULL, dd, b);
                    if ((int)lane == bo) L.take(bt, bs, bd);
                }
                continue;
            }
            // A ray's candidates sit on consecutive lanes (at most 7): the
            // closest is found among them, and the group's first lane hands
            // it to the ray's own.
            const int group = on ? own : 32 + (int)lane;
            float bt = cand ? t : INFINITY, bd = dd;
            int bs = cand ? slot : -1;  // (a candidate's distance may be infinite)
#pragma unroll
            for (int k = 1; k < 8; k <<= 1) {
                const float t2 = __shfl_down_sync(FULL, bt, k), d2 = __shfl_down_sync(FULL, bd, k);
                const int s2 = __shfl_down_sync(FULL, bs, k), g2 = __shfl_down_sync(FULL, group, k);
                if (lane + k < 32u && g2 == group && (t2 < bt || (t2 == bt && s2 > bs))) {
                    bt = t2;
                    bd = d2;
                    bs = s2;
                }
            }
            const int g0 = __shfl_up_sync(FULL, group, 1);
            W.slot[lane] = -1;
            __syncwarp();
            if (on && (lane == 0 || g0 != group) && bs >= 0) {
                W.t[own] = bt;
                W.dd[own] = bd;
                W.slot[own] = bs;
            }
            __syncwarp();
            if (W.slot[lane] >= 0) L.take(W.t[lane], W.slot[lane], W.dd[lane]);
            __syncwarp();
        }
    }
    if (has) L.leaf_done(stack, stride);
    __syncwarp();
    return count;
}

// Closest hits of a warp's rays, one per lane with `on`; every lane of the
// warp calls it.  ONE_TREE: all rays in the tree T (else each lane's own T).
template <bool ONE_TREE = true>
__device__ __forceinline__ Hit search_warp(const DevTree& T, bool on, f3 o, f3 d, float pf, bool filt, int inside,
                                           int contact, uint32_t* stack, int stride, int cap, WarpLeaves& leaves,
                                           float enough = -1.f) {
    constexpr unsigned FULL = 0xffffffffu;
    SearchLane<RayInRegs> L;
    L.clear();
    if (on) L.begin(T, o, d, pf, filt, inside, contact, enough);
    const int top = (cap - 4) * stride;
    for (;;) {
        const bool walking = L.walking();
        const unsigned wm = __ballot_sync(FULL, walking), lm = __ballot_sync(FULL, L.at_leaf());
        if (!(wm | lm)) break;
        if (lm && (wm == 0 || __popc(lm) >= 8)) {
            warp_leaves<32>(L, L.pend != NO_WORD, leaves, stack, stride,
                        [&](int from) { return ONE_TREE ? T.tris : L.ray.tris_of(from); });
        } else if (walking) {
            for (int k = 0; k < 6 && L.walking(); k++) L.visit(stack, stride, top);
        }
    }
    return on ? settle(T, L.h, o, d, pf, filt, inside, contact) : Hit{INFINITY, -1};
}

}  // namespace wr
