// kdtree_build.cpp — parallel host build of the reference scene tree
// (KDTree::build / splitBest, kdtree.cpp:141-258) and its device layout.
//
// The topology must equal the reference's exactly: the device traversal
// evaluates the reference's own box predicate on the reference's own boxes,
// which is what makes hit ids bit-exact.  The rules are therefore the
// reference's; the implementation is not: distinct vertices are found with a
// per-thread stamp array instead of an unordered_set, and subtrees above a
// size threshold are built as OpenMP tasks.
#include "kdtree_build.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#ifdef _OPENMP
#include <omp.h>
#endif

namespace wr {
namespace {

struct BNode {
    std::unique_ptr<BNode> l, r;
    float box[6];
    std::vector<uint32_t> tris;  // leaves only
    uint32_t depth = 0;
    uint32_t nodes = 1, leaves = 1, ntris = 0, max_depth = 0;  // of the subtree
};

struct Builder {
    const float* V;
    const uint32_t* T;
    uint32_t nv;

    struct Scratch {
        std::vector<uint32_t> stamp;
        uint32_t id = 0;
        std::vector<uint32_t> uniq;
        std::vector<float> coord;
    };

    Scratch& scratch() {
        thread_local Scratch s;
        thread_local const Builder* owner = nullptr;
        if (owner != this || s.stamp.size() != nv) {
            s.stamp.assign(nv, 0u);
            s.id = 0;
            owner = this;
        }
        return s;
    }

    inline float vc(uint32_t tri, int k, int d) const { return V[3 * (size_t)T[3 * (size_t)tri + k] + d]; }

    void build(BNode* nd, std::vector<uint32_t>& tl, uint32_t depth) {
        nd->depth = nd->max_depth = depth;
        const size_t cnt = tl.size();
        nd->ntris = (uint32_t)cnt;
        if (cnt == 0) {
            std::fill(nd->box, nd->box + 6, 0.f);
            return;
        }
        float mn[3], mx[3];
        for (int d = 0; d < 3; d++) mn[d] = mx[d] = vc(tl[0], 0, d);
        for (size_t i = 0; i < cnt; i++)
            for (int k = 0; k < 3; k++)
                for (int d = 0; d < 3; d++) {
                    float p = vc(tl[i], k, d);
                    mn[d] = p < mn[d] ? p : mn[d];
                    mx[d] = p > mx[d] ? p : mx[d];
                }
        for (int d = 0; d < 3; d++) {
            nd->box[d] = mn[d];
            nd->box[3 + d] = mx[d];
        }
        if (cnt <= 1) {
            nd->tris.swap(tl);
            return;
        }
        Scratch& S = scratch();
        if (++S.id == 0) {  // stamp wrap-around
            std::fill(S.stamp.begin(), S.stamp.end(), 0u);
            S.id = 1;
        }
        S.uniq.clear();
        for (size_t i = 0; i < cnt; i++)
            for (int k = 0; k < 3; k++) {
                uint32_t vi = T[3 * (size_t)tl[i] + k];
                if (S.stamp[vi] != S.id) {
                    S.stamp[vi] = S.id;
                    S.uniq.push_back(vi);
                }
            }
        const size_t nu = S.uniq.size();
        float bestRatio = 10.f, bestSplit = 0.f;
        int bestDim = 0;
        S.coord.resize(nu);
        for (int dim = 0; dim < 3; dim++) {
            for (size_t k = 0; k < nu; k++) S.coord[k] = V[3 * (size_t)S.uniq[k] + dim];
            std::nth_element(S.coord.begin(), S.coord.begin() + (nu >> 1), S.coord.end());
            const float split = S.coord[nu >> 1];
            uint32_t leftCount = 0;
            for (size_t i = 0; i < cnt; i++)
                leftCount += (vc(tl[i], 0, dim) <= split) | (vc(tl[i], 1, dim) <= split) | (vc(tl[i], 2, dim) <= split);
            const float ratio = (float)leftCount / (float)cnt;
            if (std::fabs((double)ratio - 0.5) < std::fabs((double)bestRatio - 0.5)) {
                bestRatio = ratio;
                bestDim = dim;
                bestSplit = split;
            }
        }
        if (bestRatio == 0.f || bestRatio == 1.f) {
            nd->tris.swap(tl);
            return;
        }
        std::vector<uint32_t> L, R;
        L.reserve(cnt);
        R.reserve(cnt);
        for (size_t i = 0; i < cnt; i++) {
            bool left = (vc(tl[i], 0, bestDim) <= bestSplit) | (vc(tl[i], 1, bestDim) <= bestSplit) |
                        (vc(tl[i], 2, bestDim) <= bestSplit);
            (left ? L : R).push_back(tl[i]);
        }
        std::vector<uint32_t>().swap(tl);
        nd->l.reset(new BNode);
        nd->r.reset(new BNode);
        BNode* l = nd->l.get();
        BNode* r = nd->r.get();
        if (cnt > 512) {  // worth a task (5120 triangles: 3.7 ms in one piece)
#pragma omp task default(shared) firstprivate(l, depth)
            {
                std::vector<uint32_t> Lt;
                Lt.swap(L);
                build(l, Lt, depth + 1);
            }
#pragma omp task default(shared) firstprivate(r, depth)
            {
                std::vector<uint32_t> Rt;
                Rt.swap(R);
                build(r, Rt, depth + 1);
            }
#pragma omp taskwait
        } else {
            build(l, L, depth + 1);
            build(r, R, depth + 1);
        }
        nd->nodes = 1 + l->nodes + r->nodes;
        nd->leaves = l->leaves + r->leaves;
        nd->max_depth = std::max(l->max_depth, r->max_depth);
    }
};

// Writes the subtree at `nd`, whose first node has index `id` and whose leaves'
// triangles start at `tri`, and frees what is below it.  Large subtrees are
// tasks (a node knows the size of its subtree, so each knows its place).
void flatten(BNode* nd, uint32_t id, uint32_t tri, HostTree& t) {
    // an explicit stack keeps deep trees off the call stack
    struct At {
        std::unique_ptr<BNode> own;
        BNode* n;
        uint32_t id, tri;
    };
    std::vector<At> st;
    st.push_back({nullptr, nd, id, tri});
    while (!st.empty()) {
        At a = std::move(st.back());
        st.pop_back();
        BNode* n = a.n;
        std::copy(n->box, n->box + 6, t.box.begin() + 6 * (ptrdiff_t)a.id);
        if (!n->l) {
            t.left[a.id] = t.right[a.id] = -1;
            t.leaf_first[a.id] = a.tri;
            t.leaf_count[a.id] = (uint32_t)n->tris.size();
            std::copy(n->tris.begin(), n->tris.end(), t.leaf_tris.begin() + a.tri);
            continue;
        }
        BNode *l = n->l.get(), *r = n->r.get();
        const uint32_t lid = a.id + 1, rid = lid + l->nodes, rtri = a.tri + l->ntris;
        t.left[a.id] = (int32_t)lid;
        t.right[a.id] = (int32_t)rid;
        t.leaf_first[a.id] = t.leaf_count[a.id] = 0;
        for (int k = 0; k < 2; k++) {
            At c{std::move(k ? n->r : n->l), k ? r : l, k ? rid : lid, k ? rtri : a.tri};
            if (c.n->nodes > 4096 && n->nodes > 8192) {
                BNode* root = c.own.release();
                const uint32_t cid = c.id, ctri = c.tri;
#pragma omp task default(shared) firstprivate(root, cid, ctri)
                {
                    flatten(root, cid, ctri, t);
                    delete root;
                }
            } else {
                st.push_back(std::move(c));
            }
        }
    }
#pragma omp taskwait
}

}  // namespace

HostTree build_reference_tree(const float* verts, uint32_t nv, const uint32_t* tris, uint32_t nt, int threads) {
    Builder b{verts, tris, nv};
    BNode root;
    std::vector<uint32_t> all(nt);
    for (uint32_t i = 0; i < nt; i++) all[i] = i;
#ifdef _OPENMP
    if (threads <= 0) threads = omp_get_max_threads();
#pragma omp parallel num_threads(threads)
#pragma omp single
#endif
    b.build(&root, all, 0);
    HostTree t;
    const size_t N = root.nodes;
    t.left.resize(N);
    t.right.resize(N);
    t.box.resize(6 * N);
    t.leaf_first.resize(N);
    t.leaf_count.resize(N);
    t.leaf_tris.resize(root.ntris);
    t.num_leaves = root.leaves;
    t.max_depth = root.max_depth;
#ifdef _OPENMP
#pragma omp parallel num_threads(threads)
#pragma omp single
#endif
    flatten(&root, 0, 0, t);
    (void)threads;
    return t;
}

DeviceLayout layout_for_device(const HostTree& t, const float* verts, uint32_t nv, const uint32_t* tris,
                               const int32_t* tri_obj, const uint32_t* tri_local) {
    DeviceLayout L;
    float mag = 0.f, finite = 0.f;
    for (size_t i = 0; i < 3 * (size_t)nv; i++) {
        const float a = std::fabs(verts[i]);
        mag = std::max(mag, a);
        finite = a < INFINITY ? std::max(finite, a) : finite;
    }
    L.scene_mag = mag;
    L.finite_mag = finite;
    const uint32_t N = t.num_nodes();
    if (N == 0) {
        for (int d = 0; d < 3; d++) L.root_lo[d] = L.root_hi[d] = 0.f;
        L.root_w0 = 0;
        L.root_w1 = LEAF_FLAG;
        return L;
    }
    // slots: leaves in pre-order (= left-to-right), each leaf reversed; pair
    // index of each internal node, in pre-order
    std::vector<uint32_t> slot_first(N, 0), pair_of(N, 0xffffffffu);
    uint32_t np = 0, ns = 0;
    for (uint32_t n = 0; n < N; n++) {
        if (t.left[n] >= 0) {
            pair_of[n] = np++;
        } else {
            slot_first[n] = ns;
            ns += t.leaf_count[n];
        }
    }
    L.slots.resize(ns);
    L.slot_of.assign(ns, 0u);
    L.pairs.resize(np);
    auto put_tri = [&](uint32_t slot, uint32_t gt) {
        TriRec& r = L.slots[slot];
        const uint32_t* tv = tris + 3 * (size_t)gt;
        const float* a = verts + 3 * (size_t)tv[0];
        const float* b = verts + 3 * (size_t)tv[1];
        const float* c = verts + 3 * (size_t)tv[2];
        uint32_t obj = (uint32_t)tri_obj[gt], loc = tri_local[gt];
        float w0, w1, w2;
        std::memcpy(&w0, &gt, 4);
        std::memcpy(&w1, &obj, 4);
        std::memcpy(&w2, &loc, 4);
        r.v0 = make_float4(a[0], a[1], a[2], w0);
        r.v1 = make_float4(b[0], b[1], b[2], w1);
        r.v2 = make_float4(c[0], c[1], c[2], w2);
        if (gt < L.slot_of.size()) L.slot_of[gt] = slot;
    };
    auto word = [&](uint32_t n, uint32_t& w0, uint32_t& w1) {
        if (t.left[n] < 0) {
            w0 = slot_first[n];
            w1 = t.leaf_count[n] | LEAF_FLAG;
        } else {
            w0 = pair_of[n];
            w1 = 0u;
        }
    };
#pragma omp parallel for schedule(static, 4096) if (N > 16384)
    for (uint32_t n = 0; n < N; n++) {
        if (t.left[n] < 0) {
            const uint32_t cnt = t.leaf_count[n];
            for (uint32_t k = 0; k < cnt; k++) put_tri(slot_first[n] + k, t.leaf_tris[t.leaf_first[n] + cnt - 1 - k]);
            continue;
        }
        NodePair& P = L.pairs[pair_of[n]];
        const float* lb = &t.box[6 * (size_t)t.left[n]];
        const float* rb = &t.box[6 * (size_t)t.right[n]];
        P.a = make_float4(lb[0], lb[1], lb[2], lb[3]);
        P.b = make_float4(lb[4], lb[5], rb[0], rb[1]);
        P.c = make_float4(rb[2], rb[3], rb[4], rb[5]);
        uint32_t a0, a1, b0, b1;
        word((uint32_t)t.left[n], a0, a1);
        word((uint32_t)t.right[n], b0, b1);
        P.t = make_uint4(a0, a1, b0, b1);
    }
    for (int d = 0; d < 3; d++) {
        L.root_lo[d] = t.box[d];
        L.root_hi[d] = t.box[3 + d];
    }
    word(0, L.root_w0, L.root_w1);
    return L;
}

}  // namespace wr
