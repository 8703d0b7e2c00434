// quad_build.cpp — the four-wide tree over the reference tree's leaves.
//
// The reference's median-split tree decides which triangles a ray may hit, but
// it is a poor order to search them in: on the 512,006-triangle mixed-material
// scene a bounce ray visits 52 of its nodes, 17 of this tree's.  A leaf here is
// a reference leaf with its box unchanged and a node's box is the union of
// leaf boxes, so every triangle the reference tests is under boxes that
// contain its leaf's: the search sees a superset of the reference's
// candidates, and wr_quad.cuh checks the winner against the reference's own
// boxes.
//
// Binned surface-area heuristic, in two levels so that it runs in parallel:
// the reference's subtrees of at most CLUSTER leaves are the units of the
// upper tree, and each is built over its own leaves by one thread.  The binary
// tree is then cut into four-wide nodes by the cut of least summed area
// (dynamic programming over the number of slots a subtree may take: Wald,
// Benthin, Boulos 2008; Ylitie, Karras, Laine 2017).
#include "quad_build.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#ifdef _OPENMP
#include <omp.h>
#endif

namespace wr {
namespace {

constexpr int BINS = 16;
constexpr uint32_t CLUSTER = 64;
// bin of a centre (a box of a vertex that is not finite: the first)
int bin_of(float c, float base, float scale) {
    const float x = (c - base) * scale;
    return x > 0.f ? (x < (float)BINS ? (int)x : BINS - 1) : 0;
}

constexpr float NODE_COST = 1.0f, TRI_COST = 0.6f;  // one four-wide node against one triangle test

struct QBox {
    float lo[3], hi[3];
    void clear() {
        for (int k = 0; k < 3; k++) {
            lo[k] = INFINITY;
            hi[k] = -INFINITY;
        }
    }
    void add(const QBox& b) {
        for (int k = 0; k < 3; k++) {
            lo[k] = std::min(lo[k], b.lo[k]);
            hi[k] = std::max(hi[k], b.hi[k]);
        }
    }
    bool finite() const {
        bool f = true;
        for (int k = 0; k < 3; k++) f = f && std::isfinite(lo[k]) && std::isfinite(hi[k]);
        return f;
    }
    float area() const {
        const float x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
        return x < 0.f ? 0.f : x * y + y * z + z * x;
    }
};

// a unit of a build: a leaf (or a cluster) with its box and triangle count
struct Item {
    QBox box;
    uint32_t word;   // child word of a leaf, index of a cluster
    uint32_t count;  // triangles
};

struct BinNode {
    QBox box;
    uint32_t word;       // items: Item::word
    int32_t l, r;        // -1: an item
    float cost[3];       // least cost in at most 1, 2, 3 slots
    uint8_t split[2];    // slots of the left child when given 2, 3 (0: one slot fewer)
    uint8_t split4;      // the same when given 4 (a node of its own)
};

// the box of items a[0, n), and where the surface-area heuristic parts them:
// they are partitioned, the left part's size is returned
size_t split_items(Item* a, size_t n, QBox& box) {
    QBox cen;
    box.clear();
    cen.clear();
    for (size_t i = 0; i < n; i++) {
        box.add(a[i].box);
        for (int k = 0; k < 3; k++) {
            const float c = a[i].box.lo[k] + a[i].box.hi[k];
            cen.lo[k] = std::min(cen.lo[k], c);
            cen.hi[k] = std::max(cen.hi[k], c);
        }
    }
    if (n == 1) return 1;
    float best = INFINITY;
    int best_d = -1, best_s = 0;
    // bins of all three axes in one pass (scale 0: the axis cannot be split)
    QBox bb[3][BINS];
    uint32_t bc[3][BINS] = {};
    float scale[3];
    for (int d = 0; d < 3; d++) {
        const float w = cen.hi[d] - cen.lo[d];
        scale[d] = w > 0.f && (float)BINS / w < INFINITY ? (float)BINS / w : 0.f;
        for (QBox& x : bb[d]) x.clear();
    }
    for (size_t i = 0; i < n; i++)
        for (int d = 0; d < 3; d++) {
            const int k = bin_of(a[i].box.lo[d] + a[i].box.hi[d], cen.lo[d], scale[d]);
            bb[d][k].add(a[i].box);
            bc[d][k] += a[i].count;
        }
    for (int d = 0; d < 3; d++) {
        if (scale[d] == 0.f) continue;
        float ra[BINS];
        uint32_t rc[BINS], c = 0;
        QBox acc;
        acc.clear();
        for (int k = BINS - 1; k > 0; k--) {
            acc.add(bb[d][k]);
            c += bc[d][k];
            ra[k] = acc.area();
            rc[k] = c;
        }
        acc.clear();
        c = 0;
        for (int k = 0; k + 1 < BINS; k++) {
            acc.add(bb[d][k]);
            c += bc[d][k];
            if (!c || !rc[k + 1]) continue;
            const float cost = acc.area() * (float)c + ra[k + 1] * (float)rc[k + 1];
            if (cost < best) {
                best = cost;
                best_d = d;
                best_s = k;
            }
        }
    }
    size_t m = 0;
    if (best_d >= 0) {
        const float base = cen.lo[best_d], sc = scale[best_d];
        m = (size_t)(std::partition(a, a + n, [&](const Item& it) {
                         return bin_of(it.box.lo[best_d] + it.box.hi[best_d], base, sc) <= best_s;
                     }) -
                     a);
    }
    return m == 0 || m == n ? n / 2 : m;  // equal centres: halves, in the order they have
}

// binary SAH tree over a[0, n): out[0] is its root, children come after their
// parents
void build_binary(Item* items, size_t n, std::vector<BinNode>& out) {
    struct Job {
        Item* a;
        size_t n;
        int32_t at;
    };
    out.clear();
    out.emplace_back();
    std::vector<Job> jobs{{items, n, 0}};
    while (!jobs.empty()) {
        const Job j = jobs.back();
        jobs.pop_back();
        const size_t m = split_items(j.a, j.n, out[j.at].box);
        if (j.n == 1) {
            out[j.at].word = j.a[0].word;
            out[j.at].l = out[j.at].r = -1;
            out[j.at].cost[0] = (float)j.a[0].count;  // times area and TRI_COST below
            continue;
        }
        const int32_t l = (int32_t)out.size();
        out.emplace_back();
        out.emplace_back();
        out[j.at].l = l;
        out[j.at].r = l + 1;
        jobs.push_back({j.a, m, l});
        jobs.push_back({j.a + m, j.n - m, l + 1});
    }
}

// the same by tasks: the halves of a large range are built beside each other
// and put together
void build_binary_tasks(Item* a, size_t n, std::vector<BinNode>& out) {
    if (n < 512) {
        build_binary(a, n, out);
        return;
    }
    BinNode root{};
    const size_t m = split_items(a, n, root.box);
    std::vector<BinNode> half[2];
#pragma omp task default(shared)
    build_binary_tasks(a, m, half[0]);
#pragma omp task default(shared)
    build_binary_tasks(a + m, n - m, half[1]);
#pragma omp taskwait
    root.l = 1;
    root.r = 1 + (int32_t)half[0].size();
    out.clear();
    out.reserve(1 + half[0].size() + half[1].size());
    out.push_back(root);
    for (int k = 0; k < 2; k++) {
        const int32_t by = k ? root.r : root.l;
        for (BinNode b : half[k]) {
            if (b.l >= 0) {
                b.l += by;
                b.r += by;
            }
            out.push_back(b);
        }
    }
}

// least costs of nodes [first, end) (children come after their parents).
// `cluster_cost` (may be null): the cost of the tree below each item.
void cut_costs(std::vector<BinNode>& nodes, int32_t first, const std::vector<float>* cluster_cost) {
    for (int32_t i = (int32_t)nodes.size() - 1; i >= first; i--) {
        BinNode& n = nodes[i];
        const float a = n.box.area();
        if (n.l < 0) {
            const float c = cluster_cost ? (*cluster_cost)[n.word] : n.cost[0] * a * TRI_COST;
            n.cost[0] = n.cost[1] = n.cost[2] = c;
            continue;
        }
        const BinNode &l = nodes[n.l], &r = nodes[n.r];
        const float c2 = l.cost[0] + r.cost[0];
        const float c3a = l.cost[0] + r.cost[1], c3b = l.cost[1] + r.cost[0];
        const float c4[3] = {l.cost[0] + r.cost[2], l.cost[1] + r.cost[1], l.cost[2] + r.cost[0]};
        int s4 = 0;
        for (int k = 1; k < 3; k++)
            if (c4[k] < c4[s4]) s4 = k;
        n.split4 = (uint8_t)(s4 + 1);
        n.cost[0] = c4[s4] + a * NODE_COST;  // a node of its own with four slots
        n.cost[1] = n.cost[0];
        n.split[0] = 0;
        if (c2 < n.cost[1]) {
            n.cost[1] = c2;
            n.split[0] = 1;
        }
        n.cost[2] = n.cost[1];
        n.split[1] = 0;
        if (std::min(c3a, c3b) < n.cost[2]) {
            n.cost[2] = std::min(c3a, c3b);
            n.split[1] = c3a <= c3b ? 1 : 2;
        }
    }
}

// the subtrees that fill the slots of a cut: node i with at most `slots` of them
void cut(const std::vector<BinNode>& nodes, int32_t i, int slots, int32_t* out, int* n) {
    const BinNode& b = nodes[i];
    if (b.l >= 0)
        for (; slots > 1; slots--)
            if (b.split[slots - 2]) {
                cut(nodes, b.l, b.split[slots - 2], out, n);
                cut(nodes, b.r, slots - b.split[slots - 2], out, n);
                return;
            }
    out[(*n)++] = i;
}

void set_child(QuadNode& q, int k, const QBox* b, uint32_t word) {
    // an unused slot: a box that no ray meets
    const float none_lo = 1e30f, none_hi = -1e30f;
    (&q.lox.x)[k] = b ? b->lo[0] : none_lo;
    (&q.loy.x)[k] = b ? b->lo[1] : none_lo;
    (&q.loz.x)[k] = b ? b->lo[2] : none_lo;
    (&q.hix.x)[k] = b ? b->hi[0] : none_hi;
    (&q.hiy.x)[k] = b ? b->hi[1] : none_hi;
    (&q.hiz.x)[k] = b ? b->hi[2] : none_hi;
    (&q.child.x)[k] = word;
}

// the four-wide nodes of the binary tree at `root`, breadth first from
// out[0].  Items become `word_of(item word)`; nodes' child words are indices
// into `out`.
template <class WordOf>
void emit(const std::vector<BinNode>& nodes, int32_t root, std::vector<QuadNode>& out, WordOf word_of) {
    std::vector<std::pair<int32_t, uint32_t>> todo{{root, 0u}};
    out.emplace_back();
    for (size_t at = 0; at < todo.size(); at++) {
        const auto [i, q] = todo[at];
        int32_t ch[4];
        int n = 0;
        if (nodes[i].l < 0) {
            ch[n++] = i;  // a tree of one item
        } else {
            cut(nodes, nodes[i].l, nodes[i].split4, ch, &n);
            cut(nodes, nodes[i].r, 4 - nodes[i].split4, ch, &n);
        }
        for (int k = 0; k < 4; k++) {
            if (k >= n) {
                set_child(out[q], k, nullptr, QUAD_HOLE);
                continue;
            }
            const BinNode& c = nodes[ch[k]];
            uint32_t word;
            if (c.l < 0) {
                word = word_of(c.word);
            } else {
                word = (uint32_t)out.size();
                out.emplace_back();
                todo.push_back({ch[k], word});
            }
            set_child(out[q], k, &c.box, word);
        }
    }
}

}  // namespace

// the deepest walk's stack: at every node all children but the one walked into
// wait on it
static uint32_t stack_need(const std::vector<QuadNode>& q) {
    std::vector<uint32_t> need(q.size(), 0u);  // entries waiting when the node is entered (parents come first)
    uint32_t most = 0;
    for (size_t i = 0; i < q.size(); i++) {
        uint32_t n = 0;
        for (int k = 0; k < 4; k++) n += (&q[i].child.x)[k] != QUAD_HOLE;
        const uint32_t below = need[i] + (n ? n - 1 : 0);
        most = std::max(most, below);
        for (int k = 0; k < 4; k++) {
            const uint32_t w = (&q[i].child.x)[k];
            if (!(w & QUAD_LEAF)) need[w] = below;
        }
    }
    return most;
}

// the tree over `items`, the leaves with finite boxes; node_item[n]: the first
// of them at or after node n
static void build_finite(const HostTree& t, const std::vector<uint32_t>& node_item, std::vector<Item>& items,
                         int threads, QuadLayout& L) {
    (void)threads;
    if (items.empty()) {  // no triangles: a root of holes
        L.quads.emplace_back();
        for (int k = 0; k < 4; k++) set_child(L.quads[0], k, nullptr, QUAD_HOLE);
        return;
    }
    // clusters: the reference's largest subtrees of at most CLUSTER items
    // (a subtree's leaves are consecutive in pre-order)
    std::vector<std::pair<uint32_t, uint32_t>> range;  // item ranges
    {
        std::vector<std::pair<uint32_t, uint32_t>> todo{{0u, (uint32_t)items.size()}};  // node, end of its items
        while (!todo.empty()) {
            const auto [n, end] = todo.back();
            todo.pop_back();
            const uint32_t a = node_item[n];
            if (a == end) continue;
            bool unit = t.left[n] < 0;
            if (!unit && end - a <= CLUSTER) {  // compact: no gap between what the reference's plane put together
                float sum = 0.f;
                for (uint32_t i = a; i < end; i++) sum += items[i].box.area();
                QBox b;
                std::memcpy(b.lo, &t.box[6 * (size_t)n], 12);
                std::memcpy(b.hi, &t.box[6 * (size_t)n + 3], 12);
                unit = b.area() <= sum;
            }
            if (unit) {
                range.push_back({a, end});
                continue;
            }
            const uint32_t mid = node_item[t.right[n]];
            todo.push_back({(uint32_t)t.right[n], end});
            todo.push_back({(uint32_t)t.left[n], mid});
        }
    }
    const size_t nc = range.size();
    std::vector<std::vector<QuadNode>> sub(nc);
    std::vector<Item> top(nc);
    std::vector<float> sub_cost(nc);
#ifdef _OPENMP
#pragma omp parallel num_threads(threads)
#endif
    {
        std::vector<BinNode> bin;
#ifdef _OPENMP
#pragma omp for schedule(dynamic, 4)
#endif
        for (size_t c = 0; c < nc; c++) {
            const uint32_t a = range[c].first, e = range[c].second;
            top[c].word = (uint32_t)c;
            top[c].count = 0;
            for (uint32_t i = a; i < e; i++) top[c].count += items[i].count;
            build_binary(&items[a], e - a, bin);
            cut_costs(bin, 0, nullptr);
            top[c].box = bin[0].box;
            sub_cost[c] = bin[0].cost[0];
            if (e - a > 1 || nc == 1) emit(bin, 0, sub[c], [](uint32_t w) { return w; });
        }
    }
    if (nc == 1) {
        L.quads.swap(sub[0]);
        return;
    }
    std::vector<BinNode> bin;
#ifdef _OPENMP
#pragma omp parallel num_threads(threads)
#pragma omp single
#endif
    build_binary_tasks(top.data(), nc, bin);
    cut_costs(bin, 0, &sub_cost);
    // the upper tree, its clusters marked by the leaf bit for now; the
    // clusters' nodes follow it in the order it reaches them
    std::vector<QuadNode> upper;
    std::vector<size_t> base(nc, 0);
    std::vector<uint32_t> order;
    emit(bin, 0, upper, [&](uint32_t c) {
        order.push_back(c);
        return c | QUAD_LEAF;
    });
    size_t total = upper.size();
    for (uint32_t c : order) {
        base[c] = total;
        total += sub[c].size();
    }
    for (QuadNode& q : upper)
        for (int k = 0; k < 4; k++) {
            uint32_t& w = (&q.child.x)[k];
            if (w == QUAD_HOLE || !(w & QUAD_LEAF)) continue;
            const uint32_t c = w & ~QUAD_LEAF;
            w = sub[c].empty() ? items[range[c].first].word : (uint32_t)base[c];
        }
    L.quads.resize(total);
    std::memcpy(L.quads.data(), upper.data(), sizeof(QuadNode) * upper.size());
#ifdef _OPENMP
#pragma omp parallel for num_threads(threads) schedule(dynamic, 64)
#endif
    for (size_t c = 0; c < nc; c++)
        for (size_t k = 0; k < sub[c].size(); k++) {
            QuadNode q = sub[c][k];
            for (int j = 0; j < 4; j++) {
                uint32_t& w = (&q.child.x)[j];
                if (!(w & QUAD_LEAF)) w += (uint32_t)base[c];
            }
            L.quads[base[c] + k] = q;
        }
}

// Leaves whose box has an infinite or NaN plane, above the root: their boxes say
// nothing to the search, so every ray tests their triangles (the check of the
// winner runs the reference's tests on their boxes).  The last slot of a node
// leads on, so that its word lies below the leaves on a walk's stack.  Faster
// than the walk of the reference's tree, which such a plane turns into face
// tests throughout, for any number of them (2^18 rays with 80 such words 0.42
// against 2.65 ms, with 5,115 30.5 against 155).
static void put_above(const std::vector<uint32_t>& odd, QuadLayout& L) {
    const uint32_t add = (uint32_t)(odd.size() + 2) / 3;
    std::vector<QuadNode> q(add);
    const QBox all{{-1e30f, -1e30f, -1e30f}, {1e30f, 1e30f, 1e30f}};  // met by every ray of the search
    for (uint32_t i = 0; i < add; i++) {
        for (uint32_t k = 0; k < 3; k++) {
            const size_t at = 3 * (size_t)i + k;
            set_child(q[i], k, at < odd.size() ? &all : nullptr, at < odd.size() ? odd[at] : QUAD_HOLE);
        }
        set_child(q[i], 3, &all, i + 1);
    }
    for (QuadNode b : L.quads) {
        for (int k = 0; k < 4; k++) {
            uint32_t& w = (&b.child.x)[k];
            if (!(w & QUAD_LEAF)) w += add;
        }
        q.push_back(b);
    }
    L.quads.swap(q);
}

QuadLayout build_quads(const HostTree& t, int threads) {
    QuadLayout L;
    const uint32_t N = t.num_nodes();
#ifdef _OPENMP
    if (threads <= 0) threads = omp_get_max_threads();
#endif
    (void)threads;
    // parent links of the reference tree, in the device layout's numbering
    // (pairs in pre-order, slots leaf by leaf), and the leaves as items; a leaf
    // of more than QUAD_LEAF_MAX triangles is several items with one box
    std::vector<uint32_t> pair_of(N, 0u), slot_of(N, 0u), parent(N, 0u);
    std::vector<uint32_t> node_item(N, 0u);  // first item at or after each node
    uint32_t np = 0, slots = 0, ni = 0;
    for (uint32_t n = 0; n < N; n++) {
        node_item[n] = ni;
        slot_of[n] = slots;
        if (t.left[n] >= 0) {
            pair_of[n] = np++;
            parent[t.left[n]] = parent[t.right[n]] = n;
        } else {
            ni += (t.leaf_count[n] + QUAD_LEAF_MAX - 1) / QUAD_LEAF_MAX;
            slots += t.leaf_count[n];
        }
    }
    L.leaf_up.resize(slots);
    L.pair_up.resize(np);
    std::vector<Item> items(ni);
    auto up = [&](uint32_t n) {
        return n == 0 ? UP_ROOT : pair_of[parent[n]] << 1 | (uint32_t)(t.right[parent[n]] == (int32_t)n);
    };
    bool finite = true;
#ifdef _OPENMP
#pragma omp parallel for num_threads(threads) schedule(static, 4096) reduction(&& : finite) if (N > 16384)
#endif
    for (uint32_t n = 0; n < N; n++) {
        if (t.left[n] >= 0) {
            uint32_t a[4], m = n;
            for (uint32_t& u : a) {  // (past the root: UP_ROOT again)
                u = up(m);
                m = parent[m];
            }
            L.pair_up[pair_of[n]] = make_uint4(a[0], a[1], a[2], a[3]);
            continue;
        }
        for (uint32_t k = 0, i = node_item[n]; k < t.leaf_count[n]; k += QUAD_LEAF_MAX, i++) {
            Item& it = items[i];
            std::memcpy(it.box.lo, &t.box[6 * (size_t)n], 12);
            std::memcpy(it.box.hi, &t.box[6 * (size_t)n + 3], 12);
            finite = finite && it.box.finite();
            it.count = std::min(QUAD_LEAF_MAX, t.leaf_count[n] - k);
            it.word = QUAD_LEAF | it.count << QUAD_COUNT_AT | (slot_of[n] + k);
        }
        for (uint32_t k = 0; k < t.leaf_count[n]; k++) L.leaf_up[slot_of[n] + k] = up(n);
    }
    if (slots > QUAD_MAX_SLOTS) return L;
    // leaves with an infinite or NaN bound go above the tree of the others
    std::vector<uint32_t> odd;
    if (!finite) {
        std::vector<Item> rest;
        rest.reserve(ni);
        for (uint32_t n = 0, i = 0; n < N; n++) {
            const uint32_t first = i;
            node_item[n] = (uint32_t)rest.size();
            if (t.left[n] < 0) i += (t.leaf_count[n] + QUAD_LEAF_MAX - 1) / QUAD_LEAF_MAX;
            for (uint32_t k = first; k < i; k++) {
                if (items[k].box.finite()) rest.push_back(items[k]);
                else odd.push_back(items[k].word);
            }
        }
        items.swap(rest);
    }
    build_finite(t, node_item, items, threads, L);
    if (!odd.empty()) put_above(odd, L);
    L.stack = stack_need(L.quads);
    return L;
}

}  // namespace wr
