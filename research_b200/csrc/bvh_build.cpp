// bvh_build.cpp — host binned-SAH BVH2 builder.
//
// Replaces the driver-built BLAS/TLAS of the reference
// (AccelStructure.cpp:98-330, PREFER_FAST_TRACE). Builds one binary tree
// over world-space triangles (32 centroid bins per axis, surface-area cost,
// leaves of at most 8 triangles, depth capped at 60 so a 64-entry traversal
// stack always suffices), then lays it out for the GPU: every inner node
// stores the boxes of both children, inner nodes in depth-first order.
// Large subtrees are built on separate threads. The same tree is also laid
// out 4-wide: a 4-wide node's children are a binary node's frontier of up to
// four nodes, grown by opening the inner frontier node of largest surface
// area (the leaves are the binary tree's leaves).

#include "rr_bvh.h"

#include <vector_functions.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <future>
#include <thread>

namespace rr {
namespace {

struct Box {
    float lo[3] = {INFINITY, INFINITY, INFINITY};
    float hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    void grow(const Box& b) {
        for (int a = 0; a < 3; ++a) { lo[a] = std::min(lo[a], b.lo[a]); hi[a] = std::max(hi[a], b.hi[a]); }
    }
    void grow(const float* p) {
        for (int a = 0; a < 3; ++a) { lo[a] = std::min(lo[a], p[a]); hi[a] = std::max(hi[a], p[a]); }
    }
    float area() const {
        if (!(hi[0] >= lo[0])) return 0.0f;
        const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
        return 2.0f * (dx * dy + dy * dz + dz * dx);
    }
};

struct Node {
    Box box;
    int32_t left = -1, right = -1;  // binary children; -1 = leaf
    uint32_t first = 0, count = 0;
};

constexpr int kBins = 32;
constexpr uint32_t kMaxLeaf = 8;
constexpr uint32_t kMaxDepth = 60;

struct Builder {
    const std::vector<Box>& boxes;
    const std::vector<float>& cent;  // 3 per tri
    std::vector<uint32_t>& order;
    std::vector<Node>& nodes;
    std::atomic<uint32_t> next{1};
    std::atomic<uint32_t> depth_max{0};

    void make_leaf(uint32_t idx, uint32_t first, uint32_t count) {
        nodes[idx].left = nodes[idx].right = -1;
        nodes[idx].first = first; nodes[idx].count = count;
    }

    void build(uint32_t idx, uint32_t first, uint32_t count, uint32_t depth) {
        uint32_t dm = depth_max.load();
        while (depth > dm && !depth_max.compare_exchange_weak(dm, depth)) {}
        Box box, cbox;
        for (uint32_t i = first; i < first + count; ++i) {
            box.grow(boxes[order[i]]);
            cbox.grow(&cent[3 * order[i]]);
        }
        nodes[idx].box = box;
        if (count <= 1 || depth >= kMaxDepth) { make_leaf(idx, first, count); return; }

        // Binned SAH over the three axes.
        float best_cost = INFINITY;
        int best_axis = -1, best_split = 0;
        for (int a = 0; a < 3; ++a) {
            const float ext = cbox.hi[a] - cbox.lo[a];
            if (!(ext > 0.0f)) continue;
            const float scale = float(kBins) * (1.0f - 1e-6f) / ext;
            uint32_t cnt[kBins] = {};
            Box bb[kBins];
            for (uint32_t i = first; i < first + count; ++i) {
                const uint32_t t = order[i];
                int b = int((cent[3 * t + a] - cbox.lo[a]) * scale);
                b = std::min(std::max(b, 0), kBins - 1);
                cnt[b]++;
                bb[b].grow(boxes[t]);
            }
            float right_area[kBins];
            uint32_t right_cnt[kBins];
            Box acc; uint32_t c = 0;
            for (int b = kBins - 1; b > 0; --b) {
                acc.grow(bb[b]); c += cnt[b];
                right_area[b] = acc.area(); right_cnt[b] = c;
            }
            acc = Box(); c = 0;
            for (int b = 0; b < kBins - 1; ++b) {
                acc.grow(bb[b]); c += cnt[b];
                if (c == 0 || right_cnt[b + 1] == 0) continue;
                const float cost = acc.area() * float(c) + right_area[b + 1] * float(right_cnt[b + 1]);
                if (cost < best_cost) { best_cost = cost; best_axis = a; best_split = b + 1; }
            }
        }
        const float leaf_cost = box.area() * float(count);
        const float split_cost = box.area() + best_cost;  // one node visit + children
        uint32_t mid;
        if (best_axis < 0) {
            if (count <= kMaxLeaf) { make_leaf(idx, first, count); return; }
            mid = first + count / 2;  // all centroids equal: split the list
        } else {
            if (count <= kMaxLeaf && leaf_cost <= split_cost) { make_leaf(idx, first, count); return; }
            const int a = best_axis;
            const float ext = cbox.hi[a] - cbox.lo[a];
            const float scale = float(kBins) * (1.0f - 1e-6f) / ext;
            auto it = std::partition(order.begin() + first, order.begin() + first + count, [&](uint32_t t) {
                int b = int((cent[3 * t + a] - cbox.lo[a]) * scale);
                b = std::min(std::max(b, 0), kBins - 1);
                return b < best_split;
            });
            mid = uint32_t(it - order.begin());
            if (mid == first || mid == first + count) mid = first + count / 2;
        }
        const uint32_t l = next.fetch_add(2);
        const uint32_t r = l + 1;
        nodes[idx].left = int32_t(l);
        nodes[idx].right = int32_t(r);
        const uint32_t nl = mid - first, nr = first + count - mid;
        if (depth < 8 && count > 50000) {
            auto fut = std::async(std::launch::async, [=]() { build(l, first, nl, depth + 1); });
            build(r, mid, nr, depth + 1);
            fut.get();
        } else {
            build(l, first, nl, depth + 1);
            build(r, mid, nr, depth + 1);
        }
    }
};

inline float4 mk4(float x, float y, float z, float w) { float4 v; v.x = x; v.y = y; v.z = z; v.w = w; return v; }
inline float i2f(int32_t i) { float f; std::memcpy(&f, &i, 4); return f; }

// 4-wide layout (8 float4 per node): lo.x, hi.x, lo.y, hi.y, lo.z, hi.z of
// children 0..3, then their references (>= 0 a node, < 0 a leaf starting at
// triangle ~ref) and their triangle counts. An unused child slot gets a
// point box at 1e30 on every axis, which no ray reaches within its tmax.
struct Wide4 {
    const std::vector<Node>& nodes;
    std::vector<float4>& out;
    int32_t emit(const std::vector<uint32_t>& kids) {
        const int32_t idx = int32_t(out.size() / 8);
        out.resize(out.size() + 8);
        float lo[3][4], hi[3][4];
        int32_t ref[4] = {0, 0, 0, 0}, cnt[4] = {0, 0, 0, 0};
        for (int k = 0; k < 4; ++k)
            for (int a = 0; a < 3; ++a) lo[a][k] = hi[a][k] = 1e30f;
        for (size_t k = 0; k < kids.size(); ++k) {
            const Node& c = nodes[kids[k]];
            for (int a = 0; a < 3; ++a) { lo[a][k] = c.box.lo[a]; hi[a][k] = c.box.hi[a]; }
            if (c.left < 0) { ref[k] = ~int32_t(c.first); cnt[k] = int32_t(c.count); }
            else ref[k] = emit(frontier(kids[k]));
        }
        float4* q = &out[size_t(idx) * 8];
        for (int a = 0; a < 3; ++a) {
            q[2 * a] = mk4(lo[a][0], lo[a][1], lo[a][2], lo[a][3]);
            q[2 * a + 1] = mk4(hi[a][0], hi[a][1], hi[a][2], hi[a][3]);
        }
        q[6] = mk4(i2f(ref[0]), i2f(ref[1]), i2f(ref[2]), i2f(ref[3]));
        q[7] = mk4(i2f(cnt[0]), i2f(cnt[1]), i2f(cnt[2]), i2f(cnt[3]));
        return idx;
    }
    // the up-to-four-node frontier below inner binary node b
    std::vector<uint32_t> frontier(uint32_t b) const {
        std::vector<uint32_t> kids{uint32_t(nodes[b].left), uint32_t(nodes[b].right)};
        while (kids.size() < 4) {
            int best = -1;
            float best_area = -1.0f;
            for (size_t k = 0; k < kids.size(); ++k) {
                if (nodes[kids[k]].left < 0) continue;
                const float ar = nodes[kids[k]].box.area();
                if (ar > best_area) { best_area = ar; best = int(k); }
            }
            if (best < 0) break;
            const uint32_t c = kids[best];
            kids[best] = uint32_t(nodes[c].left);
            kids.insert(kids.begin() + best + 1, uint32_t(nodes[c].right));
        }
        return kids;
    }
};

// A child's reference as the quantized nodes hold it: an inner node's index,
// or a leaf's first triangle and count (1 to 15) under the sign bit.
bool quant_ref(int32_t ref, int32_t count, uint32_t& out) {
    if (ref >= 0) { out = uint32_t(ref); return true; }
    const uint32_t first = uint32_t(~ref);
    if (first >= (1u << 27) || count < 0 || count > 15) return false;
    out = 0x80000000u | (first << 4) | uint32_t(count);
    return true;
}

// The most that grown boxes cost a ray anywhere in the tree. A ray that enters
// a node's box enters a child's with the probability of their areas' ratio, so
// the tests below a node add up from the leaves; to these come the nodes above
// it, which any ray that gets there has passed. Returned: the largest ratio, over
// all nodes, of that sum with the grown boxes to that with the tight ones. (A
// sum over the whole tree would not do: a small object on a wide ground has
// next to none of the area, and all of the rays once the camera looks at it.)
// areas: tight and grown area of both children of each node; depth-first, so a
// child's index is larger than its parent's.
double worst_cost_ratio(const std::vector<float4>& nodes, const std::vector<float4>& areas) {
    const size_t n = nodes.size() / 4;
    std::vector<float2> cost(n);      // tests below a node: tight, grown
    std::vector<float2> own(n);       // its own box's area
    std::vector<uint16_t> depth(n, 0);
    auto kids = [&](size_t g, int32_t* ref, int32_t* cnt) {
        std::memcpy(ref, &nodes[g * 4 + 3].x, 8);
        std::memcpy(cnt, &nodes[g * 4 + 3].z, 8);
    };
    for (size_t g = 0; g < n; ++g) {
        int32_t ref[2], cnt[2];
        kids(g, ref, cnt);
        const float4 a = areas[g];
        if (g == 0) own[0] = make_float2(std::max(a.x, a.z), std::max(a.y, a.w));
        for (int c = 0; c < 2; ++c)
            if (ref[c] >= 0) {
                depth[ref[c]] = uint16_t(depth[g] + 1);
                own[ref[c]] = c ? make_float2(a.z, a.w) : make_float2(a.x, a.y);
            }
    }
    double worst = 1.0;
    for (size_t g = n; g-- > 0;) {
        int32_t ref[2], cnt[2];
        kids(g, ref, cnt);
        const float4 a = areas[g];
        float2 sum = make_float2(1.0f, 1.0f);
        for (int c = 0; c < 2; ++c) {
            const float2 below = ref[c] >= 0 ? cost[ref[c]] : make_float2(float(cnt[c]), float(cnt[c]));
            const float t = c ? a.z : a.x, q = c ? a.w : a.y;
            sum.x += (own[g].x > t ? t / own[g].x : 1.0f) * below.x;
            sum.y += (own[g].y > q ? q / own[g].y : 1.0f) * below.y;
        }
        cost[g] = sum;
        worst = std::max(worst, (double(depth[g]) + sum.y) / (double(depth[g]) + sum.x));
    }
    return worst;
}

// f(first, end, chunk) over [0, n) in chunks of kChunk on the machine's threads; the
// chunks do not depend on how many there are. False as soon as a chunk says so.
constexpr size_t kChunk = 16384;
template <class F>
bool for_chunks(size_t n, F f) {
    const size_t chunks = (n + kChunk - 1) / kChunk;
    std::atomic<size_t> next{0};
    std::atomic<bool> ok{true};
    auto work = [&] {
        for (size_t c = next++; c < chunks && ok; c = next++)
            if (!f(c * kChunk, std::min(n, (c + 1) * kChunk), c)) ok = false;
    };
    const size_t threads = std::min<size_t>({chunks, std::thread::hardware_concurrency(), 16});
    std::vector<std::future<void>> others;
    for (size_t t = 1; t < threads; ++t) others.push_back(std::async(std::launch::async, work));
    work();
    for (auto& o : others) o.get();
    return ok;
}

// The quantized forms of both trees: every box plane goes outwards to a plane
// of a 15-bit grid over the scene's bounds, so a box only grows. Refused (the
// traversals then read the trees in full precision) where the boxes would
// grow by more than kQuantGrowth in surface area, summed over the tree (a
// few triangles far from all others stretch the grid), and where a leaf or a
// coordinate does not fit the format. Measured on the 1M-triangle room (960 x
// 540, 4 spp) with one mesh moved away, extension / shadow ms quantized
// against full precision (4.7 / 3.4): growth 1.003 2.6 / 1.6, 1.010 2.7 / 1.7,
// 1.036 3.4 / 2.1, 1.094 5.3 / 3.5, 1.2 10.0 / 7.3. The 10M-triangle instanced
// scenes grow by 1.006 and 1.008.
// Also refused where some part of the tree costs too much (worst_cost_ratio):
// the camera may look at just that. Path-traced 960 x 540 frames, 4 spp, both
// kinds of rays, full precision over quantized time: the room (1.17) 1.9; 4096
// instances in a box of 500 (1.56) 1.32, filled by its smallest instance 1.03
// to 1.06; a sphere of 20,000 triangles on a ground 30, 60, 100, 150 times its
// size (1.13, 1.25, 1.39, 1.85) 1.16, 1.10, 0.96, 0.92, and 3000 times 0.12; one
// of 320,000 on a ground of 10, 20, 30, 60, 1000 times (1.36, 1.62, 1.88, 2.4,
// 37) 1.25, 1.07, 1.02, 0.91, 0.085.
constexpr double kQuantGrowth = 1.06;
constexpr double kQuantWorst = 1.6;

bool quantize_trees(BvhBuild& out) {
    const size_t n = out.nodes.size() / 4, n4 = out.nodes4.size() / 8;
    if (n >= 0x7ffffff0u) return false;
    // lower and upper plane of one child on one axis
    auto planes = [&](size_t g, int child, int a, float& l, float& h) {
        const float4* q = &out.nodes[g * 4];
        const float4& xy = q[child];
        const float4& z = q[2];
        if (a == 0) { l = xy.x; h = xy.y; }
        else if (a == 1) { l = xy.z; h = xy.w; }
        else { l = child ? z.z : z.x; h = child ? z.w : z.y; }
    };
    double first[3], cell[3];   // plane 0 and the grid's step, as the kernels see them
    for (int a = 0; a < 3; ++a) {
        float l0, h0, l1, h1;
        planes(0, 0, a, l0, h0);
        planes(0, 1, a, l1, h1);
        const double lo = std::min(l0, l1), hi = std::max(h0, h1);
        const double big = std::max(std::fabs(lo), std::fabs(hi));
        if (!(big < 1e12)) return false;
        // no step finer than the coordinates' own spacing
        const double c = std::max((hi - lo) / 32760.0, std::max(big, 1e-12) * 1.2e-7);
        out.qscale[a] = std::nextafter(float(c * 256.0), INFINITY);
        cell[a] = double(out.qscale[a]) / 256.0;
        out.qbase[a] = float(lo - 2.0 * cell[a] - 128.0 * double(out.qscale[a]));
        first[a] = double(out.qbase[a]) + 128.0 * double(out.qscale[a]);
    }
    auto pack = [&](int a, float l, float h, uint32_t& w, double& extent) {
        const double ql = std::floor((double(l) - first[a]) / cell[a] - 1e-6);
        const double qh = std::ceil((double(h) - first[a]) / cell[a] + 1e-6);
        if (!(ql >= 0.0 && qh <= 32767.0 && ql <= qh)) return false;
        w = uint32_t(ql) | (uint32_t(qh) << 16);
        extent = (qh - ql) * cell[a];
        return true;
    };
    auto area = [](const double* e) { return e[0] * e[1] + e[1] * e[2] + e[2] * e[0]; };
    // One million triangles: 220 ms on one thread, 70 on eight, and 60 for
    // worst_cost_ratio. With the 4-wide layout beside the binary one a build
    // takes 1.65 s; 1.78 before there were quantized trees, 1.98 with the
    // quantization on one thread and one layout after the other.
    std::vector<double> full((n + kChunk - 1) / kChunk, 0.0), grown(full.size(), 0.0);
    std::vector<float4> areas(n);
    out.qnodes.resize(n * 2);
    const bool fits = for_chunks(n, [&](size_t first_node, size_t end, size_t chunk) {
      double f = 0.0, q = 0.0;
      for (size_t g = first_node; g < end; ++g) {
        const float4& d = out.nodes[g * 4 + 3];
        int32_t ref[2], cnt[2];
        std::memcpy(ref, &d.x, 8);
        std::memcpy(cnt, &d.z, 8);
        for (int c = 0; c < 2; ++c) {
            double e[3], eq[3];
            uint32_t w[3], r;
            for (int a = 0; a < 3; ++a) {
                float l, h;
                planes(g, c, a, l, h);
                if (!pack(a, l, h, w[a], eq[a])) return false;
                e[a] = double(h) - double(l);
            }
            const double tight = area(e), large = area(eq);
            f += tight;
            q += large;
            if (c == 0) { areas[g].x = float(tight); areas[g].y = float(large); }
            else { areas[g].z = float(tight); areas[g].w = float(large); }
            if (!quant_ref(ref[c], cnt[c], r)) return false;
            out.qnodes[g * 2 + c] = make_uint4(w[0], w[1], w[2], r);
        }
      }
      full[chunk] = f;
      grown[chunk] = q;
      return true;
    });
    if (!fits) return false;
    double sum_full = 0.0, sum_grown = 0.0;
    for (size_t c = 0; c < full.size(); ++c) {
        sum_full += full[c];
        sum_grown += grown[c];
    }
    if (!(sum_grown <= kQuantGrowth * sum_full)) return false;
    if (worst_cost_ratio(out.nodes, areas) > kQuantWorst) return false;
    out.qnodes4.resize(n4 * 4);
    return for_chunks(n4, [&](size_t first_node, size_t end, size_t) {
      for (size_t g = first_node; g < end; ++g) {
        const float* f = &out.nodes4[g * 8].x;
        for (int k = 0; k < 4; ++k) {
            uint32_t w[3], r;
            double extent;
            if (!(f[k] < 1e29f)) {   // an unused slot: lower plane above the upper one, an empty leaf
                out.qnodes4[g * 4 + k] = make_uint4(32767u, 32767u, 32767u, 0x80000000u);
                continue;
            }
            int32_t ref, cnt;
            std::memcpy(&ref, f + 24 + k, 4);
            std::memcpy(&cnt, f + 28 + k, 4);
            for (int a = 0; a < 3; ++a)
                if (!pack(a, f[a * 8 + k], f[a * 8 + 4 + k], w[a], extent)) return false;
            if (!quant_ref(ref, cnt, r)) return false;
            out.qnodes4[g * 4 + k] = make_uint4(w[0], w[1], w[2], r);
        }
      }
      return true;
    });
}

} // namespace

BvhBuild build_bvh(const std::vector<float>& tri_world, int /*threads*/) {
    const uint32_t n = uint32_t(tri_world.size() / 9);
    BvhBuild out;
    std::vector<Box> boxes(n);
    std::vector<float> cent(size_t(n) * 3);
    for (uint32_t i = 0; i < n; ++i) {
        Box b;
        b.grow(&tri_world[9 * size_t(i)]);
        b.grow(&tri_world[9 * size_t(i) + 3]);
        b.grow(&tri_world[9 * size_t(i) + 6]);
        boxes[i] = b;
        for (int a = 0; a < 3; ++a) cent[3 * size_t(i) + a] = 0.5f * (b.lo[a] + b.hi[a]);
    }
    out.order.resize(n);
    for (uint32_t i = 0; i < n; ++i) out.order[i] = i;
    std::vector<Node> nodes(std::max<size_t>(1, 2 * size_t(n)));
    Builder B{boxes, cent, out.order, nodes};
    if (n > 0) B.build(0, 0, n, 0);
    else nodes[0].box = Box();
    out.max_depth = B.depth_max.load() + 1;
    // the 4-wide layout, beside the binary one below (a small scene's after it)
    std::future<void> wide = std::async(n > 50000 ? std::launch::async : std::launch::deferred, [&] {
        Wide4 W{nodes, out.nodes4};
        if (n > 0 && nodes[0].left >= 0) W.emit(W.frontier(0));
        else if (n > 0) W.emit(std::vector<uint32_t>{0u});   // the root is a leaf
        else W.emit(std::vector<uint32_t>{});
    });

    // GPU layout: one GPU node per inner binary node, depth-first, left first.
    auto child_ref = [&](const Node& c, std::vector<int32_t>& gidx, int32_t ci, int32_t& ref, int32_t& cnt) {
        if (c.left < 0) { ref = ~int32_t(c.first); cnt = int32_t(c.count); }
        else { ref = gidx[ci]; cnt = 0; }
    };
    std::vector<int32_t> gidx(nodes.size(), -1);
    std::vector<uint32_t> dfs;
    if (nodes[0].left < 0) {
        // Root is a leaf: one GPU node with the leaf and an empty sibling.
        const Node& r = nodes[0];
        const Box& b = r.box;
        const float lo0 = n ? b.lo[0] : 0.f, hi0 = n ? b.hi[0] : 0.f;
        const float lo1 = n ? b.lo[1] : 0.f, hi1 = n ? b.hi[1] : 0.f;
        const float lo2 = n ? b.lo[2] : 0.f, hi2 = n ? b.hi[2] : 0.f;
        out.nodes.push_back(mk4(lo0, hi0, lo1, hi1));
        out.nodes.push_back(mk4(lo0, hi0, lo1, hi1));
        out.nodes.push_back(mk4(lo2, hi2, lo2, hi2));
        out.nodes.push_back(mk4(i2f(~int32_t(0)), i2f(~int32_t(0)), i2f(int32_t(r.count)), i2f(0)));
        wide.get();
        if (!quantize_trees(out)) { out.qnodes.clear(); out.qnodes4.clear(); }
        return out;
    }
    // iterative DFS to assign GPU indices
    std::vector<uint32_t> stack{0};
    while (!stack.empty()) {
        const uint32_t i = stack.back(); stack.pop_back();
        gidx[i] = int32_t(dfs.size());
        dfs.push_back(i);
        const Node& nd = nodes[i];
        if (nodes[nd.right].left >= 0) stack.push_back(uint32_t(nd.right));
        if (nodes[nd.left].left >= 0) stack.push_back(uint32_t(nd.left));
    }
    out.nodes.resize(dfs.size() * 4);
    for (size_t g = 0; g < dfs.size(); ++g) {
        const Node& nd = nodes[dfs[g]];
        const Node& c0 = nodes[nd.left];
        const Node& c1 = nodes[nd.right];
        int32_t r0, r1, k0, k1;
        child_ref(c0, gidx, nd.left, r0, k0);
        child_ref(c1, gidx, nd.right, r1, k1);
        out.nodes[g * 4 + 0] = mk4(c0.box.lo[0], c0.box.hi[0], c0.box.lo[1], c0.box.hi[1]);
        out.nodes[g * 4 + 1] = mk4(c1.box.lo[0], c1.box.hi[0], c1.box.lo[1], c1.box.hi[1]);
        out.nodes[g * 4 + 2] = mk4(c0.box.lo[2], c0.box.hi[2], c1.box.lo[2], c1.box.hi[2]);
        out.nodes[g * 4 + 3] = mk4(i2f(r0), i2f(r1), i2f(k0), i2f(k1));
    }
    wide.get();
    if (!quantize_trees(out)) { out.qnodes.clear(); out.qnodes4.clear(); }
    return out;
}

} // namespace rr
