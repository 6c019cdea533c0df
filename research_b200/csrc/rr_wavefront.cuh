// rr_wavefront.cuh — wavefront stages shared by the reference and the guided
// path tracers: ray generation, queue traversal (closest hit / any hit) with
// its schedule and occupancy variants, and queue allocation.
#pragma once

#include "rr_internal.h"

namespace rr {
namespace {

constexpr int kBlock = 256;
constexpr uint32_t kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// Slots in K output queues, for a block whose threads all take part: thread
// by thread in block order, from one atomic per queue and block. (Atomics on
// one address complete every 1.5 ns here: with one per warp the ray generation
// of a 1080p image at 4 samples took 382 us, 77 with its slots in closed
// form, and the five shade launches 2243, 1972 with one per block.)
// `turn` counts the block's calls: two tables alternate, so that a warp still
// reading one call's slots is not overtaken by the next call's counts.
template <int K>
struct AllocTable {
    uint32_t slot[2][K][kBlock / 32];
};
template <int K>
__device__ __forceinline__ void block_alloc(AllocTable<K>& table, uint32_t turn, const bool (&want)[K],
                                            uint32_t* const (&counter)[K], uint32_t (&slot)[K]) {
    static_assert(K <= kBlock / 32, "one warp per queue");
    uint32_t(&t)[K][kBlock / 32] = table.slot[turn & 1u];
    const uint32_t w = threadIdx.x >> 5, lane = lane_id();
    uint32_t mask[K];
    #pragma unroll
    for (int k = 0; k < K; ++k) {
        mask[k] = __ballot_sync(kFull, want[k]);
        if (lane == 0) t[k][w] = __popc(mask[k]);
    }
    __syncthreads();
    if (w < K) {
        // warp w: the block's warps' first slots in queue w
        const uint32_t n = lane < kBlock / 32 ? t[w][lane] : 0u;
        uint32_t end = n;
        #pragma unroll
        for (int o = 1; o < kBlock / 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, end, o);
            if (lane >= uint32_t(o)) end += v;
        }
        uint32_t base = 0;
        uint32_t* c = counter[0];
        #pragma unroll
        for (int k = 1; k < K; ++k) c = w == uint32_t(k) ? counter[k] : c;
        if (lane == kBlock / 32 - 1 && end) base = atomicAdd(c, end);
        base = __shfl_sync(kFull, base, kBlock / 32 - 1);
        if (lane < kBlock / 32) t[w][lane] = base + end - n;
    }
    __syncthreads();
    #pragma unroll
    for (int k = 0; k < K; ++k) slot[k] = t[k][w] + __popc(mask[k] & ((1u << lane) - 1u));
}

// The place of an 8 x 4 tile's pixels among those of a W x H image taken tile
// by tile (tiles at the right and bottom edges are cut).
__device__ __forceinline__ uint32_t tile_first(uint32_t tile, uint32_t tiles_x, uint32_t W, uint32_t H) {
    const uint32_t row = tile / tiles_x, col = tile % tiles_x;
    return row * 4u * W + col * 8u * min(4u, H - row * 4u);
}

struct PtLaunch {
    GpuCameraData cam;
    uint32_t frame_seed;
    uint32_t spp;
    uint32_t width, height;
    uint32_t tiles_x, tiles_per_image;
};

// One warp per 8x4 pixel tile so that primary rays of a warp are coherent.
__global__ void __launch_bounds__(kBlock) raygen_kernel(PtLaunch L, float4* __restrict__ out,
                                                        float4* qa, float4* qb, float4* qc,
                                                        uint32_t* counters) {
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t tile = gtid >> 5;
    const uint32_t lane = lane_id();
    const uint32_t total_tiles = L.tiles_per_image * L.spp;
    bool active = tile < total_tiles;
    uint32_t s = 0, px = 0, py = 0;
    if (active) {
        s = tile / L.tiles_per_image;
        const uint32_t t = tile % L.tiles_per_image;
        px = (t % L.tiles_x) * 8 + (lane & 7);
        py = (t / L.tiles_x) * 4 + (lane >> 3);
        active = px < L.width && py < L.height;
    }
    if (gtid == 0) counters[0] = L.width * L.height * L.spp;
    const uint32_t mask = __ballot_sync(kFull, active);
    if (!active) return;
    const uint32_t slot = s * L.width * L.height +
                          tile_first(tile % L.tiles_per_image, L.tiles_x, L.width, L.height) +
                          __popc(mask & ((1u << lane) - 1u));
    const uint32_t pid = (s * L.height + py) * L.width + px;
    uint32_t seed = make_seed(px, py, L.frame_seed + s);
    const float jx = rand_float(seed);
    const float jy = rand_float(seed);
    const float3 dir = primary_dir(L.cam, float(px) + jx, float(py) + jy);
    out[pid] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    qa[slot] = make_float4(L.cam.position[0], L.cam.position[1], L.cam.position[2], __uint_as_float(pid));
    qb[slot] = make_float4(dir.x, dir.y, dir.z, __uint_as_float(seed));
    qc[slot] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
}

// Adds per-thread traversal work to two 64-bit counters, one atomic per warp.
__device__ __forceinline__ void flush_work(const TraceWork& w, unsigned long long* out) {
    unsigned long long n = w.nodes, t = w.tris;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        n += __shfl_down_sync(kFull, n, o);
        t += __shfl_down_sync(kFull, t, o);
    }
    if (lane_id() == 0 && (n | t)) { atomicAdd(out, n); atomicAdd(out + 1, t); }
}

// Queue traversal. `load(i, o, d, tmax)` reads queue entry i and returns its
// scene index, `hit(i, u, v, instance, primitive)` takes a closest hit (and
// again every nearer one of the same ray), `done(i, found)` ends the entry.
// Multi: a batch of scenes, each ray traced in the scene `table[index]` (the
// lane binds that scene's arrays when it loads the ray); otherwise every ray
// is traced in `s`. Rays start at t = tmin (the path tracer's 0.001).
//
// Tree 4, 2: the quantized 4-wide / binary tree, a warp's lanes in step. Each
// turn of the loop the warp votes and does one of three things with all
// lanes that want it:
//   nodes: kNodeSteps node steps of every lane at an inner node;
//   leaves: the triangles of every lane waiting at a leaf, once more than
//     half as many lanes wait there as are at inner nodes (a lane's leaf run
//     on its own would idle the other 31 for some 100 instructions per
//     triangle: that took two thirds of the issue slots);
//   rays: idle lanes finish their rays and take the queue's next entries,
//     once at most `refill` are busy (neighbouring entries are neighbouring
//     paths after compaction, so rays stay alike). That is kBusyLanes, but 0
//     for camera rays: a warp's 32 cross the same nodes as long as all are
//     from one tile (1.92 ms for the 1080p frame's 8.3 M; refilled at 8, 16,
//     24 busy lanes 2.06 / 2.33 / 2.35. The first bounce's rays take 3.91 /
//     3.45 / 3.34 / 3.19, and shadow rays 2.91 / 2.50 / 2.18 / 2.07).
// Measured on the 1080p 4 spp frame of the 1M-triangle room, extension /
// shadow rays: one thread per ray 16.6 / 11.8 ms; this loop on the
// full-precision tree, leaf vote 1/4, 1/2, 1: 14.4 / 14.2 / 14.4 and 10.1 /
// 9.8 / 10.0 ms; with refill at 8, 16, 24 busy lanes 13.8 / 13.7 / 13.4 and
// 8.8 / 8.1 / 7.8 ms; on the quantized binary tree 12.5 / 6.9 ms; leaves as
// references and one, two, three node steps a vote 11.5 / 10.8 / 10.5 and
// 6.4 / 6.1 / 5.8 ms; 4-wide, two steps, stack in shared memory 9.3 / 5.2 ms;
// camera rays without refill 8.9 ms; with every hit tested against its
// triangle's own box (in_own_box) 9.4 / 5.3 ms.
//
// Tree 0: the binary tree in full precision, one thread per ray (scenes that
// the grid does not serve).
//
// SmemS > 0: the bottom SmemS stack entries of every thread in shared memory.
template <int SmemS, int N, class E> struct QueueStackOf { using type = SplitStack<SmemS, kBlock, N, E>; };
template <int N, class E> struct QueueStackOf<0, N, E> { using type = LocalStackN<N, E>; };

constexpr int kNodeSteps = 2;
constexpr uint32_t kBusyLanes = 24;
constexpr uint32_t kDoubtList = 64, kDoubtStop = 32;   // a warp's list of doubtful rays (traverse_queue)
static_assert(kDoubtStop - 1 + 32 <= kDoubtList, "the list holds a warp's rays on top of those it stops at");

template <bool AnyHit, bool Count, bool Multi, int Tree, int SmemS, class Load, class Hit, class Done>
__device__ __forceinline__ void traverse_queue(const DevScene& s, const DevScene* __restrict__ table, uint32_t count,
                                               uint32_t* cursor, unsigned long long* work_out, Load load, Hit hit,
                                               Done done, uint32_t refill, float tmin = 0.001f) {
    TraceWork tw;
    // an any-hit ray's bound never moves: its entries need no distance
    using Entry = typename StackEntryOf<Tree == 0 || !AnyHit>::type;
    typename QueueStackOf<SmemS, Tree == 4 ? kStackSize4 : kStackSize, Entry>::type stack;
    if constexpr (SmemS > 0) {
        __shared__ Entry stack_smem[SmemS * kBlock];
        stack.col = stack_smem + threadIdx.x;
    }
    if constexpr (Tree == 0) {
        DevScene ls{};
        while (true) {
            uint32_t base = 0;
            if (lane_id() == 0) base = atomicAdd(cursor, 32u);
            base = __shfl_sync(kFull, base, 0);
            if (base >= count) break;
            const uint32_t i = base + lane_id();
            if (i < count) {
                float3 o, d;
                float tmax;
                const uint32_t sid = load(i, o, d, tmax);
                if constexpr (Multi) {
                    ls.nodes = table[sid].nodes;
                    ls.tris = table[sid].tris;
                    ls.num_nodes = table[sid].num_nodes;
                }
                const Ray r = make_ray(o, d);
                HitRec h; TravState st;
                trav_begin(st, h, tmax);
                while (!trace_step<AnyHit, Count>(Multi ? ls : s, r, tmin, h, st, stack, &tw)) {}
                if (!AnyHit && st.found) hit(i, h.u, h.v, __uint_as_float(h.inst), __uint_as_float(h.prim));
                done(i, st.found);
            }
        }
    } else {
        const uint4* nodes = Tree == 4 ? s.qnodes4 : s.qnodes;
        const float4* tris = s.tris;
        float3 qinv = s.qinv;
        QuantRay r;
        LaneTrav st;
        st.cur = kFree;
        uint32_t i = 0;
        bool more = true;   // the queue may hold entries not taken yet
        // Doubtful rays (in_own_box), traced in the full tree at the end; a
        // warp that holds kDoubtStop of them leaves its share of the queue to
        // the loop there. Rays are taken only while fewer are listed, the
        // turn's own included, so each of the 32 lanes' rays still has a place
        // if all of them turn out doubtful.
        __shared__ uint32_t doubt_smem[kBlock / 32][kDoubtList];
        uint32_t* const doubt = doubt_smem[threadIdx.x >> 5];
        uint32_t doubts = 0;
        while (true) {
            const uint32_t leafm = __ballot_sync(kFull, st.cur < 0);
            const uint32_t nodem = __ballot_sync(kFull, st.stepping());
            bool take = more && doubts < kDoubtStop;
            if ((leafm | nodem) == 0 || (take && uint32_t(__popc(leafm | nodem)) <= refill)) {
                const bool idle = st.cur >= kDone;
                bool doubtful = false;
                if (st.cur == kDone) {
                    if (st.tri != kNoIndex)
                        doubtful = !in_own_box(tris, st.tri, r, qinv, tmin, AnyHit ? st.t : st.tl);
                    if (!doubtful) done(i, st.tri != kNoIndex);
                    st.cur = kFree;
                }
                const uint32_t m = __ballot_sync(kFull, doubtful);
                if (doubtful) doubt[doubts + __popc(m & ((1u << lane_id()) - 1u))] = i;
                doubts += __popc(m);
                take = more && doubts < kDoubtStop;
                if (!take) {
                    if ((leafm | nodem) == 0) break;
                    continue;   // the busy lanes go on
                }
                const uint32_t idlem = __ballot_sync(kFull, idle);
                uint32_t base = 0;
                if (lane_id() == 0) base = atomicAdd(cursor, __popc(idlem));
                base = __shfl_sync(kFull, base, 0);
                more = base + __popc(idlem) < count;
                if (idle) {
                    i = base + __popc(idlem & ((1u << lane_id()) - 1u));
                    if (i < count) {
                        float3 o, d;
                        float tmax;
                        const uint32_t sid = load(i, o, d, tmax);
                        if constexpr (Multi) {
                            nodes = Tree == 4 ? table[sid].qnodes4 : table[sid].qnodes;
                            tris = table[sid].tris;
                            qinv = table[sid].qinv;
                            r = make_quant_ray(table[sid], o, d);
                        } else {
                            r = make_quant_ray(s, o, d);
                        }
                        lane_begin(st, stack, tmax);
                    }
                }
                continue;
            }
            if (nodem == 0 || __popc(leafm) * 2 > __popc(nodem)) {
                if (st.cur < 0)
                    quant_leaf<AnyHit, Count>(tris, r, tmin, st, &tw, [&](float u, float v, float inst, float prim) {
                        hit(i, u, v, inst, prim);
                    });
            } else {
                #pragma unroll
                for (int k = 0; k < kNodeSteps; ++k)
                    if (st.stepping()) {
                        if constexpr (Tree == 4) quant_step4<AnyHit, Count>(nodes, r, tmin, st, stack, &tw);
                        else quant_step2<AnyHit, Count>(nodes, r, tmin, st, stack, &tw);
                    }
            }
        }
        auto trace_one = [&](uint32_t e) {
            float3 o, d;
            float tmax;
            const uint32_t sid = load(e, o, d, tmax);
            const DevScene& es = Multi ? table[sid] : s;
            HitRec h;
            const bool found = trace<AnyHit, Count>(es, make_ray(o, d), tmin, tmax, h, &tw);
            if (!AnyHit && found) hit(e, h.u, h.v, __uint_as_float(h.inst), __uint_as_float(h.prim));
            done(e, found);
        };
        __syncwarp();
        for (uint32_t k = lane_id(); k < doubts; k += 32u) trace_one(doubt[k]);
        while (more) {
            uint32_t base = 0;
            if (lane_id() == 0) base = atomicAdd(cursor, 32u);
            base = __shfl_sync(kFull, base, 0);
            more = base < count;
            if (base + lane_id() < count) trace_one(base + lane_id());
        }
    }
    if (Count) flush_work(tw, work_out);
}

// Closest hits of the ray queue (a, b) into `hits`: (u, v, instance,
// primitive), all ones for a miss.
struct StoreHit {
    float4* hits;
    __device__ __forceinline__ void operator()(uint32_t i, float u, float v, float inst, float prim) const {
        hits[i] = make_float4(u, v, inst, prim);
    }
};
struct StoreMiss {
    float4* hits;
    __device__ __forceinline__ void operator()(uint32_t i, bool found) const {
        if (!found) hits[i] = make_float4(0.0f, 0.0f, __uint_as_float(kNoIndex), __uint_as_float(kNoIndex));
    }
};
struct NoHit {
    __device__ __forceinline__ void operator()(uint32_t, float, float, float, float) const {}
};

template <bool Count, int MinBlocks, int Tree, int SmemS>
__global__ void __launch_bounds__(kBlock, MinBlocks) extend_kernel(DevScene s, const float4* __restrict__ qa,
                                                                   const float4* __restrict__ qb,
                                                                   float4* __restrict__ hits,
                                                                   const uint32_t* count_ptr, uint32_t* cursor,
                                                                   unsigned long long* work_out, uint32_t refill) {
    traverse_queue<false, Count, false, Tree, SmemS>(
        s, nullptr, *count_ptr, cursor, work_out,
        [&](uint32_t i, float3& o, float3& d, float& tmax) -> uint32_t {
            o = xyz(qa[i]);
            d = xyz(qb[i]);
            tmax = 1e9f;
            return 0u;
        },
        StoreHit{hits}, StoreMiss{hits}, refill);
}

// Any-hit shadow rays; unoccluded NEE contributions are added to the image.
template <bool Count, int MinBlocks, int Tree, int SmemS>
__global__ void __launch_bounds__(kBlock, MinBlocks) shadow_kernel(DevScene s, const float4* __restrict__ sa,
                                                                   const float4* __restrict__ sb,
                                                                   const float4* __restrict__ sc,
                                                                   float4* __restrict__ out,
                                                                   const uint32_t* count_ptr, uint32_t* cursor,
                                                                   unsigned long long* work_out) {
    traverse_queue<true, Count, false, Tree, SmemS>(
        s, nullptr, *count_ptr, cursor, work_out,
        [&](uint32_t i, float3& o, float3& d, float& tmax) -> uint32_t {
            const float4 b = sb[i];
            o = xyz(sa[i]);
            d = xyz(b);
            tmax = b.w;
            return 0u;
        },
        NoHit{},
        [&](uint32_t i, bool found) {
            if (!found) {
                const float4 c = sc[i];
                const uint32_t pid = __float_as_uint(sa[i].w);
                float4 o = out[pid];
                o.x = o.x + c.x; o.y = o.y + c.y; o.z = o.z + c.z;
                out[pid] = o;
            }
        },
        kBusyLanes);
}

// ── batches of scenes (no reference counterpart: the reference renders one
// scene per pass execute). Queue entries carry their scene index in the
// .w of the throughput (rays) and contribution (shadow rays) records.
struct BatchEntry {
    PtLaunch L;            // the scene's camera, frame seed, spp and image size
    uint32_t tile_begin;   // first raygen tile of the scene in the batch
    uint32_t path_begin;   // first path
    uint32_t _pad[2];
};

// raygen_kernel over all scenes of a batch: the global tile index picks the
// scene (binary search over tile_begin), the rest is raygen_kernel's.
__global__ void __launch_bounds__(kBlock) raygen_batch_kernel(const BatchEntry* __restrict__ E, uint32_t n_scenes,
                                                              uint32_t total_tiles, uint32_t total_paths,
                                                              float4* const* __restrict__ outs,
                                                              float4* qa, float4* qb, float4* qc,
                                                              uint32_t* counters) {
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t tile = gtid >> 5;
    const uint32_t lane = lane_id();
    bool active = tile < total_tiles;
    uint32_t sid = 0, s = 0, px = 0, py = 0;
    if (active) {
        uint32_t lo = 0, hi = n_scenes - 1;
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (E[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
        }
        sid = lo;
        const PtLaunch& L = E[sid].L;
        const uint32_t local = tile - E[sid].tile_begin;
        s = local / L.tiles_per_image;
        const uint32_t t = local % L.tiles_per_image;
        px = (t % L.tiles_x) * 8 + (lane & 7);
        py = (t / L.tiles_x) * 4 + (lane >> 3);
        active = s < L.spp && px < L.width && py < L.height;
    }
    if (gtid == 0) counters[0] = total_paths;
    const uint32_t mask = __ballot_sync(kFull, active);
    if (!active) return;
    const PtLaunch& L = E[sid].L;
    const uint32_t slot = E[sid].path_begin + s * L.width * L.height +
                          tile_first((tile - E[sid].tile_begin) % L.tiles_per_image, L.tiles_x, L.width, L.height) +
                          __popc(mask & ((1u << lane) - 1u));
    const uint32_t pid = (s * L.height + py) * L.width + px;
    uint32_t seed = make_seed(px, py, L.frame_seed + s);
    const float jx = rand_float(seed);
    const float jy = rand_float(seed);
    const float3 dir = primary_dir(L.cam, float(px) + jx, float(py) + jy);
    outs[sid][pid] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    qa[slot] = make_float4(L.cam.position[0], L.cam.position[1], L.cam.position[2], __uint_as_float(pid));
    qb[slot] = make_float4(dir.x, dir.y, dir.z, __uint_as_float(seed));
    qc[slot] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(sid));
}

template <bool Count, int MinBlocks, int Tree, int SmemS>
__global__ void __launch_bounds__(kBlock, MinBlocks) extend_batch_kernel(const DevScene* __restrict__ table,
                                                                         const float4* __restrict__ qa,
                                                                         const float4* __restrict__ qb,
                                                                         const float4* __restrict__ qc,
                                                                         float4* __restrict__ hits,
                                                                         const uint32_t* count_ptr, uint32_t* cursor,
                                                                         unsigned long long* work_out,
                                                                         uint32_t refill) {
    const DevScene none{};
    traverse_queue<false, Count, true, Tree, SmemS>(
        none, table, *count_ptr, cursor, work_out,
        [&](uint32_t i, float3& o, float3& d, float& tmax) -> uint32_t {
            o = xyz(qa[i]);
            d = xyz(qb[i]);
            tmax = 1e9f;
            return __float_as_uint(qc[i].w);
        },
        StoreHit{hits}, StoreMiss{hits}, refill);
}

template <bool Count, int MinBlocks, int Tree, int SmemS>
__global__ void __launch_bounds__(kBlock, MinBlocks) shadow_batch_kernel(const DevScene* __restrict__ table,
                                                                         float4* const* __restrict__ outs,
                                                                         const float4* __restrict__ sa,
                                                                         const float4* __restrict__ sb,
                                                                         const float4* __restrict__ sc,
                                                                         const uint32_t* count_ptr, uint32_t* cursor,
                                                                         unsigned long long* work_out) {
    const DevScene none{};
    traverse_queue<true, Count, true, Tree, SmemS>(
        none, table, *count_ptr, cursor, work_out,
        [&](uint32_t i, float3& o, float3& d, float& tmax) -> uint32_t {
            const float4 b = sb[i];
            o = xyz(sa[i]);
            d = xyz(b);
            tmax = b.w;
            return __float_as_uint(sc[i].w);
        },
        NoHit{},
        [&](uint32_t i, bool found) {
            if (!found) {
                const float4 c = sc[i];
                const uint32_t pid = __float_as_uint(sa[i].w);
                float4* out = outs[__float_as_uint(c.w)];
                float4 o = out[pid];
                o.x = o.x + c.x; o.y = o.y + c.y; o.z = o.z + c.z;
                out[pid] = o;
            }
        },
        kBusyLanes);
}

using BatchQueueKernel = void (*)(const DevScene*, const float4*, const float4*, const float4*, float4*,
                                  const uint32_t*, uint32_t*, unsigned long long*, uint32_t);
using BatchShadowKernel = void (*)(const DevScene*, float4* const*, const float4*, const float4*, const float4*,
                                   const uint32_t*, uint32_t*, unsigned long long*);
// Traversal kernel variants (rr_pathtracer_set_variants): MinBlocks x tree x
// stack entries in shared memory. A scene whose trees are not quantized is
// traced by kVariantFull's kernel whatever the variant. RR_PT_VARIANT_DEFAULT
// (4) is the fastest on the 1M-triangle room (extension / shadow rays of the 1080p
// frame 9.4 / 5.3 ms; 9.7 / 5.4 with the whole stack in local memory,
// binary tree 10.4 / 6.0). kVariantFull's form differs for the two kinds of
// rays: on the same room with one mesh 1e7 away (not quantized) 16.2 / 11.0 ms
// with 4 blocks per SM and 8 stack entries in shared memory for extension
// rays, 5 blocks and a local stack for shadow rays; 16.6 / 11.8 with 4 blocks
// and a local stack for both.
constexpr int kVariantFull = 7;
#define RR_TRAVERSAL_VARIANTS(kernel, v, full_blocks, full_smem) \
    switch (v) {                                           \
    case 0: return kernel<Count, 4, 2, 8>;                 \
    case 1: return kernel<Count, 5, 2, 0>;                 \
    case 2: return kernel<Count, 4, 2, 0>;                 \
    case 3: return kernel<Count, 4, 4, 0>;                 \
    case 5: return kernel<Count, 5, 2, 12>;                \
    case 6: return kernel<Count, 5, 4, 8>;                 \
    case kVariantFull: return kernel<Count, full_blocks, 0, full_smem>; \
    default: return kernel<Count, 4, 4, 12>;               \
    }

template <bool Count>
BatchQueueKernel extend_batch_variant(int v) { RR_TRAVERSAL_VARIANTS(extend_batch_kernel, v, 4, 8) }
template <bool Count>
BatchShadowKernel shadow_batch_variant(int v) { RR_TRAVERSAL_VARIANTS(shadow_batch_kernel, v, 5, 0) }

using QueueKernel = void (*)(DevScene, const float4*, const float4*, float4*, const uint32_t*, uint32_t*,
                             unsigned long long*, uint32_t);
using ShadowKernel = void (*)(DevScene, const float4*, const float4*, const float4*, float4*, const uint32_t*,
                              uint32_t*, unsigned long long*);
template <bool Count>
QueueKernel extend_variant(int v) { RR_TRAVERSAL_VARIANTS(extend_kernel, v, 4, 8) }
template <bool Count>
ShadowKernel shadow_variant(int v) { RR_TRAVERSAL_VARIANTS(shadow_kernel, v, 5, 0) }

// When a bounce's extension rays are refilled (traverse_queue).
uint32_t refill_of(uint32_t bounce) { return bounce == 0 ? 0u : kBusyLanes; }

// The variant a scene's rays run: the asked one, or the full-precision form.
int variant_for(const DevScene& s, int v) { return s.qnodes4 ? v : kVariantFull; }

int persistent_grid(const rr_ctx* ctx, const void* kernel) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, 0);
    return ctx->sm_count * (per_sm > 0 ? per_sm : 1);
}

// The second stream and the fork/join events of the shadow overlap.
rr_status ensure_side(rr_ctx* ctx) {
    if (ctx->side) return RR_OK;
    for (int b = 0; b < kMaxBounces; ++b) {
        RR_TRY_CUDA(ctx, cudaEventCreateWithFlags(&ctx->shaded[b], cudaEventDisableTiming));
        RR_TRY_CUDA(ctx, cudaEventCreateWithFlags(&ctx->shadowed[b], cudaEventDisableTiming));
    }
    RR_TRY_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->side, cudaStreamNonBlocking));
    return RR_OK;
}

rr_status ensure_queues(rr_ctx* ctx, size_t n) {
    rr_pt_queues& q = ctx->pt;
    if (ctx->queue_limit && n > ctx->queue_limit)
        return rr_fail(ctx, RR_ERR_QUEUE_OVERFLOW,
                       "the call needs %zu ray-queue entries; the context's queue limit is %zu "
                       "(rr_ctx_set_queue_limit)", n, ctx->queue_limit);
    if (q.capacity >= n) return RR_OK;
    for (int i = 0; i < 2; ++i) { cudaFree(q.ray_a[i]); cudaFree(q.ray_b[i]); cudaFree(q.ray_c[i]); }
    cudaFree(q.hits); cudaFree(q.shadow_a); cudaFree(q.shadow_b); cudaFree(q.shadow_c);
    q = rr_pt_queues();
    const size_t bytes = n * sizeof(float4);
    for (int i = 0; i < 2; ++i) {
        RR_TRY_CUDA(ctx, cudaMalloc(&q.ray_a[i], bytes));
        RR_TRY_CUDA(ctx, cudaMalloc(&q.ray_b[i], bytes));
        RR_TRY_CUDA(ctx, cudaMalloc(&q.ray_c[i], bytes));
    }
    RR_TRY_CUDA(ctx, cudaMalloc(&q.hits, bytes));
    RR_TRY_CUDA(ctx, cudaMalloc(&q.shadow_a, bytes));
    RR_TRY_CUDA(ctx, cudaMalloc(&q.shadow_b, bytes));
    RR_TRY_CUDA(ctx, cudaMalloc(&q.shadow_c, bytes));
    q.capacity = n;
    return RR_OK;
}

} // namespace
} // namespace rr
