// atrous.cu — edge-aware A-trous wavelet filter (AtrousPass.cpp:243-306,
// kernel atrous.slang:41-106): 5x5 B3 taps (1,4,6,4,1)/16 per axis at
// stride 1<<iter, clamped to the image, skipping G-buffer misses, weighted by
// exp(-|dp|^2/sp^2) * exp(-max(0, 1-n.n')/sn^2) * exp(-dl^2/sl^2).

#include "rr_internal.h"
#include "rr_atrous.cuh"
#include "rr_tc.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

namespace rr {
namespace {

// The G-buffer normals normalized once per call (the filter reads each
// pixel's normal for up to 25 taps per iteration; normalize is deterministic,
// so the taps see the same values as normalizing on the spot).
__global__ void __launch_bounds__(256) normalize_kernel(const float4* __restrict__ gnrm, float4* __restrict__ out,
                                                        size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 v = normalize(xyz(gnrm[i]));
    out[i] = make_float4(v.x, v.y, v.z, 0.0f);
}

// Direct-load filter, one iteration in two launches, for the strides whose
// lattice does not fill the tiles below. A pixel's tap on a
// neighbour has the same weight as the neighbour's opposite tap on the pixel
// (tap_weight), so the 24 neighbour weights of every pixel need only 12
// evaluations, each with three divisions and three exponentials:
//   atrous_pair_weights_kernel: for every pixel, the weights of its 12
//     forward taps (kPairFwd: (1,0), (2,0), then ty = 1, 2 with tx = -2..2),
//     on the clamped neighbour, -1 where either pixel is a G-buffer miss,
//     into 12 planes of W x H floats;
//   atrous_pair_sum_kernel: every pixel's 25 taps in atrous_pixel's order;
//     a forward tap reads its own weight, a backward tap whose neighbour is
//     in the image reads the neighbour's forward weight, and the centre and
//     backward taps clamped at the border are evaluated on the spot.
// The sums see the same weights in the same order as atrous_pixel: the
// same bits. `nrm`: unit normals (from normalize_kernel).
constexpr int kPairFwd = 12;
RR_D int2 pair_offset(int j) { return j < 2 ? make_int2(j + 1, 0) : make_int2((j - 2) % 5 - 2, (j - 2) / 5 + 1); }
RR_D bool pair_forward(int tx, int ty) { return ty > 0 || (ty == 0 && tx > 0); }
RR_D int pair_index(int tx, int ty) { return ty == 0 ? tx - 1 : 2 + (ty - 1) * 5 + (tx + 2); }

__global__ void __launch_bounds__(128) atrous_pair_weights_kernel(const float4* __restrict__ in,
                                                                  const float4* __restrict__ gpos,
                                                                  const float4* __restrict__ nrm,
                                                                  float* __restrict__ wt, int W, int H, int stride,
                                                                  float sp2, float sn2, float sl2) {
    const int x = blockIdx.x * 16 + (threadIdx.x & 15);
    const int y = blockIdx.y * 8 + (threadIdx.x >> 4);
    if (x >= W || y >= H) return;
    const size_t plane = size_t(W) * H;
    const size_t i = size_t(y) * W + x;
    const float4 cpos = __ldg(gpos + i);
    if (cpos.w < 0.0f) {
        #pragma unroll
        for (int j = 0; j < kPairFwd; ++j) wt[j * plane + i] = -1.0f;
        return;
    }
    const float3 cn = xyz(__ldg(nrm + i));
    const float cl = luminance601(xyz(__ldg(in + i)));
    #pragma unroll
    for (int j = 0; j < kPairFwd; ++j) {
        const int2 o = pair_offset(j);
        const int sx = min(max(x + o.x * stride, 0), W - 1);
        const int sy = min(max(y + o.y * stride, 0), H - 1);
        const size_t k = size_t(sy) * W + sx;
        // the neighbour's three values are loaded whether or not it is a miss
        // (the address is in the image), so the loads of all taps can be in
        // flight together
        const float4 spos = __ldg(gpos + k);
        const float3 sn = xyz(__ldg(nrm + k));
        const float3 srad = xyz(__ldg(in + k));
        const float w = tap_weight(o.x, o.y, xyz(cpos), cn, cl, xyz(spos), sn, srad, sp2, sn2, sl2);
        wt[j * plane + i] = spos.w < 0.0f ? -1.0f : w;
    }
}

__global__ void __launch_bounds__(128) atrous_pair_sum_kernel(const float4* __restrict__ in,
                                                              const float4* __restrict__ gpos,
                                                              const float4* __restrict__ nrm,
                                                              const float* __restrict__ wt,
                                                              float4* __restrict__ out, int W, int H, int stride,
                                                              float sp2, float sn2, float sl2) {
    const int x = blockIdx.x * 16 + (threadIdx.x & 15);
    const int y = blockIdx.y * 8 + (threadIdx.x >> 4);
    if (x >= W || y >= H) return;
    const size_t plane = size_t(W) * H;
    const size_t i = size_t(y) * W + x;
    const float4 cpos = __ldg(gpos + i);
    const float4 crad = __ldg(in + i);
    if (cpos.w < 0.0f) {
        out[i] = crad;
        return;
    }
    const float3 cn = xyz(__ldg(nrm + i));
    const float cl = luminance601(xyz(crad));
    float3 filtered = f3(0.0f, 0.0f, 0.0f);
    float wsum = 0.0f;
    #pragma unroll
    for (int ty = -2; ty <= 2; ++ty) {
        const int uy = y + ty * stride;
        const int sy = min(max(uy, 0), H - 1);
        #pragma unroll
        for (int tx = -2; tx <= 2; ++tx) {
            const int ux = x + tx * stride;
            const int sx = min(max(ux, 0), W - 1);
            const size_t k = size_t(sy) * W + sx;
            float w;
            if (tx == 0 && ty == 0) {
                w = tap_weight(0, 0, xyz(cpos), cn, cl, xyz(cpos), cn, xyz(crad), sp2, sn2, sl2);
            } else if (pair_forward(tx, ty)) {
                w = __ldg(wt + pair_index(tx, ty) * plane + i);
            } else if (ux == sx && uy == sy) {
                w = __ldg(wt + pair_index(-tx, -ty) * plane + k);
            } else {
                const float4 spos = __ldg(gpos + k);
                w = spos.w < 0.0f ? -1.0f
                                  : tap_weight(tx, ty, xyz(cpos), cn, cl, xyz(spos), xyz(__ldg(nrm + k)),
                                               xyz(__ldg(in + k)), sp2, sn2, sl2);
            }
            // loaded before the weight is known (the address is in the image)
            const float3 srad = xyz(__ldg(in + k));
            if (!(w < 0.0f)) {   // w < 0: a G-buffer miss
                filtered = filtered + srad * w;
                wsum += w;
            }
        }
    }
    const float3 o = wsum > 0.0f ? filtered / wsum : xyz(crad);
    out[i] = make_float4(o.x, o.y, o.z, crad.w);
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(tc::smem_addr(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2),
          "r"(tc::smem_addr(bar))
        : "memory");
}

// The filter over one tile of a stride's lattice. At stride s the pixels with
// the same (x mod s, y mod s) are filtered among themselves, so a block takes
// 32 x 16 of them with a halo of 2 on every side, whatever the stride: every
// tap, clamped to the image, is in its tile (a halo element stands for the
// clamped coordinate). A pixel's tap on a neighbour has the same weight, bit
// for bit, as the neighbour's opposite tap on the pixel (tap_weight), so the
// block evaluates 12 forward weights per pixel and those of the halo that
// point into the tile (13 % more) into shared memory, two at a time in
// packed FP32, and then sums every pixel's 25 taps in atrous_pixel's order.
//
// What bounds it: the FP32 lanes that run packed instructions and issue (64 %
// active at stride 1), with two blocks of 512 threads per SM. 1080p, one
// iteration: 146 us at stride 1, 149 at 4, 177 at 8 and 191 at 16 (16-byte
// loads a stride apart use half of each sector); the TMA-tiled kernel that
// evaluated all 24 weights took 381 to 389, the pair kernels below 330.
constexpr int kTileW = 32, kTileH = 16, kTileThreads = kTileW * kTileH;
constexpr int kHaloW = kTileW + 4, kHaloH = kTileH + 4;      // elements of a tile with its halo
constexpr int kTileElems = kHaloW * kHaloH;
constexpr int kWtRows = kTileH + 2, kWtElems = kHaloW * kWtRows;   // elements that own forward weights
constexpr uint32_t kTileBoxBytes = uint32_t(kTileElems * 16);      // one image's box of a TMA-staged tile

struct TileSmem {
    float4 rad[kTileElems];        // (r, g, b, 1); all zero for a G-buffer miss
    float p[7][kTileElems];        // position, unit normal, luminance
    float wt[kPairFwd][kWtElems];
};
constexpr uint32_t kTileSmem = sizeof(TileSmem);
// staged: behind the tile, from a multiple of 128 bytes on, the three boxes
// as they are copied, and an mbarrier
constexpr uint32_t kTileSmemTma = kTileSmem + 3 * kTileBoxBytes + 128;

RR_D float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
RR_D float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// -a / b for a >= 0 and b's negated reciprocal ny = RN(-1 / b), both halves
// rounded correctly: a first quotient, one correction that makes it faithful
// and one more that makes it the nearest (Markstein, IBM J. R&D 1990: with
// the reciprocal correctly rounded and the quotient within an ulp,
// RN(q + (a - b q) y) is RN(a / b)). Holds while nothing under- or
// overflows: a is clamped below 100 b by the caller, b is within
// [1e-6, 1e12], and quotients below 2^-60, where a residual may underflow,
// have exponential 1 either way. Outside: IEEE divisions, clamped where the
// exponential is zero anyway.
RR_D u64 neg_div2(u64 a, u64 b, u64 ny) {
    const u64 q0 = mul2(a, ny);
    const u64 q1 = fma2(fma2(b, q0, a), ny, q0);
    return fma2(fma2(b, q1, a), ny, q1);
}
template <bool FastDiv>
RR_D u64 neg_quotient(u64 a, u64 b, u64 ny) {
    if constexpr (FastDiv) return neg_div2(a, b, ny);
    else return pack2(max_nan(-lo2(a) / lo2(b), -200.0f), max_nan(-hi2(a) / hi2(b), -200.0f));
}

RR_D u64 both(float v) { return pack2(v, v); }

// rr_expf of two non-positive arguments (or NaN): the same operations. The
// rounding to an integer adds and takes away 1.5 2^23 (exact for |x| < 2^22),
// which leaves the integer in the sum's low bits.
RR_D u64 exp2_nonpos(u64 x) {
    const u64 s = add2(mul2(x, both(0x1.715476p+0f)), both(12582912.0f));
    const u64 k = add2(s, both(-12582912.0f));
    u64 r = fma2(k, both(-0x1.62e430p-1f), x);
    r = fma2(k, both(0x1.05c610p-29f), r);
    u64 p = both(0x1.a01a02p-16f);
    p = fma2(p, r, both(0x1.a01a02p-13f));
    p = fma2(p, r, both(0x1.6c16c2p-10f));
    p = fma2(p, r, both(0x1.111112p-7f));
    p = fma2(p, r, both(0x1.555556p-5f));
    p = fma2(p, r, both(0x1.555556p-3f));
    p = fma2(p, r, both(0.5f));
    p = fma2(p, r, both(1.0f));
    p = fma2(p, r, both(1.0f));
    auto scale = [](uint32_t bits, float v) {
        return v < -87.33654f ? 0.0f : __uint_as_float((bits << 23) + 0x3f800000u);
    };
    return mul2(p, pack2(scale(uint32_t(s), lo2(x)), scale(uint32_t(s >> 32), hi2(x))));
}

// The same for one value, as scalar instructions: packed ones run on half of
// the FP32 lanes at two values each, scalar ones also on the other half, so
// a weight's three factors are two packed and one scalar.
template <bool FastDiv>
RR_D float neg_quotient1(float a, float b, float ny) {
    if constexpr (FastDiv) {
        const float q0 = a * ny;
        const float q1 = __fmaf_rn(__fmaf_rn(b, q0, a), ny, q0);
        return __fmaf_rn(__fmaf_rn(b, q1, a), ny, q1);
    } else {
        return max_nan(-a / b, -200.0f);
    }
}
RR_D float exp1_nonpos(float x) {
    const float s = x * 0x1.715476p+0f + 12582912.0f;
    const float k = s - 12582912.0f;
    float r = __fmaf_rn(k, -0x1.62e430p-1f, x);
    r = __fmaf_rn(k, 0x1.05c610p-29f, r);
    float p = 0x1.a01a02p-16f;
    p = __fmaf_rn(p, r, 0x1.a01a02p-13f);
    p = __fmaf_rn(p, r, 0x1.6c16c2p-10f);
    p = __fmaf_rn(p, r, 0x1.111112p-7f);
    p = __fmaf_rn(p, r, 0x1.555556p-5f);
    p = __fmaf_rn(p, r, 0x1.555556p-3f);
    p = __fmaf_rn(p, r, 0.5f);
    p = __fmaf_rn(p, r, 1.0f);
    p = __fmaf_rn(p, r, 1.0f);
    return p * (x < -87.33654f ? 0.0f : __uint_as_float((__float_as_uint(s) << 23) + 0x3f800000u));
}

struct TileConsts {
    float sp2, sn2, sl2;     // the three sigma^2
    float yp, yn, yl;        // their negated reciprocals
};

// tap_weight of two taps at once: centres (element ca, cb), neighbours (na,
// nb), base weights `base`. The negated centre values are added where
// tap_weight subtracts; the clamps only replace arguments whose exponential
// is zero anyway.
template <bool FastDiv>
RR_D u64 tile_weights(const TileSmem& t, u64 cx, u64 cy, u64 cz, u64 mx_, u64 my_, u64 mz_, u64 cl, int na, int nb,
                      u64 base, const TileConsts& c) {
    auto at = [&](int k) { return pack2(t.p[k][na], t.p[k][nb]); };
    const u64 dx = add2(at(0), cx), dy = add2(at(1), cy), dz = add2(at(2), cz);
    u64 d2 = add2(add2(mul2(dx, dx), mul2(dy, dy)), mul2(dz, dz));
    u64 nd = add2(add2(mul2(mx_, at(3)), mul2(my_, at(4))), mul2(mz_, at(5)));
    nd = add2(both(1.0f), nd);
    nd = pack2(max_nan(0.0f, lo2(nd)), max_nan(0.0f, hi2(nd)));
    const float la = t.p[6][na] + lo2(cl), lb = t.p[6][nb] + hi2(cl);
    float la2 = la * la, lb2 = lb * lb;
    if constexpr (FastDiv) {
        const float ap = c.sp2 * 100.0f, al = c.sl2 * 100.0f;
        d2 = pack2(min_nan(lo2(d2), ap), min_nan(hi2(d2), ap));
        la2 = min_nan(la2, al);
        lb2 = min_nan(lb2, al);
    }
    const u64 wp = exp2_nonpos(neg_quotient<FastDiv>(d2, both(c.sp2), both(c.yp)));
    const u64 wn = exp2_nonpos(neg_quotient<FastDiv>(nd, both(c.sn2), both(c.yn)));
    const u64 wl = pack2(exp1_nonpos(neg_quotient1<FastDiv>(la2, c.sl2, c.yl)),
                         exp1_nonpos(neg_quotient1<FastDiv>(lb2, c.sl2, c.yl)));
    return mul2(mul2(mul2(base, wp), wn), wl);
}

// The halo's forward weights that point into the tile: rows -2 and -1 (15
// taps of 36 columns), then 15 (column, tap) pairs of 16 rows on the sides.
constexpr int kHaloTop = 15 * kHaloW, kHaloItems = kHaloTop + 15 * kTileH;
__constant__ signed char kHaloSide[15][3] = {
    {-1, 1, 0}, {-1, 2, 0}, {-1, 1, 1}, {-1, 2, 1}, {-1, 1, 2}, {-1, 2, 2}, {-2, 2, 0}, {-2, 2, 1}, {-2, 2, 2},
    {kTileW, -1, 1}, {kTileW, -2, 1}, {kTileW, -1, 2}, {kTileW, -2, 2}, {kTileW + 1, -2, 1}, {kTileW + 1, -2, 2}};
static_assert(kHaloItems % 2 == 0 && kHaloItems / 2 <= kTileThreads, "one packed halo item per thread");
RR_D void halo_item(int n, int& elem, int& nb, int& tap, float& base) {
    int i, j, tx, ty;
    if (n < kHaloTop) {
        const int k = n / kHaloW;
        i = n % kHaloW - 2;
        j = k < 5 ? -2 : -1;
        ty = k < 5 ? 2 : 1 + (k - 5) / 5;
        tx = k < 5 ? k - 2 : (k - 5) % 5 - 2;
    } else {
        const int k = (n - kHaloTop) / kTileH;
        j = (n - kHaloTop) % kTileH;
        i = kHaloSide[k][0]; tx = kHaloSide[k][1]; ty = kHaloSide[k][2];
    }
    elem = (j + 2) * kHaloW + i + 2;
    // a corner's tap that leaves the tile is not needed: any element will do
    nb = (j + ty + 2) * kHaloW + min(max(i + tx, -2), kTileW + 1) + 2;
    tap = pair_index(tx, ty);
    base = (kernel_weight(tx) * kernel_weight(ty)) / 256.0f;
}

// Tma: the three images' boxes are copied by TMA (stride 1), with a bounded
// wait; a block whose wait gives up sets the flag and reads global memory
// instead (same bits). nrm: unit normals. FastDiv: see neg_div2.
template <bool Tma, bool FastDiv>
__global__ void __launch_bounds__(kTileThreads, 2) atrous_tile_kernel(
    const __grid_constant__ CUtensorMap m_rad, const __grid_constant__ CUtensorMap m_pos,
    const __grid_constant__ CUtensorMap m_nrm, const float4* __restrict__ in, const float4* __restrict__ gpos,
    const float4* __restrict__ nrm, float4* __restrict__ out, int W, int H, int stride, TileConsts c, int* error,
    uint32_t wait_tries) {
    extern __shared__ __align__(128) unsigned char sm[];
    TileSmem& t = *reinterpret_cast<TileSmem*>(sm);
    const int phx = blockIdx.x % stride, phy = blockIdx.y % stride;
    const int i0 = int(blockIdx.x / stride) * kTileW, j0 = int(blockIdx.y / stride) * kTileH;
    const int tid = threadIdx.x;
    bool staged = false;
    const float4* box = reinterpret_cast<const float4*>(sm + ((kTileSmem + 127) & ~127u));
    if constexpr (Tma) {
        uint64_t* bar = reinterpret_cast<uint64_t*>(sm + ((kTileSmem + 127) & ~127u) + 3 * kTileBoxBytes);
        if (tid == 0) {
            tc::mbar_init(bar, 1);
            tc::fence_proxy_async();
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_addr(bar)),
                         "r"(3 * kTileBoxBytes)
                         : "memory");
            void* dst = const_cast<float4*>(box);
            tma_load_3d(dst, &m_rad, 0, i0 - 2, j0 - 2, bar);
            tma_load_3d(static_cast<char*>(dst) + kTileBoxBytes, &m_pos, 0, i0 - 2, j0 - 2, bar);
            tma_load_3d(static_cast<char*>(dst) + 2 * kTileBoxBytes, &m_nrm, 0, i0 - 2, j0 - 2, bar);
        }
        __syncthreads();
        const bool arrived = tc::mbar_wait(bar, 0, wait_tries);
        staged = __syncthreads_and(arrived) != 0;
        if (!staged) {
            // report it in the host-mapped flag, and give the copies one more
            // bounded wait so that none is left writing this block's shared
            // memory after it leaves
            *reinterpret_cast<volatile int*>(error) = 1;
            tc::mbar_wait(bar, 0);
        }
    }
    for (int e = tid; e < kTileElems; e += kTileThreads) {
        const int ux = phx + (i0 + e % kHaloW - 2) * stride, uy = phy + (j0 + e / kHaloW - 2) * stride;
        const int x = min(max(ux, 0), W - 1), y = min(max(uy, 0), H - 1);
        float4 r, p, n;
        if (Tma && staged && ux == x && uy == y) {
            r = box[e];
            p = box[kTileElems + e];
            n = box[2 * kTileElems + e];
        } else {
            const size_t k = size_t(y) * W + x;
            r = __ldg(in + k);
            p = __ldg(gpos + k);
            n = __ldg(nrm + k);
        }
        // A miss: no weight (it is infinitely far from every surface; where
        // sigma_position^2 is infinite too that makes a NaN, which the sum
        // below replaces), no radiance.
        const bool miss = p.w < 0.0f;
        t.rad[e] = miss ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : make_float4(r.x, r.y, r.z, 1.0f);
        t.p[0][e] = miss ? INFINITY : p.x;
        t.p[1][e] = miss ? INFINITY : p.y;
        t.p[2][e] = miss ? INFINITY : p.z;
        t.p[3][e] = miss ? 0.0f : n.x;
        t.p[4][e] = miss ? 0.0f : n.y;
        t.p[5][e] = miss ? 0.0f : n.z;
        t.p[6][e] = miss ? 0.0f : luminance601(xyz(r));
    }
    __syncthreads();
    const int i = tid % kTileW, j = tid / kTileW;
    const int ce = (j + 2) * kHaloW + i + 2;
    {
        const u64 cx = both(-t.p[0][ce]), cy = both(-t.p[1][ce]), cz = both(-t.p[2][ce]);
        const u64 mx_ = both(-t.p[3][ce]), my_ = both(-t.p[4][ce]), mz_ = both(-t.p[5][ce]);
        const u64 cl = both(-t.p[6][ce]);
        // the 12 forward taps as 6 pairs
        constexpr int kPairs[6][4] = {{1, 0, 2, 0}, {-2, 1, -1, 1}, {0, 1, 1, 1}, {2, 1, 2, 2}, {-2, 2, -1, 2}, {0, 2, 1, 2}};
        #pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int ax = kPairs[k][0], ay = kPairs[k][1], bx = kPairs[k][2], by = kPairs[k][3];
            const u64 w = tile_weights<FastDiv>(
                t, cx, cy, cz, mx_, my_, mz_, cl, ce + ay * kHaloW + ax, ce + by * kHaloW + bx,
                pack2((kernel_weight(ax) * kernel_weight(ay)) / 256.0f, (kernel_weight(bx) * kernel_weight(by)) / 256.0f),
                c);
            t.wt[pair_index(ax, ay)][ce] = lo2(w);
            t.wt[pair_index(bx, by)][ce] = hi2(w);
        }
    }
    if (tid < kHaloItems / 2) {
        int ea, na, ta, eb, nb, tb;
        float ba, bb;
        halo_item(tid, ea, na, ta, ba);
        halo_item(tid + kHaloItems / 2, eb, nb, tb, bb);
        auto neg = [&](int k) { return pack2(-t.p[k][ea], -t.p[k][eb]); };
        const u64 w = tile_weights<FastDiv>(t, neg(0), neg(1), neg(2), neg(3), neg(4), neg(5), neg(6), na, nb,
                                            pack2(ba, bb), c);
        t.wt[ta][ea] = lo2(w);
        t.wt[tb][eb] = hi2(w);
    }
    __syncthreads();
    const int x = phx + (i0 + i) * stride, y = phy + (j0 + j) * stride;
    if (x >= W || y >= H) return;
    const size_t ci = size_t(y) * W + x;
    const float4 crad = __ldg(in + ci);
    if (t.p[0][ce] == INFINITY && __ldg(gpos + ci).w < 0.0f) {
        out[ci] = crad;
        return;
    }
    // the centre's own weight: its distances are zero (NaN where a value is not finite)
    float wc;
    {
        const float px = t.p[0][ce], py = t.p[1][ce], pz = t.p[2][ce], l = t.p[6][ce];
        const float3 n = f3(t.p[3][ce], t.p[4][ce], t.p[5][ce]);
        const float nd = mx(0.0f, 1.0f - dot(n, n));
        const float none = ((px - px) + (py - py)) + ((pz - pz) + (l - l));
        wc = (kernel_weight(0) * kernel_weight(0)) / 256.0f * rr_expf(-nd / c.sn2) + none;
    }
    u64 frg = 0, fbw = 0;   // (red, green), (blue, sum of weights)
    #pragma unroll
    for (int ty = -2; ty <= 2; ++ty) {
        #pragma unroll
        for (int tx = -2; tx <= 2; ++tx) {
            const int e = ce + ty * kHaloW + tx;
            float w = tx == 0 && ty == 0 ? wc
                      : pair_forward(tx, ty) ? t.wt[pair_index(tx, ty)][ce] : t.wt[pair_index(-tx, -ty)][e];
            const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(&t.rad[e]);
            if (!FastDiv && hi2(r.y) == 0.0f) w = 0.0f;   // a miss
            frg = add2(frg, mul2(r.x, both(w)));
            fbw = add2(fbw, mul2(r.y, both(w)));
        }
    }
    const float wsum = hi2(fbw);
    const float3 f = f3(lo2(frg), hi2(frg), lo2(fbw));
    const float3 o = wsum > 0.0f ? f / wsum : xyz(crad);
    out[ci] = make_float4(o.x, o.y, o.z, crad.w);
}

} // namespace
} // namespace rr

// cuTensorMapEncodeTiled from the driver (no link-time dependency on it).
PFN_cuTensorMapEncodeTiled_v12000 rr_tensor_map_encoder() {
    // looked up once (a function-local static: initialised once, thread-safe)
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        return static_cast<PFN_cuTensorMapEncodeTiled_v12000>(nullptr);
    }();
    return fn;
}

// A W x H RGBA32F image as a 3-D tensor (4 floats, W, H) with a box of
// (4, bw, bh); false if the driver refuses it (the caller then uses the
// direct-load kernel).
static bool image_map(CUtensorMap* m, const void* img, uint32_t W, uint32_t H, uint32_t bw, uint32_t bh) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = rr_tensor_map_encoder();
    if (!enc || (reinterpret_cast<uintptr_t>(img) & 15u) != 0) return false;
    const cuuint64_t dims[3] = {4, W, H};
    const cuuint64_t strides[2] = {16, cuuint64_t(W) * 16};
    const cuuint32_t box[3] = {4, bw, bh};
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(img), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The lattice tile kernel for one iteration; false where the driver refuses
// the tensor maps (the caller then launches it without).
template <bool Tma>
static bool atrous_tile_launch(rr_ctx* ctx, const float* input, const float* gpos, const float4* nrm, float* output,
                               uint32_t W, uint32_t H, uint32_t stride, float sp2, float sn2, float sl2,
                               cudaStream_t stream) {
    CUtensorMap mr{}, mp{}, mn{};
    if (Tma && (!image_map(&mr, input, W, H, rr::kHaloW, rr::kHaloH) ||
                !image_map(&mp, gpos, W, H, rr::kHaloW, rr::kHaloH) ||
                !image_map(&mn, nrm, W, H, rr::kHaloW, rr::kHaloH)))
        return false;
    const auto in_range = [](float b) { return b >= 1e-6f && b <= 1e12f; };
    const bool fast = in_range(sp2) && in_range(sn2) && in_range(sl2);
    const auto kernel = fast ? rr::atrous_tile_kernel<Tma, true> : rr::atrous_tile_kernel<Tma, false>;
    const uint32_t smem = Tma ? rr::kTileSmemTma : rr::kTileSmem;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return false;
    const rr::TileConsts c{sp2, sn2, sl2, -1.0f / sp2, -1.0f / sn2, -1.0f / sl2};
    const uint32_t lw = (W + stride - 1) / stride, lh = (H + stride - 1) / stride;   // a phase's lattice
    const dim3 grid((lw + rr::kTileW - 1) / rr::kTileW * stride, (lh + rr::kTileH - 1) / rr::kTileH * stride);
    kernel<<<grid, rr::kTileThreads, smem, stream>>>(
        mr, mp, mn, reinterpret_cast<const float4*>(input), reinterpret_cast<const float4*>(gpos), nrm,
        reinterpret_cast<float4*>(output), int(W), int(H), int(stride), c, ctx->atrous_error_dev,
        ctx->atrous_wait_tries);
    return true;
}

// Whether a stride's lattice fills the tiles well enough for the tile kernel
// (one iteration in us, tile / pair kernels: 1920 x 1080 stride 64, 50 % full,
// 300 / 312; 957 x 541 stride 64, 26 %, 135 / 89; 333 x 217 stride 32, 15 %,
// 39 / 32, stride 16, 57 %, 19 / 33; 128 x 128 stride 16, 12 %, 17 / 31,
// stride 32, 3 %, 37 / 31; 64 x 64 stride 8, 12 %, 12 / 31). Small launches
// run at the latency of one tile, up to a few tiles per SM.
static bool atrous_tiled(uint32_t W, uint32_t H, uint32_t stride) {
    if (stride == 0 || stride > 1024u) return false;
    const uint64_t lw = (W + stride - 1) / stride, lh = (H + stride - 1) / stride;
    const uint64_t tiles = ((lw + rr::kTileW - 1) / rr::kTileW) * ((lh + rr::kTileH - 1) / rr::kTileH);
    return lw * lh * 5 >= tiles * rr::kTileThreads * 2 || tiles * stride * stride <= 300u;
}

// Unit normals of `gnrm` into the context's scratch image.
static rr_status atrous_normals(rr_ctx* ctx, const float* gnrm, uint32_t W, uint32_t H, cudaStream_t stream,
                                const float4** out) {
    const size_t n = size_t(W) * H;
    if (ctx->atrous_nrm_px < n) {
        cudaFree(ctx->atrous_nrm);
        ctx->atrous_nrm = nullptr;
        ctx->atrous_nrm_px = 0;
        RR_TRY_CUDA(ctx, cudaMalloc(&ctx->atrous_nrm, n * sizeof(float4)));
        ctx->atrous_nrm_px = n;
    }
    rr::normalize_kernel<<<unsigned((n + 255) / 256), 256, 0, stream>>>(reinterpret_cast<const float4*>(gnrm),
                                                                        ctx->atrous_nrm, n);
    RR_CHECK_LAUNCH(ctx);
    ctx->launches += 1;
    *out = ctx->atrous_nrm;
    return RR_OK;
}

static rr_status atrous_launch(rr_ctx* ctx, const float* input, const float* gpos, const float4* nrm,
                               float* output, uint32_t W, uint32_t H, uint32_t stride, float sp, float sn,
                               float sl, cudaStream_t stream) {
    const float sp2 = std::max(sp * sp, 1.0e-6f), sn2 = std::max(sn * sn, 1.0e-6f), sl2 = std::max(sl * sl, 1.0e-6f);
    if (atrous_tiled(W, H, stride)) {
        bool launched = false;
        if (ctx->atrous_tma && stride == 1) {
            if (!ctx->atrous_error) {
                // one host-mapped word: a block that gives up writes it, and the
                // next A-trous call reads it without synchronizing
                int* h = nullptr;
                RR_TRY_CUDA(ctx, cudaHostAlloc(reinterpret_cast<void**>(&h), sizeof(int), cudaHostAllocMapped));
                *reinterpret_cast<volatile int*>(h) = 0;
                void* d = nullptr;
                cudaError_t e = cudaHostGetDevicePointer(&d, h, 0);
                if (e != cudaSuccess) {
                    cudaFreeHost(h);
                    RR_TRY_CUDA(ctx, e);
                }
                ctx->atrous_error = h;
                ctx->atrous_error_dev = static_cast<int*>(d);
            }
            launched = atrous_tile_launch<true>(ctx, input, gpos, nrm, output, W, H, stride, sp2, sn2, sl2, stream);
        }
        if (!launched)
            launched = atrous_tile_launch<false>(ctx, input, gpos, nrm, output, W, H, stride, sp2, sn2, sl2, stream);
        if (launched) {
            RR_CHECK_LAUNCH(ctx);
            ctx->launches += 1;
            return RR_OK;
        }
    }
    const size_t need = size_t(rr::kPairFwd) * W * H;
    if (ctx->atrous_wt_floats < need) {
        cudaFree(ctx->atrous_wt);
        ctx->atrous_wt = nullptr;
        ctx->atrous_wt_floats = 0;
        RR_TRY_CUDA(ctx, cudaMalloc(&ctx->atrous_wt, need * sizeof(float)));
        ctx->atrous_wt_floats = need;
    }
    dim3 grid((W + 15) / 16, (H + 7) / 8);
    rr::atrous_pair_weights_kernel<<<grid, 128, 0, stream>>>(
        reinterpret_cast<const float4*>(input), reinterpret_cast<const float4*>(gpos), nrm, ctx->atrous_wt, int(W),
        int(H), int(stride), sp2, sn2, sl2);
    RR_CHECK_LAUNCH(ctx);
    rr::atrous_pair_sum_kernel<<<grid, 128, 0, stream>>>(
        reinterpret_cast<const float4*>(input), reinterpret_cast<const float4*>(gpos), nrm, ctx->atrous_wt,
        reinterpret_cast<float4*>(output), int(W), int(H), int(stride), sp2, sn2, sl2);
    RR_CHECK_LAUNCH(ctx);
    ctx->launches += 2;
    return RR_OK;
}

// An earlier call's tile copies missed their bounded wait (the flag the
// blocks write into host-mapped memory): reported once, here, at the next
// call, which then does no work. The earlier call's output is complete: the
// blocks that gave up filtered their pixels from global memory.
static rr_status atrous_report_give_up(rr_ctx* ctx, const char* who) {
    if (!ctx->atrous_error || *reinterpret_cast<volatile int*>(ctx->atrous_error) == 0) return RR_OK;
    *reinterpret_cast<volatile int*>(ctx->atrous_error) = 0;
    return rr_fail(ctx, RR_ERR_TIMEOUT,
                   "%s: an earlier A-trous call's TMA tile copies did not complete within the bounded wait "
                   "(that call's output was filtered from global memory instead); this call did no work",
                   who);
}

extern "C" rr_status rr_atrous_iteration(rr_ctx* ctx, const float* input, const float* gpos,
                                         const float* gnrm, float* output, const rr_atrous_params* p,
                                         void* stream) {
    if (!ctx) return RR_ERR_INVALID_ARGUMENT;
    if (!input || !gpos || !gnrm || !output || !p) return rr_fail(ctx, RR_ERR_INVALID_ARGUMENT, "rr_atrous_iteration: null argument");
    if (p->width == 0 || p->height == 0 || p->width > 65535u * 16u || p->height > 65535u * 8u)
        return rr_fail(ctx, RR_ERR_INVALID_ARGUMENT, "rr_atrous_iteration: bad image size");
    if (input == output) return rr_fail(ctx, RR_ERR_INVALID_ARGUMENT, "rr_atrous_iteration: input aliases output");
    if (rr_status g = atrous_report_give_up(ctx, "rr_atrous_iteration")) return g;
    RR_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    const float4* nrm = nullptr;
    rr_status st = atrous_normals(ctx, gnrm, p->width, p->height, static_cast<cudaStream_t>(stream), &nrm);
    if (st != RR_OK) return st;
    return atrous_launch(ctx, input, gpos, nrm, output, p->width, p->height, p->stride, p->sigma_position,
                         p->sigma_normal, p->sigma_luminance, static_cast<cudaStream_t>(stream));
}

extern "C" rr_status rr_atrous_execute(rr_ctx* ctx, const float* input, const float* gpos, const float* gnrm,
                                       float* ping0, float* ping1, const rr_atrous_params* p,
                                       uint32_t* out_slot, void* stream) {
    if (!ctx) return RR_ERR_INVALID_ARGUMENT;
    if (!input || !gpos || !gnrm || !ping0 || !ping1 || !p)
        return rr_fail(ctx, RR_ERR_INVALID_ARGUMENT, "rr_atrous_execute: null argument");
    if (p->width == 0 || p->height == 0 || p->width > 65535u * 16u || p->height > 65535u * 8u)
        return rr_fail(ctx, RR_ERR_INVALID_ARGUMENT, "rr_atrous_execute: bad image size");
    if (input == ping0 || input == ping1 || ping0 == ping1)
        return rr_fail(ctx, RR_ERR_INVALID_ARGUMENT, "rr_atrous_execute: buffers alias");
    if (rr_status g = atrous_report_give_up(ctx, "rr_atrous_execute")) return g;
    RR_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    // AtrousPass.cpp:265 clamps to 1..7; slot (iterations-1)&1 holds the result.
    const uint32_t iters = std::min(std::max(p->iterations, 1u), 7u);
    const float4* nrm = nullptr;
    rr_status st0 = atrous_normals(ctx, gnrm, p->width, p->height, static_cast<cudaStream_t>(stream), &nrm);
    if (st0 != RR_OK) return st0;
    const float* read = input;
    float* ping[2] = {ping0, ping1};
    for (uint32_t it = 0; it < iters; ++it) {
        float* write = ping[it & 1u];
        rr_status st = atrous_launch(ctx, read, gpos, nrm, write, p->width, p->height, 1u << it,
                                     p->sigma_position, p->sigma_normal, p->sigma_luminance,
                                     static_cast<cudaStream_t>(stream));
        if (st != RR_OK) return st;
        read = write;
    }
    if (out_slot) *out_slot = (iters - 1u) & 1u;
    return RR_OK;
}

extern "C" rr_status rr_atrous_set_tma(rr_ctx* ctx, int enable) {
    if (!ctx) return RR_ERR_INVALID_ARGUMENT;
    ctx->atrous_tma = enable != 0;
    return RR_OK;
}

extern "C" rr_status rr_atrous_tma_error(rr_ctx* ctx, int* error_out) {
    if (!ctx || !error_out) return RR_ERR_INVALID_ARGUMENT;
    *error_out = 0;
    if (!ctx->atrous_error) return RR_OK;
    RR_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    RR_TRY_CUDA(ctx, cudaDeviceSynchronize());
    *error_out = *reinterpret_cast<volatile int*>(ctx->atrous_error);
    *reinterpret_cast<volatile int*>(ctx->atrous_error) = 0;
    return RR_OK;
}

extern "C" rr_status rr_atrous_set_tma_wait_tries(rr_ctx* ctx, uint32_t tries) {
    if (!ctx) return RR_ERR_INVALID_ARGUMENT;
    ctx->atrous_wait_tries = tries;
    return RR_OK;
}
