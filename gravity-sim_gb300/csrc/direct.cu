// direct.cu -- O(N^2) direct-sum force with the integrator fused into the epilogue.
//
// Replaces src/Simulation/Direct/Shaders/SimShader.comp:37-74 (one dispatch per step,
// src/Simulation/Direct/DirectSimulation.cpp:306-319).
//
// FAST mode: j is staged 64 sources at a time in shared memory (loaded as float4 pairs of
// positions and float2 pairs of masses: j-tiles start at multiples of 64) and broadcast to
// the threads, which keep their targets in registers.  Each 64-wide tile is summed plainly
// in FP32, and the tile partials are added with Kahan compensation.
//   k_direct_small  (N <= 12,288) 32 targets per block, the tiles split over its 16 warps and
//                   the warps' compensated sums added in shared memory
//   k_direct_fast   (larger N) i-tiles of 128 threads with IPT targets each, j-chunks; every
//                   block stores its compensated partial and the last block to finish an
//                   i-tile (ticket counter, no waiting) adds the chunks in chunk order, again
//                   with Kahan, and applies the integrator
// Results do not depend on block scheduling.
//
// REFERENCE mode (k_direct_ref): j ascending over all N_al particles, plain FP32
// accumulation and correctly rounded 1/sqrt -- the shader's order, bit-identical to the CPU
// restatement; the factors of the terms are made ahead of the sums by other warps.
//
// Roofline: 14 algorithmic FLOP per pair (2 sub, 2 FMA for r^2, rsqrt, 3 mul, 2 FMA),
// 9 FP32 operations + 1 MUFU per pair, issued as packed f32x2 instructions for a thread's
// two targets (4.5 issues + 1 MUFU per pair); FP32-bound.
#include "bh_common.cuh"

namespace gsim {
namespace {

constexpr int kDirectBlock = 128;
constexpr int kDirectTileJ = 64;
constexpr int kDirectIpt = 2;  // default targets per thread (gs_shape.direct_targets: 2 or 4), in packed f32x2 pairs

// 1/sqrt of a softened squared distance.  d2 >= eps2, so with a normal eps2 (FTZ) it is
// never subnormal and the flush-to-zero form gives the same bits; the plain form also
// scales subnormal inputs, six more instructions per pair of targets.
template <bool FTZ>
__device__ __forceinline__ float direct_rsqrt(float x) {
    if (!FTZ) return rsqrtf(x);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__host__ __device__ __forceinline__ bool direct_ftz(float eps2) { return eps2 >= 1.17549435e-38f; }

// s + c carries the running sum (c: what the last additions lost); adds v to it.
__device__ __forceinline__ void kahan_add(float v, float& s, float& c) {
    const float y = v - c, u = s + y;
    c = (u - s) - y;
    s = u;
}

// Two consecutive sources (x, y, m pairs) on one target (P, Q: its position twice).  The
// sources share packed f32x2 instructions up to the two sums, which take them in order:
// dx, dy, d2 = fma(dx, dx, fma(dy, dy, eps2)), s = ((m r) r) r, t += d s, each lane rounding
// like the scalar instruction.
template <bool FTZ>
__device__ __forceinline__ void tile_pair(float2 x, float2 y, float2 m, float2 P, float2 Q, float2 E2, float& tx,
                                          float& ty) {
    const float2 dx = sub2(x, P), dy = sub2(y, Q);
    const float2 d2 = fma2(dx, dx, fma2(dy, dy, E2));
    const float2 r = make_float2(direct_rsqrt<FTZ>(d2.x), direct_rsqrt<FTZ>(d2.y));
    const float2 s = mul2(mul2(mul2(m, r), r), r);
    tx = fmaf(dx.x, s.x, tx);
    ty = fmaf(dy.x, s.x, ty);
    tx = fmaf(dx.y, s.y, tx);
    ty = fmaf(dy.y, s.y, ty);
}

// Block (bx, by) of a large system: 128 IPT targets (i-tile bx), j-chunk by.  A plain launch
// passes blockIdx.x / blockIdx.y, a batched launch the block's position inside its system's
// grid.  KAHAN false (GS_FLAG_PLAIN_SUM) adds the tile partials and the chunks plainly, for
// the precision study against the compensated sums.
//
// The loop is bound by the FMA pipe (9 packed operations of two cycles for a source and two
// targets) next to the 16 cycles that two MUFU instructions take: 18 of about 23.5 cycles a
// source.  N = 50,000: 964 us a step with the rsqrt form that scales subnormal inputs, a tile
// loaded between two barriers and chunks for one set of resident blocks; 738 us with the
// flush-to-zero form, the next tile in flight and two sets (the shorter chunks even out the
// tail).  Eight targets per thread (112 registers) took 861 us, equal contiguous runs of
// (target group, tile) units per block 827 us.
template <int IPT, bool KAHAN, bool FTZ>
__device__ __forceinline__ void direct_fast_body(uint32_t bx, uint32_t by, const float2* __restrict__ pos,
                                                 const float2* __restrict__ vel, const float* __restrict__ mass,
                                                 float2* __restrict__ pos_out, float2* __restrict__ vel_out,
                                                 float2* __restrict__ acc_rec, uint32_t n_al, int chunks,
                                                 uint32_t jchunk, float eps2, float k, float hdt,
                                                 float4* __restrict__ partials, uint32_t* __restrict__ tickets) {
    __shared__ float4 sj[2][kDirectTileJ];
    __shared__ uint32_t s_ticket;
    const int t = threadIdx.x;
    const uint32_t tile_base = bx * (kDirectBlock * IPT);
    const uint32_t j0 = by * jchunk;
    const uint32_t j1 = min(j0 + jchunk, n_al);

    static_assert(IPT % 2 == 0, "targets per thread come in packed f32x2 pairs");
    float px[IPT], py[IPT], sx[IPT], sy[IPT], cx[IPT], cy[IPT];
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        uint32_t i = tile_base + t + r * kDirectBlock;
        float2 p = i < n_al ? pos[i] : make_float2(0.f, 0.f);
        px[r] = p.x;
        py[r] = p.y;
        sx[r] = sy[r] = cx[r] = cy[r] = 0.f;
    }
    constexpr int NP = IPT / 2;
    float2 P2[NP], Q2[NP];
#pragma unroll
    for (int h = 0; h < NP; ++h) {
        P2[h] = make_float2(px[2 * h], px[2 * h + 1]);
        Q2[h] = make_float2(py[2 * h], py[2 * h + 1]);
    }
    const float2 E2 = make_float2(eps2, eps2);

    // the first half of the threads stage a tile: one float4 of two positions and one float2
    // of their masses each, loaded while the tile before is summed
    const bool stage = t < kDirectTileJ / 2;
    const float4* pos2 = reinterpret_cast<const float4*>(pos) + t;
    const float2* mass2 = reinterpret_cast<const float2*>(mass) + t;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    float2 m = make_float2(0.f, 0.f);
    if (stage) {
        q = pos2[j0 >> 1];
        m = mass2[j0 >> 1];
    }
    int buf = 0;
    for (uint32_t jt = j0; jt < j1; jt += kDirectTileJ, buf ^= 1) {
        if (stage) {  // the other buffer's readers passed the barrier of the tile before
            sj[buf][2 * t] = make_float4(q.x, q.y, m.x, 0.f);
            sj[buf][2 * t + 1] = make_float4(q.z, q.w, m.y, 0.f);
            if (jt + kDirectTileJ < j1) {
                q = pos2[(jt + kDirectTileJ) >> 1];
                m = mass2[(jt + kDirectTileJ) >> 1];
            }
        }
        __syncthreads();
        // Pairs of the thread's targets share packed f32x2 instructions (each lane rounds
        // like the scalar one, in the same order: dx, dy, d2 = fma(dx, dx, fma(dy, dy,
        // eps2)), s = ((m r) r) r, t += d s), so the bits are those of scalar evaluations.
        float2 tx2[NP], ty2[NP];
#pragma unroll
        for (int h = 0; h < NP; ++h) tx2[h] = ty2[h] = make_float2(0.f, 0.f);
#pragma unroll 16
        for (int jj = 0; jj < kDirectTileJ; ++jj) {
            const float4 g = sj[buf][jj];
#pragma unroll
            for (int h = 0; h < NP; ++h) {
                const float2 dx = sub2(make_float2(g.x, g.x), P2[h]), dy = sub2(make_float2(g.y, g.y), Q2[h]);
                const float2 d2 = fma2(dx, dx, fma2(dy, dy, E2));
                const float2 rr = make_float2(direct_rsqrt<FTZ>(d2.x), direct_rsqrt<FTZ>(d2.y));
                const float2 s = mul2(mul2(mul2(make_float2(g.z, g.z), rr), rr), rr);
                tx2[h] = fma2(dx, s, tx2[h]);
                ty2[h] = fma2(dy, s, ty2[h]);
            }
        }
#pragma unroll
        for (int r = 0; r < IPT; ++r) {  // Kahan-compensated add of the tile partial
            const float tx = r & 1 ? tx2[r / 2].y : tx2[r / 2].x, ty = r & 1 ? ty2[r / 2].y : ty2[r / 2].x;
            if (!KAHAN) {
                sx[r] += tx;
                sy[r] += ty;
                continue;
            }
            kahan_add(tx, sx[r], cx[r]);
            kahan_add(ty, sy[r], cy[r]);
        }
    }

    if (chunks > 1) {
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            uint32_t i = tile_base + t + r * kDirectBlock;
            if (i < n_al) partials[(size_t)by * n_al + i] = make_float4(sx[r], sy[r], cx[r], cy[r]);
        }
        __threadfence();
        __syncthreads();
        if (t == 0) s_ticket = atomicAdd(&tickets[bx], 1u);
        __syncthreads();
        if (s_ticket != (uint32_t)chunks - 1) return;
        __threadfence();
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            uint32_t i = tile_base + t + r * kDirectBlock;
            float ax = 0.f, ay = 0.f, kx = 0.f, ky = 0.f;
            if (i < n_al) {
#pragma unroll 8
                for (int c = 0; c < chunks; ++c) {
                    const float4 pc = __ldcg(&partials[(size_t)c * n_al + i]);
                    if (!KAHAN) {
                        ax += pc.x;
                        ay += pc.y;
                        continue;
                    }
                    kahan_add(pc.x - pc.z, ax, kx);
                    kahan_add(pc.y - pc.w, ay, ky);
                }
            }
            sx[r] = ax;
            cx[r] = kx;
            sy[r] = ay;
            cy[r] = ky;
        }
        if (t == 0) tickets[bx] = 0u;  // ready for the next step
    }

#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        uint32_t i = tile_base + t + r * kDirectBlock;
        if (i >= n_al) continue;
        float ax = sx[r] - cx[r], ay = sy[r] - cy[r];
        if (acc_rec) acc_rec[i] = make_float2(ax, ay);
        float2 v = vel[i];
        float nvx = fmaf(ax, k, v.x), nvy = fmaf(ay, k, v.y);  // SimShader.comp:68
        pos_out[i] = make_float2(fmaf(v.x + nvx, hdt, px[r]), fmaf(v.y + nvy, hdt, py[r]));  // :69
        vel_out[i] = make_float2(nvx, nvy);
    }
}

// A small system: 32 targets per block, one per lane, and the 64-wide source tiles split over
// the block's W warps.  Part p of min(16, K) parts holds tiles [p K / P, (p + 1) K / P) and
// is summed by warp p mod W with Kahan compensation; the parts are then added in part order
// in shared memory, again with Kahan.  The parts do not depend on W, so it changes no bit.
// What bounds a small system is latency (a block's chain of tile loads and sums) and the
// number of warps: N = 4096 as 16 i-tiles x 16 j-chunks of 128-thread blocks, combined
// through global partials by the last block, kept 1.7 warps per scheduler busy and took
// 20.6 us a step; 128 blocks of 16 warps, each staging its own tiles without a block barrier,
// 10.4 us (N = 1024: 16.5 -> 6.2 us, N = 8192: 41.2 -> 30.9 us).  The tiles are staged as
// separate x, y and m arrays so that two consecutive sources share packed instructions.
// Beyond kDirectSmallMax the 4-byte-per-lane broadcasts of one target per lane bound the
// loop (three 16-byte shared loads per four sources and 32 targets), and the large-system
// kernel is faster (N = 12288: 65.5 us here).
constexpr uint32_t kDirectParts = 16;
constexpr uint32_t kDirectSmallMax = 12288;
constexpr int kDirectSmallWarps = 16;

template <int W>
struct DirectSmallSmem {
    float x[W][kDirectTileJ], y[W][kDirectTileJ], m[W][kDirectTileJ];
    float4 part[kDirectParts][32];  // {sx, sy, cx, cy}
};

template <int W, bool KAHAN, bool FTZ>
__device__ __forceinline__ void direct_small_body(DirectSmallSmem<W>& g, uint32_t bx, const float2* __restrict__ pos,
                                                  const float2* __restrict__ vel, const float* __restrict__ mass,
                                                  float2* __restrict__ pos_out, float2* __restrict__ vel_out,
                                                  float2* __restrict__ acc_rec, uint32_t n_al, float eps2, float k,
                                                  float hdt) {
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tiles = n_al / kDirectTileJ, parts = min(kDirectParts, tiles);
    const uint32_t i = bx * 32 + lane;  // n_al is a multiple of 64: every target exists
    const float2 p = pos[i];
    const float2 P = make_float2(p.x, p.x), Q = make_float2(p.y, p.y), E2 = make_float2(eps2, eps2);
    const float4* X = reinterpret_cast<const float4*>(g.x[w]);
    const float4* Y = reinterpret_cast<const float4*>(g.y[w]);
    const float4* M = reinterpret_cast<const float4*>(g.m[w]);
    for (uint32_t part = w; part < parts; part += W) {
        const uint32_t t0 = part * tiles / parts, t1 = (part + 1) * tiles / parts;
        float sx = 0.f, sy = 0.f, cx = 0.f, cy = 0.f;
        float4 q = reinterpret_cast<const float4*>(pos)[t0 * 32 + lane];  // two positions and their masses
        float2 m = reinterpret_cast<const float2*>(mass)[t0 * 32 + lane];
        for (uint32_t jt = t0; jt < t1; ++jt) {
            __syncwarp();
            reinterpret_cast<float2*>(g.x[w])[lane] = make_float2(q.x, q.z);
            reinterpret_cast<float2*>(g.y[w])[lane] = make_float2(q.y, q.w);
            reinterpret_cast<float2*>(g.m[w])[lane] = m;
            __syncwarp();
            if (jt + 1 < t1) {  // in flight while this tile is summed
                q = reinterpret_cast<const float4*>(pos)[(jt + 1) * 32 + lane];
                m = reinterpret_cast<const float2*>(mass)[(jt + 1) * 32 + lane];
            }
            float tx = 0.f, ty = 0.f;
#pragma unroll
            for (int jj = 0; jj < kDirectTileJ / 4; ++jj) {
                const float4 x4 = X[jj], y4 = Y[jj], m4 = M[jj];
                tile_pair<FTZ>(make_float2(x4.x, x4.y), make_float2(y4.x, y4.y), make_float2(m4.x, m4.y), P, Q, E2, tx,
                               ty);
                tile_pair<FTZ>(make_float2(x4.z, x4.w), make_float2(y4.z, y4.w), make_float2(m4.z, m4.w), P, Q, E2, tx,
                               ty);
            }
            if (KAHAN) {
                kahan_add(tx, sx, cx);
                kahan_add(ty, sy, cy);
            } else {
                sx += tx;
                sy += ty;
            }
        }
        g.part[part][lane] = make_float4(sx, sy, cx, cy);
    }
    __syncthreads();
    if (w) return;
    float ax = 0.f, ay = 0.f, kx = 0.f, ky = 0.f;
    for (uint32_t part = 0; part < parts; ++part) {
        const float4 q = g.part[part][lane];
        if (KAHAN) {
            kahan_add(q.x - q.z, ax, kx);
            kahan_add(q.y - q.w, ay, ky);
        } else {
            ax += q.x;
            ay += q.y;
        }
    }
    ax -= kx;
    ay -= ky;
    if (acc_rec) acc_rec[i] = make_float2(ax, ay);
    const float2 v = vel[i];
    const float nvx = fmaf(ax, k, v.x), nvy = fmaf(ay, k, v.y);  // SimShader.comp:68
    pos_out[i] = make_float2(fmaf(v.x + nvx, hdt, p.x), fmaf(v.y + nvy, hdt, p.y));  // :69
    vel_out[i] = make_float2(nvx, nvy);
}

template <bool KAHAN, bool FTZ>
__global__ void __launch_bounds__(kDirectSmallWarps * 32)
k_direct_small(const float2* __restrict__ pos, const float2* __restrict__ vel, const float* __restrict__ mass,
               float2* __restrict__ pos_out, float2* __restrict__ vel_out, float2* __restrict__ acc_rec,
               uint32_t n_al, float eps2, float k, float hdt) {
    pdl_enter();
    __shared__ __align__(16) DirectSmallSmem<kDirectSmallWarps> g;
    direct_small_body<kDirectSmallWarps, KAHAN, FTZ>(g, blockIdx.x, pos, vel, mass, pos_out, vel_out, acc_rec, n_al, eps2,
                                                     k, hdt);
}

// 1 / sqrt(x) with both operations correctly rounded, for two values at once: the value of
// __frcp_rn(__fsqrt_rn(x)).  The method is Markstein's (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): from
// an approximation y of 1/sqrt(x), a Newton step in g ~ sqrt(x) and h ~ 1/(2 sqrt(x))
//     g = x y, h = y / 2, e = 1/2 - g h, g += g e, h += h e,
// then the residual x - g^2, exact in an FMA, gives the rounded root s = g + (x - g^2) h, and two
// steps r += (1 - s r) r from r = 2 h the rounded reciprocal (one leaves two mantissas, whose
// reciprocals lie 5e-8 of a unit from a rounding boundary, one unit off).  No step overflows
// or loses bits to underflow for x in [2^-100, 2^100].  Markstein's theorem on reciprocals leaves
// out a root of all-ones mantissa: r stays 2^-k, its residual half a unit that rounds away.  Such
// a root comes from the two floats just below a power of 4, mantissas 0x7ffffe and 0x7fffff.
// Those, and an x outside the range (a zero, a NaN, an overflowed distance), go to the library
// functions; with them every mantissa of both exponent parities gives the library's bits, for any
// estimate y within two units of the root's reciprocal.  In packed f32x2 form the chain is 6.5
// issues a value; the library's root and reciprocal carry their own range checks and branches,
// most of the 47 instructions that a factor cost.
__device__ __forceinline__ float2 ref_inv_sqrt2(float2 x) {
    const float2 y = make_float2(direct_rsqrt<true>(x.x), direct_rsqrt<true>(x.y));
    float2 g = mul2(x, y), h = mul2(y, make_float2(0.5f, 0.5f));
    const float2 e = fma2(make_float2(-g.x, -g.y), h, make_float2(0.5f, 0.5f));
    g = fma2(g, e, g);
    h = fma2(h, e, h);
    const float2 s = fma2(fma2(make_float2(-g.x, -g.y), g, x), h, g);
    const float2 ns = make_float2(-s.x, -s.y), one = make_float2(1.0f, 1.0f);
    const float2 r = add2(h, h), r1 = fma2(fma2(ns, r, one), r, r);
    float2 v = fma2(fma2(ns, r1, one), r1, r1);
    const float lo = 7.888609052e-31f, hi = 1.267650600e30f;  // 2^-100, 2^100
    const uint32_t ones = 0x7ffffeu;  // the last mantissa bit is free
    if (!(x.x >= lo && x.x <= hi && x.y >= lo && x.y <= hi) || (__float_as_uint(x.x) & ones) == ones ||
        (__float_as_uint(x.y) & ones) == ones) {
        v.x = __frcp_rn(__fsqrt_rn(x.x));
        v.y = __frcp_rn(__fsqrt_rn(x.y));
    }
    return v;
}

// REFERENCE math: 32 targets per block.  The shader's sum takes the sources in order
// (SimShader.comp:43-65), but only the two additions of each pair depend on the pair before;
// the factors s = ((m r) r) r with r = 1 / sqrt(d2), both correctly rounded, do not.  So 16
// warps make the factors of a 64-source tile (lane: target, four sources per warp, two per
// packed instruction) in shared memory while two more add up an earlier tile, one the x and
// one the y sums, each lane its own target in source order.  One thread per particle doing
// both was bound by its own chain of dependent divisions (N = 4096: 128 warps on the whole
// chip, 328 us a step; now 43).  A block takes 22 cycles a source, of which the dependent
// additions are 4.  No pipe is full (N = 4096: issue 58 % of the busy SMs' cycles, ALU 45, FMA
// 29): a tile takes a block 3,130 warp instructions, and its warps, 4.5 a scheduler, wait on
// their own results, branches and the hand-over's barriers.
constexpr int kRefWarps = 16;                        // warps that make factors
constexpr int kRefThreads = (kRefWarps + 2) * 32;
constexpr uint32_t kRefTargets = 32;
constexpr int kRefPer = 4;                           // sources per warp and tile: two float4 of positions, one of masses
constexpr int kRefTile = kRefWarps * kRefPer;
static_assert(kAlignment % kRefTile == 0, "whole tiles");

// Tiles of factors in flight between the making and the adding warps.
constexpr int kRefRing = 4;

struct DirectRefSmem {
    float s[kRefRing][kRefTile][kRefTargets];
    float c[kRefRing][2][kRefTile];  // the tile's x and y
    float a[kRefTargets];
};

// Named barriers of ring slot b: full (1 + b), its factors are made; empty (1 + kRefRing + b),
// they have been added up.  Both count every thread of the block: one side arrives, the other
// waits.
__device__ __forceinline__ void ref_arrive(uint32_t id) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kRefThreads) : "memory");
}
__device__ __forceinline__ void ref_wait(uint32_t id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kRefThreads) : "memory");
}

// The factors of two sources for one target: dx, dy, d2 = fma(dx, dx, fma(dy, dy, eps2)), then
// ((m r) r) r, each lane rounding like the scalar operations.
__device__ __forceinline__ float2 ref_factors(float2 x, float2 y, float2 m, float2 P, float2 Q, float2 E2, float2& dx,
                                              float2& dy) {
    dx = sub2(x, P);
    dy = sub2(y, Q);
    const float2 r = ref_inv_sqrt2(fma2(dx, dx, fma2(dy, dy, E2)));
    return mul2(mul2(mul2(m, r), r), r);
}

__device__ __forceinline__ void direct_ref_body(DirectRefSmem& g, uint32_t bx, const float2* __restrict__ pos,
                                                const float2* __restrict__ vel, const float* __restrict__ mass,
                                                float2* __restrict__ pos_out, float2* __restrict__ vel_out,
                                                float2* __restrict__ acc_rec, uint32_t n_al, float eps2, float k,
                                                float hdt) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t i = bx * kRefTargets + lane, tiles = n_al / kRefTile;
    const float2 p = pos[i];
    const float2 P = make_float2(p.x, p.x), Q = make_float2(p.y, p.y), E2 = make_float2(eps2, eps2);
    const float4* pos2 = reinterpret_cast<const float4*>(pos);
    const float4* mass4 = reinterpret_cast<const float4*>(mass);
    const int f = w * kRefPer;  // the warp's first source of a tile
    // the sources of this tile and of the next two: a tile is made in less than an L2 round trip
    float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0, m = q0, q0b = q0, q1b = q0, mb = q0;
    const auto load = [&](uint32_t jt, float4& a0, float4& a1, float4& am) {
        const uint32_t n0 = jt * kRefTile + f;
        a0 = __ldg(&pos2[n0 / 2]);
        a1 = __ldg(&pos2[n0 / 2 + 1]);
        am = __ldg(&mass4[n0 / 4]);
    };
    if (w < kRefWarps) {
        load(0, q0, q1, m);
        if (tiles > 1) load(1, q0b, q1b, mb);
    }
    const int axis = w - kRefWarps;  // of an adding warp: 0 x, 1 y
    const float pc = axis ? p.y : p.x;
    float a = 0.f;
    if (w < kRefWarps) {
        for (uint32_t jt = 0; jt < tiles; ++jt) {
            const uint32_t b = jt % kRefRing;
            const float4 p0 = q0, p1 = q1, pm = m;
            q0 = q0b;
            q1 = q1b;
            m = mb;
            if (jt + 2 < tiles) load(jt + 2, q0b, q1b, mb);
            float2 dx, dy;
            const float2 sa = ref_factors(make_float2(p0.x, p0.z), make_float2(p0.y, p0.w), make_float2(pm.x, pm.y), P,
                                          Q, E2, dx, dy);
            const float2 sb = ref_factors(make_float2(p1.x, p1.z), make_float2(p1.y, p1.w), make_float2(pm.z, pm.w), P,
                                          Q, E2, dx, dy);
            if (jt >= kRefRing) ref_wait(1 + kRefRing + b);
            g.s[b][f][lane] = sa.x;
            g.s[b][f + 1][lane] = sa.y;
            g.s[b][f + 2][lane] = sb.x;
            g.s[b][f + 3][lane] = sb.y;
            if (lane < kRefPer) {
                g.c[b][0][f + lane] = lane == 0 ? p0.x : lane == 1 ? p0.z : lane == 2 ? p1.x : p1.z;
                g.c[b][1][f + lane] = lane == 0 ? p0.y : lane == 1 ? p0.w : lane == 2 ? p1.y : p1.w;
            }
            ref_arrive(1 + b);
        }
    } else {
        for (uint32_t jt = 0; jt < tiles; ++jt) {
            const uint32_t b = jt % kRefRing;
            ref_wait(1 + b);
            // eight sources at a time, the next eight's factors and coordinates loaded before
            // the sums of this eight, so that the dependent additions do not wait for loads
            const float4* c4 = reinterpret_cast<const float4*>(g.c[b][axis]);
            float sv[8], sn[8];
            float4 c0 = c4[0], c1 = c4[1], n0 = c0, n1 = c1;
#pragma unroll
            for (int u = 0; u < 8; ++u) sv[u] = g.s[b][u][lane];
#pragma unroll
            for (int t = 0; t < kRefTile; t += 8) {
                if (t + 8 < kRefTile) {
                    n0 = c4[t / 4 + 2];
                    n1 = c4[t / 4 + 3];
#pragma unroll
                    for (int u = 0; u < 8; ++u) sn[u] = g.s[b][t + 8 + u][lane];
                }
                const float d[8] = {c0.x - pc, c0.y - pc, c0.z - pc, c0.w - pc, c1.x - pc, c1.y - pc, c1.z - pc, c1.w - pc};
#pragma unroll
                for (int u = 0; u < 8; ++u) a = fmaf(d[u], sv[u], a);
                c0 = n0;
                c1 = n1;
#pragma unroll
                for (int u = 0; u < 8; ++u) sv[u] = sn[u];
            }
            if (jt + kRefRing < tiles) ref_arrive(1 + kRefRing + b);  // one for each later wait
        }
    }
    if (axis == 1) g.a[lane] = a;
    __syncthreads();
    if (axis != 0) return;
    const float ax = a, ay = g.a[lane];
    if (acc_rec) acc_rec[i] = make_float2(ax, ay);
    const float2 v = vel[i];
    const float nvx = fmaf(ax, k, v.x), nvy = fmaf(ay, k, v.y);
    pos_out[i] = make_float2(fmaf(v.x + nvx, hdt, p.x), fmaf(v.y + nvy, hdt, p.y));
    vel_out[i] = make_float2(nvx, nvy);
}

// REFERENCE math, large systems: a warp per 32 targets makes the factors and adds them up
// itself, four sources at a time.  There are warps enough to hide each one's chain, and
// nothing is handed over.
template <int W>
struct DirectRowsSmem {
    float x[W][kDirectTileJ], y[W][kDirectTileJ], m[W][kDirectTileJ];
};
constexpr int kRowsWarps = 2;

template <int W>
__device__ __forceinline__ void direct_rows_body(DirectRowsSmem<W>& g, uint32_t bx, const float2* __restrict__ pos,
                                                 const float2* __restrict__ vel, const float* __restrict__ mass,
                                                 float2* __restrict__ pos_out, float2* __restrict__ vel_out,
                                                 float2* __restrict__ acc_rec, uint32_t n_al, float eps2, float k,
                                                 float hdt) {
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t i = (bx * W + w) * 32 + lane, tiles = n_al / kDirectTileJ;
    if (i >= n_al) return;  // the whole warp: n_al is a multiple of 64
    const float2 p = pos[i];
    const float2 P = make_float2(p.x, p.x), Q = make_float2(p.y, p.y), E2 = make_float2(eps2, eps2);
    const float4* X = reinterpret_cast<const float4*>(g.x[w]);
    const float4* Y = reinterpret_cast<const float4*>(g.y[w]);
    const float4* M = reinterpret_cast<const float4*>(g.m[w]);
    float ax = 0.f, ay = 0.f;
    float4 q = reinterpret_cast<const float4*>(pos)[lane];  // two positions and their masses
    float2 m = reinterpret_cast<const float2*>(mass)[lane];
    for (uint32_t jt = 0; jt < tiles; ++jt) {
        __syncwarp();
        reinterpret_cast<float2*>(g.x[w])[lane] = make_float2(q.x, q.z);
        reinterpret_cast<float2*>(g.y[w])[lane] = make_float2(q.y, q.w);
        reinterpret_cast<float2*>(g.m[w])[lane] = m;
        __syncwarp();
        if (jt + 1 < tiles) {  // in flight while this tile is summed
            q = reinterpret_cast<const float4*>(pos)[(jt + 1) * 32 + lane];
            m = reinterpret_cast<const float2*>(mass)[(jt + 1) * 32 + lane];
        }
#pragma unroll 2
        for (int jj = 0; jj < kDirectTileJ / 4; ++jj) {
            const float4 x = X[jj], y = Y[jj], c = M[jj];
            float2 dxa, dya, dxb, dyb;
            const float2 sa = ref_factors(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(c.x, c.y), P, Q, E2,
                                          dxa, dya);
            const float2 sb = ref_factors(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(c.z, c.w), P, Q, E2,
                                          dxb, dyb);
            ax = fmaf(dxa.x, sa.x, ax);
            ay = fmaf(dya.x, sa.x, ay);
            ax = fmaf(dxa.y, sa.y, ax);
            ay = fmaf(dya.y, sa.y, ay);
            ax = fmaf(dxb.x, sb.x, ax);
            ay = fmaf(dyb.x, sb.x, ay);
            ax = fmaf(dxb.y, sb.y, ax);
            ay = fmaf(dyb.y, sb.y, ay);
        }
    }
    if (acc_rec) acc_rec[i] = make_float2(ax, ay);
    const float2 v = vel[i];
    const float nvx = fmaf(ax, k, v.x), nvy = fmaf(ay, k, v.y);
    pos_out[i] = make_float2(fmaf(v.x + nvx, hdt, p.x), fmaf(v.y + nvy, hdt, p.y));
    vel_out[i] = make_float2(nvx, nvy);
}

// Which REFERENCE-math kernel a system takes (the same bits either way), and its blocks.
// N = 12,288: 316 us a step on k_direct_ref, 409 here; 16,384: 548 and 543; 50,000: 4464 and 2486
// (4330 with a thread per particle and the library's root and division).
constexpr uint32_t kRefSplitMax = 16384;
__host__ __device__ __forceinline__ bool ref_rows(uint32_t n_al) { return n_al > kRefSplitMax; }
static uint32_t ref_blocks(uint32_t n_al, int rows_warps) {
    return ref_rows(n_al) ? (n_al / 32 + rows_warps - 1) / rows_warps : n_al / kRefTargets;
}

__global__ void __launch_bounds__(kRowsWarps * 32)
k_direct_rows(const float2* __restrict__ pos, const float2* __restrict__ vel, const float* __restrict__ mass,
              float2* __restrict__ pos_out, float2* __restrict__ vel_out, float2* __restrict__ acc_rec, uint32_t n_al,
              float eps2, float k, float hdt) {
    pdl_enter();
    __shared__ __align__(16) DirectRowsSmem<kRowsWarps> g;
    direct_rows_body<kRowsWarps>(g, blockIdx.x, pos, vel, mass, pos_out, vel_out, acc_rec, n_al, eps2, k, hdt);
}

template <int IPT, bool KAHAN, bool FTZ>
__global__ void __launch_bounds__(kDirectBlock)
k_direct_fast(const float2* __restrict__ pos, const float2* __restrict__ vel, const float* __restrict__ mass,
              float2* __restrict__ pos_out, float2* __restrict__ vel_out, float2* __restrict__ acc_rec,
              uint32_t n_al, int chunks, uint32_t jchunk, float eps2, float k, float hdt, float4* __restrict__ partials,
              uint32_t* __restrict__ tickets) {
    pdl_enter();
    direct_fast_body<IPT, KAHAN, FTZ>(blockIdx.x, blockIdx.y, pos, vel, mass, pos_out, vel_out, acc_rec, n_al, chunks,
                                      jchunk, eps2, k, hdt, partials, tickets);
}

__global__ void __launch_bounds__(kRefThreads, 2)
k_direct_ref(const float2* __restrict__ pos, const float2* __restrict__ vel, const float* __restrict__ mass,
             float2* __restrict__ pos_out, float2* __restrict__ vel_out, float2* __restrict__ acc_rec,
             uint32_t n_al, float eps2, float k, float hdt) {
    pdl_enter();
    __shared__ __align__(16) DirectRefSmem g;
    direct_ref_body(g, blockIdx.x, pos, vel, mass, pos_out, vel_out, acc_rec, n_al, eps2, k, hdt);
}

// Batched direct sum: one launch over every direct-sum system of a plan.  Block b belongs
// to the system whose table range holds it and does the work of the plain launch's block of
// that index (small systems on four warps per block instead of sixteen, which changes no bit).
__device__ __forceinline__ uint32_t direct_batch_sys(const uint32_t* __restrict__ first, uint32_t nsys,
                                                     uint32_t b) {
    uint32_t lo = 0, hi = nsys;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&first[mid]) <= b) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <int IPT, bool KAHAN, bool FTZ>
__device__ __forceinline__ void direct_batch_body(DirectSmallSmem<kDirectBlock / 32>& g, const SysDesc& d, uint32_t b,
                                                  int in, int out) {
    if (!d.chunks)
        direct_small_body<kDirectBlock / 32, KAHAN, FTZ>(g, b, d.pos[in], d.vel[in], d.mass[in], d.pos[out], d.vel[out],
                                                         d.acc, d.n_al, d.eps2, d.k, d.hdt);
    else
        direct_fast_body<IPT, KAHAN, FTZ>(b % d.itiles, b / d.itiles, d.pos[in], d.vel[in], d.mass[in], d.pos[out],
                                          d.vel[out], d.acc, d.n_al, (int)d.chunks, d.jchunk, d.eps2, d.k, d.hdt,
                                          d.partials, d.tickets);
}

template <bool EXACT, bool KAHAN, int IPT>
__global__ void __launch_bounds__(EXACT ? kRefThreads : kDirectBlock, EXACT ? 2 : IPT == 4 ? 6 : 8)
kb_direct(const SysDesc* __restrict__ descs, const uint32_t* __restrict__ first, uint32_t nsys, uint32_t step) {
    const uint32_t s = direct_batch_sys(first, nsys, blockIdx.x);
    const SysDesc& d = descs[s];
    const uint32_t b = blockIdx.x - __ldg(&first[s]);
    const int in = (int)((d.parity + step) & 1u), out = in ^ 1;
    if constexpr (EXACT) {
        __shared__ __align__(16) union {
            DirectRefSmem split;
            DirectRowsSmem<kRefThreads / 32> rows;
        } g;
        if (ref_rows(d.n_al))
            direct_rows_body<kRefThreads / 32>(g.rows, b, d.pos[in], d.vel[in], d.mass[in], d.pos[out], d.vel[out],
                                               d.acc, d.n_al, d.eps2, d.k, d.hdt);
        else
            direct_ref_body(g.split, b, d.pos[in], d.vel[in], d.mass[in], d.pos[out], d.vel[out], d.acc, d.n_al, d.eps2,
                            d.k, d.hdt);
    } else {
        __shared__ __align__(16) DirectSmallSmem<kDirectBlock / 32> g;
        if (direct_ftz(d.eps2)) direct_batch_body<IPT, KAHAN, true>(g, d, b, in, out);
        else direct_batch_body<IPT, KAHAN, false>(g, d, b, in, out);
    }
}

__global__ void __launch_bounds__(256)
k_accel_f64(const uint32_t* __restrict__ targets, const float2* __restrict__ pos,
            const float* __restrict__ mass, uint32_t n, double eps2, double2* __restrict__ out) {
    __shared__ double sx[256], sy[256];
    const uint32_t i = targets[blockIdx.x];
    const double px = pos[i].x, py = pos[i].y;
    double ax = 0.0, ay = 0.0;
    for (uint32_t j = threadIdx.x; j < n; j += 256) {
        double dx = (double)pos[j].x - px, dy = (double)pos[j].y - py;
        double d2 = dx * dx + dy * dy + eps2;
        double s = (double)mass[j] / (d2 * sqrt(d2));
        ax += dx * s;
        ay += dy * s;
    }
    sx[threadIdx.x] = ax;
    sy[threadIdx.x] = ay;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            sx[threadIdx.x] += sx[threadIdx.x + w];
            sy[threadIdx.x] += sy[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = make_double2(sx[0], sy[0]);
}

// Energy in FP64 (diagnostic, not on the step path): per block of 256 particles i, the
// kinetic energy 1/2 m |v|^2 and m_i * sum_{j != i} m_j / sqrt(|p_j - p_i|^2 + eps^2), the
// latter over j tiles staged in shared memory; block sums in a fixed tree order.
__global__ void __launch_bounds__(256)
k_energy_f64(const float2* __restrict__ pos, const float2* __restrict__ vel, const float* __restrict__ mass,
             uint32_t n, double eps2, double2* __restrict__ part) {
    __shared__ double sx[256], sy[256], sm[256];
    const uint32_t t = threadIdx.x, i = blockIdx.x * 256 + t;
    const bool own = i < n;
    const double px = own ? (double)pos[i].x : 0.0, py = own ? (double)pos[i].y : 0.0;
    const double mi = own ? (double)mass[i] : 0.0;
    double pot = 0.0;
    for (uint32_t jt = 0; jt < n; jt += 256) {
        const uint32_t j = jt + t;
        sx[t] = j < n ? (double)pos[j].x : 0.0;
        sy[t] = j < n ? (double)pos[j].y : 0.0;
        sm[t] = j < n ? (double)mass[j] : 0.0;
        __syncthreads();
        for (uint32_t jj = 0; jj < 256; ++jj) {
            if (jt + jj == i) continue;
            const double dx = sx[jj] - px, dy = sy[jj] - py;
            pot += sm[jj] / sqrt(dx * dx + dy * dy + eps2);
        }
        __syncthreads();
    }
    const double vx = own ? (double)vel[i].x : 0.0, vy = own ? (double)vel[i].y : 0.0;
    sx[t] = 0.5 * mi * (vx * vx + vy * vy);
    sy[t] = mi * pot;
    __syncthreads();
    for (uint32_t w = 128; w > 0; w >>= 1) {
        if (t < w) {
            sx[t] += sx[t + w];
            sy[t] += sy[t + w];
        }
        __syncthreads();
    }
    if (t == 0) part[blockIdx.x] = make_double2(sx[0], sy[0]);
}

}  // namespace

gs_status energy_f64(gs_sim* s, double* kinetic, double* potential) {
    const uint32_t n = (uint32_t)s->n_al;
    const uint32_t blocks = (n + 255) / 256;
    double2* part = nullptr;
    GS_CUDA(cudaMallocAsync(&part, blocks * sizeof(double2), s->stream));
    k_energy_f64<<<blocks, 256, 0, s->stream>>>(s->pos[s->in], s->vel[s->in], s->mass[s->in], n, (double)s->eps2,
                                                 part);
    double2* host = new double2[blocks];
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, part, blocks * sizeof(double2), cudaMemcpyDeviceToHost, s->stream);
    cudaFreeAsync(part, s->stream);
    gs_status w = e == cudaSuccess ? sim_wait(s) : cuda_fail(e, "energy_f64");
    if (w != GS_OK) {  // the readback may still be pending: keep its destination alive
        if (w != GS_ERR_TIMEOUT) delete[] host;
        return w;
    }
    double ke = 0.0, pp = 0.0;
    for (uint32_t b = 0; b < blocks; ++b) {
        ke += host[b].x;
        pp += host[b].y;
    }
    delete[] host;
    *kinetic = ke;
    *potential = -0.5 * (double)s->G * pp;  // every pair was counted from both ends
    return GS_OK;
}

// j-chunks that gs_set_shape judges a shape by: enough blocks for blocks_per_sm on every SM, at
// least 256 sources per chunk, at most 64 chunks
static int pick_chunks(uint64_t n_al, int ipt, uint32_t blocks_per_sm) {
    const uint64_t itiles = (n_al + kDirectBlock * ipt - 1) / (kDirectBlock * ipt);
    const uint64_t want_blocks = 152ull * blocks_per_sm;
    uint64_t c = (want_blocks + itiles - 1) / itiles;
    uint64_t max_c = n_al / 256;  // keep at least 256 sources per chunk
    if (c > max_c) c = max_c;
    if (c < 1) c = 1;
    if (c > 64) c = 64;
    return (int)c;
}

// one ticket per i-tile of two targets per thread, the smallest
static uint64_t direct_tickets(uint64_t n_al) { return (n_al + kDirectBlock * 2 - 1) / (kDirectBlock * 2); }

// The j-split of a system: chunks of jchunk sources (a multiple of 64); chunks 0: a small
// system (k_direct_small).  Enough chunks for blocks_per_sm blocks of four targets per thread
// on every SM (twice as many blocks of two), at least 512 sources in each and at most
// max_chunks (the scratch's rows).
struct DirectGrid {
    uint32_t chunks, jchunk;
};
static uint32_t pick_rows(uint64_t n_al, uint32_t blocks_per_sm) {
    if (n_al <= kDirectSmallMax) return 0;
    const uint64_t itiles = (n_al + kDirectBlock * 4 - 1) / (kDirectBlock * 4), want = 152ull * blocks_per_sm;
    uint64_t c = (want + itiles - 1) / itiles;
    if (c > n_al / 512) c = n_al / 512;
    return (uint32_t)(c < 1 ? 1 : c > 64 ? 64 : c);
}
static DirectGrid pick_grid(uint64_t n_al, uint32_t blocks_per_sm, uint32_t max_chunks) {
    DirectGrid g{};
    uint64_t c = pick_rows(n_al, blocks_per_sm);
    if (!c) return g;
    if (c > max_chunks) c = max_chunks;
    const uint64_t j = (n_al + c - 1) / c;
    g.jchunk = (uint32_t)((j + kDirectTileJ - 1) / kDirectTileJ * kDirectTileJ);
    g.chunks = (uint32_t)((n_al + g.jchunk - 1) / g.jchunk);
    return g;
}

static int shape_ipt(const gs_shape& sh) { return sh.direct_targets == 4 ? 4 : 2; }

ShapeUse direct_shape_use(const gs_params* p, uint64_t n_al) {
    ShapeUse u;
    u.direct = p->math_mode != GS_MATH_REFERENCE && n_al > kDirectSmallMax;
    return u;
}

// Lays the j-chunk partials and tickets out in the system's slab (sizing pass: counts), for
// the j-split of the creation shape (a later shape's split is capped by it).
// direct_max_chunks is gs_set_shape's limit and no scratch: what pick_chunks gives for the
// creation shape, as callers of gs_set_shape know it.
void direct_carve(gs_sim* s) {
    DirectWork& w = s->dw;
    const int c2 = pick_chunks(s->n_al, 2, s->shape.direct_blocks_per_sm);
    const int c4 = pick_chunks(s->n_al, 4, s->shape.direct_blocks_per_sm);
    s->direct_max_chunks = (uint32_t)(c2 > c4 ? c2 : c4);
    w.partials = nullptr;
    w.tickets = nullptr;
    w.rows = pick_rows(s->n_al, s->shape.direct_blocks_per_sm);
    if (w.rows > 1) {
        sim_carve(s, (void**)&w.partials, sizeof(float4) * s->n_al * (size_t)w.rows);
        sim_carve(s, (void**)&w.tickets, sizeof(uint32_t) * direct_tickets(s->n_al));
    }
}

uint32_t direct_chunks_needed(const gs_sim* s, const gs_shape& sh) {
    return (uint32_t)pick_chunks(s->n_al, shape_ipt(sh), sh.direct_blocks_per_sm);
}

cudaError_t direct_init(gs_sim* s) {
    const DirectWork& w = s->dw;
    if (!w.tickets) return cudaSuccess;
    return cudaMemsetAsync(w.tickets, 0, sizeof(uint32_t) * direct_tickets(s->n_al), s->stream);
}

// How a system splits its sum: from its own shape, so that it sums in the same order
// whichever targets per thread run it (alone or in a batch).
static DirectGrid direct_grid(const gs_sim* s) {
    return pick_grid(s->n_al, s->shape.direct_blocks_per_sm, s->dw.rows);
}
static uint32_t direct_itiles(uint64_t n_al, int ipt) { return (uint32_t)((n_al + kDirectBlock * ipt - 1) / (kDirectBlock * ipt)); }

// The fast kernels' launch; every array as the kernels take it.  pdl: the launch may begin
// while the step before it still runs (the kernels wait for it on entry).
static cudaError_t direct_fast_launch(bool pdl, const DirectGrid& d, int ipt, bool plain, const float2* pos,
                                      const float2* vel, const float* mass, float2* pos_out, float2* vel_out,
                                      float2* acc, uint32_t n_al, float eps2, float k, float hdt, float4* partials,
                                      uint32_t* tickets, cudaStream_t st) {
    const bool ftz = direct_ftz(eps2);
    if (!d.chunks) {
        auto fn = plain ? (ftz ? k_direct_small<false, true> : k_direct_small<false, false>)
                        : (ftz ? k_direct_small<true, true> : k_direct_small<true, false>);
        return launch(pdl, fn, dim3(n_al / 32), kDirectSmallWarps * 32, st, pos, vel, mass, pos_out, vel_out, acc,
                      n_al, eps2, k, hdt);
    }
    auto fn = plain ? (ftz ? (ipt == 4 ? k_direct_fast<4, false, true> : k_direct_fast<2, false, true>)
                           : (ipt == 4 ? k_direct_fast<4, false, false> : k_direct_fast<2, false, false>))
                    : (ftz ? (ipt == 4 ? k_direct_fast<4, true, true> : k_direct_fast<2, true, true>)
                           : (ipt == 4 ? k_direct_fast<4, true, false> : k_direct_fast<2, true, false>));
    return launch(pdl, fn, dim3(direct_itiles(n_al, ipt), d.chunks), kDirectBlock, st, pos, vel, mass, pos_out, vel_out,
                  acc, n_al, (int)d.chunks, d.jchunk, eps2, k, hdt, partials, tickets);
}

cudaError_t direct_step(gs_sim* s, int in, int out, bool profile, bool chained) {
    const float k = s->dt_eff * s->G;  // SimShader.comp:68 (SIMULATION_TIME * GRAVITATIONAL_CONST)
    const float hdt = 0.5f * s->dt_eff;
    const uint32_t n_al = (uint32_t)s->n_al;
    const bool pdl = chained && !profile;
    cudaError_t e;
    stage_begin(s, kStageDirect, profile);
    if (s->p.math_mode == GS_MATH_REFERENCE)
        e = launch(pdl, ref_rows(n_al) ? k_direct_rows : k_direct_ref, dim3(ref_blocks(n_al, kRowsWarps)),
                   ref_rows(n_al) ? kRowsWarps * 32 : kRefThreads, s->stream, s->pos[in], s->vel[in], s->mass[in],
                   s->pos[out], s->vel[out], s->acc, n_al, s->eps2, k, hdt);
    else
        e = direct_fast_launch(pdl, direct_grid(s), shape_ipt(s->shape), (s->p.flags & GS_FLAG_PLAIN_SUM) != 0,
                               s->pos[in], s->vel[in], s->mass[in], s->pos[out], s->vel[out], s->acc, n_al, s->eps2, k,
                               hdt, s->dw.partials, s->dw.tickets, s->stream);
    count_launch(s);
    stage_end(s, kStageDirect, profile);
    return e;
}

void direct_batch_desc(gs_sim* s, SysDesc& d, uint32_t blocks[kTabCount], const gs_shape& batch_shape) {
    for (int t = 0; t < kTabCount; ++t) blocks[t] = 0;
    const DirectGrid g = direct_grid(s);
    d.itiles = direct_itiles(s->n_al, shape_ipt(batch_shape));
    d.chunks = g.chunks;
    d.jchunk = g.jchunk;
    d.partials = s->dw.partials;
    d.tickets = s->dw.tickets;
    blocks[kTabDirect] = s->p.math_mode == GS_MATH_REFERENCE ? ref_blocks((uint32_t)s->n_al, kRefThreads / 32)
                         : g.chunks                          ? d.itiles * g.chunks
                                                             : (uint32_t)(s->n_al / 32);
}

cudaError_t direct_batch_step(const BatchPlan& p, uint32_t step, cudaStream_t st) {
    if (!p.n_direct) return cudaSuccess;
    const SysDesc* descs = p.d_descs + p.n_bh;
    const bool four = shape_ipt(p.shape) == 4;
    if (p.direct_exact)
        kb_direct<true, false, 2><<<p.total[kTabDirect], kRefThreads, 0, st>>>(descs, p.d_tab[kTabDirect], p.n_direct, step);
    else
        (p.direct_plain ? (four ? kb_direct<false, false, 4> : kb_direct<false, false, 2>)
                        : (four ? kb_direct<false, true, 4> : kb_direct<false, true, 2>))
            <<<p.total[kTabDirect], kDirectBlock, 0, st>>>(descs, p.d_tab[kTabDirect], p.n_direct, step);
    return cudaGetLastError();
}

cudaError_t accel_f64(gs_sim* s, uint32_t n_targets, const uint32_t* d_targets, double2* d_out) {
    const double eps2 = (double)s->eps2;  // the softening the FP32 path uses, exactly
    k_accel_f64<<<n_targets, 256, 0, s->stream>>>(d_targets, s->pos[s->in], s->mass[s->in],
                                                  (uint32_t)s->n_al, eps2, d_out);
    return cudaGetLastError();
}

}  // namespace gsim

// ------------------------------------------------------------------------------------
// Direct-sum step that allocates nothing (gs_direct_step_noalloc).
//
// Some callers cannot let a library allocate device memory: a host application that owns
// every device allocation and hands its plugins fixed buffers, or a loop with a fixed
// memory budget that must not pay for (or be synchronised by) cudaMalloc / cudaFree in
// the middle of a run.  For them this entry point takes the particle buffers from the
// caller and keeps its own scratch -- the j-chunk partial sums and the per-tile tickets
// of k_direct_fast -- in the file-scope device arrays below.  Those arrays exist on every
// GPU that loads this library and stay allocated until the process exits.
// ------------------------------------------------------------------------------------
namespace gsim {
namespace {

constexpr size_t kNoAllocPartialBytes = 4u << 20;  // j-chunk partials, 4 MiB
constexpr uint32_t kNoAllocMaxTiles = GS_NOALLOC_MAX_PARTICLES / 256;

static __device__ __align__(256) float4 g_noalloc_partials[kNoAllocPartialBytes / sizeof(float4)];
static __device__ __align__(256) uint32_t g_noalloc_tickets[kNoAllocMaxTiles];

// Device addresses of the two arrays in the current context, looked up on every call:
// the lookup allocates nothing and is cheap, and a cached address could outlive the
// module it points into (cudaDeviceReset, or another context on the same ordinal).  The
// host-side names are stand-ins, not device addresses, so they are never passed to a
// kernel directly.
gs_status noalloc_scratch(float4** partials, uint32_t** tickets) {
    void* p = nullptr;
    void* t = nullptr;
    GS_CUDA(cudaGetSymbolAddress(&p, g_noalloc_partials));
    GS_CUDA(cudaGetSymbolAddress(&t, g_noalloc_tickets));
    *partials = (float4*)p;
    *tickets = (uint32_t*)t;
    return GS_OK;
}

}  // namespace
}  // namespace gsim

extern "C" gs_status gs_direct_step_noalloc(const float* d_pos_in, const float* d_vel_in, const float* d_mass,
                                            float* d_pos_out, float* d_vel_out, uint64_t n,
                                            float gravitational_const, float simulation_time, float softening_len,
                                            void* stream) {
    using namespace gsim;
    if (!d_pos_in || !d_vel_in || !d_mass || !d_pos_out || !d_vel_out) {
        set_error("gs_direct_step_noalloc: NULL buffer");
        return GS_ERR_INVALID_ARGUMENT;
    }
    if (n == 0 || n % kAlignment != 0) {
        set_error("gs_direct_step_noalloc: the particle count must be a positive multiple of 64 "
                  "(pad with zero-mass particles, as ParticleSystem does)");
        return GS_ERR_INVALID_ARGUMENT;
    }
    if (((uintptr_t)d_pos_in & 15u) || ((uintptr_t)d_mass & 7u) || ((uintptr_t)d_vel_in & 7u) ||
        ((uintptr_t)d_pos_out & 7u) || ((uintptr_t)d_vel_out & 7u)) {
        set_error("gs_direct_step_noalloc: pos_in must be 16-byte aligned and the other arrays 8-byte aligned "
                  "(the kernel reads positions as float4 pairs)");
        return GS_ERR_INVALID_ARGUMENT;
    }
    if (n > GS_NOALLOC_MAX_PARTICLES) {
        set_error("gs_direct_step_noalloc: particle count above GS_NOALLOC_MAX_PARTICLES (65536), the size "
                  "of its built-in scratch; use gs_create / gs_run for larger systems");
        return GS_ERR_CAPACITY;
    }
    const uint32_t n_al = (uint32_t)n;
    const uint32_t fit = (uint32_t)(kNoAllocPartialBytes / (sizeof(float4) * n_al));  // >= 4 for n <= 65536
    const DirectGrid split = pick_grid(n_al, 12, fit);
    cudaStream_t s = (cudaStream_t)stream;
    float4* partials = nullptr;
    uint32_t* tickets = nullptr;
    if (split.chunks > 1) {  // small systems need no scratch
        gs_status st = noalloc_scratch(&partials, &tickets);
        if (st != GS_OK) return st;
        // the tickets must start at zero; the array keeps whatever the previous call left
        GS_CUDA(cudaMemsetAsync(tickets, 0, direct_tickets(n_al) * sizeof(uint32_t), s));
    }
    const float eps2 = softening_len * softening_len;
    const float k = simulation_time * gravitational_const;
    const float hdt = 0.5f * simulation_time;
    GS_CUDA(direct_fast_launch(false, split, kDirectIpt, false, (const float2*)d_pos_in, (const float2*)d_vel_in, d_mass,
                               (float2*)d_pos_out, (float2*)d_vel_out, nullptr, n_al, eps2, k, hdt, partials, tickets,
                               s));
    return GS_OK;
}
