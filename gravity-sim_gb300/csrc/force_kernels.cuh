// force_kernels.cuh -- the Barnes-Hut traversal kernels with the integrator fused into
// their epilogue (ForceShader.comp:78-152 and the accurate group walk), plain and batched,
// templated on the math mode and on the launch shape (gs_shape: warps per block, list
// caps).  force_fast.cu and force_exact.cu instantiate them for FAST and REFERENCE math.
#pragma once
#include <type_traits>

#include "bh_common.cuh"
#include "pair_loop.h"

namespace gsim {
namespace {

// ------------------------------------------------------------------------------------
// traversal + integrator (ForceShader.comp:78-152)
// ------------------------------------------------------------------------------------

// 1/sqrt: correctly rounded (REFERENCE math) or the hardware approximation (FAST math;
// d2 >= eps^2 > 0 is never subnormal, so the flush-to-zero form loses nothing)
__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <bool EXACT>
__device__ __forceinline__ float inv_sqrt(float d2) {
    return EXACT ? __fdiv_rn(1.0f, __fsqrt_rn(d2)) : rsqrt_fast(d2);
}

// FAST math of the reference rule, whose softening may be so small that d2 is subnormal
// (FTZ false: the form that scales such inputs); with a normal eps^2 both give the same bits.
template <bool EXACT, bool FTZ>
__device__ __forceinline__ float rule_inv_sqrt(float d2) {
    if (EXACT) return __fdiv_rn(1.0f, __fsqrt_rn(d2));
    return FTZ ? rsqrt_fast(d2) : rsqrtf(d2);
}
__host__ __device__ __forceinline__ bool rule_ftz(float eps2) { return eps2 >= 1.17549435e-38f; }

// Shared memory of a warp's walk: a window of 32 records from `base` on.
struct RuleWindow {
    float4 rec[32];
    uint32_t skip[32];
};

// A warp's walk of the preorder records.  Records are taken four at a time: their distances
// and tests are made together (two records per packed instruction), and when all four are
// accepted and follow one another (particle leaves) all four are summed at once; otherwise
// the four are gone through in order with the distances at hand, as the rule does one by
// one.  After a round that left by an accepted node's skip before its last record the
// next are taken singly until one is followed by its neighbour: a walk among accepted nodes
// (the outskirts of a disk) tests few records in vain.  Force kernel, four always and so: 500k
// spiral 172 and 162 us, 80,000 53.5 and 48.5, 20,000 galaxy 61.5 and 57.6, 3,000 24.6 and 22.8.
// The sums take the records in the same order either way.
// win: the warp's window, or with STAGED (win unused) the whole tree in shared memory at
// s_rec / s_skip.
template <bool EXACT, bool COUNT, bool FTZ, bool STAGED>
__device__ __forceinline__ void force_body(Blk blk, RuleWindow* win, const float4* s_rec, const uint32_t* s_skip,
                                           const uint32_t* __restrict__ sidx, const uint32_t* __restrict__ counts,
                                           const float4* __restrict__ rec, const uint32_t* __restrict__ skip,
                                           const float2* __restrict__ pos_in, const float2* __restrict__ vel_in,
                                           float2* __restrict__ pos_out, float2* __restrict__ vel_out,
                                           float2* __restrict__ acc_rec, uint32_t n_al, float eps2, float theta2,
                                           float k, float hdt, uint32_t cap, unsigned long long* __restrict__ stat,
                                           uint32_t* __restrict__ ext) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t group = blk.id * (blockDim.x >> 5) + warp;
    const uint32_t nv = counts[0];
    const uint32_t T = min(nv + counts[1], cap);  // preorder records
    if (group * 32 >= nv) return;       // no particle in this warp: nothing to write
    const uint32_t s = group * 32 + lane;
    const uint32_t i = s < nv ? sidx[s] : 0u;
    const bool valid = s < nv && i < n_al;  // i < n_al unless the sort failed (error flag set)
    const float2 p = valid ? pos_in[i] : make_float2(0.0f, 0.0f);
    const float2 P = make_float2(p.x, p.x), Q = make_float2(p.y, p.y), E2 = make_float2(eps2, eps2);
    const float2 TH = make_float2(theta2, theta2);
    float ax = 0.0f, ay = 0.0f;
    unsigned long long n_acc = 0, n_vis = 0;
    uint32_t base = 0, ind = 0;
    bool single = false;
    if (!STAGED) {
        win->rec[lane] = rec[lane];
        win->skip[lane] = skip[lane];
        __syncwarp();
    }
    while (ind < T) {
        if (!STAGED && ind - base > 28u) {  // warp-uniform: fewer than four records left in the window
            base = ind;
            __syncwarp();
            win->rec[lane] = rec[base + lane];  // the arrays end 32 records past cap
            win->skip[lane] = skip[base + lane];
            __syncwarp();
        }
        const float4* q = STAGED ? s_rec + ind : win->rec + (ind - base);
        const uint32_t* sk = STAGED ? s_skip + ind : win->skip + (ind - base);
        if (single) {
            const float4 r0 = q[0];
            const uint32_t step = sk[0];
            const float dx = r0.x - p.x, dy = r0.y - p.y, d2 = fmaf(dx, dx, fmaf(dy, dy, eps2));
            if (COUNT) ++n_vis;
            if (__all_sync(0xffffffffu, !valid || r0.w <= d2 * theta2)) {
                const float r = rule_inv_sqrt<EXACT, FTZ>(d2);
                const float sc = ((r0.z * r) * r) * r;
                ax = fmaf(dx, sc, ax);
                ay = fmaf(dy, sc, ay);
                if (COUNT) n_acc += valid;
                ind += max(step, 1u);  // >= 1: the walk always advances
                single = step > 1u;
            } else {
                ++ind;
                single = false;
            }
            continue;
        }
        const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
        const float2 dxa = sub2(make_float2(q0.x, q1.x), P), dya = sub2(make_float2(q0.y, q1.y), Q);
        const float2 dxb = sub2(make_float2(q2.x, q3.x), P), dyb = sub2(make_float2(q2.y, q3.y), Q);
        const float2 da = fma2(dxa, dxa, fma2(dya, dya, E2)), db = fma2(dxb, dxb, fma2(dyb, dyb, E2));
        const float2 ta = mul2(da, TH), tb = mul2(db, TH);
        const bool ok[4] = {!valid || q0.w <= ta.x, !valid || q1.w <= ta.y, !valid || q2.w <= tb.x,
                            !valid || q3.w <= tb.y};
        const uint32_t sk0 = sk[0], sk1 = sk[1], sk2 = sk[2], sk3 = sk[3];
        const uint32_t left = T - ind;
        if (left >= 4u && (sk0 | sk1 | sk2) == 1u && __all_sync(0xffffffffu, ok[0] && ok[1] && ok[2] && ok[3])) {
            const float2 ra = make_float2(rule_inv_sqrt<EXACT, FTZ>(da.x), rule_inv_sqrt<EXACT, FTZ>(da.y));
            const float2 rb = make_float2(rule_inv_sqrt<EXACT, FTZ>(db.x), rule_inv_sqrt<EXACT, FTZ>(db.y));
            const float2 sa = mul2(mul2(mul2(make_float2(q0.z, q1.z), ra), ra), ra);
            const float2 sb = mul2(mul2(mul2(make_float2(q2.z, q3.z), rb), rb), rb);
            ax = fmaf(dxa.x, sa.x, ax);
            ay = fmaf(dya.x, sa.x, ay);
            ax = fmaf(dxa.y, sa.y, ax);
            ay = fmaf(dya.y, sa.y, ay);
            ax = fmaf(dxb.x, sb.x, ax);
            ay = fmaf(dyb.x, sb.x, ay);
            ax = fmaf(dxb.y, sb.y, ax);
            ay = fmaf(dyb.y, sb.y, ay);
            if (COUNT) {
                n_vis += 4;
                n_acc += valid ? 4 : 0;
            }
            ind += 3u + max(sk3, 1u);
            continue;
        }
        const float qm[4] = {q0.z, q1.z, q2.z, q3.z}, dd[4] = {da.x, da.y, db.x, db.y};
        const float dx[4] = {dxa.x, dxa.y, dxb.x, dxb.y}, dy[4] = {dya.x, dya.y, dyb.x, dyb.y};
        const uint32_t sks[4] = {sk0, sk1, sk2, sk3};
        uint32_t used = 0;
        uint32_t next = 0;  // the next record of the rule's walk, from ind
#pragma unroll
        for (uint32_t t = 0; t < 4; ++t) {
            if (next != t || t >= left) continue;  // uniform
            ++used;
            if (COUNT) ++n_vis;
            if (__all_sync(0xffffffffu, ok[t])) {
                const float r = rule_inv_sqrt<EXACT, FTZ>(dd[t]);
                const float sc = ((qm[t] * r) * r) * r;
                ax = fmaf(dx[t], sc, ax);
                ay = fmaf(dy[t], sc, ay);
                if (COUNT) n_acc += valid;
                next += max(sks[t], 1u);
            } else {
                ++next;
            }
        }
        ind += next;
        single = used <= 3u && next > used;
    }
    if (COUNT) {
        for (int o = 16; o; o >>= 1) n_acc += __shfl_xor_sync(0xffffffffu, n_acc, o);
        if (lane == 0) {
            atomicAdd(&stat[0], n_acc);
            atomicAdd(&stat[1], n_vis);
        }
    }
    float2 np = make_float2(0.0f, 0.0f);
    if (valid) {
        if (acc_rec) acc_rec[i] = make_float2(ax, ay);
        const float2 v = vel_in[i];
        const float nvx = fmaf(ax, k, v.x), nvy = fmaf(ay, k, v.y);  // ForceShader.comp:145-146
        np = make_float2(fmaf(v.x + nvx, hdt, p.x), fmaf(v.y + nvy, hdt, p.y));
        pos_out[i] = np;
        vel_out[i] = make_float2(nvx, nvy);
    }
    if (ext)  // bounding-box mode: the next step's box
        ext_add(ext, valid ? np.x : INFINITY, valid ? np.x : -INFINITY, valid ? np.y : INFINITY,
                valid ? np.y : -INFINITY);
}

template <bool EXACT, bool COUNT, bool FTZ>
__global__ void __launch_bounds__(kForceWarps * 32)
k_force(const uint32_t* __restrict__ sidx, const uint32_t* __restrict__ counts, const float4* __restrict__ rec,
        const uint32_t* __restrict__ skip, const float2* __restrict__ pos_in, const float2* __restrict__ vel_in,
        float2* __restrict__ pos_out, float2* __restrict__ vel_out, float2* __restrict__ acc_rec, uint32_t n_al,
        float eps2, float theta2, float k, float hdt, uint32_t cap, unsigned long long* __restrict__ stat,
        uint32_t* __restrict__ ext) {
    __shared__ RuleWindow win[kForceWarps];
    pdl_enter();
    force_body<EXACT, COUNT, FTZ, false>(grid_blk(), &win[threadIdx.x >> 5], nullptr, nullptr, sidx, counts, rec, skip,
                                         pos_in, vel_in, pos_out, vel_out, acc_rec, n_al, eps2, theta2, k, hdt, cap,
                                         stat, ext);
}

// Small systems: fewer blocks than SMs, so every walk's latency counts, and a window reload
// per accepted node is an L2 round trip (N = 3000: 36 us for some 150 visits a warp).  Each
// block first copies the whole tree into its shared memory; a tree that does not fit
// (kRuleStage records) is walked through windows as above.
constexpr uint32_t kRuleStage = 10240;           // records: 200 KB of records and skips
constexpr uint32_t kRuleStagedMax = 1u << 13;    // particles; one block per SM at most
struct RuleTree {
    float4 rec[kRuleStage + 8];
    uint32_t skip[kRuleStage + 8];
};

template <bool EXACT, bool COUNT, bool FTZ>
__global__ void __launch_bounds__(kForceWarps * 32)
k_force_staged(const uint32_t* __restrict__ sidx, const uint32_t* __restrict__ counts, const float4* __restrict__ rec,
               const uint32_t* __restrict__ skip, const float2* __restrict__ pos_in,
               const float2* __restrict__ vel_in, float2* __restrict__ pos_out, float2* __restrict__ vel_out,
               float2* __restrict__ acc_rec, uint32_t n_al, float eps2, float theta2, float k, float hdt, uint32_t cap,
               unsigned long long* __restrict__ stat, uint32_t* __restrict__ ext) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    RuleTree& tree = *reinterpret_cast<RuleTree*>(s_raw);
    pdl_enter();
    const uint32_t T = min(counts[0] + counts[1], cap);
    if (T > kRuleStage) {
        force_body<EXACT, COUNT, FTZ, false>(grid_blk(), reinterpret_cast<RuleWindow*>(s_raw) + (threadIdx.x >> 5),
                                             nullptr, nullptr, sidx, counts, rec, skip, pos_in, vel_in, pos_out,
                                             vel_out, acc_rec, n_al, eps2, theta2, k, hdt, cap, stat, ext);
        return;
    }
    // the last four-record round reads up to three records past the end (the arrays hold
    // cap + 32); they never enter a sum
    const uint32_t rows = (T + 3 + 3) & ~3u;
    for (uint32_t r = threadIdx.x; r < rows; r += kForceWarps * 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(&tree.rec[r])),
                     "l"(rec + r)
                     : "memory");
    for (uint32_t r = 4 * threadIdx.x; r < rows; r += 4 * kForceWarps * 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(&tree.skip[r])),
                     "l"(skip + r)
                     : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    force_body<EXACT, COUNT, FTZ, true>(grid_blk(), nullptr, tree.rec, tree.skip, sidx, counts, rec, skip, pos_in,
                                        vel_in, pos_out, vel_out, acc_rec, n_al, eps2, theta2, k, hdt, cap, stat, ext);
}

// ------------------------------------------------------------------------------------
// accurate-mode traversal (no counterpart in the reference): the 64 particles of 64
// consecutive sorted slots share one walk: 32 records are tested at once (one per lane)
// against the bounding boxes of the group; accepted nodes and runs of particle leaves are
// collected, and every lane sums them for its two particles with packed f32x2 instructions
// (quadrupole term for nodes).
//
// One warp does both (SPLIT false), or two share a group: a walking warp that tests and
// collects, and a summing warp, the lists going from one to the other through two slots in
// shared memory.  One warp spends half its time in each: at N = 20,000, where a scheduler
// has at most one warp, 46 of 103 thousand cycles a group in the walk's chain of L2 round trips
// and 53 in the sums' dependent instructions; on two warps the halves overlap.
// ------------------------------------------------------------------------------------
// Records still to test.  Pops take the top 32 and push at most four internal children
// each, one level deeper, so the stack holds at most one block of <= 128 entries per level
// and blocks of strictly increasing level: <= 96 * D + 128 = 1568 for D = 15 (checked and
// reported).  The walks of a 500k-particle spiral stay below 230, so shared memory holds the
// top 256 entries and a deeper stack's bottom goes to the walking warp's local memory, 128
// entries at a time.
constexpr int kStackCap = 1568;
static_assert(kStackCap >= 96 * (kBBoxMaxBits > kFixedDepth ? kBBoxMaxBits : kFixedDepth) + 128, "walk stack bound");
constexpr int kStackWindow = 256, kStackSpill = 128;          // of a walk
constexpr int kPairStackWindow = 512, kPairStackSpill = 256;  // of a costly group's (64-record pops)
constexpr int kSinglePerSm = 20, kSplitPerSm = 8;  // resident groups the registers are cut for

// The bottom of a stack that outgrew its window: lane l keeps entries l, 32 + l, ...
template <int CAP, int SPILL>
struct StackSpill {
    uint32_t e[(CAP + SPILL - 1) / SPILL * SPILL / 32];
    uint32_t count = 0;  // entries below the window

    // Moves the window's lowest SPILL entries out (size > SPILL of them).
    __device__ __forceinline__ uint32_t save(uint32_t* stack, uint32_t size, int lane) {
        for (uint32_t j = 0; j < SPILL; j += 32) e[(count + j) / 32] = stack[j + lane];
        for (uint32_t j = SPILL; j < size; j += 32) {  // upwards: a row's target lies below it
            const uint32_t v = j + lane < size ? stack[j + lane] : 0u;
            __syncwarp();
            if (j + lane < size) stack[j + lane - SPILL] = v;
            __syncwarp();
        }
        count += SPILL;
        return size - SPILL;
    }
    // Moves them back below the size entries of the window (size <= 64).
    __device__ __forceinline__ uint32_t restore(uint32_t* stack, uint32_t size, int lane) {
        const uint32_t v0 = (uint32_t)lane < size ? stack[lane] : 0u, v1 = lane + 32u < size ? stack[lane + 32] : 0u;
        __syncwarp();
        count -= SPILL;
        if ((uint32_t)lane < size) stack[SPILL + lane] = v0;
        if (lane + 32u < size) stack[SPILL + 32 + lane] = v1;
        for (uint32_t j = 0; j < SPILL; j += 32) stack[j + lane] = e[(count + j) / 32];
        __syncwarp();
        return size + SPILL;
    }
};

// Evaluation order.  Each particle sums the accepted nodes and the particle leaves of its
// walk separately, each in walk order, into a node and a leaf accumulator; its
// acceleration is node + leaf.  How the lists are cut into slots therefore does not change
// a bit of the result.
//
// A walk's lists are summed (SPLIT: passed on) once they hold NODE nodes or ITEM leaf runs (a
// pop adds at most 32 nodes and 64 runs).
template <int NODE, int ITEM, int SLOTS>
struct GroupSmem {
    static constexpr int kFullNode = NODE, kFullItem = ITEM, kNode = NODE + 32, kItem = (ITEM + 64 + 31) / 32 * 32;
    static constexpr bool kSplit = SLOTS == 2;
    static_assert(kItem % 32 == 0, "whole rows of runs");
    uint32_t stack[kStackWindow];
    struct Slot {
        uint32_t node[kNode];   // accepted node records
        uint2 run[kItem];       // runs of particle leaves: first record, count
        uint32_t nodes, runs, last;
    } slot[SLOTS];
    uint64_t full[2], empty[2];  // SPLIT: mbarriers of the slots
    uint32_t off[kItem];        // exclusive record offsets of a slot's runs
    // One chunk of gathered records: {x, y, m, -1.5 tr(S)}, 7.5 {Sxx, Sxy, Syy}.  A scalar
    // of a record costs one register move to pair it for the two particles; stored as
    // pairs it would cost a broadcast load's bandwidth, which goes by the bytes delivered.
    float4 ca[32], cb[32];
};

// The two warps of a walk hand slots over through mbarriers in shared memory (full and empty
// again, one arrival each).  Named barriers would do the same, but an SM has 64 of them,
// and sixteen walks with four each (or a block that reserves all sixteen ids because they
// are computed) leave no room: 14 of 32 warps resident, 360 us at N = 500,000.
__device__ __forceinline__ uint32_t bar_address(const uint64_t& bar) { return (uint32_t)__cvta_generic_to_shared(&bar); }
__device__ __forceinline__ void bar_init(uint64_t& bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_address(bar)) : "memory");
}
// The warp's earlier reads and writes of the slot come before the other side's.
__device__ __forceinline__ void bar_pass(uint64_t& bar, int lane) {
    __syncwarp();
    if (lane == 0)
        asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.release.cta.shared::cta.b64 t, [%0];\n\t}" ::"r"(bar_address(bar))
                     : "memory");
}
// Waits for the arrival that ends phase `parity`; false after kSpinLimit tries.
__device__ __forceinline__ bool bar_wait(const uint64_t& bar, uint32_t parity) {
    uint32_t done = 0;
    for (uint32_t spin = 0; !done && spin < kSpinLimit; ++spin)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(bar_address(bar)), "r"(parity)
                     : "memory");
    return __all_sync(0xffffffffu, done != 0);
}

// Barrier of a walk's two warps (a named one, by a constant so that a block reserves no more
// than its walks need).
__device__ __forceinline__ void pair_sync(int walk) {
    if (walk == 0) asm volatile("bar.sync 1, 64;" ::: "memory");
    else if (walk == 1) asm volatile("bar.sync 2, 64;" ::: "memory");
    else if (walk == 2) asm volatile("bar.sync 3, 64;" ::: "memory");
    else asm volatile("bar.sync 4, 64;" ::: "memory");
}

// One record (x, y, m) on the lane's two particles (P = their x, Q = their y):
// d = (x, y) - p, d2 = dx^2 + dy^2 + eps^2, a += d * (((m r) r) r) with r = 1/sqrt(d2),
// the CPU restatement's pair_scale sequence, two particles at once.
template <bool EXACT>
__device__ __forceinline__ void monopole_x2(float x, float y, float m, float2 P, float2 Q, float2 E2, float2& acx,
                                            float2& acy) {
    const float2 dx = sub2(make_float2(x, x), P), dy = sub2(make_float2(y, y), Q);
    const float2 d2 = fma2(dx, dx, fma2(dy, dy, E2));
    const float2 r = make_float2(inv_sqrt<EXACT>(d2.x), inv_sqrt<EXACT>(d2.y));
    const float2 sc = mul2(mul2(mul2(make_float2(m, m), r), r), r);
    acx = fma2(dx, sc, acx);
    acy = fma2(dy, sc, acy);
}

// One node with second moments on the lane's two particles.  The monopole and
// quadrupole terms of the softened potential,
//   a = d (m r^3 - 1.5 tr(S) r^5 + 7.5 (d.S.d) r^7) - 3 r^5 S d,   r = 1/sqrt(d2),
// are evaluated as r^3 (d (m + r^2 (mt + r^2 u)) - 0.4 r^2 S'' d) with the node terms
// S'' = 7.5 S and mt = -1.5 tr(S) formed once per node (eval_nodes): 21 operations per
// particle instead of 23, the CPU restatement's sequence (quad_accumulate).
template <bool EXACT>
__device__ __forceinline__ void quadrupole_x2(float x, float y, float m, float qxx, float qxy, float qyy, float mt,
                                              float2 P, float2 Q, float2 E2, float2& acx, float2& acy) {
    const float2 dx = sub2(make_float2(x, x), P), dy = sub2(make_float2(y, y), Q);
    const float2 d2 = fma2(dx, dx, fma2(dy, dy, E2));
    const float2 r = make_float2(inv_sqrt<EXACT>(d2.x), inv_sqrt<EXACT>(d2.y));
    const float2 r2 = mul2(r, r);
    const float2 r3 = mul2(r2, r);
    const float2 Sxx = make_float2(qxx, qxx), Sxy = make_float2(qxy, qxy), Syy = make_float2(qyy, qyy);
    const float2 srx = fma2(Sxx, dx, mul2(Sxy, dy));
    const float2 sry = fma2(Sxy, dx, mul2(Syy, dy));
    const float2 u = fma2(dx, srx, mul2(dy, sry));
    const float2 t = fma2(fma2(u, r2, make_float2(mt, mt)), r2, make_float2(m, m));
    const float2 k = mul2(make_float2(-0.4f, -0.4f), r2);
    const float2 ix = fma2(srx, k, mul2(dx, t));
    const float2 iy = fma2(sry, k, mul2(dy, t));
    acx = fma2(r3, ix, acx);
    acy = fma2(r3, iy, acy);
}

// A gathered node's record and moments as a chunk's entry.
template <bool QUAD>
__device__ __forceinline__ void stage_node(float4* ca, float4* cb, int lane, const float4& q, const float4& qq) {
    ca[lane] = make_float4(q.x, q.y, q.z, QUAD ? -1.5f * (qq.x + qq.z) : 0.0f);
    if (QUAD) cb[lane] = make_float4(7.5f * qq.x, 7.5f * qq.y, 7.5f * qq.z, 0.0f);
}
// Entries [klo, khi) of a chunk on the lane's two particles.
template <bool EXACT, bool QUAD>
__device__ __forceinline__ void sum_chunk(const float4* ca, const float4* cb, uint32_t klo, uint32_t khi, float2 P,
                                          float2 Q, float2 E2, float2& acx, float2& acy) {
#pragma unroll 4
    for (uint32_t j = klo; j < khi; ++j) {
        const float4 a = ca[j];
        if (QUAD) {
            const float4 b = cb[j];
            quadrupole_x2<EXACT>(a.x, a.y, a.z, b.x, b.y, b.z, a.w, P, Q, E2, acx, acy);
        } else {
            monopole_x2<EXACT>(a.x, a.y, a.z, P, Q, E2, acx, acy);
        }
    }
}

// Sum the count accepted nodes (quadrupole term with QUAD) for the lane's two particles,
// 32 at a time: lane l loads node l of the next chunk while the current one is summed.
template <bool EXACT, bool QUAD>
__device__ __forceinline__ void eval_nodes(const uint32_t* node, float4* ca, float4* cb, uint32_t count,
                                           const float4* __restrict__ rec, const float4* __restrict__ quad, float2 P,
                                           float2 Q, float2 E2, float2& acx, float2& acy, int lane) {
    if (!count) return;
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f), qq = q;
    if ((uint32_t)lane < count) {
        const uint32_t r = node[lane];
        q = __ldg(&rec[r]);
        if (QUAD) qq = __ldg(&quad[r]);
    }
    for (uint32_t f0 = 0; f0 < count; f0 += 32) {
        __syncwarp();
        stage_node<QUAD>(ca, cb, lane, q, qq);
        __syncwarp();
        const uint32_t fn = f0 + 32 + lane;
        if (fn < count) {
            const uint32_t r = node[fn];
            q = __ldg(&rec[r]);
            if (QUAD) qq = __ldg(&quad[r]);
        }
        sum_chunk<EXACT, QUAD>(ca, cb, 0, min(count - f0, 32u), P, Q, E2, acx, acy);
    }
}

// Exclusive record offsets of n_items leaf runs, and their total: lane l owns runs
// [K l, K l + K).
template <int K>
__device__ __forceinline__ uint32_t run_offsets(const uint2* run, uint32_t* off, uint32_t n_items, int lane) {
    uint32_t cnt[K], sum = 0;
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const uint32_t it = (uint32_t)lane * K + t;
        cnt[t] = it < n_items ? run[it].y : 0u;
        sum += cnt[t];
    }
    uint32_t x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    uint32_t at = x - sum;
#pragma unroll
    for (int t = 0; t < K; ++t) {
        off[lane * K + t] = at;
        at += cnt[t];
    }
    return __shfl_sync(0xffffffffu, x, 31);
}

// Record f0 + lane of the flattened leaf runs (if below total); r0 is the run that holds
// record f0, and is moved on to the one that holds f0 + 32.  The runs that start inside
// the chunk mark a bit each, and a lane's run is r0 plus the marks up to it.
__device__ __forceinline__ float4 gather_leaf(const uint2* run, const uint32_t* off, uint32_t n_items, uint32_t f0,
                                              uint32_t total, uint32_t& r0, const float4* __restrict__ rec, int lane) {
    const uint32_t r = r0 + 1 + lane, o = r < n_items ? off[r] : 0xffffffffu;
    const uint32_t marks = __reduce_or_sync(0xffffffffu, o - f0 < 32u ? 1u << (o - f0) : 0u);
    const uint32_t mine = r0 + __popc(marks & (0xffffffffu >> (31 - lane)));
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (f0 + lane < total) q = __ldg(&rec[run[mine].x + (f0 + lane - off[mine])]);
    r0 += __popc(marks);
    if (r0 + 1 < n_items && off[r0 + 1] == f0 + 32) ++r0;
    return q;
}

// Sum the particle leaves of the n_items runs as monopoles, 32 records at a time.
template <bool EXACT, int ITEM>
__device__ __forceinline__ void eval_leaves(const uint2* run, uint32_t* off, float4* ca, uint32_t n_items,
                                            const float4* __restrict__ rec, float2 P, float2 Q, float2 E2, float2& acx,
                                            float2& acy, int lane) {
    if (!n_items) return;
    __syncwarp();  // the previous slot's offsets have been read
    const uint32_t total = run_offsets<ITEM / 32>(run, off, n_items, lane);
    __syncwarp();
    uint32_t r0 = 0;
    float4 q = gather_leaf(run, off, n_items, 0, total, r0, rec, lane);
    for (uint32_t f0 = 0; f0 < total; f0 += 32) {
        __syncwarp();
        ca[lane] = q;
        __syncwarp();
        if (f0 + 32 < total) q = gather_leaf(run, off, n_items, f0 + 32, total, r0, rec, lane);
        sum_chunk<EXACT, false>(ca, nullptr, 0, min(total - f0, 32u), P, Q, E2, acx, acy);
    }
}

// The end of a group's walk: |a| for the relative criterion, then (main pass) the
// integrator and the new positions' extent.  ax, ay: node + leaf per particle (.x particle
// 0, .y particle 1).  Every lane of the warp must call it.
template <bool ESTIMATE>
__device__ __forceinline__ void group_finish(float2 ax, float2 ay, bool v0, bool v1, uint32_t i0, uint32_t i1,
                                             float2 p0, float2 p1, const float2* __restrict__ vel_in,
                                             float2* __restrict__ pos_out, float2* __restrict__ vel_out,
                                             float2* __restrict__ acc_rec, float k, float hdt,
                                             float* __restrict__ amag, uint32_t* __restrict__ ext) {
    if (amag) {
        if (v0) amag[i0] = __fsqrt_rn(fmaf(ax.x, ax.x, ay.x * ay.x));
        if (v1) amag[i1] = __fsqrt_rn(fmaf(ax.y, ax.y, ay.y * ay.y));
    }
    if (ESTIMATE) return;
    float mnx = INFINITY, mxx = -INFINITY, mny = INFINITY, mxy = -INFINITY;  // of the new positions
    if (v0) {
        if (acc_rec) acc_rec[i0] = make_float2(ax.x, ay.x);
        const float2 v = vel_in[i0];
        const float nvx = fmaf(ax.x, k, v.x), nvy = fmaf(ay.x, k, v.y);
        const float2 np = make_float2(fmaf(v.x + nvx, hdt, p0.x), fmaf(v.y + nvy, hdt, p0.y));
        pos_out[i0] = np;
        vel_out[i0] = make_float2(nvx, nvy);
        mnx = fminf(mnx, np.x);
        mxx = fmaxf(mxx, np.x);
        mny = fminf(mny, np.y);
        mxy = fmaxf(mxy, np.y);
    }
    if (v1) {
        if (acc_rec) acc_rec[i1] = make_float2(ax.y, ay.y);
        const float2 v = vel_in[i1];
        const float nvx = fmaf(ax.y, k, v.x), nvy = fmaf(ay.y, k, v.y);
        const float2 np = make_float2(fmaf(v.x + nvx, hdt, p1.x), fmaf(v.y + nvy, hdt, p1.y));
        pos_out[i1] = np;
        vel_out[i1] = make_float2(nvx, nvy);
        mnx = fminf(mnx, np.x);
        mxx = fmaxf(mxx, np.x);
        mny = fminf(mny, np.y);
        mxy = fmaxf(mxy, np.y);
    }
    if (ext) ext_add(ext, mnx, mxx, mny, mxy);  // bounding-box mode: the next step's box
}

// The outcome of testing one stacked record (an internal node) against a group's boxes:
// accepted (nn = 1), or opened into at most two runs of particle leaves {a, c} and at most
// four internal children to push, in Morton order.
struct RecTest {
    uint32_t nn, nl, a0, c0, a1, c1, npu;
    uint32_t pu[4];
};

__device__ __forceinline__ void test_record(uint32_t n, const float4* __restrict__ rec, const uint4* __restrict__ kids,
                                            const float* bx0, const float* bx1, const float* by0, const float* by1,
                                            float eps2, bool relative, float tol2, float floor2, float theta2,
                                            RecTest& r) {
    const float4 q = rec[n];
    const uint4 kd = kids[n];
    float d2 = INFINITY;  // nearest sub-box; an empty one gives +inf
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const float ex = fmaxf(fmaxf(bx0[b] - q.x, q.x - bx1[b]), 0.0f);
        const float ey = fmaxf(fmaxf(by0[b] - q.y, q.y - by1[b]), 0.0f);
        d2 = fminf(d2, fmaf(ex, ex, fmaf(ey, ey, eps2)));
    }
    bool accept;
    if (relative) {  // m^2 R^3 <= tol^2 D^5 with R <= D (R: squared opening radius), or theta
        const float lhs = (q.z * q.z) * ((q.w * q.w) * q.w);
        const float d4 = d2 * d2;
        accept = (q.w <= d2 && lhs <= tol2 * ((d4 * d4) * d2)) || q.w <= d2 * floor2;
    } else {
        accept = q.w <= d2 * theta2;
    }
    if (accept) {
        r.nn = 1;
    } else if (kd.x == kKidFinest) {
        r.a0 = kd.y;
        r.c0 = kd.z;
        r.nl = 1;
    } else {
        const uint32_t kk[4] = {kd.x, kd.y, kd.z, kd.w};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t c = kk[t];
            if (c == kKidNone) continue;
            if (c & kKidLeaf) {
                const uint32_t l = c & ~kKidLeaf;
                if (r.nl == 1 && r.a0 + r.c0 == l) ++r.c0;        // extend the open run
                else if (r.nl == 2 && r.a1 + r.c1 == l) ++r.c1;
                else if (r.nl == 0) { r.a0 = l; r.c0 = 1; r.nl = 1; }
                else { r.a1 = l; r.c1 = 1; r.nl = 2; }
            } else {
                if (r.npu == 0) r.pu[0] = c;
                else if (r.npu == 1) r.pu[1] = c;
                else if (r.npu == 2) r.pu[2] = c;
                else r.pu[3] = c;
                ++r.npu;
            }
        }
    }
}

// Sub-boxes of a group: the particles are split by their cell at the coarsest level where
// the first and last keys of the group differ, so a group that crosses a coarse Morton
// boundary is not given one box spanning the empty space between its ends.  Each box is
// the bounding box of its particles (+inf..-inf when empty).  Every lane must call it.
__device__ __forceinline__ void group_boxes(const uint32_t* __restrict__ skey, uint32_t g0, uint32_t nv, uint32_t s0,
                                            uint32_t s1, bool v0, bool v1, float2 p0, float2 p1, float* bx0,
                                            float* bx1, float* by0, float* by1) {
    const uint32_t kf = skey[g0], kl = skey[min(g0 + kGroupSize - 1, nv - 1)];
    const int shift = kf == kl ? -1 : ((31 - __clz(kf ^ kl)) & ~1);
    const int box0 = !v0 ? -1 : (shift < 0 ? 0 : (int)((skey[s0] >> shift) & 3u));
    const int box1 = !v1 ? -1 : (shift < 0 ? 0 : (int)((skey[s1] >> shift) & 3u));
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const bool in0 = box0 == b, in1 = box1 == b;
        float x0 = fminf(in0 ? p0.x : INFINITY, in1 ? p1.x : INFINITY);
        float x1 = fmaxf(in0 ? p0.x : -INFINITY, in1 ? p1.x : -INFINITY);
        float y0 = fminf(in0 ? p0.y : INFINITY, in1 ? p1.y : INFINITY);
        float y1 = fmaxf(in0 ? p0.y : -INFINITY, in1 ? p1.y : -INFINITY);
        for (int o = 16; o; o >>= 1) {
            x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
            y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
            y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
        }
        bx0[b] = x0;
        bx1[b] = x1;
        by0[b] = y0;
        by1[b] = y1;
    }
}

// What a group's two warps read of its system.
struct GroupSys {
    const uint32_t *sidx, *skey, *counts;
    const float4* rec;
    const uint32_t* skip;
    const float4* quad;
    const uint4* kids;
    const float2 *pos_in, *vel_in;
    float2 *pos_out, *vel_out, *acc_rec;
    uint32_t n_al;
    float eps2, theta2, k, hdt;
    uint32_t cap;
    unsigned long long* stat;
    int* err;
    float* amag;
    float alpha, floor2;
    uint32_t* ext;
    const uint8_t* heavy;
    uint32_t tail = 0xffffffffu;  // blocks from here on take one group on both warps (WalkShape MIXED)
};

// The walk of a group: tests the records; flush(slot, nodes, runs, done) takes the lists,
// slot by slot, and leaves the next slot free (false: a wait ran out).
template <bool COUNT, bool ESTIMATE, class SM, class Flush>
__device__ __forceinline__ bool group_walk(const GroupSys& y, SM& g, uint32_t nv, uint32_t g0, uint32_t s0,
                                           uint32_t s1, bool v0, bool v1, float2 p0, float2 p1, bool unknown, float a0,
                                           float a1, int lane, Flush&& flush) {
    const float4* __restrict__ rec = y.rec;
    const uint4* __restrict__ kids = y.kids;
    float bx0[4], bx1[4], by0[4], by1[4];
    group_boxes(y.skey, g0, nv, s0, s1, v0, v1, p0, p1, bx0, bx1, by0, by1);
    // Relative criterion: the smallest previous |a| of the group (when any is unknown the
    // group takes the theta test).  Each group reads and rewrites only its own particles'
    // |a|, so one buffer serves as input and output.
    bool relative = false;
    float tol2 = 0.0f;
    if (y.amag) {
        float amin = fminf(a0, a1);
        for (int o = 16; o; o >>= 1) amin = fminf(amin, __shfl_xor_sync(0xffffffffu, amin, o));
        relative = !ESTIMATE && !unknown;
        const float tol = y.alpha * amin;
        tol2 = tol * tol;
    }
    const float eps2 = y.eps2, floor2 = y.floor2, theta2 = y.theta2;
    unsigned long long n_int = 0, n_test = 0, n_node = 0;
    StackSpill<kStackCap, kStackSpill> spill;
    uint32_t size = 0, n_nodes = 0, n_items = 0, passed = 0;  // slots passed on
    const bool single = y.skip[0] == 1u;  // a single particle: the root is its leaf
    if (single) {
        if (lane == 0) g.slot[0].run[0] = make_uint2(0u, 1u);
        n_items = 1;
    } else {
        if (lane == 0) g.stack[0] = 0u;
        size = 1;
    }
    __syncwarp();
    const uint32_t lt = (1u << lane) - 1u;
    for (;;) {
        const bool done = size == 0 && spill.count == 0;
        if (done || n_nodes > (uint32_t)SM::kFullNode || n_items > (uint32_t)SM::kFullItem) {
            if (!flush(passed & 1u, n_nodes, n_items, done)) return false;
            ++passed;
            n_nodes = n_items = 0;
            if (done) break;
        }
        if (size < 32u && spill.count) size = spill.restore(g.stack, size, lane);
        typename SM::Slot& sl = g.slot[SM::kSplit ? passed & 1u : 0u];
        const uint32_t np = min(size, 32u);
        const uint32_t base = size - np;
        const bool act = lane < (int)np;
        const uint32_t n = act ? g.stack[base + lane] : 0u;
        __syncwarp();
        size = base;
        if (COUNT) n_test += np;
        RecTest r{};
        if (act) test_record(n, rec, kids, bx0, bx1, by0, by1, eps2, relative, tol2, floor2, theta2, r);
        // offsets in lane order from the ballots of the counts' bits: nodes 0..1, runs 0..2,
        // pushes 0..4
        const uint32_t bn = __ballot_sync(0xffffffffu, r.nn);
        const uint32_t bl0 = __ballot_sync(0xffffffffu, r.nl & 1u), bl1 = __ballot_sync(0xffffffffu, r.nl & 2u);
        const uint32_t bp0 = __ballot_sync(0xffffffffu, r.npu & 1u), bp1 = __ballot_sync(0xffffffffu, r.npu & 2u);
        const uint32_t bp2 = __ballot_sync(0xffffffffu, r.npu & 4u);
        const uint32_t ptot = __popc(bp0) + 2 * __popc(bp1) + 4 * __popc(bp2);
        if (size + ptot > (uint32_t)kStackWindow) size = spill.save(g.stack, size, lane);
        uint32_t npu = r.npu, pushed = ptot;
        if (spill.count + size + ptot > (uint32_t)kStackCap) {  // beyond the depth bound: report, do not overrun
            if (lane == 0) atomicOr(y.err, kErrTree);
            pushed = npu = 0;
        }
        if (r.nn) sl.node[n_nodes + __popc(bn & lt)] = n;
        if (r.nl) {
            uint2* run = sl.run + n_items + __popc(bl0 & lt) + 2 * __popc(bl1 & lt);
            run[0] = make_uint2(r.a0, r.c0);
            if (r.nl > 1) run[1] = make_uint2(r.a1, r.c1);
        }
        if (COUNT) {
            n_int += r.nn + (r.nl > 0 ? r.c0 : 0u) + (r.nl > 1 ? r.c1 : 0u);
            n_node += r.nn;
        }
        uint32_t* dst = g.stack + size + __popc(bp0 & lt) + 2 * __popc(bp1 & lt) + 4 * __popc(bp2 & lt);
        if (npu > 0) dst[0] = r.pu[0];
        if (npu > 1) dst[1] = r.pu[1];
        if (npu > 2) dst[2] = r.pu[2];
        if (npu > 3) dst[3] = r.pu[3];
        n_nodes += __popc(bn);
        n_items += __popc(bl0) + 2 * __popc(bl1);
        size += pushed;
        __syncwarp();
    }
    if (COUNT) {
        if (single && lane == 0) n_int += 1;
        for (int o = 16; o; o >>= 1) {
            n_int += __shfl_xor_sync(0xffffffffu, n_int, o);
            n_node += __shfl_xor_sync(0xffffffffu, n_node, o);
        }
        const unsigned long long nval = __popc(__ballot_sync(0xffffffffu, v0)) + __popc(__ballot_sync(0xffffffffu, v1));
        if (lane == 0) {
            atomicAdd(&y.stat[0], n_int * nval);
            atomicAdd(&y.stat[1], n_test);
            atomicAdd(&y.stat[2], n_node * nval);
        }
    }
    return true;
}

// The lists of one slot on the lane's two particles.
template <bool EXACT, bool QUAD, class SM>
__device__ __forceinline__ void sum_slot(const GroupSys& y, SM& g, const typename SM::Slot& sl, uint32_t nodes,
                                         uint32_t runs, float2 P, float2 Q, float2 E2, float2& anx, float2& any,
                                         float2& alx, float2& aly, int lane) {
    eval_nodes<EXACT, QUAD>(sl.node, g.ca, g.cb, nodes, y.rec, y.quad, P, Q, E2, anx, any, lane);
    eval_leaves<EXACT, SM::kItem>(sl.run, g.off, g.ca, runs, y.rec, P, Q, E2, alx, aly, lane);
}

// One group, on one warp or (SPLIT) two: `walker` says which of the two this is, `phase` holds
// this warp's phases of the slots' barriers.  False if a wait on the other warp ran out.
// ESTIMATE: the |a| estimate pass of the relative criterion.  A group whose particles all
// have a previous |a| returns at once; any other group walks with the theta test and
// writes only the |a| of its particles (no integration), which the following normal pass
// then opens nodes by.
template <bool EXACT, bool QUAD, bool COUNT, bool ESTIMATE, class SM>
__device__ __forceinline__ bool force_group_body(const GroupSys& y, uint32_t group, bool walker, uint32_t& phase, SM& g) {
    const int lane = threadIdx.x & 31;
    const uint32_t nv = y.counts[0];
    const uint32_t T = min(nv + y.counts[1], y.cap);
    const uint32_t g0 = group * kGroupSize;
    if (g0 >= nv || T == 0) return true;
    if (ESTIMATE && !y.amag) return true;  // a batch member without the relative criterion
    if (y.heavy && y.heavy[group]) return true;  // a costly group: walked by a warp pair (force_pair_body)
    // particles: slot g0 + lane (.x of every pair) and g0 + 32 + lane (.y)
    const uint32_t s0 = g0 + lane, s1 = s0 + 32;
    const uint32_t i0 = s0 < nv ? y.sidx[s0] : 0u, i1 = s1 < nv ? y.sidx[s1] : 0u;
    const bool v0 = s0 < nv && i0 < y.n_al, v1 = s1 < nv && i1 < y.n_al;  // i < n_al unless the sort failed
    const float2 p0 = v0 ? y.pos_in[i0] : make_float2(0.0f, 0.0f);
    const float2 p1 = v1 ? y.pos_in[i1] : make_float2(0.0f, 0.0f);
    bool unknown = false;
    float a0 = INFINITY, a1 = INFINITY;
    if (y.amag && (walker || ESTIMATE)) {  // |a| is rewritten only after the walk
        a0 = v0 ? y.amag[i0] : INFINITY;
        a1 = v1 ? y.amag[i1] : INFINITY;
        unknown = __any_sync(0xffffffffu, isnan(a0) || isnan(a1));
        if (ESTIMATE && !unknown) return true;  // the same in both warps: nothing to estimate
    }
    const float2 P = make_float2(p0.x, p1.x), Q = make_float2(p0.y, p1.y), E2 = make_float2(y.eps2, y.eps2);
    // node and leaf accumulators of the two particles (.x particle 0, .y particle 1)
    float2 anx = make_float2(0.0f, 0.0f), any = anx, alx = anx, aly = anx;
    bool ok = true;
    if (!SM::kSplit) {
        group_walk<COUNT, ESTIMATE>(y, g, nv, g0, s0, s1, v0, v1, p0, p1, unknown, a0, a1, lane,
                                    [&](uint32_t, uint32_t nodes, uint32_t runs, bool) {
                                        sum_slot<EXACT, QUAD>(y, g, g.slot[0], nodes, runs, P, Q, E2, anx, any, alx,
                                                              aly, lane);
                                        __syncwarp();  // the lists have been read
                                        return true;
                                    });
    } else if (walker) {
        uint32_t passed = 0;
        ok = group_walk<COUNT, ESTIMATE>(y, g, nv, g0, s0, s1, v0, v1, p0, p1, unknown, a0, a1, lane,
                                         [&](uint32_t b, uint32_t nodes, uint32_t runs, bool done) {
                                             if (lane == 0) {
                                                 g.slot[b].nodes = nodes;
                                                 g.slot[b].runs = runs;
                                                 g.slot[b].last = done ? 1u : 0u;
                                             }
                                             bar_pass(g.full[b], lane);
                                             if (passed++) {  // the other slot's lists are summed
                                                 if (!bar_wait(g.empty[b ^ 1u], phase >> (b ^ 1u) & 1u)) return false;
                                                 phase ^= 1u << (b ^ 1u);
                                             }
                                             if (done) {  // and the last: the memory is free for the next group
                                                 if (!bar_wait(g.empty[b], phase >> b & 1u)) return false;
                                                 phase ^= 1u << b;
                                             }
                                             return true;
                                         });
    } else {
        for (uint32_t b = 0, last = 0; !last; b ^= 1u) {
            ok = bar_wait(g.full[b], phase >> b & 1u);
            if (!ok) break;
            phase ^= 1u << b;
            const typename SM::Slot& sl = g.slot[b];
            last = sl.last;
            sum_slot<EXACT, QUAD>(y, g, sl, sl.nodes, sl.runs, P, Q, E2, anx, any, alx, aly, lane);
            bar_pass(g.empty[b], lane);
        }
    }
    if (!ok) {
        if (lane == 0) atomicOr(y.err, kErrBarrierWait);
        return false;
    }
    if (!SM::kSplit || !walker)
        group_finish<ESTIMATE>(add2(anx, alx), add2(any, aly), v0, v1, i0, i1, p0, p1, y.vel_in, y.pos_out, y.vel_out,
                               y.acc_rec, y.k, y.hdt, y.amag, y.ext);
    return true;
}

// ------------------------------------------------------------------------------------
// Costly groups: a warp pair per walk.  With the relative criterion a group whose smallest
// previous |a| is far below its largest (every |a| known and a_min < kHeavyRatio a_max)
// opens many more records than the others: on the 500k spiral such groups sum 2.4x the
// mean interactions and their single-warp walks trailed the traversal launch.  In systems
// of at least kHeavyMinParticles particles (more groups than the launch keeps resident)
// their walks run first, each on two warps of one block: pops take the top min(64, size)
// records (warp w tests entries [32w, 32w + 32) of the popped range), the block's pair
// scans the counts of both warps, and item i of the node list (record i of the flattened
// leaf runs) is summed by warp (i / 32) mod 2, each warp from zero in walk order; the node
// (leaf) accumulator is warp 0's + warp 1's.  The tested and accepted records are the
// same as with 32-record pops (a record is tested iff all its ancestors were opened);
// only the summation order differs, and the CPU restatement follows it.
// ------------------------------------------------------------------------------------
// 64-record pops push at most 256 children, one level deeper than the shallowest popped
// record: <= 192 D + 256 entries, the bottom of a deep stack in warp 0's local memory.
constexpr int kPairStackCap = 192 * (kBBoxMaxBits > kFixedDepth ? kBBoxMaxBits : kFixedDepth) + 256;
constexpr int kPairNode = 128, kPairItem = 192;  // a round adds <= 64 nodes and <= 128 runs

struct PairSmem {
    uint32_t stack[kPairStackWindow];
    uint32_t node[kPairNode];
    uint2 run[kPairItem];
    uint32_t off[kPairItem];
    union {
        struct {
            float4 ca[2][32], cb[2][32];  // one staged chunk per warp
        };
        float2 part[4][32];  // after the sums: warp 1's accumulators, added by warp 0
    };
    uint32_t tot[2];  // packed round counts of each warp
    uint32_t ticket;
};

// Warp wp's share of the count accepted nodes in g.node, whose global list indices are
// gbase .. gbase + count - 1: the 32-item chunks c with c mod 2 == wp, in order (each
// chunk's records loaded while the one before is summed).
template <bool EXACT, bool QUAD>
__device__ __forceinline__ void pair_eval_nodes(PairSmem& g, int wp, uint32_t count, uint32_t gbase,
                                                const float4* __restrict__ rec, const float4* __restrict__ quad,
                                                float2 P, float2 Q, float2 E2, float2& acx, float2& acy, int lane) {
    const uint32_t end = gbase + count;
    uint32_t c = gbase >> 5;
    if ((c & 1u) != (uint32_t)wp) ++c;
    if (!count || c * 32 >= end) return;
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f), qq = q;
    {
        const uint32_t f = c * 32 + (uint32_t)lane;  // global index of the lane's item
        if (f >= gbase && f < end) {
            const uint32_t r = g.node[f - gbase];
            q = __ldg(&rec[r]);
            if (QUAD) qq = __ldg(&quad[r]);
        }
    }
    for (; c * 32 < end; c += 2) {
        __syncwarp();
        stage_node<QUAD>(g.ca[wp], g.cb[wp], lane, q, qq);
        __syncwarp();
        const uint32_t fn = (c + 2) * 32 + (uint32_t)lane;  // the warp's next chunk (all past gbase)
        if (fn < end) {
            const uint32_t r = g.node[fn - gbase];
            q = __ldg(&rec[r]);
            if (QUAD) qq = __ldg(&quad[r]);
        }
        sum_chunk<EXACT, QUAD>(g.ca[wp], g.cb[wp], gbase > c * 32 ? gbase - c * 32 : 0u, min(end - c * 32, 32u), P, Q,
                               E2, acx, acy);
    }
    __syncwarp();
}

// Record fl of the flattened leaf runs of a pair (last run with off <= fl).
__device__ __forceinline__ float4 pair_gather_leaf(const PairSmem& g, uint32_t n_items, uint32_t fl,
                                                   const float4* __restrict__ rec) {
    uint32_t lo = 0, hi = n_items - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (g.off[mid] <= fl) lo = mid;
        else hi = mid - 1;
    }
    return __ldg(&rec[g.run[lo].x + (fl - g.off[lo])]);
}

// Warp wp's share of the particle leaves of the n_items runs, whose flattened records have
// global indices lbase ..; returns the number of records.  Both warps of the pair must call
// it (warp 0 writes the run offsets, then the pair synchronises).
template <bool EXACT>
__device__ __forceinline__ uint32_t pair_eval_leaves(PairSmem& g, int pair, int wp, uint32_t n_items, uint32_t lbase,
                                                     const float4* __restrict__ rec, float2 P, float2 Q, float2 E2,
                                                     float2& acx, float2& acy, int lane) {
    if (!n_items) return 0u;
    uint32_t total = 0;
    if (wp == 0) total = run_offsets<kPairItem / 32>(g.run, g.off, n_items, lane);
    pair_sync(pair);
    total = g.off[n_items - 1] + g.run[n_items - 1].y;
    const uint32_t end = lbase + total;
    uint32_t c = lbase >> 5;
    if ((c & 1u) != (uint32_t)wp) ++c;
    if (c * 32 >= end) return total;
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    {
        const uint32_t f = c * 32 + (uint32_t)lane;
        if (f >= lbase && f < end) q = pair_gather_leaf(g, n_items, f - lbase, rec);
    }
    for (; c * 32 < end; c += 2) {
        __syncwarp();
        g.ca[wp][lane] = q;
        __syncwarp();
        const uint32_t fn = (c + 2) * 32 + (uint32_t)lane;
        if (fn < end) q = pair_gather_leaf(g, n_items, fn - lbase, rec);
        sum_chunk<EXACT, false>(g.ca[wp], nullptr, lbase > c * 32 ? lbase - c * 32 : 0u, min(end - c * 32, 32u), P, Q,
                                E2, acx, acy);
    }
    __syncwarp();
    return total;
}

// The walk of costly group `group` by warp wp (0, 1) of pair `pair`; both warps call it
// with the same arguments.  Warp 0 integrates.
template <bool EXACT, bool COUNT>
__device__ __forceinline__ void force_pair_body(
    const GroupSys& y, uint32_t group, int pair, int wp, PairSmem& g) {
    const int lane = threadIdx.x & 31;
    const uint32_t nv = y.counts[0];
    const uint32_t T = min(nv + y.counts[1], y.cap);
    const uint32_t g0 = group * kGroupSize;
    if (g0 >= nv || T == 0) return;  // never for a listed group; the same for both warps
    const uint32_t s0 = g0 + lane, s1 = s0 + 32;
    const uint32_t i0 = s0 < nv ? y.sidx[s0] : 0u, i1 = s1 < nv ? y.sidx[s1] : 0u;
    const bool v0 = s0 < nv && i0 < y.n_al, v1 = s1 < nv && i1 < y.n_al;
    const float2 p0 = v0 ? y.pos_in[i0] : make_float2(0.0f, 0.0f);
    const float2 p1 = v1 ? y.pos_in[i1] : make_float2(0.0f, 0.0f);
    float bx0[4], bx1[4], by0[4], by1[4];
    group_boxes(y.skey, g0, nv, s0, s1, v0, v1, p0, p1, bx0, bx1, by0, by1);
    float amin = fminf(v0 ? y.amag[i0] : INFINITY, v1 ? y.amag[i1] : INFINITY);  // every |a| is known
    for (int o = 16; o; o >>= 1) amin = fminf(amin, __shfl_xor_sync(0xffffffffu, amin, o));
    const float tol = y.alpha * amin, tol2 = tol * tol;
    const float2 P = make_float2(p0.x, p1.x), Q = make_float2(p0.y, p1.y), E2 = make_float2(y.eps2, y.eps2);
    float2 anx = make_float2(0.0f, 0.0f), any = anx, alx = anx, aly = anx;
    unsigned long long n_int = 0, n_test = 0, n_node = 0;
    StackSpill<kPairStackCap, kPairStackSpill> spill;
    uint32_t size = 0, n_nodes = 0, n_items = 0, gnode = 0, gleaf = 0;
    if (y.skip[0] == 1u) {  // a single particle: the root is its leaf
        if (wp == 0 && lane == 0) {
            g.run[0] = make_uint2(0u, 1u);
        }
        n_items = 1;
    } else {
        if (wp == 0 && lane == 0) g.stack[0] = 0u;
        size = 1;
    }
    for (;;) {
        pair_sync(pair);  // the last round's lists, pushes and counts are visible
        if (size == 0 && spill.count == 0) break;
        if (n_nodes > (uint32_t)(kPairNode - 64)) {
            pair_eval_nodes<EXACT, true>(g, wp, n_nodes, gnode, y.rec, y.quad, P, Q, E2, anx, any, lane);
            gnode += n_nodes;
            n_nodes = 0;
            pair_sync(pair);
        }
        if (n_items > (uint32_t)(kPairItem - 128)) {
            gleaf += pair_eval_leaves<EXACT>(g, pair, wp, n_items, gleaf, y.rec, P, Q, E2, alx, aly, lane);
            n_items = 0;
            pair_sync(pair);
        }
        if (size < 64u && spill.count) {  // the same in both warps; warp 0 holds the entries
            if (wp == 0) size = spill.restore(g.stack, size, lane);
            else size += kPairStackSpill, spill.count -= kPairStackSpill;
            pair_sync(pair);
        }
        const uint32_t np = min(size, 64u);
        const uint32_t base = size - np;
        const uint32_t L = (uint32_t)(wp * 32 + lane);
        const bool act = L < np;
        const uint32_t n = act ? g.stack[base + L] : 0u;
        pair_sync(pair);  // both warps hold their records before pushes overwrite the stack top
        size = base;
        if (COUNT) n_test += __popc(__ballot_sync(0xffffffffu, act));
        RecTest r{};
        if (act) test_record(n, y.rec, y.kids, bx0, bx1, by0, by1, y.eps2, true, tol2, y.floor2, 0.0f, r);
        // offsets in pair order: this warp's scan plus warp 0's total for warp 1; nodes
        // <= 64, runs <= 128 and pushes <= 256 in pair total, so the 8/8/16-bit fields
        // never carry
        const uint32_t mine = r.nn | (r.nl << 8) | (r.npu << 16);
        uint32_t x = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) g.tot[wp] = x;
        pair_sync(pair);
        const uint32_t t0 = g.tot[0], t1 = g.tot[1];
        const uint32_t ex = x - mine + (wp ? t0 : 0u), tot = t0 + t1;
        const uint32_t noff = ex & 0xffu, loff = (ex >> 8) & 0xffu, poff = ex >> 16;
        const uint32_t ntot = tot & 0xffu, ltot = (tot >> 8) & 0xffu;
        uint32_t ptot = tot >> 16, npu = r.npu;
        if (size + ptot > (uint32_t)kPairStackWindow) {
            if (wp == 0) size = spill.save(g.stack, size, lane);
            else size -= kPairStackSpill, spill.count += kPairStackSpill;
            pair_sync(pair);
        }
        if (spill.count + size + ptot > (uint32_t)kPairStackCap) {  // beyond the depth bound: report, do not overrun
            if (wp == 0 && lane == 0) atomicOr(y.err, kErrTree);
            ptot = 0;
            npu = 0;
        }
        if (r.nn) g.node[n_nodes + noff] = n;
        if (r.nl > 0) g.run[n_items + loff] = make_uint2(r.a0, r.c0);
        if (r.nl > 1) g.run[n_items + loff + 1] = make_uint2(r.a1, r.c1);
        if (COUNT) {
            n_int += r.nn + (r.nl > 0 ? r.c0 : 0u) + (r.nl > 1 ? r.c1 : 0u);
            n_node += r.nn;
        }
        uint32_t* dst = g.stack + size + poff;
        if (npu > 0) dst[0] = r.pu[0];
        if (npu > 1) dst[1] = r.pu[1];
        if (npu > 2) dst[2] = r.pu[2];
        if (npu > 3) dst[3] = r.pu[3];
        n_nodes += ntot;
        n_items += ltot;
        size += ptot;
    }
    pair_eval_nodes<EXACT, true>(g, wp, n_nodes, gnode, y.rec, y.quad, P, Q, E2, anx, any, lane);
    pair_eval_leaves<EXACT>(g, pair, wp, n_items, gleaf, y.rec, P, Q, E2, alx, aly, lane);
    if (COUNT) {
        if (y.skip[0] == 1u && wp == 0 && lane == 0) n_int += 1;
        for (int o = 16; o; o >>= 1) {
            n_int += __shfl_xor_sync(0xffffffffu, n_int, o);
            n_node += __shfl_xor_sync(0xffffffffu, n_node, o);
        }
        const unsigned long long nval = __popc(__ballot_sync(0xffffffffu, v0)) + __popc(__ballot_sync(0xffffffffu, v1));
        if (lane == 0) {
            atomicAdd(&y.stat[0], n_int * nval);
            atomicAdd(&y.stat[1], n_test);
            atomicAdd(&y.stat[2], n_node * nval);
        }
    }
    pair_sync(pair);  // both warps are done with their staged chunks
    if (wp == 1) {
        g.part[0][lane] = anx;
        g.part[1][lane] = any;
        g.part[2][lane] = alx;
        g.part[3][lane] = aly;
    }
    pair_sync(pair);
    if (wp == 0) {
        anx = add2(anx, g.part[0][lane]);
        any = add2(any, g.part[1][lane]);
        alx = add2(alx, g.part[2][lane]);
        aly = add2(aly, g.part[3][lane]);
        group_finish<false>(add2(anx, alx), add2(any, aly), v0, v1, i0, i1, p0, p1, y.vel_in, y.pos_out,
                            y.vel_out, y.acc_rec, y.k, y.hdt, y.amag, y.ext);
    }
    pair_sync(pair);  // the pair's shared memory is free for its next group
}

// The launch of a group-walk kernel: GROUPS groups per block, on one warp each or (SPLIT) two;
// long or short lists (gs_shape).
template <int GROUPS, bool SHORT, bool SPLIT, bool MIXED = false>
struct WalkShape {
    using SplitSmem = GroupSmem<SHORT ? 31 : 63, SHORT ? 31 : 63, 2>;
    using Smem = typename std::conditional<SPLIT, SplitSmem, GroupSmem<SHORT ? 64 : 128, SHORT ? 32 : 64, 1>>::type;
    static_assert(!MIXED || (GROUPS == 2 && !SPLIT), "a block's two warps take two groups or share one");
    static constexpr bool kMixed = MIXED;
    static constexpr int kGroups = GROUPS, kThreads = GROUPS * (SPLIT ? 64 : 32);
    // resident blocks the registers are cut for: one warp per group at 96 registers a thread
    // (20 groups an SM), two at 128 (8 groups: N = 100,000, 161 us a step against 167 with 12 and 179 with 16)
    static constexpr int kBlocks = (SPLIT ? kSplitPerSm : kSinglePerSm) / GROUPS;
    static constexpr bool kSplit = SPLIT;
};

// Shared memory of a block; with HEAVY (the main pass of the relative criterion, groups on one
// warp each) each pair of warps first walks costly groups together in the bytes of its two groups.
template <class SH, bool HEAVY>
struct WalkSmem {
    union {
        typename SH::Smem g[SH::kGroups];
        typename SH::SplitSmem split;  // kMixed
    };
    PairTurn turn[(SH::kThreads + 63) / 64];
    __device__ __forceinline__ typename SH::Smem& walk(int i) { return g[i]; }
    __device__ __forceinline__ typename SH::SplitSmem& both() { return split; }
};
template <class SH>
struct WalkSmem<SH, true> {
    static_assert(!SH::kSplit && SH::kThreads % 64 == 0, "whole pairs of warps, a group each");
    union Pair {
        typename SH::Smem g[2];
        PairSmem pair;
    } p[SH::kThreads / 64];
    PairTurn turn[SH::kThreads / 64];
    __device__ __forceinline__ typename SH::Smem& walk(int i) { return p[i / 2].g[i % 2]; }
};

// The next value of a counter below cnt for both warps of a pair, or a value >= cnt when none
// is left.
__device__ __forceinline__ uint32_t pair_ticket(uint32_t* __restrict__ next, uint32_t cnt, uint32_t& s_u, int pair) {
    if ((threadIdx.x & 63u) == 0) s_u = __ldcg(next) < cnt ? atomicAdd(next, 1u) : cnt;
    pair_sync(pair);
    const uint32_t u = s_u;
    pair_sync(pair);  // read by both warps before the next ticket
    return u;
}
// The same for one warp.
__device__ __forceinline__ uint32_t warp_ticket(uint32_t* __restrict__ next, uint32_t cnt) {
    uint32_t u = 0;
    if ((threadIdx.x & 31u) == 0) u = __ldcg(next) < cnt ? atomicAdd(next, 1u) : cnt;
    return __shfl_sync(0xffffffffu, u, 0);
}

template <class SM>
__device__ __forceinline__ void walk_init(SM& g, int pair) {
    if (!SM::kSplit) return;
    if ((threadIdx.x & 63u) < 2u) {
        bar_init(g.full[threadIdx.x & 1u]);
        bar_init(g.empty[threadIdx.x & 1u]);
    }
    pair_sync(pair);
}

// Which of a walk's two warps walks: alternating over walks and blocks, so that the summing
// warps, which keep the FMA pipe busy, spread over the four schedulers.
__device__ __forceinline__ bool is_walker() {
    const uint32_t warp = threadIdx.x >> 5;
    return ((warp + (warp >> 1) + blockIdx.x) & 1u) == 0;
}

// With HEAVY every pair of warps first takes listed costly groups (heavy_list[u].y, in order
// from hwork) and then its own: the costly walks start first.
template <bool EXACT, bool QUAD, bool COUNT, bool ESTIMATE, class SH, bool HEAVY>
__global__ void __launch_bounds__(SH::kThreads, SH::kBlocks)
k_force_group(GroupSys y, const uint2* __restrict__ heavy_list, uint32_t* __restrict__ hwork) {
    __shared__ __align__(16) WalkSmem<SH, HEAVY> sm;
    pdl_enter();
    const int pair = (int)(threadIdx.x >> 6), walk = SH::kSplit ? pair : (int)(threadIdx.x >> 5);
    if constexpr (HEAVY) {
        static_assert(QUAD && !ESTIMATE, "warp pairs walk costly groups of the relative main pass");
        const uint32_t cnt = hwork[0];
        for (uint32_t u; (u = pair_ticket(hwork + 1, cnt, sm.turn[pair].unit, pair)) < cnt;)
            force_pair_body<EXACT, COUNT>(y, heavy_list[u].y, pair, (int)((threadIdx.x >> 5) & 1u), sm.p[pair].pair);
    }
    uint32_t phase = 0;
    if constexpr (SH::kMixed) {
        if (blockIdx.x >= y.tail) {
            walk_init(sm.both(), 0);
            force_group_body<EXACT, QUAD, COUNT, ESTIMATE>(y, y.tail + blockIdx.x, is_walker(), phase, sm.both());
            return;
        }
    }
    walk_init(sm.walk(walk), pair);
    force_group_body<EXACT, QUAD, COUNT, ESTIMATE>(y, blockIdx.x * SH::kGroups + walk, !SH::kSplit || is_walker(), phase,
                                                   sm.walk(walk));
}

__device__ __forceinline__ GroupSys batch_group_sys(const SysDesc& d, int in, int out, bool heavy) {
    const int f = d.passes & 1;
    return GroupSys{d.idx[f], d.keys[f], d.counters + kCtrValid, d.rec, d.skip, d.quad, d.kids, d.pos[in], d.vel[in],
                    d.pos[out], d.vel[out], d.acc, d.n_al, d.eps2, d.theta2, d.k, d.hdt, d.cap,
                    (unsigned long long*)(d.counters + kCtrStat), d.err, d.amag, d.alpha, d.floor2,
                    d.ext ? d.ext + 4 * out : nullptr, heavy ? d.heavy : nullptr};
}

// Batched: a persistent grid; with HEAVY each pair of warps first takes costly groups
// {member, group} from the batch's list, then every walk takes groups of the members from
// `work`.
template <bool EXACT, bool QUAD, bool COUNT, bool ESTIMATE, class SH, bool HEAVY>
__global__ void __launch_bounds__(SH::kThreads, SH::kBlocks)
kb_force_group(BatchArgs a, uint32_t* __restrict__ work, const uint2* __restrict__ heavy_list,
               uint32_t* __restrict__ hwork) {
    __shared__ __align__(16) WalkSmem<SH, HEAVY> sm;
    pdl_enter();
    const int pair = (int)(threadIdx.x >> 6), walk = SH::kSplit ? pair : (int)(threadIdx.x >> 5);
    if constexpr (HEAVY) {
        static_assert(QUAD && !ESTIMATE, "warp pairs walk costly groups of the relative main pass");
        const uint32_t cnt = hwork[0];
        for (uint32_t u; (u = pair_ticket(hwork + 1, cnt, sm.turn[pair].unit, pair)) < cnt;) {
            const uint2 e = heavy_list[u];
            const SysDesc& d = a.descs[e.x];
            const int in = (int)((d.parity + a.step) & 1u);
            force_pair_body<EXACT, COUNT>(batch_group_sys(d, in, in ^ 1, false), e.y, pair,
                                          (int)((threadIdx.x >> 5) & 1u), sm.p[pair].pair);
        }
    }
    if (SH::kSplit && (threadIdx.x & 63u) == 0) sm.turn[pair].failed = 0u;
    walk_init(sm.walk(walk), pair);  // SPLIT: with a barrier of the pair
    const uint32_t total = __ldg(&a.first[a.nsys]);
    const bool walker = !SH::kSplit || is_walker();
    uint32_t phase = 0;
    const auto group = [&](uint32_t u) {
        const BatchBlock bb = batch_block(a, u);
        return force_group_body<EXACT, QUAD, COUNT, ESTIMATE>(batch_group_sys(*bb.d, bb.in, bb.out, HEAVY), bb.blk.id,
                                                              walker, phase, sm.walk(walk));
    };
    if constexpr (SH::kSplit) {
        pair_loop(sm.turn[pair], (threadIdx.x & 63u) == 0, total,
                  [&] { return __ldcg(work) < total ? atomicAdd(work, 1u) : total; }, [&] { pair_sync(pair); }, group);
    } else {  // no walk of one warp waits for another
        for (uint32_t u; (u = warp_ticket(work, total)) < total;) group(u);
    }
}

template <bool EXACT, bool COUNT>
__global__ void __launch_bounds__(kForceWarps * 32, 6) kb_force(BatchArgs a, uint32_t* __restrict__ work) {
    pdl_enter();
    __shared__ RuleWindow win[kForceWarps];
    __shared__ uint32_t s_b;
    const uint32_t total = __ldg(&a.first[a.nsys]);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_b = atomicAdd(work, 1u);
        __syncthreads();
        const uint32_t b = s_b;
        if (b >= total) break;
        const BatchBlock bb = batch_block(a, b);
        const SysDesc& d = *bb.d;
        const int f = d.passes & 1;
        auto walk = [&](auto ftz) {
            force_body<EXACT, COUNT, decltype(ftz)::value, false>(
                bb.blk, &win[threadIdx.x >> 5], nullptr, nullptr, d.idx[f], d.counters + kCtrValid, d.rec, d.skip,
                d.pos[bb.in], d.vel[bb.in], d.pos[bb.out], d.vel[bb.out], d.acc, d.n_al, d.eps2, d.theta2, d.k, d.hdt,
                d.cap, (unsigned long long*)(d.counters + kCtrStat), d.ext ? d.ext + 4 * bb.out : nullptr);
        };
        if (EXACT || rule_ftz(d.eps2)) walk(std::true_type{});
        else walk(std::false_type{});
    }
}

}  // namespace
}  // namespace gsim

namespace gsim {
namespace {

using GroupFn = void (*)(GroupSys, const uint2*, uint32_t*);
using BatchGroupFn = void (*)(BatchArgs, uint32_t*, const uint2*, uint32_t*);

// The group-walk kernel of one shape (counting variants: the default shape only); heavy:
// the main pass with warp pairs for costly groups (quadrupoles, relative criterion), which
// need two warps per block at least, and have them: only systems above kSplitGroups have
// costly groups.
template <bool EXACT, bool COUNT, class SH>
GroupFn group_fn(bool quad, bool est, bool heavy) {
    if constexpr (!SH::kMixed) {
        if (est) return k_force_group<EXACT, true, COUNT, true, SH, false>;
        if constexpr (SH::kThreads >= 64 && !SH::kSplit)
            if (heavy) return k_force_group<EXACT, true, COUNT, false, SH, true>;
    }
    return quad ? k_force_group<EXACT, true, COUNT, false, SH, false>
                : k_force_group<EXACT, false, COUNT, false, SH, false>;
}
template <bool EXACT, bool COUNT, class SH>
BatchGroupFn batch_group_fn(bool quad, bool est, bool heavy) {
    if (est) return kb_force_group<EXACT, true, COUNT, true, SH, false>;
    if constexpr (SH::kThreads >= 64 && !SH::kSplit)
        if (heavy) return kb_force_group<EXACT, true, COUNT, false, SH, true>;
    return quad ? kb_force_group<EXACT, true, COUNT, false, SH, false>
                : kb_force_group<EXACT, false, COUNT, false, SH, false>;
}

// fn(shape) with the shape launched for a request, its groups and threads per block.
template <class Fn>
auto with_shape(bool count, const gs_shape& sh, bool split, bool heavy, int* groups, int* threads, Fn&& fn) {
    const auto use = [&](auto shape) {
        *groups = decltype(shape)::kGroups;
        *threads = decltype(shape)::kThreads;
        return fn(shape);
    };
    if (count) return use(WalkShape<2, false, false>{});
    const uint32_t g = heavy && sh.force_warps == 1 ? 2u : sh.force_warps;
    if (sh.force_short_lists) return split ? use(WalkShape<2, true, true>{}) : use(WalkShape<2, true, false>{});
    if (g == 1) return split ? use(WalkShape<1, false, true>{}) : use(WalkShape<1, false, false>{});
    if (g == 4) return split ? use(WalkShape<4, false, true>{}) : use(WalkShape<4, false, false>{});
    return split ? use(WalkShape<2, false, true>{}) : use(WalkShape<2, false, false>{});
}

// Two warps per group where the launch's groups cannot fill the SMs on one warp each.
constexpr uint32_t kSplitGroups = 152 * 14;
static_assert(kHeavyMinParticles / kGroupSize > kSplitGroups, "costly groups only where every group has one warp");

// Larger launches: the last groups on two warps each, so that the chip does not end on whole
// single-warp walks.  Five such groups an SM; eight where every group starts at once (3,040 on
// one warp each).  Step with none and with these, relative criterion: 140,000 particles 236 and
// 230 us, 150,000 223 and 197, 200,000 264 and 261; theta 0.35: 250,000 270 and 262, 450,000 398
// and 384.  Not with warp pairs for costly groups, which are that launch's end whatever the last
// groups do (five steps of 300,000 1.95 and 1.99 ms), nor by theta where every group starts at
// once (its walks differ little: 180,000 1.17 and 1.20 ms).
inline uint32_t tail_groups(uint32_t n_groups) { return n_groups <= 152 * kSinglePerSm ? 152 * 8 : 152 * 5; }
inline bool walk_tail(const ForceLaunch& f, uint32_t n_groups, bool heavy) {
    static_assert(kSplitGroups > 152 * 8, "some groups are left on one warp");
    return n_groups > kSplitGroups && (f.amag ? !heavy : n_groups > 152 * kSinglePerSm) && !f.count && !f.estimate &&
           f.shape.force_warps == 2 && !f.shape.force_short_lists;
}

template <bool EXACT>
GroupFn pick_group(bool count, const gs_shape& sh, uint32_t n_groups, bool mixed, bool quad, bool est, bool heavy,
                   int* groups, int* threads) {
    if (mixed) {
        using SH = WalkShape<2, false, false, true>;
        *groups = SH::kGroups;
        *threads = SH::kThreads;
        return group_fn<EXACT, false, SH>(quad, est, heavy);
    }
    return with_shape(count, sh, n_groups <= kSplitGroups, heavy, groups, threads, [&](auto s) {
        using SH = decltype(s);
        if constexpr (std::is_same<SH, WalkShape<2, false, false>>::value)
            if (count) return group_fn<EXACT, true, SH>(quad, est, heavy);
        return group_fn<EXACT, false, SH>(quad, est, heavy);
    });
}

template <bool EXACT>
BatchGroupFn pick_batch_group(bool count, const gs_shape& sh, uint32_t n_groups, bool quad, bool est, bool heavy,
                              int* groups, int* threads) {
    return with_shape(count, sh, n_groups <= kSplitGroups, heavy, groups, threads, [&](auto s) {
        using SH = decltype(s);
        if constexpr (std::is_same<SH, WalkShape<2, false, false>>::value)
            if (count) return batch_group_fn<EXACT, true, SH>(quad, est, heavy);
        return batch_group_fn<EXACT, false, SH>(quad, est, heavy);
    });
}

template <bool EXACT>
cudaError_t force_launch_impl(const ForceLaunch& f) {
    if (!f.group) {  // the reference's warp-vote walk
        const auto run = [&](auto ftz) {
            constexpr bool kFtz = decltype(ftz)::value;
            const int blocks = (int)((f.n_al / 32 + kForceWarps - 1) / kForceWarps);
            if (f.n_al <= kRuleStagedMax) {
                auto fn = f.count ? k_force_staged<EXACT, true, kFtz> : k_force_staged<EXACT, false, kFtz>;
                const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                           (int)sizeof(RuleTree));
                if (e != cudaSuccess) return e;
                return launch_shared(f.pdl, fn, blocks, kForceWarps * 32, (unsigned)sizeof(RuleTree), f.st, f.sidx,
                                     f.counts, f.rec, f.skip, f.pos_in, f.vel_in, f.pos_out, f.vel_out, f.acc, f.n_al,
                                     f.eps2, f.theta2, f.k, f.hdt, f.cap, f.stat, f.ext);
            }
            return launch(f.pdl, f.count ? k_force<EXACT, true, kFtz> : k_force<EXACT, false, kFtz>, blocks,
                          kForceWarps * 32, f.st, f.sidx, f.counts, f.rec, f.skip, f.pos_in, f.vel_in, f.pos_out,
                          f.vel_out, f.acc, f.n_al, f.eps2, f.theta2, f.k, f.hdt, f.cap, f.stat, f.ext);
        };
        if constexpr (!EXACT)
            if (!rule_ftz(f.eps2)) return run(std::false_type{});
        return run(std::true_type{});
    }
    int groups = 2, threads = 64;
    const bool heavy = f.heavy && f.quad && !f.estimate;
    const uint32_t n_groups = f.n_al / kGroupSize;
    const bool mixed = walk_tail(f, n_groups, heavy);
    GroupFn fn = pick_group<EXACT>(f.count, f.shape, n_groups, mixed, f.quad, f.estimate, heavy, &groups, &threads);
    int blocks = (int)((n_groups + groups - 1) / groups);
    GroupSys y{f.sidx, f.skey, f.counts, f.rec, f.skip, f.quad_m, f.kids, f.pos_in, f.vel_in, f.pos_out, f.vel_out,
                     f.acc, f.n_al, f.eps2, f.theta2, f.k, f.hdt, f.cap, f.stat, f.err, f.amag, f.alpha, f.floor2,
                     f.ext, heavy ? f.heavy : nullptr};
    if (mixed) {
        y.tail = (n_groups - tail_groups(n_groups)) / 2;
        blocks = (int)(n_groups - y.tail);
    }
    return launch(f.pdl, fn, blocks, threads, f.st, y, heavy ? f.heavy_list : nullptr,
                  heavy ? f.heavy_work : nullptr);
}

template <bool EXACT>
cudaError_t batch_force_launch_impl(const BatchForceLaunch& b, int* grid_out) {
    int dev = 0, sms = 0, per_sm = 0, threads = kForceWarps * 32;
    const bool heavy = b.heavy_list && b.quad && !b.estimate;
    auto resident = [&](auto fn) -> cudaError_t {  // resident blocks of the persistent launch
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0);
        if (e != cudaSuccess) return e;
        *grid_out = (sms > 0 ? sms : 152) * (per_sm > 0 ? per_sm : 1);
        return cudaSuccess;
    };
    if (!b.group) {
        auto fn = b.count ? kb_force<EXACT, true> : kb_force<EXACT, false>;
        if (grid_out) return resident(fn);
        return launch(true, fn, b.grid, threads, b.st, BatchArgs{b.descs, b.first, b.nsys, b.step}, b.work);
    }
    int groups = 2;
    BatchGroupFn fn = pick_batch_group<EXACT>(b.count, b.shape, b.units, b.quad, b.estimate, heavy, &groups, &threads);
    if (grid_out) return resident(fn);
    const int grid = (int)(b.units + groups - 1) / groups;  // no more blocks than groups need
    return launch(true, fn, b.grid < grid ? b.grid : grid, threads, b.st, BatchArgs{b.descs, b.first, b.nsys, b.step}, b.work,
                  heavy ? b.heavy_list : nullptr, heavy ? b.heavy_work : nullptr);
}

}  // namespace
}  // namespace gsim
