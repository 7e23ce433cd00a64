// Attention over the fp16 KV cache in the reference's exact arithmetic, the upload re-tiling kernels,
// and the small per-operator kernels that let the reference's graph run op by op on the device.
// All of these are HBM- or latency-bound byte/float work; none is a dense contraction.
//
// Exactness: the reference network quantizes activations at every layer, which amplifies any
// difference in f32 summation order to percent-level logit differences. Every reduction here therefore
// follows the CPU's order: the 4 x 8 accumulators and the scalar tail of Dot<FP16,FP16>, the four-wide
// grouping of std::reduce / std::transform_reduce, and the fixed horizontal-add trees.

#include <algorithm>

#include <cstdlib>

#include "spyb_common.cuh"
#include "spyb_kernels.h"
#include "spyb_tp.cuh"
#include "spyb_mv_common.cuh"

#include <math_constants.h>

namespace spyb {

static inline cudaError_t launch_check() { return cudaGetLastError(); }

// std::reduce over floats as libstdc++ evaluates it for random-access ranges: groups of four combined as
// (e0 + e1) + (e2 + e3) and added to the running sum one after the other, the remainder one by one.
// One thread's chain; `v` is in shared memory.
__device__ __forceinline__ float reduce4_chain(const float *v, int n) {
    float sum = 0.f;
    int i = 0;
    for (; i + 4 <= n; i += 4) { sum = __fadd_rn(sum, __fadd_rn(__fadd_rn(v[i], v[i + 1]), __fadd_rn(v[i + 2], v[i + 3]))); }
    for (; i < n; ++i) { sum = __fadd_rn(sum, v[i]); }
    return sum;
}

// =============================================================================================
// Attention for one (head, query token): a CTA of 8 warps, head_dim 128.
//   scores = K(f16) . fp16(Q)            MatMul with F16 weights: backend/host/operator/mat.cpp:32-42,
//                                        Dot<FP16,FP16> backend/host/include/simd/vec_dot.h:117-146
//   probs  = masked softmax, exp through the table of expf(fp16(s - max)), std::reduce sum
//                                        backend/host/operator/non-linear.cpp:129-180
//   out    = V(f16) . fp16(probs)        same MatMul rule; V is kept transposed [d][n_ctx] as the reference
//                                        graph lays it out (model/src/llm/plugin/attention.cpp:228-262)
// Dot<FP16,FP16> runs four 8-wide accumulators over 32-element steps while i + 32 < n, reduces them as
// (s0 + s2) + (s1 + s3), element l with l + 4, two horizontal adds, and leaves the rest (1..32 elements) to
// a scalar FMA chain added as tail + vector part. All 32 accumulators of a dot product live in the
// registers of ONE thread here (scores: one thread per position, the K row read with 128-bit loads) or of a
// thread pair (PV: elements 0..3 / 4..7 of the four accumulators, the V^T row read with 64-bit loads), so the
// reduction tree is register arithmetic and the dot products of a head run side by side.
// Roofline: HBM-bound, 2 * n_kv * head_dim * 2 bytes per head read once; latency-bound at short contexts.
constexpr int ATT_THREADS = 256;
constexpr int ATT_WARPS   = ATT_THREADS / WARP;
constexpr int ATT_HD      = 128;
constexpr int ATT_MANY    = 2;      // CTAs an SM holds of a launch that has more of them than the chip has SMs

// a * b + c of the f16 values in the low halves of a and b: the fmaf of the widened values (their product is exact in f32) without widening
// them; it issues as fast as fmaf, and half the bytes of its operands come out of shared memory
__device__ __forceinline__ float fma_f16(uint32_t a, uint32_t b, float c) {
    float d;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"((uint16_t)a), "h"((uint16_t)b), "f"(c));
    return d;
}
__device__ __forceinline__ uint32_t half_of(const uint32_t *w, int i) { return w[i >> 1] >> (16 * (i & 1)); }

// EARLY: a step that reads cache rows ahead of its wait (a kernel of its own: 7B steps 0.6 % slower with both in one)
// CTAS > 1: for launches of more CTAs than SMs, so many of them side by side on one: a K row and the V^T values are read when they are needed instead
// of being held ahead in 248 registers, with which one CTA fills an SM. us a step of four layers, one CTA an SM / 2 / 3 / 4: 40 heads x 32 sequences at
// 10 positions 1229 / 1162 / 1155 / 1161; 16 x 32 at 400 637 / 588 / 615 / 677; 32 x 16 at 200 740 / 717 / 726 / 753; 32 x 8 at 900 828 / 824 / 936 /
// 1063 (more CTAs share an L1 that the V^T rows then leave).
template <bool EARLY, int CTAS, bool LEAN>
__global__ void __launch_bounds__(ATT_THREADS, CTAS) attention_kernel(const AttnParams p) {
    extern __shared__ __align__(16) float att_smem[];
    __shared__ float red[ATT_WARPS];
    __shared__ float bcast;

    const int h = blockIdx.x, t = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    pdl_launch_dependents();
    if (!LEAN) { stamp(p.stamps, 0, false); stamp(p.stamps, 4, true); }

    const bool batch = p.seq_stride != 0;        // token t = sequence t of a batch in lockstep: own cache, same position, nothing else visible
    const __half *k_cache = p.k_cache + (batch ? (int64_t)t * p.seq_stride : 0), *v_cache = p.v_cache + (batch ? (int64_t)t * p.seq_stride : 0);
    // Row length of the score matrix = all positions known to the step (past + every token of the step), as the
    // reference graph shapes it (K view [hd, n_past + n_token, H], model/src/llm/plugin/attention.cpp:207-223). Entries
    // beyond the causal limit carry mask -inf: they become exact zeros, but they still decide how std::reduce groups
    // the sum and where Dot<FP16,FP16> switches from its vector loop to the scalar tail.
    auto row_length = [&](int base, int known) { return batch ? base + 1 : known > 0 ? known : base + p.T; };
    const int n_pad = (p.n_ctx + 3) & ~3;
    float *sc = att_smem;                        // [n_pad] scores, then exponentials
    float *gs = sc + n_pad;                      // [n_pad / 4] four-wide partial sums of std::reduce
    __half *qh = reinterpret_cast<__half *>(gs + ((n_pad >> 2) + 3) / 4 * 4);   // [hd] Q, on 16 bytes
    __half *ph = qh + ATT_HD;                    // [n_pad] probabilities

    // Everything this thread will need from global memory is requested up front, so that Q, the first K row and
    // the V^T values of the PV product share one memory round trip instead of three: the PV thread pair of element
    // e = tid / 2 fetches the first 32-position step and the (at most 32-position) scalar tail of its row now.
    // A step of one token does so for the positions of earlier steps before it waits for the kernel in front, which adds one position to
    // the cache and changes nothing else in it; behind the wait only Q and what holds the new position is read. Whether the position
    // counter that was read early is the step's own shows then (the kernel that advances it may not have run; all is read again). L1 is not
    // coherent with the kernel in front: only K rows of earlier steps, which share no line with the new one, go through it before the wait.
    // (7B, 8 to 40 positions: 5.5 -> 4.8 us a layer.) Passes of several tokens, batches and the layers that attention_early() leaves out read everything
    // behind the wait and through L1, where the threads' 8 bytes of V^T share sectors.
    const int pv_e = tid >> 1, pv_half = tid & 1;
    const __half *vrow = v_cache + ((int64_t)h * ATT_HD + pv_e) * p.n_ctx;
    uint2 v_first[4], v_tail[8];
    constexpr bool AHEAD = CTAS == 1;
    uint4 kv[AHEAD ? 16 : 4];                        // a whole K row in flight at once
    // the words of V^T and the K row of which positions lo <= j < n_vis (K: lo <= tid) are wanted; words that reach past n_vis, which may be
    // new in part, belong to the second pass, which goes past L1 where there was a first one
    auto request_v = [&](int lo, int n_vis, int n_main, bool last) {
        auto load_v = [&](int j) { const uint2 *src = reinterpret_cast<const uint2 *>(vrow + j); return EARLY ? __ldcg(src) : *src; };
        auto wanted = [&](int j) { return j < n_vis && j + 4 > lo && (last || j + 4 <= n_vis); };
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int j = 8 * a + 4 * pv_half;
            if (0 < n_main && wanted(j)) { v_first[a] = load_v(j); }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int j = n_main + 4 * c;
            if (wanted(j)) { v_tail[c] = load_v(j); }
        }
    };
    auto request = [&](int lo, int n_vis, int n_main, bool last) {
        request_v(lo, n_vis, n_main, last);
        if (tid >= lo && tid < n_vis) {
            const uint4 *krow = reinterpret_cast<const uint4 *>(k_cache + (int64_t)tid * p.dl + (int64_t)h * ATT_HD);
#pragma unroll
            for (int a = 0; a < (AHEAD ? 16 : 0); ++a) { kv[a] = EARLY && last ? __ldcg(krow + a) : krow[a]; }
        }
    };
#pragma unroll
    for (int a = 0; a < 4; ++a) { v_first[a] = make_uint2(0u, 0u); }
#pragma unroll
    for (int c = 0; c < 8; ++c) { v_tail[c] = make_uint2(0u, 0u); }
    int early = -1, early_tot = 0;
    if (EARLY && gridDim.y == 1 && !batch) {
        const int2 known = __ldcg(reinterpret_cast<const int2 *>(p.pos_base));
        if (known.x >= 0 && known.x < p.n_ctx) { early = known.x; early_tot = row_length(known.x, known.y); }
        request(0, early, ((early_tot - 1) / 32) * 32, false);
    }
    pdl_wait();
    if (!LEAN) { stamp(p.stamps, 1, false); stamp(p.stamps, 5, true); }
    const int2 base = __ldcg(reinterpret_cast<const int2 *>(p.pos_base));
    const __half q_mine = (tid < ATT_HD) ? p.q[(int64_t)t * p.dl + (int64_t)h * ATT_HD + tid] : __float2half(0.f);
    if (EARLY && early >= 0) { request(early & ~3, early + 1, ((early_tot - 1) / 32) * 32, true); }   // (without waiting for the counter)
    const int pos   = base.x + (batch ? 0 : t);
    const int n_vis = pos + 1;                   // causal mask: positions 0..pos are visible
    const int n_tot = row_length(base.x, base.y), n_main = ((n_tot - 1) / 32) * 32;
    if (AHEAD && (early != pos || early_tot != n_tot)) {
#pragma unroll
        for (int a = 0; a < 4; ++a) { v_first[a] = make_uint2(0u, 0u); }
#pragma unroll
        for (int c = 0; c < 8; ++c) { v_tail[c] = make_uint2(0u, 0u); }
        request(0, n_vis, n_main, true);
    }
    if (tid < ATT_HD) { qh[tid] = q_mine; }
    __syncthreads();

    // ---- scores of the visible positions: one thread per position
#pragma unroll 1
    for (int j = tid; j < n_vis; j += ATT_THREADS) {
        const uint4  *krow = reinterpret_cast<const uint4 *>(k_cache + (int64_t)j * p.dl + (int64_t)h * ATT_HD);
        const uint2  *q2   = reinterpret_cast<const uint2 *>(qh);
        float acc[4][8];
        if (AHEAD && j != tid) {
#pragma unroll
            for (int a = 0; a < (AHEAD ? 16 : 0); ++a) { kv[a] = krow[a]; }
        }
        auto part = [&](int step) {                  // 32 elements of the row
            if constexpr (!AHEAD) {
                asm volatile("" ::: "memory");       // (not all of them ahead)
#pragma unroll
                for (int a = 0; a < 4; ++a) { kv[a] = krow[4 * step + a]; }
            }
        };
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int e = 0; e < 8; ++e) { acc[a][e] = 0.f; }
        }
#pragma unroll
        for (int step = 0; step < 3; ++step) {       // elements 0..95: accumulator a takes elements 32 * step + 8a .. + 7
            part(step);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const uint4 kw = kv[AHEAD ? 4 * step + a : a];
                const uint2 qa = q2[(4 * step + a) * 2], qb = q2[(4 * step + a) * 2 + 1];
                const uint32_t kh[4] = {kw.x, kw.y, kw.z, kw.w}, qv[4] = {qa.x, qa.y, qb.x, qb.y};
#pragma unroll
                for (int e = 0; e < 8; ++e) { acc[a][e] = fma_f16(half_of(kh, e), half_of(qv, e), acc[a][e]); }
            }
        }
        float u[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float lo = __fadd_rn(__fadd_rn(acc[0][e], acc[2][e]), __fadd_rn(acc[1][e], acc[3][e]));
            const float hi = __fadd_rn(__fadd_rn(acc[0][e + 4], acc[2][e + 4]), __fadd_rn(acc[1][e + 4], acc[3][e + 4]));
            u[e] = __fadd_rn(lo, hi);
        }
        const float simd = __fadd_rn(__fadd_rn(u[0], u[1]), __fadd_rn(u[2], u[3]));
        float tail = 0.f;                             // elements 96..127: scalar chain
        part(3);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const uint4 kw = kv[AHEAD ? 12 + a : a];
            const uint2 qa = q2[(12 + a) * 2], qb = q2[(12 + a) * 2 + 1];
            const uint32_t kh[4] = {kw.x, kw.y, kw.z, kw.w}, qv[4] = {qa.x, qa.y, qb.x, qb.y};
#pragma unroll
            for (int e = 0; e < 8; ++e) { tail = fma_f16(half_of(kh, e), half_of(qv, e), tail); }
        }
        sc[j] = __fadd_rn(tail, simd);
    }
    // The V^T values of the next PV steps are requested now (the K row's registers are free), so that they arrive
    // during the softmax instead of costing one memory round trip per 32 positions afterwards.
    if (!AHEAD) { request_v(0, n_vis, n_main, true); }
    constexpr int PV_AHEAD = AHEAD ? 6 : 0;
    constexpr int n_ahead = PV_AHEAD;
    uint2 v_ahead[AHEAD ? PV_AHEAD : 1][4];
#pragma unroll
    for (int s = 0; s < PV_AHEAD; ++s) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int j0 = 32 * (s + 1), j = j0 + 8 * a + 4 * pv_half;
            v_ahead[s][a] = (s < n_ahead && j0 < n_main && j < n_vis) ? *reinterpret_cast<const uint2 *>(vrow + j) : make_uint2(0u, 0u);
        }
    }
    __syncthreads();

    // ---- masked softmax: (score + mask) * scale, subtract the maximum, table exp, std::reduce, multiply by 1/sum
    float m = -CUDART_INF_F;
#pragma unroll 1
    for (int j = tid; j < n_vis; j += ATT_THREADS) {
        const float v = __fmul_rn(__fadd_rn(sc[j], 0.0f), p.scale);
        sc[j] = v;
        m = fmaxf(m, v);
    }
    m = warp_max(m);
    if (lane == 0) { red[warp] = m; }
    __syncthreads();
    m = red[0];
#pragma unroll
    for (int w = 1; w < ATT_WARPS; ++w) { m = fmaxf(m, red[w]); }
    const int n_tot4 = (n_tot + 3) & ~3;
#pragma unroll 1
    for (int j = tid; j < n_tot4; j += ATT_THREADS) { sc[j] = (j < n_vis) ? p.exp_table[f2h(__fsub_rn(sc[j], m))] : 0.f; }
    __syncthreads();
    // std::reduce: groups of four as (e0 + e1) + (e2 + e3), formed in parallel, then one thread's running sum; the
    // remainder (n_tot % 4 elements) is added one by one
#pragma unroll 1
    for (int g = tid; g < (n_tot >> 2); g += ATT_THREADS) {
        const float4 v = reinterpret_cast<const float4 *>(sc)[g];
        gs[g] = __fadd_rn(__fadd_rn(v.x, v.y), __fadd_rn(v.z, v.w));
    }
    __syncthreads();
    if (tid == 0) {
        float sum = 0.f;
        const int ng = n_tot >> 2;
        int g = 0;
#pragma unroll 1
        for (; g + 4 <= ng; g += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(gs + g);
            sum = __fadd_rn(sum, v.x); sum = __fadd_rn(sum, v.y); sum = __fadd_rn(sum, v.z); sum = __fadd_rn(sum, v.w);
        }
#pragma unroll 1
        for (; g < ng; ++g) { sum = __fadd_rn(sum, gs[g]); }
#pragma unroll 1
        for (int j = ng << 2; j < n_tot; ++j) { sum = __fadd_rn(sum, sc[j]); }
        bcast = __fdiv_rn(1.0f, sum);
    }
    __syncthreads();
    const float inv = bcast;
    // probabilities, rounded to fp16 as the PV MatMul does with its f32 operand
#pragma unroll 1
    for (int j = tid; j < n_vis; j += ATT_THREADS) { ph[j] = __float2half_rn(__fmul_rn(sc[j], inv)); }
    __syncthreads();

    // ---- out[e] = Dot<FP16,FP16>(V_t[e][0..n_tot), probs): a thread pair per element, thread `half` holding
    // elements 4 * half .. + 3 of the four accumulators. Masked positions have probability +0 and leave every
    // accumulator unchanged, so they are skipped (their cache entries may not be written yet).
    {
        const int e = pv_e, half = pv_half;
        float acc[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int k = 0; k < 4; ++k) { acc[a][k] = 0.f; }
        }
        auto pv_step = [&](const uint2 (&vv)[4], int j0) {
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int    j  = j0 + 8 * a + 4 * half;
                const uint2  pr = *reinterpret_cast<const uint2 *>(ph + j);
                if (j + 0 < n_vis) { acc[a][0] = fma_f16(vv[a].x, pr.x, acc[a][0]); }
                if (j + 1 < n_vis) { acc[a][1] = fma_f16(vv[a].x >> 16, pr.x >> 16, acc[a][1]); }
                if (j + 2 < n_vis) { acc[a][2] = fma_f16(vv[a].y, pr.y, acc[a][2]); }
                if (j + 3 < n_vis) { acc[a][3] = fma_f16(vv[a].y >> 16, pr.y >> 16, acc[a][3]); }
            }
        };
        if (0 < n_main) { pv_step(v_first, 0); }
#pragma unroll
        for (int s = 0; s < PV_AHEAD; ++s) {
            const int j0 = 32 * (s + 1);
            if (s < n_ahead && j0 < n_main && j0 < n_vis) { pv_step(v_ahead[s], j0); }
        }
        {   // later steps: loads one step ahead of the arithmetic
            int j0 = 32 * (n_ahead + 1);
            uint2 vv[4], vn[4];
            auto fetch = [&](uint2 (&dst)[4], int jj0) {
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const int j = jj0 + 8 * a + 4 * half;
                    dst[a] = (jj0 < n_main && j < n_vis) ? *reinterpret_cast<const uint2 *>(vrow + j) : make_uint2(0u, 0u);
                }
            };
            fetch(vv, j0);
#pragma unroll 1
            for (; j0 < n_main && j0 < n_vis; j0 += 32) {
                fetch(vn, j0 + 32);
                pv_step(vv, j0);
#pragma unroll
                for (int a = 0; a < 4; ++a) { vv[a] = vn[a]; }
            }
        }
        float u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float mine = __fadd_rn(__fadd_rn(acc[0][k], acc[2][k]), __fadd_rn(acc[1][k], acc[3][k]));
            u[k] = __fadd_rn(mine, __shfl_xor_sync(0xffffffffu, mine, 1));   // element k of one half with element k + 4 of the other
        }
        const float simd = __fadd_rn(__fadd_rn(u[0], u[1]), __fadd_rn(u[2], u[3]));
        // scalar tail: positions n_main .. n_tot-1 (at most 32)
        float tail = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int j = n_main + 4 * c;
            if (j < n_vis) {
                const uint2 pr = *reinterpret_cast<const uint2 *>(ph + j);
                tail = fma_f16(v_tail[c].x, pr.x, tail);
                if (j + 1 < n_vis) { tail = fma_f16(v_tail[c].x >> 16, pr.x >> 16, tail); }
                if (j + 2 < n_vis) { tail = fma_f16(v_tail[c].y, pr.y, tail); }
                if (j + 3 < n_vis) { tail = fma_f16(v_tail[c].y >> 16, pr.y >> 16, tail); }
            }
        }
        if (half == 0) { p.out[(int64_t)t * (p.out_stride ? p.out_stride : p.dl) + (int64_t)h * ATT_HD + e] = __fadd_rn(tail, simd); }
    }
    if (!LEAN) {
        tp_publish(p.tp, p.T);
        if (p.stamps != nullptr) { __syncthreads(); stamp(p.stamps, 3, true); }
    }
}

// ---------------------------------------------------------------------------------------------
// Long contexts (n_ctx > ATT_LONG_MIN) where attn_cluster_kernel does not apply, and prompts (token-tiled forms of the first and the
// last): the same arithmetic as attention_kernel, spread over the chip in three kernels
// that meet in a scratch buffer [T][n_head][n_ctx] of floats (scores, then probabilities):
//   attn_scores_kernel   one thread per (position, head, token): Dot<FP16,FP16>(K row, Q), all 32 accumulators in registers
//   attn_softmax_kernel  one CTA per (head, token): scale, maximum, table exp, std::reduce's grouped running sum, 1/sum,
//                        probabilities rounded to fp16
//   attn_pv_kernel       one warp per output element, lane = 8 * accumulator + element of the CPU's 4 x 8 accumulators
//                        (position j of a 32-step goes to lane j % 32), sixteen elements per CTA
// HBM-bound: the K rows and the V^T rows of the visible positions are read once (2 * n_kv * 128 * 2 bytes per head).
constexpr int ATT_LONG_MIN = 1024;

// Dot<FP16,FP16>(K row, Q): kv(a) is the row's 16-byte piece a, q_s the address of Q as f16 in shared memory. 4 x 8 accumulators over
// elements 0..95, the reduction tree, the scalar chain over elements 96..127, tail + simd
template <class KV>
__device__ __forceinline__ float score_dot(KV kv, uint32_t q_s) {
    float acc[4][8];
#pragma unroll
    for (int a = 0; a < 16; ++a) {               // elements 0..95: accumulator a % 4 takes elements 8 a .. 8 a + 7
        uint32_t kw[4], qw[4];
        *reinterpret_cast<uint4 *>(kw) = kv(a); *reinterpret_cast<uint4 *>(qw) = lds128(q_s + 16 * a);
        if (a < 12) {
#pragma unroll
            for (int e = 0; e < 8; ++e) { acc[a & 3][e] = fma_f16(half_of(kw, e), half_of(qw, e), a < 4 ? 0.f : acc[a & 3][e]); }
            continue;
        }
        if (a == 12) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float lo = __fadd_rn(__fadd_rn(acc[0][e], acc[2][e]), __fadd_rn(acc[1][e], acc[3][e]));
                const float hi = __fadd_rn(__fadd_rn(acc[0][e + 4], acc[2][e + 4]), __fadd_rn(acc[1][e + 4], acc[3][e + 4]));
                acc[0][e] = __fadd_rn(lo, hi);
            }
            acc[0][0] = __fadd_rn(__fadd_rn(acc[0][0], acc[0][1]), __fadd_rn(acc[0][2], acc[0][3]));
            acc[1][0] = 0.f;                     // elements 96..127: scalar chain
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) { acc[1][0] = fma_f16(half_of(kw, e), half_of(qw, e), acc[1][0]); }
    }
    return __fadd_rn(acc[1][0], acc[0][0]);
}

__global__ void __launch_bounds__(256) attn_scores_kernel(const AttnParams p) {
    __shared__ __align__(16) __half qh[ATT_HD];
    const int h = blockIdx.y, t = blockIdx.z, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    const bool batch = p.seq_stride != 0;
    const int n_vis = p.pos_base[0] + (batch ? 0 : t) + 1;
    if ((int)blockIdx.x * 256 >= n_vis) { return; }
    const int n_pad = (p.n_ctx + 3) & ~3;
    if (tid < ATT_HD) { qh[tid] = p.q[(int64_t)t * p.dl + (int64_t)h * ATT_HD + tid]; }
    __syncthreads();
    const int j = blockIdx.x * 256 + tid;
    if (j >= n_vis) { return; }
    uint4 kv[16];
    {
        const uint4 *krow = reinterpret_cast<const uint4 *>(p.k_cache + (batch ? (int64_t)t * p.seq_stride : 0) + (int64_t)j * p.dl + (int64_t)h * ATT_HD);
#pragma unroll
        for (int a = 0; a < 16; ++a) { kv[a] = krow[a]; }
    }
    p.scratch[((int64_t)t * p.n_head + h) * n_pad + j] = score_dot([&](int a) { return kv[a]; }, smem_u32(qh));
}

// The same for a prompt, register-tiled: a CTA takes ATT_SG times ATT_ST tokens x ATT_SP positions of a head, a lane 4 tokens x 8
// positions at a time. The 32 accumulators of a dot product are walked element by element of the CPU's eight-wide vectors: element e of
// the four accumulators takes the twelve values 32 s + 8 a + e (s = 0..2, a = 0..3), four chains of three FMAs, so that only one to
// three partial sums per output live at a time instead of 32 accumulators. K and Q lie in shared memory as f16 in that order, value by
// value: [value][position] and [value][token].
// 160 f32 operations per (token, position, head). Shared memory gives a warp one word per lane and cycle however often an address
// repeats, so a word has to serve several products: 32 products per 6 words here. Bound: the FMA pipes, busy 61 % (eight warps an SM, 237
// registers). 128 tokens of 32 heads over 2000 positions on average: 67 us (f32 copies of K and Q, 4 x 4 outputs a lane, 16 products per 8
// words: 83; the 5000 FMAs of a tile unrolled, beyond the instruction caches: 87; one K row per thread: 180).
constexpr int ATT_TT = 8;                                    // tokens per CTA of the PV kernel below
constexpr int ATT_ST = 32, ATT_SP = 128, ATT_KPITCH = ATT_SP + 8, ATT_SC_THREADS = 128;
constexpr int ATT_SG = 2;                                    // token tiles a CTA walks with the same K rows
constexpr size_t ATT_SC_SMEM = (size_t)ATT_HD * (ATT_KPITCH + ATT_SG * ATT_ST) * sizeof(__half);
// value 8 c + e of a row -> its place: 12 e + c for the first 96, then 96 + 4 ((e + 1) % 8) + c - 12 (the rotation keeps the pieces c = 8..15
// of a row on different banks when they are stored side by side)
__host__ __device__ constexpr int att_value_row(int c, int e) { return c < 12 ? 12 * e + c : 96 + 4 * ((e + 1) & 7) + c - 12; }
__global__ void __launch_bounds__(ATT_SC_THREADS, 2) attn_scores_tiled_kernel(const AttnParams p) {
    extern __shared__ __align__(16) float att_smem[];
    constexpr int NQ = ATT_SG * ATT_ST;
    __half *ks = reinterpret_cast<__half *>(att_smem), *qs = ks + ATT_HD * ATT_KPITCH;
    const int h = blockIdx.y, tg = blockIdx.z * NQ, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    pdl_wait();
    const int ng = min(NQ, p.T - tg), j0 = blockIdx.x * ATT_SP;
    const int n_vis_last = p.pos_base[0] + tg + ng;          // positions the last token of the CTA sees
    if (j0 >= n_vis_last) { return; }
    const int n_pad = (p.n_ctx + 3) & ~3;
    {   // a warp reads four pairs of neighbouring rows x 128 bytes at a time and writes the pairs value by value (the pitch keeps the 8 x 4 words of a store on 32 banks)
        const int row0 = 2 * (tid >> 3), c0 = tid & 7;       // 16-byte pieces c0 and c0 + 8 of rows row0 + 32 i, row0 + 32 i + 1
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int c = c0 + 8 * half;
            const __half *src = p.k_cache + (int64_t)(j0 + row0) * p.dl + (int64_t)h * ATT_HD + 8 * c;
            uint4 w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = 32 * (i >> 1) + (i & 1);
                w[i] = j0 + row0 + r < n_vis_last ? *reinterpret_cast<const uint4 *>(src + (int64_t)r * p.dl) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                __half *dst = ks + att_value_row(c, e) * ATT_KPITCH + row0;
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const uint32_t a = e < 2 ? w[i].x : e < 4 ? w[i].y : e < 6 ? w[i].z : w[i].w, b = e < 2 ? w[i + 1].x : e < 4 ? w[i + 1].y : e < 6 ? w[i + 1].z : w[i + 1].w;
                    *reinterpret_cast<uint32_t *>(dst + 16 * i) = __byte_perm(a, b, (e & 1) ? 0x7632 : 0x5410);
                }
            }
        }
        static_assert(ATT_SC_THREADS == 8 * 16 && ATT_SP == 16 * 8, "eight pieces x 16 pairs of rows, four times");
    }
    {   // a lane takes 16-byte pieces of one token: a store's 32 halves are neighbours
        static_assert(ATT_ST == 32, "one token per lane and tile");
#pragma unroll
        for (int i = 0; i < 4 * ATT_SG; ++i) {
            const int c = 4 * (i & 3) + warp, tok = (i >> 2) * ATT_ST + lane;
            const uint4 v = *reinterpret_cast<const uint4 *>(p.q + (int64_t)(tg + min(tok, ng - 1)) * p.dl + (int64_t)h * ATT_HD + 8 * c);   // (tokens past the end repeat the last one; their scores are not stored)
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) { qs[att_value_row(c, e) * NQ + tok] = __ushort_as_half((uint16_t)half_of(w, e)); }
        }
    }
    __syncthreads();
    // warps side by side: 64 positions and 16 tokens each; lanes: 8 x 8 positions, 4 x 4 tokens
    const int jl = (warp & 1) * 64 + (lane & 7) * 8;
    if (j0 + (warp & 1) * 64 >= n_vis_last) { return; }
    const uint32_t k_s = smem_u32(ks + jl);
#pragma unroll 1
    for (int tw = (warp >> 1) * 16; tw < ng; tw += ATT_ST) {
        const int tl = tw + (lane >> 3) * 4;
        const uint32_t q_s = smem_u32(qs + tl);
        struct Row { uint32_t k[4], q[2]; };
        auto row = [&](int base, int r) {                    // place base + r
            Row x;
            const uint4 v = lds128(k_s + 2u * base * ATT_KPITCH + 2u * r * ATT_KPITCH);
            x.k[0] = v.x; x.k[1] = v.y; x.k[2] = v.z; x.k[3] = v.w;
            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(x.q[0]), "=r"(x.q[1]) : "r"(q_s + 2u * base * NQ + 2u * r * NQ));
            return x;
        };
        // u_e = v_e + v_(e + 4), then (u_0 + u_1) + (u_2 + u_3); rolled loops: the whole is 5000 FMAs, which would not stay in the instruction caches
        float out[4][8], sum[4][8];                          // [token][position]
#pragma unroll 1
        for (int e = 0; e < 4; ++e) {
            float u[4][8];
#pragma unroll
            for (int hi = 0; hi < 2; ++hi) {                 // elements e and e + 4
                float v[4][8];
#pragma unroll
                for (int ap = 0; ap < 2; ++ap) {             // accumulators ap and ap + 2
                    float x[4][8];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float a[4][8];
#pragma unroll
                        for (int s = 0; s < 3; ++s) {
                            const Row r = row(12 * e, att_value_row(4 * s + ap + 2 * i, 4 * hi));
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
#pragma unroll
                                for (int j = 0; j < 8; ++j) { a[t][j] = fma_f16(half_of(r.k, j), half_of(r.q, t), s == 0 ? 0.f : a[t][j]); }
                            }
                        }
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
#pragma unroll
                            for (int j = 0; j < 8; ++j) { x[t][j] = i == 0 ? a[t][j] : __fadd_rn(x[t][j], a[t][j]); }
                        }
                    }
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) { v[t][j] = ap == 0 ? x[t][j] : __fadd_rn(v[t][j], x[t][j]); }
                    }
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) { u[t][j] = hi == 0 ? v[t][j] : __fadd_rn(u[t][j], v[t][j]); }
                }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (e & 1) { const float w = __fadd_rn(sum[t][j], u[t][j]); out[t][j] = e == 1 ? w : __fadd_rn(out[t][j], w); }
                    else { sum[t][j] = u[t][j]; }
                }
            }
        }
        float tail[4][8];                                    // elements 96..127: scalar chain
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
            for (int j = 0; j < 8; ++j) { tail[t][j] = 0.f; }
        }
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const Row r = row(c, att_value_row(12, e));
#pragma unroll
                for (int t = 0; t < 4; ++t) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) { tail[t][j] = fma_f16(half_of(r.k, j), half_of(r.q, t), tail[t][j]); }
                }
            }
        }
        // (scores of positions a token does not see are written as they come: nothing reads them)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
            for (int j4 = 0; j4 < 8; j4 += 4) {
                const int j = j0 + jl + j4;
                if (tl + t < ng && j < n_vis_last && j < n_pad) {
                    *reinterpret_cast<float4 *>(p.scratch + ((int64_t)(tg + tl + t) * p.n_head + h) * n_pad + j) =
                        make_float4(__fadd_rn(tail[t][j4], out[t][j4]), __fadd_rn(tail[t][j4 + 1], out[t][j4 + 1]), __fadd_rn(tail[t][j4 + 2], out[t][j4 + 2]), __fadd_rn(tail[t][j4 + 3], out[t][j4 + 3]));
                }
            }
        }
    }
}

constexpr int ATT_SM_THREADS = 1024;
__global__ void __launch_bounds__(ATT_SM_THREADS) attn_softmax_kernel(const AttnParams p) {
    extern __shared__ __align__(16) float att_smem[];
    __shared__ float red[ATT_SM_THREADS / WARP];
    __shared__ float bcast;
    const int h = blockIdx.x, t = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int nthr = ATT_SM_THREADS;
    pdl_launch_dependents();
    pdl_wait();
    const bool batch = p.seq_stride != 0;
    const int n_vis = p.pos_base[0] + (batch ? 0 : t) + 1;
    const int n_tot = batch ? n_vis : (p.pos_base[1] > 0) ? p.pos_base[1] : p.pos_base[0] + p.T;
    const int n_pad = (p.n_ctx + 3) & ~3;
    float *sc = att_smem, *gs = sc + n_pad;
    float *row = p.scratch + ((int64_t)t * p.n_head + h) * n_pad;
    // masked softmax: (score + mask) * scale, subtract the maximum, table exp, std::reduce, multiply by 1/sum
    float m = -CUDART_INF_F;
    for (int j = tid; j < n_vis; j += nthr) {
        const float v = __fmul_rn(__fadd_rn(row[j], 0.0f), p.scale);
        sc[j] = v;
        m = fmaxf(m, v);
    }
    m = warp_max(m);
    if (lane == 0) { red[warp] = m; }
    __syncthreads();
    m = red[0];
#pragma unroll
    for (int w = 1; w < ATT_SM_THREADS / WARP; ++w) { m = fmaxf(m, red[w]); }
    // (masked positions are exact zeros: they decide which elements form a group of four, but a group of zeros leaves the sum as it is,
    // so the groups behind the last visible position are left out)
    const int n_sum = min(n_tot, (n_vis + 3) & ~3), n_sum4 = (n_sum + 3) & ~3;
    for (int j = tid; j < n_sum4; j += nthr) { sc[j] = (j < n_vis) ? p.exp_table[f2h(__fsub_rn(sc[j], m))] : 0.f; }
    __syncthreads();
    const int ng = min(n_tot >> 2, n_sum4 >> 2);
    for (int g = tid; g < ng; g += nthr) {
        const float4 v = reinterpret_cast<const float4 *>(sc)[g];
        gs[g] = __fadd_rn(__fadd_rn(v.x, v.y), __fadd_rn(v.z, v.w));
    }
    __syncthreads();
    if (tid == 0) {
        float sum = 0.f;
        int g = 0;
        for (; g + 4 <= ng; g += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(gs + g);
            sum = __fadd_rn(sum, v.x); sum = __fadd_rn(sum, v.y); sum = __fadd_rn(sum, v.z); sum = __fadd_rn(sum, v.w);
        }
        for (; g < ng; ++g) { sum = __fadd_rn(sum, gs[g]); }
        for (int j = ng << 2; j < n_sum; ++j) { sum = __fadd_rn(sum, sc[j]); }
        bcast = __fdiv_rn(1.0f, sum);
    }
    __syncthreads();
    const float inv = bcast;
    // probabilities, rounded to fp16 as the PV MatMul does with its f32 operand
    for (int j = tid; j < n_vis; j += nthr) { row[j] = __half2float(__float2half_rn(__fmul_rn(sc[j], inv))); }
}

// The same for a token of a prompt, in front of the tiled PV kernel: four neighbouring positions per thread and pass, whose exponentials are
// one of std::reduce's groups; the running sum of the groups on the CTA's four warps (running_sum_wide). The probabilities become f16
// values in the first half of the row - all of it is in shared memory by then - with zeros behind the last position, as far as a PV tile
// reads. Up to ten CTAs per SM (contexts below some 3900; nine at 4096, five at 8192: the shared memory is that of the whole context): one CTA's sum
// overlaps the others' passes. Bound: the gathers from the table of exponentials, 20 to 30 lines of
// L1 a warp. 128 tokens of 32 heads over 2000 positions on average: 36 -> 33 us.
constexpr int ATT_SMT_THREADS = 128;
static_assert(ATT_SMT_THREADS == RS_THREADS, "all warps form the running sum");
__host__ __device__ static inline size_t att_smt_smem(int n_ctx) { const size_t n4 = ((size_t)n_ctx + 3) / 4; return (4 * n4 + (n4 + 3) / 4 * 4 + rs_scratch_words(4)) * sizeof(float); }
__global__ void __launch_bounds__(ATT_SMT_THREADS, 10) attn_softmax_tiled_kernel(const AttnParams p) {
    extern __shared__ __align__(16) float att_smem[];
    __shared__ float red[ATT_SMT_THREADS / WARP], inv_s;
    const int h = blockIdx.x, t = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_pad = (p.n_ctx + 3) & ~3;
    float4 *sc4 = reinterpret_cast<float4 *>(att_smem);
    float  *gs = att_smem + n_pad, *rs = gs + ((n_pad >> 2) + 3) / 4 * 4;
    pdl_launch_dependents();
    pdl_wait();
    const int n_vis = p.pos_base[0] + t + 1;
    const int n_tot = (p.pos_base[1] > 0) ? p.pos_base[1] : p.pos_base[0] + p.T;
    float *row = p.scratch + ((int64_t)t * p.n_head + h) * n_pad;
    const int n4 = (n_vis + 3) >> 2;
    // masked softmax: (score + mask) * scale, subtract the maximum, table exp, std::reduce, multiply by 1/sum
    float m = -CUDART_INF_F;
    for (int g = tid; g < n4; g += ATT_SMT_THREADS) {
        const float4 x = reinterpret_cast<const float4 *>(row)[g];
        const int left = n_vis - 4 * g;
        auto scaled = [&](float s, int i) { return i < left ? __fmul_rn(__fadd_rn(s, 0.0f), p.scale) : -CUDART_INF_F; };
        const float4 v = make_float4(scaled(x.x, 0), scaled(x.y, 1), scaled(x.z, 2), scaled(x.w, 3));
        sc4[g] = v;
        m = fmaxf(m, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
    }
    m = warp_max(m);
    if (lane == 0) { red[warp] = m; }
    __syncthreads();
    m = red[lane & (ATT_SMT_THREADS / WARP - 1)];
#pragma unroll
    for (int o = ATT_SMT_THREADS / WARP / 2; o > 0; o >>= 1) { m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o)); }
    // (masked positions are exact zeros: they decide which elements form a group of four, but a group of zeros leaves the sum as it is,
    // so the groups behind the last visible position are left out)
    for (int g = tid; g < n4; g += ATT_SMT_THREADS) {
        const float4 v = sc4[g];
        const int left = n_vis - 4 * g;
        auto ex = [&](float s, int i) { return i < left ? p.exp_table[f2h(__fsub_rn(s, m))] : 0.f; };
        const float4 e = make_float4(ex(v.x, 0), ex(v.y, 1), ex(v.z, 2), ex(v.w, 3));
        sc4[g] = e;
        gs[g] = __fadd_rn(__fadd_rn(e.x, e.y), __fadd_rn(e.z, e.w));
    }
    __syncthreads();
    const int n_sum = min(n_tot, 4 * n4), ng = min(n_tot >> 2, n4);
    const float sum4 = running_sum_wide(smem_u32(gs), ng, smem_u32(rs), rs_scratch_words(4), tid, 1);
    if (tid == 0) {
        float sum = sum4;
        for (int j = ng << 2; j < n_sum; ++j) { sum = __fadd_rn(sum, att_smem[j]); }
        inv_s = __fdiv_rn(1.0f, sum);
    }
    __syncthreads();
    const float inv = inv_s;
    uint2 *row16 = reinterpret_cast<uint2 *>(row);   // probabilities, rounded to fp16 as the PV MatMul does with its f32 operand
    const int n_read = min(n_pad, (n_vis + ATT_TT - 1 + 31) & ~31) >> 2;
    for (int g = tid; g < n_read; g += ATT_SMT_THREADS) {
        uint2 v = make_uint2(0u, 0u);
        if (g < n4) {
            const float4 e = sc4[g];
            auto prob = [inv](float x) { return (uint32_t)__half_as_ushort(__float2half_rn(__fmul_rn(x, inv))); };
            v = make_uint2(prob(e.x) | (prob(e.y) << 16), prob(e.z) | (prob(e.w) << 16));
        }
        row16[g] = v;
    }
}

constexpr int ATT_PV_WARPS = 16;
__global__ void __launch_bounds__(ATT_PV_WARPS * WARP) attn_pv_kernel(const AttnParams p) {
    extern __shared__ __align__(16) float att_smem[];
    const int per_head = ATT_HD / ATT_PV_WARPS;
    const int h = blockIdx.x / per_head, e = (blockIdx.x % per_head) * ATT_PV_WARPS + (threadIdx.x >> 5), t = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31;
    pdl_launch_dependents();
    pdl_wait();
    const bool batch = p.seq_stride != 0;
    const int n_vis = p.pos_base[0] + (batch ? 0 : t) + 1;
    const int n_tot = batch ? n_vis : (p.pos_base[1] > 0) ? p.pos_base[1] : p.pos_base[0] + p.T;
    const int n_pad = (p.n_ctx + 3) & ~3;
    const int n_main = ((n_tot - 1) / 32) * 32;
    float *pr = att_smem;
    const float *row = p.scratch + ((int64_t)t * p.n_head + h) * n_pad;
    for (int j = tid; j < n_vis; j += ATT_PV_WARPS * WARP) { pr[j] = row[j]; }
    __syncthreads();
    // out[e] = Dot<FP16,FP16>(V_t[e][0..n_tot), probs); masked positions have probability +0 and leave every accumulator
    // unchanged, so they are skipped (their cache entries may not be written yet)
    const __half *vrow = p.v_cache + (batch ? (int64_t)t * p.seq_stride : 0) + ((int64_t)h * ATT_HD + e) * p.n_ctx;
    float acc = 0.f;
    int j0 = 0;
    for (; j0 + 8 * 32 <= n_main && j0 + 8 * 32 <= n_vis; j0 += 8 * 32) {   // eight steps' loads in flight
        float v[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) { v[s] = __half2float(vrow[j0 + 32 * s + lane]); }
#pragma unroll
        for (int s = 0; s < 8; ++s) { acc = fmaf(v[s], pr[j0 + 32 * s + lane], acc); }
    }
    for (; j0 < n_main; j0 += 32) {
        const int j = j0 + lane;
        if (j < n_vis) { acc = fmaf(__half2float(vrow[j]), pr[j], acc); }
    }
    acc = reduce_f16dot_lanes(acc);
    const float vt = (n_main + lane < n_vis) ? __half2float(vrow[n_main + lane]) : 0.f;
    float tail = 0.f;                         // positions n_main .. n_tot-1 (at most 32): scalar chain
#pragma unroll 1
    for (int i = 0; i < 32; ++i) {
        const float v = __shfl_sync(0xffffffffu, vt, i);
        if (n_main + i < n_vis) { tail = fmaf(v, pr[n_main + i], tail); }
    }
    if (lane == 0) { p.out[(int64_t)t * (p.out_stride ? p.out_stride : p.dl) + (int64_t)h * ATT_HD + e] = __fadd_rn(tail, acc); }
    tp_publish(p.tp, p.T);
}

// ---------------------------------------------------------------------------------------------
// A step over a long context in one kernel: ATL_C CTAs (a cluster) take a head. Each CTA scores its quarter of the positions, the quarters'
// exponentials meet in every CTA's shared memory, each CTA forms the softmax sum (its order allows no split) and then its quarter of the
// head's output elements over all positions. Same arithmetic as attention_kernel. HBM-bound: K and V^T are read once. Four warps copy
// both through one ring of stages (32 K rows of 256 bytes, or 512 positions of eight V^T rows) without regard to the phases: while the
// softmax is formed, V^T fills the ring. (cp.async, 512 bytes an instruction: bulk copies of a row each cost the warp 50 cycles, 54 us in all.) A stage is filled for one warp: no CTA-wide waits on the way.
// 32 heads over 4000 positions, three kernels (scores, softmax, PV) before: 41 us, now about 22; the reads take 10.3.
// (Q as f16 and products of f16 values by one instruction, stages counted by shifts, the other CTAs' rows mapped once: steps of eight layers, Q8_0 at 3968
// positions 520.4 -> 518.4 us, Q4_0 at 250 335.3 -> 333.4, at 900 355.9 -> 353.7.)
constexpr int ATL_C = 4, ATL_WARPS = 8, ATL_COPY_WARPS = 4, ATL_THREADS = (ATL_WARPS + ATL_COPY_WARPS) * WARP;
constexpr int ATL_KPITCH = 272, ATL_VCH = 512, ATL_VROWS = 8, ATL_VPITCH = 2 * ATL_VCH + 64, ATL_STAGE = 32 * ATL_KPITCH;   // pitches without bank conflicts
static_assert(ATL_VROWS * ATL_VPITCH == ATL_STAGE && ATL_C * 4 * ATL_VROWS == ATT_HD, "both kinds of stages fill the slot; four warps take a CTA's elements");
// Which warps meet in a slot of the ring: a barrier's parity tells a phase only from its neighbours, so a warp may wait for a slot's next phase
// only when it knows the one before to be complete. Slot g % NS therefore always has the same copy warp (NS is a multiple of their number)
// and, K stage after K stage and V stage after V stage, the same reader (NS is a multiple of the score warps, of which small rings use
// fewer); between the two kinds lies the exchange of the exponentials, which follows every K stage.
constexpr int ATL_MAX_STAGES = 16, ATL_MIN_STAGES = 4;   // 4, 8 or 16
__host__ __device__ constexpr int atl_copy_warp(int g) { return g % ATL_COPY_WARPS; }
__host__ __device__ constexpr int atl_score_warps(int ns) { return ns < ATL_WARPS ? ns : ATL_WARPS; }
__host__ __device__ constexpr int atl_reader(int g, int nK, int ns) { return g < nK ? g % atl_score_warps(ns) : (g - nK) & 3; }
struct AtlSmem { size_t ex, gs, rs, red, bars, ring; };   // gs: the sums of four, then the probabilities as f16
__host__ __device__ static inline AtlSmem atl_smem(int n_ctx) {   // offsets in bytes; q lies in front
    const size_t n32 = ((size_t)n_ctx + 31) & ~(size_t)31;
    AtlSmem L;
    L.ex = ATT_HD * 2; L.gs = L.ex + n32 * 4; L.rs = L.gs + 2 * n32; L.red = L.rs + rs_scratch_words(4) * 4; L.bars = L.red + (ATL_C * ATL_WARPS + 4) * 4;
    L.ring = (L.bars + (2 * ATL_MAX_STAGES + 2) * 8 + 127) / 128 * 128;
    return L;
}
__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(__cvta_generic_to_global(src)) : "memory");
}
__device__ __forceinline__ void atl_wait(uint32_t bar, uint32_t parity, uint64_t &limit_ns) {
    if (mbar_try_wait(bar, parity)) { return; }
    if (limit_ns == 0 || !mbar_wait_prompt(bar, parity, limit_ns)) { limit_ns = 0; }
}

__global__ void __launch_bounds__(ATL_THREADS, 2) attn_cluster_kernel(const AttnParams p, const int ns_log) {
    const int NS = 1 << ns_log;
    extern __shared__ __align__(128) uint8_t atl_raw[];
    const AtlSmem L = atl_smem(p.n_ctx);
    __half *qh = reinterpret_cast<__half *>(atl_raw);
    float *ex = reinterpret_cast<float *>(atl_raw + L.ex), *gs = reinterpret_cast<float *>(atl_raw + L.gs);
    float *rs = reinterpret_cast<float *>(atl_raw + L.rs), *red = reinterpret_cast<float *>(atl_raw + L.red);
    const uint32_t ring_s = smem_u32(atl_raw + L.ring), full_s = smem_u32(atl_raw + L.bars), empty_s = full_s + 8 * ATL_MAX_STAGES;
    const uint32_t max_s = empty_s + 8 * ATL_MAX_STAGES, exp_s = max_s + 8;
    const int h = blockIdx.x / ATL_C, rank = blockIdx.x % ATL_C, t = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int i = 0; i < NS; ++i) { mbar_init(full_s + 8 * i, WARP); mbar_init(empty_s + 8 * i, 1); }
        mbar_init(max_s, ATL_C * ATL_WARPS); mbar_init(exp_s, ATL_C * ATL_WARPS);
        mbar_init_fence();
    }
    cluster_sync();   // every CTA of the cluster is there, its barriers too
    pdl_wait();
    const bool batch = p.seq_stride != 0;
    const int n_vis = p.pos_base[0] + (batch ? 0 : t) + 1;
    const int n_tot = batch ? n_vis : (p.pos_base[1] > 0) ? p.pos_base[1] : p.pos_base[0] + p.T;
    const int slice = ((n_vis + ATL_C * 32 - 1) / (ATL_C * 32)) * 32, start = rank * slice;
    const int cnt = max(0, min(slice, n_vis - start)), nK = (cnt + 31) >> 5, nC = (n_vis + ATL_VCH - 1) / ATL_VCH;
    uint64_t limit = WAIT_LIMIT_NS;
    if (warp >= ATL_WARPS) {
        const __half *K = p.k_cache + (batch ? (int64_t)t * p.seq_stride : 0) + (int64_t)start * p.dl + (int64_t)h * ATT_HD;
        const __half *V = p.v_cache + (batch ? (int64_t)t * p.seq_stride : 0) + ((int64_t)h * ATT_HD + rank * (ATT_HD / ATL_C)) * p.n_ctx;
        const int total = nK + 4 * nC;
        for (int g = warp - ATL_WARPS; g < total; g += ATL_COPY_WARPS) {   // (atl_copy_warp)
            const int slot = g & (NS - 1);
            if (g >= NS) { atl_wait(empty_s + 8 * slot, (uint32_t)((g >> ns_log) - 1) & 1u, limit); }
            if (!__all_sync(0xffffffffu, limit != 0)) { break; }
            const uint32_t bar = full_s + 8 * slot, dst = ring_s + slot * ATL_STAGE;
            if (g < nK) {
                const __half *row = K + (int64_t)(32 * g + (lane >> 4)) * p.dl + (lane & 15) * 8;
                const int rows = cnt - 32 * g - (lane >> 4);
#pragma unroll
                for (int i = 0; i < 16; ++i) { if (2 * i < rows) { cp_async16(dst + (2 * i + (lane >> 4)) * ATL_KPITCH + (lane & 15) * 16, row + (int64_t)2 * i * p.dl); } }
            } else {
                const int c = (g - nK) >> 2, w = (g - nK) & 3;
                const __half *row = V + (int64_t)(w * ATL_VROWS) * p.n_ctx + c * ATL_VCH + lane * 8;
                const int left = n_vis - c * ATL_VCH - lane * 8;   // (a whole piece lies inside the row: n_ctx is a multiple of 8)
#pragma unroll
                for (int i = 0; i < 16; ++i) { if ((i & 1) * 256 < left) { cp_async16(dst + (i >> 1) * ATL_VPITCH + (i & 1) * 512 + lane * 16, row + (int64_t)(i >> 1) * p.n_ctx + (i & 1) * 256); } }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");   // no copy is in flight when the CTA ends, also when its readers gave up
    } else {
        if (tid < ATT_HD) { qh[tid] = p.q[(int64_t)t * p.dl + (int64_t)h * ATT_HD + tid]; }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        // scores of this CTA's positions, a tile of 32 per warp, a position per lane
        float m = -CUDART_INF_F;
        const int n_score = atl_score_warps(NS);
        for (int k = warp; warp < n_score && k < nK; k += n_score) {   // (atl_reader)
            const int slot = k & (NS - 1);
            atl_wait(full_s + 8 * slot, (uint32_t)(k >> ns_log) & 1u, limit);
            const uint32_t src = ring_s + slot * ATL_STAGE + lane * ATL_KPITCH;
            const float s = score_dot([=](int a) { return lds128(src + 16 * a); }, smem_u32(qh));
            __syncwarp();
            if (lane == 0) { mbar_arrive(empty_s + 8 * slot); }
            const int  j = 32 * k + lane;
            const float v = j < cnt ? __fmul_rn(__fadd_rn(s, 0.0f), p.scale) : -CUDART_INF_F;
            ex[start + j] = v;
            m = fmaxf(m, v);
        }
        m = warp_max(m);
        __syncwarp();   // (the warp's scores are read by others when small rings have fewer score warps)
        if (lane < ATL_C) {
            cluster_store(cluster_map(smem_u32(red + rank * ATL_WARPS + warp), lane), m);
            cluster_arrive(cluster_map(max_s, lane));
        }
        cluster_wait(max_s, 0u, limit);
        m = warp_max(red[lane]);
        // exponentials and their sums of four, to all CTAs of the cluster
        uint32_t there[ATL_C];   // the rows `ex` of the CTAs
#pragma unroll
        for (int r = 0; r < ATL_C; ++r) { there[r] = cluster_map(smem_u32(ex), r); }
#pragma unroll 1
        for (int k0 = warp; k0 < nK; k0 += 4 * ATL_WARPS) {
            float e[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int j = 32 * (k0 + i * ATL_WARPS) + lane;
                e[i] = j < cnt ? p.exp_table[f2h(__fsub_rn(ex[start + j], m))] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int k = k0 + i * ATL_WARPS, j = 32 * k + lane;
                if (k < nK) {   // uniform in the warp
                    const float two = __fadd_rn(e[i], __shfl_xor_sync(0xffffffffu, e[i], 1)), four = __fadd_rn(two, __shfl_xor_sync(0xffffffffu, two, 2));
                    const uint32_t to = 4u * (start + j), to4 = (uint32_t)(L.gs - L.ex) + start + j;   // (4 bytes per four values)
#pragma unroll
                    for (int r = 0; r < ATL_C; ++r) {
                        cluster_store(there[r] + to, e[i]);
                        if ((lane & 3) == 0) { cluster_store(there[r] + to4, four); }
                    }
                }
            }
        }
        __syncwarp();
        if (lane < ATL_C) { cluster_arrive(cluster_map(exp_s, lane)); }
        cluster_wait(exp_s, 0u, limit);
        // std::reduce: groups of four, in order; masked positions are exact zeros that decide which elements form a group
        const int n_sum = min(n_tot, (n_vis + 3) & ~3), ng = min(n_tot >> 2, (n_vis + 3) >> 2);
        if (warp < RS_THREADS / WARP) {
            float sum = running_sum_wide(smem_u32(gs), ng, smem_u32(rs), rs_scratch_words(4), tid, 1);
            if (tid == 0) {
                for (int j = ng << 2; j < n_sum; ++j) { sum = __fadd_rn(sum, ex[j]); }
                red[ATL_C * ATL_WARPS] = __fdiv_rn(1.0f, sum);
            }
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        const float inv = red[ATL_C * ATL_WARPS];
        auto prob = [inv](float e) { return (uint32_t)__half_as_ushort(__float2half_rn(__fmul_rn(e, inv))); };   // as the PV MatMul rounds its f32 operand
        for (int g = tid; g < (n_vis + 3) >> 2; g += ATL_WARPS * WARP) {
            const float4 e = reinterpret_cast<const float4 *>(ex)[g];
            reinterpret_cast<uint2 *>(gs)[g] = make_uint2(prob(e.x) | (prob(e.y) << 16), prob(e.z) | (prob(e.w) << 16));
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        // PV: accumulators 8 (lane % 4) .. + 7 of row lane / 4 of the warp's eight (position j of a 32-step belongs to accumulator j % 32)
        if (warp < 4) {
            const int n_main = ((n_tot - 1) / 32) * 32, n_full = min(n_main, n_vis) >> 5;
            const int q = lane & 3;
            const uint32_t pr_s = smem_u32(gs);
            float acc[8], tail = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) { acc[i] = 0.f; }
            auto step = [&](uint32_t v_s, int pos, int valid) {
                uint32_t vw[4], pw[4];
                *reinterpret_cast<uint4 *>(vw) = lds128(v_s); *reinterpret_cast<uint4 *>(pw) = lds128(pr_s + 2 * pos);
#pragma unroll
                for (int i = 0; i < 8; ++i) { if (i < valid) { acc[i] = fma_f16(vw[i >> 1] >> (16 * (i & 1)), pw[i >> 1] >> (16 * (i & 1)), acc[i]); } }
            };
            for (int c = 0; c < nC; ++c) {
                const int g = nK + 4 * c + warp, slot = g & (NS - 1);
                atl_wait(full_s + 8 * slot, (uint32_t)(g >> ns_log) & 1u, limit);
                const uint32_t row = ring_s + slot * ATL_STAGE + (lane >> 2) * ATL_VPITCH;
                const int p0 = c * ATL_VCH, steps = min(ATL_VCH / 32, n_full - c * (ATL_VCH / 32));
#pragma unroll 4
                for (int s = 0; s < steps; ++s) { step(row + s * 64 + q * 16, p0 + s * 32 + q * 8, 8); }
                const int part = n_full * 32;   // a step that the causal limit cuts (several tokens in a pass)
                if (part >= p0 && part < p0 + ATL_VCH && part < n_main && part < n_vis) { step(row + (part - p0) * 2 + q * 16, part + q * 8, n_vis - part - q * 8); }
                if (n_main >= p0 && n_main < p0 + ATL_VCH) {   // positions n_main .. : scalar chain (at most 32)
                    const int n = n_vis - n_main;
                    for (int i0 = 0; i0 < n; i0 += 8) {
                        uint32_t vw[4], pw[4];
                        *reinterpret_cast<uint4 *>(vw) = lds128(row + (n_main - p0 + i0) * 2); *reinterpret_cast<uint4 *>(pw) = lds128(pr_s + 2 * (n_main + i0));
#pragma unroll
                        for (int i = 0; i < 8; ++i) { if (i0 + i < n) { tail = fma_f16(vw[i >> 1] >> (16 * (i & 1)), pw[i >> 1] >> (16 * (i & 1)), tail); } }
                    }
                }
                __syncwarp();
                if (lane == 0) { mbar_arrive(empty_s + 8 * slot); }
            }
            float u[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) {   // FP16::block_reduce: (s0 + s2) + (s1 + s3), then elements e and e + 4, then the two pair steps
                acc[i] = __fadd_rn(acc[i], __shfl_xor_sync(0xffffffffu, acc[i], 2));
                acc[i] = __fadd_rn(acc[i], __shfl_xor_sync(0xffffffffu, acc[i], 1));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) { u[i] = __fadd_rn(acc[i], acc[i + 4]); }
            const float simd = __fadd_rn(__fadd_rn(u[0], u[1]), __fadd_rn(u[2], u[3]));
            if (q == 0) {
                p.out[(int64_t)t * (p.out_stride ? p.out_stride : p.dl) + (int64_t)h * ATT_HD + rank * (ATT_HD / ATL_C) + warp * ATL_VROWS + (lane >> 2)] = __fadd_rn(tail, simd);
            }
        }
    }
    if (limit == 0 && p.error_flag != nullptr) { atomicExch(p.error_flag, 1); }   // a copy or a CTA of the cluster did not arrive
    cluster_sync();   // no CTA ends while another may still write into its shared memory
}

// PV for a prompt: a CTA takes ATT_PVT_ELEMS output elements of a head for ATT_TT consecutive tokens. The 32 accumulators of an output
// (position j of a 32-step belongs to accumulator j % 32) lie in the registers of eight lanes, four each, so that a lane reads four
// neighbouring positions at once (64 bits of V^T, 128 bits of a token's probabilities); a lane takes two output elements, a warp eight,
// for all ATT_TT tokens. The eight lanes of an output meet once at the end, halving the number of tokens a lane keeps at every step of
// the tree, and each lane then runs the scalar tails of its token.
// 128 f32 operations per (token, position, head). V^T and the probabilities (f16; the softmax kernel leaves zeros behind a token's last
// position, as far as a tile reads) of ATT_CH positions at a time run through a ring in shared memory with cp.async; a lane takes four
// elements of V^T for eight tokens, 24 words of shared memory per 128 products. Bound: instruction issue (73 %; the FMA pipes 53 %).
// 128 tokens of 32 heads over 2000 positions on average: 73 us (f32 probabilities and two elements a lane, whose V^T came straight from
// L1: 101; whole rows staged first, one CTA per SM: 119).
constexpr int ATT_PVT_WARPS = 4, ATT_EE = 4, ATT_PVT_ELEMS = ATT_PVT_WARPS * 4 * ATT_EE;
constexpr int ATT_CH = 128, ATT_CH_RING = 3, ATT_VPITCH = 2 * ATT_CH + 16;   // bytes: the rows of two lane groups lie on different banks
constexpr size_t ATT_PV_STAGE = (size_t)ATT_PVT_ELEMS * ATT_VPITCH + ATT_TT * 2 * ATT_CH, ATT_PV_SMEM = ATT_CH_RING * ATT_PV_STAGE;
__global__ void __launch_bounds__(ATT_PVT_WARPS * WARP, 3) attn_pv_tiled_kernel(const AttnParams p) {
    extern __shared__ __align__(16) float att_smem[];
    constexpr int PER_HEAD = ATT_HD / ATT_PVT_ELEMS, THREADS = ATT_PVT_WARPS * WARP;
    const int h = blockIdx.x / PER_HEAD, t0 = blockIdx.y * ATT_TT, tid = threadIdx.x, lane = tid & 31, grp = lane >> 3, lg = lane & 7;
    const int el = (tid >> 5) * 4 * ATT_EE + grp * ATT_EE, e0 = (blockIdx.x % PER_HEAD) * ATT_PVT_ELEMS + el;   // the lane's first element, in the CTA and in the head
    pdl_launch_dependents();
    pdl_wait();
    const int nt = min(ATT_TT, p.T - t0);
    const int n_tot = (p.pos_base[1] > 0) ? p.pos_base[1] : p.pos_base[0] + p.T;
    const int n_pad = (p.n_ctx + 3) & ~3;
    const int n_main = ((n_tot - 1) / 32) * 32;
    const int vis0 = p.pos_base[0] + t0 + 1;                  // positions token t0 + tt sees: vis0 + tt
    const int vis_last = vis0 + nt - 1;
    const int n_steps = (min(n_main, vis_last) + 31) >> 5;    // (steps behind the tile's last visible position add nothing)
    // staged: all visible positions, with the scalar tails' (n_main .. n_tot - 1) in the last chunk, and what the steps read behind them
    const int n_chunks = (vis_last + ATT_CH - 1) / ATT_CH, staged = max(vis_last, 32 * n_steps);
    const __half *vrow = p.v_cache + ((int64_t)h * ATT_HD + e0 - el) * p.n_ctx;   // the CTA's first row
    const int64_t row_pitch = 2 * (int64_t)p.n_head * n_pad;  // (tokens past the end repeat the last one; their results are not stored)
    const __half *rows = reinterpret_cast<const __half *>(p.scratch + ((int64_t)t0 * p.n_head + h) * n_pad);
    const uint32_t ring = smem_u32(att_smem);
    const bool wide = (p.n_ctx & 7) == 0 && (reinterpret_cast<uintptr_t>(p.v_cache) & 15) == 0;   // V^T rows lie on 16 bytes, else on 8
    auto stage = [&](int c) {   // one commit group per chunk, empty ones behind the last
        if (c < n_chunks) {
            const uint32_t dst = ring + (uint32_t)(c % ATT_CH_RING) * (uint32_t)ATT_PV_STAGE;
            if (wide) {
#pragma unroll
                for (int i = 0; i < ATT_PVT_ELEMS * ATT_CH / 8 / THREADS; ++i) {
                    const int q = tid + i * THREADS, e = q >> 4, j = 8 * (q & 15);
                    if (c * ATT_CH + j < staged) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + e * ATT_VPITCH + 2 * j), "l"(__cvta_generic_to_global(vrow + (int64_t)e * p.n_ctx + c * ATT_CH + j)) : "memory"); }
                }
            } else {
#pragma unroll 4
                for (int i = 0; i < ATT_PVT_ELEMS * ATT_CH / 4 / THREADS; ++i) {
                    const int q = tid + i * THREADS, e = q >> 5, j = 4 * (q & 31);
                    if (c * ATT_CH + j < staged) { asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + e * ATT_VPITCH + 2 * j), "l"(__cvta_generic_to_global(vrow + (int64_t)e * p.n_ctx + c * ATT_CH + j)) : "memory"); }
                }
            }
            const int tt = tid >> 4, j = 8 * (tid & 15);      // (a row of probabilities has room for twice n_pad f16 values)
            if (c * ATT_CH + j < staged) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + ATT_PVT_ELEMS * ATT_VPITCH + tt * 2 * ATT_CH + 2 * j), "l"(__cvta_generic_to_global(rows + min(tt, nt - 1) * row_pitch + c * ATT_CH + j)) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    static_assert(THREADS == ATT_TT * ATT_CH / 8, "one piece of the probabilities per thread");
#pragma unroll
    for (int c = 0; c < ATT_CH_RING - 1; ++c) { stage(c); }
    float acc[ATT_TT][ATT_EE][4];
#pragma unroll
    for (int tt = 0; tt < ATT_TT; ++tt) {
#pragma unroll
        for (int ee = 0; ee < ATT_EE; ++ee) {
#pragma unroll
            for (int k = 0; k < 4; ++k) { acc[tt][ee][k] = 0.f; }
        }
    }
    auto lds64 = [](uint32_t addr, uint32_t (&w)[2]) { asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr)); };
    for (int c = 0; c < n_chunks; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ATT_CH_RING - 2) : "memory");
        __syncthreads();                                      // chunk c is there for everyone, and everyone is done with chunk c - 1
        stage(c + ATT_CH_RING - 1);
        const uint32_t v_s = ring + (uint32_t)(c % ATT_CH_RING) * (uint32_t)ATT_PV_STAGE + el * ATT_VPITCH + 8 * lg;
        const uint32_t p_s = ring + (uint32_t)(c % ATT_CH_RING) * (uint32_t)ATT_PV_STAGE + ATT_PVT_ELEMS * ATT_VPITCH + 8 * lg;
        const int steps = min(ATT_CH / 32, n_steps - c * (ATT_CH / 32));
#pragma unroll 1
        for (int s = 0; s < steps; ++s) {
            uint32_t v[ATT_EE][2];
#pragma unroll
            for (int ee = 0; ee < ATT_EE; ++ee) { lds64(v_s + ee * ATT_VPITCH + 64 * s, v[ee]); }
            const int over = c * ATT_CH + 32 * s + 4 * lg + 4 - vis_last;   // (cache entries behind the last visible position may not be written yet)
            if (over > 0) {
#pragma unroll
                for (int ee = 0; ee < ATT_EE; ++ee) {
                    if (over >= 1) { v[ee][1] &= 0xffffu; }
                    if (over >= 2) { v[ee][1] = 0u; }
                    if (over >= 3) { v[ee][0] &= 0xffffu; }
                    if (over >= 4) { v[ee][0] = 0u; }
                }
            }
#pragma unroll
            for (int tt = 0; tt < ATT_TT; ++tt) {
                uint32_t pv[2];
                lds64(p_s + tt * 2 * ATT_CH + 64 * s, pv);
#pragma unroll
                for (int ee = 0; ee < ATT_EE; ++ee) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) { acc[tt][ee][k] = fma_f16(half_of(v[ee], k), half_of(pv, k), acc[tt][ee][k]); }
                }
            }
        }
    }
    // FP16::block_reduce (vec_util.h:61-71): lane lg holds accumulator lg / 2, elements 4 (lg % 2) .. + 3. (s0 + s2) + (s1 + s3) are the
    // exchanges with lanes lg ^ 4 and lg ^ 2, element l with l + 4 the one with lg ^ 1. At each exchange a lane hands over half of its
    // tokens and keeps the sums of the others: in the end lane lg holds token lg.
#pragma unroll
    for (int half = ATT_TT / 2; half > 0; half >>= 1) {       // 4, 2, 1: also the lane distance
        const bool up = (lg & half) != 0;
#pragma unroll
        for (int tt = 0; tt < half; ++tt) {
#pragma unroll
            for (int ee = 0; ee < ATT_EE; ++ee) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float keep = up ? acc[tt + half][ee][k] : acc[tt][ee][k], give = up ? acc[tt][ee][k] : acc[tt + half][ee][k];
                    acc[tt][ee][k] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, half));
                }
            }
        }
    }
    static_assert(ATT_TT == 8, "one lane of a group of eight per token");
    // the scalar tails (positions n_main .. n_tot - 1, at most 32, as far as the lane's token sees them; in the last chunk), one FMA chain per output
    if (lg >= nt) { return; }
    const int n_tail = min(32, vis0 + lg - n_main);
    const uint32_t last = ring + (uint32_t)((n_chunks - 1) % ATT_CH_RING) * (uint32_t)ATT_PV_STAGE + 2 * (n_main % ATT_CH);
    float tail[ATT_EE] = {};
    for (int i = 0; i < n_tail; i += 4) {
        uint32_t q[2];
        lds64(last + ATT_PVT_ELEMS * ATT_VPITCH + lg * 2 * ATT_CH + 2 * i, q);
#pragma unroll
        for (int ee = 0; ee < ATT_EE; ++ee) {
            uint32_t w[2];
            lds64(last + (el + ee) * ATT_VPITCH + 2 * i, w);
#pragma unroll
            for (int k = 0; k < 4; ++k) { if (i + k < n_tail) { tail[ee] = fma_f16(half_of(w, k), half_of(q, k), tail[ee]); } }
        }
    }
    float *dst = p.out + (int64_t)(t0 + lg) * (p.out_stride ? p.out_stride : p.dl) + (int64_t)h * ATT_HD + e0;
#pragma unroll
    for (int ee = 0; ee < ATT_EE; ++ee) {
        const float vec = __fadd_rn(__fadd_rn(acc[0][ee][0], acc[0][ee][1]), __fadd_rn(acc[0][ee][2], acc[0][ee][3]));
        dst[ee] = __fadd_rn(tail[ee], vec);
    }
}

static cudaError_t launch_with_pdl(const void *kernel, dim3 grid, dim3 block, size_t smem, const AttnParams &p, const LaunchCfg &cfg) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid; lc.blockDim = block; lc.dynamicSmemBytes = smem; lc.stream = cfg.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr; lc.numAttrs = cfg.pdl ? 1 : 0;
    void *args[] = {const_cast<AttnParams *>(&p)};
    return cudaLaunchKernelExC(&lc, kernel, args);
}

// the cluster kernel: single steps and batches, whole 16-byte pieces of the cache rows, ATL_MIN_STAGES stages beside the exponentials
// (contexts up to 31,840 positions). One CTA per SM with a deep ring while all fit so, else two with eight stages each where they fit.
static int atl_stage_count(int n_ctx, int64_t ctas, int num_sms) {
    const size_t fixed = atl_smem(n_ctx).ring;
    auto stages = [&](size_t b) {
        for (int ns = ATL_MAX_STAGES; ns >= ATL_MIN_STAGES; ns /= 2) { if (fixed + (size_t)ns * ATL_STAGE <= b) { return ns; } }
        return 0;
    };
    const int ns = stages(ctas <= num_sms ? 224 * 1024 : 112 * 1024);
    return ns >= 8 ? ns : stages(224 * 1024);
}
static int atl_stages(const AttnParams &p, const LaunchCfg &cfg) { return atl_stage_count(p.n_ctx, (int64_t)ATL_C * p.n_head * p.T, cfg.num_sms); }
// host-only: 0 when, for every ring that the rule above gives, a slot's successive stages have one copy warp and, within K and within V, one reader
int attn_ring_selftest() {
    for (int ctas = 4; ctas <= 4096; ctas *= 8) {
        for (int n_ctx = 8; n_ctx <= 40000; n_ctx += 8) {
            const int ns = atl_stage_count(n_ctx, ctas, 140);
            if (ns == 0) { continue; }
            if (ns > ATL_MAX_STAGES || atl_smem(n_ctx).ring + (size_t)ns * ATL_STAGE > 224 * 1024) { return 101; }
            for (int nK = 0; nK <= 2 * ns; ++nK) {
                for (int g = 0; g < nK + 3 * ns; ++g) {
                    if (atl_copy_warp(g) != atl_copy_warp(g + ns)) { return 102; }
                    if ((g < nK) == (g + ns < nK) && atl_reader(g, nK, ns) != atl_reader(g + ns, nK, ns)) { return 103; }
                }
            }
        }
    }
    return 0;
}
static bool atl_fits(const AttnParams &p, const LaunchCfg &cfg) {
    return (p.T < ATT_TT || p.seq_stride != 0) && p.tp.counter == nullptr && (p.n_ctx & 7) == 0 && (p.seq_stride & 7) == 0 &&
           (((uintptr_t)p.k_cache | (uintptr_t)p.v_cache) & 15) == 0 && atl_stages(p, cfg) >= ATL_MIN_STAGES;
}
static cudaError_t launch_attn_cluster(const AttnParams &p, const LaunchCfg &cfg) {
    int ns = atl_stages(p, cfg);
    const size_t smem = atl_smem(p.n_ctx).ring + (size_t)ns * ATL_STAGE;
    cudaError_t err = allow_dynamic_smem(reinterpret_cast<const void *>(attn_cluster_kernel), smem);
    if (err != cudaSuccess) { return err; }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(ATL_C * p.n_head), (unsigned)p.T); lc.blockDim = dim3(ATL_THREADS); lc.dynamicSmemBytes = smem; lc.stream = cfg.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ATL_C; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr; lc.numAttrs = cfg.pdl ? 2 : 1;
    AttnParams q = p;
    if (q.error_flag == nullptr) { q.error_flag = cfg.error_flag; }
    int ns_log = ns == 16 ? 4 : ns == 8 ? 3 : 2;   // (atl_stage_count: 4, 8 or 16)
    void *args[] = {&q, &ns_log};
    return cudaLaunchKernelExC(&lc, reinterpret_cast<const void *>(attn_cluster_kernel), args);
}

size_t attention_scratch_floats(int n_ctx, int n_head, int T) {   // 0: the single-kernel path serves this context length
    if (n_ctx <= ATT_LONG_MIN) { return 0; }
    return (size_t)T * n_head * (((size_t)n_ctx + 3) & ~(size_t)3);
}

// Whether the steps of a model read the cache rows of earlier steps before they wait for the QKV kernel. One attention CTA fills an SM, and the
// mat-vec grids leave eight SMs free: CTAs of further heads start when a QKV CTA ends and hide nothing. The CTAs of the K-quant kernel end together,
// and with up to 24 heads, where V^T's rows do not begin on lines (reads of eight bytes past L1 then take more sectors), the late reads cost more than
// the early ones save. Steps of 4 layers, us, reads behind the wait / early, behind 20, 60, 220 positions. A context of 844: Q4_K_M 8 heads 104.7 /
// 103.2, 106.5 / 103.4, 113.1 / 107.5; 12 heads 110.8 / 112.1, 113.1 / 114.7, 122.3 / 130.0; 20 heads 158.7 / 159.2, 160.7 / 161.8, 170.2 / 176.9; 32 heads 192.5 /
// 191.7, 194.0 / 192.5, 203.8 / 201.5; Q4_0 12 heads 99.3 / 98.3, 101.1 / 99.6, 107.2 / 107.8. A context of 512: Q4_K_M 12 heads 111.6 / 111.1, 113.6 / 111.9, 123.6 /
// 128.3; 24 heads 170.2 / 167.9, 172.3 / 168.9, 184.1 / 185.3. (With the kernels as they are, 8 layers, a context of 844, behind 10, 150 and 215: 10 heads
// 185.2 / 184.0, 199.8 / 202.7, 209.1 / 217.8; 16 heads 206.8 / 206.9, 222.1 / 222.1, 231.2 / 237.4; 24 heads 293.4 / 292.3, 311.4 / 311.4, 324.9 / 330.9.)
int attention_early(int n_head, int n_ctx, bool kq) { return !kq || n_head <= 8 || n_head > 24 || n_ctx % 64 == 0 ? 1 : 0; }

// The form for a single token at position pos, where both kernels take the context. A layer's attention, us, one CTA a head / a cluster of four, 32
// heads: position 8: 4.8 / 7.5; 100: 5.3 / 8.0; 250: 8.2 / 8.2; 460: 14.3 / 8.9; 900: 28 / 10.7. The line for other numbers of heads, from steps
// of 8-layer models with little beside the attention, us a layer: 2 heads 248: 17.7 / 18.2, 280: 18.7 / 18.4; 8 heads 248: 20.6 / 21.4, 280: 21.5 / 21.5;
// 16 heads 216: 24.9 / 24.7, 248: 25.5 / 24.7; 24 heads 248: 29.0 / 29.1, 280: 29.9 / 29.3; 32 heads 248: 32.0 / 32.5, 280: 33.1 / 32.7; 40 heads 248:
// 41.7 / 42.2, 280: 42.7 / 42.5. They meet between 210 (16 heads) and 280: 240 is off by at most 4 % of such a layer.
// (With the kernels as they are, steps of 8 layers at 220: Q4_0 8 heads 161.5 / 169.9, 16 209.3 / 207.8, 24 249.8 / 254.5, 32 302.4 / 307.6, 40 403.4 / 407.1;
// Q4_K_M 204.5 / 201.2, 235.4 / 225.4, 327.4 / 320.5, 361.1 / 361.6, 507.3 / 494.9; at 190 one CTA is ahead or level everywhere.)
constexpr int ATT_CLUSTER_POS = 240, ATT_ONE_CTA_CTX = 8192;   // (the rows of the longest context: 57 KB)
int attention_form(const AttnParams &p, const LaunchCfg &cfg, int pos) {
    if (p.T != 1 || p.seq_stride != 0 || p.n_ctx > ATT_ONE_CTA_CTX || !atl_fits(p, cfg)) { return ATT_BY_CONTEXT; }
    return pos < ATT_CLUSTER_POS ? ATT_ONE_CTA : ATT_CLUSTER;
}

cudaError_t launch_attention(const AttnParams &p, const LaunchCfg &cfg) {
    if (p.hd != ATT_HD || p.T < 1 || p.n_ctx < 1 || (p.n_ctx & 3) || (p.dl & 7)) { return cudaErrorInvalidValue; }
    const size_t n_pad = ((size_t)p.n_ctx + 3) & ~(size_t)3;
    if (p.form == ATT_CLUSTER && atl_fits(p, cfg)) { return launch_attn_cluster(p, cfg); }
    if (p.form != ATT_ONE_CTA && (p.n_ctx > ATT_LONG_MIN || p.force_long) && p.scratch != nullptr) {
        if (atl_fits(p, cfg)) { return launch_attn_cluster(p, cfg); }
        // a prompt: tokens share the K rows and the V^T rows, read in pieces of 16 (K, Q) and 8 bytes (V^T); Q and V^T of any other alignment go
        // through the kernels that read them value by value
        const bool tiled = p.T >= ATT_TT && p.tp.counter == nullptr && p.seq_stride == 0 && ((uintptr_t)p.q & 15) == 0 && ((uintptr_t)p.v_cache & 7) == 0;
        cudaError_t err = tiled ? allow_dynamic_smem(reinterpret_cast<const void *>(attn_scores_tiled_kernel), ATT_SC_SMEM) : cudaSuccess;
        if (err != cudaSuccess) { return err; }
        err = tiled
            ? launch_with_pdl(reinterpret_cast<const void *>(attn_scores_tiled_kernel), dim3((unsigned)((p.n_ctx + ATT_SP - 1) / ATT_SP), p.n_head, (unsigned)((p.T + ATT_SG * ATT_ST - 1) / (ATT_SG * ATT_ST))), dim3(ATT_SC_THREADS), ATT_SC_SMEM, p, cfg)
            : launch_with_pdl(reinterpret_cast<const void *>(attn_scores_kernel), dim3((unsigned)((p.n_ctx + 255) / 256), p.n_head, p.T), dim3(256), 0, p, cfg);
        if (err != cudaSuccess) { return err; }
        const void  *softmax = tiled ? reinterpret_cast<const void *>(attn_softmax_tiled_kernel) : reinterpret_cast<const void *>(attn_softmax_kernel);
        const size_t sm_smem = tiled ? att_smt_smem(p.n_ctx) : (n_pad + n_pad / 4) * sizeof(float) + 16;
        if ((n_pad + n_pad / 4) * sizeof(float) + 16 > 200 * 1024) { return cudaErrorInvalidValue; }
        err = allow_dynamic_smem(softmax, sm_smem);
        if (err != cudaSuccess) { return err; }
        err = launch_with_pdl(softmax, dim3(p.n_head, p.T), dim3(tiled ? ATT_SMT_THREADS : ATT_SM_THREADS), sm_smem, p, cfg);
        if (err != cudaSuccess) { return err; }
        if (tiled) {
            err = allow_dynamic_smem(reinterpret_cast<const void *>(attn_pv_tiled_kernel), ATT_PV_SMEM);
            if (err != cudaSuccess) { return err; }
            return launch_with_pdl(reinterpret_cast<const void *>(attn_pv_tiled_kernel), dim3(p.n_head * (ATT_HD / ATT_PVT_ELEMS), (unsigned)((p.T + ATT_TT - 1) / ATT_TT)), dim3(ATT_PVT_WARPS * WARP), ATT_PV_SMEM, p, cfg);
        }
        const size_t pv_smem = n_pad * sizeof(float) + 16;
        err = allow_dynamic_smem(reinterpret_cast<const void *>(attn_pv_kernel), pv_smem);
        if (err != cudaSuccess) { return err; }
        return launch_with_pdl(reinterpret_cast<const void *>(attn_pv_kernel), dim3(p.n_head * (ATT_HD / ATT_PV_WARPS), p.T), dim3(ATT_PV_WARPS * WARP), pv_smem, p, cfg);
    }
    const size_t smem = (n_pad + (n_pad / 4 + 3) / 4 * 4) * sizeof(float) + (n_pad + ATT_HD) * sizeof(__half) + 16;   // (contexts of up to ATT_ONE_CTA_CTX positions; longer ones have a scratch)
    if (smem > 200 * 1024) { return cudaErrorInvalidValue; }
    const bool many = (int64_t)p.n_head * p.T > device_sms();
    const void *kernel = reinterpret_cast<const void *>(many ? attention_kernel<false, ATT_MANY, false> : !(p.early && p.T == 1 && p.seq_stride == 0) ? attention_kernel<false, 1, false>
                                                          : p.stamps == nullptr && p.tp.counter == nullptr ? attention_kernel<true, 1, true> : attention_kernel<true, 1, false>);
    cudaError_t err = allow_dynamic_smem(kernel, smem);
    if (err != cudaSuccess) { return err; }
    return launch_with_pdl(kernel, dim3(p.n_head, p.T, 1), dim3(ATT_THREADS), smem, p, cfg);
}

// =============================================================================================
// upload-time re-tiling: raw 18-byte / 34-byte blocks -> the record stream described at DevMatrix
// (one thread per padded block; blocks beyond nb are written as zeros with a zero scale)
template <int WORDS, bool MMA>   // WORDS 4: Q4_0 (16 nibble bytes), 8: Q8_0 (32 int8 values); MMA: the fragment-ordered record of DevMatrix::mma
__global__ void retile_kernel(const uint8_t *raw, int64_t row_stride, int64_t n_rows, int nb, int nbp, uint8_t *base, int tile_rows,
                              int64_t dst_row0, int64_t src_row0, int sub_rows, int sub_off) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows * nbp) { return; }
    const int64_t  lrow = i / nbp;
    const int      b = (int)(i - lrow * nbp);
    const uint8_t *src = raw + lrow * row_stride + (int64_t)b * (2 + 4 * WORDS);
    const bool     real = b < nb;
    constexpr int  ROWB = WORDS * 32 + 16;
    const int64_t  srow = src_row0 + lrow;
    const int64_t  row  = dst_row0 + (sub_rows > 0 ? (srow / sub_rows) * tile_rows + sub_off + srow % sub_rows : srow);
    const int      r    = (int)(row % tile_rows);
    uint8_t  *rec = base + ((row / tile_rows) * (nbp >> 3) + (b >> 3)) * ((int64_t)tile_rows * ROWB);
    const uint16_t d = real ? (uint16_t)(src[0] | (src[1] << 8)) : (uint16_t)0;
    const int      grp_bytes = tile_rows * WORDS * 16;   // MMA: quants of one group of four blocks, all rows of the tile
    if (MMA) { reinterpret_cast<uint16_t *>(rec + 2 * grp_bytes + r * 16)[b & 7] = d; }
    else     { reinterpret_cast<uint16_t *>(rec + r * ROWB + WORDS * 32)[b & 7] = d; }
#pragma unroll
    for (int k = 0; k < WORDS; ++k) {
        uint32_t v = real ? (uint32_t)(src[2 + 4 * k] | (src[3 + 4 * k] << 8) | (src[4 + 4 * k] << 16) | ((uint32_t)src[5 + 4 * k] << 24)) : 0u;
        if (WORDS == 4) { v ^= 0x88888888u; }
        if (MMA) {   // [group][half of the block][row][word of the half] x 16 B, the four blocks of the group side by side
            reinterpret_cast<uint32_t *>(rec + ((b >> 2) & 1) * grp_bytes + (((k >> 2) * tile_rows + r) * 4 + (k & 3)) * 16)[b & 3] = v;
        } else {
            reinterpret_cast<uint32_t *>(rec + r * ROWB + ((b >> 2) & 1) * (WORDS * 16))[(b & 3) + 4 * k] = v;
        }
    }
}

cudaError_t launch_retile(int type, const uint8_t *raw, int64_t row_stride, int64_t n_rows, int nb, uint8_t *matrix_base, int tile_rows, bool mma,
                          int64_t dst_row0, int64_t src_row0, int sub_rows, int sub_off, cudaStream_t s) {
    const int     nbp = padded_blocks(nb);
    const int64_t n = n_rows * nbp;
    if (n == 0) { return cudaSuccess; }
    if (tile_rows != 4 && tile_rows != 8 && tile_rows != 16 && tile_rows != 32) { return cudaErrorInvalidValue; }
    if (mma && tile_rows != 8 && tile_rows != 16) { return cudaErrorInvalidValue; }
    const unsigned grid = (unsigned)((n + 255) / 256);
    if (type == 2) {
        if (mma) { retile_kernel<4, true><<<grid, 256, 0, s>>>(raw, row_stride, n_rows, nb, nbp, matrix_base, tile_rows, dst_row0, src_row0, sub_rows, sub_off); }
        else     { retile_kernel<4, false><<<grid, 256, 0, s>>>(raw, row_stride, n_rows, nb, nbp, matrix_base, tile_rows, dst_row0, src_row0, sub_rows, sub_off); }
    } else if (type == 8) {
        if (mma) { retile_kernel<8, true><<<grid, 256, 0, s>>>(raw, row_stride, n_rows, nb, nbp, matrix_base, tile_rows, dst_row0, src_row0, sub_rows, sub_off); }
        else     { retile_kernel<8, false><<<grid, 256, 0, s>>>(raw, row_stride, n_rows, nb, nbp, matrix_base, tile_rows, dst_row0, src_row0, sub_rows, sub_off); }
    } else { return cudaErrorNotSupported; }
    return launch_check();
}

// =============================================================================================
// Q8_0 quantizer writing the reference's 34-byte blocks (backend/host/include/simd/vec_convert.h:178-261)
__global__ void quantize_q8_0_ref_kernel(const float *x, int64_t n4, uint8_t *blocks) {
    const int64_t base = (int64_t)blockIdx.x * blockDim.x;
    const int64_t g    = base + threadIdx.x;
    const bool    valid = g < n4;
    const float4  v = valid ? reinterpret_cast<const float4 *>(x)[g] : make_float4(0.f, 0.f, 0.f, 0.f);
    uint16_t dh; int s;
    const uint32_t q = quantize_q8_lane4(v, dh, s);
    if (!valid) { return; }
    uint8_t *o = blocks + (g >> 3) * 34;
    const int li = (int)(g & 7);
    if (li == 0) { o[0] = (uint8_t)(dh & 0xff); o[1] = (uint8_t)(dh >> 8); }
    o[2 + 4 * li] = (uint8_t)(q & 0xff); o[3 + 4 * li] = (uint8_t)((q >> 8) & 0xff);
    o[4 + 4 * li] = (uint8_t)((q >> 16) & 0xff); o[5 + 4 * li] = (uint8_t)(q >> 24);
}

cudaError_t launch_quantize_q8_0_ref_layout(const float *x, int64_t n, uint8_t *blocks, cudaStream_t s) {
    if (n % QK != 0) { return cudaErrorInvalidValue; }
    if (n == 0) { return cudaSuccess; }
    const int64_t n4 = n / 4;
    quantize_q8_0_ref_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, s>>>(x, n4, blocks);
    return launch_check();
}

// per-block int32 dots through the same device functions the mat-vec uses (one thread per block)
__global__ void block_dots_kernel(int wtype, const uint8_t *w, const uint8_t *xb, int64_t nblk, int32_t *out) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nblk) { return; }
    const uint8_t *y = xb + b * 34 + 2;
    uint32_t yw[8];
    for (int k = 0; k < 8; ++k) {
        yw[k] = y[4 * k] | (y[4 * k + 1] << 8) | (y[4 * k + 2] << 16) | ((uint32_t)y[4 * k + 3] << 24);
    }
    int total = 0;
    if (wtype == 2) {
        const uint8_t *q = w + b * 18 + 2;
        for (int k = 0; k < 4; ++k) {
            const uint32_t ww = q[4 * k] | (q[4 * k + 1] << 8) | (q[4 * k + 2] << 16) | ((uint32_t)q[4 * k + 3] << 24);
            const float hi = lane_sum16_q4_0(ww ^ 0x88888888u, 1u, yw[4 + k]);   // both come scaled by 16
            const float lo = lane_sum16_q4_0(ww ^ 0x88888888u, 16u, yw[k]);
            total += (int)hi / 16 + (int)lo / 16;
        }
    } else {
        const uint8_t *q = w + b * 34 + 2;
        for (int k = 0; k < 8; ++k) {
            const uint32_t ww = q[4 * k] | (q[4 * k + 1] << 8) | (q[4 * k + 2] << 16) | ((uint32_t)q[4 * k + 3] << 24);
            total += (int)lane_sum_q8_0(ww, yw[k]);
        }
    }
    out[b] = total;
}

cudaError_t launch_block_dots(int wtype, const uint8_t *w_row, const uint8_t *x_blocks, int64_t n, int32_t *out, cudaStream_t s) {
    if ((wtype != 2 && wtype != 8) || n % QK != 0) { return cudaErrorInvalidValue; }
    const int64_t nblk = n / QK;
    if (nblk == 0) { return cudaSuccess; }
    block_dots_kernel<<<(unsigned)((nblk + 127) / 128), 128, 0, s>>>(wtype, w_row, x_blocks, nblk, out);
    return launch_check();
}

// =============================================================================================
// K-quant weights (Q4_K: 144 B / 256 elements, Q6_K: 210 B / 256 elements; layouts
// orchestration/include/number/number_impl/k-quant.h:79-117, 162-188). The reference defines only the block layouts
// and has no compute for them, so there is nothing to be bit-identical to: the kernel multiplies the decoded weights
// with the f32 activations (the reference's MatMul semantics without an activation quantizer) and is checked against
// a numpy decode within the stated tolerance. One warp per output row and column; a lane decodes 8 consecutive
// elements of every 256-element super-block, so a warp reads each 144 / 210-byte block once, contiguously.
// HBM-bound: rows * K/256 * 144 (210) bytes per launch; activations stay in L2.
__device__ __forceinline__ void kq_scale_min_k4(const uint8_t *sc12, int j, float &sc, float &mn) {
    if (j < 4) { sc = (float)(sc12[j] & 63); mn = (float)(sc12[4 + j] & 63); }
    else { sc = (float)((sc12[4 + j] & 0xF) | ((sc12[j - 4] >> 6) << 4)); mn = (float)((sc12[4 + j] >> 4) | ((sc12[j] >> 6) << 4)); }
}

template <int TYPE>   // 12: Q4_K, 14: Q6_K
__global__ void __launch_bounds__(256) matmul_kquant_kernel(const uint8_t *w, int64_t row_bytes, const float *x, float *out, int64_t n_rows,
                                                            int64_t k, int64_t n_cols) {
    const int     lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t nsb = k >> 8;
    for (int64_t item = gw; item < n_rows * n_cols; item += nw) {
        const int64_t  row = item % n_rows, col = item / n_rows;
        const uint8_t *wr = w + row * row_bytes;
        const float   *xc = x + col * k;
        float acc = 0.f;
        for (int64_t b = 0; b < nsb; ++b) {
            const float4 x0 = *reinterpret_cast<const float4 *>(xc + b * 256 + lane * 8), x1 = *reinterpret_cast<const float4 *>(xc + b * 256 + lane * 8 + 4);
            const float  xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
            if (TYPE == 12) {
                const uint8_t *blk = wr + b * 144;
                const float d = h2f((uint16_t)(blk[0] | (blk[1] << 8))), dmin = h2f((uint16_t)(blk[2] | (blk[3] << 8)));
                // elements 8*lane .. 8*lane+7 lie in sub-block j = lane / 4; 64-element group g = j / 2 keeps its first 32
                // elements in the low nibbles and the next 32 in the high nibbles of bytes 32g .. 32g+31
                const int j = lane >> 2, g = j >> 1, hi = j & 1, off = (lane & 3) * 8;
                float sc, mn; kq_scale_min_k4(blk + 4, j, sc, mn);
                const uint2 q = *reinterpret_cast<const uint2 *>(blk + 16 + 32 * g + off);
                const float dl = __fmul_rn(d, sc), ml = __fmul_rn(dmin, mn);
                float part = 0.f, xs = 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint32_t byte = ((e < 4 ? q.x : q.y) >> (8 * (e & 3))) & 0xff;
                    part = fmaf((float)(hi ? (byte >> 4) : (byte & 0xF)), xv[e], part);
                    xs += xv[e];
                }
                acc += dl * part - ml * xs;
            } else {
                const uint8_t *blk = wr + b * 210;
                const float d = h2f((uint16_t)(blk[208] | (blk[209] << 8)));
                // element i = 8*lane + e: half h = i / 128, quarter qq = (i % 128) / 32, l = i % 32; six bits =
                // nibble of ql[64h + 32(qq & 1) + l] (low for qq < 2, high else) | two bits (2*qq) of qh[32h + l]
                const int i0 = lane * 8, h = i0 >> 7, qq = (i0 & 127) >> 5, l0 = i0 & 31;
                const uint8_t *ql = blk + 64 * h + 32 * (qq & 1) + l0;   // 210-byte blocks: only 2-byte alignment holds, byte loads
                const uint8_t *qh = blk + 128 + 32 * h + l0;
                const float sc = (float)(int8_t)blk[192 + (i0 >> 4)];
                float part = 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint32_t byte = ql[e];
                    const int      six  = (int)((qq < 2 ? (byte & 0xF) : (byte >> 4)) | (((qh[e] >> (2 * qq)) & 3) << 4)) - 32;
                    part = fmaf((float)six, xv[e], part);
                }
                acc += __fmul_rn(d, sc) * part;
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) { out[col * n_rows + row] = acc; }
    }
}

cudaError_t launch_matmul_kquant(int type, const uint8_t *w, int64_t n_rows, int64_t k, const float *x, int64_t n_cols, float *out, cudaStream_t s) {
    if ((type != 12 && type != 14) || k % 256 != 0) { return cudaErrorInvalidValue; }
    if (n_rows == 0 || n_cols == 0) { return cudaSuccess; }
    const int64_t warps = n_rows * n_cols;
    const unsigned grid = (unsigned)std::min<int64_t>((warps + 7) / 8, 148 * 8);
    if (type == 12) { matmul_kquant_kernel<12><<<grid, 256, 0, s>>>(w, k / 256 * 144, x, out, n_rows, k, n_cols); }
    else            { matmul_kquant_kernel<14><<<grid, 256, 0, s>>>(w, k / 256 * 210, x, out, n_rows, k, n_cols); }
    return launch_check();
}

// =============================================================================================
// per-operator kernels (each mirrors one OperatorImpl of backend/host/operator/*.cpp)

// OperatorNormRMSImpl::execute, non-linear.cpp:194-223; one CTA per row. Sum of squares in the order of
// std::transform_reduce: (x0^2 + x1^2) + (x2^2 + x3^2) per group of four (second product of each pair fused into the first),
// groups added to the running sum in order.
__global__ void rmsnorm_kernel(const float *x, float *out, int64_t n, float eps) {
    extern __shared__ __align__(16) float v3[];
    __shared__ float scale_s;
    const float *xr = x + (int64_t)blockIdx.x * n;
    float       *o  = out + (int64_t)blockIdx.x * n;
    const int n4 = (int)(n >> 2);
    pdl_launch_dependents();
    pdl_wait();
    for (int g = threadIdx.x; g < n4; g += blockDim.x) {
        const float4 v = reinterpret_cast<const float4 *>(xr)[g];
        v3[g] = __fadd_rn(fmaf(v.y, v.y, __fmul_rn(v.x, v.x)), fmaf(v.w, v.w, __fmul_rn(v.z, v.z)));
    }
    __syncthreads();
    __shared__ __align__(16) float rs_scratch[rs_scratch_words(4)];
    if (threadIdx.x < RS_THREADS) {
        float sum = running_sum_wide(smem_u32(v3), n4, smem_u32(rs_scratch), rs_scratch_words(4), threadIdx.x, 1);
        if (threadIdx.x == 0) {
            for (int64_t i = (int64_t)n4 * 4; i < n; ++i) { sum = fmaf(xr[i], xr[i], sum); }
            scale_s = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)n), eps)));
        }
    }
    __syncthreads();
    const float scale = scale_s;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) { o[i] = __fmul_rn(xr[i], scale); }
}
cudaError_t launch_rmsnorm(const float *x, float *out, int64_t n, int64_t rows, float eps, cudaStream_t s, bool pdl) {
    if (rows == 0 || n == 0) { return cudaSuccess; }
    if ((n & 3) != 0 || n > 180 * 1024) { return cudaErrorNotSupported; }   // rows are read as float4 groups
    const size_t smem = (size_t)n;   // n/4 floats
    static size_t smem_allowed = 48 * 1024;
    if (smem > smem_allowed) {
        cudaError_t err = cudaFuncSetAttribute(rmsnorm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) { return err; }
        smem_allowed = smem;
    }
    return launch_maybe_pdl(rmsnorm_kernel, dim3((unsigned)rows), 256, smem, s, pdl, x, out, n, eps);
}

// binary_execution<plus / multiplies>, basic.cpp:15-50: row r of `a` with row (r % b_rows) of `b`
__global__ void binary_rows_kernel(int op, const float *a, const float *b, float *out, int64_t n, int64_t rows, int64_t b_rows) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, r = i / n, c = i - r * n;
    pdl_launch_dependents();
    pdl_wait();
    if (i >= n * rows) { return; }
    const float   y = b[(r % b_rows) * n + c];
    out[i] = op == 0 ? __fadd_rn(a[i], y) : __fmul_rn(a[i], y);
}
cudaError_t launch_binary_rows(int op, const float *a, const float *b, float *out, int64_t n, int64_t rows, int64_t b_rows, cudaStream_t s, bool pdl) {
    const int64_t tot = n * rows;
    if (tot == 0) { return cudaSuccess; }
    return launch_maybe_pdl(binary_rows_kernel, dim3((unsigned)((tot + 255) / 256)), 256, 0, s, pdl, op, a, b, out, n, rows, b_rows);
}

// OperatorSiluImpl::execute, non-linear.cpp:57-77
__global__ void silu_kernel(const float *x, float *out, int64_t n, const float *table) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (i < n) { out[i] = table[f2h(x[i])]; }
}
cudaError_t launch_silu(const float *x, float *out, int64_t n, const float *silu_table, cudaStream_t s, bool pdl) {
    if (n == 0) { return cudaSuccess; }
    return launch_maybe_pdl(silu_kernel, dim3((unsigned)((n + 255) / 256)), 256, 0, s, pdl, x, out, n, silu_table);
}

// operator_masked_softmax_execute, non-linear.cpp:129-180; one CTA per row (i1, i2), row length ne0,
// the row kept in shared memory; the sum follows std::reduce's order (reduce4_chain).
template <class Mask>   // mask_at(i): the row's additive mask
__device__ __forceinline__ void softmax_masked_row(const float *src, float *dst, int64_t ne0, float scale, const float *exp_table, const Mask &mask_at) {
    extern __shared__ __align__(16) float row_s[];
    __shared__ float red[8];
    __shared__ float bcast;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    pdl_launch_dependents();
    pdl_wait();
    float m = -CUDART_INF_F;
    for (int64_t i = threadIdx.x; i < ne0; i += blockDim.x) {
        const float v = __fmul_rn(__fadd_rn(src[i], mask_at(i)), scale);
        row_s[i] = v;
        m = fmaxf(m, v);
    }
    m = warp_max(m);
    if (lane == 0) { red[warp] = m; }
    __syncthreads();
    m = red[0];
    for (int w = 1; w < nw; ++w) { m = fmaxf(m, red[w]); }
    for (int64_t i = threadIdx.x; i < ne0; i += blockDim.x) {
        row_s[i] = (mask_at(i) == -CUDART_INF_F) ? 0.f : exp_table[f2h(__fsub_rn(row_s[i], m))];
    }
    __syncthreads();
    if (threadIdx.x == 0) { bcast = __fdiv_rn(1.0f, reduce4_chain(row_s, (int)ne0)); }
    __syncthreads();
    const float inv = bcast;
    for (int64_t i = threadIdx.x; i < ne0; i += blockDim.x) { dst[i] = __fmul_rn(row_s[i], inv); }
}
__global__ void softmax_masked_kernel(const float *scores, const float *mask, float *out, int64_t ne0, int64_t ne1,
                                      int64_t mask_stride, float scale, const float *exp_table) {
    const int64_t row = blockIdx.x;
    const float  *mk  = mask + (row % ne1) * mask_stride;
    softmax_masked_row(scores + row * ne0, out + row * ne0, ne0, scale, exp_table, [mk](int64_t i) { return mk[i]; });
}
__global__ void softmax_bits_kernel(const float *scores, const __grid_constant__ MaskBits mask, float *out, int64_t ne0, int64_t ne1, float scale, const float *exp_table) {
    const int64_t row = blockIdx.x;
    const int     bit0 = (int)((row % ne1) * ne0);
    softmax_masked_row(scores + row * ne0, out + row * ne0, ne0, scale, exp_table, [&mask, bit0](int64_t i) {
        const int b = bit0 + (int)i;
        return (mask.w[b >> 5] >> (b & 31)) & 1u ? 0.f : -CUDART_INF_F;
    });
}
cudaError_t launch_softmax_bits(const float *scores, const MaskBits &mask, float *out, int64_t ne0, int64_t ne1, int64_t ne2, float scale, const float *exp_table, cudaStream_t s, bool pdl) {
    if (ne0 < 1 || ne1 < 1 || ne2 < 1 || ne0 * ne1 > MASK_BITS) { return cudaErrorInvalidValue; }
    return launch_maybe_pdl(softmax_bits_kernel, dim3((unsigned)(ne1 * ne2)), 256, (size_t)ne0 * sizeof(float), s, pdl, scores, mask, out, ne0, ne1, scale, exp_table);   // (at most 32 KB of shared memory)
}
cudaError_t launch_softmax_masked(const float *scores, const float *mask, float *out, int64_t ne0, int64_t ne1, int64_t ne2,
                                  int64_t mask_stride, float scale, const float *exp_table, cudaStream_t s, bool pdl) {
    if (ne0 == 0 || ne1 * ne2 == 0) { return cudaSuccess; }
    const size_t smem = (size_t)ne0 * sizeof(float);
    if (smem > 200 * 1024) { return cudaErrorNotSupported; }
    static size_t smem_allowed = 48 * 1024;
    if (smem > smem_allowed) {
        cudaError_t err = cudaFuncSetAttribute(softmax_masked_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) { return err; }
        smem_allowed = smem;
    }
    return launch_maybe_pdl(softmax_masked_kernel, dim3((unsigned)(ne1 * ne2)), 256, smem, s, pdl, scores, mask, out, ne0, ne1, mask_stride, scale, exp_table);
}

__device__ __forceinline__ int64_t soff(const Strided &t, int64_t i0, int64_t i1, int64_t i2, int64_t i3) {
    return i0 * t.nb[0] + i1 * t.nb[1] + i2 * t.nb[2] + i3 * t.nb[3];
}

// OperatorRopeImpl::execute in mode Norm with default YaRN settings, non-linear.cpp:270-371.
// One thread per (pair, head, token); the (cos, sin) of every (token, pair) comes from a table the host
// fills with the same libm calls and the same repeated f32 multiplication of theta as the CPU operator.
__device__ __forceinline__ void rope_pair(const Strided &x, const Strided &out, float2 cs, int64_t k, int64_t i1, int64_t i2) {
    const float *src = reinterpret_cast<const float *>(reinterpret_cast<const uint8_t *>(x.data) + soff(x, 2 * k, i1, i2, 0));
    float       *dst = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(out.data) + soff(out, 2 * k, i1, i2, 0));
    const float x0 = src[0], x1 = src[1];
    dst[0] = __fsub_rn(__fmul_rn(x0, cs.x), __fmul_rn(x1, cs.y));
    dst[1] = __fadd_rn(__fmul_rn(x0, cs.y), __fmul_rn(x1, cs.x));
}
__global__ void rope_kernel(const Strided x, const float2 *cos_sin, const Strided out) {
    const int64_t npair = x.ne[0] >> 1;
    const int64_t i     = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (i >= npair * x.ne[1] * x.ne[2]) { return; }
    const int64_t k = i % npair, i1 = (i / npair) % x.ne[1], i2 = i / (npair * x.ne[1]);
    rope_pair(x, out, cos_sin[i2 * npair + k], k, i1, i2);
}
__global__ void rope_rows_kernel(const Strided x, const float2 *cos_sin, const __grid_constant__ RopeRows rows, const Strided out) {
    const int64_t npair = x.ne[0] >> 1;
    const int64_t i     = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (i >= npair * x.ne[1] * x.ne[2]) { return; }
    const int64_t k = i % npair, i1 = (i / npair) % x.ne[1], i2 = i / (npair * x.ne[1]);
    rope_pair(x, out, cos_sin[(int64_t)rows.row[i2] * npair + k], k, i1, i2);
}
cudaError_t launch_rope(const Strided &x, const float2 *cos_sin, const Strided &out, cudaStream_t s, bool pdl) {
    const int64_t tot = (x.ne[0] >> 1) * x.ne[1] * x.ne[2];
    if (tot == 0) { return cudaSuccess; }
    return launch_maybe_pdl(rope_kernel, dim3((unsigned)((tot + 127) / 128)), 128, 0, s, pdl, x, cos_sin, out);
}
cudaError_t launch_rope_rows(const Strided &x, const float2 *cos_sin, const RopeRows &rows, const Strided &out, cudaStream_t s, bool pdl) {
    const int64_t tot = (x.ne[0] >> 1) * x.ne[1] * x.ne[2];
    if (tot == 0) { return cudaSuccess; }
    if (x.ne[2] > ROPE_ROWS) { return cudaErrorInvalidValue; }
    return launch_maybe_pdl(rope_rows_kernel, dim3((unsigned)((tot + 127) / 128)), 128, 0, s, pdl, x, cos_sin, rows, out);
}

// dup_execute (Copy / Contiguous), view.cpp:83-227, 285-321: element (i0..i3) of src in source order goes to
// the element with the same flat index of dst (dst indexed through its own shape and strides).
__global__ void copy_strided_kernel(const Strided src, int src_type, const Strided dst, int dst_type) {
    const int64_t tot = src.ne[0] * src.ne[1] * src.ne[2] * src.ne[3];
    const int64_t i   = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (i >= tot) { return; }
    const int64_t s0 = i % src.ne[0], s1 = (i / src.ne[0]) % src.ne[1], s2 = (i / (src.ne[0] * src.ne[1])) % src.ne[2],
                  s3 = i / (src.ne[0] * src.ne[1] * src.ne[2]);
    const int64_t d0 = i % dst.ne[0], d1 = (i / dst.ne[0]) % dst.ne[1], d2 = (i / (dst.ne[0] * dst.ne[1])) % dst.ne[2],
                  d3 = i / (dst.ne[0] * dst.ne[1] * dst.ne[2]);
    const uint8_t *sp = reinterpret_cast<const uint8_t *>(src.data) + soff(src, s0, s1, s2, s3);
    uint8_t       *dp = reinterpret_cast<uint8_t *>(dst.data) + soff(dst, d0, d1, d2, d3);
    const float v = (src_type == 0) ? *reinterpret_cast<const float *>(sp) : h2f(*reinterpret_cast<const uint16_t *>(sp));
    if (dst_type == 0) { *reinterpret_cast<float *>(dp) = v; } else { *reinterpret_cast<uint16_t *>(dp) = f2h(v); }
}
cudaError_t launch_copy_strided(const Strided &src, int src_type, const Strided &dst, int dst_type, cudaStream_t s, bool pdl) {
    if ((src_type != 0 && src_type != 1) || (dst_type != 0 && dst_type != 1)) { return cudaErrorNotSupported; }
    const int64_t tot = src.ne[0] * src.ne[1] * src.ne[2] * src.ne[3];
    if (tot == 0) { return cudaSuccess; }
    return launch_maybe_pdl(copy_strided_kernel, dim3((unsigned)((tot + 255) / 256)), 256, 0, s, pdl, src, src_type, dst, dst_type);
}

// bytes of one table row of ne0 elements
__host__ __device__ __forceinline__ int64_t table_row_bytes(int type, int64_t ne0) {
    return type == 0 ? ne0 * 4 : type == 1 ? ne0 * 2 : type == 8 ? ne0 / 32 * 34 : type == 12 ? ne0 / 256 * 144 : type == 14 ? ne0 / 256 * 210 : ne0 / 32 * 18;
}
// embedding row -> f32: memcpy for F32, Q8_0 -> F32 as OperatorGetRowImpl::execute (view.cpp:33-81);
// Q4_0 rows (which the CPU backend cannot gather) decode as (nibble - 8) * d; K-quant rows (no reference arithmetic; the block
// layouts of number_impl/k-quant.h) as (d * sc) * q - dmin * m (Q4_K) and q * (d * sc) (Q6_K), every operation a separate f32 one.
__device__ __forceinline__ float embd_value(const uint8_t *row, int type, int64_t i) {
    if (type == 0) { return reinterpret_cast<const float *>(row)[i]; }
    if (type == 1) { return h2f(reinterpret_cast<const uint16_t *>(row)[i]); }
    if (type == 12) {
        const uint8_t *s = row + (i >> 8) * 144;
        const int e = (int)(i & 255), j = e >> 5, l = e & 31;
        const float d = h2f((uint16_t)(s[0] | (s[1] << 8))), dmin = h2f((uint16_t)(s[2] | (s[3] << 8)));
        const uint8_t *sc12 = s + 4;
        uint32_t sc, mn;
        if (j < 4) { sc = sc12[j] & 63u; mn = sc12[j + 4] & 63u; }
        else { sc = (sc12[j + 4] & 0xFu) | ((uint32_t)(sc12[j - 4] >> 6) << 4); mn = (uint32_t)(sc12[j + 4] >> 4) | ((uint32_t)(sc12[j] >> 6) << 4); }
        const uint8_t qb = s[16 + 32 * (j >> 1) + l];
        const int q = (j & 1) ? (qb >> 4) : (qb & 0xF);
        return __fsub_rn(__fmul_rn(__fmul_rn(d, (float)sc), (float)q), __fmul_rn(dmin, (float)mn));
    }
    if (type == 14) {
        const uint8_t *s = row + (i >> 8) * 210;
        const int e = (int)(i & 255), hf = e >> 7, seg = (e >> 5) & 3, l = e & 31;
        const uint8_t lo = s[64 * hf + 32 * (seg & 1) + l], h = s[128 + 32 * hf + l];
        const int q = (((seg & 2) ? (lo >> 4) : (lo & 0xF)) | (((h >> (2 * seg)) & 3) << 4)) - 32;
        const float d = h2f((uint16_t)(s[208] | (s[209] << 8)));
        const int sc = (int)(int8_t)s[192 + (e >> 4)];
        return __fmul_rn((float)q, __fmul_rn(d, (float)sc));
    }
    const int64_t b = i >> 5; const int k = (int)(i & 31);
    if (type == 8) {
        const uint8_t *blk = row + b * 34;
        return __fmul_rn((float)(int8_t)blk[2 + k], h2f((uint16_t)(blk[0] | (blk[1] << 8))));
    }
    const uint8_t *blk = row + b * 18;   // Q4_0
    const int nib = (k < 16) ? (blk[2 + k] & 0xF) : (blk[2 + k - 16] >> 4);
    return __fmul_rn((float)(nib - 8), h2f((uint16_t)(blk[0] | (blk[1] << 8))));
}

__global__ void getrow_kernel(const uint8_t *table, int type, int64_t row_bytes, int64_t ne0, const int32_t *ids, float *out) {
    const int64_t r   = blockIdx.x;
    const uint8_t *row = table + (int64_t)ids[r] * row_bytes;
    for (int64_t i = threadIdx.x; i < ne0; i += blockDim.x) { out[r * ne0 + i] = embd_value(row, type, i); }
}
cudaError_t launch_getrow(const uint8_t *table, int table_type, int64_t row_bytes, int64_t ne0, const int32_t *ids, int64_t n_ids, float *out, cudaStream_t s) {
    if (table_type != 0 && table_type != 1 && table_type != 2 && table_type != 8 && table_type != 12 && table_type != 14) { return cudaErrorNotSupported; }
    if (n_ids == 0) { return cudaSuccess; }
    getrow_kernel<<<(unsigned)n_ids, 256, 0, s>>>(table, table_type, row_bytes, ne0, ids, out);
    return launch_check();
}
cudaError_t launch_embed(const int32_t *ids, int n_ids, const uint8_t *embd, int embd_type, int64_t d_model, float *x_out, cudaStream_t s) {
    return launch_getrow(embd, embd_type, table_row_bytes(embd_type, d_model), d_model, ids, n_ids, x_out, s);
}

// MatMul with an F16 weight and f32 activations (the attention products when run op by op): activations
// are rounded to fp16 first (mat.cpp:32-42), then Dot<FP16,FP16> (vec_dot.h:117-146) in its exact order.
// One warp per output element; arbitrary byte strides.
__global__ void matmul_f16_kernel(const Strided w, const Strided x, const Strided out) {
    const int64_t n_out = out.ne[0] * out.ne[1] * out.ne[2];
    const int64_t o     = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int     lane  = threadIdx.x & 31;
    const int64_t i01 = o % out.ne[0], i11 = (o / out.ne[0]) % out.ne[1], i02 = o / (out.ne[0] * out.ne[1]);
    const uint8_t *wp = reinterpret_cast<const uint8_t *>(w.data) + soff(w, 0, i01, i02, 0);
    const uint8_t *xp = reinterpret_cast<const uint8_t *>(x.data) + soff(x, 0, i11, i02, 0);
    const int64_t n = w.ne[0];
    const int64_t n_main = n > 0 ? ((n - 1) / 32) * 32 : 0;
    pdl_launch_dependents();
    pdl_wait();
    if (o >= n_out) { return; }
    auto w_at = [&](int64_t k) { return h2f(*reinterpret_cast<const uint16_t *>(wp + k * w.nb[0])); };
    auto x_at = [&](int64_t k) { return h2f(f2h(*reinterpret_cast<const float *>(xp + k * x.nb[0]))); };
    // the scalar tail's (at most 32) elements, one to a lane, in flight with the rest: 32 x 200 scores of heads of 128 7.9 -> 6.8 us
    const float wt = n_main + lane < n ? w_at(n_main + lane) : 0.f, xt = n_main + lane < n ? x_at(n_main + lane) : 0.f;
    float acc = 0.f;
#pragma unroll 4
    for (int64_t k = 0; k < n_main; k += 32) { acc = fmaf(w_at(k + lane), x_at(k + lane), acc); }
    acc = reduce_f16dot_lanes(acc);
    float tail = 0.f;
    const int n_tail = (int)(n - n_main);
    for (int k = 0; k < n_tail; ++k) { tail = fmaf(__shfl_sync(0xffffffffu, wt, k), __shfl_sync(0xffffffffu, xt, k), tail); }
    if (lane == 0) { *reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(out.data) + soff(out, i01, i11, i02, 0)) = __fadd_rn(tail, acc); }
}
cudaError_t launch_matmul_f16(const Strided &w, const Strided &x, const Strided &out, cudaStream_t s, bool pdl) {
    const int64_t n_out = out.ne[0] * out.ne[1] * out.ne[2];
    if (n_out == 0) { return cudaSuccess; }
    return launch_maybe_pdl(matmul_f16_kernel, dim3((unsigned)((n_out * 32 + 255) / 256)), 256, 0, s, pdl, w, x, out);
}

// Greedy sampling on the device (first maximum wins, model/include/llm/sampler/greedy.h:20-25), followed by
// the next step's embedding gather and the position increment, so a decode step needs no host round trip.
__global__ void __launch_bounds__(1024) argmax_embed_kernel(const float *logits, int64_t n_vocab, int32_t *token_out, int32_t *history,
                                                           int *pos_counter, const uint8_t *embd, int embd_type, int64_t d_model, float *x_out) {
    __shared__ float bv[32];
    __shared__ int   bi[32];
    __shared__ int   winner;
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float best = -CUDART_INF_F; int idx = 0x7fffffff;
    for (int64_t i = tid; i < n_vocab; i += blockDim.x) {
        const float v = logits[i];
        if (v > best || (v == best && (int)i < idx)) { best = v; idx = (int)i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int   oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
    }
    if (lane == 0) { bv[warp] = best; bi[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        best = (lane < (int)(blockDim.x >> 5)) ? bv[lane] : -CUDART_INF_F;
        idx  = (lane < (int)(blockDim.x >> 5)) ? bi[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int   oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
        }
        if (lane == 0) {
            if (idx == 0x7fffffff) { idx = 0; }   // all-NaN row: the CPU's max_element returns the first element
            winner = idx;
            *token_out = idx;
            const int step_pos = *pos_counter;
            if (history != nullptr) { history[step_pos] = idx; }
            *pos_counter = step_pos + 1;
            pos_counter[2] += 1;   // exchange epoch of the next step (tensor parallel)
        }
    }
    __syncthreads();
    if (embd != nullptr) {
        const uint8_t *row = embd + (int64_t)winner * table_row_bytes(embd_type, d_model);
        for (int64_t i = tid; i < d_model; i += blockDim.x) { x_out[i] = embd_value(row, embd_type, i); }
    }
}
cudaError_t launch_argmax_embed(const float *logits, int64_t n_vocab, int32_t *token_out, int32_t *history, int *pos_counter,
                                const uint8_t *embd, int embd_type, int64_t d_model, float *x_out, const LaunchCfg &cfg) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(1); lc.blockDim = dim3(1024); lc.dynamicSmemBytes = 0; lc.stream = cfg.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr; lc.numAttrs = cfg.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&lc, argmax_embed_kernel, logits, n_vocab, token_out, history, pos_counter, embd, embd_type, d_model, x_out);
}

// Greedy sampling for a batch of sequences in lockstep: block c takes the logits of sequence c, writes its token (for the next
// step's embedding gather and into ids_out[step][c]) and gathers the embedding into column c of x. The position is advanced
// by advance_pos_kernel afterwards (one word for the whole batch).
__global__ void __launch_bounds__(1024) argmax_embed_batch_kernel(const float *logits, int64_t n_vocab, int32_t *tokens, int32_t *ids_out,
                                                                 const uint8_t *embd, int embd_type, int64_t d_model, float *x_out, int64_t x_stride) {
    __shared__ float bv[32];
    __shared__ int   bi[32];
    __shared__ int   winner;
    const int c = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *row_logits = logits + (int64_t)c * n_vocab;
    float best = -CUDART_INF_F; int idx = 0x7fffffff;
    for (int64_t i = tid; i < n_vocab; i += blockDim.x) {
        const float v = row_logits[i];
        if (v > best || (v == best && (int)i < idx)) { best = v; idx = (int)i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int   oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
    }
    if (lane == 0) { bv[warp] = best; bi[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        best = (lane < (int)(blockDim.x >> 5)) ? bv[lane] : -CUDART_INF_F;
        idx  = (lane < (int)(blockDim.x >> 5)) ? bi[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int   oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
        }
        if (lane == 0) {
            if (idx == 0x7fffffff) { idx = 0; }   // all-NaN row: the CPU's max_element returns the first element
            winner = idx;
            tokens[c] = idx;
            ids_out[c] = idx;
        }
    }
    __syncthreads();
    if (embd != nullptr && x_out != nullptr) {
        const uint8_t *row = embd + (int64_t)winner * table_row_bytes(embd_type, d_model);
        for (int64_t i = tid; i < d_model; i += blockDim.x) { x_out[(int64_t)c * x_stride + i] = embd_value(row, embd_type, i); }
    }
}
__global__ void advance_pos_kernel(int *pos_counter) { pos_counter[0] += 1; pos_counter[2] += 1; }

cudaError_t launch_argmax_embed_batch(const float *logits, int64_t n_vocab, int n_seq, int32_t *tokens, int32_t *ids_out, const uint8_t *embd, int embd_type,
                                      int64_t d_model, float *x_out, int64_t x_stride, int *pos_counter, cudaStream_t s) {
    argmax_embed_batch_kernel<<<n_seq, 1024, 0, s>>>(logits, n_vocab, tokens, ids_out, embd, embd_type, d_model, x_out, x_stride);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) { return err; }
    advance_pos_kernel<<<1, 1, 0, s>>>(pos_counter);
    return cudaGetLastError();
}

}  // namespace spyb
