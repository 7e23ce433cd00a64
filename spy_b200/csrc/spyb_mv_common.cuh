// Pieces shared by the mat-vec kernels of every weight format: the RMSNorm running sum and the fused epilogues.
#pragma once

#include "spyb_common.cuh"
#include "spyb_kernels.h"

namespace spyb {

// Single-column mat-vecs on matvec_rows_kernel and matvec_kq_kernel that are launched ahead of their predecessor's end: stages of each warp's ring
// whose copies are issued before the previous kernel's results are waited for; the rest follow when the reads of x are on their way. Issuing
// takes the warp some 50 cycles a copy, which the last CTA to start (its SM was the last to become free) would add to the step, and x does not
// queue behind a ring full of weights on every SM. Operators of one column on K-quants keep to it: submitted one after the other over several
// matrices, 4096 x 11008 Q6_K 11.2 us and 11008 x 4096 Q4_K 7.15 (all stages first: 11.8 and 7.4); a submit on an idle stream takes the same
// time either way. Plain launches (no programmatic launch) issue all stages first.
constexpr int MV_STAGES_EARLY = 1;

// the RMSNorm running sum: one thread's chain of dependent f32 additions, in the CPU's order
__device__ __forceinline__ float running_sum_serial(uint32_t v3, int n4) {   // v3: shared-space address
    float sum = 0.f;
    int g = 0;
    if (n4 >= 16) {   // the 128-bit reads run one step (16 values) ahead of the dependent adds
        float4 q0 = lds128f(v3), q1 = lds128f(v3 + 16), q2 = lds128f(v3 + 32), q3 = lds128f(v3 + 48);
        for (g = 16; g + 16 <= n4; g += 16) {
            const float4 n0 = lds128f(v3 + 4 * g), n1 = lds128f(v3 + 4 * g + 16), n2 = lds128f(v3 + 4 * g + 32), n3 = lds128f(v3 + 4 * g + 48);
            sum = __fadd_rn(sum, q0.x); sum = __fadd_rn(sum, q0.y); sum = __fadd_rn(sum, q0.z); sum = __fadd_rn(sum, q0.w);
            sum = __fadd_rn(sum, q1.x); sum = __fadd_rn(sum, q1.y); sum = __fadd_rn(sum, q1.z); sum = __fadd_rn(sum, q1.w);
            sum = __fadd_rn(sum, q2.x); sum = __fadd_rn(sum, q2.y); sum = __fadd_rn(sum, q2.z); sum = __fadd_rn(sum, q2.w);
            sum = __fadd_rn(sum, q3.x); sum = __fadd_rn(sum, q3.y); sum = __fadd_rn(sum, q3.z); sum = __fadd_rn(sum, q3.w);
            q0 = n0; q1 = n1; q2 = n2; q3 = n3;
        }
        sum = __fadd_rn(sum, q0.x); sum = __fadd_rn(sum, q0.y); sum = __fadd_rn(sum, q0.z); sum = __fadd_rn(sum, q0.w);
        sum = __fadd_rn(sum, q1.x); sum = __fadd_rn(sum, q1.y); sum = __fadd_rn(sum, q1.z); sum = __fadd_rn(sum, q1.w);
        sum = __fadd_rn(sum, q2.x); sum = __fadd_rn(sum, q2.y); sum = __fadd_rn(sum, q2.z); sum = __fadd_rn(sum, q2.w);
        sum = __fadd_rn(sum, q3.x); sum = __fadd_rn(sum, q3.y); sum = __fadd_rn(sum, q3.z); sum = __fadd_rn(sum, q3.w);
    }
    for (; g < n4; ++g) { sum = __fadd_rn(sum, __uint_as_float(lds32(v3 + 4 * g))); }
    return sum;
}

// (out of line: what is rarely taken shall not lie between what always is)
static __device__ __noinline__ float running_sum_cold(uint32_t v3, int n4) { return running_sum_serial(v3, n4); }

// The same sum, the same bits, by four consecutive warps: the chain is 4.4 cycles per value (4450 cycles for the 1024 groups of a row of
// 4096), which every RMSNorm of a decode step would wait for; this takes 2200. While the running sum stays in one binade it is an integer S
// times its ulp, and adding v >= 0 adds the integer nearest to v / ulp - at a tie the one that leaves S even, so that only S's parity
// matters. Each thread holds a chunk of 4 CQ values and learns its binade from approximate prefix sums: a chunk that stays inside one
// becomes one increment for an even and one for an odd S, and runs of such chunks are added up by a segmented scan. The chunks in which a
// binade may end (some eight of 128) become slots with their values, in order, and the first warp goes through the slots: the increment
// of the run before it, then the slot's values one after the other. The binades are checked with the exact sums afterwards; when one does
// not hold, or there are too many slots (long runs of zeros, values that are not numbers), the plain chain is taken.
// lt: the thread's index in the four warps, bar: their named barrier. The first warp gets the sum.
constexpr int RS_THREADS = 128, RS_SLOTS = 32, RS_SLOTS0 = 14, RS_SLOTS1 = 6;   // slots: of the first warp's chunks, of each other warp's
__host__ __device__ constexpr int rs_scratch_words(int cq) { return 8 + RS_SLOTS * 4 * (1 + cq); }
template <int CQ>
__device__ __forceinline__ float running_sum_chunks(uint32_t v3, int n4, uint32_t scratch, int lt, int bar) {
    constexpr float TWO23 = 8388608.f;
    const int lane = lt & 31, w = lt >> 5;
    const int q4 = n4 >> 2, q0 = lt * CQ;
    const uint32_t count = scratch + 16, slots = scratch + 32;
    constexpr int SLOT = 16 * (1 + CQ);
    auto first_slot = [](int warp) { return warp == 0 ? 0 : RS_SLOTS0 + (warp - 1) * RS_SLOTS1; };
    float v[4 * CQ], own = 0.f;
#pragma unroll
    for (int q = 0; q < CQ; ++q) {
        const float4 x = q0 + q < q4 ? lds128f(v3 + 16 * (q0 + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
        own += (x.x + x.y) + (x.z + x.w);
    }
    float hi = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const float l = __shfl_up_sync(0xffffffffu, hi, o); if (lane >= o) { hi += l; } }
    if (lane == 31) { sts32(scratch + 4 * w, __float_as_uint(hi)); }
    float lo = __shfl_up_sync(0xffffffffu, hi, 1);
    if (lane == 0) { lo = 0.f; }
    asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
    const float4 tot = lds128f(scratch);
    const float base = (w > 0 ? tot.x : 0.f) + (w > 1 ? tot.y : 0.f) + (w > 2 ? tot.z : 0.f);
    // binades of the sum before and after the chunk, with room for the difference between these sums and the chain's (2048 roundings)
    const int el = (int)(__float_as_uint((base + lo) * (1.f - 1.f / 4096.f)) >> 23), eh = (int)(__float_as_uint((base + hi) * (1.f + 1.f / 4096.f)) >> 23);
    bool serial = el != eh || el < 40 || el >= 250;
    const float to_ulps = __uint_as_float((uint32_t)(277 - el) << 23);
    int a0 = 0, before = 0, d = 0, ties = 0;
#pragma unroll
    for (int k = 0; k < 4 * CQ; ++k) {
        const float x = __fmul_rn(v[k], to_ulps), t = __fadd_rn(x, TWO23), f = __fsub_rn(x, __fsub_rn(t, TWO23));   // nearest integer (even at a tie), rest
        if (fabsf(f) == 0.5f) { ++ties; before = a0; d = f > 0.f ? 1 : -1; }
        a0 += (int)(__float_as_uint(t) - __float_as_uint(TWO23));
    }
    serial = serial || ties > 1;
    int a1 = a0 + ((before & 1) ? 0 : d);
    a0 += (before & 1) ? d : 0;
    if (serial) { a0 = 0; a1 = 0; }
    const uint32_t flags = __ballot_sync(0xffffffffu, serial);
    const int last = 31 - __clz((int)(flags & (0xffffffffu >> (31 - lane))));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int l0 = __shfl_up_sync(0xffffffffu, a0, o), l1 = __shfl_up_sync(0xffffffffu, a1, o);
        if (lane - o > last) {
            const int r0 = l0 + ((l0 & 1) ? a1 : a0), r1 = l1 + ((l1 & 1) ? a0 : a1);
            a0 = r0; a1 = r1;
        }
    }
    int p0 = __shfl_up_sync(0xffffffffu, a0, 1), p1 = __shfl_up_sync(0xffffffffu, a1, 1), pe = __shfl_up_sync(0xffffffffu, serial ? -1 : el, 1);
    const int rank = __popc(flags & ((1u << lane) - 1u));
    if (lane == 0) { p0 = 0; p1 = 0; pe = -1; }
    if (lane == 31) {   // the warp's last slot: its last chunk, or the run it ends with
        sts32(count + 4 * w, (uint32_t)(rank + 1));
        if (!serial) { p0 = a0; p1 = a1; pe = el; }
    }
    if ((serial || lane == 31) && rank < (w == 0 ? RS_SLOTS0 : RS_SLOTS1)) {
        const uint32_t s = slots + (first_slot(w) + rank) * SLOT;
        sts128(s, make_uint4((uint32_t)p0, (uint32_t)(p1 - p0), (uint32_t)pe, 0u));
        auto bits = [&](float x) { return serial ? __float_as_uint(x) : 0u; };
#pragma unroll
        for (int q = 0; q < CQ; ++q) { sts128(s + 16 * (1 + q), make_uint4(bits(v[4 * q]), bits(v[4 * q + 1]), bits(v[4 * q + 2]), bits(v[4 * q + 3]))); }
    }
    asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
    if (w != 0) { return 0.f; }
    float s = 0.f;
    const uint4 cn = lds128(count);
    const int4  cnt = make_int4((int)cn.x, (int)cn.y, (int)cn.z, (int)cn.w);
    bool ok = cnt.x <= RS_SLOTS0 && max(max(cnt.y, cnt.z), cnt.w) <= RS_SLOTS1;
    if (ok) {   // one slot to a lane; the sum goes from lane to lane (lanes past the last slot add nothing)
        const int s1 = cnt.x, s2 = s1 + cnt.y, s3 = s2 + cnt.z, total = s3 + cnt.w;
        const int sw = (lane >= s1) + (lane >= s2) + (lane >= s3);
        const uint32_t mine = slots + (first_slot(sw) + lane - (lane >= s3 ? s3 : lane >= s2 ? s2 : lane >= s1 ? s1 : 0)) * SLOT;
        const uint4 en = lane < total ? lds128(mine) : make_uint4(0u, 0u, 0xffffffffu, 0u);
        const int ez = (int)en.z;
        float c[4 * CQ];
#pragma unroll
        for (int q = 0; q < CQ; ++q) {
            const float4 x = lane < total ? lds128f(mine + 16 * (1 + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
            c[4 * q] = x.x; c[4 * q + 1] = x.y; c[4 * q + 2] = x.z; c[4 * q + 3] = x.w;
        }
        uint32_t from = 0;
#pragma unroll 1
        for (int i0 = 0; i0 < total; i0 += 4) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t b = __float_as_uint(s);
                if (lane == i0 + i) { from = b; }
                float t = __uint_as_float(b + en.x + (b & 1u) * en.y);
#pragma unroll
                for (int k = 0; k < 4 * CQ; ++k) { t = __fadd_rn(t, c[k]); }
                s = __shfl_sync(0xffffffffu, t, i0 + i);
            }
        }
        const uint32_t to = from + en.x + (from & 1u) * en.y;
        ok = __all_sync(0xffffffffu, ez < 0 || ((int)(from >> 23) == ez && (int)(to >> 23) == ez));
    }
    if (!ok) { return running_sum_cold(v3, n4); }
#pragma unroll 1
    for (int g = 4 * q4; g < n4; ++g) { s = __fadd_rn(s, __uint_as_float(lds32(v3 + 4 * g))); }
    return s;
}
// Called by four whole warps. From RS_MIN values on (640: 2200 cycles against 2900; 512: 1900 against 2400, less what the extra code costs a
// cold instruction cache) the chunks, where `words` of scratch hold them; the chain by the first warp otherwise.
constexpr int RS_MIN = 576, RS_MAX = 2048;
static __device__ __noinline__ float running_sum_wide(uint32_t v3, int n4, uint32_t scratch, int words, int lt, int bar) {
    if (n4 >= RS_MIN && n4 <= 1024 && words >= rs_scratch_words(2)) { return running_sum_chunks<2>(v3, n4, scratch, lt, bar); }
    if (n4 > 1024 && n4 <= 1536 && words >= rs_scratch_words(3)) { return running_sum_chunks<3>(v3, n4, scratch, lt, bar); }
    if (n4 > 1536 && n4 <= RS_MAX && words >= rs_scratch_words(4)) { return running_sum_chunks<4>(v3, n4, scratch, lt, bar); }
    return lt < 32 ? running_sum_serial(v3, n4) : 0.f;
}
// ---------------------------------------------------------------------------------------------
// epilogue for one finished dot product `v` (identical on the 8 lanes of its row) of row `row`, column t.
// `partner` is the value of the neighbouring row (row ^ 1), needed by RoPE. Called by all lanes; lane l == 0 writes.
// EPI >= 0: the epilogue of a kernel that has this one only
template <int EPI = -1>
__device__ __forceinline__ void matvec_epilogue(const MatvecParams &p, int64_t row, int t, float v, float partner, bool writer) {
    switch (EPI >= 0 ? EPI : p.epi) {
    case EPI_STORE:
        if (writer) { p.out[(int64_t)t * p.out_stride + row] = v; }
        break;
    case EPI_RESID:   // Add(attn_out, x) / Add(ffn_inp, ffn_out): model/src/llm/model/llama.cpp:194-211
        if (writer) { const int64_t i = (int64_t)t * p.out_stride + row; p.out[i] = __fadd_rn(v, p.resid[i]); }
        break;
    case EPI_QKV_ROPE: {
        if (!writer) { break; }
        const int sec = (int)row >= 2 * p.dl ? 2 : (int)row >= p.dl ? 1 : 0;
        const int e   = (int)row - sec * p.dl;
        const int pos = *p.pos_base + (p.seq_stride ? 0 : t);          // a batch in lockstep: every column at the same position,
        const int64_t seq_off = p.seq_stride ? (int64_t)t * p.seq_stride : 0;   // each in its own cache
        if (sec == 2) {   // V: f32 -> f16 RNE into the transposed cache [dl][n_ctx] (dup_execute, backend/host/operator/view.cpp:163-191)
            p.v_cache[seq_off + (int64_t)e * p.n_ctx + pos] = __float2half_rn(v);
        } else {          // RoPE, mode Norm: backend/host/operator/non-linear.cpp:270-371 (rows 2i, 2i+1 rotate together)
            const float2 cs = p.rope_table[(int64_t)pos * (p.hd >> 1) + ((e % p.hd) >> 1)];
            const float x0 = (e & 1) ? partner : v, x1 = (e & 1) ? v : partner;
            const float a = (e & 1) ? __fadd_rn(__fmul_rn(x0, cs.y), __fmul_rn(x1, cs.x))
                                    : __fsub_rn(__fmul_rn(x0, cs.x), __fmul_rn(x1, cs.y));
            __half *dst = (sec == 0) ? p.q_out + (int64_t)t * p.dl + e : p.k_cache + seq_off + (int64_t)pos * p.dl + e;
            *dst = __float2half_rn(a);
        }
    } break;
    default: break;
    }
}

// up * silu(gate): model/src/llm/plugin/ffn.cpp:28-35; silu = table on the fp16-rounded argument
__device__ __forceinline__ void matvec_epilogue_silu(const MatvecParams &p, int64_t row, int t, float up, float gate, bool writer) {
    if (writer) { p.out[(int64_t)t * p.out_stride + row] = __fmul_rn(up, p.silu_table[f2h(gate)]); }
}

}  // namespace spyb
