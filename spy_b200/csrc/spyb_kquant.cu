// Dequant-fused mat-vec for K-quant weights (Q4_K: 144 B / 256 values, Q6_K: 210 B / 256 values; block layouts
// orchestration/include/number/number_impl/k-quant.h:79-117, 162-188) inside the fused step plan.
//
// Parity is unpinned by the reference: it defines these layouts but no arithmetic for them (a K-quant weight makes its
// MatMul pick a quantizer that throws, backend/host/include/simd/vec_convert.h:30-36). What is reproduced here, bit for
// bit, is the CPU restatement used as the checker: the reference's MatMul rule for quantized weights - activations
// quantized to Q8_0 first (backend/host/operator/mat.cpp:32-42, 95-128) - with, per 256-value super-block,
//   Q4_K:  acc = 0; for the 8 sub-blocks j of 32 values: acc = fma((d * sc_j) * dx_j, (float)sum(q * y), acc);
//                                                         acc = fma(-((dmin * m_j) * dx_j), (float)sum(y), acc)
//   Q6_K:  acc = 0; for the 16 groups g of 16 values:    acc = fma((d * sc_g) * dx_(g/2), (float)sum(q * y), acc)
// and the row's result = the super-blocks' values added in order. The integer sums are exact, so only this order matters.
//
// Mapping: a super-block's value depends on nothing before it, so the lanes of a warp take the super-blocks of a unit (NP pairs of
// neighbouring rows: rows 2q, 2q+1 rotate together in RoPE; FFN up row q and gate row q meet in the SiLU epilogue) side by side, 32 at a
// time (a round), leave their values in shared memory, and one lane per row and column adds a row's values in order.
// Streaming: every warp pulls its rounds through a private ring with cp.async.bulk (a round is one or two contiguous runs of 32 x 144 or
// 208 bytes); the first copies are issued before griddepcontrol.wait, so the previous kernel's tail and the serial prologue pass while
// the weights arrive; a lane takes its super-block into registers (the 144- and 208-byte pitches are odd multiples of 16: conflict-free
// 128-bit reads) and the stage is refilled before the arithmetic begins.
// Roofline: HBM-bound, rows * K/256 * 144 (210) bytes per launch, read once; Q4_K rows as the file has them, Q6_K rows re-laid at upload so
// that every piece is 16-byte aligned (208-byte bodies, the fp16 scales of a row together at its end).
// Activations in shared memory as one record per super-block: 64 words of Q8_0 values, 8 scales, 16 sums of 16 values as floats, at a
// pitch of 92 words, again an odd multiple of 16 bytes, so that the lanes' 128-bit reads of different super-blocks are conflict-free.
// Against lanes that read their super-blocks from global memory when they got to them: 11008 x 4096 Q4_K, four columns, 22.5 -> 15.4 us; a
// decode step of eight 7B layers (Q4_K / Q6_K) 0.75 -> 0.52 ms.

#include <algorithm>
#include <type_traits>

#include "spyb_common.cuh"
#include "spyb_kernels.h"
#include "spyb_tp.cuh"
#include "spyb_mv_common.cuh"

namespace spyb {

constexpr int KQ_THREADS = 512;
constexpr int KQ_WARPS   = KQ_THREADS / WARP;
constexpr int KQ_REC = 92;               // words per super-block of activations: 64 values, 8 scales, 16 half-block sums, 4 of padding
constexpr int KQ_MAX_STAGES = 4;

// PG groups of eight values (groups g0, g0 + KQ_THREADS, ... of the column's n8) -> their words of the column's records, the blocks' scales
// and half-block sums; called by whole warps
template <int PG>
__device__ __forceinline__ void kq_quantize(const float (&v)[PG][8], int g0, int n8, uint32_t *rec) {
    const int npass = min(PG, (n8 - (g0 & ~31) + KQ_THREADS - 1) / KQ_THREADS);   // (n8 is a multiple of 32: the same in the whole warp)
    uint2 q[PG];
    int kd;
    const float d = quantize_q8_groups<PG>(v, npass, q, kd);
#pragma unroll
    for (int k = 0; k < PG; ++k) {
        if (k < npass) {
            int s = q8_sum8(q[k]);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            const int g = g0 + k * KQ_THREADS, b = g >> 2, w = g & 3;
            uint32_t *r = rec + (b >> 3) * KQ_REC;
            *reinterpret_cast<uint2 *>(r + (b & 7) * 8 + 2 * w) = q[k];
            if ((w & 1) == 0) { r[72 + 2 * (b & 7) + (w >> 1)] = __float_as_uint((float)s); }
        }
    }
    if (kd >= 0) { const int b = (g0 + kd * KQ_THREADS) >> 2; rec[(b >> 3) * KQ_REC + 64 + (b & 7)] = __float_as_uint(h2f(f2h(d))); }
}

// NormRMS + Mul(weight) (optional) + Quantizator<FP32,Q8_0> of the pass's columns into the activation records (column t lies col words
// further); the arithmetic is that of the Q4_0 / Q8_0 kernels' prologue (same device functions). The columns' running sums of squares run
// side by side, one warp each.
template <bool NORM>
__device__ __forceinline__ void kq_prologue(const MatvecParams &p, int nT, uint32_t *rec, int col, float *scale_s) {
    const int tid = threadIdx.x;
    const int n4  = (int)(p.A.k >> 2);
    if (NORM) {
#pragma unroll 1
        for (int t = 0; t < nT; ++t) {
            const float4 *x4 = reinterpret_cast<const float4 *>(p.x + (int64_t)t * p.x_stride);
            float *v3 = reinterpret_cast<float *>(rec + t * col);   // (n4 = 64 words per super-block: inside the column's records)
            for (int g = tid; g < n4; g += KQ_THREADS) {
                const float4 v = __ldcg(x4 + g);
                const float v1 = fmaf(v.y, v.y, __fmul_rn(v.x, v.x));
                const float v2 = fmaf(v.w, v.w, __fmul_rn(v.z, v.z));
                v3[g] = __fadd_rn(v1, v2);
            }
        }
        __syncthreads();
        if ((tid & 31) == 0 && (tid >> 5) < nT) {
            const float sum  = running_sum_cold(smem_u32(rec + (tid >> 5) * col), n4);
            const float mean = __fdiv_rn(sum, (float)p.A.k);
            scale_s[tid >> 5] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, p.eps)));
        }
        __syncthreads();   // also: the partials (aliasing the records) are dead from here on
    }
    const int n8 = n4 >> 1;
#pragma unroll 1
    for (int t = 0; t < nT; ++t) {
        const float *x = p.x + (int64_t)t * p.x_stride;
        const float scale = NORM ? scale_s[t] : 1.f;
        for (int base = 0; base < n8; base += KQ_THREADS) {   // n8 is a multiple of 32: whole warps, whole blocks
            const int g = base + tid;
            const bool valid = g < n8;
            float v[1][8];
            if (valid) { load8_cg(x + 8 * g, v[0]); }
            else {
#pragma unroll
                for (int i = 0; i < 8; ++i) { v[0][i] = 0.f; }
            }
            if (NORM && valid) {
                float w[8];
                load8_cg(p.norm_w + 8 * g, w);
#pragma unroll
                for (int i = 0; i < 8; ++i) { v[0][i] = __fmul_rn(__fmul_rn(v[0][i], scale), w[i]); }
            }
            kq_quantize<1>(v, g, n8, rec + t * col);
        }
    }
}

// One column of at most 512 PG groups of eight: every thread keeps its groups of x in registers from the one global read on; x_requested() is
// called when the reads are on their way. wearly: the norm weights when the kernel read them at its start (PG <= KQ_NORM_EARLY).
constexpr int KQ_NORM_EARLY = 2, KQ_PRO_GROUPS = 3;
template <int PG, bool NORM, class Requested>
__device__ __forceinline__ void kq_prologue_1col(const MatvecParams &p, uint32_t *rec, float *scale_s, const float (*wearly)[8], Requested x_requested) {
    constexpr int CQ = PG == 1 ? 2 : 3;                          // (quads per thread of the wide sum: rows of at most 4096 or 6144 values)
    const int tid = threadIdx.x;
    const int n4  = (int)(p.A.k >> 2), n8 = (int)(p.A.k >> 3);   // multiples of 64 and 32: whole warps, whole blocks
    float xv[PG][8], wv[PG][8];
    auto zero = [](float (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 8; ++i) { v[i] = 0.f; }
    };
#pragma unroll
    for (int k = 0; k < PG; ++k) {
        const int g = tid + k * KQ_THREADS;
        if (g < n8) { load8_cg(p.x + 8 * g, xv[k]); } else { zero(xv[k]); }
    }
    if (NORM) {
#pragma unroll
        for (int k = 0; k < PG; ++k) {
            const int g = tid + k * KQ_THREADS;
            if (PG <= KQ_NORM_EARLY) {
#pragma unroll
                for (int i = 0; i < 8; ++i) { wv[k][i] = wearly[k][i]; }
            } else if (g < n8) { load8_cg(p.norm_w + 8 * g, wv[k]); } else { zero(wv[k]); }
        }
    }
    x_requested();
    if (NORM) {
        float *v3 = reinterpret_cast<float *>(rec);   // (n4 = 64 words per super-block: inside the records; the scratch of the sum behind it)
#pragma unroll
        for (int k = 0; k < PG; ++k) {
            const int g = tid + k * KQ_THREADS;
            if (g < n8) { reinterpret_cast<float2 *>(v3)[g] = squares8(xv[k]); }
        }
        __syncthreads();
        float sum = 0.f;
        if (PG <= KQ_NORM_EARLY && n4 >= RS_MIN && n4 <= CQ * 512 && (n4 >> 6) * (KQ_REC - 64) >= rs_scratch_words(CQ)) {
            if (tid < RS_THREADS) { sum = running_sum_chunks<PG <= KQ_NORM_EARLY ? CQ : 2>(smem_u32(v3), n4, smem_u32(v3 + n4), tid, 1); }
        } else if (tid == 0) { sum = running_sum_cold(smem_u32(v3), n4); }
        if (tid == 0) { scale_s[0] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)p.A.k), p.eps))); }
        __syncthreads();   // also: the partials (aliasing the records) are dead from here on
        const float scale = scale_s[0];
#pragma unroll
        for (int k = 0; k < PG; ++k) {
#pragma unroll
            for (int i = 0; i < 8; ++i) { xv[k][i] = __fmul_rn(__fmul_rn(xv[k][i], scale), wv[k][i]); }
        }
    }
    kq_quantize<PG>(xv, tid, n8, rec);
}

// byte i of w (a constant) as the float 2^23 + byte: the byte becomes the low bits of a float's mantissa
template <int I> __device__ __forceinline__ float kq_byte_magic(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | I)); }

// values of one Q4_K super-block (its 144 bytes in w) for the TM activation columns of a pass: rec_s = shared-space address of the
// super-block's activation record of column 0, the next column's col_bytes further. The weights are unpacked once for all columns.
template <int TM, int NW>
__device__ __forceinline__ void kq_values_q4k(const uint4 (&w)[NW], uint32_t rec_s, uint32_t col_bytes, float (&acc)[TM]) {
    const float2 dm = __half22float2(*reinterpret_cast<const __half2 *>(&w[0].x));   // d, dmin
    // the eight 6-bit scales and minima, four to a word
    const uint32_t scw[2] = {w[0].y & 0x3f3f3f3fu, (w[0].w & 0x0f0f0f0fu) | ((w[0].y >> 2) & 0x30303030u)};
    const uint32_t mnw[2] = {w[0].z & 0x3f3f3f3fu, ((w[0].w >> 4) & 0x0f0f0f0fu) | ((w[0].z >> 2) & 0x30303030u)};
#pragma unroll
    for (int t = 0; t < TM; ++t) { acc[t] = 0.f; }
#pragma unroll
    for (int jp = 0; jp < 4; ++jp) {           // sub-blocks 2 jp and 2 jp + 1: the low and the high nibbles of bytes 32 jp .. + 31 of qs
        const uint4 qa = w[1 + 2 * jp], qb = w[2 + 2 * jp];
        const uint32_t w8[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
        uint32_t nib[2][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) { nib[0][i] = w8[i] & 0x0f0f0f0fu; nib[1][i] = (w8[i] >> 4) & 0x0f0f0f0fu; }
        const uint32_t sw = scw[jp >> 1], mw = mnw[jp >> 1];
        const float s0 = (jp & 1) ? kq_byte_magic<2>(sw) : kq_byte_magic<0>(sw), s1 = (jp & 1) ? kq_byte_magic<3>(sw) : kq_byte_magic<1>(sw);
        const float m0 = (jp & 1) ? kq_byte_magic<2>(mw) : kq_byte_magic<0>(mw), m1 = (jp & 1) ? kq_byte_magic<3>(mw) : kq_byte_magic<1>(mw);
        // (2^23 is taken off before the product, not with it: an infinite d would meet its own opposite)
        const float dsc[2] = {__fmul_rn(dm.x, s0 - 8388608.f), __fmul_rn(dm.x, s1 - 8388608.f)}, dmn[2] = {__fmul_rn(-dm.y, m0 - 8388608.f), __fmul_rn(-dm.y, m1 - 8388608.f)};   // (dmn: negated)
#pragma unroll
        for (int t = 0; t < TM; ++t) {
            {
                const uint32_t r = rec_s + t * col_bytes;
                const float4 ys = lds128f(r + 288u + 16u * jp);   // sums of the four halves
                float dx[2];
                asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(dx[0]), "=f"(dx[1]) : "r"(r + 256u + 8u * jp));
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    const uint4 ya = lds128(r + 64u * jp + 32u * o), yb = lds128(r + 64u * jp + 32u * o + 16u);
                    const uint32_t y8[8] = {ya.x, ya.y, ya.z, ya.w, yb.x, yb.y, yb.z, yb.w};
                    int isum = (int)MAGIC_I;   // (the sum as the bits of the float MAGIC_F + sum)
#pragma unroll
                    for (int i = 0; i < 8; ++i) { isum = __dp4a((int)nib[o][i], (int)y8[i], isum); }
                    acc[t] = fmaf(__fmul_rn(dsc[o], dx[o]), __int_as_float(isum) - MAGIC_F, acc[t]);
                    acc[t] = fmaf(__fmul_rn(dmn[o], dx[o]), o ? __fadd_rn(ys.z, ys.w) : __fadd_rn(ys.x, ys.y), acc[t]);   // (small integers: the sum is exact)
                }
            }
        }
    }
}

// values of one Q6_K super-block in the upload layout: w = its 208 bytes (ql 128, qh 64, 16 int8 scales), d_half = its fp16 scale
template <int TM, int NW>
__device__ __forceinline__ void kq_values_q6k(const uint4 (&wv)[NW], uint16_t d_half, uint32_t rec_s, uint32_t col_bytes, float (&acc)[TM]) {
    const float d = h2f(d_half);
    const uint32_t scs[4] = {wv[12].x, wv[12].y, wv[12].z, wv[12].w};
#pragma unroll
    for (int t = 0; t < TM; ++t) { acc[t] = 0.f; }
#pragma unroll
    for (int gq = 0; gq < 4; ++gq) {
        uint32_t v6[4][4];                      // the values 0..63 of groups 4 gq .. + 3, four per word
        float    dsc[4];
#pragma unroll
        for (int gi = 0; gi < 4; ++gi) {
            // group g = values 16g .. 16g+15: half h of the super-block, segment s of 32 values, l = 16 * (g & 1) .. + 15
            //   s 0: ql[64h + l] low | qh[32h + l] bits 0-1     s 1: ql[64h + 32 + l] low  | bits 2-3
            //   s 2: ql[64h + l] high | bits 4-5                s 3: ql[64h + 32 + l] high | bits 6-7
            const int g = 4 * gq + gi, h = g >> 3, sg = (g >> 1) & 3, l0 = 16 * (g & 1);
            const uint4 lv = wv[(64 * h + 32 * (sg & 1) + l0) >> 4], hv = wv[8 + ((32 * h + l0) >> 4)];
            const uint32_t lw[4] = {lv.x, lv.y, lv.z, lv.w}, hw[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t lo = (sg & 2) ? (lw[i] >> 4) & 0x0f0f0f0fu : lw[i] & 0x0f0f0f0fu;
                const uint32_t hi = sg == 0 ? hw[i] << 4 : sg == 1 ? hw[i] << 2 : sg == 2 ? hw[i] : hw[i] >> 2;
                v6[gi][i] = lo | (hi & 0x30303030u);
            }
            const uint32_t su = scs[gq] ^ 0x80808080u;   // scale + 128
            const float sm = gi == 0 ? kq_byte_magic<0>(su) : gi == 1 ? kq_byte_magic<1>(su) : gi == 2 ? kq_byte_magic<2>(su) : kq_byte_magic<3>(su);
            dsc[gi] = __fmul_rn(d, sm - 8388736.f);
        }
#pragma unroll
        for (int t = 0; t < TM; ++t) {
            {
                const uint32_t r = rec_s + t * col_bytes;
                const float4 ys4 = lds128f(r + 288u + 16u * gq);   // sums of the groups' activations
                float dx[2];
                asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(dx[0]), "=f"(dx[1]) : "r"(r + 256u + 8u * gq));
                const float ys[4] = {ys4.x, ys4.y, ys4.z, ys4.w};
#pragma unroll
                for (int gi = 0; gi < 4; ++gi) {
                    const uint4 y = lds128(r + 16u * (4 * gq + gi));
                    int isum = __dp4a((int)v6[gi][0], (int)y.x, (int)MAGIC_I);
                    isum = __dp4a((int)v6[gi][1], (int)y.y, isum); isum = __dp4a((int)v6[gi][2], (int)y.z, isum); isum = __dp4a((int)v6[gi][3], (int)y.w, isum);
                    const float sum = fmaf(-32.f, ys[gi], __int_as_float(isum)) - MAGIC_F;   // value = stored - 32 (integers below 2^24 throughout: exact)
                    acc[t] = fmaf(__fmul_rn(dsc[gi], dx[gi >> 1]), sum, acc[t]);
                }
            }
        }
    }
}

struct KqRow { const uint8_t *w; int64_t pitch; int type; };
// where row `row` of the virtual matrix lies (static indexes: the segments stay in the parameter bank)
__device__ __forceinline__ KqRow kq_row(const MatvecParams &p, int64_t row) {
    const int64_t n0 = p.kq[0].n_rows, n1 = p.kq[1].n_rows;
    const bool b1 = p.kq_n > 1 && row >= n0, b2 = p.kq_n > 2 && row >= n0 + n1;
    KqRow r;
    r.pitch = b2 ? p.kq[2].row_bytes : b1 ? p.kq[1].row_bytes : p.kq[0].row_bytes;
    r.type  = b2 ? p.kq[2].type : b1 ? p.kq[1].type : p.kq[0].type;
    r.w     = (b2 ? p.kq[2].w : b1 ? p.kq[1].w : p.kq[0].w) + (row - (b2 ? n0 + n1 : b1 ? n0 : 0)) * r.pitch;
    return r;
}
// first row of the unit that begins at pair `pair0` (side 1: of the second matrix in pair mode). Row r of a unit is row r of the first, or,
// in pair mode, row r / 2 of side r % 2.
template <int EPI>
__device__ __forceinline__ KqRow kq_unit(const MatvecParams &p, int64_t pair0, int side) {
    if constexpr (EPI == EPI_RESID || EPI == EPI_STORE) { return {p.kq[0].w + 2 * pair0 * p.kq[0].row_bytes, p.kq[0].row_bytes, p.kq[0].type}; }   // (one matrix)
    if (EPI >= 0 ? EPI != EPI_SILU_MUL : !p.pair_mode) { return kq_row(p, 2 * pair0); }
    KqRow r;
    r.pitch = side ? p.kq[1].row_bytes : p.kq[0].row_bytes; r.type = side ? p.kq[1].type : p.kq[0].type;
    r.w = (side ? p.kq[1].w : p.kq[0].w) + pair0 * r.pitch;
    return r;
}

struct KqPlan { int np, wact, ns, stage_bytes; };   // pairs per unit, streaming warps per CTA, ring stages per warp, bytes per stage
struct KqSmem { size_t part, bars, ring, total; };
__host__ __device__ static inline KqSmem kq_smem_layout(int nsb, int TM, const KqPlan &q) {
    KqSmem m;
    m.part = (size_t)TM * nsb * KQ_REC * 4;
    m.bars = (m.part + (size_t)q.wact * TM * 2 * q.np * nsb * 4 + 15) / 16 * 16;
    m.ring = (m.bars + (size_t)q.wact * q.ns * 8 + 127) / 128 * 128;
    m.total = m.ring + (size_t)q.wact * q.ns * q.stage_bytes;
    return m;
}

// TM: columns of the pass, rounded up to 1, 2 or 4 (columns past p.T compute on whatever their records hold and are not stored); TYPE: 12 or
// 14 when every row is of that type, else 0
// PRO: the prologue the kernel is built with - one column of at most 1024 groups of four (with the norm also 1536) or a longer one, with and without the norm;
// else any
// EPI >= 0: of one epilogue (SILU_MUL: in pair mode; STORE and RESID: of one matrix), without the exchange between GPUs, as in matvec_rows_kernel
enum { KQP_ANY, KQP_NORM, KQP_NORM_MID, KQP_PLAIN, KQP_NORM_LONG, KQP_PLAIN_LONG };
template <int TM, int TYPE, int PRO, int EPI = -1>
__global__ void __launch_bounds__(KQ_THREADS, 1) matvec_kq_kernel(const MatvecParams p, const KqPlan pl) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ float scale_s[TM];
    const bool pair_mode = EPI >= 0 ? EPI == EPI_SILU_MUL : p.pair_mode != 0;
    const int  epi = EPI >= 0 ? EPI : p.epi;
    const int nsb = p.A.nb >> 3, nT = (TM == 1) ? 1 : p.T;
    const int col = nsb * KQ_REC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const KqSmem L = kq_smem_layout(nsb, TM, pl);
    const int n_row = 2 * pl.np, items = n_row * nsb, n_round = (items + 31) >> 5;   // per unit
    const int64_t n_units  = (pair_mode ? p.kq[0].n_rows : (p.A.n_rows >> 1)) / pl.np;
    const int64_t unit_lo  = n_units * blockIdx.x / gridDim.x, unit_hi = n_units * (blockIdx.x + 1) / gridDim.x;
    const int64_t my_first = unit_lo + warp;
    const int     my_units = (warp < pl.wact && my_first < unit_hi) ? (int)((unit_hi - my_first + pl.wact - 1) / pl.wact) : 0;
    const int     n_stage  = my_units * n_round;
    const uint32_t ring_s = smem_u32(smem_raw + L.ring) + (uint32_t)warp * pl.ns * pl.stage_bytes;
    const uint32_t bar_s  = smem_u32(smem_raw + L.bars) + (uint32_t)warp * pl.ns * 8;
    float *part = reinterpret_cast<float *>(smem_raw + L.part) + (size_t)warp * TM * items;
    const bool mixed = TYPE == 0 && pair_mode && p.kq[0].type != p.kq[1].type;   // (items of a stage then lie at the larger pitch)

    // lane 0: the next 32 super-blocks of the unit at lunit (from super-block lsb of its row lr on) into slot lslot
    int64_t lunit = my_first; int lr = 0, lsb = 0, lslot = 0, issued = 0;
    KqRow l0 = {}, l1 = {};
    auto load_unit = [&]() { l0 = kq_unit<EPI>(p, lunit * pl.np, 0); if (pair_mode) { l1 = kq_unit<EPI>(p, lunit * pl.np, 1); } };
    const uint64_t policy = l2_evict_first();
    // the loop over a stage's pieces of Q6_K rows: unrolled for two columns (17376 x 5632 29.7 -> 28.9 us, 4096 x 11008 18.0 -> 17.6, 1024 x 2048 4.81 -> 4.75), rolled in the
    // kernels of a step, which the instruction cache has to hold side by side
    constexpr int PIECES = TM == 2 && TYPE == 14 ? 4 : 1;
    // the end of a row's sum, up to seven super-blocks: unrolled for two columns too (Q4_K rows of fifteen super-blocks, 12564 x 3840 12.2 -> 12.0 us, 10620 x 3840 11.3 -> 11.1)
    constexpr int TAIL = TM == 2 ? 4 : 1;
    auto issue_next = [&]() {
        const uint32_t bar = bar_s + lslot * 8;
        uint32_t dst = ring_s + (uint32_t)(lslot * pl.stage_bytes);
        int left = min(32, items - (lr * nsb + lsb));
        if (!pair_mode && (TYPE != 0 ? TYPE : l0.type) == 12) {   // the unit's rows are one contiguous run
            const uint32_t bytes = (uint32_t)left * 144u;
            mbar_expect_tx(bar, bytes);
            bulk_copy_g2s_once(dst, l0.w + (size_t)(lr * nsb + lsb) * 144, bytes, bar, policy);
            lsb += left;
#pragma unroll 1
            while (lsb >= nsb) { lsb -= nsb; ++lr; }
        } else {
            uint32_t bytes = (uint32_t)left * ((TYPE != 0 ? TYPE : l0.type) == 12 ? 144u : 208u);
            if (mixed) {
                bytes = 0;
#pragma unroll 1
                for (int q = left, r = lr, o = lsb; q > 0; ++r, o = 0) { const int m = min(q, nsb - o); bytes += (uint32_t)m * (((r & 1) ? l1.type : l0.type) == 12 ? 144u : 208u); q -= m; }
            }
            mbar_expect_tx(bar, bytes);
#pragma unroll PIECES
            while (left > 0) {
                const int m = min(left, nsb - lsb);
                const bool second = pair_mode && (lr & 1);
                const uint32_t body = (TYPE != 0 ? TYPE : second ? l1.type : l0.type) == 12 ? 144u : 208u;
                const uint8_t *src = (second ? l1.w : l0.w) + (int64_t)(pair_mode ? lr >> 1 : lr) * (second ? l1.pitch : l0.pitch) + (uint32_t)lsb * body;
                bulk_copy_g2s_once(dst, src, (uint32_t)m * body, bar, policy);
                dst += (uint32_t)m * (mixed ? 208u : body);
                left -= m; lsb += m;
                if (lsb == nsb) { lsb = 0; ++lr; }
            }
        }
        ++issued;
        if (++lslot == pl.ns) { lslot = 0; }
        if (lr == n_row) { lr = 0; lunit += pl.wact; if (issued < n_stage) { load_unit(); } }
    };

    // weights never change during a step: the copies may run ahead of the previous kernel's results
    pdl_launch_dependents();
    constexpr int PG = (PRO == KQP_NORM || PRO == KQP_PLAIN) ? 1 : PRO == KQP_NORM_MID ? 2 : KQ_PRO_GROUPS;
    float wearly[PRO == KQP_NORM_MID ? 2 : 1][8];
    if (PRO == KQP_NORM || PRO == KQP_NORM_MID) {
#pragma unroll
        for (int k = 0; k < (PG < 4 ? PG : 0); ++k) {
            const int g = threadIdx.x + k * KQ_THREADS;
            if (g < (int)(p.A.k >> 3)) { load8_cg(p.norm_w + 8 * g, wearly[k]); }
            else {
#pragma unroll
                for (int i = 0; i < 8; ++i) { wearly[k][i] = 0.f; }
            }
        }
    }
    if (lane == 0 && n_stage > 0) {
#pragma unroll 1
        for (int s = 0; s < pl.ns; ++s) { mbar_init(bar_s + s * 8, 1); }
        mbar_init_fence();
        load_unit();
#pragma unroll 1
        for (int s = 0; s < (PRO == KQP_ANY ? pl.ns : min(pl.ns, p.stages_early)) && issued < n_stage; ++s) { issue_next(); }
    }
    __syncwarp();
    pdl_wait();
    if (EPI < 0) { tp_wait(p.tp, p.error_flag); }
    uint32_t *rec = reinterpret_cast<uint32_t *>(smem_raw);
    if constexpr (PRO == KQP_ANY) {
        if (p.pro == PRO_NORM_QUANT) { kq_prologue<true>(p, nT, rec, col, scale_s); } else { kq_prologue<false>(p, nT, rec, col, scale_s); }
    } else {
        auto rest = [&]() {
            if (lane == 0) {
#pragma unroll 1
                while (issued < min(pl.ns, n_stage)) { issue_next(); }
            }
        };
        constexpr bool NORM = PRO == KQP_NORM || PRO == KQP_NORM_MID || PRO == KQP_NORM_LONG;
        kq_prologue_1col<PG, NORM>(p, rec, scale_s, wearly, rest);
    }
    __syncthreads();

    const uint32_t rec_s = smem_u32(rec), col_bytes = (uint32_t)col * 4u;
    int64_t unit = my_first;
    int round = 0, slot = 0, n = 0;
    uint32_t parity = 0;
    bool ok = true;
    // this lane's super-block in the round: sb of row r of the unit, `first` = the first super-block of that row in the round
    int r = lane / nsb, sb = lane - r * nsb;
    const int r_0 = r, sb_0 = sb;
    // the rows' results are finished one unit later: the residual or the SiLU table entry they meet is on its way meanwhile
    float pend_a = 0.f, pend_b = 0.f;
    float *pend = nullptr;
    auto finish_pending = [&]() { if (pend != nullptr) { *pend = epi == EPI_SILU_MUL ? __fmul_rn(pend_a, pend_b) : __fadd_rn(pend_a, pend_b); pend = nullptr; } };
    for (; n < n_stage; ++n) {
        const int  i = 32 * round + lane;
        const bool have = i < items;
        int        type = TYPE;
        uint16_t   dh = 0;
        if (TYPE != 12) {
            const KqRow u = kq_unit<EPI>(p, unit * pl.np, r & 1);
            type = u.type;
            if (have && type != 12) { dh = __ldg(reinterpret_cast<const uint16_t *>(u.w + (int64_t)(pair_mode ? r >> 1 : r) * u.pitch + (size_t)nsb * 208) + sb); }   // (arrives while the copy is waited for)
        }
        const uint32_t body = type == 12 ? 144u : 208u;
        const int before = min(lane, sb);        // super-blocks of the same row in front of this one in the round
        ok = mbar_wait_bounded(bar_s + slot * 8, parity, WAIT_LIMIT_NS);
        if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
        uint4 w[TYPE == 12 ? 9 : 13];
        const uint32_t src = ring_s + (uint32_t)(slot * pl.stage_bytes) + (uint32_t)(lane - before) * (mixed ? 208u : body) + (uint32_t)before * body;
        if (have) {
#pragma unroll
            for (int k = 0; k < 9; ++k) { w[k] = lds128(src + 16u * k); }
            if (TYPE != 12 && type != 12) {
#pragma unroll
                for (int k = 9; k < 13; ++k) { w[k] = lds128(src + 16u * k); }
            }
        }
        __syncwarp();   // every lane has its super-block in registers: the stage can be refilled
        if (lane == 0 && issued < n_stage) { issue_next(); }
        if (++slot == pl.ns) { slot = 0; parity ^= 1u; }
        if (have) {
            float v[TM];
            if constexpr (TYPE == 12) { kq_values_q4k<TM>(w, rec_s + (uint32_t)(sb * KQ_REC * 4), col_bytes, v); }
            else if constexpr (TYPE == 14) { kq_values_q6k<TM>(w, dh, rec_s + (uint32_t)(sb * KQ_REC * 4), col_bytes, v); }
            else if (type == 12) { kq_values_q4k<TM>(w, rec_s + (uint32_t)(sb * KQ_REC * 4), col_bytes, v); }
            else                 { kq_values_q6k<TM>(w, dh, rec_s + (uint32_t)(sb * KQ_REC * 4), col_bytes, v); }
#pragma unroll
            for (int t = 0; t < TM; ++t) { part[t * items + i] = v[t]; }
        }
        sb += 32;
#pragma unroll 1
        while (sb >= nsb) { sb -= nsb; ++r; }
        if (++round == n_round) {   // the unit is complete: lane = (column, row) adds a row's values in order
            __syncwarp();
            const int ur = lane % n_row, t = lane / n_row;
            float sum = 0.f;
            if (t < nT) {
                const float *q = part + t * items + ur * nsb;
                int k = 0;
#pragma unroll 1
                for (; k + 8 <= nsb; k += 8) {
                    float f[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) { f[e] = q[k + e]; }
#pragma unroll
                    for (int e = 0; e < 8; ++e) { sum = __fadd_rn(sum, f[e]); }
                }
#pragma unroll TAIL
                for (; k < nsb; ++k) { sum = __fadd_rn(sum, q[k]); }
            }
            const float partner = __shfl_xor_sync(0xffffffffu, sum, 1);
            finish_pending();
            if (epi == EPI_SILU_MUL) {
                if (t < nT && (ur & 1) == 0) { pend = p.out + (int64_t)t * p.out_stride + unit * pl.np + (ur >> 1); pend_a = sum; pend_b = p.silu_table[f2h(partner)]; }
            } else if (epi == EPI_RESID) {
                if (t < nT) { const int64_t o = (int64_t)t * p.out_stride + 2 * unit * pl.np + ur; pend = p.out + o; pend_a = sum; pend_b = p.resid[o]; }
            } else { matvec_epilogue<EPI>(p, 2 * unit * pl.np + ur, t, sum, partner, t < nT); }
            __syncwarp();   // (the values are overwritten by the next unit)
            r = r_0; sb = sb_0;
            round = 0; unit += pl.wact;
        }
    }
    finish_pending();
    if (!ok) {
        // a copy did not arrive: report, give the copies still in flight a last bounded chance to land and stop; the host sees the
        // flag at its next synchronisation
        if (lane == 0 && p.error_flag != nullptr) { atomicExch(p.error_flag, 1); }
#pragma unroll 1
        for (int k = n; k < __shfl_sync(0xffffffffu, issued, 0); ++k) {
            mbar_wait_bounded(bar_s + slot * 8, parity, 10000000ull);
            if (++slot == pl.ns) { slot = 0; parity ^= 1u; }
        }
    }
    if (EPI < 0) { tp_publish(p.tp, p.T); }
}

cudaError_t launch_matvec_kq(const MatvecParams &p, const LaunchCfg &cfg) {
    if (p.T < 1 || p.T > KQ_MAX_COLUMNS || p.kq_n < 1 || p.kq_n > 3 || p.A.k % 256 != 0 || p.A.k > 256 * 32 * 4 || p.A.nb != (int)(p.A.k / QK)) { return cudaErrorInvalidValue; }
    if (p.pair_mode ? (p.kq_n != 2 || p.kq[0].n_rows != p.kq[1].n_rows || p.epi != EPI_SILU_MUL) : (p.epi == EPI_SILU_MUL || (p.A.n_rows & 1))) { return cudaErrorInvalidValue; }
    bool q6 = false, q4 = false;
    for (int i = 0; i < p.kq_n; ++i) {
        if ((p.kq[i].type != 12 && p.kq[i].type != 14) || p.kq[i].w == nullptr || (p.kq[i].n_rows & 1) || (reinterpret_cast<uintptr_t>(p.kq[i].w) & 15) || (p.kq[i].row_bytes & 15)) { return cudaErrorInvalidValue; }
        q6 = q6 || p.kq[i].type == 14; q4 = q4 || p.kq[i].type == 12;
    }
    const int nsb = (int)(p.A.k / 256);
    const int TM  = p.T <= 2 ? p.T : KQ_MAX_COLUMNS;
    const int64_t pairs = p.pair_mode ? p.kq[0].n_rows : (p.A.n_rows >> 1);
    const int64_t grid  = std::max<int64_t>(1, std::min<int64_t>(cfg.num_sms, pairs));
    // Pairs per unit: a round costs the same however few of its 32 lanes have a super-block, so short rows share a unit; but a CTA's warps
    // take whole units, so the choice is the one whose busiest warp has the fewest rounds (plus the ordered sum, about 0.7 of a round).
    // Units do not straddle the segments of a virtual matrix. Single columns take the larger of two equal units: half as many warps issue the
    // same instructions (4096 x 2048 Q6_K: 8.2 -> 7.2 us, 3000 x 1536 8.2 -> 6.6).
    KqPlan pl = {1, KQ_WARPS, 1, 32 * (q6 ? 208 : 144)};
    double best = 0.0;
    for (int np = 1; np <= 4; np *= 2) {
        bool whole = pairs % np == 0;
        for (int i = 0; i < p.kq_n && !p.pair_mode; ++i) { whole = whole && p.kq[i].n_rows % (2 * np) == 0; }
        if (!whole) { break; }
        const int64_t units_cta = (pairs / np + grid - 1) / grid;
        const double cost = (double)((units_cta + KQ_WARPS - 1) / KQ_WARPS) * ((2 * np * nsb + 31) / 32 + 0.7);
        if (np == 1 || cost < best || (TM == 1 && cost == best)) { best = cost; pl.np = np; }
    }
    // Warps that stream: all sixteen when two stages each fit the shared memory, fewer otherwise (Q6_K with four columns), down to one
    const size_t budget = 224 * 1024;
    for (pl.wact = KQ_WARPS; pl.wact > 1; --pl.wact) {
        pl.ns = 2;
        if (kq_smem_layout(nsb, TM, pl).total <= budget) { break; }
    }
    if (pl.wact == 1) { pl.ns = 1; }
    while (pl.ns < KQ_MAX_STAGES) { ++pl.ns; if (kq_smem_layout(nsb, TM, pl).total > budget) { --pl.ns; break; } }
    const size_t smem = kq_smem_layout(nsb, TM, pl).total;
    if (smem > budget) { return cudaErrorInvalidValue; }
    using Kernel = void (*)(const MatvecParams, const KqPlan);
    const int ty = q4 && q6 ? 2 : q6 ? 1 : 0;
    Kernel kernel;
    if (TM == 1) {
        static const Kernel one[6][3] = {
            {matvec_kq_kernel<1, 12, KQP_ANY>, matvec_kq_kernel<1, 14, KQP_ANY>, matvec_kq_kernel<1, 0, KQP_ANY>},
            {matvec_kq_kernel<1, 12, KQP_NORM>, matvec_kq_kernel<1, 14, KQP_NORM>, matvec_kq_kernel<1, 0, KQP_NORM>},
            {matvec_kq_kernel<1, 12, KQP_NORM_MID>, matvec_kq_kernel<1, 14, KQP_NORM_MID>, matvec_kq_kernel<1, 0, KQP_NORM_MID>},
            {matvec_kq_kernel<1, 12, KQP_PLAIN>, matvec_kq_kernel<1, 14, KQP_PLAIN>, matvec_kq_kernel<1, 0, KQP_PLAIN>},
            {matvec_kq_kernel<1, 12, KQP_NORM_LONG>, matvec_kq_kernel<1, 14, KQP_NORM_LONG>, matvec_kq_kernel<1, 0, KQP_NORM_LONG>},
            {matvec_kq_kernel<1, 12, KQP_PLAIN_LONG>, matvec_kq_kernel<1, 14, KQP_PLAIN_LONG>, matvec_kq_kernel<1, 0, KQP_PLAIN_LONG>}};
        const int64_t n4 = p.A.k >> 2;
        const bool norm = p.pro == PRO_NORM_QUANT;
        // (One kernel for all of a layer's matrices, whose instructions the next launch finds in the caches, was the faster one below d = 3072 while
        // each held the code of every epilogue. Eight layers of Q4_K / Q6_K, that kernel / these: d = 512, ff 1024: 197.8 / 188.5 us a step; 1536, 3072:
        // 223.6 / 203.7; 2560, 5120: 320.4 / 285.2; 3072, 6144: 341.0 / 299.5.)
        const int pro = n4 <= 2 * KQ_THREADS ? (norm ? KQP_NORM : KQP_PLAIN) : norm && n4 <= 3 * KQ_THREADS ? KQP_NORM_MID : n4 <= 2 * KQ_PRO_GROUPS * KQ_THREADS ? (norm ? KQP_NORM_LONG : KQP_PLAIN_LONG) : KQP_ANY;
        kernel = one[pro][ty];
        if (p.tp.counter == nullptr && p.tp.flag_in == nullptr && (p.epi == EPI_SILU_MUL || p.epi == EPI_QKV_ROPE || p.kq_n == 1)) {
            auto of_type = [&](auto pr, auto ep) -> Kernel {
                constexpr int P = decltype(pr)::value, E = decltype(ep)::value;
                return ty == 0 ? matvec_kq_kernel<1, 12, P, E> : ty == 1 ? matvec_kq_kernel<1, 14, P, E> : matvec_kq_kernel<1, 0, P, E>;
            };
            auto normed = [&](auto pr) -> Kernel {
                return p.epi == EPI_QKV_ROPE ? of_type(pr, std::integral_constant<int, EPI_QKV_ROPE>{}) : p.epi == EPI_SILU_MUL ? of_type(pr, std::integral_constant<int, EPI_SILU_MUL>{})
                     : p.epi == EPI_STORE ? of_type(pr, std::integral_constant<int, EPI_STORE>{}) : kernel;
            };
            if (pro == KQP_NORM) { kernel = normed(std::integral_constant<int, KQP_NORM>{}); }
            else if (pro == KQP_NORM_MID) { kernel = normed(std::integral_constant<int, KQP_NORM_MID>{}); }
            else if (pro == KQP_NORM_LONG) { kernel = normed(std::integral_constant<int, KQP_NORM_LONG>{}); }
            else if (pro == KQP_PLAIN && p.epi == EPI_RESID) { kernel = of_type(std::integral_constant<int, KQP_PLAIN>{}, std::integral_constant<int, EPI_RESID>{}); }
            else if (pro == KQP_PLAIN_LONG && p.epi == EPI_RESID) { kernel = of_type(std::integral_constant<int, KQP_PLAIN_LONG>{}, std::integral_constant<int, EPI_RESID>{}); }
        }
    } else {
        static const Kernel more[2][3] = {{matvec_kq_kernel<2, 12, KQP_ANY>, matvec_kq_kernel<2, 14, KQP_ANY>, matvec_kq_kernel<2, 0, KQP_ANY>},
                                          {matvec_kq_kernel<KQ_MAX_COLUMNS, 12, KQP_ANY>, matvec_kq_kernel<KQ_MAX_COLUMNS, 14, KQP_ANY>, matvec_kq_kernel<KQ_MAX_COLUMNS, 0, KQP_ANY>}};
        kernel = more[TM == 2 ? 0 : 1][ty];
    }
    cudaError_t err = allow_dynamic_smem(reinterpret_cast<const void *>(kernel), smem);
    if (err != cudaSuccess) { return err; }
    MatvecParams q = p;
    if (q.error_flag == nullptr) { q.error_flag = cfg.error_flag; }
    if (cfg.pdl) { q.stages_early = MV_STAGES_EARLY; }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)grid); lc.blockDim = dim3(KQ_THREADS); lc.dynamicSmemBytes = smem; lc.stream = cfg.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr; lc.numAttrs = cfg.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&lc, kernel, q, pl);
}

// upload-time re-layout of Q6_K rows: [sb][ql 128 | qh 64 | scales 16 | d 2] (210 bytes each) ->
// [sb][ql 128 | qh 64 | scales 16] (208 bytes each), then the row's fp16 d values, the row padded to a multiple of 16 bytes
__global__ void kq_relayout_q6k_kernel(const uint8_t *raw, int64_t n_rows, int nsb, uint8_t *dst, int64_t dst_row_bytes) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows * nsb) { return; }
    const int64_t row = i / nsb; const int sb = (int)(i - row * nsb);
    const uint8_t *s = raw + (row * nsb + sb) * 210;
    uint8_t *d = dst + row * dst_row_bytes + (size_t)sb * 208;
    for (int k = 0; k < 208; ++k) { d[k] = s[k]; }
    uint8_t *dd = dst + row * dst_row_bytes + (size_t)nsb * 208 + 2 * sb;
    dd[0] = s[208]; dd[1] = s[209];
}
int64_t kq_row_bytes(int type, int64_t k) {
    const int64_t nsb = k / 256;
    return type == 12 ? nsb * 144 : ((nsb * 210 + 15) / 16) * 16;
}
cudaError_t launch_kq_relayout_q6k(const uint8_t *raw, int64_t n_rows, int64_t k, uint8_t *dst, cudaStream_t s) {
    const int nsb = (int)(k / 256);
    const int64_t n = n_rows * nsb;
    if (n == 0) { return cudaSuccess; }
    kq_relayout_q6k_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(raw, n_rows, nsb, dst, kq_row_bytes(14, k));
    return cudaGetLastError();
}

}  // namespace spyb
