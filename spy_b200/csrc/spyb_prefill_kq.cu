// Prompt evaluation for K-quant weights (Q4_K, Q6_K) as a GEMM on the tcgen05 tensor cores: the K-quant counterpart of
// spyb_prefill.cu, same roles and rings, a different tile and epilogue.
//
// Parity is unpinned by the reference (it defines the K-quant block layouts, orchestration/include/number/number_impl/
// k-quant.h:79-117, 162-188, but no arithmetic for them); what is reproduced bit for bit is the restatement the single-token
// kernel of spyb_kquant.cu follows: activations quantized to Q8_0 first, and per 256-value super-block
//   Q4_K:  acc = 0; for the 8 sub-blocks j of 32 values: acc = fma((d * sc_j) * dx_j, (float)sum(q * y), acc);
//                                                         acc = fma(-((dmin * m_j) * dx_j), (float)sum(y), acc)
//   Q6_K:  acc = 0; for the 16 groups g of 16 values:    acc = fma((d * sc_g) * dx_(g/2), (float)sum(q * y), acc)
// the row's result being the super-blocks' values added in order.
//
// The contraction is dense here: A (128 x 32) = the block's integer weights (Q4_K: 0..15, Q6_K: -32..31), B (TT x 32) = the tokens'
// activation values, both as f16 (8-bit integers are exact in it, products and sums of a block's 32 products are exact in f32). Q4_K takes
// one sum per (row, token, block): two MMAs of K = 16 onto the same columns; Q6_K one per half block (its scales are per 16 values): two
// MMAs onto columns of their own. The quantizer writes the activations as the B operand itself (K-major, no swizzle), so that no warp
// has to expand anything. The weight tile carries, per row, the two f32 products the restatement forms first (Q4_K: d * sc_j and
// dmin * m_j; Q6_K: d * sc of the two groups), made at upload with the same f32 multiplication.
#include "spyb_tc.cuh"

#include <algorithm>
#include <type_traits>

namespace spyb {

namespace {

constexpr int KQ_WT = PF_KQ_WTILE;
constexpr int KQ_EPI_WARPS = 16, KQ_GEMM_THREADS = 608;   // sixteen epilogue warps, the copy warp, two MMA warps: 104 registers each
// Persistent CTAs (one per SM), tiles of 128 rows x TT tokens walked along K in steps of NB blocks, two D buffers of up to 256 columns, as in
// prefill_gemm_kernel. Wide tiles for prompts; narrow ones, whose steps are mostly weights, when wide ones would be mostly padding.
//
// Bound of the wide tile: issue slots. Per (row, token, block) two multiplications and two FMAs, packed two tokens at a time, and eight
// uniform 128-bit shared-memory reads of the token scales per 16 tokens.
// Q4_K_M, 8 layers, 512 tokens: 8.2 ms in all (whole tiles only: 8.7; one 64-token tile per CTA with 8-bit operands: 14.3); 4 layers, 16 tokens: 0.86 (2.43).
template <int TT> struct KqGeom {
    static constexpr int NB    = TT == 64 ? 2 : 4;            // blocks per step
    static constexpr int YB    = TT * 72;                     // a block's activations: TT x 32 f16, TT scales, TT sums
    static constexpr int STAGE = NB * (KQ_WT + YB);
    static constexpr int NS    = TT == 64 ? 6 : 4;            // steps in the ring
    static constexpr int PW    = TT / 8;                      // token pairs per epilogue warp
    static constexpr size_t SMEM = (size_t)NS * STAGE + 8 * (2 * NS + 4) + 16;
};

__device__ __forceinline__ float2 lds64f(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
template <int N> __device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t *r) {
    if constexpr (N == 16) { tmem_ld16(taddr, r); } else if constexpr (N == 8) { tmem_ld8(taddr, r); } else { tmem_ld4(taddr, r); }
}

template <int WT, int TT, bool SHARE, bool LATE>   // WT: 12 = Q4_K, 14 = Q6_K; SHARE: the last tiles are cut among the CTAs, between super-blocks (PfItem)
__global__ void __launch_bounds__(KQ_GEMM_THREADS, 1) prefill_kq_gemm_kernel(PrefillGemm g) {
    using G = KqGeom<TT>;
    constexpr int NB = G::NB, NS = G::NS, PW = G::PW, YB = G::YB, H = WT == 14 ? 2 : 1, TW = TT / 4;   // H sums per (row, token, block), TW tokens per epilogue warp
    static_assert(NB * TT * H <= 256 && 8 % NB == 0, "a step fits a D buffer and super-blocks end with a step");
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem), bars = sbase + NS * G::STAGE;
    // a stage: [NB weight tiles][NB blocks of activations]
    auto raw_full = [&](int s) { return bars + 8u * s; };                       // the step's weights and activations have landed
    auto st_free  = [&](int s) { return bars + 8u * (NS + s); };                // the stage may be refilled (arrival by the MMA warp that waits for the step's D buffer)
    auto d_full   = [&](int i) { return bars + 8u * (2 * NS + i); };            // the MMAs into buffer i have completed
    auto d_free   = [&](int i) { return bars + 8u * (2 * NS + 2 + i); };        // buffer i has been read (one arrival per epilogue warp)
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + (size_t)NS * G::STAGE + 8 * (2 * NS + 4));

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nb = g.nb;                                                        // (a multiple of 8)
    const int n_tok = (g.T + TT - 1) / TT;
    const int n_tile = n_tok * (int)((g.n_rows + PF_M - 1) / PF_M);
    const uint64_t limit = g.wait_limit_ns;
    constexpr int SB = 8 / NB;                                                  // steps of a super-block
    const int n_super = nb / 8;
    auto first_item = [&]() -> PfItem {
        if constexpr (SHARE) { return pf_share_item(g.share, n_tile, n_super, (int)blockIdx.x, (int)gridDim.x, 0); }
        return {(int)blockIdx.x, 0, n_super, 0};
    };
    auto next_item = [&](PfItem &it) {
        if constexpr (SHARE) { it = pf_share_item(g.share, n_tile, n_super, (int)blockIdx.x, (int)gridDim.x, it.q + 1); }
        else { it.tile += gridDim.x; }
    };

    pdl_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) { mbar_init(raw_full(s), 1); mbar_init(st_free(s), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(d_full(i), 1); mbar_init(d_free(i), KQ_EPI_WARPS); }
        mbar_init_fence();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    uint64_t left_ns = limit;   // (zero once a wait has run out)

    if (warp == KQ_EPI_WARPS) {
        // ---- copies; the weights of the first tile's first steps do not wait for the previous kernel
        int st = 0, k = 0, issued = 0;
        uint32_t par = 1;
        bool ok = true;
        const PfItem first = first_item();
        const int early = first.tile < n_tile ? min(NS, (first.to - first.from) * SB) : 0;
        if (elect_one()) {
            for (int i = 0; i < early; ++i) {
                mbar_expect_tx(raw_full(i), (uint32_t)G::STAGE);
                bulk_copy_g2s(sbase + (uint32_t)i * G::STAGE, g.w + ((int64_t)(first.tile / n_tok) * nb + first.from * 8 + i * NB) * KQ_WT, (uint32_t)(NB * KQ_WT), raw_full(i));
            }
        }
        __syncwarp();
        pdl_wait();
        for (PfItem it = first; it.tile < n_tile && ok; next_item(it)) {
            const uint8_t *wsrc = g.w + ((int64_t)(it.tile / n_tok) * nb + it.from * 8) * KQ_WT;
            const uint8_t *ysrc = g.yq + ((int64_t)(it.tile % n_tok) * nb + it.from * 8) * YB;
            for (int i = it.from * SB; i < it.to * SB; ++i, ++k) {
                if (k >= NS) {
                    ok = __all_sync(0xffffffffu, mbar_wait_relaxed(st_free(st), par, limit));
                    if (!ok) { break; }
                }
                if (elect_one()) {
                    const uint32_t dst = sbase + (uint32_t)st * G::STAGE;
                    if (k >= early) {
                        mbar_expect_tx(raw_full(st), (uint32_t)G::STAGE);
                        bulk_copy_g2s(dst, wsrc, (uint32_t)(NB * KQ_WT), raw_full(st));
                    }
                    bulk_copy_g2s(dst + NB * KQ_WT, ysrc, (uint32_t)(NB * YB), raw_full(st));
                }
                __syncwarp();
                issued = k + 1;
                wsrc += NB * KQ_WT; ysrc += NB * YB;
                if (++st == NS) { st = 0; par ^= 1u; }
            }
        }
        if (!ok && lane == 0) { pf_report(g.error_flag, 4); }
        // no copy of this CTA is in flight when it leaves
        for (int j = max(0, issued - NS); j < issued; ++j) {
            if (!mbar_wait_relaxed(raw_full(j % NS), (uint32_t)(j / NS) & 1u, limit)) { if (lane == 0) { pf_report(g.error_flag, 4); } break; }
        }
    } else if (warp > KQ_EPI_WARPS) {
        // ---- MMAs: warp m takes the steps of D buffer m; columns of block j and sum h: (j H + h) TT + token
        const int m = warp - (KQ_EPI_WARPS + 1);
        const uint32_t d0 = tmem + (uint32_t)m * 256u;
        int st = 0, k = 0, mine = 0;
        uint32_t par = 0;
        for (PfItem it = first_item(); it.tile < n_tile && left_ns != 0; next_item(it)) {
            for (int i = it.from * SB; i < it.to * SB; ++i, ++k) {
                if ((k & 1) == m) {
                    mbar_wait_lean(d_free(m), (uint32_t)mine & 1u, left_ns);
                    if (left_ns != 0 && mine > 0 && lane == 0) { mbar_arrive(st_free(st >= 2 ? st - 2 : st + NS - 2)); }   // (the step before on this buffer has been read)
                    mbar_wait_lean(raw_full(st), par, left_ns);
                    if (left_ns == 0) { break; }
                    tc_fence_after();
                    const uint32_t base = sbase + (uint32_t)st * G::STAGE;
                    const uint64_t a0 = operand_desc(base, 2048u, 128u), b0 = operand_desc(base + NB * KQ_WT, 16u * TT, 128u);
                    if (elect_one()) {
#pragma unroll
                        for (int j = 0; j < NB; ++j) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                mma_f16_ss(d0 + (uint32_t)((j * H + (H == 2 ? h : 0)) * TT), a0 + (uint64_t)((j * KQ_WT + h * 4096) >> 4), b0 + (uint64_t)((j * YB + h * 32 * TT) >> 4),
                                           idesc_f16(TT), H == 1 && h == 1 ? 1u : 0u);
                            }
                        }
                        mma_commit(d_full(m));
                    }
                    __syncwarp();
                    ++mine;
                }
                if (++st == NS) { st = 0; par ^= 1u; }
            }
        }
        if (left_ns == 0 && lane == 0) { pf_report(g.error_flag, 5); }
        // every MMA has completed (it reads shared memory and writes tensor memory) before the CTA leaves
        if (mine > 0 && !mbar_wait_relaxed(d_full(m), (uint32_t)(mine - 1) & 1u, limit)) { if (lane == 0) { pf_report(g.error_flag, 5); } }
    } else {
        pdl_wait();
        // ---- epilogue: row 32 (warp % 4) + lane, tokens part * TW .. of the tile as PW packed pairs
        const int quad = warp & 3, part = warp >> 2;
        const int row = 32 * quad + lane;
        const uint32_t tbase = tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(part * TW);
        const uint32_t sc_addr = sbase + 8192u + 8u * (uint32_t)row, dx_addr = sbase + NB * KQ_WT + TT * 64 + 4u * (uint32_t)(part * TW);
        uint64_t acc[PW], tot[PW];
#pragma unroll
        for (int u = 0; u < PW; ++u) { acc[u] = 0ull; tot[u] = 0ull; }
        if (lane == 0) { mbar_arrive(d_free(0)); mbar_arrive(d_free(1)); }
        int st = 0, k = 0;
        for (PfItem it = first_item(); it.tile < n_tile; next_item(it)) {
            const int tile = it.tile;
            if constexpr (SHARE) if (it.from > 0) {   // the sums of the super-blocks in front are another CTA's
                const int64_t at = (int64_t)((int)blockIdx.x - 1) * KQ_EPI_WARPS + warp;
                handoff_wait(g.handoff_flags + at, left_ns);
#pragma unroll
                for (int u = 0; u < PW; ++u) { tot[u] = __ldcg(reinterpret_cast<const unsigned long long *>(g.handoff) + (at * 16 + u) * 32 + lane); }
                __syncwarp();
                if (lane == 0) { g.handoff_flags[at] = 0u; }
            }
#pragma unroll 1
            for (int i = SHARE ? it.from * SB : 0; i < it.to * SB; ++i, ++k) {
                const int buf = k & 1;
                const uint32_t stage = (uint32_t)st * G::STAGE, tb = tbase + (uint32_t)buf * 256u;
                mbar_wait_lean(d_full(buf), (uint32_t)(k >> 1) & 1u, left_ns);
                tc_fence_after();
                uint32_t r[2][TW * H];
#pragma unroll
                for (int h = 0; h < H; ++h) { tmem_ld_n<TW>(tb + (uint32_t)(h * TT), r[0] + h * TW); }
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    const float2 sc = lds64f(sc_addr + stage + (uint32_t)j * KQ_WT);
                    const uint64_t scx = f2_pack(sc.x, sc.x), scy = WT == 12 ? f2_pack(-sc.y, -sc.y) : f2_pack(sc.y, sc.y);   // (the negation commutes with the rounding of the product)
                    uint64_t dx[PW], ys[PW];
                    const uint32_t xa = dx_addr + stage + (uint32_t)j * YB;
#pragma unroll
                    for (int u = 0; u < PW; u += 2) {
                        lds128_2x64(xa + 8u * u, dx[u], dx[u + 1]);
                        if (WT == 12) { lds128_2x64(xa + 4u * TT + 8u * u, ys[u], ys[u + 1]); }
                    }
                    tmem_ld_wait();
                    if (j + 1 < NB) {   // the next block's columns arrive while this one's are folded
#pragma unroll
                        for (int h = 0; h < H; ++h) { tmem_ld_n<TW>(tb + (uint32_t)(((j + 1) * H + h) * TT), r[(j + 1) & 1] + h * TW); }
                    } else {            // the whole buffer is in registers and the step's scales have been read
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) { mbar_arrive(d_free(buf)); }
                    }
                    const uint32_t *rj = r[j & 1];
#pragma unroll
                    for (int u = 0; u < PW; ++u) {
                        acc[u] = f2_fma(f2_mul(scx, dx[u]), f2_pack_bits(rj[2 * u], rj[2 * u + 1]), acc[u]);
                        acc[u] = f2_fma(f2_mul(scy, dx[u]), WT == 12 ? ys[u] : f2_pack_bits(rj[TW * (H - 1) + 2 * u], rj[TW * (H - 1) + 2 * u + 1]), acc[u]);
                    }
                }
                if (((i + 1) * NB) % 8 == 0) {   // a super-block ends: its value joins the row's sum
#pragma unroll
                    for (int u = 0; u < PW; ++u) { tot[u] = f2_add(tot[u], acc[u]); acc[u] = 0ull; }
                }
                if (++st == NS) { st = 0; }
            }
            if constexpr (SHARE) if (it.to < n_super) {   // another CTA goes on with these sums
                const int64_t at = (int64_t)blockIdx.x * KQ_EPI_WARPS + warp;
#pragma unroll
                for (int u = 0; u < PW; ++u) { __stcg(reinterpret_cast<unsigned long long *>(g.handoff) + (at * 16 + u) * 32 + lane, (unsigned long long)tot[u]); tot[u] = 0ull; }
                if constexpr (LATE) { const uint64_t t0 = global_timer_ns(); while (global_timer_ns() - t0 < 3 * limit) {} }   // (failure-path check)
                __syncwarp();
                if (lane == 0) { handoff_publish(g.handoff_flags + at); }
                continue;
            }
            const int64_t orow = (int64_t)(tile / n_tok) * PF_M + row;
            const int     tok0 = (tile % n_tok) * TT + part * TW;
#pragma unroll
            for (int u = 0; u < PW; ++u) {
                float v[2];
                f2_unpack(tot[u], v[0], v[1]);
                tot[u] = 0ull;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int token = tok0 + 2 * u + e;
                    if (token < g.T && orow < g.n_rows) {   // (the last row tile may be partly padding)
                        const int64_t o = (int64_t)token * g.out_stride + orow;
                        g.out[o] = g.resid != nullptr ? __fadd_rn(v[e], g.resid[o]) : v[e];
                    }
                }
            }
        }
        if (left_ns == 0 && lane == 0) { pf_report(g.error_flag, 6); }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// element k of a block's row at its place in the f16 operand tile (core matrices of 8 rows x 16 bytes, 2048 bytes per eight elements)
__device__ __forceinline__ __half *tile_elem(uint8_t *tile, int r, int k) { return reinterpret_cast<__half *>(tile + (k >> 3) * 2048 + r * 16) + (k & 7); }

// upload-time re-layout: GGUF super-blocks (Q4_K 144 B, Q6_K 210 B per 256 values) of rows [0, n_rows) -> tiles of 128 rows x one
// 32-element block: the integer weights as f16, then per row the two f32 scale products of the block. One thread per (row, block),
// consecutive threads consecutive rows: their stores are contiguous.
template <int WT>
__global__ void prefill_kq_retile_kernel(const uint8_t *raw, int64_t row_stride, int64_t n_rows, int nb, uint8_t *base, int64_t dst_row0) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows * nb) { return; }
    const int     b = (int)(i / n_rows), sb = b >> 3, j = b & 7;
    const int64_t lrow = i - (int64_t)b * n_rows;
    const int64_t row = dst_row0 + lrow;
    const int     r = (int)(row % PF_M);
    uint8_t *tile = base + ((row / PF_M) * nb + b) * (int64_t)KQ_WT;
    float *scales = reinterpret_cast<float *>(tile + 8192 + 8 * r);
    if (WT == 12) {
        const uint8_t *s = raw + lrow * row_stride + (int64_t)sb * 144;
        const float d = h2f((uint16_t)(s[0] | (s[1] << 8))), dmin = h2f((uint16_t)(s[2] | (s[3] << 8)));
        const uint8_t *sc12 = s + 4, *qs = s + 16 + 32 * (j >> 1);
        uint32_t sc, mn;
        if (j < 4) { sc = sc12[j] & 63u; mn = sc12[j + 4] & 63u; }
        else { sc = (sc12[j + 4] & 0xFu) | ((sc12[j - 4] >> 6) << 4); mn = (uint32_t)(sc12[j + 4] >> 4) | ((uint32_t)(sc12[j] >> 6) << 4); }
        scales[0] = __fmul_rn(d, (float)sc);
        scales[1] = __fmul_rn(dmin, (float)mn);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int q0 = qs[8 * c + 2 * e], q1 = qs[8 * c + 2 * e + 1];
                v[e] = (uint32_t)__half_as_ushort(__int2half_rn((j & 1) ? q0 >> 4 : q0 & 15)) | ((uint32_t)__half_as_ushort(__int2half_rn((j & 1) ? q1 >> 4 : q1 & 15)) << 16);
            }
            *reinterpret_cast<uint4 *>(tile_elem(tile, r, 8 * c)) = make_uint4(v[0], v[1], v[2], v[3]);
        }
    } else {
        const uint8_t *s = raw + lrow * row_stride + (int64_t)sb * 210;
        const uint8_t *ql = s, *qh = s + 128;
        const int8_t *sc = reinterpret_cast<const int8_t *>(s + 192);
        const float d = h2f((uint16_t)(s[208] | (s[209] << 8)));
        const int hf = j >> 2, seg = j & 3;                  // half of the super-block, segment of 32 values
        scales[0] = __fmul_rn(d, (float)sc[2 * j]);
        scales[1] = __fmul_rn(d, (float)sc[2 * j + 1]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t v[4];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int l = 8 * c + e, lo = ql[64 * hf + 32 * (seg & 1) + l], h = qh[32 * hf + l];
                const int q = ((seg & 2) ? (lo >> 4) : (lo & 0xF)) | (((h >> (2 * seg)) & 3) << 4);
                const uint32_t x = __half_as_ushort(__int2half_rn(q - 32));
                v[e >> 1] = (e & 1) ? v[e >> 1] | (x << 16) : x;
            }
            *reinterpret_cast<uint4 *>(tile_elem(tile, r, 8 * c)) = make_uint4(v[0], v[1], v[2], v[3]);
        }
    }
}

template <int WT, int TT, bool SHARE, bool LATE = false>
cudaError_t launch_kq_t(const PrefillGemm &g, cudaStream_t stream, bool pdl) {
    const size_t smem = KqGeom<TT>::SMEM;
    cudaError_t err = allow_dynamic_smem(reinterpret_cast<const void *>(prefill_kq_gemm_kernel<WT, TT, SHARE, LATE>), smem);
    if (err != cudaSuccess) { return err; }
    const int64_t tiles = (int64_t)((g.T + TT - 1) / TT) * ((g.n_rows + PF_M - 1) / PF_M), walkers = std::min<int64_t>(tiles, device_sms());
    PrefillGemm h = g;
    h.share = {(int)(tiles / walkers), 0, (int)(tiles % walkers), 0};
    if (SHARE) { h.share = pf_share((int)tiles, g.nb / 8, (int)walkers); }
    return launch_maybe_pdl(prefill_kq_gemm_kernel<WT, TT, SHARE, LATE>, dim3((unsigned)walkers), KQ_GEMM_THREADS, smem, stream, pdl, h);
}

}  // namespace

// Tokens a tile: 16, 32 or 64 (tok 0: any), and whether the last tiles are shared; by the cost of pf_cost, one for both types, so that the matrices of a layer that read the
// same activations agree on a width. Fitted to 1353 sizes of both (1024 x 1536 to 32000 x 11264, 5 to 512 tokens), timed with the submits of one backend and with those of three
// in turn. At 626 other sizes a model's choice is 0.13 % behind the fastest on average, more than 3 % at 8 (Q6_K 12232 x 8192 x 83 7.5 %). An operator's, against
// widths by whole rounds alone: one backend 3.7 % faster on average (more than 3 % slower at 4 of 476), three 1.1 % (at 40); with a model's rule 4.2 % and 0 % (at 72).
// us a submit from one backend / three, whole and shared tiles: Q4_K 11008 x 4096 x 64, 32 tokens a tile 45.4 / 28.5 and 32.5 / 29.7; 64 tokens a tile: Q4_K
// 5120 x 5120 x 512 141.8 / 110.2 and 108.4 / 105.1, 4096 x 4096 x 512 79.0 / 73.7 and 72.9 / 70.3; Q6_K 4096 x 11008 x 512 196.7 / 171.5 and 175.0 / 169.7.
int prefill_kq_tile_tokens(int64_t n_rows, int nb, int T, int tok, int how, bool beside, int sms, bool *share) {
    static constexpr struct { int tok; PfCost cost; } WIDTHS[3] = {
        {16, {3420, 100, 98.6, 78.2, 4010, 0.003, 250}}, {32, {4370, 230, 137.6, 61.1, 3310, -0.026, 1560}}, {64, {4610, 800, 271.1, 2.6, 5760, -0.052, 1260}}};
    static constexpr PfRule RULE = {0.91, 1.22, 430};
    int best = 0;
    double best_ns = 0.0;
    for (const auto &w : WIDTHS) {
        if (tok != 0 && tok != w.tok) { continue; }
        const int64_t row_tiles = (n_rows + PF_M - 1) / PF_M;
        bool shared;
        const double ns = pf_cost(w.cost, RULE, row_tiles, row_tiles * ((T + w.tok - 1) / w.tok), sms, nb, sms, how, nb >= 16, beside, &shared);
        if (best == 0 || ns < best_ns) { best = w.tok; best_ns = ns; *share = shared; }
    }
    return best;
}

cudaError_t launch_prefill_gemm_kq(const PrefillGemm &g, cudaStream_t stream, bool pdl) {
    if (g.w == nullptr || g.yq == nullptr || g.out == nullptr || g.T < 1 || g.nb < 8 || (g.nb & 7) || g.n_rows < 1 || (g.type != 12 && g.type != 14)) { return cudaErrorInvalidValue; }
    bool share = false;
    prefill_kq_tile_tokens(g.n_rows, g.nb, g.T, g.tile_tok, g.tiles, g.beside, device_sms(), &share);
    auto of_width = [&](auto tt) {
        constexpr int TT = decltype(tt)::value;
        if (share && g.handoff != nullptr) { return g.type == 12 ? launch_kq_t<12, TT, true>(g, stream, pdl) : launch_kq_t<14, TT, true>(g, stream, pdl); }
        return g.type == 12 ? launch_kq_t<12, TT, false>(g, stream, pdl) : launch_kq_t<14, TT, false>(g, stream, pdl);
    };
    if (g.selftest_late) { return !share || g.handoff == nullptr || g.type != 12 || g.tile_tok != 16 ? cudaErrorInvalidValue : launch_kq_t<12, 16, true, true>(g, stream, pdl); }
    switch (g.tile_tok) {
    case 64: return of_width(std::integral_constant<int, 64>{});
    case 32: return of_width(std::integral_constant<int, 32>{});
    case 16: return of_width(std::integral_constant<int, 16>{});
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_prefill_retile_kq(int type, const uint8_t *raw, int64_t row_stride, int64_t n_rows, int nb, uint8_t *base, int64_t dst_row0, cudaStream_t stream) {
    if ((type != 12 && type != 14) || n_rows < 1 || nb < 8 || (nb & 7)) { return cudaErrorInvalidValue; }
    const int64_t n = n_rows * nb;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (type == 12) { prefill_kq_retile_kernel<12><<<blocks, 256, 0, stream>>>(raw, row_stride, n_rows, nb, base, dst_row0); }
    else            { prefill_kq_retile_kernel<14><<<blocks, 256, 0, stream>>>(raw, row_stride, n_rows, nb, base, dst_row0); }
    return cudaGetLastError();
}

}  // namespace spyb
