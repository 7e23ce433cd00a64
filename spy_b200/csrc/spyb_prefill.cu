// Prompt evaluation as a dequant-fused GEMM on the 5th-generation tensor cores (tcgen05, accumulators in tensor memory).
//
// The reference evaluates MatMul(W[Q4_0 | Q8_0], x) for a prompt of T tokens as T independent dot products per row
// (backend/host/operator/mat.cpp:95-128 with Dot<Q4_0,Q8_0> / Dot<Q8_0,Q8_0>, backend/host/include/simd/vec_dot.h:42-115):
// per 32-element block the eight integer "lane sums" (4 products each) are converted to f32 and folded into eight f32
// accumulators with acc = fma(d_w * d_x, lane_sum, acc), block after block, and the eight accumulators meet in the
// hsum_float_8 tree at the end of the row. Only the integer lane sums are a contraction; everything after them is
// order-bound f32 work. So the tensor core computes the lane sums of a block for 128 rows x TT tokens, half a block at a time:
//
//   A (128 x 16)   = the half block's weights of 128 rows
//   B (4 TT x 16)  = for token t and accumulator n (four per half) the row 8 (t / 2) + 2 n + t % 2 holds the four activation values of
//                    accumulator n at their place and zeros elsewhere
//   D (128 x 4 TT, tensor memory) = A B^T: one lane sum per row, token and accumulator
//
// with f16 operands and f32 accumulators (tcgen05.mma kind::f16, K = 16). Every 8-bit integer is exact in f16, products and sums of four
// of them are exact in f32: D holds (float)lane_sum itself, for Q4_0 and Q8_0 weights alike. (An earlier form with e4m3 operands, K = 32,
// had to split every 8-bit value in two and take two MMAs of twice the columns per block for Q4_0 and four for Q8_0.)
// The epilogue warps read D back with tcgen05.ld (lane = row) and run the CPU's FMA chains in block order on f32 accumulators held as
// packed f32x2 pairs of neighbouring tokens, whose scales come as pairs from shared memory. Operands reach shared memory by
// cp.async.bulk (weights in a 128-row x 1-block tile layout made at upload, activations as compact blocks); an expander warp writes the
// activations into the canonical K-major no-swizzle operand layout (core matrices of 8 rows x 16 bytes). Every wait is bounded.
#include "spyb_tc.cuh"
#include "spyb_mv_common.cuh"

#include <algorithm>
#include <type_traits>
#include <vector>

namespace spyb {

namespace {

constexpr int PF_HALF = 4096;   // bytes of half a block's weights: 16 f16 values of 128 rows
constexpr int PF_QUANT_THREADS = 512;
constexpr int PF_QUANT_GROUPS  = (PF_MAX_K + 8 * PF_QUANT_THREADS - 1) / (8 * PF_QUANT_THREADS);   // groups of eight values per thread of the widest row

// ---------------------------------------------------------------------------------------------
// the GEMM: persistent CTAs (one per SM, all 512 tensor-memory columns), each walking tiles of 128 rows x TT tokens along K in
// steps of NB = 32 S / TT blocks, so that a step is 256 columns of D whatever the tile's width; two D buffers. 20 warps (96 registers):
//   warps 0-15  epilogue: row = 32 (warp % 4) + lane, a quarter of the tile's tokens; four warps per scheduler hide the latency of tensor
//               memory and of the hand-offs behind one another's FMAs
//   warp 16     streams the operands of step after step with cp.async.bulk (weights: A operands as they are; compact activations)
//   warp 17     expands the compact activations into the B operands
//   warps 18-19 issue the MMAs of alternate steps and one commit each
// The pipeline does not drain between tiles: copies, expansion and MMAs run on into the next tile while a tile's rows are stored.
//
// Bound: no unit is full. A step is 32 packed FMAs and 4 packed multiplies per epilogue warp, 144 a scheduler, each measured at 2.2-2.4 cycles, and 157 other
// instructions a scheduler; the loop is written for few of them (waits of one test and one branch, D buffers as constants of the unrolled code, one
// arrival per step) and measures 548 cycles per step, the FMA pipes 56 % busy, the issue slots 55 %, the tensor pipe 23 %: the folds wait for what they read from
// tensor and shared memory, four warps a scheduler hide part of that, and no register is left to ask for it earlier. 4096 x 4096 x 448 tokens 127 us (138
// with whole tiles only), 22016 rows 628 us (the e4m3 form: 216 and 1017 us). Tiles of
// 32 tokens halve the weight bytes per FMA but need 110 registers: spills, 265 us. Eight epilogue warps with 216 registers each: 186-208 us. (The
// epilogue's registers are all taken, which is why its loop is written as PTX, pf_fold_steps: the compiler's own order of the same loop measured
// between 640 and 709 us on the 22016 rows, depending on code beside it.)
//
// S = 2: few tokens of a matrix of few rows are fewer tiles than SMs, and a CTA takes no more than some 55 GB/s of weights. A cluster of two
// CTAs then shares a tile by the halves of its blocks: the eight accumulators of an output are independent chains until the row's end, four
// of them read the first 16 values of every block and four the others, so each CTA streams and multiplies one half of the weights (the
// scales lie between the halves) for four chains of twice the blocks per step, and at the end of a tile the second CTA's epilogue warps leave their sums in
// the first one's shared memory, where they are added in the tree's order. 4096 x 11008 x 8 tokens 52 -> 32.5 us, 4096 x 4096 x 8 20.8 -> 15.1.
// Where the tiles fill the chip it costs more (a scale product for every four FMAs, the scales twice): best_form has the line.
template <int TT, int S, bool MANY> struct PfGeom {
    static constexpr int NB     = 32 * S / TT;                            // blocks per step
    static constexpr int YB     = TT * 64 + TT * 4;                       // a block's compact activations: TT x 32 f16, TT f32 scales
    static constexpr int HS     = 2 / S;                                  // halves of a block that a CTA takes
    static constexpr int WB     = HS * PF_HALF + 512;                     // a block's weights: its halves, the scales (between them, so that both lie beside either)
    static constexpr int RAW    = NB * (WB + YB);                         // a step as it arrives
    static constexpr int STAGE  = RAW + 8192;                             // ... and its B operands
    // steps in the ring (even). Few tokens of wide tiles wait for weights: eight steps, 22016 x 4096 x 32 tokens 63.4 -> 57.9 us, 15360 x 5120 x 32 57.6 ->
    // 53.2. Many tokens find them in L2: 4096 x 4096 x 448 126.0 with six, 127.8 with eight; 4096 x 11008 x 448 327.7 / 320.8; 22016 x 4096 x 448 640 / 648.
    static constexpr int NS     = TT == 16 ? (S == 1 && !MANY ? 8 : 6) : 4;
    static constexpr int PW     = TT / 8;                                 // token pairs per epilogue warp
    static constexpr int PC     = PW < 2 ? 1 : 2;                         // pairs per chunk of tensor-memory columns (8 columns each)
    static constexpr int NC     = NB * HS * (PW / PC);                    // chunks per step and warp
    static constexpr int XCH    = S == 2 ? PF_GEMM_EPI_WARPS * 32 * PW * 4 * 8 : 0;   // the other CTA's accumulators
    static constexpr int BARS   = NS * STAGE + XCH;
    static constexpr int N_BAR  = 3 * NS + 4 + (S == 2 ? 2 * PF_GEMM_EPI_WARPS : 0);
    static constexpr size_t SMEM = (size_t)BARS + 8 * N_BAR + 16;
};


// The epilogue's loop over the steps of 16-token tiles, two a turn (D buffers 0 and 1), as one piece of PTX: the accumulators stay where they are. The same
// loop in C++ is at the mercy of what surrounds it: its accumulators are given other registers from copy to copy of the step, and some ten moves
// per step and warp bring them back (12288 x 4096 x 448 tokens, shared tiles: 412 us; as PTX 366).
// A step's chunks are 16 columns of D, half a block's sums of the warp's four tokens; the second block's are requested under the folds of
// the first one's. (Each chunk requested, waited for and folded in turn: 401 us where this takes 381; one chunk ahead 426, its registers spill.)
// Operands: %0-%15 accumulators [pair][4 half + n], %16 tensor-memory address, %17 limit (ns), %18 stage offset, %19 parity, %20 turns; %21, %22 addresses of the
// row's and the tokens' scales in stage 0, %23 d_full(0), %24 lane; %25 bytes of a stage, %26 of the ring, %27 of a block's weights, %28 of its activations.
#define PF_FMA(A, SC, X, Y) "mov.b64 t, {" X ", " Y "};\n\tfma.rn.f32x2 %" A ", " SC ", t, %" A ";\n\t"
#define PF_FOLD(R, A0, A1, A2, A3, A4, A5, A6, A7) PF_FMA(A0, "s0", R "0", R "1") PF_FMA(A1, "s0", R "2", R "3") PF_FMA(A2, "s0", R "4", R "5") PF_FMA(A3, "s0", R "6", R "7") \
    PF_FMA(A4, "s1", R "8", R "9") PF_FMA(A5, "s1", R "10", R "11") PF_FMA(A6, "s1", R "12", R "13") PF_FMA(A7, "s1", R "14", R "15")
#define PF_FOLD_FIRST(R)  PF_FOLD(R, "0", "1", "2", "3", "8", "9", "10", "11")
#define PF_FOLD_SECOND(R) PF_FOLD(R, "4", "5", "6", "7", "12", "13", "14", "15")
#define PF_READ(R, COL) "add.u32 a, %16, " COL ";\n\ttcgen05.ld.sync.aligned.32x32b.x16.b32 {" R "0," R "1," R "2," R "3," R "4," R "5," R "6," R "7," R "8," R "9," R "10," R "11," R "12," R "13," R "14," R "15}, [a];\n\t"
#define PF_READ_WAIT "tcgen05.wait::ld.sync.aligned;\n\t"
#define PF_SCALES(W, Y) "add.u32 a, %21, %18;\n\tld.shared.f32 dw, [a+" W "];\n\tadd.u32 a, %22, %18;\n\tld.shared.v2.b64 {x0, x1}, [a+" Y "];\n\t"
#define PF_PRODUCTS "mov.b64 t, {dw, dw};\n\tmul.rn.f32x2 s0, t, x0;\n\tmul.rn.f32x2 s1, t, x1;\n\t"
#define PF_D_FULL(OFF, L) "mbarrier.try_wait.parity.shared::cta.b64 p, [%23+" OFF "], %19;\n\t@p bra D" L "_%=;\n\tmov.u64 t0, %%globaltimer;\nA" L "_%=:\n\t" \
    "mbarrier.try_wait.parity.shared::cta.b64 p, [%23+" OFF "], %19;\n\t@p bra D" L "_%=;\n\tmov.u64 t1, %%globaltimer;\n\tsub.u64 t1, t1, t0;\n\tsetp.lt.u64 q, t1, %17;\n\t@q bra A" L "_%=;\n\tmov.u64 %17, 0;\nD" L "_%=:\n\ttcgen05.fence::after_thread_sync;\n\t"
#define PF_D_FREE(OFF) "tcgen05.fence::before_thread_sync;\n\tbar.warp.sync 0xffffffff;\n\t@lead mbarrier.arrive.shared::cta.b64 _, [%23+" OFF "];\n\t"
#define PF_STEP(C0, C1, C2, C3, FULL, FREE, L) PF_D_FULL(FULL, L) \
    PF_READ("r", C0) PF_READ("u", C1) PF_SCALES("0", "0") PF_PRODUCTS PF_READ_WAIT PF_FOLD_FIRST("r") PF_READ("r", C2) PF_SCALES("%27", "%28") PF_FOLD_SECOND("u") PF_PRODUCTS \
    PF_READ("u", C3) PF_READ_WAIT PF_D_FREE(FREE) PF_FOLD_FIRST("r") PF_FOLD_SECOND("u") "add.u32 %18, %18, %25;\n\t"
template <class G>
__device__ __forceinline__ void pf_fold_steps(uint64_t (&acc)[2][8], int turns, uint32_t tbase, uint32_t dw_addr, uint32_t dx_addr, uint32_t d_bars, int lane, uint32_t &stage, uint32_t &par, uint64_t &limit_ns) {
    static_assert(G::NB == 2 && G::HS == 2 && G::PW == 2 && G::NS % 2 == 0, "16 tokens, whole blocks");
    asm volatile("{\n\t.reg .b32 r<16>, u<16>, a;\n\t.reg .f32 dw;\n\t.reg .b64 t, x0, x1, s0, s1, t0, t1;\n\t.reg .pred p, q, lead;\n\tsetp.eq.u32 lead, %24, 0;\nLOOP_%=:\n\t"
                 PF_STEP("0", "64", "128", "192", "0", "16", "0") PF_STEP("256", "320", "384", "448", "8", "24", "1")
                 "setp.eq.u32 p, %18, %26;\n\t@p mov.u32 %18, 0;\n\txor.b32 %19, %19, 1;\n\tsub.u32 %20, %20, 1;\n\tsetp.ne.u32 p, %20, 0;\n\t@p bra LOOP_%=;\n\t}"
                 : "+l"(acc[0][0]), "+l"(acc[0][1]), "+l"(acc[0][2]), "+l"(acc[0][3]), "+l"(acc[0][4]), "+l"(acc[0][5]), "+l"(acc[0][6]), "+l"(acc[0][7]),
                   "+l"(acc[1][0]), "+l"(acc[1][1]), "+l"(acc[1][2]), "+l"(acc[1][3]), "+l"(acc[1][4]), "+l"(acc[1][5]), "+l"(acc[1][6]), "+l"(acc[1][7]),
                   "+r"(tbase), "+l"(limit_ns), "+r"(stage), "+r"(par), "+r"(turns)
                 : "r"(dw_addr), "r"(dx_addr), "r"(d_bars), "r"(lane), "n"(G::STAGE), "n"(G::NS * G::STAGE), "n"(G::WB), "n"(G::YB) : "memory");
}
#undef PF_FMA
#undef PF_FOLD
#undef PF_FOLD_FIRST
#undef PF_FOLD_SECOND
#undef PF_READ
#undef PF_READ_WAIT
#undef PF_SCALES
#undef PF_PRODUCTS
#undef PF_D_FULL
#undef PF_D_FREE
#undef PF_STEP

// SHARE: the last tiles are cut among the CTAs or clusters (PfItem in spyb_tc.cuh)
template <int TT, int S, bool MANY, bool SHARE, bool LATE>
__global__ void __launch_bounds__(PF_GEMM_THREADS, 1) prefill_gemm_kernel(PrefillGemm g) {
    using G = PfGeom<TT, S, MANY>;
    constexpr int NB = G::NB, NS = G::NS, PW = G::PW, PC = G::PC, YB = G::YB, HS = G::HS, WB = G::WB;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem), bars = sbase + G::BARS;
    // a stage: [NB blocks of weights: first half, 128 scales, second half (S = 2: the CTA's half and the scales)][NB compact activation blocks][8192 bytes of B operands]
    auto raw_full = [&](int s) { return bars + 8u * s; };                       // the step's weights and activations have landed
    auto ops_full = [&](int s) { return bars + 8u * (NS + s); };                // its B operands are written and fenced
    auto st_free  = [&](int s) { return bars + 8u * (2 * NS + s); };            // the stage may be refilled: its step's D buffer and scales have been read (arrival by the MMA warp, which waits for that anyway)
    auto d_full   = [&](int i) { return bars + 8u * (3 * NS + i); };            // the MMAs into buffer i have completed
    auto d_free   = [&](int i) { return bars + 8u * (3 * NS + 2 + i); };        // buffer i has been read (one arrival per epilogue warp)
    auto x_full   = [&](int w) { return bars + 8u * (3 * NS + 4 + w); };        // (S = 2) epilogue warp w of the other CTA has left its accumulators here
    auto x_free   = [&](int w) { return bars + 8u * (3 * NS + 4 + PF_GEMM_EPI_WARPS + w); };   // ... and here: the other CTA has read them
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + G::BARS + 8 * G::N_BAR);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nb = g.nb, n_step = (nb + NB - 1) / NB;
    const int n_tok = (g.T + TT - 1) / TT;
    const int n_tile = n_tok * (int)((g.n_rows + PF_M - 1) / PF_M);
    const int rank = S == 2 ? (int)(blockIdx.x & 1) : 0;   // (the CTAs of a cluster walk the same tiles)
    const uint64_t limit = g.wait_limit_ns;

    // The barriers, the zeroed B operands, the tensor memory and the first weights need nothing of the previous kernel; every role waits
    // for it before it touches activations or results.
    pdl_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) { mbar_init(raw_full(s), 1); mbar_init(ops_full(s), 1); mbar_init(st_free(s), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(d_full(i), 1); mbar_init(d_free(i), PF_GEMM_EPI_WARPS); }
        if (S == 2) {
            for (int w = 0; w < PF_GEMM_EPI_WARPS; ++w) { mbar_init(x_full(w), 1); mbar_init(x_free(w), 1); }
        }
        mbar_init_fence();
    }
    // the B operands are zero except where the expansion writes, and it writes the same places in every step
    for (int i = tid; i < NS * 512; i += PF_GEMM_THREADS) { sts128(sbase + (uint32_t)(i >> 9) * G::STAGE + G::RAW + (uint32_t)(i & 511) * 16u, make_uint4(0u, 0u, 0u, 0u)); }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (S == 2) { cluster_sync(); }   // (the other CTA's barriers are there)
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // How the expanding and multiplying warps walk: items and their steps, or (COUNTED) one count over all of them; and who releases the stage before a step's: the
    // thread that issues its MMAs, or (EARLY_FREE) lane 0 beforehand. Measured over 8 to 30 sizes a form, against one count throughout and lane 0 for two CTAs only: whole
    // tiles of 16 tokens by one CTA -3 to -4 % of the time (lane 0: -0.5 to -1.5), their shared ones of up to 64 tokens -2 %, above +0.6 %; 8 tokens by one CTA -1.3 to
    // -1.9 % (the issuing thread: -0.6), by two -0.3 to -0.5; 16 by two +0.7. Without the blocks past a row's end, tiles of 16 tokens +0.7 to +1.3 %, of 8 -0.5.
    constexpr bool COUNTED = TT == 16 && (S == 2 || (SHARE && MANY)), EARLY_FREE = TT == 8 || S == 2;
    const int walker = (int)blockIdx.x / S;
    [[maybe_unused]] const int total_steps = SHARE ? g.share.rounds * n_step + g.share.len + ((int)gridDim.x / S - 1 - walker < g.share.rem ? 1 : 0) : (g.share.rounds + (walker < g.share.rem ? 1 : 0)) * n_step;
    auto first_item = [&]() -> PfItem {
        if constexpr (SHARE) { return pf_share_item(g.share, n_tile, n_step, (int)blockIdx.x / S, (int)gridDim.x / S, 0); }
        return {(int)blockIdx.x / S, 0, n_step, 0};
    };
    auto next_item = [&](PfItem &it) {
        if constexpr (SHARE) { it = pf_share_item(g.share, n_tile, n_step, (int)blockIdx.x / S, (int)gridDim.x / S, it.q + 1); }
        else { it.tile += gridDim.x / S; }
    };
    // calls step(i, count) for the walker's steps, i the step of its tile (COUNTED: of none), until one returns false
    auto each_step = [&](auto step) {
        if constexpr (COUNTED) { for (int k = 0; k < total_steps; ++k) { if (!step(0, k)) { return; } } }
        else {
            int k = 0;
            for (PfItem it = first_item(); it.tile < n_tile; next_item(it)) {
                for (int i = it.from; i < it.to; ++i, ++k) { if (!step(i, k)) { return; } }
            }
        }
    };

    // CTAs that run together take neighbouring token tiles of the same rows: a weight tile crosses HBM once
    if (warp >= PF_GEMM_EPI_WARPS) {
        uint64_t left_ns = limit;   // (zero once a wait has run out)
        if (warp == PF_GEMM_EPI_WARPS) {
            // ---- copies
            int st = 0, k = 0, issued = 0;
            uint32_t par = 1;
            bool ok = true;
            // the weights of the first tile's first steps, then (the previous kernel is done) their activations with all that follows
            const PfItem first = first_item();
            const int early = first.tile < n_tile ? min(NS, first.to - first.from) : 0;
            // n blocks of weights at `w` into stage st
            auto copy_weights = [&](int st, const uint8_t *w, int n) {
                const uint32_t dst = sbase + (uint32_t)st * G::STAGE;
                if (S == 1 && !MANY) { bulk_copy_g2s(dst, w, (uint32_t)(n * WB), raw_full(st)); }
                else if (S == 1) {
#pragma unroll
                    for (int j = 0; j < 2 * NB; ++j) {
                        if (j < 2 * n) { bulk_copy_g2s(dst + j * (WB / 2), w + (int64_t)j * (WB / 2), WB / 2, raw_full(st)); }
                    }
                }
                else {
#pragma unroll
                    for (int j = 0; j < NB; ++j) {
                        if (j < n) { bulk_copy_g2s(dst + j * WB, w + (int64_t)j * PF_WTILE_F16 + rank * PF_HALF, WB, raw_full(st)); }
                    }
                }
            };
            if (elect_one()) {
                for (int i = 0; i < early; ++i) {
                    if (i == g.selftest_skip_step) { continue; }
                    const int n = min(NB, nb - (first.from + i) * NB);
                    mbar_expect_tx(raw_full(i), (uint32_t)(n * (WB + YB)));
                    copy_weights(i, g.w + ((int64_t)(first.tile / n_tok) * nb + (first.from + i) * NB) * PF_WTILE_F16, n);
                }
            }
            __syncwarp();
            pdl_wait();
            for (PfItem it = first; it.tile < n_tile && ok; next_item(it)) {
                const uint8_t *wsrc = g.w + ((int64_t)(it.tile / n_tok) * nb + it.from * NB) * PF_WTILE_F16;
                const uint8_t *ysrc = g.yq + ((int64_t)(it.tile % n_tok) * nb + it.from * NB) * YB;
                for (int i = it.from; i < it.to; ++i, ++k) {
                    if (k >= NS) {
                        ok = __all_sync(0xffffffffu, mbar_wait_relaxed(st_free(st), par, limit));
                        if (!ok) { break; }
                    }
                    const int n = min(NB, nb - i * NB);
                    if (k != g.selftest_skip_step && elect_one()) {   // (failure-path check: that step never arrives)
                        const uint32_t dst = sbase + (uint32_t)st * G::STAGE;
                        if (k >= early) {
                            mbar_expect_tx(raw_full(st), (uint32_t)(n * (WB + YB)));
                            copy_weights(st, wsrc, n);
                        }
                        bulk_copy_g2s(dst + NB * WB, ysrc, (uint32_t)(n * YB), raw_full(st));
                    }
                    __syncwarp();
                    issued = k + 1;
                    wsrc += NB * PF_WTILE_F16; ysrc += NB * YB;
                    if (++st == NS) { st = 0; par ^= 1u; }
                }
            }
            if (!ok && lane == 0) { pf_report(g.error_flag, 4); }
            // no copy of this CTA is in flight when it leaves
            for (int j = max(0, issued - NS); j < issued; ++j) {
                if (j != g.selftest_skip_step && !mbar_wait_relaxed(raw_full(j % NS), (uint32_t)(j / NS) & 1u, limit)) { if (lane == 0) { pf_report(g.error_flag, 4); } break; }
            }
        } else if (warp == PF_GEMM_EPI_WARPS + 1) {
            // ---- expansion. The four values of accumulator n of token t in half h of a block go to row 8 (t / 2) + 2 n + t % 2 of the half's
            // B operand (4 TT rows x 16), at their place 4 n; the rest of B stays zero. A lane takes 16 bytes (accumulators 2 np and
            // 2 np + 1) at a time, four times in a step.
            int st = 0;
            uint32_t par = 0;
            constexpr int TK = 8 * S;   // token t0 + TK k of the step (block (t0 + TK k) / TT), of the one half that a CTA takes or of both
            const int h = S == 2 ? 0 : (lane >> 1) & 1, np = lane & 1, t0 = S == 2 ? lane >> 1 : lane >> 2;
            const uint32_t dst_lane = (uint32_t)((S == 2 ? (t0 / TT) * 128 * TT : 0) + h * 128 * TT + np * (64 * TT + 64) + ((S == 2 ? t0 % TT : t0) >> 1) * 128 + (t0 & 1) * 16);
            const uint32_t src_lane = (uint32_t)(S == 2 ? (t0 / TT) * YB + (t0 % TT) * 64 + rank * 32 + np * 16 : lane * 16);
            each_step([&](int, int) {
                mbar_wait_lean(raw_full(st), par, left_ns);
                if (left_ns == 0) { return false; }
                const uint32_t base = sbase + (uint32_t)st * G::STAGE, src = base + NB * WB + src_lane, dst = base + G::RAW + dst_lane;
                uint4 v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) { v[k] = lds128(src + (uint32_t)((k * TK / TT) * YB + (k * TK % TT) * 64)); }   // all loads in flight before the first store
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t d = dst + (uint32_t)((k * TK / TT) * HS * 128 * TT + (k * TK % TT) * 64);
                    sts64(d, v[k].x, v[k].y);
                    sts64(d + 40u, v[k].z, v[k].w);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) { mbar_arrive(ops_full(st)); }
                if (++st == NS) { st = 0; par ^= 1u; }
                return true;
            });
            if (left_ns == 0 && lane == 0) { pf_report(g.error_flag, 4); }
        } else {
            // ---- MMAs: per block and half of 16 elements one 128 x 4 TT x 16 product; warp m takes the steps of D buffer m (issuing a step's
            // MMAs and their commit takes one warp up to 400 cycles)
            const int m = warp - (PF_GEMM_EPI_WARPS + 2);
            const uint32_t d0 = tmem + (uint32_t)m * 256u;
            int st = 0, mine = 0;
            uint32_t par = 0;
            each_step([&](int i, int k) {
                if ((k & 1) == m) {
                    mbar_wait_lean(ops_full(st), par, left_ns);
                    mbar_wait_lean(d_free(m), (uint32_t)mine & 1u, left_ns);
                    if (left_ns == 0) { return false; }
                    if (EARLY_FREE && mine > 0 && lane == 0) { mbar_arrive(st_free(st >= 2 ? st - 2 : st + NS - 2)); }   // (the step before on this buffer has been read)
                    tc_fence_after();
                    const uint32_t base = sbase + (uint32_t)st * G::STAGE;
                    const uint64_t a0 = operand_desc(base + (uint32_t)rank * 512u, 2048u, 128u), b0 = operand_desc(base + G::RAW, 64u * TT, 128u);
                    [[maybe_unused]] const int n = min(NB, nb - i * NB);
                    if (elect_one()) {
                        if (!EARLY_FREE && mine > 0) { mbar_arrive(st_free(st >= 2 ? st - 2 : st + NS - 2)); }   // (the step before on this buffer has been read)
#pragma unroll
                        for (int j = 0; j < NB; ++j) {
                            if (TT == 8 && j >= n) { continue; }   // (TT = 16: blocks past the end of a row are multiplied too, whatever lies there: nobody folds them)
#pragma unroll
                            for (int h = 0; h < HS; ++h) {
                                mma_f16_ss(d0 + (uint32_t)((j * HS + h) * 4 * TT), a0 + (uint64_t)((j * WB + h * (PF_HALF + 512)) >> 4), b0 + (uint64_t)(((j * HS + h) * 128 * TT) >> 4),
                                           idesc_f16(4 * TT), 0u);
                            }
                        }
                        mma_commit(d_full(m));
                    }
                    __syncwarp();
                    ++mine;
                }
                if (++st == NS) { st = 0; par ^= 1u; }
                return true;
            });
            if (left_ns == 0 && lane == 0) { pf_report(g.error_flag, 5); }
            // every MMA has completed (it reads shared memory and writes tensor memory) before the CTA leaves
            if (mine > 0 && !mbar_wait_relaxed(d_full(m), (uint32_t)(mine - 1) & 1u, limit)) { if (lane == 0) { pf_report(g.error_flag, 5); } }
        }
    } else {
        pdl_wait();
        // ---- epilogue: tokens part * TT / 4 .. of the tile as PW packed pairs (tokens 2 u, 2 u + 1), eight accumulators each. D's columns
        // of block j and half h: 8 TT j + 4 TT h + 8 (t / 2) + 2 n + t % 2, i.e. a pair's accumulator n is a neighbouring pair of columns.
        const int quad = warp & 3, part = warp >> 2;
        const int row = 32 * quad + lane;
        const uint32_t tbase = tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(part * TT);
        const uint32_t dw_addr = sbase + (rank == 0 ? (uint32_t)PF_HALF : 0u) + 4u * (uint32_t)row, dx_addr = sbase + NB * WB + TT * 64 + (uint32_t)(part * TT);
        uint64_t acc[PW][4 * HS];
#pragma unroll
        for (int u = 0; u < PW; ++u) {
#pragma unroll
            for (int n = 0; n < 4 * HS; ++n) { acc[u][n] = 0ull; }
        }
        if (lane == 0) { mbar_arrive(d_free(0)); mbar_arrive(d_free(1)); }
        uint32_t stage = 0, par = 0;   // (the ring has an even number of stages: a step's stage and its D buffer are even or odd together)
        uint64_t left_ns = limit;      // (zero once a wait has run out)
        // one step, its D buffer a constant of the unrolled code; n of its NB blocks lie inside the row
        auto step = [&](auto buf_c, int n) {
            constexpr int buf = decltype(buf_c)::value;
            mbar_wait_lean(d_full(buf), par, left_ns);
            tc_fence_after();
            uint64_t sc[PC];
#pragma unroll
            for (int c = 0; c < G::NC; ++c) {   // chunk c: half c % HS of PC pairs of block c / HS / (PW / PC)
                const int cu = (c / HS) % (PW / PC), j = (c / HS) / (PW / PC);
                const uint32_t col = (uint32_t)(buf * 256 + (j * HS + c % HS) * 4 * TT + cu * 8 * PC);
                uint32_t r[8 * PC];
                if (PC == 2) { tmem_ld16(tbase + col, r); } else { tmem_ld8(tbase + col, r); }
                if (c % HS == 0) {
                    const float dw = lds32f(dw_addr + stage + (uint32_t)(j * WB));
                    const uint64_t dw2 = f2_pack(dw, dw);
                    const uint32_t xa = dx_addr + stage + (uint32_t)(j * YB + cu * 8 * PC);
                    if (PC == 2) { uint64_t x0, x1; lds128_2x64(xa, x0, x1); sc[0] = f2_mul(dw2, x0); sc[PC - 1] = f2_mul(dw2, x1); }
                    else { sc[0] = f2_mul(dw2, lds64u(xa)); }
                }
                tmem_ld_wait();
                if (c == G::NC - 1) {           // the whole buffer is in registers and the step's scales have been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) { mbar_arrive(d_free(buf)); }
                }
                if (NB == 1 || j < n) {         // (blocks past the end of the row in a tile's last step are not folded)
#pragma unroll
                    for (int p = 0; p < PC; ++p) {
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            uint64_t &a = acc[PC * cu + p][4 * (c % HS) + m];
                            a = f2_fma(sc[p], f2_pack_bits(r[8 * p + 2 * m], r[8 * p + 2 * m + 1]), a);
                        }
                    }
                }
            }
            stage += G::STAGE;
            if (buf) { par ^= 1u; if (stage == NS * G::STAGE) { stage = 0; } }
        };
        using B0 = std::integral_constant<int, 0>;
        using B1 = std::integral_constant<int, 1>;
        const int rest = nb % NB;
        uint32_t x_par = 0;      // phase of the hand-over between the CTAs of a cluster
        bool odd = false;        // an item with an odd number of steps leaves the next one starting on buffer 1
        [[maybe_unused]] bool joined = false;   // (S = 2) a tile's halves have been joined already
        for (PfItem it = first_item(); it.tile < n_tile; next_item(it)) {
            const int n_full = SHARE ? min(it.to, nb / NB) - it.from : nb / NB;
            const int tile = it.tile;
            if constexpr (SHARE) if (it.from > 0) {   // another walker's accumulators
                const int64_t at = (int64_t)((int)blockIdx.x - S) * PF_GEMM_EPI_WARPS + warp;
                handoff_wait(g.handoff_flags + at, left_ns);
#pragma unroll
                for (int n = 0; n < 4 * HS * PW; ++n) { acc[n / (4 * HS)][n % (4 * HS)] = __ldcg(reinterpret_cast<const unsigned long long *>(g.handoff) + (at * 16 + n) * 32 + lane); }
                __syncwarp();
                if (lane == 0) { g.handoff_flags[at] = 0u; }
            }
            int i = 0;
            if (odd && n_full > 0) { step(B1{}, NB); i = 1; }
            if constexpr (TT == 16 && S == 1) {
                const int turns = (n_full - i) >> 1;
                if (turns > 0) { pf_fold_steps<G>(acc, turns, tbase, dw_addr, dx_addr, d_full(0), lane, stage, par, left_ns); }
                i += 2 * turns;
            } else {
#pragma unroll 1
                for (; i + 2 <= n_full; i += 2) { step(B0{}, NB); step(B1{}, NB); }
            }
            bool second = odd && n_full == 0;
            if (i < n_full) { step(B0{}, NB); second = true; }
            if (rest != 0 && (!SHARE || it.to == n_step)) {
                if (second) { step(B1{}, rest); } else { step(B0{}, rest); }
                second = !second;
            }
            odd = second;
            if constexpr (SHARE) if (it.to < n_step) {   // another walker goes on with these accumulators
                const int64_t at = (int64_t)blockIdx.x * PF_GEMM_EPI_WARPS + warp;
#pragma unroll
                for (int n = 0; n < 4 * HS * PW; ++n) {
                    uint64_t &a = acc[n / (4 * HS)][n % (4 * HS)];
                    __stcg(reinterpret_cast<unsigned long long *>(g.handoff) + (at * 16 + n) * 32 + lane, (unsigned long long)a);
                    a = 0ull;
                }
                if constexpr (LATE) { const uint64_t t0 = global_timer_ns(); while (global_timer_ns() - t0 < 3 * limit) {} }   // (failure-path check)
                __syncwarp();
                if (lane == 0) { handoff_publish(g.handoff_flags + at); }
                continue;
            }
            // hsum_float_8 (vec_util.h:74-81): accumulator n of a half is CPU accumulator 4 + n / n (Q4_0: low / high nibbles) or n / 4 + n
            // (Q8_0); either way the tree is (c0 + c4) + (c2 + c6) and (c1 + c5) + (c3 + c7)
            const int64_t orow = (int64_t)(tile / n_tok) * PF_M + row;
            const int     tok0 = (tile % n_tok) * TT + part * (TT / 4);
            if constexpr (S == 2) {   // the second half's accumulators are those of the same thread of the cluster's other CTA
                const uint32_t xch = sbase + (uint32_t)(NS * G::STAGE) + 8u * (uint32_t)tid;
                if (rank == 1) {
                    if (SHARE ? joined : tile != blockIdx.x / S) { cluster_wait(x_free(warp), x_par ^ 1u, left_ns); }   // (the tile before has been read)
                    joined = true;
                    const uint32_t to = cluster_map(xch, 0);
#pragma unroll
                    for (int i = 0; i < 4 * PW; ++i) { cluster_store64(to + (uint32_t)(i * PF_GEMM_EPI_WARPS * 32 * 8), acc[i >> 2][i & 3]); }
                    __syncwarp();
                    if (lane == 0) { cluster_arrive(cluster_map(x_full(warp), 0)); }
                } else {
                    cluster_wait(x_full(warp), x_par, left_ns);
#pragma unroll
                    for (int i = 0; i < 4 * PW; ++i) { acc[i >> 2][i & 3] = f2_add(acc[i >> 2][i & 3], lds64u(xch + (uint32_t)(i * PF_GEMM_EPI_WARPS * 32 * 8))); }
                    __syncwarp();
                    if (lane == 0) { cluster_arrive(cluster_map(x_free(warp), 1)); }
                }
                x_par ^= 1u;
            }
#pragma unroll
            for (int u = 0; u < PW; ++u) {
                if (S == 1 || rank == 0) {
                    if constexpr (S == 1) {
#pragma unroll
                        for (int m = 0; m < 4; ++m) { acc[u][m] = f2_add(acc[u][m], acc[u][4 + m]); }
                    }
                    float v[2];
                    f2_unpack(f2_add(f2_add(acc[u][0], acc[u][2]), f2_add(acc[u][1], acc[u][3])), v[0], v[1]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int token = tok0 + 2 * u + e;
                        if (token < g.T && orow < g.n_rows) {   // (the last row tile may be partly padding)
                            const int64_t o = (int64_t)token * g.out_stride + orow;
                            g.out[o] = g.resid != nullptr ? __fadd_rn(v[e], g.resid[o]) : v[e];
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < 4 * HS; ++m) { acc[u][m] = 0ull; }
            }
        }
        if (left_ns == 0 && lane == 0) { pf_report(g.error_flag, 6); }
    }
    tc_fence_before();
    __syncthreads();
    if (S == 2) { cluster_sync(); }   // (neither CTA's shared memory goes while the other may still reach into it)
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------
// activations of T tokens -> compact Q8_0 blocks grouped by (tile of tile_tok tokens, block). One CTA per token; RMSNorm and the
// quantizer as in the mat-vec prologue (NormRMS, backend/host/operator/non-linear.cpp:194-223: groups of four squares formed in
// parallel, the running sum on four warps; Quantizator<FP32,Q8_0>, simd/vec_convert.h:178-261). Bound: that sum's chain; the
// norm's weights are read before the wait for the previous kernel. PG groups of eight values a thread: one fits most models, and two CTAs an
// SM. us with the norm, one thread's sum / this: 8 tokens x 5120 9.8 / 7.4, 32 x 5120 9.6 / 7.0, 448 x 4096 26.5 / 10.7.
// KQ false (Q4_0 / Q8_0 weights): [token][32 values as f16], the scales. KQ true: the f16 B operand itself (16 bytes of eight values of a token at
// (value / 8) * 16 TOKT + 16 token), the scales, the blocks' integer sums as floats.
// SILU: a token's row is [K up | K gate] as the stacked GEMM leaves it, and what is quantized is up * silu(gate) (model/src/llm/plugin/ffn.cpp:28-35),
// which goes to act only where somebody wants it. (As two kernels, 512 x 11008: 27 + 14 us, 90 MB; this 22-27 us, 46 MB.)
template <bool NORM, bool KQ, int PG, bool SILU>
__global__ void __launch_bounds__(PF_QUANT_THREADS, PG <= 2 ? 2 : 1) prefill_quant_kernel(const float *x, int64_t x_stride, int K, const float *norm_w, float eps, uint8_t *yq,
                                                                         int TOKT, int part_len, int64_t part_stride, uint8_t *tap, const float *silu_table, float *act) {
    static_assert(!(NORM && SILU), "");
    const int SCALES = TOKT * 64;                         // offset of the scales inside a block's record
    const int YQB = SCALES + TOKT * (KQ ? 8 : 4);
    extern __shared__ __align__(16) float v3[];
    __shared__ float scale_s;
    const int tid = threadIdx.x, token = blockIdx.x;
    const int n4 = K >> 2, n8 = K >> 3, nb = K >> 5;
    const int npass = (n8 + PF_QUANT_THREADS - 1) / PF_QUANT_THREADS;
    pdl_launch_dependents();
    float wv[NORM ? PG : 1][8];
    if (NORM) {   // the norm's weights are constants: they are there before the previous kernel is done
#pragma unroll
        for (int k = 0; k < PG; ++k) {
            const int gi = tid + k * PF_QUANT_THREADS;
            if (k < npass && gi < n8) { load8_cg(norm_w + 8 * gi, wv[NORM ? k : 0]); }
            else {
#pragma unroll
                for (int i = 0; i < 8; ++i) { wv[NORM ? k : 0][i] = 0.f; }
            }
        }
    }
    pdl_wait();
    // a row may lie in parts (the slices the ranks of a tensor-parallel group gathered): elements [i part_len, (i + 1) part_len)
    // of token t at x + i part_stride + t x_stride; one part = the plain row (parts are multiples of four values)
    const float *xrow = x + (int64_t)token * x_stride;
    float xv[PG][8];
#pragma unroll
    for (int k = 0; k < PG; ++k) {
        const int gi = tid + k * PF_QUANT_THREADS;
        if (k < npass && gi < n8) {
            if (SILU) {
                float gate[8];
                load8_cg(xrow + 8 * gi, xv[k]);
                load8_cg(xrow + K + 8 * gi, gate);
#pragma unroll
                for (int i = 0; i < 8; ++i) { xv[k][i] = __fmul_rn(xv[k][i], silu_table[f2h(gate[i])]); }
                if (act != nullptr) {
                    float4 *to = reinterpret_cast<float4 *>(act + (int64_t)token * K + 8 * gi);
                    to[0] = make_float4(xv[k][0], xv[k][1], xv[k][2], xv[k][3]); to[1] = make_float4(xv[k][4], xv[k][5], xv[k][6], xv[k][7]);
                }
            }
            else if (part_len == K) { load8_cg(xrow + 8 * gi, xv[k]); }
            else {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int e = 8 * gi + 4 * h, part = e / part_len;
                    const float4 v = *reinterpret_cast<const float4 *>(xrow + (int64_t)part * part_stride + (e - part * part_len));
                    xv[k][4 * h] = v.x; xv[k][4 * h + 1] = v.y; xv[k][4 * h + 2] = v.z; xv[k][4 * h + 3] = v.w;
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) { xv[k][i] = 0.f; }
        }
    }
    if (NORM) {
#pragma unroll
        for (int k = 0; k < PG; ++k) {
            const int gi = tid + k * PF_QUANT_THREADS;
            if (k < npass && gi < n8) { reinterpret_cast<float2 *>(v3)[gi] = squares8(xv[k]); }
        }
        __syncthreads();
        __shared__ __align__(16) float rs[rs_scratch_words(4)];
        float sum = 0.f;
        if (tid < RS_THREADS) { sum = running_sum_wide(smem_u32(v3), n4, smem_u32(rs), rs_scratch_words(4), tid, 1); }
        if (tid == 0) {
            scale_s = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)K), eps)));
        }
        __syncthreads();
        const float scale = scale_s;
#pragma unroll
        for (int k = 0; k < PG; ++k) {
#pragma unroll
            for (int i = 0; i < 8; ++i) { xv[k][i] = __fmul_rn(__fmul_rn(xv[k][i], scale), wv[NORM ? k : 0][i]); }
        }
    }
    uint8_t *tile = yq + ((int64_t)(token / TOKT) * nb) * YQB;
    const int tt = token % TOKT;
    uint2 qv[PG];
    int kd;
    const float d = quantize_q8_groups<PG>(xv, npass, qv, kd);   // (npass is uniform over the CTA: the quantizer's shuffles see full warps)
    if (kd >= 0 && tid + kd * PF_QUANT_THREADS < n8) {
        const int b = (tid + kd * PF_QUANT_THREADS) >> 2;
        const uint16_t dh = f2h(d);
        reinterpret_cast<float *>(tile + (int64_t)b * YQB + SCALES)[tt] = h2f(dh);
        if (tap != nullptr && token == 0) { *reinterpret_cast<uint16_t *>(tap + (int64_t)b * 34) = dh; }
    }
#pragma unroll
    for (int k = 0; k < PG; ++k) {
        if (k < npass) {
            const int gi = tid + k * PF_QUANT_THREADS;
            const uint2 q = qv[k];
            int sum = 0;
            if (KQ) {   // the block's sum over its four lanes
                sum = q8_sum8(q);
                sum += __shfl_xor_sync(0xffffffffu, sum, 1); sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            }
            if (gi < n8) {
                const int b = gi >> 2, w = gi & 3;
                uint8_t *blk = tile + (int64_t)b * YQB;
                // byte + 128 as the low byte of the f16 1024 + (byte + 128), less 1152: the value as f16
                auto halves = [](uint32_t bytes, uint32_t sel) {
                    uint32_t h = __byte_perm(bytes ^ 0x80808080u, 0x64646464u, sel);
                    *reinterpret_cast<__half2 *>(&h) = __hsub2(*reinterpret_cast<__half2 *>(&h), __float2half2_rn(1152.f));
                    return h;
                };
                const uint4 v = make_uint4(halves(q.x, 0x4140), halves(q.x, 0x4342), halves(q.y, 0x4140), halves(q.y, 0x4342));
                if (tap != nullptr && token == 0) {   // reference-layout blocks of token 0 (34-byte records: only 2-byte alignment holds)
                    uint16_t *o = reinterpret_cast<uint16_t *>(tap + (int64_t)b * 34) + 1 + 4 * w;
                    o[0] = (uint16_t)q.x; o[1] = (uint16_t)(q.x >> 16); o[2] = (uint16_t)q.y; o[3] = (uint16_t)(q.y >> 16);
                }
                *reinterpret_cast<uint4 *>(KQ ? blk + w * 16 * TOKT + tt * 16 : blk + tt * 64 + w * 16) = v;
                if (KQ && w == 0) { reinterpret_cast<float *>(blk + SCALES + TOKT * 4)[tt] = (float)sum; }
            }
        }
    }
}

// upload-time re-layout: raw 18-byte / 34-byte blocks of rows [0, n_rows) -> tiles of 128 rows x 1 block: the first half of the block's
// values, the 128 scales as f32, the second half. A half is an f16 A operand (core matrices of 8 rows x 16 bytes: element k of row r at
// (k / 8) * 2048 + (r / 8) * 128 + (r % 8) * 16 + 2 (k % 8)); Q4_0: element k of the first half is the low nibble of byte k minus 8, of
// the second half the high one. A warp takes 8 rows x 4 neighbouring blocks: its stores are runs of 128 bytes, its loads runs of 72 or 136.
template <int WT>
__global__ void prefill_retile_kernel(const uint8_t *raw, int64_t row_stride, int64_t n_rows, int nb, uint8_t *base, int64_t dst_row0) {
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int     lane = threadIdx.x & 31, bq = (nb + 3) >> 2;
    const int64_t lrow = w / bq * 8 + (lane & 7);
    const int     b = (int)(w % bq) * 4 + (lane >> 3);
    if (lrow >= n_rows || b >= nb) { return; }
    uint16_t src[WT == 2 ? 9 : 17];   // (blocks are 2-byte aligned)
    const uint16_t *raw16 = reinterpret_cast<const uint16_t *>(raw + lrow * row_stride + (int64_t)b * (WT == 2 ? 18 : 34));
#pragma unroll
    for (int i = 0; i < (WT == 2 ? 9 : 17); ++i) { src[i] = raw16[i]; }
    const int64_t row = dst_row0 + lrow;
    const int     r = (int)(row % PF_M);
    uint8_t *tile = base + ((row / PF_M) * nb + b) * (int64_t)PF_WTILE_F16;
    reinterpret_cast<float *>(tile + PF_HALF)[r] = h2f(src[0]);
    auto byte_of = [&](int i) { return (i & 1) ? src[1 + (i >> 1)] >> 8 : src[1 + (i >> 1)] & 0xff; };
    auto value = [&](int k) {
        if (WT == 2) { const int byte = byte_of(k & 15); return (k < 16 ? (byte & 15) : (byte >> 4)) - 8; }
        return (int)(int8_t)byte_of(k);
    };
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[e] = (uint32_t)__half_as_ushort(__int2half_rn(value(8 * c + 2 * e))) | ((uint32_t)__half_as_ushort(__int2half_rn(value(8 * c + 2 * e + 1))) << 16);
        }
        *reinterpret_cast<uint4 *>(tile + c * 2048 + (c >> 1) * 512 + (r >> 3) * 128 + (r & 7) * 16) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// RoPE(Q, K) + fp16 stores of Q / K / V after the QKV GEMM (the arithmetic of the mat-vec epilogue EPI_QKV_ROPE:
// backend/host/operator/non-linear.cpp:270-371, view.cpp:163-191). The first qk_blocks blocks rotate, a thread per pair of neighbouring elements of a
// token; the others turn 64 elements x 32 tokens of V over in shared memory, because the cache holds a row per element: a warp then writes
// 32 neighbouring positions of a row, 64 bytes, where a thread per element wrote two bytes into a line of its own (512 tokens x 12288: 31.5 us,
// 16-17 now; 38 MB). A batch in lockstep (seq_stride > 0: token t is sequence t, with its own cache) has nothing to turn over: a thread per element.
constexpr int PF_POST_THREADS = 256, PF_POST_E = 64, PF_POST_T = 32;
__global__ void __launch_bounds__(PF_POST_THREADS) prefill_qkv_post_kernel(const float *qkv, int T, int dl, int hd, const int *pos_base, const float2 *rope, __half *q_out, __half *k_cache,
                                        __half *v_cache, int n_ctx, int64_t seq_stride, int qk_blocks) {
    __shared__ __half vt[PF_POST_T][PF_POST_E + 2];
    pdl_launch_dependents();
    pdl_wait();
    if ((int)blockIdx.x < qk_blocks) {
        const int64_t i = (int64_t)blockIdx.x * PF_POST_THREADS + threadIdx.x;
        if (i >= (int64_t)dl * T) { return; }
        const int t = (int)(i / dl), col = 2 * (int)(i - (int64_t)t * dl);
        const bool is_k = col >= dl;
        const int e = is_k ? col - dl : col, pos = *pos_base + (seq_stride ? 0 : t);
        const float2 x = *reinterpret_cast<const float2 *>(qkv + (int64_t)t * 3 * dl + col), cs = rope[(int64_t)pos * (hd >> 1) + ((e % hd) >> 1)];
        const float a0 = __fsub_rn(__fmul_rn(x.x, cs.x), __fmul_rn(x.y, cs.y));
        const float a1 = __fadd_rn(__fmul_rn(x.x, cs.y), __fmul_rn(x.y, cs.x));
        __half *dst = is_k ? k_cache + (seq_stride ? (int64_t)t * seq_stride : 0) + (int64_t)pos * dl + e : q_out + (int64_t)t * dl + e;
        *reinterpret_cast<__half2 *>(dst) = __halves2half2(__float2half_rn(a0), __float2half_rn(a1));
        return;
    }
    const int vb = (int)blockIdx.x - qk_blocks;
    if (seq_stride) {
        const int64_t i = (int64_t)vb * PF_POST_THREADS + threadIdx.x;
        if (i >= (int64_t)dl * T) { return; }
        const int t = (int)(i / dl), e = (int)(i - (int64_t)t * dl);
        v_cache[(int64_t)t * seq_stride + (int64_t)e * n_ctx + *pos_base] = __float2half_rn(qkv[(int64_t)t * 3 * dl + 2 * dl + e]);
        return;
    }
    const int e_tiles = (dl + PF_POST_E - 1) / PF_POST_E, e0 = vb % e_tiles * PF_POST_E, t0 = vb / e_tiles * PF_POST_T;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int t = w; t < PF_POST_T; t += PF_POST_THREADS / 32) {
        const int e = e0 + 2 * lane;   // (dl is even: heads are rotated in pairs)
        if (t0 + t < T && e < dl) {
            const float2 x = *reinterpret_cast<const float2 *>(qkv + (int64_t)(t0 + t) * 3 * dl + 2 * dl + e);
            *reinterpret_cast<__half2 *>(&vt[t][2 * lane]) = __halves2half2(__float2half_rn(x.x), __float2half_rn(x.y));
        }
    }
    __syncthreads();
    if (t0 + lane >= T) { return; }
    __half *row = v_cache + (int64_t)e0 * n_ctx + *pos_base + t0 + lane;
    for (int e = w; e < min(PF_POST_E, dl - e0); e += PF_POST_THREADS / 32) { row[(int64_t)e * n_ctx] = vt[lane][e]; }
}

// up * silu(gate) (model/src/llm/plugin/ffn.cpp:28-35) on the output [T][2 F] of the stacked up|gate GEMM
__global__ void prefill_silu_mul_kernel(const float *upgate, int T, int F, const float *silu_table, float *act) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (i >= (int64_t)T * F) { return; }
    const int t = (int)(i / F);
    const int64_t f = i - (int64_t)t * F;
    const float up = upgate[(int64_t)t * 2 * F + f], gate = upgate[(int64_t)t * 2 * F + F + f];
    act[i] = __fmul_rn(up, silu_table[f2h(gate)]);
}

template <int TT, int S, bool MANY = false, bool SHARE = false, bool LATE = false>
cudaError_t launch_gemm_t(const PrefillGemm &g, cudaStream_t stream, bool pdl) {
    const void *kernel = reinterpret_cast<const void *>(prefill_gemm_kernel<TT, S, MANY, SHARE, LATE>);
    const size_t smem = PfGeom<TT, S, MANY>::SMEM;
    cudaError_t err = allow_dynamic_smem(kernel, smem);
    if (err != cudaSuccess) { return err; }
    const int64_t tiles = (int64_t)((g.T + TT - 1) / TT) * ((g.n_rows + PF_M - 1) / PF_M), walkers = std::min<int64_t>(tiles, device_sms() / S);
    PrefillGemm h = g;
    h.share = {(int)(tiles / walkers), 0, (int)(tiles % walkers), 0};
    if (SHARE) { h.share = pf_share((int)tiles, (g.nb + PfGeom<TT, S, MANY>::NB - 1) / PfGeom<TT, S, MANY>::NB, (int)walkers); }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(S * walkers)); lc.blockDim = dim3(PF_GEMM_THREADS); lc.dynamicSmemBytes = smem; lc.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = S; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    lc.attrs = attr; lc.numAttrs = S > 1 ? 2 : 1;
    void *args[] = {&h};
    return cudaLaunchKernelExC(&lc, kernel, args);
}

}  // namespace

int device_sms() {
    static int sms[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { return 148; }
    if (sms[dev] == 0) {
        int n = 0;
        sms[dev] = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
    }
    return sms[dev];
}

// The form of the Q4_0 / Q8_0 kernel for a matrix and a number of tokens: tiles of 16 or of 8 tokens, by one CTA each or by a cluster of two, the last ones whole or
// shared; the one whose cost (pf_cost) is least. Fitted to 1068 sizes, fifteen matrices of models and 160 drawn ones from 1024 x 1536 to 32000 x 11264, with 5 to 512
// tokens, every form timed with the submits of one backend and with those of three in turn. At 636 other sizes a model's choice is 0.25 % behind the fastest on average,
// more than 3 % at 21 (28620 x 1728 x 8 tokens 10 %). An operator's, against a rule of whole tiles by rounds alone: one backend 5.9 % faster on average (more
// than 3 % slower at 2 of 587), three 3.6 % (at 24); with a model's rule 6.7 % and 1.7 % (at 76). us a submit from one backend / three, with the quantizer,
// 16 tokens a tile by one CTA, 8 by one, 16 by two, 8 by two: 4096 x 4096 x 8 tokens 24.0 / 9.9, 19.0 / 10.3, 19.0 / 14.2, 15.7 / 13.9; 4096 x 11008 x 16 57.4 /
// 20.3, 54.9 / 25.9, 39.3 / 19.7, 35.9 / 30.0; 22016 x 4096 x 448 628 / 617, 998 / 974, 820 / 809, 1199 / 1190. The first and third with shared tiles: 12288 x 4096
// x 32 whole 45.6 / 29.8, 46.2 / 39.3, shared 37.1 / 34.0, 47.6 / 44.3; 5120 x 13824 x 32 whole 70.9 / 40.4, 86.8 / 50.7, the third shared 57.8 / 54.2.
struct PfForm { int tok, split; PfCost cost; };
static PfForm best_form(int64_t n_rows, int nb, int T, int tok, int split, int how, bool beside, int sms, bool *share) {   // tok, split, how 0: any
    static constexpr PfForm FORMS[4] = {{16, 1, {4320, 790, 143.9, 27.1, 5490, 0.044, 1850}}, {8, 1, {2430, 0, 118.7, 100.1, 4060, -0.019, 870}},
                                        {16, 2, {6920, 1830, 87.9, 23.3, 4550, 0.079, 1420}}, {8, 2, {4890, 650, 63.3, 89.7, 6320, 0.004, 2300}}};
    static constexpr PfRule RULE = {0.83, 0.46, 2340};
    PfForm best = {};
    double best_ns = 0.0;
    for (const PfForm &f : FORMS) {
        if ((tok != 0 && tok != f.tok) || (split != 0 && split != f.split)) { continue; }
        const int64_t row_tiles = (n_rows + PF_M - 1) / PF_M;
        bool shared;
        const double ns = pf_cost(f.cost, RULE, row_tiles, row_tiles * ((T + f.tok - 1) / f.tok), std::max(1, sms / f.split), nb, sms, how, true, beside, &shared);
        if (best.tok == 0 || ns < best_ns) { best = f; best_ns = ns; *share = shared; }
    }
    return best;
}
void prefill_form(int64_t n_rows, int nb, int T, int sms, int *tile_tok, int *split) {
    bool share;
    const PfForm f = best_form(n_rows, nb, T, 0, 0, 0, true, sms, &share);
    *tile_tok = f.tok; *split = f.split;
}
void prefill_plan(int type, int64_t n_rows, int nb, int T, int sms, int *tile_tok, int *split, int *tiles) {
    bool share = false;
    if (type == 12 || type == 14) { *tile_tok = prefill_kq_tile_tokens(n_rows, nb, T, *tile_tok, *tiles, true, sms, &share); *split = 1; }
    else { const PfForm f = best_form(n_rows, nb, T, *tile_tok, *split, *tiles, true, sms, &share); *tile_tok = f.tok; *split = f.split; }
    *tiles = share ? 2 : 1;
}
// host-only check of the shared tiles: every step of every tile is some walker's exactly once, and a tile's first steps are the lower neighbour's of the
// walker that goes on with it, and done by the time it does
int prefill_share_selftest() {
    for (int walkers : {2, 3, 74, 148}) {
        for (int n_step : {1, 2, 3, 7, 64, 65, 172, 448}) {
            for (int n_tile = walkers + 1; n_tile < 4 * walkers; n_tile += 1 + walkers / 20) {
                const PfShare h = pf_share(n_tile, n_step, walkers);
                std::vector<int> begun(n_tile, 0), begun_by(n_tile, -1), begun_at(n_tile, 0), done(n_tile, 0);
                for (int w = 0; w < walkers; ++w) {
                    int at = 0;
                    for (PfItem it = pf_share_item(h, n_tile, n_step, w, walkers, 0); it.tile < n_tile; it = pf_share_item(h, n_tile, n_step, w, walkers, it.q + 1)) {
                        if (it.tile < 0 || it.from < 0 || it.from >= it.to || it.to > n_step) { return 101; }
                        if (it.from > 0 && (begun[it.tile] != it.from || begun_by[it.tile] != w - 1 || begun_at[it.tile] > at)) { return 102; }
                        at += it.to - it.from;
                        done[it.tile] += it.to - it.from;
                        if (it.to < n_step) { begun[it.tile] = it.to; begun_by[it.tile] = w; begun_at[it.tile] = at; }
                    }
                    if (at != h.rounds * n_step + h.len + (walkers - 1 - w < h.rem ? 1 : 0)) { return 103; }
                }
                for (int t = 0; t < n_tile; ++t) { if (done[t] != n_step) { return 104; } }
            }
        }
    }
    return 0;
}
int prefill_tile_tokens(int type, int64_t n_rows, int nb, int T, bool beside) {
    bool share;
    if (type == 12 || type == 14) { return prefill_kq_tile_tokens(n_rows, nb, T, 0, 0, beside, device_sms(), &share); }
    return best_form(n_rows, nb, T, 0, 0, 0, beside, device_sms(), &share).tok;
}

size_t prefill_weight_bytes(int type, int64_t n_rows, int nb) {
    const size_t tile = (type == 12 || type == 14) ? (size_t)PF_KQ_WTILE : (size_t)PF_WTILE_F16;
    return (size_t)((n_rows + PF_ROWS - 1) / PF_ROWS) * nb * tile;
}
size_t prefill_act_bytes(int T, int nb) {   // (the largest of the layouts)
    return std::max((size_t)((T + PF_TOK - 1) / PF_TOK) * PF_TOK * nb * 68,
                    (size_t)((T + PF_KQ_TOK_MAX - 1) / PF_KQ_TOK_MAX) * PF_KQ_TOK_MAX * nb * 72);
}

cudaError_t launch_prefill_retile(int type, const uint8_t *raw, int64_t row_stride, int64_t n_rows, int nb, uint8_t *base, int64_t dst_row0, cudaStream_t stream) {
    if (type == 12 || type == 14) { return launch_prefill_retile_kq(type, raw, row_stride, n_rows, nb, base, dst_row0, stream); }
    if ((type != 2 && type != 8) || n_rows < 1 || nb < 1) { return cudaErrorInvalidValue; }
    if ((reinterpret_cast<uintptr_t>(raw) & 1) || (row_stride & 1)) { return cudaErrorInvalidValue; }
    const int64_t warps = (n_rows + 7) / 8 * ((nb + 3) / 4);
    const unsigned blocks = (unsigned)((warps + 7) / 8);
    if (type == 2) { prefill_retile_kernel<2><<<blocks, 256, 0, stream>>>(raw, row_stride, n_rows, nb, base, dst_row0); }
    else           { prefill_retile_kernel<8><<<blocks, 256, 0, stream>>>(raw, row_stride, n_rows, nb, base, dst_row0); }
    return cudaGetLastError();
}

template <bool SILU>
static cudaError_t launch_quant_t(const float *x, int64_t x_stride, int T, int K, const float *norm_w, float eps, uint8_t *yq, cudaStream_t stream, int weight_type,
                                  int tile_tok, int part_len, int64_t part_stride, bool pdl, uint8_t *tap, const float *silu_table, float *act) {
    if (weight_type != 2 && weight_type != 8 && weight_type != 12 && weight_type != 14) { return cudaErrorInvalidValue; }
    if (part_len <= 0) { part_len = K; part_stride = 0; }
    if ((part_len & 3) || (part_stride & 3) || K % part_len != 0) { return cudaErrorInvalidValue; }
    if (T < 1 || tile_tok < 1 || K < 32 || (K & 31) || K > PF_MAX_K || (x_stride & 3) || ((uintptr_t)x & 15) || ((uintptr_t)act & 15)) { return cudaErrorInvalidValue; }
    const size_t smem = norm_w != nullptr ? (size_t)K : 0;   // K / 4 floats
    const bool kq = weight_type == 12 || weight_type == 14;
    auto of_groups = [&](auto pg) {
        constexpr int PG = decltype(pg)::value;
        if constexpr (SILU) { return kq ? prefill_quant_kernel<false, true, PG, true> : prefill_quant_kernel<false, false, PG, true>; }
        else { return kq ? (norm_w ? prefill_quant_kernel<true, true, PG, false> : prefill_quant_kernel<false, true, PG, false>) : (norm_w ? prefill_quant_kernel<true, false, PG, false> : prefill_quant_kernel<false, false, PG, false>); }
    };
    const int groups = (K / 8 + PF_QUANT_THREADS - 1) / PF_QUANT_THREADS;
    auto *kernel = groups == 1 ? of_groups(std::integral_constant<int, 1>{}) : groups == 2 ? of_groups(std::integral_constant<int, 2>{}) : of_groups(std::integral_constant<int, PF_QUANT_GROUPS>{});
    return launch_maybe_pdl(kernel, dim3((unsigned)T), PF_QUANT_THREADS, smem, stream, pdl, x, x_stride, K, norm_w, eps, yq, tile_tok, part_len, part_stride, tap, silu_table, act);
}
cudaError_t launch_prefill_quant(const float *x, int64_t x_stride, int T, int K, const float *norm_w, float eps, uint8_t *yq, cudaStream_t stream, int weight_type,
                                 int tile_tok, int part_len, int64_t part_stride, bool pdl, uint8_t *tap) {
    return launch_quant_t<false>(x, x_stride, T, K, norm_w, eps, yq, stream, weight_type, tile_tok, part_len, part_stride, pdl, tap, nullptr, nullptr);
}
cudaError_t launch_prefill_silu_quant(const float *upgate, int T, int F, const float *silu_table, float *act, uint8_t *yq, cudaStream_t stream, int weight_type, int tile_tok, bool pdl) {
    return launch_quant_t<true>(upgate, 2 * (int64_t)F, T, F, nullptr, 0.f, yq, stream, weight_type, tile_tok, 0, 0, pdl, nullptr, silu_table, act);
}

cudaError_t launch_prefill_gemm(const PrefillGemm &g, cudaStream_t stream, bool pdl) {
    if (g.type == 12 || g.type == 14) { return launch_prefill_gemm_kq(g, stream, pdl); }
    if ((g.type != 2 && g.type != 8) || g.w == nullptr || g.yq == nullptr || g.out == nullptr || g.T < 1 || g.nb < 1 || g.n_rows < 1) { return cudaErrorInvalidValue; }
    if ((g.tile_tok != 16 && g.tile_tok != 8) || g.split < 0 || g.split > 2) { return cudaErrorInvalidValue; }
    bool share = false;
    const bool pair = best_form(g.n_rows, g.nb, g.T, g.tile_tok, g.split, g.tiles, g.beside, device_sms(), &share).split == 2;
    share = share && g.handoff != nullptr;
    if (g.selftest_late) { return !share || g.T <= 64 || g.tile_tok != 16 ? cudaErrorInvalidValue : pair ? launch_gemm_t<16, 2, false, true, true>(g, stream, pdl) : launch_gemm_t<16, 1, true, true, true>(g, stream, pdl); }
    // Many tokens (MANY): the epilogue is the bound and the weights come out of L2; copies of half a block are in its way for less long.
    // 22016 x 4096 x 448 tokens 659 us with one copy a step, 649 by blocks, 642 by halves, 646 by quarters. Where the weights' way
    // through HBM is the bound one copy is better: 4096 x 11008 x 64 tokens 55.8 us, by halves 56.2.
    const bool many = g.T > 64;
    if (g.tile_tok == 8) {
        if (share) { return pair ? launch_gemm_t<8, 2, false, true>(g, stream, pdl) : launch_gemm_t<8, 1, false, true>(g, stream, pdl); }
        return pair ? launch_gemm_t<8, 2>(g, stream, pdl) : launch_gemm_t<8, 1>(g, stream, pdl);
    }
    if (share) { return pair ? launch_gemm_t<16, 2, false, true>(g, stream, pdl) : many ? launch_gemm_t<16, 1, true, true>(g, stream, pdl) : launch_gemm_t<16, 1, false, true>(g, stream, pdl); }
    return pair ? launch_gemm_t<16, 2>(g, stream, pdl) : many ? launch_gemm_t<16, 1, true>(g, stream, pdl) : launch_gemm_t<16, 1>(g, stream, pdl);
}

cudaError_t launch_prefill_qkv_post(const float *qkv, int T, int dl, int hd, const int *pos_base, const float2 *rope, __half *q_out, __half *k_cache,
                                    __half *v_cache, int n_ctx, int64_t seq_stride, cudaStream_t stream, bool pdl) {
    const int64_t qk_blocks = ((int64_t)dl * T + PF_POST_THREADS - 1) / PF_POST_THREADS;
    const int64_t v_blocks = seq_stride ? qk_blocks : (int64_t)((dl + PF_POST_E - 1) / PF_POST_E) * ((T + PF_POST_T - 1) / PF_POST_T);
    return launch_maybe_pdl(prefill_qkv_post_kernel, dim3((unsigned)(qk_blocks + v_blocks)), PF_POST_THREADS, 0, stream, pdl, qkv, T, dl, hd, pos_base, rope, q_out, k_cache, v_cache, n_ctx, seq_stride, (int)qk_blocks);
}

// the last pass's columns into the buffers the mat-vec passes leave them in
__global__ void prefill_keep_kernel(const PrefillKeep k) {
    for (int s = 0; s < 4; ++s) {
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k.n4[s]; i += (int64_t)gridDim.x * blockDim.x) { k.dst[s][i] = k.src[s][i]; }
    }
}
cudaError_t launch_prefill_keep(const PrefillKeep &k, cudaStream_t stream) {
    prefill_keep_kernel<<<64, 256, 0, stream>>>(k);
    return cudaGetLastError();
}

cudaError_t launch_prefill_silu_mul(const float *upgate, int T, int F, const float *silu_table, float *act, cudaStream_t stream, bool pdl) {
    const int64_t n = (int64_t)T * F;
    return launch_maybe_pdl(prefill_silu_mul_kernel, dim3((unsigned)((n + 255) / 256)), 256, 0, stream, pdl, upgate, T, F, silu_table, act);
}

}  // namespace spyb
