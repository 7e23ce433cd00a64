// Device helpers shared by the tcgen05 prompt kernels (spyb_prefill.cu: Q4_0 / Q8_0, spyb_prefill_kq.cu: Q4_K / Q6_K):
// shared-memory and mbarrier accessors, operand descriptors, the MMA / commit / tensor-memory instructions, bounded waits.
#pragma once

#include <algorithm>

#include "spyb_common.cuh"
#include "spyb_kernels.h"

namespace spyb {
namespace {

constexpr int PF_M           = PF_ROWS;            // weight rows per CTA = M of the MMA
constexpr int PF_GEMM_EPI_WARPS = 16, PF_GEMM_THREADS = 640;   // the Q4_0 / Q8_0 kernel: sixteen epilogue warps and four feeder warps, 96 registers each
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) { asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(addr), "r"(a), "r"(b) : "memory"); }
__device__ __forceinline__ float lds32f(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void lds128_2x64(uint32_t addr, uint64_t &a, uint64_t &b) {
    asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ uint64_t lds64u(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// f16 operands, f32 accumulators, 128 x N x 16: D (+)= A B^T. 8-bit integers are exact in f16, their products and the sums of a
// block's few products are exact in f32
__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__host__ __device__ constexpr uint32_t idesc_f16(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(PF_M >> 4) << 24); }
// K-major operand without swizzle, core matrices of 8 rows x 16 bytes: `lbo` bytes between neighbouring 16-byte K chunks, `sbo` bytes
// between neighbouring groups of eight rows
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// one lane of a converged warp, the same one every time. Instructions whose operands go through uniform registers (tcgen05.mma,
// tcgen05.commit, bulk copies) issue at half the cost under this predicate than under `lane == 0` (measured: 69 against 140 cycles
// per MMA), because the compiler knows that one thread at most is active.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// feeder roles (copy, expansion, MMA issue) run ahead of the epilogue: their waits back off instead of competing with the
// epilogue warps for issue slots
__device__ __forceinline__ bool mbar_wait_relaxed(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try_wait(bar, parity)) { return true; }
    const uint64_t t0 = global_timer_ns();
    for (;;) {
        __nanosleep(100);
        if (mbar_try_wait(bar, parity)) { return true; }
        if (global_timer_ns() - t0 > limit_ns) { return false; }
    }
}
// A wait whose fast path is one test and one branch, for loops that count instructions. When it runs out of time it sets limit_ns to
// zero and returns, and every later wait with the same limit gives up at once: the caller may run through to its end and report then.
__device__ __forceinline__ void mbar_wait_lean(uint32_t bar, uint32_t parity, uint64_t &limit_ns) {
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .u64 t0, t;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\tmov.u64 t0, %%globaltimer;\n"
                 "AGAIN:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\tmov.u64 t, %%globaltimer;\n\tsub.u64 t, t, t0;\n\t"
                 "setp.lt.u64 q, t, %0;\n\t@q bra AGAIN;\n\tmov.u64 %0, 0;\nDONE:\n\t}"
                 : "+l"(limit_ns) : "r"(bar), "r"(parity) : "memory");
}
__device__ __forceinline__ void pf_report(int *error_flag, int code) {
    if (error_flag != nullptr) { atomicExch(error_flag, code); }
}

// Shared tiles: where the tiles are no whole number of rounds, what is left after all rounds but one - one to two tiles a walker (CTA or cluster) - is laid end
// to end and cut into equal stretches, one a walker, from the last one down. A tile on a cut is two walkers': the lower one takes its first
// steps before the rest of its stretch and leaves the accumulators in the handoff buffer, the higher one takes the last steps at the end of
// its own. Whoever waits thus waits for a CTA that was started before itself, and for steps that were done by then if all walk at one pace
// (a stretch is at least a tile long). Whole rounds come first, in step: walkers that are beside each other then read the same weights at the same time.
// Whole tiles / shared, us with the quantizer: 4096 x 4096 x 448 tokens (6.05 rounds) 142.5 / 126, 5120 x 13824 x 32 (1.08 rounds of clusters) 73.3 / 54, 12288
// x 4096 x 32 (1.30 rounds) 45.8 / 37. What a cut costs, 2.5 to 6.3 us, is in pf_cost. Whole rounds keep a kernel of their own,
// whose registers do not suffer from the handing over.
struct PfItem { int tile, from, to, q; };   // steps (K-quants: super-blocks) [from, to) of a tile: a walker's item q
__host__ __device__ __forceinline__ PfItem pf_share_item(const PfShare &h, int n_tile, int n_step, int walker, int walkers, int q) {
    const int base = h.rounds * walkers, r = walkers - 1 - walker;
    const int lo = r * h.len + (r < h.rem ? r : h.rem), hi = lo + h.len + (r < h.rem ? 1 : 0);   // (a stretch is at least a tile long)
    const int t0 = (int)(((uint64_t)lo * h.magic) >> 32), x0 = lo - t0 * n_step, t1 = (int)(((uint64_t)hi * h.magic) >> 32), x1 = hi - t1 * n_step;
    const int early = x0 != 0 ? 1 : 0, mid = q - h.rounds - early, n_mid = t1 - t0 - early;
    if (q < h.rounds) { return {walker + q * walkers, 0, n_step, q}; }
    if (mid < 0) { return {base + t0, 0, n_step - x0, q}; }
    if (mid < n_mid) { return {base + t0 + early + mid, 0, n_step, q}; }
    return {mid == n_mid && x1 != 0 ? base + t1 : n_tile, n_step - x1, n_step, q};
}
inline PfShare pf_share(int n_tile, int n_step, int walkers) {   // n_tile > walkers
    const int rounds = n_tile / walkers - 1, steps = (n_tile - rounds * walkers) * n_step;
    return {rounds, steps / walkers, steps % walkers, (0x100000000ull + n_step - 1) / n_step};
}
// What a launch costs, in ns, with its last tiles whole or shared, whichever is less (how: PrefillGemm::tiles). What fills its pipelines; for every block of the
// matrix some time for its bytes, in proportion to the chip; then rounds of tiles: what a tile does once (its drain, and for two CTAs the joining of the
// halves) and a time for each block of the row (less for narrow tiles, whose weights bound them, and about half for two CTAs). A last round that is full beyond
// `full_from` costs up to full_ns more: what it leaves idle, the next launch begins on. Shared tiles make the rounds a fraction, for the handing over and somewhat slower
// blocks. That is a launch with nothing beside it but its successor, a model's prompt. An operator (beside) also pays for the SMs' time that its tiles take, `idle`
// times, and `margin_ns` for sharing: other backends' operators run on the SMs that a whole last round leaves, and shared tiles leave none. Three backends' submits in turn /
// one's, us a submit, whole and shared: Q4_0 10024 x 3328 x 27 tokens 21.7 and 25.4 / 38.2 and 27.9; Q6_K 6520 x 6144 x 39 21.9 and 26.8 / 33.3 and 31.9.
struct PfCost { double launch_ns, tile_ns, block_ns, rows_ns, handoff_ns, slower, full_ns; };
struct PfRule { double full_from, idle, margin_ns; };
inline double pf_cost(const PfCost &c, const PfRule &r, int64_t row_tiles, int64_t tiles, int64_t walkers, int nb, int sms, int how, bool sharable, bool beside, bool *shared) {
    const double once = c.launch_ns + (double)row_tiles / sms * nb * c.rows_ns, busy = (double)tiles / walkers * (c.tile_ns + nb * c.block_ns);
    const double fill = (double)((tiles - 1) % walkers + 1) / walkers;   // of the last round
    const double whole = once + (double)((tiles + walkers - 1) / walkers) * (c.tile_ns + nb * c.block_ns) + c.full_ns * std::max(0.0, (fill - r.full_from) / (1.0 - r.full_from)) + (beside ? r.idle * busy : 0.0);
    *shared = false;
    if (how == 1 || !sharable || tiles <= walkers || (how != 2 && tiles % walkers == 0)) { return whole; }
    const double cut = (double)tiles / walkers * (c.tile_ns + nb * c.block_ns * (1.0 + c.slower));
    const double share = once + c.handoff_ns + cut + (beside ? r.margin_ns + r.idle * (cut + c.handoff_ns) : 0.0);
    *shared = how == 2 || share < whole;
    return *shared ? share : whole;
}
// The word that says that a warp's accumulators lie in the handoff buffer; only the walker they are meant for clears it again. One that gave up may clear it
// before it is set: after any reported error the words are the host's to clear (spyb_backend::clear_device_error).
__device__ __forceinline__ void handoff_publish(unsigned *flag) { asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(1u) : "memory"); }
__device__ __forceinline__ void handoff_wait(const unsigned *flag, uint64_t &limit_ns) {
    const uint64_t t0 = global_timer_ns();
    for (;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (__all_sync(0xffffffffu, v != 0u)) { return; }
        if (__any_sync(0xffffffffu, global_timer_ns() - t0 >= limit_ns)) { limit_ns = 0; return; }
    }
}

}  // namespace
}  // namespace spyb
