// Device helpers shared by the tcgen05 prompt kernels (spyb_prefill.cu: Q4_0 / Q8_0, spyb_prefill_kq.cu: Q4_K / Q6_K):
// shared-memory and mbarrier accessors, operand descriptors, the MMA / commit / tensor-memory instructions, bounded waits.
#pragma once

#include "spyb_common.cuh"
#include "spyb_kernels.h"

namespace spyb {
namespace {

constexpr int PF_M           = PF_ROWS;            // weight rows per CTA = M of the MMA
constexpr int PF_NCOL        = 128;                // columns of D per block step = N of the MMA
constexpr int PF_TILE        = PF_M * 32;          // bytes of one s8 operand tile
constexpr int PF_EPI_WARPS   = 8;                  // epilogue warps: (row quadrant 0..3) x (half of the columns); 12 warps in all leave them 168 registers
constexpr int PF_BATCH       = 4;                  // blocks per batch: the unit of the copies, of the expansion and of stage reuse
constexpr int PF_RING        = 4;                  // batches in the shared-memory rings
constexpr int PF_MMA_WARPS   = 2;                  // warps whose first thread issues the MMAs of every PF_MMA_WARPS-th block
constexpr int PF_THREADS     = (PF_EPI_WARPS + 2 + PF_MMA_WARPS) * 32;   // + the copy warp and the expander warp
constexpr int PF_GEMM_EPI_WARPS = 16, PF_GEMM_THREADS = 640;   // the Q4_0 / Q8_0 kernel: sixteen epilogue warps and four feeder warps, 96 registers each
constexpr int PF_DBUF        = 4;                  // accumulator buffers in tensor memory, PF_NCOL columns each (512 columns = all of it)

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
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

// shared-memory operand descriptor: K-major, no swizzle; element (row r, byte k) of the tile lies at
// (r / 8) * 256 + (k / 16) * 128 + (r % 8) * 16 + k % 16: leading (K-chunk) offset 128, stride (8-row group) offset 256
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(256u >> 4) << 32) | (1ull << 46);
}
// instruction descriptor: D s32, A and B s8 K-major, N = 128, M = 128
constexpr uint32_t PF_IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(PF_NCOL >> 3) << 17) | ((uint32_t)(PF_M >> 4) << 24);

__device__ __forceinline__ void mma_s8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc) {
    const uint32_t zero = 0, accumulate = 1;   // D += A B^T: D holds the offset pattern
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(PF_IDESC), "r"(accumulate), "r"(zero) : "memory");
}
// e4m3 operands (kind::f8f6f4), f32 accumulators: D (+)= A B^T. Small integers are exact in e4m3 (|v| <= 16, and multiples of 16
// up to 128), their products and the sums of a block's few products are exact in f32, so D holds (float)(integer sum) itself.
constexpr uint32_t PF_IDESC_F8 = (1u << 4) | ((uint32_t)(PF_NCOL >> 3) << 17) | ((uint32_t)(PF_M >> 4) << 24);
__device__ __forceinline__ void mma_f8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
    const uint32_t zero = 0;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(PF_IDESC_F8), "r"(accumulate), "r"(zero) : "memory");
}
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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// the same 32-bit word into 32 consecutive columns of this thread's lane
__device__ __forceinline__ void tmem_st32_same(uint32_t taddr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(v) : "memory");
}
// 16 consecutive columns of this thread's lane from 16 registers (callers keep a register set that holds the offset
// pattern alive across the loop, so that no copies are made per store)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                   "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// e4m3 code of the integer v, 0 <= v <= 15 (exact: three mantissa bits cover 8..15), and of a signed value in [-15, 15]
__host__ __device__ __forceinline__ uint32_t e4m3_of_small(uint32_t v) {
    if (v == 0) { return 0u; }
    const int e = v >= 8 ? 3 : v >= 4 ? 2 : v >= 2 ? 1 : 0;
    return ((uint32_t)(e + 7) << 3) | ((v << (3 - e)) & 7u);
}
__host__ __device__ __forceinline__ uint32_t e4m3_of_signed(int v) { return v < 0 ? (0x80u | e4m3_of_small((uint32_t)-v)) : e4m3_of_small((uint32_t)v); }
// a Q8_0 activation byte y in [-127, 127] as two e4m3 values: y = hi + lo with lo = y mod 16 in [0, 15] and hi = y - lo a
// multiple of 16 in [-128, 112] (the code of |hi| / 16 with the exponent raised by four)
__device__ __forceinline__ void e4m3_split4(uint32_t q, uint32_t &hi, uint32_t &lo) {
    hi = 0u; lo = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int y = (int)(int8_t)((q >> (8 * i)) & 0xffu);
        const int yl = y & 15, yh = (y - yl) >> 4;   // yh in [-8, 7]
        const uint32_t ch = yh == 0 ? 0u : (e4m3_of_signed(yh) + 0x20u);
        hi |= ch << (8 * i);
        lo |= e4m3_of_small((uint32_t)yl) << (8 * i);
    }
}

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

}  // namespace
}  // namespace spyb
