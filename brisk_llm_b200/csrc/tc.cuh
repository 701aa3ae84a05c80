// Fifth-generation tensor-core primitives of the prompt multiplies (gemm_k_tc.cu, gemm_tc.cu): mbarriers with bounded waits,
// shared-memory descriptors, tcgen05 instructions.
#pragma once

#include <cuda.h>

#include "kernels.h"

namespace bk {

// A row-major byte matrix [rows][row_bytes] as a TMA descriptor whose box is box_rows x box_bytes (16, 32, 64 or 128; the swizzle is
// as wide as the box, none for 16). Rows past the last arrive as zeros.
CUtensorMap tensor_map(const void* base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows);

#ifdef __CUDACC__
constexpr uint32_t kTmemCols = 512;

__device__ __forceinline__ uint32_t saddr(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory"); }
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(saddr(b)), "r"(parity) : "memory");
    return ok != 0;
}
// The waits of a kernel's warps are bounded: one that lasts longer than `limit` cycles gives up, and whoever gave up says so in the error
// word at the kernel's end. What follows a wait that gave up:
//   - No copy is asked for any more: one into a slot whose last is still on its way overdraws the slot's barrier. Nobody arrives whose
//     own wait did not succeed, so that the waits of others give up in turn.
//   - What had been asked for is waited for at the kernel's end (mbar_drain): copies, MMAs and commits that outlive their CTA write into
//     shared and tensor memory that is another's by then.
//   - A warp stays together. Lanes that went on where others gave up would meet those at no vote and no barrier again.
//
// By every lane of a warp for itself: `dead` where it gave up, at which its later waits return at once; all go on to the same end. A
// __syncwarp follows: behind waits of single lanes even a vote need not bring the warp together again, and .sync.aligned instructions
// (tcgen05.ld, tcgen05.st) that lanes reach apart have ended in an illegal memory access.
__device__ __forceinline__ void mbar_wait(uint64_t* b, uint32_t parity, bool& dead, long long limit) {
    if (dead || mbar_try_wait(b, parity)) return;
    const long long start = clock64();
    while (!mbar_try_wait(b, parity)) {
        if (clock64() - start > limit) {  // bounded in time, not in tries: one try may itself sleep for a while
            dead = true;
            return;
        }
    }
}
// A warp waits for several barriers at once, lanes first .. end - 1 for one each: even where the barriers are long
// complete one wait costs 71 cycles, several at once 111. Every try is voted on, so that all lanes have one answer. False: gave up.
__device__ __forceinline__ bool mbar_wait_all(uint64_t* mine, uint32_t parity, uint32_t first, uint32_t end, long long limit) {
    const uint32_t lane = threadIdx.x & 31;
    const bool waits = lane >= first && lane < end;
    bool done = __all_sync(0xffffffffu, !waits || mbar_try_wait(mine, parity));
    if (!done) {
        const long long start = clock64();
        do {
            done = __all_sync(0xffffffffu, !waits || mbar_try_wait(mine, parity));
        } while (!done && !__any_sync(0xffffffffu, clock64() - start > limit));
    }
    __syncwarp();
    return done;
}
// At the kernel's end, for what is sure to complete: a copy or a commit that was issued. (A second is far more than
// either can take; it is there so that nothing waits without an end.)
__device__ __forceinline__ void mbar_drain(uint64_t* b, uint32_t parity) {
    const long long start = clock64();
    while (!mbar_try_wait(b, parity)) {
        if (clock64() - start > kTcWaitCycles) break;
    }
}

// K-major operand tile without swizzle: core matrices of 8 rows x 16 bytes; `lbo` bytes between the two 16-byte halves of
// K, `sbo` bytes between groups of 8 rows. Bit 46: the descriptor version of this architecture.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) | (uint64_t((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// K-major operand tile with rows of 128 bytes and the 128-byte swizzle (what a TMA load with that swizzle leaves); `addr` may point
// at any 32-byte step inside the first row. The tile starts on a 1024-byte boundary.
__device__ __forceinline__ uint64_t smem_desc_swizzled(uint32_t addr) {
    return uint64_t((addr >> 4) & 0x3FFF) | (1ull << 16) | (uint64_t(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Box at byte x, row y of the map; x is a multiple of 16. Counted on `bar`.
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(saddr(bar))
                 : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes) : "memory");
}
// s32 accumulator, 8-bit A (signed or not) x s8 B, both K-major, M = 128
constexpr uint32_t instr_i8(bool a_signed, uint32_t n) { return (2u << 4) | (uint32_t(a_signed) << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24); }
// f32 accumulator, f16 x f16, both K-major, M = 128
constexpr uint32_t instr_f16(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

// One lane of a converged warp. Issue tcgen05 and TMA instructions under `if (elect_one())` in a warp whose control flow is uniform:
// the operands then stay in uniform registers. Under `lane == 0` each is moved there for every instruction, 45 to 57 cycles an MMA
// against 23 (and 32 for the MMA itself at 64 tokens).
__device__ __forceinline__ bool elect_one() {
    uint32_t mine;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(mine));
    return mine != 0;
}
// D = (accumulate ? D : 0) + A x B, 128 x N x 32 bytes of K; A in tensor memory (lane = row, four values a column)
__device__ __forceinline__ void mma_i8_ts(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t instr, bool accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}" ::"r"(d), "r"(a), "l"(b_desc), "r"(instr),
                 "r"(uint32_t(accumulate))
                 : "memory");
}
// D = A x B, 128 x N x 16 values of K, both operands in shared memory
__device__ __forceinline__ void mma_f16_ss(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t instr) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a_desc), "l"(b_desc), "r"(instr), "r"(0u)
                 : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void async_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 16 columns of the warp's 32 lanes := v
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
// 16 lanes x 16 columns as a warp's fragment: v[4 c + k] holds lane g + 8 (k / 2) and column 8 c + 2 t + k % 2 (g = lane / 4, t = lane % 4)
__device__ __forceinline__ void tmem_ld_frag2(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
// 16 lanes x 8 columns as a warp's fragment: v[k] holds lane g + 8 (k / 2) and column 2 t + k % 2
__device__ __forceinline__ void tmem_ld_frag1(uint32_t taddr, uint32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
}
#endif

}  // namespace bk
