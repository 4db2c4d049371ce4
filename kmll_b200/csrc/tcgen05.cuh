// mbarriers with bounded waits, and the tcgen05 instructions that the tensor-core kernels share.
#pragma once

#include <stdint.h>

namespace kmll {

constexpr unsigned long long kWaitLimitTicks = 4000000000ull;  // every mbarrier wait gives up after this many cycles (2 to 4 s)
__device__ inline uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ inline void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ inline void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ inline bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait; false = timed out (the caller raises the status word and unwinds).  Roles meet at hardware barriers only where every warp
// comes by, time-out or not: ahead of the roles' loops and behind them.
template <bool BACKOFF = true>
__device__ inline bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();  // (not %globaltimer: reading that register costs a good fraction of a microsecond)
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i) {
            if (mbar_try_wait(bar, parity)) return true;
            if (BACKOFF) __nanosleep(64);  // leave the issue slots to the warps that share the scheduler
        }
        if ((unsigned long long)(clock64() - t0) > kWaitLimitTicks) return false;
    }
}
__device__ inline void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ inline void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ inline void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Tensor memory is allocated before the block releases its dependents, that is, a block barrier stands between tcgen05.alloc and
// pdl_wait(): a dependent block that held the columns while it waits for this grid would keep this grid in alloc, the one wait without a bound.
// shared-memory matrix descriptor: K-major operand tile with 128-byte rows in the 128-byte swizzle (what TMA writes with
// CU_TENSOR_MAP_SWIZZLE_128B): groups of 8 rows are 1024 bytes apart; version 1 (sm_100); layout type 2 = SWIZZLE_128B
__device__ inline uint64_t gemm_smem_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor of kind::f16: D = f32, A = B = binary16, both K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t gemm_idesc_f16(int m, int n) {
    return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// the same with A = B = bf16
__host__ __device__ constexpr uint32_t gemm_idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// ---- issue by a converged warp -------------------------------------------------------------------------------------------
// A role that issues MMAs, commits or copies walks its loops as a whole warp, and one elected lane's predicate does the issuing.  The
// operands are then values the compiler knows to be the same in every lane, and stay in uniform registers.  With
// `if (lane == 0)` around the loops every operand of every instruction goes through vector registers first, and an issue costs the
// thread 70 to 230 cycles (attention of 2048 x 128 x 32 heads: 234 cycles per 128 x 128 x 16 MMA; this way 61, the tensor core's own time).
__device__ inline int uniform_warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
__device__ inline uint32_t elect_lead() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p;
}
// all lanes leave a bounded wait together
__device__ inline bool warp_wait(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait<false>(bar, parity)) != 0; }
// The last of the first `issued` uses of a ring of `stages` that is one of stage st; -1: none.
__host__ __device__ constexpr int ring_last_use(int issued, int st, int stages) { return issued <= st ? -1 : st + (issued - 1 - st) / stages * stages; }
static_assert(ring_last_use(0, 0, 1) == -1 && ring_last_use(1, 0, 1) == 0 && ring_last_use(7, 0, 1) == 6, "one stage");
static_assert(ring_last_use(0, 0, 2) == -1 && ring_last_use(1, 0, 2) == 0 && ring_last_use(1, 1, 2) == -1 && ring_last_use(2, 1, 2) == 1, "two stages, first uses");
static_assert(ring_last_use(5, 0, 2) == 4 && ring_last_use(5, 1, 2) == 3 && ring_last_use(20, 1, 9) == 19 && ring_last_use(20, 2, 9) == 11, "later uses");
// A block does not end with copies under way: whoever began the copies of the first `issued` uses of a ring waits, before it leaves its
// role after a time-out, for the last one of each stage.  (It has seen the uses before end, so the parity is that one's.)
__device__ inline bool ring_landed(uint64_t* full, int issued, int stages) {
    bool ok = true;
    for (int st = 0; st < stages; ++st) {
        const int last = ring_last_use(issued, st, stages);
        if (last >= 0) ok = warp_wait(&full[st], (uint32_t)(last / stages) & 1u) && ok;
    }
    return ok;
}
__device__ inline void lead_mma_f16(uint32_t lead, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(lead) : "memory");
}
// the A operand from tensor memory: lane = row, a 32-bit column holds two consecutive 16-bit entries of K
__device__ inline void lead_mma_f16_ts(uint32_t lead, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(lead) : "memory");
}
__device__ inline void lead_mma_i8(uint32_t lead, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t@e tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(lead) : "memory");
}
__device__ inline void lead_mma_i8_ts(uint32_t lead, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t@e tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(lead) : "memory");
}
__device__ inline void lead_commit(uint32_t lead, uint64_t* bar) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
                 ::"r"(smem_u32(bar)), "r"(lead) : "memory");
}
__device__ inline void lead_expect_tx(uint32_t lead, uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
                 ::"r"(smem_u32(bar)), "r"(bytes), "r"(lead) : "memory");
}
// tiled TMA loads into this block's shared memory (no multicast), completion on an mbarrier
__device__ inline void lead_tma_2d(uint32_t lead, uint32_t smem_dst, const void* map, int x, int y, uint64_t* bar) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %5, 0;\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}"
                 ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)), "r"(lead) : "memory");
}
__device__ inline void lead_tma_3d(uint32_t lead, uint32_t smem_dst, const void* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %6, 0;\n\t"
                 "@e cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n\t}"
                 ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)), "r"(lead) : "memory");
}

// 32 columns of this warp's 32 lanes; the values are there when the call returns
__device__ inline void tmem_load_x32(uint32_t taddr, uint32_t (&d)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]),
          "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]), "=r"(d[16]), "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]),
          "=r"(d[21]), "=r"(d[22]), "=r"(d[23]), "=r"(d[24]), "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]), "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// the reverse (tmem_store_wait before anybody else is told)
__device__ inline void tmem_store_x32(uint32_t taddr, const uint32_t (&d)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
        ::"r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]), "r"(d[8]), "r"(d[9]), "r"(d[10]),
          "r"(d[11]), "r"(d[12]), "r"(d[13]), "r"(d[14]), "r"(d[15]), "r"(d[16]), "r"(d[17]), "r"(d[18]), "r"(d[19]), "r"(d[20]),
          "r"(d[21]), "r"(d[22]), "r"(d[23]), "r"(d[24]), "r"(d[25]), "r"(d[26]), "r"(d[27]), "r"(d[28]), "r"(d[29]), "r"(d[30]), "r"(d[31]), "r"(taddr)
        : "memory");
}
__device__ inline void tmem_store_x16(uint32_t taddr, const uint32_t (&d)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
        ::"r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]), "r"(d[8]), "r"(d[9]), "r"(d[10]),
          "r"(d[11]), "r"(d[12]), "r"(d[13]), "r"(d[14]), "r"(d[15]), "r"(taddr)
        : "memory");
}
__device__ inline void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ inline void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

}  // namespace kmll
