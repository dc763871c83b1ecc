// PTX wrappers of the tensor-core kernels: mbarriers, bulk copies, tensor memory, tcgen05.mma.
#pragma once

#include "sm100_common.cuh"

namespace sm100 {
namespace {

__device__ __forceinline__ uint32_t smem_addr(const void * p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// non-blocking look at a barrier phase
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
constexpr uint32_t TC_WAIT_LIMIT = 1u << 21;  // polls of one mbarrier wait before the CTA gives up (~1 s)
// Bounded wait.  Returns false when the CTA is giving up (this wait ran out, or another one did).
// Waiters off the critical path (`patient`) sleep between polls so that they leave the issue slots alone.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, volatile int * abort_flag, int * fault, int site, bool patient) {
    for (uint32_t i = 0; i < TC_WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (patient || i >= 64) {
            if (*abort_flag != 0) return false;
            __nanosleep(patient ? 100 : 32);
        }
    }
    *abort_flag = 1 + site;
    *(volatile int *) fault = 1 + site;
    return false;
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// global -> shared bulk copy through the TMA unit; src, dst and bytes are multiples of 16
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void * src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

// Shared-memory matrix descriptor of a K-major operand without swizzle (8-row x 16-byte core matrices), as two
// words.  Low: bits 0-13 start address >> 4, bits 16-29 (bytes between the two core matrices an instruction
// spans along K) >> 4.  High: bits 0-13 (bytes between 8-row groups) >> 4, bit 14 = descriptor version of sm_100;
// base offset, swizzle mode = 0.
// Instruction descriptor of kind::f16: f16 A and B, both K-major, f32 accumulator, M x N tile.
__host__ __device__ constexpr uint32_t instr_desc_f16(int m, int n) {
    return (1u << 4) | ((uint32_t) (n >> 3) << 17) | ((uint32_t) (m >> 4) << 24);
}
// MMAs are executed by a whole (converged) warp: one elected lane issues.  Keeping the warp converged around the issue lets the
// operands live in uniform registers - issued from inside a divergent `if (lane == 0)` each MMA cost ~86 cycles.  A in tensor memory:
// lane = row, 32-bit column j of the 8 columns of a step = the row's K elements 2j (low half) and 2j + 1.
// The four MMAs of a 64-wide chunk (A in tensor memory) as one block of instructions: the issuing lane is given as a
// flag, the descriptors and addresses of the K steps are derived inside.  `b_desc` is the whole 64-bit descriptor
// of the first K step, `b_step` what a K step adds to it.
__device__ __forceinline__ void mma4_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint64_t b_step, uint32_t idesc, uint32_t accumulate,
                                            uint32_t issuer) {
    asm volatile(
        "{\n\t.reg .pred pi, pacc, pone;\n\t.reg .b64 d1, d2, d3;\n\t.reg .b32 a1, a2, a3;\n\t"
        "elect.sync _|pi, 0xffffffff;\n\t"
        "setp.ne.b32 pacc, %5, 0;\n\t"
        "setp.eq.b32 pone, %6, %6;\n\t"
        "add.u64 d1, %2, %3;\n\t"
        "add.u64 d2, d1, %3;\n\t"
        "add.u64 d3, d2, %3;\n\t"
        "add.u32 a1, %1, 8;\n\t"
        "add.u32 a2, %1, 16;\n\t"
        "add.u32 a3, %1, 24;\n\t"
        "@pi tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %4, pacc;\n\t"
        "@pi tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], d1, %4, pone;\n\t"
        "@pi tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], d2, %4, pone;\n\t"
        "@pi tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], d3, %4, pone;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "l"(b_step), "r"(idesc), "r"(accumulate), "r"(issuer)
        : "memory");
}
// two commits (weight stage, activation stage) by the issuing lane
__device__ __forceinline__ void mma_commit2(uint32_t bar_a, uint32_t bar_b, uint32_t issuer) {
    asm volatile(
        "{\n\t.reg .pred pi;\n\t"
        "elect.sync _|pi, 0xffffffff;\n\t"
        "@pi tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
        "@pi tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}" ::"r"(bar_a),
        "r"(bar_b), "r"(issuer)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// arrives on `bar` when every MMA issued so far by the elected lane has finished reading shared memory and writing
// TMEM (whole converged warp: elect.sync picks the lane that issued them)
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
        : "memory");
}
// 32 lanes x 16 consecutive f32 columns of the accumulator: thread i of the warp receives lane (base lane + i)
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// How the tiles of a launch are dealt: as many as fill whole waves go to one CTA each, the rest - the last wave, or all when there
// are fewer than SMs - have their K range cut over `splits` CTAs, whose partial tiles a second launch adds in order.  (160 tiles of 96
// chunks on 148 SMs: 96 + 12 chunks' time with the last 12 cut in eight, 192 without.)
struct TilePlan {
    int64_t whole;   // tiles [0, whole): one CTA each
    int64_t cut;     // tiles [whole, whole + cut): `splits` CTAs each
    int splits;
    int64_t cost;    // of the whole launch
};
// Costs in tenths of a chunk's time of a 128 x 128 tile (about 0.3 us).  A wave costs its chunks (`per_chunk` each) plus about eight chunks of
// start and epilogue; partial tiles cost another six for the launch that adds them and a write and a read of every partial output
// (`outputs` per tile).  Ties go to fewer CTAs.
// `least` > 1: no CTA may take the whole of K, every tile is cut.
inline TilePlan plan_tiles(int64_t tiles, int nchunks, int per_chunk, int64_t outputs, int least) {
    const int64_t sms = sm_count();
    TilePlan p = {least > 1 ? 0 : tiles / sms * sms, least > 1 ? tiles : tiles % sms, 1, 0};
    const int64_t waves = p.whole / sms;
    int64_t best = 0;
    if (p.cut > 0) {
        best = INT64_MAX;
        for (int s = least; s <= least + 7 && s <= nchunks; ++s) {
            const int64_t cost = (p.cut * s + sms - 1) / sms * ((int64_t) ((nchunks + s - 1) / s) * per_chunk + 80) + (s > 1 ? 60 + s * p.cut * outputs / 20000 : 0);
            if (cost < best) { best = cost; p.splits = s; }
        }
    }
    p.cost = waves * ((int64_t) nchunks * per_chunk + 80) + best;
    if (p.splits == 1) p = {tiles, 0, 1, p.cost};
    return p;
}
inline int64_t plan_ctas(const TilePlan & p) { return p.whole + p.cut * p.splits; }

}  // namespace
}  // namespace sm100
