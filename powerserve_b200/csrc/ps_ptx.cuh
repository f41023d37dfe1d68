// ps_ptx.cuh - inline-PTX building blocks shared by every kernel file: mbarrier, 1-D TMA bulk copies, programmatic dependent
// launch, and the tcgen05 (5th-generation tensor core) wrappers - shared-memory operand descriptors for the canonical
// K-major no-swizzle layout, the single-thread MMA issue, commit, fences, tensor-memory loads and the bounded mbarrier wait.
#pragma once
#include "ps_math.cuh"

#include <cstdint>

// ---------------------------------------------------------------------------------------------------- PTX helpers
PS_D uint32_t ps_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
PS_D void ps_mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ps_smem_u32(bar)), "r"(count));
}
PS_D void ps_mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ps_smem_u32(bar)), "r"(bytes) : "memory");
}
PS_D void ps_mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ps_smem_u32(bar)) : "memory");
}
PS_D void ps_mbar_wait(uint64_t *bar, uint32_t parity) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "WAIT_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1;\n\t"
        "@p bra DONE_%=;\n\t"
        "bra WAIT_%=;\n\t"
        "DONE_%=:\n\t}" ::"r"(ps_smem_u32(bar)),
        "r"(parity)
        : "memory");
}
// 1-D TMA: global -> shared, completion counted in bytes on an mbarrier
PS_D void ps_bulk_g2s(void *dst_smem, const void *src_gmem, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(ps_smem_u32(dst_smem)),
                 "l"(src_gmem), "r"(bytes), "r"(ps_smem_u32(bar))
                 : "memory");
}
PS_D void ps_fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
PS_D void ps_grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
PS_D void ps_grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Programmatic dependent launch.  A kernel launched by launch_k / pa_launch_dep may start while the one before it in the stream still runs; nothing
// that other kernels write is read, and nothing they read is written, before this wait, which ends when the kernel before is complete (and, as that one
// waited too, all before it).  Every kernel launched that way waits in all threads that touch global memory.  After it the next kernel may start
PS_D void ps_grid_dep() {
    ps_grid_dep_wait();
    ps_grid_dep_launch();
}
PS_D void ps_bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// ---------------------------------------------------------------------------------------------------- tcgen05 helpers
PS_D uint64_t ps_tc_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    // cute::UMMA::SmemDescriptor: start address [0,14) >> 4, leading byte offset [16,30) >> 4, stride byte offset [32,46) >> 4,
    // version [46,48) = 1 (Blackwell), layout type [61,64) = 0 (no swizzle)
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) | ((uint64_t)(sbo_bytes >> 4) << 32) | (1ull << 46);
}
PS_D void ps_tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
PS_D void ps_tc_mma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) { // A operand from tensor memory
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// one thread of a converged warp; unlike `lane == 0` it tells the compiler that the branch has a single active thread
PS_D bool ps_elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
PS_D void ps_tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ps_smem_u32(bar)) : "memory");
}
PS_D void ps_tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
PS_D void ps_tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
PS_D void ps_tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// bounded mbarrier wait: a mis-sequenced pipeline must never hang the GPU.  A poll that fails has suspended the thread for 7 800 cycles, so
// 2^18 polls are about a second; then it gives up (returns false)
PS_D bool ps_tc_poll(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
PS_D bool ps_tc_wait(uint64_t *bar, uint32_t parity, int polls = 1 << 18) {
    for (int spin = 0; spin < polls; spin++)
        if (ps_tc_poll(ps_smem_u32(bar), parity)) return true;
    return false;
}
// the same by a converged warp that goes on together: giving up is the warp's decision, not a lane's (elect.sync and the .aligned tcgen05
// instructions that follow need all lanes).  The limit is a time here, 2^31 SM cycles unless a test asks for less
#define PS_TC_WAIT_CYCLES 0x80000000u
// limits where a block goes on after a wait that gave up, and meets the slot of the missing copy again dozens of times: some 30 ms, so that all of them together end
// within seconds (a copy takes microseconds; a flag that ended the later waits at once cost the kernels 2 to 16 %)
#define PS_COPY_POLLS (1 << 13)
#define PS_COPY_CYCLES (1u << 26)
PS_D uint32_t ps_clock32() {
    uint32_t t;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(t));
    return t;
}
PS_D bool ps_tc_wait_warp(uint64_t *bar, uint32_t parity, uint32_t cycles = PS_TC_WAIT_CYCLES) {
    bool ok = ps_tc_poll(ps_smem_u32(bar), parity);
    if (!ok) {
        const uint32_t t0 = ps_clock32();
        do ok = ps_tc_poll(ps_smem_u32(bar), parity);
        while (!ok && ps_clock32() - t0 < cycles);
    }
    return __all_sync(0xffffffffu, ok);
}
// named barrier that says whether `ok` holds in every one of its n threads
PS_D bool ps_bar_all(int id, int n, bool ok) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\tbar.red.and.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(id), "r"(n), "r"((uint32_t)ok) : "memory");
    return r != 0;
}

// position in a ring of N: index and the parity of the round
template <int N> struct PsRing {
    int i = 0;
    uint32_t round = 0;
    PS_D void step() {
        if (++i == N) { i = 0; round ^= 1; }
    }
};
