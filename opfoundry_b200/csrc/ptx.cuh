// Thin inline-PTX wrappers for the sm_100a features the sparse-MLA kernels use:
// mbarrier (with bounded waits), TMA tile loads into this CTA's shared memory,
// tcgen05 MMA / TMEM alloc / ld / st / commit, and the shared-memory and
// instruction descriptors tcgen05.mma consumes.
#pragma once
#include <cstdint>
#include <cuda.h>

namespace dsa {

// ------------------------------------------------------------------ addresses
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {   // no arrival
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
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

// Non-blocking probe of a phase (try_wait may park the thread for a while; this never does).
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

// try_wait with an explicit suspend-time hint: the thread is parked by the hardware until the phase
// completes or about `ns` nanoseconds have passed, so a waiting warp neither takes issue slots from the
// warps that have work nor sleeps past the completion (as a nanosleep back-off does).
__device__ __forceinline__ bool mbar_try_wait_hint(uint32_t bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Every wait in these kernels is bounded, by time: a wait that has not been satisfied after
// DSA_WAIT_BUDGET_NS gives up.  When the bound runs out, or another thread of the CTA already gave
// up, the wait returns false; the caller records a status code and the CTA drains to its normal
// exit (TMEM is freed there).  Nothing spins forever and nothing traps.
#ifndef DSA_WAIT_LIMIT
#define DSA_WAIT_LIMIT (1u << 24)      // iteration bound of the polling loops that are not mbarrier waits
#endif
#ifndef DSA_WAIT_HINT_NS
#define DSA_WAIT_HINT_NS 20000u        // one parked try_wait
#endif
#ifndef DSA_WAIT_TRIES
#define DSA_WAIT_TRIES (1u << 28)      // the last bound of warp_wait_short: more than two seconds even if a try came back at once
#endif
#ifndef DSA_WAIT_BUDGET_NS
#define DSA_WAIT_BUDGET_NS 2000000000ull
#endif
__device__ __forceinline__ bool mbar_wait_budget(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint64_t budget_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
#pragma unroll 1
    for (uint32_t it = 0; it < DSA_WAIT_LIMIT; ++it) {
        if (mbar_try_wait_hint(bar, parity, DSA_WAIT_HINT_NS)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > budget_ns) break;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return mbar_wait_budget(bar, parity, abort_flag, DSA_WAIT_BUDGET_NS);
}

// After a wait has given up, copies and MMAs issued before it may still be on their way into shared memory and TMEM.  Nothing waits
// for them any more, so the CTA gives them time to land before it gives that memory back: they end by themselves within microseconds.
#ifndef DSA_SETTLE_NS
#define DSA_SETTLE_NS 200000ull
#endif
__device__ __forceinline__ void settle_in_flight() {
    const uint64_t t0 = global_ns();
#pragma unroll 1
    for (uint32_t it = 0; it < DSA_WAIT_LIMIT && global_ns() - t0 < DSA_SETTLE_NS; ++it) {
    }
}

// Warp-uniform forms for warps that run converged code (shuffles, tcgen05.ld/st) after a wait:
// either every lane saw the phase complete or the whole warp gives up together.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// The same in few instructions, for code whose size counts (seven warps of a scheduler on five different loops miss the instruction
// cache): these end by the abort flag, which a warp of the CTA that waits by time for what the others bring (warp_wait) raises after two seconds,
// and by themselves after DSA_WAIT_TRIES.  (A time in each of them: 128 sequences of 2 x 16 heads 142 -> 149 us.)
__device__ __forceinline__ bool mbar_try_wait_all(uint32_t bar, uint32_t parity) {   // parked as above; what the whole warp has seen
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "vote.sync.all.pred q, p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(DSA_WAIT_HINT_NS)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool warp_wait_short(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
    for (uint32_t n = 0; !mbar_try_wait_all(bar, parity); ++n) {
        if (*abort_flag) return false;
        if (n > DSA_WAIT_TRIES) {
            *abort_flag = 1;
            return false;
        }
    }
    return true;
}

// Three barriers at once: none can leave its phase before this warp has gone on.
__device__ __forceinline__ bool warp_wait_short3(uint32_t bar_a, uint32_t parity_a, uint32_t bar_b, uint32_t parity_b, uint32_t bar_c, uint32_t parity_c,
                                                 volatile int* abort_flag) {
    uint32_t ok;
#pragma unroll 1
    for (uint32_t n = 0;; ++n) {
        asm volatile(
            "{\n\t.reg .pred p, q, r;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %7;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4, %7;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 r, [%5], %6, %7;\n\t"
            "and.pred p, p, q;\n\t"
            "and.pred p, p, r;\n\t"
            "vote.sync.all.pred q, p, 0xffffffff;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(ok)
            : "r"(bar_a), "r"(parity_a), "r"(bar_b), "r"(parity_b), "r"(bar_c), "r"(parity_c), "r"(DSA_WAIT_HINT_NS)
            : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
        if (n > DSA_WAIT_TRIES) {
            *abort_flag = 1;
            return false;
        }
    }
}

// Two barriers at once: neither can leave its phase before this warp has gone on.
__device__ __forceinline__ bool warp_wait_short2(uint32_t bar_a, uint32_t parity_a, uint32_t bar_b, uint32_t parity_b, volatile int* abort_flag) {
    uint32_t ok;
#pragma unroll 1
    for (uint32_t n = 0;; ++n) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %5;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4, %5;\n\t"
            "and.pred p, p, q;\n\t"
            "vote.sync.all.pred q, p, 0xffffffff;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(ok)
            : "r"(bar_a), "r"(parity_a), "r"(bar_b), "r"(parity_b), "r"(DSA_WAIT_HINT_NS)
            : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
        if (n > DSA_WAIT_TRIES) {
            *abort_flag = 1;
            return false;
        }
    }
}

// Programmatic dependent launch: blocks until the kernels this one depends on have completed and their
// writes are visible (a no-op when the kernel was launched without the attribute).
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// 16-byte read-only global load that does not allocate in L1 (a gathered row is read once per SM).
__device__ __forceinline__ uint4 ldg_stream_16(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// 32-byte global store (sm_100).
__device__ __forceinline__ void stg_256(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f, uint32_t g, uint32_t h) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d), "r"(e), "r"(f), "r"(g), "r"(h)
                 : "memory");
}

// The same for addresses that may be aligned to 16 bytes only; kMaybe = false: the caller knows that they are not.
template <bool kMaybe>
__device__ __forceinline__ void stg_32(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f, uint32_t g, uint32_t h, bool wide) {
    if (!kMaybe || wide) {
        stg_256(p, a, b, c, d, e, f, g, h);
    } else {
        reinterpret_cast<uint4*>(p)[0] = make_uint4(a, b, c, d);
        reinterpret_cast<uint4*>(p)[1] = make_uint4(e, f, g, h);
    }
}

// ------------------------------------------------------------------ thread-block cluster
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cta address of this CTA -> shared::cluster address of the same offset in CTA `rank`
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t caddr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(caddr), "r"(v) : "memory");
}
// Asynchronous 16-byte store into another CTA's shared memory; its arrival is counted (in bytes)
// on an mbarrier of that CTA, so the receiver needs no fence from the sender.
__device__ __forceinline__ void st_async_b32x4(uint32_t caddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t cbar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(caddr),
                 "r"(a), "r"(b), "r"(c), "r"(d), "r"(cbar)
                 : "memory");
}
__device__ __forceinline__ void st_async_u32(uint32_t caddr, uint32_t v, uint32_t cbar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(caddr), "r"(v), "r"(cbar)
                 : "memory");
}
// arrive on an mbarrier of another CTA of the cluster; releases this thread's earlier writes
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t caddr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(caddr) : "memory");
}
// The same at CTA scope: what it orders must already be visible where it is needed - TMEM accesses before a
// tcgen05.fence::before_thread_sync, shared memory made visible to the async proxy by fence.proxy.async - and a release at
// cluster scope, which waits for every earlier write of the thread, is then not paid for.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t caddr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(caddr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_try_wait_cluster_hint(uint32_t bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
// bounded like mbar_wait; acquires at cluster scope (the data was written by the peer CTA)
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const uint64_t t0 = global_ns();
#pragma unroll 1
    for (uint32_t it = 0; it < DSA_WAIT_LIMIT; ++it) {
        if (mbar_try_wait_cluster_hint(bar, parity, DSA_WAIT_HINT_NS)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > DSA_WAIT_BUDGET_NS) break;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ bool warp_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait_cluster(bar, parity, abort_flag));
}
// Both CTAs of the cluster arrive and wait (start-up after barrier init, and before exit so that
// no CTA leaves while its peer can still write into its shared memory).
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// generic-proxy writes to shared memory -> visible to the async proxy (TMA, tcgen05.mma operands)
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ------------------------------------------------------------------ TMA
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// 3-D tiled load (global -> this CTA's shared memory), completion on an mbarrier.
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        :
        : "r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// Asks for `bytes` bytes (a multiple of 16, 16-byte aligned) to be brought into L2.
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// 4-byte asynchronous copy global -> shared (src_bytes = 0 writes zeros without reading), and an
// mbarrier arrival that happens when all earlier cp.async of this thread have landed (it counts
// against the barrier's expected arrivals).
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ uint4 lds_16(uint32_t src) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(src) : "memory");
    return v;
}
__device__ __forceinline__ void sts_16(uint32_t dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void cp_async_mbar_arrive_noinc(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Register budget of the executing warpgroup (all four warps execute the same one).
template <int N> __device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N> __device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// ------------------------------------------------------------------ TMEM
// Executed by one full warp.  Writes the allocated base address to *smem_dst.
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32-bit, N consecutive columns: thread t of the warp gets lane (base lane + t).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        :
        : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
          "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]),
          "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        :
        : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :
                 : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// N consecutive columns, N in {8, 16, 32}
template <int N> __device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t (&r)[N]);
template <> __device__ __forceinline__ void tmem_ld_n<8>(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8(taddr, r); }
template <> __device__ __forceinline__ void tmem_ld_n<16>(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
template <> __device__ __forceinline__ void tmem_ld_n<32>(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }
template <int N> __device__ __forceinline__ void tmem_st_n(uint32_t taddr, const uint32_t (&r)[N]);
template <> __device__ __forceinline__ void tmem_st_n<8>(uint32_t taddr, const uint32_t (&r)[8]) { tmem_st8(taddr, r); }
template <> __device__ __forceinline__ void tmem_st_n<16>(uint32_t taddr, const uint32_t (&r)[16]) { tmem_st16(taddr, r); }
template <> __device__ __forceinline__ void tmem_st_n<32>(uint32_t taddr, const uint32_t (&r)[32]) { tmem_st32(taddr, r); }

// Ties values that tcgen05.ld delivers to the wait before this, where other work stands between the load and the wait.
__device__ __forceinline__ void tmem_loaded(uint32_t (&r)[16]) {
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]),
                 "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
}

// ------------------------------------------------------------------ tcgen05.mma
// Shared-memory matrix descriptor, 128-byte swizzle: start address, leading / stride byte
// offsets (all >> 4), descriptor version 1 (bits 46-47), swizzle mode 2 = 128B (bits 61-63).
//   K-major operand  (rows of 128 B = 64 bf16 along K, 8-row groups 1024 B apart):
//       SBO = 1024, LBO unused; step 16 elements along K = +32 bytes on the start address.
//   MN-major operand (rows of 128 B = 64 bf16 along MN, one K index per row, 8-row groups
//       1024 B apart): SBO = 1024, LBO = distance between consecutive 64-element MN blocks;
//       step 16 along K = +16 rows = +2048 bytes on the start address.
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

// MN-major operand whose rows hold N = 16 or 32 bf16 (one K index per row): 32- or 64-byte swizzle (mode 6 or 4), groups of
// eight rows follow one another.  There is a single MN block, so the leading offset is not used.
template <int N>
__device__ __forceinline__ uint64_t make_smem_desc_mn_narrow(uint32_t saddr, uint32_t lbo_bytes) {
    static_assert(N == 16 || N == 32, "32- or 64-byte rows");
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((8 * 2 * N) >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(N == 16 ? 6 : 4) << 61;
    return d;
}

// Instruction descriptor for kind::f16 with bf16 A and B, fp32 accumulate.
//   bits 4-5 D format (1 = f32), 7-9 A format (1 = bf16), 10-12 B format (1 = bf16),
//   bit 15 A major (0 = K), bit 16 B major (0 = K, 1 = MN), bits 17-22 N >> 3, bits 24-28 M >> 4.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) |
           (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}
// The same for f16 A and B, and for kind::f8f6f4 with e4m3 A and B (both K-major).
__host__ __device__ constexpr uint32_t make_idesc_f16(int M, int N, bool b_mn_major) { return make_idesc_bf16(M, N, b_mn_major) & ~((1u << 7) | (1u << 10)); }
__host__ __device__ constexpr uint32_t make_idesc_e4m3(int M, int N) { return make_idesc_f16(M, N, false); }
constexpr uint32_t kIdescAE5m2 = 1u << 7;          // of kind::f8f6f4: A is e5m2
constexpr uint32_t kIdescATransposed = 1u << 15;   // A is MN-major

// D[tmem] (+)= A * B, A in shared memory (ss) or TMEM (ts), B in shared memory; accumulate == 0 overwrites D.
// Forms for an issuing warp that stays converged: every lane executes the call, the lane whose
// `elected` is non-zero issues.  Descriptors then stay warp-uniform values.
__device__ __forceinline__ void umma_ss_el(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
        : "memory");
}
// Four MMAs of one 64-column block (K = 16 each) in one piece of assembly: the election predicate is
// set up once and the operands of the steps differ by immediates (A: +8 TMEM columns or +32 bytes,
// B: +32 bytes = +2 in descriptor units), so a step costs the issuing warp three instructions instead
// of eight.  `first_accumulates` = 0 lets the first step overwrite D.  b_lo / b_hi (a_lo / a_hi): the two
// halves of the shared-memory descriptor; adding to the low half cannot carry out of its 14-bit address
// field because shared memory ends below 2^18 bytes.
__device__ __forceinline__ void umma_ss_x4_el(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                              uint32_t idesc, uint32_t first_accumulates, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q, pt, pf;\n\t.reg .b32 la, lb;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 q, %7, 0;\n\t"
        "setp.ne.b32 pf, %6, 0;\n\t"
        "setp.eq.b32 pt, %7, %7;\n\t"
        "mov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %5, pf;\n\t"
        "add.u32 la, %1, 2;\n\tadd.u32 lb, %3, 2;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %5, pt;\n\t"
        "add.u32 la, %1, 4;\n\tadd.u32 lb, %3, 4;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %5, pt;\n\t"
        "add.u32 la, %1, 6;\n\tadd.u32 lb, %3, 6;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %5, pt;\n\t}"
        :
        : "r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first_accumulates), "r"(elected)
        : "memory");
}
// All tcgen05.mma the elected lane has issued arrive (once) on the mbarrier when complete.
__device__ __forceinline__ void tc_commit_el(uint32_t bar, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        :
        : "r"(bar), "r"(elected)
        : "memory");
}

// ------------------------------------------------------------------ the pair forms (cta_group::2)
// One instruction over the tensor cores of both CTAs of a cluster, issued by the even one: each CTA's shared memory holds
// its half of A's rows and its half of B's N rows at the same offsets, and each CTA's TMEM gets its half of D's rows.
// With M = 128 a CTA has 64 rows: TMEM lanes 0-63 hold columns [0, N / 2) of them and lanes 64-127 columns [N / 2, N), so
// all lanes work and the rate is the full one; an A operand in TMEM has its 64 rows in both halves of the lanes.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {   // one warp of either CTA
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// All pair MMAs this thread has issued arrive, when complete, on the barrier at this offset in both CTAs.
__device__ __forceinline__ void tc_commit_pair_el(uint32_t bar, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b16 m;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "mov.b16 m, 3;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}"
        :
        : "r"(bar), "r"(elected)
        : "memory");
}
__device__ __forceinline__ void umma_pair_ss_el(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
        : "memory");
}
// four K = 16 steps of one 64-column block, as umma_ss_x4_el
__device__ __forceinline__ void umma_pair_ts_x4_el(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                                   uint32_t first_accumulates, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q, pt, pf;\n\t.reg .b32 a, l;\n\t.reg .b64 bd;\n\t"
        "setp.ne.b32 q, %6, 0;\n\t"
        "setp.ne.b32 pf, %5, 0;\n\t"
        "setp.eq.b32 pt, %6, %6;\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], bd, %4, pf;\n\t"
        "add.u32 a, %1, 8;\n\tadd.u32 l, %2, 2;\n\tmov.b64 bd, {l, %3};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a], bd, %4, pt;\n\t"
        "add.u32 a, %1, 16;\n\tadd.u32 l, %2, 4;\n\tmov.b64 bd, {l, %3};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a], bd, %4, pt;\n\t"
        "add.u32 a, %1, 24;\n\tadd.u32 l, %2, 6;\n\tmov.b64 bd, {l, %3};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a], bd, %4, pt;\n\t}"
        :
        : "r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first_accumulates), "r"(elected)
        : "memory");
}
__device__ __forceinline__ void umma_pair_ss_x4_el(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                                   uint32_t idesc, uint32_t first_accumulates, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q, pt, pf;\n\t.reg .b32 la, lb;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 q, %7, 0;\n\t"
        "setp.ne.b32 pf, %6, 0;\n\t"
        "setp.eq.b32 pt, %7, %7;\n\t"
        "mov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %5, pf;\n\t"
        "add.u32 la, %1, 2;\n\tadd.u32 lb, %3, 2;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %5, pt;\n\t"
        "add.u32 la, %1, 4;\n\tadd.u32 lb, %3, 4;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %5, pt;\n\t"
        "add.u32 la, %1, 6;\n\tadd.u32 lb, %3, 6;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %5, pt;\n\t}"
        :
        : "r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first_accumulates), "r"(elected)
        : "memory");
}
// four K = 32 steps of one block of 128 e4m3 columns
__device__ __forceinline__ void umma_pair_f8_ss_x4_el(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                                   uint32_t idesc, uint32_t first_accumulates, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q, pt, pf;\n\t.reg .b32 la, lb;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 q, %7, 0;\n\t"
        "setp.ne.b32 pf, %6, 0;\n\t"
        "setp.eq.b32 pt, %7, %7;\n\t"
        "mov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], ad, bd, %5, pf;\n\t"
        "add.u32 la, %1, 2;\n\tadd.u32 lb, %3, 2;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], ad, bd, %5, pt;\n\t"
        "add.u32 la, %1, 4;\n\tadd.u32 lb, %3, 4;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], ad, bd, %5, pt;\n\t"
        "add.u32 la, %1, 6;\n\tadd.u32 lb, %3, 6;\n\tmov.b64 ad, {la, %2};\n\tmov.b64 bd, {lb, %4};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], ad, bd, %5, pt;\n\t}"
        :
        : "r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first_accumulates), "r"(elected)
        : "memory");
}

// ------------------------------------------------------------------ small helpers
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t pack_bf16x2_from2(uint64_t v);   // below

// Two fp32 values in one 64-bit register and the two-wide fp32 arithmetic of sm_100 on them.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t pack2u(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ uint32_t pack_bf16x2_from2(uint64_t v) {
    float lo, hi;
    unpack2(v, lo, hi);
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// D += A B of one warp, bf16 operands: A 16 x 16, B 16 x 8
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// e4m3 and e5m2 (saturating, to nearest even) and f16, two at a time: element 0 in the low half
__device__ __forceinline__ uint32_t f16x2_to_e4m3x2(uint32_t v) {   // in the low half
    uint32_t r;
    asm("{\n\t.reg .b16 t;\n\tcvt.rn.satfinite.e4m3x2.f16x2 t, %1;\n\tmov.b32 %0, {t, 0};\n\t}" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t f16x2_to_e5m2x2(uint32_t v) {
    uint32_t r;
    asm("{\n\t.reg .b16 t;\n\tcvt.rn.satfinite.e5m2x2.f16x2 t, %1;\n\tmov.b32 %0, {t, 0};\n\t}" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t sub_f16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t e4m3x2_to_f16x2(uint32_t v) {   // the two low bytes; exact
    uint32_t r;
    asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, a;\n\t}" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void unpack_f16x2(uint32_t v, float& lo, float& hi) {
    asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.f32.f16 %0, a;\n\tcvt.f32.f16 %1, b;\n\t}" : "=f"(lo), "=f"(hi) : "r"(v));
}
__device__ __forceinline__ uint32_t mul_f16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// 2^n in f16, n from -24 to 15
__device__ __forceinline__ uint32_t pow2_f16(int n) { return n >= -14 ? static_cast<uint32_t>(n + 15) << 10 : 1u << (n + 24); }
// s = hi + lo in f16, hi in the low half: 22 significant bits from 2^-3 on, 2^-25 off below
__device__ __forceinline__ uint32_t split_f16(float s) {
    const uint32_t hi = pack_f16x2(s, s);
    float a, b;
    unpack_f16x2(hi, a, b);
    return pack_f16x2(a, s - a);
}
// v (hi + lo): the product with lo is small, so the sum is rounded once for all that matters
__device__ __forceinline__ uint32_t scale_f16x2(uint32_t v, uint32_t hi, uint32_t lo) {
    uint32_t r;
    asm("{\n\t.reg .b32 t;\n\tmul.rn.f16x2 t, %1, %3;\n\tfma.rn.f16x2 %0, %1, %2, t;\n\t}" : "=r"(r) : "r"(v), "r"(hi), "r"(lo));
    return r;
}
// two bf16 times a power of two
__device__ __forceinline__ uint32_t scale_bf16x2(uint32_t v, float mul) { return pack_bf16x2(__uint_as_float(v << 16) * mul, __uint_as_float(v & 0xFFFF0000u) * mul); }
__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

}  // namespace dsa
