// tbl_sync.cuh -- device-side synchronisation primitives of the sweep
// kernels: acquire/release words, bounded mbarrier waits, st.async pushes into
// another CTA's shared memory and cluster barriers.
#pragma once
#include <cuda_runtime.h>

namespace tbl {

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Programmatic dependent launch: a kernel started with launch_dependent
// (tbl_internal.cuh) begins when the blocks of the kernel in front of it have
// left, before its end has been processed and its writes are all visible.  Every
// thread executes dependent_wait before it touches what other kernels write; the
// kernel before the one in front has ended by then, because that one has waited
// for it.  (No kernel lets the next one begin earlier than that: its blocks came
// to lie two to an SM, beside the last of a sweep, 303 -> 350 ms a mixed step at
// 768 x 194 x 144, for 1% at 32 x 18 x 24.)
__device__ __forceinline__ void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the same, p being read afterwards only (also where the compiler takes what p
// points to for constant)
template <typename T>
__device__ __forceinline__ void dependent_wait(T*& p) {
    asm volatile("griddepcontrol.wait;" : "+l"(p)::"memory");
}

constexpr long long SPIN_LIMIT = 1LL << 24;  // ~1 s of polling memory, then the wait gives up
constexpr long long MBAR_LIMIT = 1LL << 18;  // ~1 s at an mbarrier: a try_wait that fails takes 3.75 us

constexpr long long XLINGER = 1LL << 27;  // bounded wait for the partner at the end

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned mapa_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(unsigned raddr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(raddr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Whether the phase of the given parity has completed (no waiting).
__device__ __forceinline__ bool mbar_test(unsigned long long* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for the completion of the phase of the given parity.  (A limit by
// the clock instead of a count cost the sweeps 1.5%.)
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity) {
    long long spins = 0;
    while (!mbar_try_wait(b, parity)) {
        if (++spins > MBAR_LIMIT) return false;
    }
    return true;
}
// One lane's CH values of a step into the consumer's ring slot.
template <int CH>
__device__ __forceinline__ void xpush(unsigned rd, unsigned rb, const double (&v)[CH]) {
#pragma unroll
    for (int b = 0; b < CH / 2; ++b)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(
                         rd + 16u * b),
                     "d"(v[2 * b]), "d"(v[2 * b + 1]), "r"(rb)
                     : "memory");
}
template <int CH>
__device__ __forceinline__ void xpush(unsigned rd, unsigned rb, const float (&v)[CH]) {
#pragma unroll
    for (int b = 0; b < CH / 4; ++b)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                         rd + 16u * b),
                     "f"(v[4 * b]), "f"(v[4 * b + 1]), "f"(v[4 * b + 2]), "f"(v[4 * b + 3]), "r"(rb)
                     : "memory");
}
__device__ __forceinline__ void st_remote_s32(unsigned raddr, int v) {
    asm volatile("st.relaxed.cluster.shared::cluster.s32 [%0], %1;" ::"r"(raddr), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed_cluster(const int* p) {
    int v;
    asm volatile("ld.relaxed.cluster.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}
// Bounded wait until a word of this CTA (written by the partner CTA) is non-zero.
__device__ __forceinline__ int wait_word(const int* p) {
    for (long long spins = 0; spins < XLINGER; ++spins) {
        const int v = ld_relaxed_cluster(p);
        if (v) return v;
        if (spins > 64) __nanosleep(64);
    }
    return 0;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace tbl
