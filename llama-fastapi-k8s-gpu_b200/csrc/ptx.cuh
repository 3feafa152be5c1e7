// Thin inline-PTX wrappers used by the sm_100a kernels: mbarrier, 1-D TMA bulk copies
// (cp.async.bulk), programmatic dependent launch, warp helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b2 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// make mbarrier.init visible to the async (TMA) proxy
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Spin with a watchdog: if a barrier never completes (a protocol bug) the kernel records `code`
// in the host-visible error word and carries on with garbage instead of hanging the GPU; every
// engine call checks that word after it synchronises and fails loudly.
// try_wait already suspends the thread for a hardware time slice.
__device__ __forceinline__ void mbar_give_up(uint32_t parity, unsigned int* err, unsigned int code, unsigned int info) {
    if (err) {          // plain stores: the words live in host memory. [0] code [1] block [2] thread [3] info [4] parity
        volatile unsigned int* e = reinterpret_cast<volatile unsigned int*>(err);
        if (e[0] == 0) { e[1] = blockIdx.x; e[2] = threadIdx.x; e[3] = info; e[4] = parity; e[0] = code; }
    }
}
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, unsigned int* err, unsigned int code,
                                          unsigned int info = 0) {
    uint32_t spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (++spins > (1u << 22)) { mbar_give_up(parity, err, code, info); return; }
    }
}
// The wait of a loop that a whole warp runs while one lane issues copies or products. The lanes leave it together: what is issued next
// lets the barrier move on, and a lane still waiting when it has moved two phases on would read the parity of the phase before its own.
__device__ __forceinline__ void mbar_wait_warp(uint64_t* bar, uint32_t parity, unsigned int* err, unsigned int code, unsigned int info = 0) {
    mbar_wait(bar, parity, err, code, info);
    __syncwarp();
}
// 1-D bulk async copy global -> shared, completion signalled on an mbarrier (complete_tx).
// dst and src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// 2-D tensor copy global -> shared (box of the tensor map at element coordinates {c0, c1}), completion on an mbarrier
__device__ __forceinline__ void tma_load_2d(void* dst, const void* tmap, int c0, int c1, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(tmap), "r"(c0), "r"(c1), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const void* tmap, int c0, int c1, int c2, int c3, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(smem_u32(dst)), "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar)) : "memory");
}
// Programmatic dependent launch (PDL): `launch` lets the next kernel in the stream start
// its prologue (weight prefetch) early; `wait` blocks until the previous kernel has fully
// completed and its global writes are visible.
__device__ __forceinline__ void griddep_launch() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void griddep_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// one lane of a converged warp, the same one every time
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// ---- thread-block clusters: all threads of all CTAs meet (ordering nothing but what a fence before it orders); an address in CTA `rank`'s shared memory
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// the same with what was written to shared memory before it visible to the cluster behind it
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_address(uint32_t own, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(own), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 cluster_load4(uint32_t address) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(address) : "memory");
    return v;
}
__device__ __forceinline__ float2 cluster_load2(uint32_t address) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(address) : "memory");
    return v;
}
// an arrival at another CTA's barrier: what its thread has done and seen before is before what whoever waits with mbar_wait_cluster does next
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// the wait for a barrier that another CTA arrives at, or counts bytes of (st_async_16)
__device__ __forceinline__ void mbar_wait_cluster(uint64_t* bar, uint32_t parity, unsigned int* err, unsigned int code, unsigned int info = 0) {
    for (uint32_t spins = 0, ok = 0; !ok;) {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (!ok && ++spins > (1u << 22)) { mbar_give_up(parity, err, code, info); return; }
    }
}
// 16 bytes into another CTA's shared memory, counted by a barrier there
__device__ __forceinline__ void st_async_16(uint32_t to, const uint32_t* v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(to), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar) : "memory");
}

// timeline records (debugging aid, B2_TIMELINE=1): slot 0 keeps the earliest time, the others the latest
__device__ __forceinline__ void tl_stamp(unsigned long long* tl, int slot) {
    if (!tl) return;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (slot == 0) atomicMin(tl, t); else atomicMax(tl + slot, t);
}

// two f32 in one register pair: one instruction for two multiply-adds
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ float rcp_approx(float y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return r;
}
// z / (1 + exp(w)) without a branch (a division has one): the approximate quotient and one correction by its remainder (a step of Newton's
// method); within two units of the last place of expf's denominator. The reciprocal is taken of a quarter: past 2^126 it would be flushed to 0. Past
// the largest number (w > 88.7) the quotient is 0. NaN and an infinite z come out as from a division.
__device__ __forceinline__ float over_one_plus_exp(float z, float w) {
    const float y = 1.f + expf(w), r = 0.25f * rcp_approx(0.25f * y), v = z * r, q = fmaf(fmaf(-y, v, z), r, v);
    return y == 1.f ? z : y == INFINITY ? 0.f * z : q;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

}  // namespace b2
