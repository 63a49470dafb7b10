// sweep_common.cuh -- device helpers shared by the Metropolis sweep kernels
// (sampler.cu, sampler_screen.cu): shared-memory loads, configuration bits,
// chain start and finish, the FP32 acceptance sum.
#pragma once

#include "common.cuh"
#include "sampler.cuh"

namespace rbmnqs {

// Shared-memory loads by 32-bit shared address: the gather tables may also
// live in global memory, so their generic pointers would otherwise compile
// to generic loads.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float2 lds_f2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
// N / 4 words from a 4 N-byte aligned shared address (N = 4, 8, 16)
template <int N> __device__ __forceinline__ void lds_words(uint32_t addr, uint32_t (&w)[N / 4]) {
    if constexpr (N == 16) {
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
    } else if constexpr (N == 8) {
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr));
    } else {
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[0]) : "r"(addr));
    }
}

// word i of the configuration with constant indices only (a runtime index
// would place the array in local memory)
__device__ __forceinline__ uint32_t spin_word(const uint32_t sp[4], int i) {
    return i == 0 ? sp[0] : (i == 1 ? sp[1] : (i == 2 ? sp[2] : sp[3]));
}
__device__ __forceinline__ int spin_bit(const uint32_t sp[4], int i) {
    const uint32_t w = i < 32 ? sp[0] : (i < 64 ? sp[1] : (i < 96 ? sp[2] : sp[3]));
    return (w >> (i & 31)) & 1;
}
__device__ __forceinline__ void flip_bit(uint32_t sp[4], int i) {
    const uint32_t b = 1u << (i & 31);
    if (i < 32) sp[0] ^= b;
    else if (i < 64) sp[1] ^= b;
    else if (i < 96) sp[2] ^= b;
    else sp[3] ^= b;
}

// Initial configuration of a chain: Philox stream 1 bits for a fresh chain,
// else the persisted configuration.
__device__ __forceinline__ void chain_start(const SamplerArgs& a, int chain, uint2 key, uint32_t epoch, uint32_t sp[4]) {
    const int n = a.m.n;
    if (a.ctl[1] && a.sweep0 == 0) {
        const uint4 r = philox4x32(make_uint4(0, epoch, (uint32_t)chain, 1), key);
        const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const int lo = 32 * w;
            const uint32_t mask = n >= lo + 32 ? 0xffffffffu : (n > lo ? ((1u << (n - lo)) - 1) : 0u);
            sp[w] = rw[w] & mask;
        }
    } else {
#pragma unroll
        for (int w = 0; w < 4; w++) sp[w] = a.spins[4 * chain + w];
    }
}

// Proposal counter at the start of a segment: 32-aligned (proposals are
// drawn 32 at a time) and past every proposal of earlier segments (a sweep
// makes at most n proposals).
__device__ __forceinline__ uint32_t prop_base(const SamplerArgs& a) {
    return (uint32_t)a.sweep0 * (uint32_t)(32 * ((a.m.n + 31) / 32));
}
__device__ __forceinline__ int segment_sweeps(const SamplerArgs& a) {
    return a.nsweeps ? a.nsweeps : a.spc * a.step + a.warmup;
}
// sample slot of global sweep sg, or -1
__device__ __forceinline__ int sample_slot(const SamplerArgs& a, int st) {
    const int sg = a.sweep0 + st;
    if (!a.record || sg < a.warmup || (sg - a.warmup) % a.step) return -1;
    return (sg - a.warmup) / a.step;
}

__device__ __forceinline__ void chain_finish(const SamplerArgs& a, int chain, int lane, const uint32_t sp[4],
                                             uint32_t nacc, uint32_t prop) {
    if (lane < 4) a.spins[4 * chain + lane] = spin_word(sp, lane);
    if (lane == 0) {
        const uint32_t made = prop - prop_base(a);
        a.n_acc[chain] = (a.sweep0 ? a.n_acc[chain] : 0u) + nacc;
        a.n_prop[chain] = (a.sweep0 ? a.n_prop[chain] : 0u) + made;
    }
}

// MUFU operations in their flush-to-zero forms (the sweeps' ln|cosh|).
__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_ftz(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float cos_ftz(float x) {
    float y;
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Sum over the warp of the lanes' ln|cosh| differences for the acceptance
// test.  The partials are summed as fixed-point integers (2^-22 steps, one
// redux.sync instead of a five-level shuffle butterfly) when every lane's
// partial is below 16 in magnitude, which keeps the 32-lane total inside
// int32; otherwise the FP32 butterfly.  The quantisation (2.4e-7) is that of
// an FP32 sum of this size, so decisions differ from the FP64 chains only at
// ties, as with any FP32 sum.
constexpr float kFixScale = 4194304.f;  // 2^22
__device__ __forceinline__ int fix22(float v) { return __float2int_rn(v * kFixScale); }
__device__ __forceinline__ float sweep_sum(float v) {
    const int isum = __reduce_add_sync(kFull, fix22(v));
    if (__any_sync(kFull, !(fabsf(v) < 16.f))) return warp_sum(v);
    return (float)isum * (1.f / kFixScale);
}

}  // namespace rbmnqs
