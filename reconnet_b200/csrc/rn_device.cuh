// Device helpers: mbarrier + bulk (TMA, non-tensor) copies for sm_100a, and
// small numeric utilities.  Every wait is bounded (rn::kSpinLimit).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "rn_internal.h"

namespace rn {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile(
        "{\n\t.reg .b64 st;\n\t"
        "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
        "r"(bytes)
        : "memory");
}

// Returns true when the phase with the given parity has completed, false if
// the bounded spin (`limit` polls) ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit = kSpinLimit) {
    uint32_t addr = smem_u32(bar);
    for (long long it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Bulk global -> shared copy completing on an mbarrier (cp.async.bulk, no
// multicast).  dst/src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// 16-byte global -> shared copy (cp.async, L2 only); `valid` false writes 16
// zero bytes and reads nothing.  Completion: cp_async_commit / cp_async_wait.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most N of this thread's committed groups are still in flight
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Two FP32 lanes in one 64-bit register: the packed FP32 instructions of
// sm_100 do two IEEE operations per issue slot.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// round-down add (for floors against 1.5 * 2^23)
__device__ __forceinline__ f32x2 f2_add_rd(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// shared-memory load at a byte address
__device__ __forceinline__ float4 lds4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// floor(x) and frac(x) for 0 <= x < 2^22 on the FMA/ALU pipes: the integer
// part comes from rounding (x - 0.5) with a 1.5 * 2^23 bias.  At exact
// integers it may return (n-1, 1.0) instead of (n, 0.0); both evaluate the
// same prefix value because entry n-1 plus one full pixel is entry n.
__device__ __forceinline__ int floor_frac(float x, float& frac) {
    const float kBias = 12582912.0f;  // 1.5 * 2^23
    float y = (x - 0.5f) + kBias;
    int k = __float_as_int(y) - 0x4B400000;
    frac = x - (y - kBias);
    return k;
}

// Error-free split of a double into hi + lo floats.
__device__ __forceinline__ float2 split_double(double v) {
    float hi = __double2float_rn(v);
    float lo = __double2float_rn(v - (double)hi);
    return make_float2(hi, lo);
}

// 1 / d in FP64 from the FP32 reciprocal by two Newton steps (each squares the
// relative error: 1e-7, 1e-14, below FP64's own rounding), a fifth of a
// division's instructions; outside FP32's comfortable range the division.
__device__ __forceinline__ double reciprocal(double d) {
    const double a = fabs(d);
    if (!(a > 1e-30 && a < 1e30)) return 1.0 / d;
    double r = (double)__frcp_rn((float)d);
    r = fma(r, fma(-d, r, 1.0), r);
    return fma(r, fma(-d, r, 1.0), r);
}

// Inclusive prefix sum over the 32 lanes of a warp (all lanes participate).
__device__ __forceinline__ double warp_incl_scan(double v) {
    const unsigned full = 0xffffffffu;
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        double t = __shfl_up_sync(full, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

}  // namespace rn
