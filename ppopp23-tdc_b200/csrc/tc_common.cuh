// What every tensor-core kernel of the library is made of: mbarriers with bounded waits, bulk copies, the shared-memory
// matrix descriptor of the un-swizzled K-major operand layout, the MMA instruction and its descriptor, reads of tensor
// memory, division by multiplication, and the power-of-two range scaling of fp16 operands.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tdc_tc {

constexpr int M_TILE   = 128;   // positions per CTA = MMA M

constexpr int CB       = 8;     // 4-byte words per operand row and K step (32 bytes): 8 TF32 channels, or 16 fp16 channels

// Division of a non-negative number below 2^31 by a fixed divisor as one widening multiply and a shift: the index
// arithmetic of the loaders, the producer and the epilogue divides by the row pitch, the positions per image and the
// number of output-channel blocks once or more per tile and work item, and an integer division is 20 (32-bit) to
// 100 (64-bit) dependent instructions of a single warp.  mul = floor(2^(31+s) / d) + 1 with 2^(s-1) < d <= 2^s:
// n * mul >> (31 + s) == n / d for every 0 <= n < 2^31 (the excess mul * d - 2^(31+s) is at most d <= 2^s, so the
// product overshoots n / d by less than 1 / d).
struct FastDiv { uint32_t mul, shift; };

inline FastDiv fastdiv_make(uint32_t d) {
    uint32_t s = 0;
    while ((1ull << s) < d) ++s;
    FastDiv f;
    f.mul = (uint32_t)(((1ull << (31 + s)) / d) + 1ull);
    f.shift = 31 + s;
    return f;
}

__host__ __device__ __forceinline__ uint32_t fastdiv(uint32_t n, FastDiv f) { return (uint32_t)(((unsigned long long)n * f.mul) >> f.shift); }

constexpr int ABSMAX_SLOTS = 1024;

// The power of two that brings a magnitude m just under 2^target; 1 for a zero or non-finite m.
__host__ __device__ __forceinline__ float range_scale(float m, int target = 14) {
    if (!(m > 0.f) || !(m < 3.0e38f)) return 1.f;
    int e;
    frexpf(m, &e);                                  // m = f * 2^e, 0.5 <= f < 1
    int k = target - e;
    k = k < -60 ? -60 : (k > 60 ? 60 : k);
    return ldexpf(1.f, k);
}

// The larger of two values; a NaN wins.  fmaxf drops it: an input that left fp16's range arrives in an epilogue as inf - inf, and a
// ReLU or a maximum by fmaxf would make it a zero that nothing reports.
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Bounded wait: true when the phase with `parity` has completed, false after ~1 s.
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try(bar, parity)) return true;          // the common case costs no clock read
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try(bar, parity)) return true;
        if (clock64() - t0 > 2000000000ll) return false;
    }
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Shared-memory matrix descriptor: K-major, no swizzle.  lbo = bytes between the two core
// matrices of one K step (channels 0-3 / 4-7), sbo = bytes between 8-row groups.
__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= 1ull << 46;                 // descriptor version of sm_100
    return d;                        // layout type 0 (no swizzle), base offset 0
}

template <bool F16>
__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if constexpr (F16)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 32 consecutive columns of this warp's 32 tensor-memory lanes -> 32 registers per thread.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

// ... and 16 of them (the persistent kernel's epilogue works in half chunks: it has fewer registers per thread).
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// One lane of a converged warp, chosen by the hardware.  The MMA issue loops run warp-uniform
// (every lane waits on the barriers and computes the same descriptors) and only the MMA and
// commit instructions sit under this predicate: operands the compiler can prove warp-uniform
// stay in uniform registers, which is what the tensor-core instructions read.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred != 0;
}

// Instruction descriptor: D fp32, A and B tf32 (format 2) or fp16 (format 0), both K-major, M = 128, N = n.
template <bool F16>
__device__ __forceinline__ uint32_t make_idesc(int n) {
    const uint32_t fmt = F16 ? 0u : 2u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(M_TILE >> 4) << 24);
}

}  // namespace tdc_tc
