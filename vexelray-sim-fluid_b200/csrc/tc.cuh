// tc.cuh -- tcgen05, tensor-memory and mbarrier helpers shared by the network's tensor-core kernels.
#pragma once

#include "common.cuh"

namespace vf {

constexpr int TC_SPINS = 1 << 22;   // mbarrier polls before a role gives up

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// K-major operand in the 32-byte swizzle: 8-row groups 256 bytes apart, version 1, layout type 6.
__device__ __forceinline__ uint64_t desc_sw32(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46) |
           (6ull << 61);
}

// K-major operand without swizzle: 8-row core matrices of 16-byte rows, LBO between the two k halves, SBO between
// 8-row groups.
__device__ __forceinline__ uint64_t desc_plain(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)((lbo >> 4) & 0x3fff) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3fff) << 32) | (1ull << 46);
}

// K-major operands in the 64-byte and 128-byte swizzles (8-row groups 512 and 1024 bytes apart).
__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46) |
           (4ull << 61);
}

__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

__host__ __device__ constexpr uint32_t sw32(uint32_t r, uint32_t h) { return r * 32 + ((h ^ ((r >> 2) & 1)) << 4); }

// kind::f16 instruction descriptor: fp32 accumulate, bf16 A and B, both K-major, or both MN-major.
__host__ __device__ constexpr uint32_t idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__host__ __device__ constexpr uint32_t idesc_mn(int m, int n) { return idesc(m, n) | (1u << 15) | (1u << 16); }

// MN-major operands. In the 64-byte swizzle: blocks of 32 consecutive M (or N) elements, 64 bytes, `block` bytes apart;
// within a block 8 k rows of 64 bytes, the next 8 k rows 512 bytes on. Without swizzle: blocks of 8 elements, 16 bytes,
// `block` bytes apart; 8 k rows of 16 bytes, the next 8 k rows 128 bytes on.
__device__ __forceinline__ uint64_t desc_mn64(uint32_t addr, uint32_t block) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)((block >> 4) & 0x3fff) << 16) | ((uint64_t)(512 >> 4) << 32) |
           (1ull << 46) | (4ull << 61);
}

__device__ __forceinline__ uint64_t desc_mn16(uint32_t addr, uint32_t block) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)((block >> 4) & 0x3fff) << 32) |
           (1ull << 46);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for the phase of `parity`; on expiry sets the status and the CTA's abort flag.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_cta, uint32_t* status) {
    for (int spin = 0; spin < TC_SPINS; spin++) {
        if (mbar_try(bar, parity)) return true;
        if ((spin & 1023) == 1023 && *abort_cta) return false;
    }
    set_status(status, ST_TIMEOUT);
    *abort_cta = 1;
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// D += A B (the accumulators start at zero: the epilogue clears what it reads).
__device__ __forceinline__ void umma_acc(uint32_t tmem, uint64_t a, uint64_t b, uint32_t id) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(id));
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// CW consecutive fp32 columns of this thread's tensor-memory lane, without the wait (tmem_wait_ld after a batch).
template <int CW>
__device__ __forceinline__ void tmem_ld_nowait(uint32_t taddr, uint32_t (&r)[CW]) {
    if constexpr (CW == 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
            "%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr));
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
    }
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

template <int CW>
__device__ __forceinline__ void tmem_zero_cols(uint32_t taddr) {
    const uint32_t z = 0;
    if constexpr (CW == 16) {
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
            "%1};" ::"r"(taddr),
            "r"(z)
            : "memory");
    } else {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(z)
                     : "memory");
    }
}

// 32 bytes of global memory in one access (a whole sector a thread); p is 32-byte aligned.
__device__ __forceinline__ void st_global_32(void* p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ void ld_global_32(uint32_t (&v)[8], const void* p) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
}

}  // namespace vf
