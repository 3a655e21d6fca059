// Warp-level bfloat16 products (mma.sync m16n8k16, float sums) and float operands as sums of three bfloat16 numbers.
//
// A float is the sum of three bfloat16 numbers up to its last bit (8 bits each of 24), so a product whose one operand
// is bfloat16 and whose other one is float is three products of bfloat16 operands, each exact in float.
#pragma once

#include "common.cuh"

namespace janis {

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldmatrix4(uint32_t (&v)[4], uint32_t shared) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(shared) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&v)[4], uint32_t shared) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(shared) : "memory");
}

// (x, y) as three pairs of bfloat16 numbers: hi the nearest, mid the nearest to what is left, lo the rest
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    x -= __uint_as_float(hi << 16);
    y -= __uint_as_float(hi & 0xffff0000u);
    const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
    mid = *reinterpret_cast<const uint32_t*>(&m);
    x -= __uint_as_float(mid << 16);
    y -= __uint_as_float(mid & 0xffff0000u);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x, y);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Whether four pairs of bfloat16 numbers hold no infinity and no NaN: an exponent of ones carries into the sign's place
__device__ __forceinline__ bool all_finite(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t m = 0x7f807f80u, one = 0x00800080u;
    return ((((a & m) + one) | ((b & m) + one) | ((c & m) + one) | ((d & m) + one)) & 0x80008000u) == 0;
}

// 16 bytes from global to shared memory; zeros where !ok
__device__ __forceinline__ void copy16_or_zero(uint32_t shared, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(shared), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

}  // namespace janis
