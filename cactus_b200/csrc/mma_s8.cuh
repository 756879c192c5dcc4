// int8 m16n8k32 MMA whose accumulator starts at 0x4B400000 (the result read as a float is 12582912 + dot), the packed fp32
// arithmetic of its epilogue (mmq.cu: head comment), and the f16 MMA of attention.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace b200 {

// k=32 MMA step alone, accumulator pairs returned packed (aligned register pairs for the f32x2 epilogue)
__device__ __forceinline__ void mma_s8_magic2(uint64_t &p01, uint64_t &p23, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("{\n"
        ".reg .b32 c0, c1, c2, c3;\n"
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {c0,c1,c2,c3}, {%2,%3,%4,%5}, {%6,%7}, {%8,%8,%8,%8};\n"
        "mov.b64 %0, {c0,c1};\n"
        "mov.b64 %1, {c2,c3};\n"
        "}\n"
        : "=l"(p01), "=l"(p23)
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0x4B400000u));
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    uint32_t a, b;
    asm("mov.b64 {%0,%1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
    lo = __uint_as_float(a);
    hi = __uint_as_float(b);
}

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

}  // namespace b200
