// packed_f32.cuh -- float32 arithmetic on register pairs (f32x2) for the
// kernels that follow the reference's order of roundings: each half of a pair
// is rounded as the scalar instruction would round it.
#pragma once

#include <cstdint>

namespace bf {

struct F2 {
    float x, y;
};
__device__ __forceinline__ uint64_t pack2(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ F2 unpack2(uint64_t v) {
    F2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Sums of products are written as a x (+-1) + b, one rounding, with the factor from a
// kernel parameter: the compiler contracts an f32x2 product feeding an f32x2
// addition into one fused operation (also with .rn on both), which would drop
// the product's rounding; it cannot contract into an operation that is fused
// already.
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The signed nibble at bit 4 s of w as a float: the nibble with its sign bit
// flipped is its value + 8, placed in the mantissa of 2^23.
__device__ __forceinline__ float nibble_float(uint32_t w, int bit) {
    return __fsub_rn(__uint_as_float(((w >> bit) & 0xFu) ^ 0x4B000008u), 8388616.0f);
}

}  // namespace bf
