// tracker_common.cuh -- register-level pieces of the streaming trackers
// (tracker_stream.cu, and the served batch in serve_kernels.cu): the int4 ->
// fp16 decode, the m16n8k16 MMA, and the FP64-phase steering weight.
#pragma once

#include <cuda_fp16.h>

#include "bf_internal.cuh"

namespace bf {
namespace trk {

__device__ __forceinline__ uint32_t lop3_and_xor(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(a), "r"(b), "r"(c));  // (a & b) ^ c
    return r;
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) {
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ __half2 bits_h2(uint32_t u) {
    return *reinterpret_cast<__half2*>(&u);
}

// Decode one 32-bit word (bytes b0..b3) into four fp16 pairs:
//   re02 = (re b0, re b2), im02 = (im b0, im b2), re13, im13.
__device__ __forceinline__ void decode_word(uint32_t w, uint32_t& re02, uint32_t& im02,
                                            uint32_t& re13, uint32_t& im13) {
    const __half2 bias_lo = __floats2half2_rn(1032.0f, 1032.0f);
    const __half2 sixteenth = __floats2half2_rn(0.0625f, 0.0625f);
    const __half2 bias_hi = __floats2half2_rn(-72.0f, -72.0f);
    const uint32_t w1 = w >> 8;
    re02 = h2_bits(__hsub2(bits_h2(lop3_and_xor(w, 0x000F000Fu, 0x64086408u)), bias_lo));
    im02 = h2_bits(__hfma2(bits_h2(lop3_and_xor(w, 0x00F000F0u, 0x64806480u)), sixteenth, bias_hi));
    re13 = h2_bits(__hsub2(bits_h2(lop3_and_xor(w1, 0x000F000Fu, 0x64086408u)), bias_lo));
    im13 = h2_bits(__hfma2(bits_h2(lop3_and_xor(w1, 0x00F000F0u, 0x64806480u)), sixteenth, bias_hi));
}

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                          uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Steering weight w = exp(i * k * (p . d)) in two steps: the FP64 delay
// p . d (shared by all channels of a direction), then the FP64 phase
// k * delay reduced to a quadrant n and r = phase - n pi / 2 in [-pi/4, pi/4]
// (one fused multiply-add), and sin r, cos r from their Taylor series
// through r^11 and r^12 (truncation error below 3e-11 on the interval)
// evaluated in FP32 by Horner's rule.  Every operation is an explicitly
// rounded intrinsic, so any kernel that composes these two gets
// bit-identical weights.
__device__ __forceinline__ float2 sincos_quadrant(float r, int quad) {
    const float r2 = __fmul_rn(r, r);
    float ps = -2.5052108385441718775e-8f;               // -1/11!
    ps = __fmaf_rn(ps, r2, 2.7557319223985890653e-6f);   //  1/9!
    ps = __fmaf_rn(ps, r2, -1.9841269841269841270e-4f);  // -1/7!
    ps = __fmaf_rn(ps, r2, 8.3333333333333333333e-3f);   //  1/5!
    ps = __fmaf_rn(ps, r2, -1.6666666666666666667e-1f);  // -1/3!
    const float sn = __fmaf_rn(__fmul_rn(ps, r2), r, r);
    float pc = 2.0876756987868098979e-9f;                //  1/12!
    pc = __fmaf_rn(pc, r2, -2.7557319223985890653e-7f);  // -1/10!
    pc = __fmaf_rn(pc, r2, 2.4801587301587301587e-5f);   //  1/8!
    pc = __fmaf_rn(pc, r2, -1.3888888888888888889e-3f);  // -1/6!
    pc = __fmaf_rn(pc, r2, 4.1666666666666666667e-2f);   //  1/4!
    pc = __fmaf_rn(pc, r2, -0.5f);
    const float cs = __fmaf_rn(pc, r2, 1.0f);
    // (cos, sin) of n pi / 2 + r: quadrants 1 and 3 swap, 1 and 2 negate
    // cos, 2 and 3 negate sin
    const float c1 = (quad & 1) != 0 ? sn : cs;
    const float s1 = (quad & 1) != 0 ? cs : sn;
    return make_float2(quad == 1 || quad == 2 ? -c1 : c1, (quad & 2) != 0 ? -s1 : s1);
}
__device__ __forceinline__ double steering_delay(const float* pos, int a, double dx, double dy, double dz) {
    return __dadd_rn(__dadd_rn(__dmul_rn(static_cast<double>(pos[3 * a]), dx),
                               __dmul_rn(static_cast<double>(pos[3 * a + 1]), dy)),
                     __dmul_rn(static_cast<double>(pos[3 * a + 2]), dz));
}
// n = rint(x) and n mod 4.  Below 2^51 in magnitude, x + 1.5 * 2^52 lands
// where the ulp is 1, so the addition rounds x to an integer exactly as rint
// does (to nearest, ties to even) and the low bits of the sum hold n mod 4
// (1.5 * 2^52 is a multiple of 4): two additions instead of a rounding and a
// 64-bit conversion.  Larger |x| takes rint.
__device__ __forceinline__ double round_quadrant(double x, int& quad) {
    constexpr double kShift = 6755399441055744.0;  // 1.5 * 2^52
    if (fabs(x) < 0x1p51) {
        const double s = __dadd_rn(x, kShift);
        quad = __double2loint(s) & 3;
        return __dsub_rn(s, kShift);
    }
    const double n = rint(x);
    quad = static_cast<int>(static_cast<long long>(n) & 3);
    return n;
}
__device__ __forceinline__ float2 steering_from_delay(double k, double delay) {
    constexpr double kHalfPi = 1.5707963267948966192313216916398;
    constexpr double kTwoOverPi = 0.63661977236758134307553505349006;
    const double phase = __dmul_rn(k, delay);
    int quad;
    const double n = round_quadrant(__dmul_rn(phase, kTwoOverPi), quad);
    const float r = __double2float_rn(__fma_rn(-kHalfPi, n, phase));
    return sincos_quadrant(r, quad);
}
__device__ __forceinline__ float2 steering_weight(const float* pos, int a, double k, double dx,
                                                  double dy, double dz) {
    return steering_from_delay(k, steering_delay(pos, a, dx, dy, dz));
}

__device__ __forceinline__ uint16_t split_part(float c, bool lo) {
    const __half h = __float2half_rn(c);
    if (!lo) return __half_as_ushort(h);
    return __half_as_ushort(__float2half_rn(c - __half2float(h)));
}

// Integer form (windows above 16 spectra).  A weight w is the integer
// q = rint(w 2^30) in four signed base-256 digits, exact for float weights of
// at least 2^-7 and within 2^-31 below; voltages are 16 x the int4 values, one
// mask per four components.  mma.m16n8k32 on int8 multiplies 16 spectra by 16
// antennas (re in k 0-15, im in k 16-31) into the eight columns (re, im) x
// (d3, d2, d1, d0), exactly.  Against the fp16 hi + lo form it halves the MMAs,
// takes a third of the decode's instructions and rounds only when the digit
// sums are put together; weights cost a third more to form, which a window of
// one block does not earn back.

// A weight has digits when it is finite and of the size a phasor can have; a
// direction or wave number that is not finite gives one that has none.  Such a
// (window, channel) must not come out as a finite power, as it does not in the
// forms that keep weights as floats: its powers are NaN.  Weights are looked at
// only where a delay or a wave number is out of the ordinary: inside both bounds
// a phase is below 2^51 quadrants and its weight a phasor.
__device__ __forceinline__ bool odd_delay(double delay) { return !(fabs(delay) < 0x1p40); }
__device__ __forceinline__ bool odd_wave_number(double k) { return !(fabs(k) < 0x1p11); }
__device__ __forceinline__ bool has_digits(float2 w) { return fabsf(w.x) < 1.5f && fabsf(w.y) < 1.5f; }
// All of a window's weights, for the warp.
template <int A>
__device__ __forceinline__ bool weights_have_digits(double k, const double* delays, int lane) {
    bool all = true;
#pragma unroll 1
    for (int a = lane; a < A; a += 32) all = all && has_digits(steering_from_delay(k, delays[a]));
    return __all_sync(0xffffffffu, all);
}

// The digits of rint(w 2^30) as the bytes d0 .. d3, and those of its negative.
struct Digits {
    uint32_t pos, neg;
};
__device__ __forceinline__ Digits weight_digits(float w) {
    const uint32_t q = static_cast<uint32_t>(__float2int_rn(__fmul_rn(w, 0x1p30f)));
    return Digits{(q + 0x80808080u) ^ 0x80808080u, (0x80808080u - q) ^ 0x80808080u};
}
// Digit rows of a channel's weights in shared memory, one byte per antenna:
// d3 .. d0 of Re w, of -Im w, of Im w.
constexpr int kDigitRows = 12;
// Antennas 2 pair and 2 pair + 1 of the rows.
template <int A>
__device__ __forceinline__ void store_digits(uint8_t* rows, int pair, float2 w0, float2 w1) {
    const Digits x0 = weight_digits(w0.x), x1 = weight_digits(w1.x);
    const Digits y0 = weight_digits(w0.y), y1 = weight_digits(w1.y);
    uint16_t* dst = reinterpret_cast<uint16_t*>(rows) + pair;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const uint32_t sel = 0x0073u - 0x11u * d;  // byte 3 - d of both
        dst[d * (A / 2)] = static_cast<uint16_t>(__byte_perm(x0.pos, x1.pos, sel));
        dst[(4 + d) * (A / 2)] = static_cast<uint16_t>(__byte_perm(y0.neg, y1.neg, sel));
        dst[(8 + d) * (A / 2)] = static_cast<uint16_t>(__byte_perm(y0.pos, y1.pos, sel));
    }
}
// Antennas 4 quad .. + 3 of the rows.
template <int A>
__device__ __forceinline__ void store_digit_quad(uint8_t* rows, int quad, const float2 (&w)[4]) {
    uint32_t words[3][4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const Digits im = weight_digits(w[a].y);
        words[0][a] = weight_digits(w[a].x).pos;
        words[1][a] = im.neg;
        words[2][a] = im.pos;
    }
    uint32_t* dst = reinterpret_cast<uint32_t*>(rows) + quad;
#pragma unroll
    for (int part = 0; part < 3; ++part) {
        // bytes 0 and 1, 2 and 3 of two antennas, then each byte of all four
        const uint32_t* x = words[part];
        const uint32_t lo0 = __byte_perm(x[0], x[1], 0x5140), lo1 = __byte_perm(x[2], x[3], 0x5140);
        const uint32_t hi0 = __byte_perm(x[0], x[1], 0x7362), hi1 = __byte_perm(x[2], x[3], 0x7362);
        dst[(4 * part) * (A / 4)] = __byte_perm(hi0, hi1, 0x7632);
        dst[(4 * part + 1) * (A / 4)] = __byte_perm(hi0, hi1, 0x5410);
        dst[(4 * part + 2) * (A / 4)] = __byte_perm(lo0, lo1, 0x7632);
        dst[(4 * part + 3) * (A / 4)] = __byte_perm(lo0, lo1, 0x5410);
    }
}
// B fragments (b0: re inputs, b1: im inputs) of a column's two rows, over word
// j of the A / 4 antennas of a lane quad.
template <int A>
__device__ __forceinline__ void load_row_frags(const uint8_t* r0, const uint8_t* r1, uint32_t (&b)[A / 16][2]) {
    if constexpr (A == 32) {
        const uint2 x = *reinterpret_cast<const uint2*>(r0), y = *reinterpret_cast<const uint2*>(r1);
        b[0][0] = x.x; b[1][0] = x.y; b[0][1] = y.x; b[1][1] = y.y;
    } else {
#pragma unroll
        for (int j = 0; j < A / 16; j += 4) {
            const uint4 x = *reinterpret_cast<const uint4*>(r0 + 4 * j), y = *reinterpret_cast<const uint4*>(r1 + 4 * j);
            b[j][0] = x.x; b[j + 1][0] = x.y; b[j + 2][0] = x.z; b[j + 3][0] = x.w;
            b[j][1] = y.x; b[j + 1][1] = y.y; b[j + 2][1] = y.z; b[j + 3][1] = y.w;
        }
    }
}
// One source: column g of (re, im) x (d3, d2, d1, d0).
template <int A>
__device__ __forceinline__ void load_digit_frags(const uint8_t* rows, int g, int q, uint32_t (&b)[A / 16][2]) {
    load_row_frags<A>(rows + (g < 4 ? g : g + 4) * A + q * (A / 4),       // re: Re w; im: Im w
                      rows + (g < 4 ? g + 4 : g - 4) * A + q * (A / 4), b);  // re: -Im w; im: Re w
}
// Two sources: columns (re, im) x (first, second source) x two digits, d3 and
// d2 in one tile, d1 and d0 in the other, so that a lane holds all digits of
// one component of one source.
template <int A>
__device__ __forceinline__ void load_pair_frags(const uint8_t* first, const uint8_t* second, int g, int q,
                                                uint32_t (&b)[2][A / 16][2]) {
    const uint8_t* rows = ((g & 2) == 0 ? first : second) + q * (A / 4);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int d = 2 * h + (g & 1);
        load_row_frags<A>(rows + (g < 4 ? d : d + 8) * A, rows + (g < 4 ? d + 4 : d) * A, b[h]);
    }
}
__device__ __forceinline__ void mma_16832(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 x the real and imaginary parts of a word's four samples.
__device__ __forceinline__ uint32_t word_re16(uint32_t w) { return (w << 4) & 0xF0F0F0F0u; }
__device__ __forceinline__ uint32_t word_im16(uint32_t w) { return w & 0xF0F0F0F0u; }
// What lane q's digit sums count: the lanes of d3 and d2 (q even), of d1 and d0.
__device__ __forceinline__ float digit_scale(int q) { return (q & 1) == 0 ? 0x1p-18f : 0x1p-34f; }
// The squared part of rows g and g + 8: re^2 in lanes q = 0 and 1, im^2 in 2
// and 3.  Lane q even holds the sums of d3 and d2, odd those of d1 and d0; a
// sum is at most 2 A 2^14 in magnitude, so 256 x one fits 32 bits up to 128
// antennas.  scale: digit_scale(q), or NaN for a window without digits.
template <int A>
__device__ __forceinline__ void digit_squares(const int (&d)[4], float scale, float& sq_g, float& sq_h) {
    float f[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if constexpr (A <= 128) {
            f[h] = __fmul_rn(__int2float_rn(d[2 * h] * 256 + d[2 * h + 1]), scale);
        } else {
            f[h] = __fmul_rn(__fmaf_rn(__int2float_rn(d[2 * h]), 256.0f, __int2float_rn(d[2 * h + 1])), scale);
        }
        f[h] = __fadd_rn(f[h], __shfl_xor_sync(0xffffffffu, f[h], 1));
    }
    sq_g = __fmul_rn(f[0], f[0]);
    sq_h = __fmul_rn(f[1], f[1]);
}

}  // namespace trk
}  // namespace bf
