// One 32-element block of the int8 activation quantizer on one warp, lane k holding element k: the arithmetic of
// quantize-act-blocks! (src/raster/compiler/backend/cpu/quant.clj:282-305): mx = max|x|, d = mx / 127 and
// id = 1 / d in double, q = clamp(round_half_up((double)x * id), -127, 127), xs = (float)d, sum = sum of q.
#pragma once
#include <stdint.h>

namespace rstq {

__device__ __forceinline__ int quant_round_half_up(double v) {
    const double f = floor(v);
    return (int)f + ((v - f) >= 0.5 ? 1 : 0);
}

// The double arithmetic decides few codes: t = x * fl32(127 / mx), a quotient of 2 ulp, is within 127 * 2^-22 = 3.1e-5 of the
// double product, so where t is further than 5e-5 from every k + 0.5, rounding t to nearest gives the same code; u = fma(x, id,
// 1.5 * 2^23) holds that code in its low bits.  xs = fl32(mx / 127) equals (float)((double)mx / 127.0): the quotient
// of a 24-bit integer by 127 is no midpoint.  Blocks whose maximum is zero, tiny, huge or infinite, and elements
// near a tie or not a number, take the double path.  (The decode kernel, the pre-pass and the super-block quantizer, which hold
// their elements in other places, go by the same margin.)
constexpr float kQuantSure = 0.5f - 5e-5f;
// (An SM does 64 double operations per clock, and a decode step's 4096-element norm quantizes its row on one SM: two
// divisions per lane were half a microsecond of each such launch.  7B-class MLP at 8 tokens, whose quantizer
// kernels ran them too: 23.3 -> 22.6 us; a step of four 7B layers 227 -> 224 us.)
__device__ __forceinline__ void quant_block32(float v, int* q, int* sum, float* xs) {
    constexpr float kMagic = 12582912.0f;   // 2^23 + 2^22
    // non-negative floats order as their bits; elements that are no number do not count unless all are
    float mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(v), 0.f))));
    if (__all_sync(0xffffffffu, v != v)) mx = v;
    bool exact = !(mx >= 1e-30f && mx <= 1e37f);
    int code = 0;
    if (!exact) {
        const float id = __fdividef(127.f, mx);
        const float u = fmaf(v, id, kMagic);
        exact = !(fabsf(fmaf(v, id, kMagic - u)) <= kQuantSure);
        code = __float_as_int(u) - __float_as_int(kMagic);
        *xs = __fdiv_rn(mx, 127.f);
    }
    if (exact) {
        const double d = (double)mx / 127.0;
        const double id = d == 0.0 ? 0.0 : 1.0 / d;
        code = max(-127, min(127, quant_round_half_up((double)v * id)));
        *xs = (float)d;
    }
    *q = code;
    *sum = __reduce_add_sync(0xffffffffu, code);
}

// The same on eight lanes (of eight neighbours each), lane j with elements 4j .. 4j + 3: their codes as one word; sum and
// scale of the whole block.
__device__ __forceinline__ void quant_block32_words(const float (&v)[4], uint32_t* codes, int* sum, float* xs) {
    constexpr float kMagic = 12582912.0f;   // 2^23 + 2^22
    float mx = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));   // (fmaxf: numbers before NaNs)
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    bool exact = !(mx >= 1e-30f && mx <= 1e37f);
    uint32_t w = 0;
    if (!exact) {
        const float id = __fdividef(127.f, mx);
        uint32_t u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float t = fmaf(v[k], id, kMagic);
            const float frac = fabsf(fmaf(v[k], id, kMagic - t));
            exact |= !(frac <= kQuantSure);
            u[k] = __float_as_uint(t);
        }
        w = __byte_perm(__byte_perm(u[0], u[1], 0x0040), __byte_perm(u[2], u[3], 0x0040), 0x5410);
        *xs = __fdiv_rn(mx, 127.f);
    }
    if (exact) {
        const double d = (double)mx / 127.0;
        const double id = d == 0.0 ? 0.0 : 1.0 / d;
        w = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            w |= (uint32_t)(max(-127, min(127, quant_round_half_up((double)v[k] * id))) & 0xFF) << (8 * k);
        *xs = (float)d;
    }
    *codes = w;
    int s = __dp4a((int)w, 0x01010101, 0);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    *sum = s;
}

}  // namespace rstq
