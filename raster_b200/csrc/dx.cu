// Backward-data of the frozen-weight linear, qlinear-q8-dx (src/raster/quant/train.clj:110-142):
//   dx[m, i] = sum over o of scales[o, i / 32] * codes[o, i] * dy[m, o]
// the dequant-transpose GEMM dX = dY . dequant(W), W = [out, in] signed 8-bit codes in the
// reference's row-major layout with one f32 scale per 32 columns.
//
// Two launches.  dx_prep_kernel writes dy as terms of 16 bits, dx_tmem_kernel is a tcgen05 GEMM over them with the
// weights dequantized, in f32, and split the same way on their way into tensor memory:
//
//   D[128 columns i, NT tokens] += W'[i, o] * dy[m, o]
//
// in one of two forms, tile by tile:
//
//   pairs of fp16     W' = H + 2^-11 L, dy = h + 2^-11 l:  H h + 2^-11 (H l + L h)                             3 MMAs
//   triples of bf16   W' = W1 + W2 + W3, dy = Y1 + Y2 + Y3:  W1 Y1 + (W1 Y2 + W2 Y1) + (W1 Y3 + W2 Y2 + W3 Y1)  6 MMAs
//
// A pair (11 bits, a sign, 11 bits) holds an element of dy to 2 * 2^-24 of itself, one unit of f32's last place, and a weight to
// 6 * 2^-24 (4.0 seen, 0.95 rms): its scale is a pair itself, times the code in packed fp16.  The second term is kept 2^11 larger than it is, in a sum of its own, and a power of
// two per token row and per 32-column block brings the largest of them close to fp16's, so an element down to 2^-27 of its row's
// largest (a scale down to 2^-20 of its column block's) is held so: the tiles whose rows and column blocks hold nothing
// smaller but zeros, and no infinity, take pairs.  Triples hold all 24 bits at any spread (2^-90 is tested); a tile with
// one such row or column block takes them.  dx_prep_kernel writes both forms of dy and says which rows are which.
//
// The sums on the tensor core decide the error of a long sum, its products that of a short one.  2-norm against the f64 product,
// over that of the product, triples / pairs: 4096 x 4096, m = 512 9.2e-6 / 4.9e-6 (pairs add half as often to the first sum), m = 64
// 9.7e-7 / 6.5e-7 (even and odd steps have sums of their own), 1024 x 1024, m = 16 4.5e-7 / 3.5e-7; sums over 256, 192, 128, 64, 32 rows
// up to 64 tokens 2.2e-7 / 2.1e-7, 1.7 / 1.9, 1.1 / 1.4, 0.68 / 1.4, 0.53 / 1.1; more tokens, over 64 rows 1.7 / 1.4, over 32 1.09 / 1.11.
// So sums that short are triples: pairs are nowhere further from the f64 product (dx_pair_rows).
//
// What bounds it: the tensor core at the power cap, for pairs nominally 768 cycles per 64 rows of a 128 x 128 tile; with the
// conversions taken out the same MMAs take 1050, with them 1160.  us per call back to back, all tiles triples -> pairs
// where they hold: 4096 x 4096, m = 512 98.4 -> 62.5, m = 64 29.0 -> 25.5; 1024 x 1024, m = 16 16.3 -> 15.0; 11008 x 2048, m = 300
// 135 -> 82.8.  With a row of small elements per tile, so triples: 91.6, 30.0, 17.4 (dy waits for the tile's form), 126 (92.0, 29.2, 16.6 without pairs).
#include <type_traits>

#include "internal.h"
#include "mma_helpers.cuh"
#include "tcgen05_helpers.cuh"

namespace rstq {

constexpr int kDxStep = 64;                    // rows o per pipeline stage
constexpr int kDxRaw = 8;                      // stages of codes and scales in shared memory
constexpr int kDxSet = 8;                      // dequant warps of a stage: 4 blocks of 32 columns x 2 halves of its rows
constexpr int kDxDq = 2 * kDxSet;              // two sets on alternate stages
constexpr int kDxThreads = (kDxDq + 3) * 32;   // + two copy warps and the MMA warp
constexpr int kDxCodes = kDxStep * 128;        // bytes of codes per stage
constexpr int kDxScales = 1024;                // bytes of scales per stage: 64 rows x 4 blocks
constexpr int kDxRawBytes = kDxCodes + kDxScales;
// A form's rings.  dy, in shared memory: four stages of pairs or three of triples (nine planes of nt x 128 bytes hold
// either).  W', in tensor memory behind the accumulators (nt columns each): 32 columns per term and stage.
template <int NT, bool PAIRS>
struct DxForm {
    static constexpr int terms = PAIRS ? 2 : 3;
    static constexpr int ybytes = terms * NT * 128;
    static constexpr int ystages = PAIRS ? 4 : 3;
    static constexpr int accs = PAIRS ? (NT > 64 ? 2 : 4) : (NT > 64 ? 2 : 3);
    static constexpr int wcols = 32 * terms;
    static constexpr int wstages = (512 - accs * NT) / wcols < 4 ? (512 - accs * NT) / wcols : 4;   // 4; triples 2, 3 or 4
};
constexpr int kDxMaxY = 4, kDxMaxW = 4;        // barriers of either ring
__host__ __device__ constexpr int dx_yring_bytes(int nt) { return 9 * nt * 128; }
__host__ __device__ constexpr int dx_ring_bytes(int nt) { return dx_yring_bytes(nt) + kDxRaw * kDxRawBytes; }

// Position p of an element inside its group of 16 rows o: the order in which a lane of the dequant warps holds
// them (rows 2t, 2t + 1, 2t + 8, 2t + 9 for t = p / 4).  Any order serves, as long as dy has the same one; this
// one reads the 128-byte-swizzled code tile without bank conflicts.
__host__ __device__ constexpr int dx_row_of(int p) { return 2 * (p >> 2) + (p & 1) + ((p & 2) ? 8 : 0); }

// ---- what the GEMM needs beforehand: dy in both forms, the largest and the smallest scale of every column block ------
constexpr int kDxParts = 64;                   // thread blocks that look at the scales, each at its share of the rows o
struct DxPrep {
    const float* dy;
    const float* scales;
    uint16_t* y;            // [3][m][opad]: bf16 terms of dy * 2^-e
    uint16_t* y16;          // [2][m][opad]: fp16 terms of dy * 2^-(e + 5)
    int* rowexp;            // [m]: 2 e, which brings max|dy| of the row into [2^19, 2^20), + 1 if pairs do not hold the row
    float* colmax;          // [2][kDxParts][nb]: max|scale| of a part's rows; min|scale| of those that are not zero
    int64_t m, out, nb, opad;
};

// The exponent e that brings a finite maximum into [2^(top-1), 2^top) as max * 2^-e, and 2^-e as two factors (a
// subnormal maximum needs more than one f32 holds).
__device__ __forceinline__ int dx_exponent(float mx, int top, float* down, float* down2) {
    int e = 0;
    if (mx > 0.f && mx < __int_as_float(0x7F800000)) {
        int ex;
        frexpf(mx, &ex);
        e = ex - top;
    }
    const int e1 = e < -100 ? -100 : e;
    *down = ldexpf(1.0f, -e1);
    *down2 = ldexpf(1.0f, e1 - e);
    return e;
}
// v * 2^e.  In two halves, whose powers f32 holds and between which nothing leaves its range that the result does
// not leave; below 2^-252 every v here (< 2^71) ends as zero.  (ldexpf does the same 3 us slower over 512 x 4096 results.)
__device__ __forceinline__ float dx_scale(float v, int e) {
    e = e < -252 ? -252 : e;
    const int h = e >> 1;
    return v * __int_as_float((h + 127) << 23) * __int_as_float((e - h + 127) << 23);
}
// What pairs hold whole: with the largest magnitude of dy in [2^19, 2^20), of the scales in [2^12, 2^13), no element
// and no scale but zeros below 2^-8.  (As fp16 both carry 2^-5 less: |dy| and |code * scale| stay below fp16's largest, and
// 2^-13 is where the second term, 2^11 larger than it is, still has its 11 bits.)
constexpr int kDxPrepMax = 512;     // threads per block of the pre-pass, at most
constexpr float kDxPairMin = 0.00390625f;
constexpr int kDxPairExp = 5;
constexpr float kDxLow = 2048.0f;   // what the second terms of pairs are larger by
__host__ __device__ constexpr int dx_pair_rows(int nt) { return nt <= 64 ? 256 : 64; }   // shorter sums: triples
__device__ __forceinline__ float dx_nonzero(float v) { return v == 0.f ? __int_as_float(0x7F800000) : fabsf(v); }
__device__ __forceinline__ void dx_block_range(float& mx, float& mn, float (*red)[kDxPrepMax / 32]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = mx;
        red[1][threadIdx.x >> 5] = mn;
    }
    __syncthreads();
    mx = red[0][0];
    mn = red[1][0];
    for (int i = 1; i < (int)blockDim.x / 32; ++i) {
        mx = fmaxf(mx, red[0][i]);
        mn = fminf(mn, red[1][i]);
    }
    __syncthreads();
}
__device__ __forceinline__ uint32_t pack_f16x2(float hi, float lo) {
    uint32_t d;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ float2 unpack_f16x2(uint32_t h) {
    const __half2 v = *reinterpret_cast<const __half2*>(&h);
    return __half22float2(v);
}
// b (upper half) and a (lower half) as pairs of fp16 terms
__device__ __forceinline__ void dx_pair(float b, float a, uint32_t* t1, uint32_t* t2) {
    *t1 = pack_f16x2(b, a);
    const float2 h = unpack_f16x2(*t1);
    *t2 = pack_f16x2((b - h.y) * kDxLow, (a - h.x) * kDxLow);
}
// b (upper half) and a (lower half) as three bf16 terms each.  INF: an infinity goes into the last term, which meets the
// first term of the other factor alone -- next to the zeros among the other terms it would come out as a NaN.
template <bool INF>
__device__ __forceinline__ void dx_terms(float b, float a, uint32_t* t1, uint32_t* t2, uint32_t* t3) {
    uint32_t keep = 0xFFFFFFFFu;
    if (INF) {
        if (isinf(a)) keep &= 0xFFFF0000u;
        if (isinf(b)) keep &= 0x0000FFFFu;
    }
    const uint32_t p1 = pack_bf16x2(b, a) & keep;
    a -= __uint_as_float(p1 << 16);
    b -= __uint_as_float(p1 & 0xFFFF0000u);
    const uint32_t p2 = pack_bf16x2(b, a) & keep;
    a -= __uint_as_float(p2 << 16);
    b -= __uint_as_float(p2 & 0xFFFF0000u);
    *t1 = p1;
    *t2 = p2;
    *t3 = pack_bf16x2(b, a);
}

// Latency-bound: every element is read once into registers (rows up to 16384), found the range of, and written in
// both forms; the blocks that look at the scales read theirs as one run and leave a range per column block
// (a strip of column blocks per thread block instead took 45 us at 4096 x 4096: 16 bytes of every row).  Adds 6.2 us to the
// GEMM behind it at 4096 x 4096, m = 512 (9.4 with a whole group of 16 rows per thread: half sectors), 2.2 of them for the triples.
constexpr int kDxMaxCols = 4096;
__global__ void __launch_bounds__(kDxPrepMax, 2)
dx_prep_kernel(const DxPrep p) {
    __shared__ float s_red[2][kDxPrepMax / 32];
    __shared__ uint32_t s_max[kDxMaxCols], s_min[kDxMaxCols];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int nt = (int)blockDim.x;
    if (blockIdx.x < kDxParts) {
        const int64_t o0 = p.out * blockIdx.x / kDxParts, o1 = p.out * (blockIdx.x + 1) / kDxParts;
        for (int64_t c0 = 0; c0 < p.nb; c0 += kDxMaxCols) {     // (one pass up to 131 072 columns i)
            const int nc = (int)(p.nb - c0 < kDxMaxCols ? p.nb - c0 : kDxMaxCols);
            for (int c = threadIdx.x; c < nc; c += nt) {
                s_max[c] = 0u;
                s_min[c] = 0x7F800000u;
            }
            __syncthreads();
            // a thread keeps its columns (four where rows are whole 16 bytes) and steps over the rows
            const bool vec = (p.nb & 3) == 0;
            const int cols = vec ? nc >> 2 : nc, groups = cols < nt ? nt / cols : 1;
            const int rg = (int)threadIdx.x / cols;
            if (rg < groups || cols >= nt) {
                for (int c = (int)threadIdx.x - rg * cols; c < cols; c += nt) {
                    float mx[4] = {0.f, 0.f, 0.f, 0.f}, mn[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) mn[j] = __int_as_float(0x7F800000);
                    const float* q = p.scales + c0 + (vec ? 4 * c : c);
#pragma unroll 8
                    for (int64_t o = o0 + (cols < nt ? rg : 0); o < o1; o += groups) {
                        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (vec) f = __ldg(reinterpret_cast<const float4*>(q + o * p.nb));
                        else f.x = __ldg(q + o * p.nb);
                        const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            mx[j] = fmaxf(mx[j], fabsf(v[j]));
                            mn[j] = fminf(mn[j], dx_nonzero(v[j]));
                        }
                    }
                    // (the bits of magnitudes order like the magnitudes)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (vec || j == 0) {
                            atomicMax(&s_max[vec ? 4 * c + j : c], __float_as_uint(mx[j]));
                            atomicMin(&s_min[vec ? 4 * c + j : c], __float_as_uint(mn[j]));
                        }
                }
            }
            __syncthreads();
            for (int c = threadIdx.x; c < nc; c += nt) {
                p.colmax[(int64_t)blockIdx.x * p.nb + c0 + c] = __uint_as_float(s_max[c]);
                p.colmax[(int64_t)(kDxParts + blockIdx.x) * p.nb + c0 + c] = __uint_as_float(s_min[c]);
            }
            __syncthreads();
        }
        return;
    }
    const int64_t m = (int64_t)blockIdx.x - kDxParts;
    const float* src = p.dy + m * p.out;
    const bool vec = (p.out & 3) == 0;
    // Half a group of 16 rows o per thread and step: rows 4h .. 4h + 3 and 8 + 4h .. are positions 8h .. 8h + 7, so that a
    // warp reads and writes whole 32-byte sectors.
    auto load8 = [&](int64_t at, float (&v)[8]) {   // at: position, a multiple of 8
        const int64_t o = (at & ~15ll) + ((at & 8) >> 1);
        if (vec && o + 12 <= p.out) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 f = __ldg(reinterpret_cast<const float4*>(src + o + 8 * j));
                v[4 * j] = f.x; v[4 * j + 1] = f.y; v[4 * j + 2] = f.z; v[4 * j + 3] = f.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = o + (j & 3) + 2 * (j & 4) < p.out ? __ldg(src + o + (j & 3) + 2 * (j & 4)) : 0.f;
        }
    };
    float mx = 0.f, mn = __int_as_float(0x7F800000);
    auto range8 = [&](const float (&v)[8]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            mx = fmaxf(mx, fabsf(v[j]));
            mn = fminf(mn, dx_nonzero(v[j]));
        }
    };
    constexpr int kKeep = 4;   // x threads x 8 elements
    const bool keep = p.opad <= (int64_t)kKeep * nt * 8;
    float held[kKeep][8];
    if (keep) {
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int64_t at = (int64_t)(i * nt + threadIdx.x) * 8;
            if (at < p.opad) load8(at, held[i]);
        }
#pragma unroll
        for (int i = 0; i < kKeep; ++i)
            if ((int64_t)(i * nt + threadIdx.x) * 8 < p.opad) range8(held[i]);
    } else {
        for (int64_t at = threadIdx.x * 8; at < p.opad; at += nt * 8) {
            load8(at, held[0]);
            range8(held[0]);
        }
    }
    float down, down2;
    dx_block_range(mx, mn, s_red);
    const int e = dx_exponent(mx, 20, &down, &down2);
    const bool wide = isinf(mx) || mn * down * down2 < kDxPairMin;
    auto store8 = [&](int64_t at, const float (&v)[8]) {
        constexpr float kPair = 1.0f / (1 << kDxPairExp);
        uint32_t t[5][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {   // positions at + 2q, + 1
            const int r = 2 * (q >> 1) + 4 * (q & 1);
            const float a = v[r] * down * down2, b = v[r + 1] * down * down2;
            dx_terms<true>(b, a, &t[0][q], &t[1][q], &t[2][q]);
            dx_pair(b * kPair, a * kPair, &t[3][q], &t[4][q]);
        }
#pragma unroll
        for (int k = 0; k < 5; ++k)
            *reinterpret_cast<uint4*>((k < 3 ? p.y + (k * p.m + m) * p.opad : p.y16 + ((k - 3) * p.m + m) * p.opad) + at) =
                make_uint4(t[k][0], t[k][1], t[k][2], t[k][3]);
    };
    if (keep) {
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int64_t at = (int64_t)(i * nt + threadIdx.x) * 8;
            if (at < p.opad) store8(at, held[i]);
        }
    } else {
        for (int64_t at = threadIdx.x * 8; at < p.opad; at += nt * 8) {
            load8(at, held[0]);
            store8(at, held[0]);
        }
    }
    if (threadIdx.x == 0) p.rowexp[m] = 2 * e + (wide ? 1 : 0);
}

// ---- the GEMM -----------------------------------------------------------------------------------
struct DxParams {
    const float* scales;
    const int* rowexp;
    const float* colmax;
    float* dx;
    int* status;
    int64_t in, out;
    int tma_scales;          // nb % 4 == 0: the scales of a stage come with its copies, else by loads of the lanes
    int m, steps, ttiles, split;   // split: thread blocks (one cluster) that share a tile, each a range of o
};

__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
// A copy thread that gave up: let the copies it has issued land before this block's shared memory goes away.
__device__ __noinline__ void dx_drain(uint32_t bars, int issued, int ring) {
    for (int k = issued > ring ? issued - ring : 0; k < issued; ++k) {
        const unsigned long long t0 = gtime_ns();
        while (!mbar_try(bars + 8 * (k % ring), (uint32_t)(k / ring) & 1u) && gtime_ns() - t0 < kWaitLimitNs) {
        }
    }
}

// The MMAs of 16 rows o, triples.  The three terms of dy lie one above the other in shared memory, so a term of W' times several
// of them is one instruction as far as the width allows (256): a tcgen05 instruction costs its issuer 50 - 60
// cycles, and A is read from tensor memory once for both.  Up to 64 tokens the accumulators are the three sums in
// the order of their size.  Above, W2 Y1 goes to the first product for the sake of that (4096 x 4096, m = 512: 102.6 ->
// 91.9 us).
template <int NT>
__device__ __forceinline__ void dx_mma16(uint32_t d, uint32_t w, uint32_t b_lo, uint32_t b_hi, uint32_t accumulate, uint32_t leader) {
    constexpr uint32_t id1 = idesc_bf16(NT), id2 = idesc_bf16(2 * NT), id3 = idesc_bf16(NT <= 64 ? 3 * NT : NT);
    if constexpr (NT <= 64) {
        asm volatile(
            "{\n"
            ".reg .pred p, q, t;\n"
            ".reg .b64 b0;\n"
            "setp.ne.b32 p, %10, 0;\n"
            "setp.ne.b32 q, %11, 0;\n"
            "setp.eq.b32 t, 0, 0;\n"
            "mov.b64 b0, {%6, %7};\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%3], b0, %12, p;\n"   // W1 (Y1, Y2, Y3)
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%4], b0, %9, t;\n"    // W2 (Y1, Y2)
            "@q tcgen05.mma.cta_group::1.kind::f16 [%2], [%5], b0, %8, t;\n"    // W3 Y1
            "}" ::"r"(d), "r"(d + NT), "r"(d + 2 * NT), "r"(w), "r"(w + 32), "r"(w + 64), "r"(b_lo), "r"(b_hi), "r"(id1), "r"(id2),
            "r"(accumulate), "r"(leader), "r"(id3)
            : "memory");
    } else {
        asm volatile(
            "{\n"
            ".reg .pred p, q, t;\n"
            ".reg .b64 b0, b2;\n"
            "setp.ne.b32 p, %8, 0;\n"
            "setp.ne.b32 q, %9, 0;\n"
            "setp.eq.b32 t, 0, 0;\n"
            "mov.b64 b0, {%5, %7};\n"
            "mov.b64 b2, {%6, %7};\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], b0, %11, p;\n"   // W1 (Y1, Y2)
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], b2, %10, t;\n"   // W1 Y3
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%3], b0, %11, t;\n"   // W2 (Y1, Y2)
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%4], b0, %10, t;\n"   // W3 Y1
            "}" ::"r"(d), "r"(d + NT), "r"(w), "r"(w + 32), "r"(w + 64), "r"(b_lo), "r"(b_lo + 2 * NT * 8), "r"(b_hi), "r"(accumulate),
            "r"(leader), "r"(id1), "r"(id2)
            : "memory");
    }
}

// The same of pairs: H (h, l) as one instruction over 2 NT columns, L h to the sum of the second terms.
template <int NT>
__device__ __forceinline__ void dx_mma16_pairs(uint32_t d, uint32_t w, uint32_t b_lo, uint32_t b_hi, uint32_t accumulate, uint32_t leader) {
    constexpr uint32_t id1 = idesc_f16(NT), id2 = idesc_f16(2 * NT);
    asm volatile(
        "{\n"
        ".reg .pred p, q, t;\n"
        ".reg .b64 b0;\n"
        "setp.ne.b32 p, %6, 0;\n"
        "setp.ne.b32 q, %7, 0;\n"
        "setp.eq.b32 t, 0, 0;\n"
        "mov.b64 b0, {%4, %5};\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], b0, %9, p;\n"   // H (h, l)
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%3], b0, %8, t;\n"   // L h
        "}" ::"r"(d), "r"(d + NT), "r"(w), "r"(w + 32), "r"(b_lo), "r"(b_hi), "r"(accumulate), "r"(leader), "r"(id1), "r"(id2)
        : "memory");
}

// Warps 0 .. 15 dequantize and store the tile (warp & 3 = 32-column block = its tensor-memory lanes, (warp >> 2) & 1 =
// half of the stage's rows o, warp >> 3 = even / odd stages), warp 16 copies codes and scales, 17 issues the MMAs, 18
// copies dy.  Warps 0 .. 15 also find out which form the tile takes.  Codes, dy and W' have rings of their own: with one ring a stage waited for copy, conversion and MMA in turn.
// Tensor-memory lane gid + 8 r of a block is column 4 gid + r of it: a lane of the dequant warp reads the codes
// of four neighbouring columns as one word per row, and the 16x256b store wants exactly these four lanes of it.
// Every mbarrier wait is time-bounded; on expiry the block reports through the status word, lets its copies
// land, still meets its barriers and frees its tensor memory.
template <int NT>
__global__ void __launch_bounds__(kDxThreads, 1)
dx_tmem_kernel(const DxParams p, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_y,
               const __grid_constant__ CUtensorMap map_y16, const __grid_constant__ CUtensorMap map_s) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_abort, s_wide;
    __shared__ uint32_t s_tmem;
    __shared__ int s_colexp[4];
    __shared__ __align__(8) uint64_t s_bar[2 * kDxMaxY + 2 * kDxMaxW + 2 * kDxRaw + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem), bar0 = smem_u32(s_bar);
    // y_full: a stage of dy has arrived; w_full: a stage of W' is in tensor memory; y_free, w_free: their MMAs are done;
    // raw: codes and scales of a step have arrived; taken: they are in registers
    const uint32_t y_full = bar0, y_free = y_full + 8 * kDxMaxY, w_full = y_free + 8 * kDxMaxY, w_free = w_full + 8 * kDxMaxW;
    const uint32_t raw = w_free + 8 * kDxMaxW, taken = raw + 8 * kDxRaw, acc_full = taken + 8 * kDxRaw;
    const uint32_t rbase = sbase + dx_yring_bytes(NT);
    const int part = blockIdx.x % p.split, tile = blockIdx.x / p.split;
    const int ft = tile / p.ttiles, tok0 = (tile - ft * p.ttiles) * NT;
    const int k0 = (int)((int64_t)p.steps * part / p.split), k1 = (int)((int64_t)p.steps * (part + 1) / p.split);
    volatile int* abort_flag = &s_abort;

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_y16)) : "memory");
    }
    if (tid < kDxMaxY) {
        mbar_init(y_full + 8 * tid, 1);
        mbar_init(y_free + 8 * tid, 1);
    }
    if (tid < kDxMaxW) {
        mbar_init(w_full + 8 * tid, kDxSet);
        mbar_init(w_free + 8 * tid, 1);
    }
    if (tid < kDxRaw) {
        mbar_init(raw + 8 * tid, 1);
        mbar_init(taken + 8 * tid, kDxSet);
    } else if (tid == kDxRaw) {
        mbar_init(acc_full, 1);
        s_abort = 0;
        s_wide = 0;
    }
    if (tid <= kDxRaw) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == kDxDq + 1) {
        tmem_alloc(smem_u32(&s_tmem), 512);
        tmem_relinquish();
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    bool ok = true, wide = false;
    auto exp_of = [&](int tok) { return (__ldg(p.rowexp + tok) >> 1) + (wide ? 0 : 2 * kDxPairExp); };
    // The dequant warps decide the tile's form; they, the MMA warp and the warp that copies dy meet here.
    auto form_known = [] { asm volatile("bar.sync 1, %0;" ::"r"((kDxDq + 2) * 32) : "memory"); };
    if (warp == kDxDq) {
        // ---------------- codes and scales ----------------
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const uint32_t bytes = p.tma_scales ? kDxRawBytes : kDxCodes;
            int s = 0, issued = 0;
            uint32_t ph = 0;
            for (int k = k0; k < k1; ++k) {
                ok = mbar_block(taken + 8 * s, ph ^ 1u, abort_flag);
                if (!ok) break;
                const uint32_t dst = rbase + s * kDxRawBytes, bar = raw + 8 * s;
                mbar_expect_tx(bar, bytes);
                tma_load_2d(dst, &map_w, ft * 128, k * kDxStep, bar);
                if (p.tma_scales) tma_load_2d(dst + kDxCodes, &map_s, ft * 4, k * kDxStep, bar);
                ++issued;
                if (++s == kDxRaw) { s = 0; ph ^= 1u; }
            }
            if (!ok) dx_drain(raw, issued, kDxRaw);
        }
    } else if (warp == kDxDq + 2) {
        // ---------------- dy ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        form_known();
        auto copy = [&](auto pairs, const CUtensorMap* map) {
            using F = DxForm<NT, decltype(pairs)::value>;
            int s = 0, issued = 0;
            uint32_t ph = 0;
            for (int k = k0; k < k1; ++k) {
                ok = mbar_block(y_free + 8 * s, ph ^ 1u, abort_flag);
                if (!ok) break;
                mbar_expect_tx(y_full + 8 * s, F::ybytes);
                tma_load_3d(sbase + s * F::ybytes, map, k * kDxStep, tok0, 0, y_full + 8 * s);
                ++issued;
                if (++s == F::ystages) { s = 0; ph ^= 1u; }
            }
            if (!ok) dx_drain(y_full, issued, F::ystages);
        };
        if (lane == 0) {
            if (s_wide) copy(std::false_type{}, &map_y);
            else copy(std::true_type{}, &map_y16);
        }
    } else if (warp == kDxDq + 1) {
        // ---------------- MMAs ----------------
        const uint32_t leader = lane == 0;
        const uint64_t d0 = smem_desc_sw128(sbase);
        const uint32_t d_lo = (uint32_t)d0, d_hi = (uint32_t)(d0 >> 32);
        bool any = false;
        form_known();
        auto issue = [&](auto pairs) {
            constexpr bool P = decltype(pairs)::value;
            using F = DxForm<NT, P>;
            int ys = 0, ws = 0;
            uint32_t yph = 0, wph = 0;
            bool ready = false;
            for (int k = k0; k < k1; ++k) {
                if (!ready) ok = mbar_spin(y_full + 8 * ys, yph, abort_flag) && mbar_spin(w_full + 8 * ws, wph, abort_flag);
                if (!ok) break;
                tc_fence_after();
                // pairs of up to 64 tokens: even and odd steps have sums of their own
                const uint32_t set = P && NT <= 64 ? (uint32_t)(k - k0) & 1u : 0u, d = tmem + set * 2 * NT;
                const uint32_t w = tmem + F::accs * NT + ws * F::wcols, b = d_lo + (uint32_t)ys * (F::ybytes >> 4);
                const int ys2 = ys + 1 == F::ystages ? 0 : ys + 1, ws2 = ws + 1 == F::wstages ? 0 : ws + 1;
                const uint32_t yph2 = ys2 ? yph : yph ^ 1u, wph2 = ws2 ? wph : wph ^ 1u;
                auto mma16 = [&](int j, uint32_t accumulate) {
                    if constexpr (P) dx_mma16_pairs<NT>(d, w + 8 * j, b + 2 * j, d_hi, accumulate, leader);
                    else dx_mma16<NT>(d, w + 8 * j, b + 2 * j, d_hi, accumulate, leader);
                };
                mma16(0, (uint32_t)(k - k0) > set);
                mma16(1, 1u);
                mma16(2, 1u);
                // (the next stage's barriers are tested ahead of the last MMAs: their round trips run beside them)
                ready = mbar_test(y_full + 8 * ys2, yph2) & mbar_test(w_full + 8 * ws2, wph2);
                mma16(3, 1u);
                umma_commit_if(w_free + 8 * ws, leader);
                umma_commit_if(y_free + 8 * ys, leader);
                any = true;
                ys = ys2; ws = ws2; yph = yph2; wph = wph2;
            }
        };
        if (s_wide) issue(std::false_type{});
        else issue(std::true_type{});
        if (any) {
            umma_commit_if(acc_full, leader);
            if (!ok) {  // gave up: the tensor core must be idle before tensor memory is freed
                const unsigned long long t0 = gtime_ns();
                while (!mbar_try(acc_full, 0) && gtime_ns() - t0 < kWaitLimitNs) {
                }
            }
        }
    } else {
        // ---------------- dequant ----------------
        const int blk = warp & 3, half = (warp >> 2) & 1, set = warp >> 3, gid = lane >> 2, t = lane & 3;
        // rows 2t, 2t + 1 (and + 8, the same swizzle) of a group of 16, columns 32 blk + 4 gid .. + 3
        const int chunk = 2 * blk + (gid >> 2);
        const uint32_t off0 = (2 * t) * 128 + ((chunk ^ (2 * t)) << 4) + (gid & 3) * 4 + half * 32 * 128;
        const uint32_t off1 = (2 * t + 1) * 128 + ((chunk ^ (2 * t + 1)) << 4) + (gid & 3) * 4 + half * 32 * 128;
        // the scale this lane splits for its warp: of row 2t + ... of group gid >> 2, the one a lane of the same t
        // holds as element gid & 3 (eight lanes hold the same eight rows)
        const int my_row = half * 32 + (gid >> 2) * 16 + 2 * t + (gid & 1) + (gid & 2) * 4;
        const uint32_t soff = kDxCodes + my_row * 16 + blk * 4;
        const int64_t nb = p.in >> 5, b = (int64_t)ft * 4 + blk;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        float mx = 0.f, mn = __int_as_float(0x7F800000);
        if (b < nb)
            for (int i = lane; i < kDxParts; i += 32) {
                mx = fmaxf(mx, __ldg(p.colmax + i * nb + b));
                mn = fminf(mn, __ldg(p.colmax + (kDxParts + i) * nb + b));
            }
        // a quarter of the tile's rows per (half, set): do pairs hold them all?
        const int tok = tok0 + (warp >> 2) * (NT / 4) + lane;
        const int row_wide = lane < NT / 4 && tok < p.m ? __ldg(p.rowexp + tok) & 1 : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        }
        float down, down2;   // the block's scales are used times 2^-ce, the largest in [2^12, 2^13)
        const int ce = dx_exponent(mx, 13, &down, &down2);
        const bool infinite = isinf(mx);   // a scale of this column block (of the whole matrix)
        const bool any_wide = p.out < dx_pair_rows(NT) || __any_sync(0xffffffffu, row_wide) || infinite || mn * down * down2 < kDxPairMin;
        if (lane == 0) {
            s_colexp[blk] = ce;   // (the four warps of a block of columns agree)
            if (any_wide) s_wide = 1;
        }
        form_known();
        wide = s_wide != 0;
        // one stage after the other: body(codes, scales, where the stage's W' of this warp goes)
        auto stages = [&](auto pairs, auto body) {
            using F = DxForm<NT, decltype(pairs)::value>;
            const uint32_t tdst = tmem + F::accs * NT + ((uint32_t)(blk * 32) << 16) + half * 16;
            int ws = set % F::wstages, rs = set;
            uint32_t wph = 0, rph = 0;
            for (int k = k0 + set; k < k1; k += 2) {
                float sf = 0.f;
                if (!p.tma_scales) {
                    const int64_t o = (int64_t)k * kDxStep + my_row;
                    if (o < p.out && b < nb) sf = __ldg(p.scales + o * nb + b);
                }
                ok = __all_sync(0xffffffffu, mbar_block(raw + 8 * rs, rph, abort_flag));
                if (!ok) break;
                const uint32_t st = rbase + rs * kDxRawBytes;
                uint32_t w[2][4];
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    w[g][0] = lds_u32(st + off0 + g * 2048);
                    w[g][1] = lds_u32(st + off1 + g * 2048);
                    w[g][2] = lds_u32(st + off0 + g * 2048 + 1024);
                    w[g][3] = lds_u32(st + off1 + g * 2048 + 1024);
                }
                if (p.tma_scales) sf = __uint_as_float(lds_u32(st + soff));
                // gather the eight scales the lane's rows need: as f32, or as pairs of fp16 (the first term below)
                sf *= down;
                sf *= down2;
                uint32_t own = __float_as_uint(sf);
                if constexpr (decltype(pairs)::value) {
                    const float first = __half2float(__float2half_rn(sf));
                    own = pack_f16x2((sf - first) * kDxLow, first);
                }
                uint32_t sc[2][4];
#pragma unroll
                for (int g = 0; g < 2; ++g)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        sc[g][j] = __shfl_sync(0xffffffffu, own, (g * 4 + j) * 4 + t);
                        w[g][j] ^= 0x80808080u;   // code + 128
                    }
                __syncwarp();
                if (lane == 0) mbar_arrive(taken + 8 * rs);
                rs += 2;
                if (rs >= kDxRaw) { rs -= kDxRaw; rph ^= 1u; }
                ok = __all_sync(0xffffffffu, mbar_block(w_free + 8 * ws, wph ^ 1u, abort_flag));
                if (!ok) break;
                tc_fence_after();
                body(w, sc, tdst + ws * F::wcols);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(w_full + 8 * ws);
                ws += 2;
                if (ws >= F::wstages) { ws -= F::wstages; wph ^= 1u; }
            }
        };
        // the code of column 4 gid + j, row h of group g: under the upper half of 2^23 the byte is 2^23 + 128 + code exactly
        auto code = [](const uint32_t (&w)[2][4], int g, int h, int j) {
            return __uint_as_float(__byte_perm(w[g][h], 0x4B000000u, 0x7440u | (uint32_t)j)) - 8388736.0f;
        };
        auto triples = [&](auto inf, const uint32_t (&w)[2][4], const uint32_t (&sc)[2][4], uint32_t dst) {
#pragma unroll
            for (int q = 0; q < 2; ++q, dst += 16u << 16) {      // columns 4 gid + 2q, + 2q + 1
                uint32_t v1[8], v2[8], v3[8];
#pragma unroll
                for (int g = 0; g < 2; ++g)
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {   // rows 2t + 8h, 2t + 8h + 1
                            const int e = g * 4 + c * 2 + h;
                            dx_terms<decltype(inf)::value>(code(w, g, 2 * h + 1, 2 * q + c) * __uint_as_float(sc[g][2 * h + 1]),
                                                           code(w, g, 2 * h, 2 * q + c) * __uint_as_float(sc[g][2 * h]), &v1[e],
                                                           &v2[e], &v3[e]);
                        }
                tmem_st_16x256b_x2(dst, v1);
                tmem_st_16x256b_x2(dst + 32, v2);
                tmem_st_16x256b_x2(dst + 64, v3);
            }
        };
        if (wide) {
            stages(std::false_type{}, [&](const uint32_t (&w)[2][4], const uint32_t (&sc)[2][4], uint32_t dst) {
                if (infinite) triples(std::true_type{}, w, sc, dst);
                else triples(std::false_type{}, w, sc, dst);
            });
        } else {
            down *= 1.0f / (1 << kDxPairExp);      // (no scale of such a block comes near f32's limits on the way)
            stages(std::true_type{}, [&](const uint32_t (&w)[2][4], const uint32_t (&sc)[2][4], uint32_t dst) {
                // Two rows at a time in packed fp16, scale = s1 + 2^-11 s2: H = code * (s1 + 2^-11 s2) to within a little more than half a
                // step (the second product is rounded, and absorbed), what it left of code * s1 is exact (a multiple of s1's
                // last place, below 2^8 of them), L = 2^11 times that + code * s2 rounded once.  (Eight instructions per two weights.
                // Without the second product in H, L is up to three times as large and rounded as much more: weights off
                // by up to 9 units of 2^-24, 1.21 rms, now 4.0 and 0.95; from f32 products it would be
                // 3.0 and 0.83, but fourteen instructions.  4096 x 4096, m = 512: 62.3, 62.5 and 67.4 us.)
                uint32_t v1[2][8], v2[2][8];
#pragma unroll
                for (int g = 0; g < 2; ++g)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {       // rows 2t + 8h, 2t + 8h + 1
                        const uint32_t s1 = __byte_perm(sc[g][2 * h], sc[g][2 * h + 1], 0x5410);
                        const uint32_t s2 = __byte_perm(sc[g][2 * h], sc[g][2 * h + 1], 0x7632);
                        const uint32_t s3 = hmul2_u32(s2, 0x10001000u);   // 2^-11 s2
#pragma unroll
                        for (int q = 0; q < 2; ++q) {   // columns 4 gid + 2q, + 2q + 1
                            const uint32_t both = __byte_perm(w[g][2 * h], w[g][2 * h + 1], q ? 0x7362 : 0x5140);
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                // under the upper byte of 1024 the code + 128 is 1152 + code
                                const uint32_t n = hadd2_u32(__byte_perm(both, 0x64u, c ? 0x4342 : 0x4140), 0xE480E480u);
                                const uint32_t hi = hfma2_u32(n, s1, hmul2_u32(n, s3));
                                const uint32_t left = hfma2_u32(n, s1, hi ^ 0x80008000u);
                                const int e = g * 4 + c * 2 + h;
                                v1[q][e] = hi;
                                v2[q][e] = hfma2_u32(n, s2, hmul2_u32(left, 0x68006800u));
                            }
                        }
                    }
#pragma unroll
                for (int q = 0; q < 2; ++q, dst += 16u << 16) {
                    tmem_st_16x256b_x2(dst, v1[q]);
                    tmem_st_16x256b_x2(dst + 32, v2[q]);
                }
            });
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_block(acc_full, 0, abort_flag));
        tc_fence_after();
        // ---------------- the tile: a warp holds 32 columns i x NT / 4 tokens ----------------
        const int64_t i = (int64_t)ft * 128 + blk * 32 + 4 * (lane & 7) + (lane >> 3);
        const bool i_ok = i < p.in;
        constexpr int TPW = NT / 4, CH = TPW < 32 ? TPW : 32;
        float* s_out = reinterpret_cast<float*>(smem);           // [NT][128], split tiles only (the ring is idle)
#pragma unroll 1
        for (int c0 = 0; c0 < TPW && ok; c0 += CH) {
            const int col = (warp >> 2) * TPW + c0;
            uint32_t a[CH], b[CH];
            const uint32_t ta = tmem + ((uint32_t)(blk * 32) << 16) + col;
#pragma unroll
            for (int j = 0; j < CH; j += 8) {
                tmem_ld8(ta + j, *reinterpret_cast<uint32_t(*)[8]>(&a[j]));
                tmem_ld8(ta + NT + j, *reinterpret_cast<uint32_t(*)[8]>(&b[j]));
            }
            tmem_ld_wait();
            if constexpr (NT <= 64) {
                // triples: the third sum; pairs: the sums of the odd steps (a block has eight of them at least, or the whole of four)
                uint32_t c[CH];
#pragma unroll
                for (int j = 0; j < CH; j += 8) tmem_ld8(ta + 2 * NT + j, *reinterpret_cast<uint32_t(*)[8]>(&c[j]));
                tmem_ld_wait();
                uint32_t (&to)[CH] = wide ? b : a;
#pragma unroll
                for (int j = 0; j < CH; ++j) to[j] = __float_as_uint(__uint_as_float(to[j]) + __uint_as_float(c[j]));
                if (!wide) {
#pragma unroll
                    for (int j = 0; j < CH; j += 8) tmem_ld8(ta + 3 * NT + j, *reinterpret_cast<uint32_t(*)[8]>(&c[j]));
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < CH; ++j) b[j] = __float_as_uint(__uint_as_float(b[j]) + __uint_as_float(c[j]));
                }
            }
            const float low = wide ? 1.0f : 1.0f / kDxLow;
#pragma unroll
            for (int j = 0; j < CH; ++j) {
                const float v = fmaf(__uint_as_float(b[j]), low, __uint_as_float(a[j]));
                const int tok = tok0 + col + j;
                // (both exponents at once: one of them alone can take a finite result through infinity or zero)
                if (p.split > 1) s_out[(col + j) * 128 + blk * 32 + 4 * (lane & 7) + (lane >> 3)] = v;
                else if (tok < p.m && i_ok) p.dx[(int64_t)tok * p.in + i] = dx_scale(v, ce + exp_of(tok));
            }
        }
    }
    if (p.split > 1) {
        // The blocks of the cluster add their ranges of o through distributed shared memory, always in the same
        // order, each for its share of the tile's tokens.
        __syncwarp();
        cluster_sync();
        const int per = NT / p.split;
        if (warp < kDxDq && ok) {
            for (int e = tid; e < per * 128; e += kDxDq * 32) {
                const int row = part * per + (e >> 7), c = e & 127, tok = tok0 + row;
                const uint32_t at = sbase + (uint32_t)(row * 128 + c) * 4;
                float v = 0.f;
                for (int r = 0; r < p.split; ++r) {
                    uint32_t ra;
                    float x;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(at), "r"(r));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(ra) : "memory");
                    v += x;
                }
                const int64_t i = (int64_t)ft * 128 + c;
                if (tok < p.m && i < p.in)
                    p.dx[(int64_t)tok * p.in + i] = dx_scale(v, s_colexp[c >> 5] + exp_of(tok));
            }
        }
        __syncwarp();
        cluster_sync();   // nobody leaves while its shared memory is read
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kDxDq + 1) tmem_dealloc(tmem, 512);
    if (tid == 0 && s_abort) atomicExch(p.status, 2);
}

// dims, box: innermost first; strides: bytes between rows and, of three dimensions, planes
static bool dx_map(EncodeTiledFn enc, CUtensorMap* map, CUtensorMapDataType type, const void* base, int rank, const cuuint64_t (&dims)[3],
                   const cuuint64_t (&strides)[2], const cuuint32_t (&box)[3], bool swizzle = true) {
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(map, type, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static constexpr int dx_smem_bytes(int nt) { return dx_ring_bytes(nt) + 1024; }

int32_t dx_configure() {
    RSTQ_CUDA(cudaFuncSetAttribute(dx_tmem_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, dx_smem_bytes(32)));
    RSTQ_CUDA(cudaFuncSetAttribute(dx_tmem_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, dx_smem_bytes(64)));
    RSTQ_CUDA(cudaFuncSetAttribute(dx_tmem_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, dx_smem_bytes(128)));
    return RSTQ_OK;
}

template <int NT>
static cudaError_t dx_launch(const DeviceState& ds, const DxParams& p, int tiles, const CUtensorMap& w, const CUtensorMap& y,
                             const CUtensorMap& y16, const CUtensorMap& s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * p.split));
    cfg.blockDim = dim3(kDxThreads);
    cfg.dynamicSmemBytes = dx_smem_bytes(NT);
    cfg.stream = ds.stream;
    cudaLaunchAttribute a[2];
    int n = 0;
    if (p.split > 1) {
        a[n].id = cudaLaunchAttributeClusterDimension;
        a[n].val.clusterDim.x = (unsigned)p.split;
        a[n].val.clusterDim.y = a[n].val.clusterDim.z = 1;
        ++n;
    }
    if (ds.pdl) {
        a[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        a[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = a;
    cfg.numAttrs = (unsigned)n;
    return cudaLaunchKernelEx(&cfg, dx_tmem_kernel<NT>, p, w, y, y16, s);
}

int32_t launch_qlinear_q8_dx(rstq_ctx* ctx, DeviceState& ds, const float* dy, const int8_t* codes,
                             const float* scales, float* dx, int64_t m, int64_t in, int64_t out) {
    EncodeTiledFn enc = encode_tiled_fn();
    RSTQ_REQUIRE(enc, RSTQ_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    const int64_t nb = in / 32, steps = (out + kDxStep - 1) / kDxStep, opad = steps * kDxStep, ftiles = (in + 127) / 128;
    // Tile width: MMAs of fewer than 128 tokens cost their issue (50 - 60 cycles), so narrow tiles only save
    // work for padding below 128 tokens.
    const int nt = m <= 32 ? 32 : (m <= 64 ? 64 : 128);
    const int64_t ttiles = (m + nt - 1) / nt, tiles = ftiles * ttiles;
    RSTQ_REQUIRE(m < (1ll << 30) && tiles < (1ll << 28) && in < (1ll << 31) && out < (1ll << 31), RSTQ_E_LIMIT,
                 "m = %lld, in = %lld, out = %lld too large for one launch", (long long)m, (long long)in, (long long)out);
    // Tiles that leave half the SMs idle are shared by a cluster of 2, 4 or 8 blocks, each with at least eight
    // stages of its own (below that the set-up and the exchange cost what the shorter loop gains).
    int split = 1;
    while (split < 8 && tiles * split * 2 <= ds.sm_count && steps >= 16 * split) split *= 2;

    const int64_t yb = (3 * m * opad * 2 + 255) & ~255ll, hb = (2 * m * opad * 2 + 255) & ~255ll, rb = (m * 4 + 255) & ~255ll;
    const int64_t cb = 2 * kDxParts * nb * 4;
    int32_t rc = dx_reserve(ds, yb + hb + rb + cb);
    if (rc != RSTQ_OK) return rc;
    char* base = (char*)ds.dx_scratch;
    DxPrep q{dy, scales, (uint16_t*)base, (uint16_t*)(base + yb), (int*)(base + yb + hb), (float*)(base + yb + hb + rb), m, out, nb, opad};
    CUtensorMap mw, my, mh, ms;
    const bool tma_scales = nb % 4 == 0;   // rows of whole 16 bytes
    const cuuint64_t i_ = (cuuint64_t)in, o_ = (cuuint64_t)out, m_ = (cuuint64_t)m, op_ = (cuuint64_t)opad, nb_ = (cuuint64_t)nb;
    RSTQ_REQUIRE(dx_map(enc, &mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, codes, 2, {i_, o_, 1}, {i_, 0}, {128, kDxStep, 1}) &&
                     dx_map(enc, &my, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, q.y, 3, {op_, m_, 3}, {op_ * 2, op_ * m_ * 2},
                            {kDxStep, (cuuint32_t)nt, 3}) &&
                     dx_map(enc, &mh, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, q.y16, 3, {op_, m_, 2}, {op_ * 2, op_ * m_ * 2},
                            {kDxStep, (cuuint32_t)nt, 2}) &&
                     (!tma_scales || dx_map(enc, &ms, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, scales, 2, {nb_, o_, 1}, {nb_ * 4, 0},
                                            {4, kDxStep, 1}, false)),
                 RSTQ_E_CUDA, "cuTensorMapEncodeTiled failed (m = %lld, in = %lld, out = %lld)", (long long)m, (long long)in,
                 (long long)out);
    if (!tma_scales) ms = mw;   // not used then
    RSTQ_CUDA(launch_pdl(dx_prep_kernel, dim3((unsigned)(m + kDxParts)), dim3(opad > 4096 ? kDxPrepMax : opad > 2048 ? 256 : 128), 0, ds, q));
    ctx->launches++;
    DxParams p{scales, q.rowexp, q.colmax, dx, ds.status, in, out, tma_scales, (int)m, (int)steps, (int)ttiles, split};
    RSTQ_CUDA(nt == 32   ? dx_launch<32>(ds, p, (int)tiles, mw, my, mh, ms)
              : nt == 64 ? dx_launch<64>(ds, p, (int)tiles, mw, my, mh, ms)
                         : dx_launch<128>(ds, p, (int)tiles, mw, my, mh, ms));
    ctx->launches++;
    return RSTQ_OK;
}

}  // namespace rstq
