// Host-side weight codecs: quantize-weight (src/raster/compiler/backend/cpu/quant.clj:42-70),
// quantize-weight-q4k (:95-150) and quantize-weight-q6k (:222-262), over flat f32 arrays.
//
// Load-time work on host memory, bit for bit the double-precision arithmetic of the reference (divide,
// reciprocal, multiply, round half up, clamp).  What bounds it: for q4_0 and q8_0 the read of the f32 matrix and the
// first touch of the results, for the K-quants the double arithmetic of a block (4 ns per element and core); blocks are
// independent, so the array is cut over the host's cores.
// Only finite inputs are taken, and of q4_K only minima that do not dwarf their block's spread: the callers keep the
// general path for the rest (return value 1).
//
// Compiled for AVX2 (on x86) and for the base architecture, without contraction into fused multiply-adds: a contracted
// product would round differently from the reference's two steps.
// (no trapping math: comparisons may then be turned into masks; results do not change)
#pragma GCC optimize("no-trapping-math", "fp-contract=off")
#include <math.h>
#include <string.h>
#if defined(__x86_64__) && !defined(RSTQ_NO_AVX2)
#include <immintrin.h>
#endif

#include <thread>
#include <vector>

#include "internal.h"

namespace rstq {

#if defined(__x86_64__) && !defined(RSTQ_NO_AVX2)
#define RSTQ_AVX2 __attribute__((target("avx2")))
#define RSTQ_HAS_AVX2() ((bool)__builtin_cpu_supports("avx2"))
#else   // other hosts: the base architecture's form alone
#define RSTQ_AVX2
#define RSTQ_HAS_AVX2() false
#endif
#define RSTQ_INLINE static inline __attribute__((always_inline))

// Math.round of v (nearest integer, ties upward) for |v| < 2^31: v - trunc(v) is exact, so the two
// comparisons decide exactly as floor(v) and its remainder do.
// (clamped, and all in double: one lane width throughout, so the loops over a block vectorize)
RSTQ_INLINE int round_clamp(double v, double zp, double lo, double hi) {
    const double i = (double)(int)v, f = v - i;
    double q = i + (f >= 0.5 ? 1.0 : 0.0) - (f < -0.5 ? 1.0 : 0.0) + zp;
    q = q < lo ? lo : q;
    q = q > hi ? hi : q;
    return (int)q;
}
// Largest magnitude of n values (n % 8 == 0); false when one is an infinity or a NaN.  The bits of
// magnitudes order like the magnitudes, and their integer maximum vectorizes.
RSTQ_INLINE bool largest(const float* w, int n, float* mx) {
    uint32_t m[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = 0; i < n; i += 8)
        for (int j = 0; j < 8; ++j) {
            uint32_t b;
            memcpy(&b, w + i + j, 4);
            b &= 0x7FFFFFFFu;
            m[j] = b > m[j] ? b : m[j];
        }
    uint32_t worst = 0;
    for (int j = 0; j < 8; ++j) worst = m[j] > worst ? m[j] : worst;
    memcpy(mx, &worst, 4);
    return worst < 0x7F800000u;
}
// 32 codes -> element k in the low, element k + 16 in the high nibble of byte k
RSTQ_INLINE void put_nibbles(const int (&q)[32], uint8_t* dst) {
    for (int k = 0; k < 16; ++k) dst[k] = (uint8_t)(q[k] | (q[k + 16] << 4));
}

// One 32-element block of q4_0 / q8_0.
RSTQ_INLINE bool block_plain(const float* w, uint8_t* codes, float* scale, int bits) {
    float mx;
    if (!largest(w, 32, &mx)) return false;
    int at = 0;
    while (fabsf(w[at]) != mx) ++at;   // the first element of largest magnitude
    const double zp = bits == 4 ? 8.0 : 128.0, top = bits == 4 ? 15.0 : 255.0;
    const double d = (double)w[at] / -zp, inv = d == 0.0 ? 0.0 : 1.0 / d;
    int q[32];
    for (int k = 0; k < 32; ++k) q[k] = round_clamp((double)w[k] * inv, zp, 0.0, top);
    if (bits == 4) put_nibbles(q, codes);
    else
        for (int k = 0; k < 32; ++k) codes[k] = (uint8_t)q[k];
    *scale = (float)d;
    return true;
}

#if defined(__x86_64__) && !defined(RSTQ_NO_AVX2)
// The same with the codes from f32 arithmetic where that provably gives the double result: t = x * fl32(1 / d) lies within
// 128 * 2^-23 of the double product (a rounding of the reciprocal, one of the product), so a t further than 1e-4 from
// every tie rounds the same way.  A block with one that is not, or whose scale leaves the normal f32 range, takes
// block_plain.  (Left to the compiler, these loops come out scalar: 2.7 - 3.0 ns per element and core, 0.7 so;
// 4096 x 4096 on 8 cores of one host 8.6 -> 3.8 ms, the rest the read of the f32 matrix and the pages of the results.)
template <int BITS>
RSTQ_AVX2 static inline bool block_plain_avx2(const float* w, uint8_t* codes, float* scale) {
    const __m256 sign = _mm256_set1_ps(-0.0f);
    __m256 x[4], a[4];
    for (int j = 0; j < 4; ++j) {
        x[j] = _mm256_loadu_ps(w + 8 * j);
        a[j] = _mm256_andnot_ps(sign, x[j]);
    }
    // (the bits of magnitudes order like the magnitudes)
    __m256i m = _mm256_max_epi32(_mm256_max_epi32(_mm256_castps_si256(a[0]), _mm256_castps_si256(a[1])),
                                 _mm256_max_epi32(_mm256_castps_si256(a[2]), _mm256_castps_si256(a[3])));
    m = _mm256_max_epi32(m, _mm256_permute2x128_si256(m, m, 1));
    m = _mm256_max_epi32(m, _mm256_shuffle_epi32(m, 0x4E));
    m = _mm256_max_epi32(m, _mm256_shuffle_epi32(m, 0xB1));
    const int bits = _mm256_cvtsi256_si32(m);
    if (bits >= 0x7F800000) return false;
    float mx;
    memcpy(&mx, &bits, 4);
    if (!(mx >= 1e-30f && mx <= 1e30f)) return block_plain(w, codes, scale, BITS);
    uint32_t at = 0;      // the elements of largest magnitude
    for (int j = 0; j < 4; ++j)
        at |= (uint32_t)_mm256_movemask_ps(_mm256_castsi256_ps(_mm256_cmpeq_epi32(_mm256_castps_si256(a[j]), m))) << (8 * j);
    constexpr int zp = BITS == 4 ? 8 : 128, top = BITS == 4 ? 15 : 255;
    const double d = (double)w[__builtin_ctz(at)] / -(double)zp;
    const __m256 inv = _mm256_set1_ps((float)(1.0 / d)), magic = _mm256_set1_ps(12582912.0f), edge = _mm256_set1_ps(0.4999f);
    const __m256i shift = _mm256_set1_epi32(zp - 0x4B400000), most = _mm256_set1_epi32(top);
    __m256 near = _mm256_setzero_ps();
    __m256i q[4];
    for (int j = 0; j < 4; ++j) {
        const __m256 t = _mm256_mul_ps(x[j], inv), r = _mm256_add_ps(t, magic);    // 2^23 + 2^22: rounds to the nearest integer
        near = _mm256_or_ps(near, _mm256_cmp_ps(_mm256_andnot_ps(sign, _mm256_sub_ps(t, _mm256_sub_ps(r, magic))), edge, _CMP_GT_OQ));
        q[j] = _mm256_add_epi32(_mm256_castps_si256(r), shift);
        q[j] = _mm256_min_epi32(_mm256_max_epi32(q[j], _mm256_setzero_si256()), most);
    }
    if (_mm256_movemask_ps(near)) return block_plain(w, codes, scale, BITS);
    const __m256i order = _mm256_setr_epi32(0, 4, 1, 5, 2, 6, 3, 7);
    if (BITS == 8) {
        const __m256i p = _mm256_packus_epi16(_mm256_packs_epi32(q[0], q[1]), _mm256_packs_epi32(q[2], q[3]));
        _mm256_storeu_si256((__m256i*)codes, _mm256_permutevar8x32_epi32(p, order));
    } else {              // element k in the low, k + 16 in the high nibble of byte k
        const __m256i b = _mm256_packs_epi32(_mm256_or_si256(q[0], _mm256_slli_epi32(q[2], 4)), _mm256_or_si256(q[1], _mm256_slli_epi32(q[3], 4)));
        _mm_storeu_si128((__m128i*)codes, _mm256_castsi256_si128(_mm256_permutevar8x32_epi32(_mm256_packus_epi16(b, b), order)));
    }
    *scale = (float)d;
    return true;
}
#endif

RSTQ_INLINE double maxd(double a, double b) { return a > b ? a : b; }

// One 256-element super-block of q4_K: eight sub-blocks of 32 with a 6-bit scale and minimum.
RSTQ_INLINE bool block_q4k(const float* w, uint8_t* wq, float* da, float* db, int8_t* aq, int8_t* bq) {
    float mx;
    if (!largest(w, 256, &mx)) return false;
    double a[8], b[8], amax = 0.0, bmax = 0.0;
    for (int s = 0; s < 8; ++s) {
        float l8[8], h8[8];
        for (int j = 0; j < 8; ++j) l8[j] = h8[j] = w[s * 32 + j];
        for (int k = 8; k < 32; k += 8)
            for (int j = 0; j < 8; ++j) {
                const float v = w[s * 32 + k + j];
                l8[j] = v < l8[j] ? v : l8[j];
                h8[j] = v > h8[j] ? v : h8[j];
            }
        float lo = l8[0], hi = h8[0];
        for (int j = 1; j < 8; ++j) {
            lo = l8[j] < lo ? l8[j] : lo;
            hi = h8[j] > hi ? h8[j] : hi;
        }
        a[s] = ((double)hi - (double)lo) / 15.0;
        b[s] = (double)lo;
        amax = maxd(amax, a[s]);
        bmax = maxd(bmax, fabs(b[s]));
    }
    const double dav = amax / 63.0, dbv = bmax / 31.0;
    const double ida = dav == 0.0 ? 0.0 : 1.0 / dav, idb = dbv == 0.0 ? 0.0 : 1.0 / dbv;
    for (int s = 0; s < 8; ++s) {
        const int ai = round_clamp(a[s] * ida, 0.0, 0.0, 63.0), bi = round_clamp(b[s] * idb, 0.0, -32.0, 31.0);
        const double a1 = dav * (double)ai, b1 = dbv * (double)bi, ia1 = a1 == 0.0 ? 0.0 : 1.0 / a1;
        // beyond the integer range of the rounding (a minimum that dwarfs the spread): the general path
        if (!(((double)mx + fabs(b1)) * ia1 < 2147483000.0)) return false;
        int q[32];
        for (int k = 0; k < 32; ++k) q[k] = round_clamp(((double)w[s * 32 + k] - b1) * ia1, 0.0, 0.0, 15.0);
        put_nibbles(q, wq + s * 16);
        aq[s] = (int8_t)ai;
        bq[s] = (int8_t)bi;
    }
    *da = (float)dav;
    *db = (float)dbv;
    return true;
}

// One 256-element super-block of q6_K: sixteen sub-blocks of 16 with an integer scale.
RSTQ_INLINE bool block_q6k(const float* w, uint8_t* wq, int8_t* sc, float* ds) {
    double a[16], amax = 0.0;
    for (int s = 0; s < 16; ++s) {
        float mx;
        if (!largest(w + s * 16, 16, &mx)) return false;
        a[s] = (double)mx / 32.0;
        amax = maxd(amax, a[s]);
    }
    const double dv = amax / 127.0, idv = dv == 0.0 ? 0.0 : 1.0 / dv;
    for (int s = 0; s < 16; ++s) {
        const int si = round_clamp(a[s] * idv, 0.0, 0.0, 127.0);
        const double a1 = dv * (double)si, ia1 = a1 == 0.0 ? 0.0 : 1.0 / a1;
        int q[16];
        for (int k = 0; k < 16; ++k) q[k] = round_clamp((double)w[s * 16 + k] * ia1, 32.0, 0.0, 63.0);
        for (int k = 0; k < 16; ++k) wq[s * 16 + k] = (uint8_t)q[k];
        sc[s] = (int8_t)si;
    }
    *ds = (float)dv;
    return true;
}

// Ranges of blocks, per instruction set.
struct PlainJob {
    const float* w;
    uint8_t* codes;
    float* scales;
    int bits;
    template <int BITS>
    RSTQ_INLINE bool range(const PlainJob& j, int64_t b0, int64_t b1) {
        for (int64_t b = b0; b < b1; ++b)
            if (!block_plain(j.w + b * 32, j.codes + b * (4 * BITS), j.scales + b, BITS)) return false;
        return true;
    }
#if defined(__x86_64__) && !defined(RSTQ_NO_AVX2)
    template <int BITS>
    RSTQ_AVX2 static bool range_avx2(const PlainJob& j, int64_t b0, int64_t b1) {
        for (int64_t b = b0; b < b1; ++b)
            if (!block_plain_avx2<BITS>(j.w + b * 32, j.codes + b * (4 * BITS), j.scales + b)) return false;
        return true;
    }
    bool avx2(int64_t b0, int64_t b1) const { return bits == 4 ? range_avx2<4>(*this, b0, b1) : range_avx2<8>(*this, b0, b1); }
#else
    bool avx2(int64_t b0, int64_t b1) const { return base(b0, b1); }
#endif
    bool base(int64_t b0, int64_t b1) const { return bits == 4 ? range<4>(*this, b0, b1) : range<8>(*this, b0, b1); }
};
struct Q4kJob {
    const float* w;
    uint8_t* wq;
    float *da, *db;
    int8_t *aq, *bq;
    RSTQ_INLINE bool range(const Q4kJob& j, int64_t b0, int64_t b1) {
        for (int64_t b = b0; b < b1; ++b)
            if (!block_q4k(j.w + b * 256, j.wq + b * 128, j.da + b, j.db + b, j.aq + b * 8, j.bq + b * 8)) return false;
        return true;
    }
    RSTQ_AVX2 bool avx2(int64_t b0, int64_t b1) const { return range(*this, b0, b1); }
    bool base(int64_t b0, int64_t b1) const { return range(*this, b0, b1); }
};
struct Q6kJob {
    const float* w;
    uint8_t* wq;
    int8_t* sc;
    float* ds;
    RSTQ_INLINE bool range(const Q6kJob& j, int64_t b0, int64_t b1) {
        for (int64_t b = b0; b < b1; ++b)
            if (!block_q6k(j.w + b * 256, j.wq + b * 256, j.sc + b * 16, j.ds + b)) return false;
        return true;
    }
    RSTQ_AVX2 bool avx2(int64_t b0, int64_t b1) const { return range(*this, b0, b1); }
    bool base(int64_t b0, int64_t b1) const { return range(*this, b0, b1); }
};

// fn(begin, end) over [0, n) on the host's cores, at least `least` items a thread (a thread costs about
// 20 us to start: less work than that is not worth one); the caller takes the first part itself.
void host_parallel(int64_t n, int64_t least, void (*fn)(void*, int, int64_t, int64_t), void* arg) {
    int64_t t = std::thread::hardware_concurrency();
    if (t > 32) t = 32;
    if (t > n / least) t = n / least;
    if (t < 1) t = 1;
    std::vector<std::thread> extra;
    int64_t from = n / t;
    try {
        for (int64_t i = 1; i < t; ++i) {
            const int64_t to = n * (i + 1) / t;
            extra.emplace_back(fn, arg, (int)i, from, to);
            from = to;
        }
    } catch (...) {      // no thread to be had: this one does the rest
        fn(arg, 0, from, n);
    }
    fn(arg, 0, 0, n / t);
    for (auto& e : extra) e.join();
}

// Largest scale magnitude below 3e38 (infinities and NaNs do not count).
float largest_scale(const float* s, int64_t n) {
    float m[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int64_t n8 = n & ~7ll;
    for (int64_t i = 0; i < n8; i += 8)
        for (int j = 0; j < 8; ++j) {
            float a = fabsf(s[i + j]);
            a = a < 3.0e38f ? a : 0.f;
            m[j] = a > m[j] ? a : m[j];
        }
    for (int64_t i = n8; i < n; ++i) {
        const float a = fabsf(s[i]);
        if (a < 3.0e38f && a > m[0]) m[0] = a;
    }
    float mx = m[0];
    for (int j = 1; j < 8; ++j) mx = m[j] > mx ? m[j] : mx;
    return mx;
}

template <typename Job>
static int32_t run_codec(const Job& job, int64_t blocks, int64_t block_elems) {
    struct Arg {
        const Job* job;
        bool avx2;
        int bad[33];
    } arg{&job, RSTQ_HAS_AVX2(), {0}};
    host_parallel(blocks, 65536 / block_elems, [](void* p, int slot, int64_t b0, int64_t b1) {
        Arg& a = *(Arg*)p;
        const bool ok = a.avx2 ? a.job->avx2(b0, b1) : a.job->base(b0, b1);
        if (!ok) a.bad[slot] = 1;
    }, &arg);
    for (int b : arg.bad)
        if (b) return 1;
    return RSTQ_OK;
}

}  // namespace rstq

using namespace rstq;

extern "C" {

int32_t rstq_quantize_weight(const float* w, void* codes, float* scales, int64_t n, int32_t format) {
    RSTQ_REQUIRE(w && codes && scales, RSTQ_E_INVALID, "null argument");
    RSTQ_REQUIRE(format == RSTQ_FMT_Q4_0 || format == RSTQ_FMT_Q8_0, RSTQ_E_INVALID, "no codec for format %d", format);
    RSTQ_REQUIRE(n >= 0 && n % 32 == 0, RSTQ_E_SHAPE, "n = %lld is not a multiple of 32", (long long)n);
    return run_codec(PlainJob{w, (uint8_t*)codes, scales, format == RSTQ_FMT_Q4_0 ? 4 : 8}, n / 32, 32);
}

int32_t rstq_quantize_weight_q4k(const float* w, void* wq, float* da, float* db, int8_t* aq, int8_t* bq, int64_t n) {
    RSTQ_REQUIRE(w && wq && da && db && aq && bq, RSTQ_E_INVALID, "null argument");
    RSTQ_REQUIRE(n >= 0 && n % 256 == 0, RSTQ_E_SHAPE, "n = %lld is not a multiple of 256", (long long)n);
    return run_codec(Q4kJob{w, (uint8_t*)wq, da, db, aq, bq}, n / 256, 256);
}

int32_t rstq_quantize_weight_q6k(const float* w, void* wq, int8_t* sc, float* ds, int64_t n) {
    RSTQ_REQUIRE(w && wq && sc && ds, RSTQ_E_INVALID, "null argument");
    RSTQ_REQUIRE(n >= 0 && n % 256 == 0, RSTQ_E_SHAPE, "n = %lld is not a multiple of 256", (long long)n);
    return run_codec(Q6kJob{w, (uint8_t*)wq, sc, ds}, n / 256, 256);
}

}  // extern "C"
