// Prefill-shape (M > 16) dequant-fused GEMM on the 5th-generation tensor cores.
//
// Replaces qmatmul-i8-gemm! (src/raster/quant/kernels_k.clj:344-370) and
// qlinear-q8 at large M (src/raster/quant/train.clj:77-108): where the
// reference runs one work-item per (token, output) with a serial K loop, this
// is a tiled tcgen05 GEMM:
//
//   D[128 features, NTOK tokens] (f32, in tensor memory)
//       += A[128, 128] (fp16, dequantized weights) * B[NTOK, 128]^T (fp16 activations)
//
//  * A is produced on the fly: 16 warps read the packed 4/8-bit codes and f32
//    block scales of the mma32 layout straight from global memory (register
//    prefetch four K-steps ahead, behind requests into L2 eight more ahead),
//    turn code and block scale into fp16 (exact integers times the rounded
//    scale) and hand them to the tensor core: gemm_tmem_kernel, the default,
//    stores them into a ring in tensor memory; gemm_tc_kernel stores 16-byte
//    rows into shared memory in the K-major 128-byte-swizzled layout.  fp16
//    (11-bit significand) rather than bf16 keeps the result within 1e-3 of the
//    f32 reference; a per-matrix power of two keeps scaled weights in fp16 range.
//  * B comes from a small pre-pass that rewrites the activations as fp16 with
//    one power-of-two exponent per token row (exact for bf16 inputs), loaded by
//    TMA (cp.async.bulk.tensor, 128-byte swizzle) by one producer thread.
//  * One thread (gemm_tmem_kernel: one of two, on alternate K-steps) issues
//    tcgen05.mma (cta_group::1, kind::f16, M = 128, N = NTOK, K = 16 per
//    instruction); tcgen05.commit releases a stage to the producers.
//  * The 16 dequant warps then read the accumulator with tcgen05.ld, undo the two
//    exponents and store y (f32 or bf16) row-major [token, feature].
// Every mbarrier wait is time-bounded; on expiry the CTA reports through the
// status word, drains and still frees its tensor memory.

#include <algorithm>
#include <type_traits>

#include "internal.h"
#include "mma_helpers.cuh"
#include "quant_helpers.cuh"
#include "sync_helpers.cuh"
#include "tcgen05_helpers.cuh"

namespace rstq {

constexpr int kDqWarps = 16;
constexpr int kGemmThreads = (2 + kDqWarps) * 32;  // TMA warp, MMA warp, 16 dequant/epilogue warps
constexpr int kKStep = 128;                        // K elements per pipeline stage (4 blocks)
constexpr int kAStage = 128 * kKStep * 2;          // 32 KB of fp16 weights per stage
constexpr int kPrefetch = 4;                       // K-steps of packed weights held in registers

// Eight elements of a 32-element block, the block's other three eighths in the neighbouring lanes (lane & ~3):
// replaced by code * scale of the int8 quantizer, as quant_block32 (quant_helpers.cuh) forms them.
__device__ __forceinline__ void quant_dequant8(float (&v)[8]) {
    constexpr float kMagic = 12582912.0f;   // 2^23 + 2^22
    const unsigned mask = 0xFu << (threadIdx.x & 28);
    float mx = fabsf(v[0]);
#pragma unroll
    for (int j = 1; j < 8; ++j) mx = fmaxf(mx, fabsf(v[j]));
    mx = fmaxf(mx, __shfl_xor_sync(mask, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(mask, mx, 2));
    bool exact = !(mx >= 1e-30f && mx <= 1e37f);
    if (!exact) {
        const float id = __fdividef(127.f, mx), xs = __fdiv_rn(mx, 127.f);
        float code[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            code[j] = fmaf(v[j], id, kMagic) - kMagic;
            exact |= !(fabsf(fmaf(v[j], id, -code[j])) <= kQuantSure);
        }
        if (!exact) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = code[j] * xs;
            return;
        }
    }
    const double d = (double)mx / 127.0;
    const double id = d == 0.0 ? 0.0 : 1.0 / d;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = (float)max(-127, min(127, quant_round_half_up((double)v[j] * id))) * (float)d;
}

// ---- activation pre-pass: x (f32 / bf16, as it is or int8-quantized) -> fp16 * 2^-e(row) ---
// One CTA per token row.  rowscale[m] = 2^e so that max|x| * 2^-e lies in [2^13, 2^14).
// SRC 2, 3: the int8 quantizer on the way (MODE_A8): code * scale of every element, without the quantizer's own
// launch and its arrays' trip through memory (int4, 11000 x 4128, M = 100: 26.9 us a call with both kernels, 23.1
// with one; 14336 x 4096, M = 64: 22.4 -> 19.9).
template <int SRC, int T>  // 0 = f32, 1 = bf16, 2 = f32 quantized here, 3 = bf16 quantized here
__global__ void __launch_bounds__(T)
act_to_f16_kernel(const void* __restrict__ x, __half* __restrict__ x16,
                  float* __restrict__ rowscale, int64_t in) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t m = blockIdx.x;
    // eight consecutive elements (one 16-byte fp16 store) per thread and step
    auto load8 = [&](int64_t k, float (&v)[8]) {
        if (SRC == 0 || SRC == 2) {
            const float4* q = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + m * in + k);
            const float4 a = __ldg(q), b = __ldg(q + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(x) + m * in + k));
            const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[2 * j] = __uint_as_float(w[j] << 16);
                v[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
            }
        }
        if (SRC >= 2) quant_dequant8(v);
    };
    // Rows of up to 32 T elements stay in registers between the two passes (max, convert); longer rows are read twice.
    constexpr int kKeep = 4;  // x T threads x 8 elements
    const bool keep = in <= (int64_t)kKeep * T * 8;
    float held[kKeep][8];
    float mx = 0.f;
    if (keep) {
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int64_t k = (int64_t)(i * T + threadIdx.x) * 8;
            if (k < in) {
                load8(k, held[i]);
#pragma unroll
                for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(held[i][j]));
            }
        }
    } else {
        for (int64_t k = threadIdx.x * 8; k < in; k += T * 8) {
            float v[8];
            load8(k, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(v[j]));
        }
    }
    __shared__ float s_mx[T / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) s_mx[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = s_mx[0];
#pragma unroll
    for (int i = 1; i < T / 32; ++i) mx = fmaxf(mx, s_mx[i]);
    int e = 0;
    if (mx > 0.f && mx < 3.0e38f) {
        int ex;
        frexpf(mx, &ex);  // mx = f * 2^ex, f in [0.5, 1)
        e = ex - 14;
    }
    const float down = ldexpf(1.0f, -e);
    auto store8 = [&](int64_t k, const float (&v)[8]) {
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __half2 t = __floats2half2_rn(v[2 * j] * down, v[2 * j + 1] * down);
            h[j] = *reinterpret_cast<const uint32_t*>(&t);
        }
        *reinterpret_cast<uint4*>(x16 + m * in + k) = make_uint4(h[0], h[1], h[2], h[3]);
    };
    if (keep) {
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int64_t k = (int64_t)(i * T + threadIdx.x) * 8;
            if (k < in) store8(k, held[i]);
        }
    } else {
        for (int64_t k = threadIdx.x * 8; k < in; k += T * 8) {
            float v[8];
            load8(k, v);
            store8(k, v);
        }
    }
    if (threadIdx.x == 0) rowscale[m] = ldexpf(1.0f, e);
}

// ---- the GEMM kernel ---------------------------------------------------------------------
constexpr int kNST = 3;  // pipeline stages

struct GemmParams {
    const uint8_t* w;       // mma32 units
    void* y;                // [M, out] f32 or bf16
    const float* rowscale;  // 2^e per token row (activation pre-pass)
    int* status;
    int64_t out;            // output features
    int nb, ngroups;        // K blocks per row, 32-row groups stored
    int M, ksteps, ttiles;  // ksteps: K-steps of a tile
    // gemm_tmem_kernel: the K-steps of all tiles, tile after tile, are one sequence and CTA c runs the range
    // [range_start(c), range_start(c + 1)) of it
    int64_t uq, ur;         // uq steps each, the first ur CTAs one more
    int half;               // > 0 instead: two CTAs per tile, the first runs the tile's first `half` steps
    int parts;              // > 0 instead: that many CTAs per tile, each an equal part of its steps
    float* part;            // a range that begins inside a tile leaves that tile's f32 sums here ([CTA][warp][column]
                            // [lane]); the CTA that holds the tile's first step adds them to its own and stores y
    int* part_flags;        // one word per CTA, zero between launches: set when its `part` is complete
    float wmul, wdiv;       // 2^ew applied to the block scales, 2^-ew applied to the result
    int out_dtype;
    int cols;               // columns of a tile that are computed (pairs of CTAs: a multiple of 32)
    unsigned long long* dbg;  // optional timeline of CTA 0 (see RSTQ_TUNE_TIMELINE), or null
};

// packed weights of one dequant task, as loaded from global memory
template <int BITS>
struct RawW;
template <>
struct RawW<4> {
    uint2 a, b;  // slot 2t', 2t'+1: words (2q, 2q+1)
    float2 s;    // scales of rows gid + 16q, gid + 16q + 8
};
template <>
struct RawW<8> {
    uint4 a, b;  // plane p, slot 2t', 2t'+1: rows gid + 8i
    float4 s;
};

__device__ __forceinline__ uint32_t hsub_hmul(uint32_t v, uint32_t off, uint32_t scale2) {
    __half2 h = *reinterpret_cast<__half2*>(&v);
    h = __hmul2(__hsub2(h, *reinterpret_cast<__half2*>(&off)), *reinterpret_cast<__half2*>(&scale2));
    return *reinterpret_cast<uint32_t*>(&h);
}
// four unsigned bytes (each < 256) -> four fp16 (value - zero) * scale, in byte order
__device__ __forceinline__ uint2 bytes_to_h4(uint32_t bytes, uint32_t off, uint32_t scale2) {
    uint2 r;
    r.x = hsub_hmul(__byte_perm(bytes, 0x64646464u, 0x4140), off, scale2);
    r.y = hsub_hmul(__byte_perm(bytes, 0x64646464u, 0x4342), off, scale2);
    return r;
}
__device__ __forceinline__ uint32_t scale_h2(float s) {
    __half2 h = __half2half2(__float2half_rn(s));
    return *reinterpret_cast<uint32_t*>(&h);
}

// The conversion of gemm_tmem_kernel: one fused multiply-add per pair of weights.  A byte b placed
// in the low byte of a half (0x00bb) IS the fp16 subnormal b * 2^-24, so
//     fma(0x00bb, s, -zero * 2^-24 * s) = (b - zero) * s * 2^-24, rounded once:
// the product is exact inside the fma and the addend, a power of two times the already rounded
// scale s, is exact as well, which makes the result the same bits as subtracting the zero point
// first (exact integers) and multiplying by s afterwards, in half the instructions.  The caller
// folds the 2^-24 into the scale.
// bytes 0..3 of `bytes` (other bits of each byte pair must be zero) -> four halves v * scale + add
__device__ __forceinline__ uint2 bytes_fma_h4(uint32_t bytes, uint32_t scale2, uint32_t add2) {
    uint2 r;
    r.x = hfma2_u32(__byte_perm(bytes, 0u, 0x4140), scale2, add2);
    r.y = hfma2_u32(__byte_perm(bytes, 0u, 0x4342), scale2, add2);
    return r;
}
constexpr int kSubnormalShift = 8;  // block scales carry 2^8 more: code * 2^-24 * (s * 2^8) stays in fp16 range

template <int BITS, int NTOK>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tc_kernel(const GemmParams p, const __grid_constant__ CUtensorMap tmap) {
    constexpr int UNIT = BITS == 4 ? kUnitBytesQ4 : kUnitBytesQ8;
    constexpr int CODES = BITS == 4 ? kUnitCodesQ4 : kUnitCodesQ8;
    constexpr int BSTAGE = NTOK * kKStep * 2;
    constexpr int STAGE = kAStage + BSTAGE;
    constexpr uint32_t TMEM_COLS = NTOK < 32 ? 32 : NTOK;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_abort;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_bar[3 * kNST + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // 128-byte swizzle atoms need 1024-byte alignment
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar0 = smem_u32(s_bar);
    const uint32_t full_a = bar0, full_b = bar0 + 8 * kNST, empty = bar0 + 16 * kNST, acc_full = bar0 + 24 * kNST;
    const int ft = blockIdx.x / p.ttiles, tt = blockIdx.x - ft * p.ttiles;
    const int tok0 = tt * NTOK;
    volatile int* abort_flag = &s_abort;

    if (tid < kNST) {
        mbar_init(full_a + 8 * tid, kDqWarps);
        mbar_init(full_b + 8 * tid, 1);
        mbar_init(empty + 8 * tid, 1);
    }
    if (tid == kNST) {
        mbar_init(acc_full, 1);
        s_abort = 0;
    }
    if (tid <= kNST) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == 1) {
        tmem_alloc(smem_u32(&s_tmem), TMEM_COLS);
        tmem_relinquish();
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int ksteps = p.ksteps;

    if (warp == 0) {
        // ---------------- TMA producer of the activation tiles ----------------
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // activations come from the pre-pass
            int s = 0, issued = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int ks = 0; ks < ksteps; ++ks) {
                ok = mbar_spin(empty + 8 * s, ph ^ 1u, abort_flag);
                if (!ok) break;
                const uint32_t dst = sbase + s * STAGE + kAStage;
                mbar_expect_tx(full_b + 8 * s, BSTAGE);
                tma_load_2d(dst, &tmap, ks * kKStep, tok0, full_b + 8 * s);
                tma_load_2d(dst + NTOK * 128, &tmap, ks * kKStep + 64, tok0, full_b + 8 * s);
                ++issued;
                if (++s == kNST) { s = 0; ph ^= 1u; }
            }
            if (!ok) {  // let the copies already issued land before this CTA's shared memory goes away
                for (int k = issued > kNST ? issued - kNST : 0; k < issued; ++k) {
                    const unsigned long long t0 = gtime_ns();
                    while (!mbar_try(full_b + 8 * (k % kNST), (uint32_t)(k / kNST) & 1u) &&
                           gtime_ns() - t0 < kWaitLimitNs) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            constexpr uint32_t idesc = idesc_f16(NTOK);
            int s = 0;
            uint32_t ph = 0;
            bool ok = true, any = false;
            for (int ks = 0; ks < ksteps; ++ks) {
                ok = mbar_spin(full_a + 8 * s, ph, abort_flag) && mbar_spin(full_b + 8 * s, ph, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a0 = sbase + s * STAGE, b0 = a0 + kAStage;
#pragma unroll
                for (int kk = 0; kk < kKStep / 16; ++kk) {
                    const uint32_t aa = a0 + (kk >> 2) * (128 * 128) + (kk & 3) * 32;
                    const uint32_t bb = b0 + (kk >> 2) * (NTOK * 128) + (kk & 3) * 32;
                    umma_f16(tmem, smem_desc_sw128(aa), smem_desc_sw128(bb), idesc, (ks | kk) != 0);
                }
                any = true;
                umma_commit(empty + 8 * s);  // stage free once these MMAs have read it
                if (++s == kNST) { s = 0; ph ^= 1u; }
            }
            if (ok || any) {
                umma_commit(acc_full);
                if (!ok) {  // gave up: tensor core must be idle before tensor memory is freed
                    const unsigned long long t0 = gtime_ns();
                    while (!mbar_try(acc_full, 0) && gtime_ns() - t0 < kWaitLimitNs) {
                    }
                }
            }
        }
    } else {
        // ---------------- dequant warps: group = dq >> 2, block of the K-step = dq & 3 ----------------
        const int dq = warp - 2, grp = dq >> 2, sub = dq & 3;
        const int sel = (lane >> 4) & 1;  // 4-bit: row pair q; 8-bit: plane p
        const int tp = (lane >> 3) & 1, gid = lane & 7;
        const int64_t g_glob = (int64_t)ft * 4 + grp;
        const bool g_valid = g_glob < p.ngroups;
        // running pointer to this task's unit of the current prefetch K-step
        const uint8_t* wptr = p.w + (g_glob * p.nb + sub) * UNIT + (gid * 4 + 2 * tp) * 16 +
                              (BITS == 4 ? sel * 8 : sel * 512);
        const uint8_t* sptr = p.w + (g_glob * p.nb + sub) * UNIT + CODES + gid * 16 + (BITS == 4 ? sel * 8 : 0);
        int bk_next = sub;  // block index the next load refers to

        auto load = [&](RawW<BITS>& r) {
            if (g_valid && bk_next < p.nb) {
                if constexpr (BITS == 4) {
                    r.a = __ldg(reinterpret_cast<const uint2*>(wptr));
                    r.b = __ldg(reinterpret_cast<const uint2*>(wptr + 16));
                    r.s = __ldg(reinterpret_cast<const float2*>(sptr));
                } else {
                    r.a = __ldg(reinterpret_cast<const uint4*>(wptr));
                    r.b = __ldg(reinterpret_cast<const uint4*>(wptr + 16));
                    r.s = __ldg(reinterpret_cast<const float4*>(sptr));
                }
            } else {
                r = RawW<BITS>{};  // zero scale: rows / blocks beyond the matrix contribute 0
            }
            wptr += 4 * UNIT;
            sptr += 4 * UNIT;
            bk_next += 4;
        };
        // Shared-memory byte offsets of this task's 16-byte chunks inside a stage (K-major,
        // 128-byte swizzle: chunk c of row r sits at (r/8)*1024 + (r%8)*128 + ((c ^ r%8) * 16)).
        // Rows of one task differ by multiples of 8, so they share the xor and sit 1024 B apart.
        const uint32_t katom_off = (sub >> 1) * (128 * 128);
        uint32_t soff0, soff1;
        if (BITS == 4) {
            const uint32_t rbase = katom_off + (grp * 4 + 2 * sel) * 1024 + gid * 128;
            soff0 = rbase + (((4 * (sub & 1) + tp) ^ gid) << 4);      // h = 0
            soff1 = rbase + (((4 * (sub & 1) + 2 + tp) ^ gid) << 4);  // h = 1
        } else {
            soff0 = katom_off + (grp * 4) * 1024 + gid * 128 + (((4 * (sub & 1) + 2 * sel + tp) ^ gid) << 4);
            soff1 = 0;
        }
        const float wmul = p.wmul;
        auto convert = [&](const RawW<BITS>& r, uint32_t stage) {
            if constexpr (BITS == 4) {
                const uint32_t off = 0x64086408u;  // 1024 + zero point 8
                const uint32_t s_lo = scale_h2(r.s.x * wmul), s_hi = scale_h2(r.s.y * wmul);
                const uint32_t wa[2] = {r.a.x, r.a.y}, wb[2] = {r.b.x, r.b.y};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t dst = stage + (h ? soff1 : soff0);
                    const uint2 l0 = bytes_to_h4(wa[h] & 0x0F0F0F0Fu, off, s_lo);
                    const uint2 l1 = bytes_to_h4(wb[h] & 0x0F0F0F0Fu, off, s_lo);
                    sts128(dst, l0.x, l0.y, l1.x, l1.y);            // row gid + 16q
                    const uint2 h0 = bytes_to_h4((wa[h] >> 4) & 0x0F0F0F0Fu, off, s_hi);
                    const uint2 h1 = bytes_to_h4((wb[h] >> 4) & 0x0F0F0F0Fu, off, s_hi);
                    sts128(dst + 1024, h0.x, h0.y, h1.x, h1.y);     // row gid + 16q + 8
                }
            } else {
                const uint32_t off = 0x64806480u;  // 1024 + zero point 128
                const uint32_t wa[4] = {r.a.x, r.a.y, r.a.z, r.a.w}, wb[4] = {r.b.x, r.b.y, r.b.z, r.b.w};
                const float sc[4] = {r.s.x, r.s.y, r.s.z, r.s.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t s2 = scale_h2(sc[i] * wmul);
                    const uint2 l0 = bytes_to_h4(wa[i], off, s2);
                    const uint2 l1 = bytes_to_h4(wb[i], off, s2);
                    sts128(stage + soff0 + i * 1024, l0.x, l0.y, l1.x, l1.y);  // row gid + 8i
                }
            }
        };

        RawW<BITS> raw[kPrefetch];
#pragma unroll
        for (int j = 0; j < kPrefetch; ++j) load(raw[j]);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int ks0 = 0; ks0 < ksteps && ok; ks0 += kPrefetch) {
#pragma unroll
            for (int j = 0; j < kPrefetch; ++j) {
                const int ks = ks0 + j;
                if (ks < ksteps && ok) {
                    const bool got = mbar_spin(empty + 8 * s, ph ^ 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, got);
                    if (ok) {
                        convert(raw[j], sbase + s * STAGE);
                        fence_async_smem();  // generic-proxy stores -> visible to the tensor core
                        __syncwarp();
                        if (lane == 0) mbar_arrive(full_a + 8 * s);
                        load(raw[j]);
                        if (++s == kNST) { s = 0; ph ^= 1u; }
                    }
                }
            }
        }

        // ---------------- epilogue: tensor memory -> y ----------------
        if (ok) {
            const bool got = mbar_spin(acc_full, 0, abort_flag);
            ok = __all_sync(0xffffffffu, got);
        }
        if (ok) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // y may still be read by the grid before us
            tc_fence_after();
            const int sp = warp & 3;          // tensor-memory lanes 32*sp .. 32*sp + 31
            const int cq = dq >> 2;           // column quarter
            const int64_t f = (int64_t)ft * 128 + sp * 32 + lane;
            constexpr int CPW = NTOK / 4;     // columns per warp
#pragma unroll
            for (int c0 = 0; c0 < CPW; c0 += 8) {
                uint32_t v[8];
                const int col = cq * CPW + c0;
                tmem_ld8(tmem + ((uint32_t)(sp * 32) << 16) + (uint32_t)col, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int tok = tok0 + col + j;
                    if (tok < p.M && f < p.out) {
                        const float val = __uint_as_float(v[j]) * p.wdiv * __ldg(p.rowscale + tok);
                        store_out(p.y, p.out_dtype, (int64_t)tok * p.out + f, val);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, TMEM_COLS);
    if (tid == 0 && s_abort) atomicExch(p.status, 2);
}

// ---- GEMM with the dequantized weights kept in tensor memory ------------------------------------
// Same tile and pipeline as gemm_tc_kernel, but A never touches shared memory: the
// tcgen05.st.16x256b fragment layout (lane = 4*gid + tig writes rows gid and gid + 8,
// 32-bit columns 2*tig and 2*tig + 1) is exactly how the mma32 layout hands a lane its 16-byte
// slot, so every lane converts its slot in registers and stores it to the A ring in tensor
// memory (64 columns per 128-element K-step); tcgen05.mma reads A from tensor memory and only B
// from shared memory, which halves the shared-memory traffic of the K loop.
// Warp roles: 0 = TMA (activations) and the L2 requests for the weights, 1 and 18 = MMA (even / odd
// K-steps), 2..17 = dequant, then epilogue: warp & 3 = 32-row group (= its tensor-memory
// sub-partition); t = (warp - 2) >> 2 picks the set (t & 1: even / odd K-steps) and the pair of
// blocks (2 (t >> 1), + 1) of a K-step.
constexpr int kGemmThreadsT = (3 + kDqWarps) * 32;  // TMA warp, MMA warp (even K-steps), 16 dequant / epilogue warps, MMA warp (odd K-steps)
// pipeline stages (B in shared memory, A in tensor memory): what is left of the 512 columns after two
// accumulators, at most 4: with exactly four the dequant warps run their two-set schedule, which
// measured faster than six stages on the one-set schedule where six would fit (M <= 64: 76 -> 68 us
// at M = 16 on 28672 x 8192)
__host__ __device__ constexpr int gemm_stages(int ntok, bool duo) { return ntok > 128 && !duo ? 3 : 4; }
// A 256-token tile has one accumulator (256 columns) and one issuing thread: an MMA then takes the
// tensor core 128 cycles, more than its issue costs; its activation stage is 64 KB, so three stages.
__host__ __device__ constexpr int gemm_issuers(int ntok) { return ntok > 128 ? 1 : 2; }
constexpr int kAColsPerStage = kKStep / 2;
constexpr int kEpiLd = 36;   // floats per token row of the epilogue's staging tiles (16-byte aligned rows)
// bytes of activations per stage and CTA: a pair of CTAs shares a tile's tokens
__host__ __device__ constexpr int gemm_bstage(int ntok, bool duo) { return ntok * kKStep * 2 / (duo ? 2 : 1); }
__host__ __device__ constexpr int gemm_smem(int ntok, bool duo) {
    const int ring = gemm_stages(ntok, duo) * gemm_bstage(ntok, duo), epi = kDqWarps * (ntok / 4 < 32 ? ntok / 4 : 32) * kEpiLd * 4;
    return (ring > epi ? ring : epi) + 1024;
}
constexpr int kWeightPfSteps = 8;  // K-steps of packed weights requested into L2 ahead of the loads

// One 128-element K-step as a single block of instructions, so that nothing but a branch sits
// between the last MMA of a step and the first of the next: eight MMAs (A columns a0 + 8 kk, B
// descriptor b_lo + 2 (kk & 3) + BHALF (kk >> 2) in 16-byte units, BHALF = second 64-element half
// of the stage), with a non-blocking test of the NEXT stage's barrier tucked in between them, where the
// issuing lane is waiting for the tensor core anyway; its answer is read at the end.  first = 0
// makes MMA 0 overwrite the accumulator; lanes with leader = 0 issue no tensor-core instruction.
template <int BHALF, bool DUO>
__device__ __forceinline__ uint32_t umma_f16_ts_step(uint32_t d_tmem, uint32_t a0, uint32_t b_lo, uint32_t b_hi,
                                                     uint32_t idesc, uint32_t first, uint32_t leader,
                                                     uint32_t next_full, uint32_t next_parity) {
    uint32_t next_ready;
    if constexpr (DUO) {   // the pair's barrier, which the other CTA arrives on as well
        asm volatile(
            "{\n"
            ".reg .pred p, q, t, r;\n"
            ".reg .b64 bd0, bd1, bd2, bd3, bd4, bd5, bd6, bd7;\n"
            ".reg .b32 a1, a2, a3, a4, a5, a6, a7, b;\n"
            "setp.ne.b32 p, %6, 0;\n"
            "setp.ne.b32 q, %7, 0;\n"
            "setp.eq.b32 t, 0, 0;\n"
            "mov.b64 bd0, {%3, %4};\n"
            "add.u32 a1, %2, 8;  add.u32 b, %3, 2;   mov.b64 bd1, {b, %4};\n"
            "add.u32 a2, %2, 16; add.u32 b, %3, 4;   mov.b64 bd2, {b, %4};\n"
            "add.u32 a3, %2, 24; add.u32 b, %3, 6;   mov.b64 bd3, {b, %4};\n"
            "add.u32 a4, %2, 32; add.u32 b, %3, %8;  mov.b64 bd4, {b, %4};\n"
            "add.u32 a5, %2, 40; add.u32 b, %3, %9;  mov.b64 bd5, {b, %4};\n"
            "add.u32 a6, %2, 48; add.u32 b, %3, %10; mov.b64 bd6, {b, %4};\n"
            "add.u32 a7, %2, 56; add.u32 b, %3, %11; mov.b64 bd7, {b, %4};\n"
            "tcgen05.fence::after_thread_sync;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [%2], bd0, %5, p;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [a1], bd1, %5, t;\n"
            "mbarrier.test_wait.parity.shared::cta.b64 r, [%12], %13;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [a2], bd2, %5, t;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [a3], bd3, %5, t;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [a4], bd4, %5, t;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [a5], bd5, %5, t;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [a6], bd6, %5, t;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%1], [a7], bd7, %5, t;\n"
            "selp.u32 %0, 1, 0, r;\n"
            "}"
            : "=r"(next_ready)
            : "r"(d_tmem), "r"(a0), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first), "r"(leader), "n"(BHALF),
              "n"(BHALF + 2), "n"(BHALF + 4), "n"(BHALF + 6), "r"(next_full), "r"(next_parity)
            : "memory");
    } else {
        asm volatile(
            "{\n"
            ".reg .pred p, q, t, r;\n"
            ".reg .b64 bd0, bd1, bd2, bd3, bd4, bd5, bd6, bd7;\n"
            ".reg .b32 a1, a2, a3, a4, a5, a6, a7, b;\n"
            "setp.ne.b32 p, %6, 0;\n"
            "setp.ne.b32 q, %7, 0;\n"
            "setp.eq.b32 t, 0, 0;\n"
            "mov.b64 bd0, {%3, %4};\n"
            "add.u32 a1, %2, 8;  add.u32 b, %3, 2;   mov.b64 bd1, {b, %4};\n"
            "add.u32 a2, %2, 16; add.u32 b, %3, 4;   mov.b64 bd2, {b, %4};\n"
            "add.u32 a3, %2, 24; add.u32 b, %3, 6;   mov.b64 bd3, {b, %4};\n"
            "add.u32 a4, %2, 32; add.u32 b, %3, %8;  mov.b64 bd4, {b, %4};\n"
            "add.u32 a5, %2, 40; add.u32 b, %3, %9;  mov.b64 bd5, {b, %4};\n"
            "add.u32 a6, %2, 48; add.u32 b, %3, %10; mov.b64 bd6, {b, %4};\n"
            "add.u32 a7, %2, 56; add.u32 b, %3, %11; mov.b64 bd7, {b, %4};\n"
            "tcgen05.fence::after_thread_sync;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], bd0, %5, p;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [a1], bd1, %5, t;\n"
            "mbarrier.test_wait.parity.shared::cta.b64 r, [%12], %13;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [a2], bd2, %5, t;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [a3], bd3, %5, t;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [a4], bd4, %5, t;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [a5], bd5, %5, t;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [a6], bd6, %5, t;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [a7], bd7, %5, t;\n"
            "selp.u32 %0, 1, 0, r;\n"
            "}"
            : "=r"(next_ready)
            : "r"(d_tmem), "r"(a0), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first), "r"(leader), "n"(BHALF),
              "n"(BHALF + 2), "n"(BHALF + 4), "n"(BHALF + 6), "r"(next_full), "r"(next_parity)
            : "memory");
    }
    return next_ready;
}
template <int BITS>
struct RawT;
template <>
struct RawT<4> {
    uint4 c;    // the lane's slot: words 2q + h
    float4 s;   // scales of rows gid + 8i
};
template <>
struct RawT<8> {
    uint4 c0, c1;  // plane 0 / 1 slot: word i = row gid + 8i
    float4 s;
};

static __device__ __align__(16) uint8_t g_zero_unit[kUnitBytesQ8];   // never written
__device__ __forceinline__ int64_t gemm_range_start(const GemmParams& p, int64_t c) {
    if (p.half > 0) return (c >> 1) * p.ksteps + (c & 1) * p.half;
    if (p.parts > 0) {
        const uint32_t t = (uint32_t)c / (uint32_t)p.parts;
        return t * p.ksteps + ((uint32_t)c - t * p.parts) * p.ksteps / p.parts;
    }
    return c * p.uq + (c < p.ur ? c : p.ur);
}

// SEGS: ranges that touch several tiles, and rows whose last K-step is a partial one.  A kernel of its own: with the
// loop over segments and the second K loop around it a single tile ran 3 % slower (4096 x 4096, M = 512: 21.3 ->
// 22.0 us); with what is left of the bookkeeping (ring positions, segment lengths, a division per role) as constants
// there, int8 4096 x 4096 takes 24.42 us at M = 512 (24.58 without, 24.38 before there were segments), 18.6 at
// M = 256 (18.8).
// DUO: a pair of CTAs (a cluster of two) works on a tile of 256 features x 256 tokens with MMAs of cta_group::2: each CTA
// dequantizes its 128 features into its own tensor memory and brings half of the tokens into its shared memory, one thread
// of the first issues for both.  Half the activation bytes per SM, half the MMA instructions, and four stages fit instead of
// three: K-step 1110 -> 1030 cycles with all SMs busy (the tensor core's own time is 1024).  The second CTA keeps barriers of its own;
// its warp 1 passes every full stage on to the first CTA's barrier (an arrival with cluster scope instead of the default one
// takes 180 cycles per step: a fence; what it would order, TMA bytes and tensor memory, other instructions order already).
template <int BITS, int NTOK, bool SEGS, bool DUO>
__global__ void __launch_bounds__(kGemmThreadsT, 1)
gemm_tmem_kernel(const GemmParams p, const __grid_constant__ CUtensorMap tmap) {
    constexpr int UNIT = BITS == 4 ? kUnitBytesQ4 : kUnitBytesQ8;
    constexpr int CODES = BITS == 4 ? kUnitCodesQ4 : kUnitCodesQ8;
    constexpr int BSTAGE = gemm_bstage(NTOK, DUO);
    constexpr int kNSTT = gemm_stages(NTOK, DUO);
    constexpr int CS = DUO ? 2 : 1, BROWS = NTOK / CS;        // CTAs of a tile; its tokens in this CTA's shared memory
    constexpr int ISS = gemm_issuers(NTOK);
    constexpr uint32_t TMEM_COLS = 512;                       // ISS accumulators (NTOK columns each) + A ring, power of two
    constexpr uint32_t A_COL0 = ISS * NTOK;                   // A ring starts after the accumulators
    static_assert(ISS * NTOK + kNSTT * kAColsPerStage <= 512 && kNSTT >= 3,
                  "tensor memory holds the accumulators and the A ring");
    static_assert(!DUO || ISS == 1, "the second CTA of a pair has one warp that passes its stages on");
    extern __shared__ uint8_t smem_raw[];
    if (p.dbg && blockIdx.x == 0 && threadIdx.x == 64) { p.dbg[300] = (unsigned long long)clock64(); p.dbg[304] = gtime_ns(); }
    __shared__ int s_abort;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_bar[2 * 6 + 2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar0 = smem_u32(s_bar);
    // full[s]: the eight dequant warps of the step's set have stored A of the stage and the TMA bytes of B have
    // landed; empty[s]: the MMAs that read the stage have completed (tcgen05.commit); acc_full: a segment's sums are
    // complete; acc_free: the epilogue has read them (and is done with the activation stages it borrows)
    const uint32_t full = bar0, empty = bar0 + 8 * kNSTT, acc_full = bar0 + 16 * kNSTT, acc_free = acc_full + 8;
    volatile int* abort_flag = &s_abort;
    // This CTA's range of the step sequence.  It is worked off in segments, one per tile it touches; step q of the
    // range (counted over all segments) uses ring stage q mod kNSTT.  Where tiles are shared the ranges are dealt out
    // from the back: a CTA then waits only for CTAs launched before it.
    const int KS = p.ksteps, units = (int)gridDim.x / CS, unit = (int)blockIdx.x / CS;
    const int cta = SEGS || p.half > 0 ? units - 1 - unit : unit;   // (DUO: the pair's number)
    const uint32_t rank = DUO ? blockIdx.x & 1 : 0;                 // (its place in the cluster: clusters are two neighbours)
    int tile_first, k_first, steps_own;   // first tile, first step in it, number of steps
    if (p.half > 0) {
        tile_first = cta >> 1;
        k_first = (cta & 1) * p.half;
        steps_own = (cta & 1) ? KS - p.half : p.half;
    } else if (!SEGS || (p.uq == KS && p.ur == 0 && p.parts == 0)) {
        tile_first = cta;
        k_first = 0;
        steps_own = KS;
    } else {
        const uint32_t r0 = (uint32_t)gemm_range_start(p, cta);
        tile_first = (int)(r0 / (uint32_t)KS);
        k_first = (int)(r0 - (uint32_t)tile_first * KS);
        steps_own = (int)((uint32_t)gemm_range_start(p, cta + 1) - r0);
    }
    const int fd = tile_first / p.ttiles, ft_first = fd * CS + (int)rank, tok_first = (tile_first - fd * p.ttiles) * NTOK;

    // DUO: the columns of a tile that hold tokens, in thirty-twos (N of an MMA of cta_group::2 with M = 256), where one tile takes all tokens: narrower MMAs.  (The rest of its
    // columns is never written, and what is read there goes nowhere.  int4 28672 x 8192 at M = 160 91.4 -> 85.6 us; in
    // sixteens M = 200 would be 208 columns and 104.2 us at 8192 x 28672, it is 224 and 105.0.  Worked out per tile, for several, full
    // tiles lose 1.4 %.)
    const int cols = DUO ? p.cols : NTOK;

    if (tid == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
    if (warp >= 2 && warp < 2 + kDqWarps) {
        // the first weights this warp will load: ask for them now, so that the HBM round trip
        // runs while the CTA sets itself up (barriers, tensor memory, the CTA-wide sync)
        const int t = (warp - 2) >> 2, pset = t & 1, blk0 = 2 * (t >> 1);
        int64_t g = (int64_t)ft_first * 4 + (warp & 3);
        g = g < p.ngroups ? g : (int64_t)p.ngroups - 1;
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            const int b = 4 * (k_first + pset + 2 * d) + blk0;
            if ((SEGS ? b + 1 < p.nb : pset + 2 * d < steps_own) && lane * 128 < 2 * UNIT)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w + (g * p.nb + b) * UNIT + lane * 128));
        }
    }
    if (tid < kNSTT) {
        mbar_init(full + 8 * tid, kDqWarps / 2 + 1 + (DUO && rank == 0 ? 1 : 0));   // (+ 1: the other CTA's stage, passed on)
        mbar_init(empty + 8 * tid, 1);
    } else if (tid == kNSTT) {
        mbar_init(acc_full, ISS == 2 && (SEGS || steps_own >= 2) ? 2 : 1);   // one arrival per MMA issuer (that has steps) and segment
        mbar_init(acc_free, kDqWarps);
        s_abort = 0;
    }
    if (tid <= kNSTT) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == 1) {
        if constexpr (DUO) {
            tmem_alloc2(smem_u32(&s_tmem), TMEM_COLS);
            tmem_relinquish2();
        } else {
            tmem_alloc(smem_u32(&s_tmem), TMEM_COLS);
            tmem_relinquish();
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    // (the other CTA's barriers: only the warps that arrive on them wait for it here, the others at the end)
    if constexpr (DUO) cluster_arrive();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    unsigned long long* dbg = (p.dbg && blockIdx.x == 0) ? p.dbg : nullptr;
    if (dbg && tid == 64) dbg[301] = (unsigned long long)clock64();

    if (warp == 0) {
        // ---------------- TMA producer of the activation tiles ----------------
        if (lane == 0) {
            // The dequant warps read the packed weights with plain loads a few K-steps ahead, which
            // covers an L2 round trip but not one to HBM.  This thread therefore asks for the
            // weights to be brought into L2 kPfSteps K-steps ahead of those loads, four K-steps (16
            // units, one contiguous run per row group) per request.
            constexpr int kPfSteps = kWeightPfSteps;
            int s = 0, issued = 0, seg = 0, left = steps_own;
            uint32_t ph = 0;
            bool ok = true;
            for (int tile = tile_first, k0 = k_first, ft = ft_first, tok0 = tok_first; ok; k0 = 0) {
                const int n = SEGS ? min(KS - k0, left) : steps_own;
                const int nb_end = min(p.nb, 4 * (k0 + n));
                auto request = [&](int ks) {  // K-steps ks .. ks + 3 of this segment
                    const int b0 = 4 * (k0 + ks);
                    const int nblk = min(16, nb_end - b0);
                    if (nblk <= 0) return;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const int64_t gg = (int64_t)ft * 4 + g;
                        if (gg < p.ngroups) {
                            const uint8_t* q = p.w + (gg * p.nb + b0) * UNIT;
                            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(q), "r"((uint32_t)(nblk * UNIT))
                                         : "memory");
                        }
                    }
                };
                if (!SEGS || seg == 0) {
                    asm volatile("griddepcontrol.wait;" ::: "memory");  // activations come from the pre-pass
                } else {
                    // a further tile: its first weights on their way while the epilogue of the one before runs
                    for (int k2 = 0; k2 < 8 + kPfSteps; k2 += 4) request(k2);
                    ok = mbar_block(acc_free, (uint32_t)(seg - 1) & 1u, abort_flag);
                }
                const int row0 = tok0 + (DUO ? (int)rank * (cols / 2) : 0);   // a pair's second CTA holds the upper half of the columns
                for (int ks = 0; ks < n && ok; ++ks) {
                    // weight requests: none before the wait above (they would compete for HBM with the
                    // pre-pass this kernel waits for) nor before the first activation tiles are on their
                    // way; the dequant warps load K-steps 0 .. 3 themselves
                    if ((!SEGS || seg == 0) && ks == kNSTT)
                        for (int k2 = 4; k2 < 8 + kPfSteps; k2 += 4) request(k2);
                    if ((ks & 3) == 0 && ks >= 4) request(ks + 4 + kPfSteps);
                    ok = mbar_block(empty + 8 * s, ph ^ 1u, abort_flag);
                    if (!ok) break;
                    const uint32_t dst = sbase + s * BSTAGE;
                    mbar_expect_tx(full + 8 * s, BSTAGE);
                    tma_load_2d(dst, &tmap, (k0 + ks) * kKStep, row0, full + 8 * s);
                    tma_load_2d(dst + BROWS * 128, &tmap, (k0 + ks) * kKStep + 64, row0, full + 8 * s);
                    ++issued;
                    if (++s == kNSTT) { s = 0; ph ^= 1u; }
                }
                if (!SEGS || (left -= n) == 0) break;
                ++seg;
                ++tile;
                const int fd2 = tile / p.ttiles;
                ft = fd2 * CS + (int)rank;
                tok0 = (tile - fd2 * p.ttiles) * NTOK;
            }
            if constexpr (DUO)   // the last arrivals from the pair's MMAs: none may find this CTA's shared memory gone
                for (int i = 0; i < kNSTT && ok; ++i) {   // (stages never used pass at once)
                    ok = mbar_block(empty + 8 * s, ph ^ 1u, abort_flag);
                    if (++s == kNSTT) { s = 0; ph ^= 1u; }
                }
            if (!ok) {  // let the copies already issued land before this CTA's shared memory goes away
                for (int k = issued > kNSTT ? issued - kNSTT : 0; k < issued; ++k) {
                    const unsigned long long t0 = gtime_ns();
                    while (!mbar_try(full + 8 * (k % kNSTT), (uint32_t)(k / kNSTT) & 1u) &&
                           gtime_ns() - t0 < kWaitLimitNs) {
                    }
                }
            }
        }
    } else if (DUO && rank == 1 && warp == 1) {
        // ---------------- the second CTA of a pair: its stages, passed on to the issuer ----------------
        // (A further segment's first stage goes on only after this CTA's epilogue is done with the accumulators.)
        bool ok = true;
        int q = 0, seg = 0, left = steps_own;
        cluster_wait();
        for (int k0 = k_first; ok; k0 = 0) {
            const int n = SEGS ? min(KS - k0, left) : steps_own;
            if (SEGS && seg > 0) ok = __all_sync(0xffffffffu, mbar_spin(acc_free, (uint32_t)(seg - 1) & 1u, abort_flag));
            for (int ks = 0; ks < n && ok; ++ks, ++q) {
                const uint32_t bar = full + 8 * (q % kNSTT);
                ok = __all_sync(0xffffffffu, mbar_spin(bar, (uint32_t)(q / kNSTT) & 1u, abort_flag));
                if (!ok) break;
                tc_fence_after();
                tc_fence_before();
                if (lane == 0) mbar_arrive_at(bar, 0);
                __syncwarp();
            }
            if (!SEGS || (left -= n) == 0) break;
            ++seg;
        }
    } else if (warp == 1 || (ISS == 2 && warp == 2 + kDqWarps)) {
        // ---------------- MMA issuers ----------------
        // Issuing is what limits the tensor core here: a tcgen05 instruction costs the issuing
        // thread 50 - 60 cycles (measured: an MMA, a commit and a barrier test alike, whatever N
        // is), so the eight MMAs of a step plus its barrier work take one thread about 900 cycles
        // while the tensor core needs 512 for them.  Two warps on different schedulers therefore
        // take alternate K-steps, each into an accumulator of its own (the epilogue adds them);
        // each commits its own stages, so the rest of the pipeline does not notice.
        // The whole warp runs the loop with identical values (the address arithmetic stays
        // warp-uniform) and lane 0 alone issues the tensor-core instructions.
        const int m = warp == 1 ? 0 : 1;
        const uint32_t leader = lane == 0;
        const uint32_t idesc = DUO ? idesc_f16_pair(cols) : idesc_f16(NTOK);
        auto commit = [&](uint32_t bar) {
            if constexpr (DUO) umma_commit2_if(bar, leader);
            else umma_commit_if(bar, leader);
        };
        const uint64_t d0 = smem_desc_sw128(sbase);
        const uint32_t d_lo = (uint32_t)d0, d_hi = (uint32_t)(d0 >> 32);
        const uint32_t dcol = tmem + (uint32_t)(m * NTOK);
        static_assert(kKStep == 128, "eight MMAs per step");
        if constexpr (DUO) cluster_wait();
        bool any = false, ok = true;
        int q0 = 0, seg = 0, left = steps_own;
        for (int k0 = k_first; ok; k0 = 0) {
            const int n = SEGS ? min(KS - k0, left) : steps_own;
            const int first = ISS == 2 ? (SEGS ? (m + q0) & 1 : m) : 0;   // this issuer's first step of the segment: q0 + first = m (mod 2)
            int s = SEGS ? (q0 + first) % kNSTT : first;
            uint32_t ph = SEGS ? (uint32_t)((q0 + first) / kNSTT) & 1u : 0u;
            if (SEGS && seg > 0) ok = mbar_spin(acc_free, (uint32_t)(seg - 1) & 1u, abort_flag);
            if (ok && first < n) ok = mbar_spin(full + 8 * s, ph, abort_flag);
            if (dbg && lane == 0 && seg == 0) dbg[306 + 2 * m] = (unsigned long long)clock64();
            for (int ks = first; ks < n && ok; ks += ISS) {
                int s2 = s + ISS;
                uint32_t ph2 = ph;
                if (s2 >= kNSTT) { s2 -= kNSTT; ph2 ^= 1u; }
                const uint32_t a0 = tmem + A_COL0 + s * kAColsPerStage, b_lo = d_lo + (uint32_t)s * (BSTAGE >> 4);
                // the block also tests the barrier of this issuer's next step (ks + ISS) early
                const uint32_t n2 = umma_f16_ts_step<BROWS * 8, DUO>(dcol, a0, b_lo, d_hi, idesc, ks != first, leader, full + 8 * s2,
                                                               ph2);
                commit(empty + 8 * s);  // the stage is free once these MMAs have read it
                any = true;
                if (ks + ISS < n && !n2) ok = mbar_spin(full + 8 * s2, ph2, abort_flag);
                s = s2;
                ph = ph2;
            }
            if (dbg && lane == 0) dbg[307 + 2 * m] = (unsigned long long)clock64();
            if (any || (SEGS && ok)) commit(acc_full);   // (arrives at once where this issuer had no step)
            if (!ok && any) {  // gave up: the tensor core must be idle before tensor memory is freed
                const unsigned long long t0 = gtime_ns();
                while (!mbar_try(acc_full, (uint32_t)seg & 1u) && gtime_ns() - t0 < kWaitLimitNs) {
                }
            }
            if (!SEGS || (left -= n) == 0) break;
            ++seg;
            q0 += n;
        }
    } else if (warp == 2 + kDqWarps) {
        // the second issuer warp of the two-accumulator tiles: nothing to do on a 256-token tile
    } else {
        // ---------------- dequant warps ----------------
        const int dq = warp - 2, grp = warp & 3;
        const int gid = lane >> 2;
        const float wmul = p.wmul;
        // this warp's rows are tensor-memory lanes 32*grp .. 32*grp + 31; its block is 16 columns wide
        const uint32_t t_lane = (uint32_t)(grp * 32) << 16;
        auto convert_store = [&](const RawT<BITS>& r, uint32_t a_stage, int blk) {
            const uint32_t dst = a_stage + t_lane + blk * 16;
            const float sc[4] = {r.s.x, r.s.y, r.s.z, r.s.w};
            if constexpr (BITS == 4) {
                constexpr uint32_t kZero = 0x80088008u;   // -8 * 2^-24 twice
                constexpr uint32_t kSixteenth = 0x2C002C00u;
                const uint32_t w[4] = {r.c.x, r.c.y, r.c.z, r.c.w};
#pragma unroll
                for (int q = 0; q < 2; ++q) {  // rows gid + 16q (low nibbles) and gid + 16q + 8 (high)
                    const uint32_t s_lo = scale_h2(sc[2 * q] * wmul), s_hi = scale_h2(sc[2 * q + 1] * wmul);
                    const uint32_t z_lo = hmul2_u32(s_lo, kZero), z_hi = hmul2_u32(s_hi, kZero);
                    const uint32_t s_hi16 = hmul2_u32(s_hi, kSixteenth);  // high nibbles stay where they are: 16 n
                    uint32_t v[8];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {  // columns 8h .. 8h + 7: elements 16h + 4tig ..
                        const uint2 lo = bytes_fma_h4(w[2 * q + h] & 0x0F0F0F0Fu, s_lo, z_lo);
                        const uint2 hi = bytes_fma_h4(w[2 * q + h] & 0xF0F0F0F0u, s_hi16, z_hi);
                        v[4 * h + 0] = lo.x;
                        v[4 * h + 1] = lo.y;
                        v[4 * h + 2] = hi.x;
                        v[4 * h + 3] = hi.y;
                    }
                    tmem_st_16x256b_x2(dst + ((uint32_t)(16 * q) << 16), v);
                }
            } else {
                constexpr uint32_t kZero = 0x80808080u;  // -128 * 2^-24 twice
                const uint32_t w0[4] = {r.c0.x, r.c0.y, r.c0.z, r.c0.w}, w1[4] = {r.c1.x, r.c1.y, r.c1.z, r.c1.w};
#pragma unroll
                for (int q = 0; q < 2; ++q) {  // rows gid + 16q (i = 2q) and gid + 16q + 8 (i = 2q + 1)
                    const uint32_t s_a = scale_h2(sc[2 * q] * wmul), s_b = scale_h2(sc[2 * q + 1] * wmul);
                    const uint32_t z_a = hmul2_u32(s_a, kZero), z_b = hmul2_u32(s_b, kZero);
                    uint32_t v[8];
                    const uint2 a0 = bytes_fma_h4(w0[2 * q], s_a, z_a), b0 = bytes_fma_h4(w0[2 * q + 1], s_b, z_b);
                    const uint2 a1 = bytes_fma_h4(w1[2 * q], s_a, z_a), b1 = bytes_fma_h4(w1[2 * q + 1], s_b, z_b);
                    v[0] = a0.x; v[1] = a0.y; v[2] = b0.x; v[3] = b0.y;   // plane 0: columns 0..7
                    v[4] = a1.x; v[5] = a1.y; v[6] = b1.x; v[7] = b1.y;   // plane 1: columns 8..15
                    tmem_st_16x256b_x2(dst + ((uint32_t)(16 * q) << 16), v);
                }
            }
        };
        // Two sets of eight warps take alternate K-steps, a warp converting two adjacent
        // blocks of its row group per step: while one set converts, the other waits for its
        // stage or stores, so the issue slots do not idle between bursts, and the fixed cost
        // of a step (barrier test, store wait, arrival) is paid once per two units.
        // Blocks past the end of a row (nb no multiple of 4) are read from a unit of zeros.
        const int t = dq >> 2, pset = t & 1, blk0 = 2 * (t >> 1);
        const uint32_t s_delta = (uint32_t)(CODES + gid * 16 - lane * 16);
        bool ok = true;
        int q0 = 0, seg = 0, left = steps_own;
        for (int tile = tile_first, k0 = k_first, ft = ft_first, tok0 = tok_first;; k0 = 0) {   // (also when a wait ran out: the warps meet at a barrier)
        const int n = SEGS ? min(KS - k0, left) : steps_own;
        {
            const int first = SEGS ? (pset + q0) & 1 : pset;   // own steps: q0 + first + 2 i
            const int n_own = (n - first + 1) >> 1;
            int64_t g_ld = (int64_t)ft * 4 + grp;         // (groups beyond the matrix: any valid rows, never stored)
            g_ld = g_ld < p.ngroups ? g_ld : (int64_t)p.ngroups - 1;
            int b_own = 4 * (k0 + first) + blk0;          // first block of own step i
            const uint8_t* wl = p.w + (g_ld * p.nb + b_own) * UNIT + lane * 16;
            auto fetch2 = [&](auto partial, RawT<BITS> (&r)[2], int own_off) {
                const uint8_t* q = wl + (size_t)own_off * (8 * UNIT);
#pragma unroll
                for (int u = 0; u < 2; ++u, q += UNIT) {
                    const uint8_t* a = q;
                    if (decltype(partial)::value && b_own + own_off * 8 + u >= p.nb) a = g_zero_unit + lane * 16;
                    if constexpr (BITS == 4) {
                        r[u].c = __ldg(reinterpret_cast<const uint4*>(a));
                    } else {
                        r[u].c0 = __ldg(reinterpret_cast<const uint4*>(a));
                        r[u].c1 = __ldg(reinterpret_cast<const uint4*>(a + 512));
                    }
                    r[u].s = __ldg(reinterpret_cast<const float4*>(a + s_delta));
                }
            };
            auto step2 = [&](const RawT<BITS> (&r)[2], int q) -> bool {
                // ring position q % stages, pass q / stages (the first pass finds every stage free: parity 1)
                const int st = q % kNSTT;
                const uint32_t parity = (uint32_t)(((q / kNSTT) & 1) ^ 1);
                if (!__all_sync(0xffffffffu, mbar_block(empty + 8 * st, parity, abort_flag))) return false;
                tc_fence_after();
                const uint32_t a_stage = tmem + A_COL0 + st * kAColsPerStage;
                convert_store(r[0], a_stage, blk0);
                convert_store(r[1], a_stage, blk0 + 1);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(full + 8 * st);
                return true;
            };
            auto k_loop = [&](auto partial) {
                RawT<BITS> raw[2][2];
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    raw[d][0] = RawT<BITS>{};
                    raw[d][1] = RawT<BITS>{};
                    if (d < n_own) fetch2(partial, raw[d], d);
                }
                int i = 0;
                for (; i + 2 <= n_own && ok; i += 2) {
                    const int q = q0 + first + 2 * i;
                    ok = step2(raw[0], q);
                    if (i + 2 < n_own) fetch2(partial, raw[0], 2);
                    if (ok) {
                        ok = step2(raw[1], q + 2);
                        if (i + 3 < n_own) fetch2(partial, raw[1], 3);
                    }
                    wl += (size_t)16 * UNIT;
                    if (decltype(partial)::value) b_own += 16;
                }
                if (ok && i < n_own) ok = step2(raw[0], q0 + first + 2 * i);
            };
            if constexpr (SEGS) {
                if (4 * (k0 + n) > p.nb) k_loop(std::true_type{});   // the row's last K-step is a partial one
                else k_loop(std::false_type{});
            } else {
                k_loop(std::false_type{});
            }
        }

        // ---------------- epilogue: tensor memory -> y ----------------
        // A warp owns 32 features (its tensor-memory lanes) x CPW tokens, handled CH <= 32 tokens at a
        // time.  Its token scales, one per lane and chunk, are fetched while the last MMAs run (the
        // pre-pass that wrote them completed before any activation tile was loaded).
        constexpr int CPW = NTOK / 4;                 // columns per warp
        constexpr int CH = CPW < 32 ? CPW : 32;       // columns per chunk
        constexpr int NCH = CPW / CH;
        const int cq = dq >> 2;                       // column quarter
        float rs_lane[NCH];
#pragma unroll
        for (int h = 0; h < NCH; ++h) rs_lane[h] = 0.f;
        if (ok) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
            for (int h = 0; h < NCH; ++h) {
                const int tl = tok0 + cq * CPW + h * CH + lane;
                if (lane < CH && tl < p.M) rs_lane[h] = __ldg(p.rowscale + tl);
            }
        }
        if (ok) {
            const bool got = mbar_block(acc_full, (uint32_t)seg & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, got);
        }
        if (dbg && tid == 64) dbg[302] = (unsigned long long)clock64();
        // A tile cut between CTAs: those holding its later steps (as the first segment of their ranges, so early)
        // hand their sums over through L2; the CTA holding its first step (its last segment) adds them to its own,
        // always in CTA order, and writes y.  A giver waits for nobody, and all CTAs are resident together.
        const bool giver = (SEGS || p.half > 0) && k0 > 0;
        int takes = 0;   // CTAs behind this one with steps of this tile
        if (!SEGS) takes = p.half > 0 && !giver;
        else if (p.parts > 0) takes = giver ? 0 : p.parts - 1;
        else if (!giver && n < KS)
            while (cta + 1 + takes < units && gemm_range_start(p, cta + 1 + takes) < (int64_t)(tile + 1) * KS) ++takes;
        constexpr size_t kPart = (size_t)kDqWarps * CPW * 32;   // floats per CTA
        const int slot = cta * CS + (int)rank;        // of this CTA's sums and flag
        float* part = p.part + slot * kPart + (size_t)dq * (CPW * 32);
        if (ok && takes > 0) {
            // (a lane per flag: one after the other they cost a trip to L2 each, 850 cycles)
            int got = 1;
            const unsigned long long t0 = gtime_ns();
            for (int k = 1 + lane; k <= (SEGS ? takes : 1) && got; k += 32) {
                for (;;) {
                    int v;
                    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p.part_flags + slot + k * CS) : "memory");
                    if (v != 0) break;
                    if (*abort_flag || gtime_ns() - t0 > kWaitLimitNs) {
                        *abort_flag = 1;
                        got = 0;
                        break;
                    }
                    __nanosleep(64);
                }
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, got);
        }
        if (ok) {
            tc_fence_after();
            const int sp = warp & 3;          // tensor-memory lanes 32*sp .. 32*sp + 31
            const int64_t f = (int64_t)ft * 128 + sp * 32 + lane;
            const float wdiv = p.wdiv;
            constexpr int LD = kEpiLd;
            float* tile_s = reinterpret_cast<float*>(smem) + dq * (CH * LD);
#pragma unroll
            for (int h = 0; h < NCH; ++h) {
                // all loads of the chunk first, one wait, then the stores with the output type decided
                // once (a lane owns one feature: consecutive lanes write consecutive elements of a row)
                uint32_t v[CH];
                // (a segment of one step has its sums in that step's accumulator alone)
                const uint32_t t0 = tmem + ((uint32_t)(sp * 32) << 16) + (uint32_t)(cq * CPW + h * CH) +
                                    (SEGS && ISS == 2 && n == 1 ? (uint32_t)(q0 & 1) * NTOK : 0u);
#pragma unroll
                for (int c0 = 0; c0 < CH; c0 += 8) tmem_ld8(t0 + c0, *reinterpret_cast<uint32_t(*)[8]>(&v[c0]));
                tmem_ld_wait();
                if (ISS == 2 && n >= 2) {  // the odd K-steps went into the second accumulator
                    uint32_t v2[CH];
#pragma unroll
                    for (int c0 = 0; c0 < CH; c0 += 8) tmem_ld8(t0 + NTOK + c0, *reinterpret_cast<uint32_t(*)[8]>(&v2[c0]));
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < CH; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(v2[j]));
                }
                const int tokb = tok0 + cq * CPW + h * CH;
                if (giver) {   // raw sums, 128 bytes per column and warp
#pragma unroll
                    for (int j = 0; j < CH; ++j) part[(h * CH + j) * 32 + lane] = __uint_as_float(v[j]);
                    continue;
                }
                for (int k = 1; k <= (SEGS ? takes : (takes > 0 ? 1 : 0)); ++k) {
                    const float* from = part + k * CS * kPart + (h * CH) * 32 + lane;
#pragma unroll
                    for (int j = 0; j < CH; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __ldcg(from + j * 32));
                }
                if ((p.out & 7) == 0) {
                    // Fast path: transpose the warp's 32-feature x CH-token tile through shared memory
                    // (the B ring is idle: every MMA has completed) so that a lane stores eight
                    // consecutive features of one token with one 16-byte (bf16) or two (f32) stores,
                    // instead of one element per store.
                    if (h) __syncwarp();   // the tile of the previous chunk has been read
#pragma unroll
                    for (int j = 0; j < CH; ++j) tile_s[j * LD + lane] = __uint_as_float(v[j]);
                    __syncwarp();
                    const int fg = (lane & 3) * 8;
                    const int64_t f0 = (int64_t)ft * 128 + sp * 32 + fg;
#pragma unroll
                    for (int t0c = 0; t0c < CH; t0c += 8) {
                        const int t = t0c + (lane >> 2), tok = tokb + t;
                        const float sc = wdiv * __shfl_sync(0xffffffffu, rs_lane[h], t);
                        if (tok < p.M && f0 < p.out) {
                            const float4 a = *reinterpret_cast<const float4*>(tile_s + t * LD + fg);
                            const float4 c = *reinterpret_cast<const float4*>(tile_s + t * LD + fg + 4);
                            if (p.out_dtype == RSTQ_BF16) {
                                uint4 o;
                                o.x = pack_bf16x2(a.y * sc, a.x * sc);
                                o.y = pack_bf16x2(a.w * sc, a.z * sc);
                                o.z = pack_bf16x2(c.y * sc, c.x * sc);
                                o.w = pack_bf16x2(c.w * sc, c.z * sc);
                                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.y) + (int64_t)tok * p.out + f0) = o;
                            } else {
                                float* y = reinterpret_cast<float*>(p.y) + (int64_t)tok * p.out + f0;
                                *reinterpret_cast<float4*>(y) = make_float4(a.x * sc, a.y * sc, a.z * sc, a.w * sc);
                                *reinterpret_cast<float4*>(y + 4) = make_float4(c.x * sc, c.y * sc, c.z * sc, c.w * sc);
                            }
                        }
                    }
                } else {
                    // one element per store (a lane owns one feature)
                    const bool f_ok = f < p.out;
#pragma unroll
                    for (int j = 0; j < CH; ++j) {
                        const float val = __uint_as_float(v[j]) * wdiv * __shfl_sync(0xffffffffu, rs_lane[h], j);
                        if (f_ok && tokb + j < p.M) {
                            store_out(p.y, p.out_dtype, (int64_t)(tokb + j) * p.out + f, val);
                        }
                    }
                }
            }
        }
        if (giver || takes > 0) {
            // giver: every warp's part is out before the flag goes up; taker: every warp has read the
            // parts before the flags go down again (the next launch's givers write only after this
            // grid has completed).  All sixteen warps meet here whether or not a wait ran out.
            if (giver && ok) __threadfence();
            asm volatile("bar.sync 6, %0;" ::"r"(kDqWarps * 32) : "memory");
            if (dq == 0) {
                if (!giver)
                    for (int k = 1 + lane; k <= (SEGS ? takes : 1); k += 32) p.part_flags[slot + k * CS] = 0;
                else if (ok && lane == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p.part_flags + slot), "r"(1) : "memory");
            }
        }
        if (!SEGS || (left -= n) == 0) break;
        q0 += n;
        ++seg;
        ++tile;
        const int fd2 = tile / p.ttiles;
        ft = fd2 * CS + (int)rank;
        tok0 = (tile - fd2 * p.ttiles) * NTOK;
        if (ok) {   // the accumulators and the activation stages are free for the next segment
            fence_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free);
        }
        }
    }
    if (dbg && tid == 64) { dbg[303] = (unsigned long long)clock64(); dbg[305] = gtime_ns(); }
    tc_fence_before();
    __syncthreads();
    if constexpr (DUO) {
        if (warp != 1) cluster_wait();
        __syncwarp();
        cluster_sync();   // neither CTA leaves, nor frees its tensor memory, under the other's MMAs and arrivals
    }
    if (warp == 1) {
        if constexpr (DUO) tmem_dealloc2(tmem, TMEM_COLS);
        else tmem_dealloc(tmem, TMEM_COLS);
    }
    if (tid == 0 && s_abort) atomicExch(p.status, 2);
}

// ---- host side --------------------------------------------------------------------------
template <int BITS, int NTOK>
static int32_t gemm_attr() {
    if constexpr (NTOK <= 128)
        RSTQ_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<BITS, NTOK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kNST * (kAStage + NTOK * kKStep * 2) + 1024));
    auto smem = [](auto kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
    RSTQ_CUDA(smem(gemm_tmem_kernel<BITS, NTOK, false, false>, gemm_smem(NTOK, false)));
    RSTQ_CUDA(smem(gemm_tmem_kernel<BITS, NTOK, true, false>, gemm_smem(NTOK, false)));
    if constexpr (NTOK == 256) {
        RSTQ_CUDA(smem(gemm_tmem_kernel<BITS, NTOK, false, true>, gemm_smem(NTOK, true)));
        RSTQ_CUDA(smem(gemm_tmem_kernel<BITS, NTOK, true, true>, gemm_smem(NTOK, true)));
    }
    return RSTQ_OK;
}

template <int BITS, int NTOK>
static cudaError_t gemm_launch(const DeviceState& ds, const GemmParams& p, const CUtensorMap& tmap, int ctas, bool general, bool duo) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kGemmThreadsT);
    cfg.dynamicSmemBytes = gemm_smem(NTOK, duo);
    cfg.stream = ds.stream;
    cudaLaunchAttribute a[2];
    int n = 0;
    if (duo) {
        a[n].id = cudaLaunchAttributeClusterDimension;
        a[n].val.clusterDim.x = 2;
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
    if constexpr (NTOK == 256) {
        if (duo) return general ? cudaLaunchKernelEx(&cfg, gemm_tmem_kernel<BITS, NTOK, true, true>, p, tmap)
                                : cudaLaunchKernelEx(&cfg, gemm_tmem_kernel<BITS, NTOK, false, true>, p, tmap);
    }
    return general ? cudaLaunchKernelEx(&cfg, gemm_tmem_kernel<BITS, NTOK, true, false>, p, tmap)
                   : cudaLaunchKernelEx(&cfg, gemm_tmem_kernel<BITS, NTOK, false, false>, p, tmap);
}

int32_t gemm_configure(DeviceState& ds) {
    (void)ds;
    int32_t rc;
    if ((rc = gemm_attr<4, 32>()) != RSTQ_OK) return rc;
    if ((rc = gemm_attr<4, 64>()) != RSTQ_OK) return rc;
    if ((rc = gemm_attr<4, 128>()) != RSTQ_OK) return rc;
    if ((rc = gemm_attr<8, 32>()) != RSTQ_OK) return rc;
    if ((rc = gemm_attr<8, 64>()) != RSTQ_OK) return rc;
    if ((rc = gemm_attr<8, 128>()) != RSTQ_OK) return rc;
    if ((rc = gemm_attr<4, 256>()) != RSTQ_OK) return rc;
    if ((rc = gemm_attr<8, 256>()) != RSTQ_OK) return rc;
    return RSTQ_OK;
}

// x (src 0 = f32, 1 = bf16, 2 / 3 = f32 / bf16 through the int8 quantizer) -> fp16 rows x16 and 2^e per row
template <int SRC>
static cudaError_t act_launch(const DeviceState& ds, const void* x, void* x16, float* rowscale, int64_t M, int64_t in) {
    const dim3 grid((unsigned)M);
    auto go = [&](auto kernel, int t) { return launch_pdl(kernel, grid, dim3((unsigned)t), 0, ds, x, (__half*)x16, rowscale, in); };
    // 32 elements per thread at most, so that a row stays in registers up to 32768 (8192 with 256 threads for any row,
    // before): 4096 x 11008, M = 70, quantized on the way 34.0 -> 28.0 us a call, 8192 x 28672, M = 100 73.5 -> 66.0.  128 threads
    // for short rows: 1000 x 1024, M = 2048 12.8 -> 12.0; at in = 4096 they lose (4096 x 4096, M = 512 22.2 -> 23.2), as 512 threads
    // do at 6016 (3000 x 6016, M = 30 16.9 -> 17.5).  Where the quantizer is on the way a thread has more to do, and fewer of
    // them pay only once 256 for each row do not run at once, eight rows per SM: int8 7520 x 1632, 128 / 256 threads, M = 74 12.5 / 12.1, M = 150
    // 14.3 / 13.6, M = 600 26.5 / 25.9, M = 1200 40.4 / 41.5; 2000 x 2048, M = 600 16.0 / 15.1, M = 2000 24.7 / 26.4; 4096 x 1024, M = 300
    // 10.6 / 10.3, M = 1200 24.9 / 26.3.  Without it 128 are as fast or faster at every M (M = 150 11.8 / 12.7, M = 20 10.2 / 10.2).
    if (in <= 2048 && (SRC < 2 || M > 8 * ds.sm_count)) return go(act_to_f16_kernel<SRC, 128>, 128);
    if (in <= 8192) return go(act_to_f16_kernel<SRC, 256>, 256);
    // Many rows: an SM holds one block of 1024 threads or two of 512, so that loads of the next rows wait for the last ones' reductions;
    // bf16 rows are then read twice by four blocks of 256 per SM sooner (1024 features, 256 / 512 threads: in = 16384, M = 2000 87.6 / 93.4,
    // M = 1000 50.8 / 52.5, M = 520 35.8 / 36.1, M = 300 29.3 / 28.2; f32 102.7 / 102.0 at 2000, quantized 123.5 / 112.1), and others by
    // 512 threads instead of 1024 (in = 20000, M = 2000 f32 130.4 / 140.7; M = 520 47.9 / 48.6, M = 300 34.4 / 34.5, quantized 40.4 / 38.9).
    const int64_t sm = ds.sm_count;
    if (SRC == 1 && M > 4 * sm) return go(act_to_f16_kernel<SRC, 256>, 256);
    if (in <= 16384 || M > (SRC >= 2 ? 3 : 2) * sm) return go(act_to_f16_kernel<SRC, 512>, 512);
    return go(act_to_f16_kernel<SRC, 1024>, 1024);
}
static int32_t launch_act_to_f16(rstq_ctx* ctx, DeviceState& ds, const void* x, int src, void* x16,
                                 float* rowscale, int64_t M, int64_t in) {
    const cudaError_t le = src == 0   ? act_launch<0>(ds, x, x16, rowscale, M, in)
                           : src == 1 ? act_launch<1>(ds, x, x16, rowscale, M, in)
                           : src == 2 ? act_launch<2>(ds, x, x16, rowscale, M, in)
                                      : act_launch<3>(ds, x, x16, rowscale, M, in);
    ctx->launches++;
    RSTQ_CUDA(le);
    return RSTQ_OK;
}

// Token-tile width and split along K of a prefill GEMM on a device of `sm_count` SMs: whichever of
// 128- / 256-wide tiles, one, two or more CTAs per tile, needs the fewest cycles over the waves of CTAs
// the grid makes.  `tmem_kernel`: the call runs gemm_tmem_kernel with a pair scratch (wide tiles and
// the split exist only there); `wide`: RSTQ_TUNE_GEMM_WIDE.
// (measured: a 128-wide K-step 690 cycles; a 256-wide one 1140 with 64 CTAs running, 1240 with 96,
// 1400 with all 148 -- their activation tiles are twice as large and all come from L2; set-up, first
// loads and epilogue of a CTA about 8000 resp. 9000 cycles; the hand-over of a pair about 1500)
// (kRangeCycles: what the second segment of a range costs, in cycles over the plain model.  The model counts neither
// further segments nor the power cap, under which idle SMs buy the others a higher clock: ranges are taken only over at
// most four tiles each, and where it sees 15 % saved; up to 64 tokens, far from the cap, 6 %; against pairs, which wait for no last wave, anything
// (8192 x 28672 at M = 256, bf16: over seconds 124.9 / 126.2, but a first call of both matrices of the 70B-class MLP 228 -> 219).  Measured over seconds, int4 /
// int8, whole tiles or pairs -> ranges, us.  Above the line: 24576 x 3072 at M = 64 29.5 -> 27.0, at M = 20 31.3 -> 26.4;
// 28672 x 4096 at M = 64 43.1 -> 42.3; 28672 x 8192 at M = 32 62.1 -> 57.3, at M = 256 128.3 -> 124.9; 11008 x 4096 at M = 512
// 65.2 -> 64.2 (in a burst 60.4 -> 55.9); 20000 x 2048 at M = 200 37.0 -> 34.2; 14336 x 4096 at M = 512 70.2 -> 69.9.
// Below it, where the model alone would take them: 26000 x 2048 at M = 32 21.5 -> 22.2; 4096 x 4096 at M = 2048 79.6 -> 82.9, 4096 x 11008 at M = 2048
// 189 -> 200, 9000 x 6144 at M = 900 107 -> 112, 27648 x 1024 at M = 256 29.0 -> 31.1, 6144 x 8192 at M = 1024 130 -> 134,
// 5120 x 13824 at M = 300 65.9 -> 67.3.  More than four tiles per range:
// 11008 x 4096 at M = 1024 and 2048, as fast either way.)
constexpr int64_t kRangeCycles = 13000;
// (More than two CTAs per tile, where the tiles are few: equal parts of a tile's steps, one segment each.  The first part's CTA
// waits for all the others' flags at once and adds their sums in order: beside a pair's hand-over about 1500 cycles for the
// kernel that knows segments, and 10 x (tokens of the tile) - 100 per part, which is reading it from L2.  With seven eighths of
// the SMs taken the last CTAs queue behind the pre-pass (6000 x 4096 over 141 of them: M = 64 15.5 -> 16.5 us).  Two CTAs per
// tile, or ranges -> parts, int4 / int8 with bf16 tokens, us: 1024 x 16384 at M = 32 23.4 -> 14.6 (16 parts), 1608 x 9248 at M = 17
// 17.9 -> 13.1, 4096 x 11008 at M = 64 24.3 -> 22.1, at M = 128 28.3 -> 24.8, 4096 x 4096 at M = 32 13.9 -> 12.1 (four), 2592 x 4064 at
// M = 128 17.3 -> 15.8.  On the other side: 1024 x 4096 at M = 128 over 8 parts 16.7, over 16 21.6 (pairs 15.8, four 15.2); 2048 x 2048
// at M = 128 13.6 over three, 12.8 over two; 512 x 1024, K too short to cut, 8.2 whole and 9.1 over four.  256-token tiles are left as they are.
// Ranges instead of parts where they save 2500 cycles' steps: 4096 x 16384 at M = 32 24.2 against 25.2 over four, but
// 4096 x 8192 19.4 against 18.2.)
constexpr int64_t kPartsCycles = 3000, kPartsFull = 2000, kMaxParts = 64, kPartsToRange = 2500;
// (256-token tiles on pairs of CTAs, where every SM has 80 K-steps to do: a K-step takes 7 % less, a launch of clusters about 1.2 us more
// (both SMs of a pair have to be free of the pre-pass), a tile 1800 cycles more, and the tiles are counted in twos: an odd number of
// feature tiles idles a CTA of the last pair, and may need a wave that single CTAs do not.  In a burst / over 0.1 s, us: 70B-class
// MLP at M = 256 (97 steps each) 103.3 -> 97.0 / 116.9 -> 112.1 and 104.7 -> 98.6 / 118.6 -> 114.9; int4 4096 x 8192 at M = 2048 (110)
// 122.3 -> 113.5 / 135.1 -> 128.7; 7168 x 16384 at M = 512 (97) 103.8 -> 99.2 / 118.6 -> 114.4.  Fewer steps: 8192 x 8192 at
// M = 512 (55) 54.5 -> 53.0 / 58.7 -> 60.0, 16384 x 6144 at M = 250 (41) 43.0 -> 41.2 / 43.7 -> 46.1.  Where pairs take a wave more: 6272 x 11008 at
// M = 768 (147 tiles) 98 -> 132, 2688 x 10752 at M = 1792 107 -> 137, 4736 x 5120 at M = 2048 (two waves, three) 101 -> 115, 6272 x 5632 at M = 1536
// 108 -> 122.  Short rows, where the tile's own cycles decide: 28672 x 1056 at M = 2048 201 -> 206, 28280 x 2112 at M = 1177 188 -> 189,
// 28672 x 2048 at M = 1024 149 -> 148.  40 others of 80 .. 180 steps: 0.93 .. 0.99.  Tiles of 128 tokens, as fast
// in the kernel either way, only lose the launch (int8 4096 x 4096 at M = 512 21.5 -> 22.8).)
constexpr int64_t kPairSteps = 80, kPairStep = 93, kPairFixed = 1800;
GemmPlan gemm_plan(int64_t out, int64_t in, int64_t M, int sm_count, bool tmem_kernel, int wide) {
    const int64_t ftiles = (out + 127) / 128, sm = sm_count > 0 ? sm_count : 1;
    const int64_t ksteps_total = (in / 32 + 3) / 4;
    // cs: CTAs of a tile, 1 or 2 (a pair, on a tile of two feature tiles: an odd number of them leaves a CTA of the last pair idle)
    auto tiles_of = [&](int nt, int cs) { return (ftiles + cs - 1) / cs * ((M + nt - 1) / nt); };
    // CTAs that may share tiles: a slot of the scratch (128 x nt sums) and a flag for every one, and all of them on the device at once
    auto sharers = [&](int nt) { return std::min({sm, (int64_t)kGemmSharers, kPairScratchBytes / (128 * 4 * nt)}); };
    auto step_cycles = [&](int nt, int64_t active) { return nt == 256 ? 1140 + (active > 64 ? (active - 64) * 31 / 10 : 0) : (int64_t)690; };
    auto cycles = [&](int nt, int cs, int* parts) {
        const int64_t tiles = tiles_of(nt, cs), places = std::max<int64_t>(1, sm / cs), cap = sharers(nt) / cs;
        const bool split = tmem_kernel && tiles * 2 <= cap && ksteps_total >= 16 && wide != 3;
        const int64_t ctas = (split ? tiles * 2 : tiles) * cs, c = step_cycles(nt, ctas < sm ? ctas : sm) * (cs == 2 ? kPairStep : 100) / 100;
        const int64_t fixed = (nt == 256 ? 9000 : 8000) + (cs == 2 ? kPairFixed : 0);
        int64_t best = split ? (ksteps_total + 1) / 2 * c + 1500 + fixed : (tiles + places - 1) / places * (ksteps_total * c + fixed);
        *parts = split ? 2 : 1;
        for (int64_t k = 3; split && nt <= 128 && k <= ksteps_total && k <= kMaxParts && tiles * k <= cap; ++k) {
            const int64_t n = tiles * k;
            const int64_t t = (ksteps_total + k - 1) / k * c + kPartsCycles + (n * 8 > sm * 7 ? kPartsFull : 0) + (k - 1) * (nt * 10 - 100) + fixed;
            if (t < best) {
                best = t;
                *parts = (int)k;
            }
        }
        return best;
    };
    GemmPlan pl{};
    pl.ntok = M <= 32 ? 32 : (M <= 64 ? 64 : 128);
    int64_t best = cycles(pl.ntok, 1, &pl.parts);
    if (M > 128 && tmem_kernel && wide != 1) {
        int parts = 1;
        const int64_t c = cycles(256, 1, &parts);
        if (wide == 2 || wide >= 5 || c < best) {
            pl.ntok = 256;
            pl.parts = parts;
            best = c;
        }
    }
    // Equal ranges of the step sequence on all SMs instead of whole tiles (or pairs) per thread block: no SM waits
    // for the last wave, at the price of a second segment per thread block (an epilogue, a refill of the pipeline,
    // a hand-over).
    if (tmem_kernel && wide != 3) {
        const int64_t steps = tiles_of(pl.ntok, 1) * ksteps_total, G = std::min(sharers(pl.ntok), steps);
        const int64_t per = (steps + G - 1) / G, c = step_cycles(pl.ntok, G), fixed = pl.ntok == 256 ? 9000 : 8000;
        const int p2 = pl.parts;
        const bool pays = p2 > 2 ? per * c + kPartsToRange + (ksteps_total / per - p2) * (pl.ntok * 10 - 100) < (ksteps_total + p2 - 1) / p2 * c
                                 : per <= 3 * ksteps_total && (per * c + fixed + kRangeCycles) * 100 < best * (p2 == 2 ? 100 : (pl.ntok <= 64 ? 94 : 85));
        if (steps < (1ll << 30) && (wide == 4 || wide == 6 || pays)) {
            pl.ranges = (int)G;
            pl.parts = 1;
        }
    }
    // Pairs, by their own count of tiles, places and slots
    if (pl.ntok == 256 && tmem_kernel && (wide >= 5 || (wide == 0 && tiles_of(256, 1) * ksteps_total >= kPairSteps * sm && ((ftiles & 1) == 0 || ftiles >= 9)))) {
        if (pl.ranges > 0) {
            const int64_t steps = tiles_of(256, 2) * ksteps_total, G = std::max<int64_t>(1, std::min<int64_t>(pl.ranges / 2, steps));
            const int64_t one = tiles_of(256, 1) * ksteps_total, per1 = (one + pl.ranges - 1) / pl.ranges;
            pl.duo = wide >= 5 || (steps + G - 1) / G * kPairStep < per1 * 100;
            if (pl.duo) pl.ranges = (int)G;
        } else {
            int parts = 1;
            const int64_t c = cycles(256, 2, &parts);
            pl.duo = wide >= 5 || c < best;
            if (pl.duo) pl.parts = parts;
        }
    }
    const int cs = pl.duo ? 2 : 1;
    pl.cols = pl.duo && M < 256 ? (int)((M + 31) & ~31ll) : pl.ntok;
    pl.grid = (pl.ranges > 0 ? pl.ranges : tiles_of(pl.ntok, cs) * pl.parts) * cs;
    return pl;
}

// y[M, out] = x[M, in] . dequant(W)^T on the tensor cores.  src: 0 = f32 x, 1 = bf16 x,
// 2 / 3 = f32 / bf16 x through the int8 quantizer.  x16 / rowscale are caller-provided scratch
// (M*in fp16, M floats).
int32_t launch_gemm(rstq_ctx* ctx, DeviceState& ds, const rstq_weight* w, const void* x, int src, void* y,
                    int out_dtype, int64_t M, void* x16, float* rowscale, float* acc32) {
    RSTQ_REQUIRE(M >= 1 && M < (1ll << 30), RSTQ_E_SHAPE, "M = %lld", (long long)M);
    RSTQ_REQUIRE(((uintptr_t)x16 & 15) == 0 && (w->in * 2) % 16 == 0, RSTQ_E_ALIGN,
                 "activation scratch must be 16-byte aligned");
    EncodeTiledFn enc = encode_tiled_fn();
    RSTQ_REQUIRE(enc, RSTQ_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    const bool a_in_tmem = ctx->tune_gemm_kernel != 1;
    // Token-tile width and the split along K.  Above 128 tokens a tile may be 256 wide (gemm_tmem_kernel
    // only): the K loop is bound by the issue of the tensor-core instructions, and an instruction of
    // twice the width does twice the work -- a K-step of a 256-wide tile takes 1140 cycles against
    // 690 of a 128-wide one (measured) -- but halves the number of tiles.  When a grid would fill at
    // most half the SMs and K is long, two CTAs share a tile, each taking half of K; the second hands
    // its accumulator to the first through L2 (about 1500 cycles).  Whichever combination needs the
    // fewest cycles over the waves of CTAs it makes on this device is taken (4096 features: M <= 256: 128
    // wide, split; M = 512: 128 wide, one wave of 128 tiles; M = 768: 256 wide, one wave of 96 tiles
    // instead of two of 192; M >= 1024: 256 wide).
    const GemmPlan pl = gemm_plan(w->out, w->in, M, ds.sm_count, a_in_tmem && acc32 != nullptr, (int)ctx->tune_gemm_wide);
    const int ntok = pl.ntok;
    const bool duo = pl.duo, shared = pl.parts > 1 || pl.ranges > 0;
    // (as gemm_plan has it: a slot of the sums' scratch and a flag for every CTA)
    RSTQ_REQUIRE(!shared || (pl.grid <= kGemmSharers && pl.grid * 128 * ntok * 4 <= kPairScratchBytes), RSTQ_E_LIMIT,
                 "%lld thread blocks share tiles of %d tokens", (long long)pl.grid, ntok);
    // pre-pass: activations -> fp16 with one exponent per token row.  kind::f16 wants A and B of
    // one type (fp16 weights against bf16 activations raise "illegal instruction"), and fp16 on
    // both sides keeps three more mantissa bits of the weights than bf16 would.
    int32_t rc = launch_act_to_f16(ctx, ds, x, src, x16, rowscale, M, w->in);
    if (rc != RSTQ_OK) return rc;
    cudaError_t le;

    CUtensorMap tmap;
    const cuuint64_t dims[2] = {(cuuint64_t)w->in, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)w->in * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)(duo ? ntok / 2 : ntok)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult cr = enc(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x16, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    RSTQ_REQUIRE(cr == CUDA_SUCCESS, RSTQ_E_CUDA, "cuTensorMapEncodeTiled failed with %d", (int)cr);

    GemmParams p{};
    p.w = w->data;
    p.y = y;
    p.rowscale = rowscale;
    p.status = ds.status;
    p.out = w->out;
    p.nb = (int)w->nb;
    p.ngroups = (int)(w->outp / 32);
    p.M = (int)M;
    p.ksteps = (int)((w->nb + 3) / 4);
    p.ttiles = (int)((M + ntok - 1) / ntok);
    // gemm_tmem_kernel converts codes as fp16 subnormals (code * 2^-24): its block scales carry
    // 2^kSubnormalShift more and the result the remaining 2^(24 - kSubnormalShift)
    p.wmul = ldexpf(1.0f, w->gemm_exp + (a_in_tmem ? kSubnormalShift : 0));
    p.wdiv = ldexpf(1.0f, -w->gemm_exp + (a_in_tmem ? 24 - kSubnormalShift : 0));
    p.out_dtype = out_dtype;
    p.cols = pl.cols;
    p.dbg = ds.dbg;
    RSTQ_REQUIRE(pl.grid < (1ll << 30), RSTQ_E_LIMIT, "grid too large");
    // (units: thread blocks, or pairs of them on tiles of 256 features)
    const int64_t cs = duo ? 2 : 1, steps = ((w->out + 127) / 128 + cs - 1) / cs * p.ttiles * p.ksteps;
    p.half = pl.parts == 2 ? (p.ksteps + 1) / 2 : 0;
    p.parts = pl.parts > 2 ? pl.parts : 0;
    p.uq = pl.ranges > 0 ? steps / pl.ranges : p.ksteps;
    p.ur = pl.ranges > 0 ? steps % pl.ranges : 0;
    p.part = acc32;   // [CTA][16 warps][columns per warp][32 lanes] f32: 128 * ntok floats each
    p.part_flags = ds.counters + ds.counters_len - kGemmSharers;
    const bool general = pl.ranges > 0 || pl.parts > 2 || (w->nb & 3) != 0;
    const int grid = (int)pl.grid;
    const size_t smem1 = kNST * (kAStage + (size_t)ntok * kKStep * 2) + 1024;
#define GL(B, N) \
    le = a_in_tmem ? gemm_launch<B, N>(ds, p, tmap, grid, general, duo) \
                   : launch_pdl(gemm_tc_kernel<B, N>, dim3((unsigned)grid), dim3(kGemmThreads), smem1, ds, p, tmap)
    if (w->bits == 4) {
        if (ntok == 32) GL(4, 32);
        else if (ntok == 64) GL(4, 64);
        else if (ntok == 128) GL(4, 128);
        else le = gemm_launch<4, 256>(ds, p, tmap, grid, general, duo);
    } else {
        if (ntok == 32) GL(8, 32);
        else if (ntok == 64) GL(8, 64);
        else if (ntok == 128) GL(8, 128);
        else le = gemm_launch<8, 256>(ds, p, tmap, grid, general, duo);
    }
#undef GL
    ctx->launches++;
    RSTQ_CUDA(le);
    RSTQ_CUDA(cudaGetLastError());
    return RSTQ_OK;
}

}  // namespace rstq
