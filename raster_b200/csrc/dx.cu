// Backward-data of the frozen-weight linear, qlinear-q8-dx (src/raster/quant/train.clj:110-142):
//   dx[m, i] = sum over o of scales[o, i / 32] * codes[o, i] * dy[m, o]
// the dequant-transpose GEMM dX = dY . dequant(W), W = [out, in] signed 8-bit codes in the
// reference's row-major layout with one f32 scale per 32 columns.
//
// Two launches.  dx_prep_kernel rewrites the f32 factors as pairs of fp16 (value = hi + lo, 22 significant
// bits; a power of two per token row / per 32-column block keeps both in range), dx_tmem_kernel is a
// tcgen05 GEMM over them with the weights dequantized on the way into tensor memory:
//
//   D[128 columns i, NT tokens] += W'[i, o] * dy[m, o],  W' = Wh + Wl, dy = Yh + Yl
//                                = Wh Yh + Wh Yl + Wl Yh      (Wl Yl is below 2^-22 of the product)
//
// which is an f32-grade product (measured <= 4e-7 of max|dx| against the f64 oracle) at three fp16 MMAs.
// The f32 scale times an integer code needs no wider arithmetic: with s = sh + sl in fp16,
// Wh = rn(c sh), the residual c sh - Wh is exact in an fp16 fma, Wl = rn(c sl + residual).
//
// What bounds it: the tensor core, nominally 192 cycles per 16 rows o of a 128 x 128 tile.  Yh and Yl lie one
// above the other in shared memory, so Wh times both is ONE instruction of twice the width: two MMAs per 16 rows
// (128 + 64 cycles) instead of three of 64, because a tcgen05 instruction costs its issuer 50 - 60 cycles.
// Measured, us per call back to back (before: bf16 mma.sync with three terms, 263 / 898):
//   4096 x 4096, m = 512: 56.5 (0.91 PFLOP/s of fp16 MMAs; the loop 49, at 1200 cycles per 64 rows and 1.68 GHz:
//   with neither copies nor conversions 1028 -- 1.6 PFLOP/s for the chip, cuBLAS's own rate on it, so what is left
//   is power), m = 2048: 213, m = 64: 23.5
#include "internal.h"
#include "mma_helpers.cuh"
#include "tcgen05_helpers.cuh"

namespace rstq {

constexpr int kDxStep = 64;                    // rows o per pipeline stage
constexpr int kDxStages = 4;                   // dy in shared memory and W' in tensor memory
constexpr int kDxRaw = 8;                      // codes and scales in shared memory
constexpr int kDxSet = 8;                      // dequant warps of a stage: 4 blocks of 32 columns x 2 halves of its rows
constexpr int kDxDq = 2 * kDxSet;              // two sets on alternate stages
constexpr int kDxThreads = (kDxDq + 3) * 32;   // + two copy warps and the MMA warp
constexpr int kDxCodes = kDxStep * 128;        // bytes of codes per stage
constexpr int kDxScales = 1024;                // bytes of scales per stage: 64 rows x 4 blocks
constexpr int kDxRawBytes = kDxCodes + kDxScales;
__host__ __device__ constexpr int dx_ring_bytes(int nt) { return kDxStages * 2 * nt * 128 + kDxRaw * kDxRawBytes; }

// Position p of an element inside its group of 16 rows o: the order in which a lane of the dequant warps holds
// them (rows 2t, 2t + 1, 2t + 8, 2t + 9 for t = p / 4).  Any order serves, as long as dy has the same one; this
// one reads the 128-byte-swizzled code tile without bank conflicts.
__host__ __device__ constexpr int dx_row_of(int p) { return 2 * (p >> 2) + (p & 1) + ((p & 2) ? 8 : 0); }

// ---- what the GEMM needs beforehand: dy as fp16 pairs, the largest scale of every column block ------
constexpr int kDxParts = 64;                   // thread blocks that look at the scales, each at its share of the rows o
struct DxPrep {
    const float* dy;
    const float* scales;
    __half *yh, *yl;        // [m][opad]
    int* rowexp;            // [m]: e, the row holds dy * 2^-e with max|.| in [2^13, 2^14)
    float* colmax;          // [kDxParts][nb]: max|scale| of a part's rows
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
    e = e < -149 ? -149 : e;   // 2^-149 is the smallest f32
    const int e1 = e < -100 ? -100 : e;
    *down = ldexpf(1.0f, -e1);
    *down2 = ldexpf(1.0f, e1 - e);
    return e;
}
// v * 2^e.  In two halves, whose powers f32 holds and between which nothing leaves its range that the result does
// not leave; below 2^-252 every v here (< 2^60) ends as zero.  (ldexpf does the same 3 us slower over 512 x 4096 results.)
__device__ __forceinline__ float dx_scale(float v, int e) {
    e = e < -252 ? -252 : e;
    const int h = e >> 1;
    return v * __int_as_float((h + 127) << 23) * __int_as_float((e - h + 127) << 23);
}
__device__ __forceinline__ float dx_block_max(float mx, float* red) {   // 256 threads
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) mx = fmaxf(mx, red[i]);
    __syncthreads();
    return mx;
}
__device__ __forceinline__ void dx_split(float a, float b, uint32_t* hi, uint32_t* lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    // (an infinity has no remainder)
    const __half2 l = __floats2half2_rn(fabsf(f.x) < 7e4f ? a - f.x : 0.f, fabsf(f.y) < 7e4f ? b - f.y : 0.f);
    *hi = *reinterpret_cast<const uint32_t*>(&h);
    *lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Latency-bound: every element is read once into registers (rows up to 8192), found the maximum of, and written
// as two halves; the blocks that look at the scales read theirs as one run and leave a maximum per column block
// (a strip of column blocks per thread block instead took 45 us at 4096 x 4096: 16 bytes of every row).
constexpr int kDxMaxCols = 4096;
__global__ void __launch_bounds__(256)
dx_prep_kernel(const DxPrep p) {
    __shared__ float s_red[8];
    __shared__ uint32_t s_max[kDxMaxCols];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x < kDxParts) {
        const int64_t o0 = p.out * blockIdx.x / kDxParts, o1 = p.out * (blockIdx.x + 1) / kDxParts;
        for (int64_t c0 = 0; c0 < p.nb; c0 += kDxMaxCols) {     // (one pass up to 131 072 columns i)
            const int nc = (int)(p.nb - c0 < kDxMaxCols ? p.nb - c0 : kDxMaxCols);
            for (int c = threadIdx.x; c < nc; c += 256) s_max[c] = 0u;
            __syncthreads();
            // a thread keeps its columns (four where rows are whole 16 bytes) and steps over the rows
            const bool vec = (p.nb & 3) == 0;
            const int cols = vec ? nc >> 2 : nc, groups = cols < 256 ? 256 / cols : 1;
            const int rg = (int)threadIdx.x / cols;
            if (rg < groups || cols >= 256) {
                for (int c = (int)threadIdx.x - rg * cols; c < cols; c += 256) {
                    float4 mx = make_float4(0.f, 0.f, 0.f, 0.f);
                    const float* q = p.scales + c0 + (vec ? 4 * c : c);
#pragma unroll 8
                    for (int64_t o = o0 + (cols < 256 ? rg : 0); o < o1; o += groups) {
                        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (vec) v = __ldg(reinterpret_cast<const float4*>(q + o * p.nb));
                        else v.x = __ldg(q + o * p.nb);
                        mx.x = fmaxf(mx.x, fabsf(v.x));
                        mx.y = fmaxf(mx.y, fabsf(v.y));
                        mx.z = fmaxf(mx.z, fabsf(v.z));
                        mx.w = fmaxf(mx.w, fabsf(v.w));
                    }
                    // (the bits of magnitudes order like the magnitudes)
                    if (vec) {
                        atomicMax(&s_max[4 * c], __float_as_uint(mx.x));
                        atomicMax(&s_max[4 * c + 1], __float_as_uint(mx.y));
                        atomicMax(&s_max[4 * c + 2], __float_as_uint(mx.z));
                        atomicMax(&s_max[4 * c + 3], __float_as_uint(mx.w));
                    } else {
                        atomicMax(&s_max[c], __float_as_uint(mx.x));
                    }
                }
            }
            __syncthreads();
            for (int c = threadIdx.x; c < nc; c += 256) p.colmax[(int64_t)blockIdx.x * p.nb + c0 + c] = __uint_as_float(s_max[c]);
            __syncthreads();
        }
        return;
    }
    const int64_t m = (int64_t)blockIdx.x - kDxParts;
    const float* src = p.dy + m * p.out;
    const bool vec = (p.out & 3) == 0;
    auto load16 = [&](int64_t o, float (&v)[16]) {   // o a multiple of 16
        if (vec && o + 16 <= p.out) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 f = __ldg(reinterpret_cast<const float4*>(src + o) + j);
                v[4 * j] = f.x; v[4 * j + 1] = f.y; v[4 * j + 2] = f.z; v[4 * j + 3] = f.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = o + j < p.out ? __ldg(src + o + j) : 0.f;
        }
    };
    constexpr int kKeep = 2;   // x 256 threads x 16 elements
    const bool keep = p.opad <= kKeep * 256 * 16;
    float held[kKeep][16];
    float mx = 0.f;
    if (keep) {
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int64_t o = (int64_t)(i * 256 + threadIdx.x) * 16;
            if (o < p.opad) {
                load16(o, held[i]);
#pragma unroll
                for (int j = 0; j < 16; ++j) mx = fmaxf(mx, fabsf(held[i][j]));
            }
        }
    } else {
        for (int64_t o = threadIdx.x * 16; o < p.opad; o += 256 * 16) {
            load16(o, held[0]);
#pragma unroll
            for (int j = 0; j < 16; ++j) mx = fmaxf(mx, fabsf(held[0][j]));
        }
    }
    float down, down2;
    const int e = dx_exponent(dx_block_max(mx, s_red), 14, &down, &down2);
    auto store16 = [&](int64_t o, const float (&v)[16]) {
        uint32_t h[8], l[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)   // half2 q: positions 2q, 2q + 1
            dx_split(v[dx_row_of(2 * q)] * down * down2, v[dx_row_of(2 * q + 1)] * down * down2, &h[q], &l[q]);
        uint4* dh = reinterpret_cast<uint4*>(p.yh + m * p.opad + o);
        uint4* dl = reinterpret_cast<uint4*>(p.yl + m * p.opad + o);
        dh[0] = make_uint4(h[0], h[1], h[2], h[3]);
        dh[1] = make_uint4(h[4], h[5], h[6], h[7]);
        dl[0] = make_uint4(l[0], l[1], l[2], l[3]);
        dl[1] = make_uint4(l[4], l[5], l[6], l[7]);
    };
    if (keep) {
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int64_t o = (int64_t)(i * 256 + threadIdx.x) * 16;
            if (o < p.opad) store16(o, held[i]);
        }
    } else {
        for (int64_t o = threadIdx.x * 16; o < p.opad; o += 256 * 16) {
            load16(o, held[0]);
            store16(o, held[0]);
        }
    }
    if (threadIdx.x == 0) p.rowexp[m] = e;
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

__device__ __forceinline__ uint32_t hsub2_u32(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds_u128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
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
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The MMAs of one stage (64 rows o) as one block of instructions: per 16 rows Wh against (Yh, Yl) and Wl against
// Yh.  The barrier of the next stage is tested among them and the answer read at the end: tested after the last
// MMA instead, the round trips of the tests left the tensor core idle for 400 of 1225 cycles per stage.
__device__ __forceinline__ uint32_t dx_mma_step(uint32_t d, uint32_t w, uint32_t b_lo, uint32_t b_hi, uint32_t id_both, uint32_t id_hi,
                                                uint32_t accumulate, uint32_t leader, uint32_t next_bar, uint32_t next_parity) {
    uint32_t next_ready;
    asm volatile(
        "{\n"
        ".reg .pred p, q, t, r;\n"
        ".reg .b64 b0, b1, b2, b3;\n"
        ".reg .b32 h1, h2, h3, l0, l1, l2, l3, b;\n"
        "setp.ne.b32 p, %7, 0;\n"
        "setp.ne.b32 q, %8, 0;\n"
        "setp.eq.b32 t, 0, 0;\n"
        "mov.b64 b0, {%3, %4};\n"
        "add.u32 b, %3, 2; mov.b64 b1, {b, %4};\n"
        "add.u32 b, %3, 4; mov.b64 b2, {b, %4};\n"
        "add.u32 b, %3, 6; mov.b64 b3, {b, %4};\n"
        "add.u32 h1, %2, 8;  add.u32 h2, %2, 16; add.u32 h3, %2, 24;\n"
        "add.u32 l0, %2, 32; add.u32 l1, %2, 40; add.u32 l2, %2, 48; add.u32 l3, %2, 56;\n"
        "tcgen05.fence::after_thread_sync;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], b0, %5, p;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [l0], b0, %6, t;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [h1], b1, %5, t;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [l1], b1, %6, t;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [h2], b2, %5, t;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [l2], b2, %6, t;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 r, [%9], %10;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [h3], b3, %5, t;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [l3], b3, %6, t;\n"
        "selp.u32 %0, 1, 0, r;\n"
        "}"
        : "=r"(next_ready)
        : "r"(d), "r"(w), "r"(b_lo), "r"(b_hi), "r"(id_both), "r"(id_hi), "r"(accumulate), "r"(leader), "r"(next_bar), "r"(next_parity)
        : "memory");
    return next_ready;
}

// Warps 0 .. 15 dequantize and store the tile (warp & 3 = 32-column block = its tensor-memory lanes, (warp >> 2) & 1 =
// half of the stage's rows o, warp >> 3 = even / odd stages), warp 16 copies codes and scales, 17 issues the MMAs, 18 copies dy.  The codes have a
// ring of their own, twice as deep: one ring for everything made a stage wait for copy, conversion and MMA in turn
// (3000 cycles; with four stages 1250 per step against the 768 of the MMAs).  Tensor memory: columns 0 .. NT-1 hold
// Wh Yh + Wl Yh, NT .. 2 NT-1 Wh Yl, 256 .. 511 the ring of W' (32 columns Wh, 32 Wl per stage).
// Tensor-memory lane gid + 8 r of a block is column 4 gid + r of it: a lane of the dequant warp reads the codes
// of four neighbouring columns as one word per row, and the 16x256b store wants exactly these four lanes of it.
// Every mbarrier wait is time-bounded; on expiry the block reports through the status word, lets its copies
// land, still meets its barriers and frees its tensor memory.
template <int NT>
__global__ void __launch_bounds__(kDxThreads, 1)
dx_tmem_kernel(const DxParams p, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_h,
               const __grid_constant__ CUtensorMap map_l, const __grid_constant__ CUtensorMap map_s) {
    constexpr int YB = NT * 128;                 // bytes of Yh (or Yl) per stage
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_abort;
    __shared__ uint32_t s_tmem;
    __shared__ int s_colexp[4];
    __shared__ __align__(8) uint64_t s_bar[2 * kDxStages + 2 * kDxRaw + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem), bar0 = smem_u32(s_bar);
    // ready: the stage of dy has arrived and its W' is in tensor memory; empty: its MMAs are done;
    // raw: codes and scales of a step have arrived; taken: they are in registers
    const uint32_t ready = bar0, empty = bar0 + 8 * kDxStages;
    const uint32_t raw = bar0 + 16 * kDxStages, taken = raw + 8 * kDxRaw, acc_full = taken + 8 * kDxRaw;
    const uint32_t rbase = sbase + kDxStages * 2 * YB;
    const int part = blockIdx.x % p.split, tile = blockIdx.x / p.split;
    const int ft = tile / p.ttiles, tok0 = (tile - ft * p.ttiles) * NT;
    const int k0 = (int)((int64_t)p.steps * part / p.split), k1 = (int)((int64_t)p.steps * (part + 1) / p.split);
    volatile int* abort_flag = &s_abort;

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_h)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_l)) : "memory");
    }
    if (tid < kDxStages) {
        mbar_init(ready + 8 * tid, kDxSet + 1);
        mbar_init(empty + 8 * tid, 1);
    }
    if (tid < kDxRaw) {
        mbar_init(raw + 8 * tid, 1);
        mbar_init(taken + 8 * tid, kDxSet);
    } else if (tid == kDxRaw) {
        mbar_init(acc_full, 1);
        s_abort = 0;
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

    bool ok = true;
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
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int s = 0, issued = 0;
            uint32_t ph = 0;
            for (int k = k0; k < k1; ++k) {
                ok = mbar_block(empty + 8 * s, ph ^ 1u, abort_flag);
                if (!ok) break;
                const uint32_t dst = sbase + s * 2 * YB, bar = ready + 8 * s;
                mbar_expect_tx(bar, 2 * YB);
                tma_load_2d(dst, &map_h, k * kDxStep, tok0, bar);
                tma_load_2d(dst + YB, &map_l, k * kDxStep, tok0, bar);
                ++issued;
                if (++s == kDxStages) { s = 0; ph ^= 1u; }
            }
            if (!ok) dx_drain(ready, issued, kDxStages);
        }
    } else if (warp == kDxDq + 1) {
        // ---------------- MMAs ----------------
        constexpr uint32_t id_both = idesc_f16(2 * NT), id_hi = idesc_f16(NT);
        const uint32_t leader = lane == 0;
        const uint64_t d0 = smem_desc_sw128(sbase);
        const uint32_t d_lo = (uint32_t)d0, d_hi = (uint32_t)(d0 >> 32);
        int s = 0;
        uint32_t ph = 0;
        bool any = false;
        ok = mbar_spin(ready, 0, abort_flag);
        for (int k = k0; k < k1 && ok; ++k) {
            const int s2 = s + 1 == kDxStages ? 0 : s + 1;
            const uint32_t ph2 = s2 ? ph : ph ^ 1u;
            const uint32_t n2 = dx_mma_step(tmem, tmem + 256 + s * 64, d_lo + (uint32_t)s * (2 * YB >> 4), d_hi, id_both, id_hi, k != k0,
                                            leader, ready + 8 * s2, ph2);
            umma_commit_if(empty + 8 * s, leader);
            any = true;
            if (k + 1 < k1 && !n2) ok = mbar_spin(ready + 8 * s2, ph2, abort_flag);
            s = s2;
            ph = ph2;
        }
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
        const uint32_t tdst = tmem + 256 + ((uint32_t)(blk * 32) << 16) + half * 16;
        const int64_t nb = p.in >> 5, b = (int64_t)ft * 4 + blk;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        float mx = 0.f;
        if (b < nb)
            for (int i = lane; i < kDxParts; i += 32) mx = fmaxf(mx, __ldg(p.colmax + i * nb + b));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float down, down2;   // the block's scales are used times 2^-ce, the largest in [2^6, 2^7)
        const int ce = dx_exponent(mx, 7, &down, &down2);
        if (lane == 0) s_colexp[blk] = ce;   // (the four warps of a block of columns agree)
        int s = set, rs = set;
        uint32_t ph = 0, rph = 0;
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
            // split it, and gather the eight the lane's rows need: (sh, sh), (sh, sh), (sl, sl), (sl, sl) per group
            uint32_t mine;
            {
                const float v = sf * down * down2;
                const __half h = __float2half_rn(v), l = __float2half_rn(v - __half2float(h));
                mine = (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(l) << 16);
            }
            uint4 sc[2];
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                uint32_t v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = __shfl_sync(0xffffffffu, mine, (g * 4 + j) * 4 + t);
                sc[g] = make_uint4(__byte_perm(v[0], v[1], 0x5410), __byte_perm(v[2], v[3], 0x5410),
                                   __byte_perm(v[0], v[1], 0x7632), __byte_perm(v[2], v[3], 0x7632));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(taken + 8 * rs);
            rs += 2;
            if (rs >= kDxRaw) { rs -= kDxRaw; rph ^= 1u; }
            ok = __all_sync(0xffffffffu, mbar_block(empty + 8 * s, ph ^ 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int q = 0; q < 2; ++q) {      // columns 4 gid + 2q, + 2q + 1
                uint32_t vh[8], vl[8];
#pragma unroll
                for (int g = 0; g < 2; ++g)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const uint32_t sel = (2 * q + c) | ((4 + 2 * q + c) << 8);   // this column's byte of the two rows; the odd bytes are masked away
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t sh = h ? sc[g].y : sc[g].x, sl = h ? sc[g].w : sc[g].z;
                            // (code ^ 0x80) under the exponent byte of 1024 is 1024 + 128 + code exactly
                            const uint32_t e = __byte_perm(w[g][2 * h], w[g][2 * h + 1], sel);
                            const uint32_t v = hsub2_u32((e & 0x00FF00FFu) ^ 0x64806480u, 0x64806480u);
                            const uint32_t hi = hmul2_u32(v, sh);
                            const uint32_t rest = hfma2_u32(v, sh, hi ^ 0x80008000u);
                            vh[g * 4 + c * 2 + h] = hi;
                            vl[g * 4 + c * 2 + h] = hfma2_u32(v, sl, rest);
                        }
                    }
                tmem_st_16x256b_x2(tdst + s * 64 + ((uint32_t)(16 * q) << 16), vh);
                tmem_st_16x256b_x2(tdst + s * 64 + 32 + ((uint32_t)(16 * q) << 16), vl);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * s);
            s += 2;
            if (s >= kDxStages) { s -= kDxStages; ph ^= 1u; }
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
#pragma unroll
            for (int j = 0; j < CH; ++j) {
                const float v = __uint_as_float(a[j]) + __uint_as_float(b[j]);
                const int tok = tok0 + col + j;
                // (both exponents at once: one of them alone can take a finite result through infinity or zero)
                if (p.split > 1) s_out[(col + j) * 128 + blk * 32 + 4 * (lane & 7) + (lane >> 3)] = v;
                else if (tok < p.m && i_ok) p.dx[(int64_t)tok * p.in + i] = dx_scale(v, ce + __ldg(p.rowexp + tok));
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
                    p.dx[(int64_t)tok * p.in + i] = dx_scale(v, s_colexp[c >> 5] + __ldg(p.rowexp + tok));
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

static bool dx_map(EncodeTiledFn enc, CUtensorMap* map, CUtensorMapDataType type, const void* base, int64_t x, int64_t y,
                   int64_t stride, int box_x, int box_y, bool swizzle = true) {
    const cuuint64_t dims[2] = {(cuuint64_t)x, (cuuint64_t)y}, strides[1] = {(cuuint64_t)stride};
    const cuuint32_t box[2] = {(cuuint32_t)box_x, (cuuint32_t)box_y}, estr[2] = {1, 1};
    return enc(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
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
static cudaError_t dx_launch(const DeviceState& ds, const DxParams& p, int tiles, const CUtensorMap& w, const CUtensorMap& h,
                             const CUtensorMap& l, const CUtensorMap& s) {
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
    return cudaLaunchKernelEx(&cfg, dx_tmem_kernel<NT>, p, w, h, l, s);
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

    const int64_t yb = (m * opad * 2 + 255) & ~255ll, rb = (m * 4 + 255) & ~255ll, cb = kDxParts * nb * 4;
    int32_t rc = dev_reserve_any_time(ds, &ds.dx_scratch, &ds.dx_scratch_bytes, 2 * yb + rb + cb);
    if (rc != RSTQ_OK) return rc;
    char* base = (char*)ds.dx_scratch;
    DxPrep q{dy, scales, (__half*)base, (__half*)(base + yb), (int*)(base + 2 * yb), (float*)(base + 2 * yb + rb),
             m, out, nb, opad};
    CUtensorMap mw, mh, ml, ms;
    const bool tma_scales = nb % 4 == 0;   // rows of whole 16 bytes
    RSTQ_REQUIRE(dx_map(enc, &mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, codes, in, out, in, 128, kDxStep) &&
                     dx_map(enc, &mh, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, q.yh, opad, m, opad * 2, kDxStep, nt) &&
                     dx_map(enc, &ml, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, q.yl, opad, m, opad * 2, kDxStep, nt) &&
                     (!tma_scales || dx_map(enc, &ms, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, scales, nb, out, nb * 4, 4, kDxStep, false)),
                 RSTQ_E_CUDA, "cuTensorMapEncodeTiled failed (m = %lld, in = %lld, out = %lld)", (long long)m, (long long)in,
                 (long long)out);
    if (!tma_scales) ms = mw;   // not used then
    RSTQ_CUDA(launch_pdl(dx_prep_kernel, dim3((unsigned)(m + kDxParts)), dim3(256), 0, ds, q));
    ctx->launches++;
    DxParams p{scales, q.rowexp, q.colmax, dx, ds.status, in, out, tma_scales, (int)m, (int)steps, (int)ttiles, split};
    RSTQ_CUDA(nt == 32   ? dx_launch<32>(ds, p, (int)tiles, mw, mh, ml, ms)
              : nt == 64 ? dx_launch<64>(ds, p, (int)tiles, mw, mh, ml, ms)
                         : dx_launch<128>(ds, p, (int)tiles, mw, mh, ml, ms));
    ctx->launches++;
    return RSTQ_OK;
}

}  // namespace rstq
