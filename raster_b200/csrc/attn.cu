// The attention steps of the decoder layer's decode chain (one token), f32, so that the chain
// norm -> quantize -> q/k/v matmuls -> rope -> cache append -> attention -> o matmul stays on the
// device and in one CUDA graph:
//   rope      rope-pos-gpu! / rope-pos-buf!            src/raster/dl/attention.clj:386-408, :482-499
//   append    kv-append! / kv-append-buf!              attention.clj:413-416, :501-504
//   attention gqa-decode-attention-gpu! / -buf!        attention.clj:423-471, :514-575
// The position / cache length is a host scalar or, when a one-element int64 device buffer is given,
// read inside the kernel (the reference's -buf variants), so a captured graph serves every token.
//
// Attention is one kernel where the reference has three phases: a CTA owns one KV head, a slice of
// the cache positions and up to four (eight in the general kernel) query heads of the group, which it serves from the K / V rows
// it reads once (the reference reads them once per query head); warps walk the positions with an online
// softmax (running max, sum and weighted V in registers), the warps of a CTA are merged through
// shared memory, and the slices of a KV head through distributed shared memory where they are a cluster, else through
// a small scratch in device memory, from which one CTA writes out = sum_j p_j v_j.  The reference's score scratch `sc` is not used.
// head_dim 64 and 128 take gqa_decode_stream_kernel (rows through shared memory, eight positions per
// warp step); every other head_dim % 4 == 0 up to 256 takes the general gqa_decode_kernel (a
// warp per position).
#include <algorithm>

#include "internal.h"
#include "quant_helpers.cuh"
#include "sync_helpers.cuh"

namespace rstq {

constexpr int kAttnWarps = 8;
constexpr int kAttnGroup = 8;     // query heads of one KV head served by a CTA
constexpr int kAttnVec = 2;       // float4 per lane along head_dim: head_dim <= 256
constexpr int kAttnCounters = 1024;
constexpr float kNegInf = -1.0e38f;   // the reference's sentinel below any real score

// A position or length in device memory, read from L2: a kernel that looks at it before its wait for the kernel
// ahead, which may still write it, looks again afterwards.
__device__ __forceinline__ int64_t ld_i64(const int64_t* p) {
    int64_t v;
    asm volatile("ld.volatile.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__global__ void __launch_bounds__(256)
rope_pos_kernel(const float* __restrict__ x, float* __restrict__ out, int64_t heads, int64_t head_dim, double ln_theta,
                int64_t pos, const int64_t* __restrict__ posbuf) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t h2 = head_dim >> 1;
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= heads * h2) return;
    const int64_t h = idx / h2, i = idx - h * h2;
    const double p = (double)(posbuf ? posbuf[0] : pos);
    const double freq = exp((-2.0 * (double)i) / (double)head_dim * ln_theta);
    double s, c;
    sincos(p * freq, &s, &c);
    const double x0 = (double)x[h * head_dim + i], x1 = (double)x[h * head_dim + i + h2];
    out[h * head_dim + i] = (float)(x0 * c - x1 * s);
    out[h * head_dim + i + h2] = (float)(x1 * c + x0 * s);
}

__global__ void __launch_bounds__(256)
kv_append_kernel(const float* __restrict__ src, float* __restrict__ cache, int64_t kvrow, int64_t pos,
                 const int64_t* __restrict__ posbuf) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t p = posbuf ? posbuf[0] : pos;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < kvrow; i += (int64_t)gridDim.x * blockDim.x)
        cache[p * kvrow + i] = src[i];
}

// rope(q), rope(k), append k, append v of one token in ONE launch (four steps of the reference's
// chain): q is turned in place; k is turned, stored back and written to its cache row; v is copied
// to its cache row.  One thread per rotation pair of q and k, and per pair of v elements.
__global__ void __launch_bounds__(256)
rope_append_kernel(float* __restrict__ q, float* __restrict__ k, const float* __restrict__ v,
                   float* __restrict__ kcache, float* __restrict__ vcache, int64_t n_q, int64_t n_kv, int64_t head_dim,
                   double ln_theta, int64_t pos, const int64_t* __restrict__ posbuf) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t h2 = head_dim >> 1, kvrow = n_kv * head_dim;
    const int64_t nrot = (n_q + n_kv) * h2, idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t h = idx / h2, i = idx - h * h2;
    // The double-precision chain (exp, then sincos) is this kernel's time: it runs while the kernel before this one
    // finishes, for a position in device memory from what it holds by then and again should that change (four 7B
    // layers at one token: exp alone 222.3 -> 220.0 us, the rest 208.6 -> 206.6).
    const double freq = exp((-2.0 * (double)i) / (double)head_dim * ln_theta);
    const int64_t early = posbuf ? ld_i64(posbuf) : pos;
    double s, c;
    sincos((double)early * freq, &s, &c);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t p = posbuf ? ld_i64(posbuf) : pos;
    if (p != early) sincos((double)p * freq, &s, &c);
    if (idx < nrot) {
        const bool isk = h >= n_q;
        float* x = isk ? k + (h - n_q) * head_dim : q + h * head_dim;
        const double x0 = (double)x[i], x1 = (double)x[i + h2];
        const float y0 = (float)(x0 * c - x1 * s), y1 = (float)(x1 * c + x0 * s);
        x[i] = y0;
        x[i + h2] = y1;
        if (isk) {
            float* dst = kcache + p * kvrow + (h - n_q) * head_dim;
            dst[i] = y0;
            dst[i + h2] = y1;
        }
    } else if (idx < nrot + n_kv * h2) {
        const int64_t e = (idx - nrot) * 2;
        *reinterpret_cast<float2*>(vcache + p * kvrow + e) = *reinterpret_cast<const float2*>(v + e);
    }
}

struct AttnParams {
    const float *q, *k, *v;
    float* out;
    float* part;     // [n_kv][gz][S][kAttnGroup][head_dim + 4]: weighted V, running max, sum, 2 pad
    int* counters;   // [n_kv * gz], zero between launches
    const int64_t* clenbuf;
    int64_t cache_len;
    int n_q, group, n_kv, head_dim, S;
    float scale;
    int gs;          // query heads per CTA as the scratch is laid out
    int64_t maxpos;
    int* status;
    // optional: the output quantized to int8 blocks of 32 as well (the o projection's input), by the
    // CTA that writes it; only with head_dim % 32 == 0 (a warp then owns whole blocks)
    int8_t* xq;
    float* xs;
    int32_t* xsum;
};

// (a length in device memory never reaches beyond the caches)
__device__ __forceinline__ int64_t attn_len(const AttnParams& p) {
    const int64_t n = p.clenbuf ? ld_i64(p.clenbuf) : p.cache_len;
    return n < 0 ? 0 : (n > p.maxpos ? p.maxpos : n);
}

// one value of the output, and with it -- when asked for -- its 32-element quantizer block (the 32
// lanes of the warp hold 32 consecutive elements of one head)
__device__ __forceinline__ void attn_store(const AttnParams& p, int64_t e, float v, int lane) {
    p.out[e] = v;
    if (p.xq) {
        int q, sm;
        float scale;
        quant_block32(v, &q, &sm, &scale);
        uint32_t word = (uint32_t)(q & 0xFF) << (8 * (lane & 3));
        word |= __shfl_xor_sync(0xffffffffu, word, 1);
        word |= __shfl_xor_sync(0xffffffffu, word, 2);
        const int64_t blk = e >> 5;
        if ((lane & 3) == 0) reinterpret_cast<uint32_t*>(p.xq)[blk * 8 + (lane >> 2)] = word;
        if (lane == 0) {
            p.xs[blk] = scale;
            if (p.xsum) p.xsum[blk] = sm;
        }
    }
}

// Second half of the general kernel: the per-warp states in shared memory ([warps][gc][row]: weighted V, max, sum) are
// merged per CTA, then per KV head across the slices of the cache.
__device__ __forceinline__ void attn_finish(const AttnParams& p, float* s_part, int* s_last_p, int gc, int g0, int hkv,
                                            int split, int gz, int hd, int row) {
    __shared__ float s_cw[kAttnGroup][kAttnWarps];   // weight of each warp's state in the CTA's state
    __shared__ float s_cM[kAttnGroup], s_cL[kAttnGroup];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (warp < gc && lane < kAttnWarps) {            // warp g merges the eight (max, sum) pairs of head g
        const float* st = s_part + (lane * gc + warp) * row + hd;
        const float mw = st[0], lw = st[1];
        float M = mw;
#pragma unroll
        for (int o = kAttnWarps / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFu, M, o));
        const float e = expf(mw - M);
        float L = lw * e;
#pragma unroll
        for (int o = kAttnWarps / 2; o > 0; o >>= 1) L += __shfl_xor_sync(0xFFu, L, o);
        s_cw[warp][lane] = e;
        if (lane == 0) {
            s_cM[warp] = M;
            s_cL[warp] = L;
        }
    }
    __syncthreads();
    // CTA state per (g, d): straight to out when there is one slice, else to the scratch
    float* mine = p.part + ((((int64_t)hkv * gridDim.z + gz) * p.S + split) * kAttnGroup) * row;
    for (int i = threadIdx.x; i < gc * hd; i += blockDim.x) {
        const int g = i / hd, d = i - g * hd;
        const float* base = s_part + g * row + d;
        float O = 0.f;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) O = fmaf(base[w * gc * row], s_cw[g][w], O);
        if (p.S == 1) attn_store(p, (int64_t)(hkv * p.group + g0 + g) * hd + d, O * (1.0f / s_cL[g]), lane);
        else mine[g * row + d] = O;
    }
    if (p.S > 1 && threadIdx.x < gc) {
        mine[threadIdx.x * row + hd] = s_cM[threadIdx.x];
        mine[threadIdx.x * row + hd + 1] = s_cL[threadIdx.x];
    }
    if (p.S == 1) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const int prev = atomicAdd(p.counters + hkv * gridDim.z + gz, 1);
        *s_last_p = prev == p.S - 1;
        if (*s_last_p) p.counters[hkv * gridDim.z + gz] = 0;   // ready for the next launch / graph replay
        __threadfence();
    }
    __syncthreads();
    if (!*s_last_p) return;
    // The last CTA of this KV head merges the S slices.  What it reads -- maxima, sums, weighted V -- lies a trip to L2
    // away, and three such trips in a row were most of this tail: warp g takes the (max, sum) pairs of head g, up
    // to kPairs per lane at once (128 slices: more than one per SM is rare), while every thread requests its first kHold
    // weighted values; then the slice weights exp(m_s - M) go round through shared memory (the per-warp states are dead
    // by now; the host keeps S + 1 <= 8 * row).
    const float* all = p.part + (((int64_t)hkv * gridDim.z + gz) * p.S * kAttnGroup) * row;
    const int S = p.S;
    float* s_w = s_part;            // [gc][S] weights
    float* s_L = s_part + gc * S;   // [gc]
    constexpr int kPairs = 4, kHold = 20;
    float held[kHold];
    {
        const int i = threadIdx.x, g = i / hd, d = i - g * hd;
        const float* col = all + (int64_t)g * row + d;
#pragma unroll
        for (int k = 0; k < kHold; ++k) held[k] = i < gc * hd && k < S ? __ldcg(col + (int64_t)k * kAttnGroup * row) : 0.f;
    }
    if (warp < gc) {
        const float* st = all + (int64_t)warp * row + hd;
        float M = kNegInf, Lsum = 0.f, mv[kPairs], lv[kPairs];
#pragma unroll
        for (int k = 0; k < kPairs; ++k) {
            const int sl = lane + 32 * k;
            mv[k] = sl < S ? __ldcg(st + (int64_t)sl * kAttnGroup * row) : kNegInf;
            lv[k] = sl < S ? __ldcg(st + (int64_t)sl * kAttnGroup * row + 1) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < kPairs; ++k) M = fmaxf(M, mv[k]);
        for (int sl = lane + 32 * kPairs; sl < S; sl += 32) M = fmaxf(M, __ldcg(st + (int64_t)sl * kAttnGroup * row));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
        for (int k = 0; k < kPairs; ++k) {
            const int sl = lane + 32 * k;
            if (sl < S) {
                const float e = expf(mv[k] - M);
                Lsum = fmaf(lv[k], e, Lsum);
                s_w[warp * S + sl] = e;
            }
        }
        for (int sl = lane + 32 * kPairs; sl < S; sl += 32) {
            const float e = expf(__ldcg(st + (int64_t)sl * kAttnGroup * row) - M);
            Lsum = fmaf(__ldcg(st + (int64_t)sl * kAttnGroup * row + 1), e, Lsum);
            s_w[warp * S + sl] = e;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) Lsum += __shfl_xor_sync(0xffffffffu, Lsum, o);
        if (lane == 0) s_L[warp] = Lsum;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < gc * hd; i += blockDim.x) {
        const int g = i / hd, d = i - g * hd;
        const float* col = all + (int64_t)g * row + d;
        float O = 0.f;
        int sl = 0;
        if (i == (int)threadIdx.x) {
#pragma unroll
            for (int k = 0; k < kHold; ++k)
                if (k < S) O = fmaf(held[k], s_w[g * S + k], O);
            sl = kHold;
        }
#pragma unroll 8
        for (; sl < S; ++sl) O = fmaf(__ldcg(col + (int64_t)sl * kAttnGroup * row), s_w[g * S + sl], O);
        attn_store(p, (int64_t)(hkv * p.group + g0 + g) * hd + d, O * (1.0f / s_L[g]), lane);
    }
}

__global__ void __launch_bounds__(kAttnWarps * 32)
gqa_decode_kernel(const AttnParams p) {
    extern __shared__ __align__(16) float s_part[];   // [kAttnWarps][gc][hd + 4]
    __shared__ int s_last;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hkv = blockIdx.x, split = blockIdx.y, gz = blockIdx.z;
    const int hd = p.head_dim, hd4 = hd >> 2, row = hd + 4;   // row: weighted V, max, sum, 2 pad (16-byte rows)
    const int g0 = gz * kAttnGroup;
    const int gc = min(kAttnGroup, p.group - g0);            // query heads this CTA serves
    const int64_t clen = attn_len(p);
    const int64_t chunk = (clen + p.S - 1) / p.S;
    const int64_t j0 = split * chunk, j1 = min(clen, j0 + chunk);
    const int64_t kvstride = (int64_t)p.n_kv * hd;
    const float4* kb = reinterpret_cast<const float4*>(p.k + (int64_t)hkv * hd);
    const float4* vb = reinterpret_cast<const float4*>(p.v + (int64_t)hkv * hd);

    // this lane's slice of every served query head, pre-multiplied by the score scale
    float4 qv[kAttnGroup][kAttnVec];
    float4 acc[kAttnGroup][kAttnVec];
    float m[kAttnGroup], l[kAttnGroup];
#pragma unroll
    for (int g = 0; g < kAttnGroup; ++g) {
        m[g] = kNegInf;
        l[g] = 0.f;
#pragma unroll
        for (int u = 0; u < kAttnVec; ++u) {
            acc[g][u] = make_float4(0.f, 0.f, 0.f, 0.f);
            const int c = lane + u * 32;
            qv[g][u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (g < gc && c < hd4) {
                const float4 t = reinterpret_cast<const float4*>(p.q + (int64_t)(hkv * p.group + g0 + g) * hd)[c];
                qv[g][u] = make_float4(t.x * p.scale, t.y * p.scale, t.z * p.scale, t.w * p.scale);
            }
        }
    }
    for (int64_t j = j0 + warp; j < j1; j += kAttnWarps) {
        float4 kk[kAttnVec], vv[kAttnVec];
#pragma unroll
        for (int u = 0; u < kAttnVec; ++u) {
            const int c = lane + u * 32;
            kk[u] = vv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c < hd4) {
                kk[u] = __ldg(kb + j * (kvstride >> 2) + c);
                vv[u] = __ldg(vb + j * (kvstride >> 2) + c);
            }
        }
#pragma unroll
        for (int g = 0; g < kAttnGroup; ++g) {
            if (g < gc) {
                float s = 0.f;
#pragma unroll
                for (int u = 0; u < kAttnVec; ++u)
                    s = fmaf(qv[g][u].x, kk[u].x, fmaf(qv[g][u].y, kk[u].y, fmaf(qv[g][u].z, kk[u].z, fmaf(qv[g][u].w, kk[u].w, s))));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                const float mn = fmaxf(m[g], s);
                const float corr = expf(m[g] - mn), pj = expf(s - mn);
                m[g] = mn;
                l[g] = fmaf(l[g], corr, pj);
#pragma unroll
                for (int u = 0; u < kAttnVec; ++u) {
                    acc[g][u].x = fmaf(acc[g][u].x, corr, pj * vv[u].x);
                    acc[g][u].y = fmaf(acc[g][u].y, corr, pj * vv[u].y);
                    acc[g][u].z = fmaf(acc[g][u].z, corr, pj * vv[u].z);
                    acc[g][u].w = fmaf(acc[g][u].w, corr, pj * vv[u].w);
                }
            }
        }
    }
    // warps -> shared memory
#pragma unroll
    for (int g = 0; g < kAttnGroup; ++g) {
        if (g < gc) {
            float* dst = s_part + (warp * gc + g) * row;
#pragma unroll
            for (int u = 0; u < kAttnVec; ++u) {
                const int c = lane + u * 32;
                if (c < hd4) reinterpret_cast<float4*>(dst)[c] = acc[g][u];
            }
            if (lane == 0) {
                dst[hd] = m[g];
                dst[hd + 1] = l[g];
            }
        }
    }
    attn_finish(p, s_part, &s_last, gc, g0, hkv, split, gz, hd, row);
}

// ---- head_dim 64 and 128 ----------------------------------------------------------------------
// Streams its slice of K and V through shared memory: a CTA of 16 warps per SM (with many KV heads four CTAs of four), serving
// up to four query heads of a KV head from rows that it reads once (larger groups find them in L2).  Each warp works alone on
// tiles of eight positions, with a ring of its own that cp.async keeps full, so the bytes in flight do not depend on registers:
//   scores   eight lanes share a position; the sums of 8 positions x H heads over those lanes are reduced by halving
//            (7 shuffles for 32 values), which leaves one (position, head) per lane: one exp per value
//   softmax  online per tile (a maximum over eight positions, a rescale only where a maximum moved)
//   output   a lane owns four dims of all heads, p comes back as one broadcast load per position
// and the warps' states meet once, at the end.  The slices of a KV head then meet in one of two ways (attention_impl says
// which): as a cluster of up to eight, each CTA merging its share of the output from the others' shared memory; or
// through slots in device memory that hold kEmpty between launches: the CTA of the last slice polls for the values
// themselves (no fence, counter or flag stands between a store and its reader), merges and empties them.  It waits only
// for CTAs launched before it.
// What bounds it: an SM takes in its 190 - 230 KB at about 65 B/ns, whether they come from HBM or L2; then a tail (the last
// tile, the warps' merge, the slices' merge) of about 4 us through slots and 2.5 as a cluster, of which little is arithmetic.
// us, back to back over 0.3 GB of caches in turn, against the kernel before it (two heads per CTA, rows through registers):
// through slots 32 q / 8 kv heads x 4096 13.9 -> 11.7, 64 / 8 x 2000 12.8 -> 10.7, 28 / 4 x 5000 14.4 -> 12.2, 32 / 16 x 2000
// 11.8 -> 10.2, x 40000 99.7 -> 100.2, 64 / 8 x 8000 of 64 elements 23.7 -> 14.8; as clusters 32 / 32 x 1000 11.1 -> 9.1, 32 / 8 x 1000
// 8.9 -> 7.7, 32 / 16 x 500 8.6 -> 6.3; four 7B layers at 1024 positions 222.5 -> 195.4.  Slower than that: two KV heads of 64 elements at 2500
// positions (7.3 -> 8.5), 15 / 5 x 1800 of 64 (8.3 -> 8.7).
// Tried and slower: one bulk copy per row instead of cp.async (20 cycles each, the first tile 2.3 us after the wait); a counter
// that the last CTA to arrive reads instead of the polled slots (a tail of 4.4 us); slots read before the weights are
// ready (most are empty then, and the second look costs a trip: 11.5 -> 12.4); eight heads per CTA in two passes
// (28 / 4 x 5000 16.1); packed f32x2 arithmetic (11.8 -> 12.4).
constexpr int kTilePos = 8;
constexpr int kStreamWarps = 16;                      // one such CTA per SM ...
constexpr int kNarrowWarps = 4;                       // ... or, with many KV heads, four of these
constexpr int kStreamHeads = 4;                       // query heads of one KV head per CTA
constexpr int kHintPos = 16;                          // positions per warp of a CTA requested into L2 ahead of time
constexpr uint32_t kEmpty = 0xFFFFFFFFu;              // a NaN that no arithmetic produces
__host__ __device__ constexpr int attn_unit_bytes(int hd) { return kTilePos * hd * 4; }      // a tile's rows of K, or of V
// A warp's ring: K and V of one tile of 128 elements, of two of 64 (128 KB in flight per SM).  192 KB, as at first, was slower almost
// everywhere, as if SMs got in each other's way: 32 q / 8 kv heads x 4096 12.6 -> 11.7 us, 32 / 32 x 1000 9.7 -> 9.1, x 16384 83.7 ->
// 78.8, 32 / 16 x 40000 105.7 -> 101.5.  The CTAs of four warps stay with that, which also keeps them at four per SM: with less, a
// fifth finds room and the slices no longer spread evenly (160 / 160 x 2000 of 64 elements 29.4 -> 34.9).
__host__ __device__ constexpr int attn_ring(int warps) { return warps == kStreamWarps ? 8192 : 12288; }
__host__ __device__ constexpr int attn_units(int hd, int warps) { return attn_ring(warps) / attn_unit_bytes(hd); }
// shared memory: the warps' rings, the query heads, the warps' p
__host__ __device__ constexpr int attn_q_off(int warps) { return warps * attn_ring(warps); }
__host__ __device__ constexpr int attn_p_off(int hd, int warps) { return attn_q_off(warps) + kStreamHeads * hd * 4; }
__host__ __device__ constexpr int attn_smem(int hd, int warps) { return attn_p_off(hd, warps) + warps * kTilePos * kStreamHeads * 4; }
// ... and, once the rings are drained, in their place: the warps' states, then the merge of the slices
constexpr int kClusterMax = 8;                        // slices of a KV head that may be one cluster
// bytes of K and V that a slice may grow by for it: about 1 us of its stream at four query heads, half as much again at one or
// two, whose positions cost less arithmetic
constexpr int64_t attn_cluster_extra(int64_t heads) { return heads > 2 ? 65000 : 96000; }
constexpr int kMaxSlices = 160;                       // five (max, sum) pairs per lane of the merging warps
__host__ __device__ constexpr int attn_w_off(int hd, int warps) { return warps * kStreamHeads * (hd + 4) * 4; }       // slice weights
__host__ __device__ constexpr int attn_o_off(int hd, int warps) { return attn_w_off(hd, warps) + kStreamHeads * kMaxSlices * 4; }  // partial outputs
static_assert(attn_o_off(128, kStreamWarps) + kStreamWarps * 32 * 16 <= attn_q_off(kStreamWarps) &&
                  attn_o_off(128, kNarrowWarps) + kNarrowWarps * 32 * 16 <= attn_q_off(kNarrowWarps),
              "the merge fits where the rings were");
static_assert(kNarrowWarps >= kStreamHeads && kNarrowWarps * 32 >= kStreamHeads * 128 / 4, "a warp per head, a thread per four dims in the merge");

// slots: a value is there once it is not kEmpty.  Written and polled with strong (relaxed) accesses, for the value is the
// hand-over; each word says for itself that it is there, so no order between them is needed.
__device__ __forceinline__ float4 slot_read4(const float4* a) {
    float4 v;
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ float2 slot_read2(const float2* a) {
    float2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ bool slot_full(float v) { return __float_as_uint(v) != kEmpty; }
__device__ __forceinline__ bool slot_full(const float4 v) { return slot_full(v.x) && slot_full(v.y) && slot_full(v.z) && slot_full(v.w); }
__device__ __forceinline__ bool slot_full(const float2 v) { return slot_full(v.x) && slot_full(v.y); }
__device__ __forceinline__ float slot_value(float v) { return slot_full(v) ? v : __uint_as_float(0x7FFFFFFFu); }
__device__ __forceinline__ void slot_write(float4* a, float4 v) {
    asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(a), "f"(slot_value(v.x)), "f"(slot_value(v.y)),
                 "f"(slot_value(v.z)), "f"(slot_value(v.w))
                 : "memory");
}
__device__ __forceinline__ void slot_write(float2* a, float2 v) {
    asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1,%2};" ::"l"(a), "f"(slot_value(v.x)), "f"(slot_value(v.y)) : "memory");
}
__device__ __forceinline__ float4 slot_empty4() {
    const float e = __uint_as_float(kEmpty);
    return make_float4(e, e, e, e);
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void attn_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a value at the same place of a cluster's CTA `rank`
__device__ __forceinline__ float ld_cluster(uint32_t at, int rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(at), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// H = query heads of the KV head that a CTA serves at most (1, 2 or 4).  CL: the slices of a KV head are one cluster.
// WARPS: of the CTA; an SM holds kStreamWarps in all.
template <int HD, int H, bool CL, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, kStreamWarps / WARPS)
gqa_decode_stream_kernel(const AttnParams p) {
    constexpr int THREADS = WARPS * 32;
    constexpr int VEC = HD / 32, ROW = HD + 4;      // VEC: float4 per lane of a position's eight lanes
    constexpr uint32_t ROWB = HD * 4, UNITB = attn_unit_bytes(HD);
    constexpr int NU = attn_units(HD, WARPS);                              // units of the ring: K and V of a tile in turn
    constexpr int LPP = HD / 4, PPS = 32 / LPP;                     // output: lanes per position, positions per step
    extern __shared__ __align__(128) uint8_t s_raw[];
    __shared__ int s_abort;
    __shared__ float s_cw[kStreamHeads][WARPS], s_cM[kStreamHeads], s_cL[kStreamHeads], s_L[kStreamHeads];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = lane >> 3, sub = lane & 7;
    const int hkv = blockIdx.x, split = blockIdx.y, gz = blockIdx.z;
    const int g0 = gz * kStreamHeads, gc = min(kStreamHeads, p.group - g0);
    const int64_t kvrow = (int64_t)p.n_kv * HD;
    const float* kb = p.k + (int64_t)hkv * HD;
    const float* vb = p.v + (int64_t)hkv * HD;
    const uint32_t base = smem_u32(s_raw), ring = base + warp * attn_ring(WARPS);
    volatile int* abort_flag = &s_abort;

    if (tid == 0) s_abort = 0;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // (a length in device memory may still change: here it only says which rows of the cache to ask for)
    auto range = [&](int64_t* j0, int64_t* j1) {
        const int64_t clen = attn_len(p);
        const int64_t chunk = (clen + p.S - 1) / p.S;
        *j0 = min(clen, split * chunk);
        *j1 = min(clen, *j0 + chunk);
    };
    int64_t j0, j1;
    range(&j0, &j1);
    for (int i = tid; i < kHintPos * WARPS * 2 * (HD / 32); i += THREADS) {     // (128 bytes each)
        const int r = i / (HD / 32), c = i % (HD / 32);
        const int64_t j = j0 + (r >> 1);
        if (j < j1) asm volatile("prefetch.global.L2 [%0];" ::"l"(((r & 1) ? vb : kb) + j * kvrow + c * 32));
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (p.clenbuf) range(&j0, &j1);

    const int tiles = (int)((j1 - j0 + kTilePos - 1) / kTilePos);
    const int mine = tiles > warp ? (tiles - warp + WARPS - 1) / WARPS : 0;   // tiles warp, warp + WARPS, ...
    auto request = [&](int u) {    // unit u: K (even) or V (odd) of this warp's tile u / 2; an empty group beyond the last
        if (u < 2 * mine) {
            const int64_t j = j0 + (int64_t)(warp + (u >> 1) * WARPS) * kTilePos;
            const int np = (int)(j1 - j < kTilePos ? j1 - j : kTilePos);
            const uint32_t dst = ring + (u % NU) * UNITB + lane * 16;
            const float* src = ((u & 1) ? vb : kb) + (j + lane / LPP) * kvrow + (lane % LPP) * 4;
#pragma unroll
            for (int t = 0; t < kTilePos / PPS; ++t)
                if (t * PPS + lane / LPP < np)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + t * PPS * ROWB), "l"(src + t * PPS * kvrow) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto arrived = [&]() {         // the oldest unit requested is in shared memory
        asm volatile("cp.async.wait_group %0;" ::"n"(NU - 1) : "memory");
        __syncwarp();
    };
#pragma unroll 1
    for (int u = 0; u < NU; ++u) request(u);
    float4* s_q = reinterpret_cast<float4*>(s_raw + attn_q_off(WARPS));
    for (int i = tid; i < H * (HD / 4); i += THREADS) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < gc * (HD / 4)) t = reinterpret_cast<const float4*>(p.q + (int64_t)(hkv * p.group + g0) * HD)[i];
        s_q[i] = make_float4(t.x * p.scale, t.y * p.scale, t.z * p.scale, t.w * p.scale);
    }
    __syncthreads();

    const uint32_t qa = base + attn_q_off(WARPS) + sub * 16;
    float* s_p = reinterpret_cast<float*>(s_raw + attn_p_off(HD, WARPS)) + warp * (kTilePos * H);
    const uint32_t pa = smem_u32(s_p);
    float4 acc[H];
    float m = kNegInf, l = 0.f;     // of the head this lane holds scores of
#pragma unroll
    for (int h = 0; h < H; ++h) acc[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    // what the halving leaves in this lane: position 4 (sub & 1) + grp, head lane_h
    const int lane_pos = 4 * (sub & 1) + grp;
    const int lane_h = H == 4 ? ((sub >> 1) & 1) * 2 + (sub >> 2) : (H == 2 ? (sub >> 1) & 1 : 0);
#pragma unroll 1
    for (int i = 0; i < mine; ++i) {
        const int64_t j = j0 + (int64_t)(warp + i * WARPS) * kTilePos;
        const int np = (int)(j1 - j < kTilePos ? j1 - j : kTilePos);
        const uint32_t ka = ring + (2 * i % NU) * UNITB, va = ring + ((2 * i + 1) % NU) * UNITB;
        arrived();
        float4 kk[2][VEC];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int u = 0; u < VEC; ++u) kk[t][u] = ld_shared_f4(ka + (4 * t + grp) * ROWB + (sub + 8 * u) * 16);
        __syncwarp();
        request(2 * i + NU);
        float v[2 * H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int u = 0; u < VEC; ++u) {
                const float4 qq = ld_shared_f4(qa + h * ROWB + u * 128);
                s0 = fmaf(qq.x, kk[0][u].x, fmaf(qq.y, kk[0][u].y, fmaf(qq.z, kk[0][u].z, fmaf(qq.w, kk[0][u].w, s0))));
                s1 = fmaf(qq.x, kk[1][u].x, fmaf(qq.y, kk[1][u].y, fmaf(qq.z, kk[1][u].z, fmaf(qq.w, kk[1][u].w, s1))));
            }
            v[h] = s0;
            v[H + h] = s1;
        }
#pragma unroll
        for (int n = H, o = 1; o < 8; n >>= 1, o <<= 1) {
            if (n >= 1) {        // 2 n values -> n: the lane keeps the half its bit names
                const bool up = sub & o;
#pragma unroll
                for (int k = 0; k < n; ++k) {
                    const float give = up ? v[k] : v[n + k], keep = up ? v[n + k] : v[k];
                    v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            } else {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            }
        }
        const bool valid = lane_pos < np;
        float mx = valid ? v[0] : kNegInf;
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float mn = fmaxf(m, mx);
        const float pj = valid ? expf(v[0] - mn) : 0.f;
        if (__any_sync(0xffffffffu, mn != m)) {
            const float corr = expf(m - mn);
            l *= corr;
            m = mn;
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const float c = __shfl_sync(0xffffffffu, corr, H == 4 ? (h >> 1) * 2 + (h & 1) * 4 : 2 * h);
                float4& a = acc[h];
                a = make_float4(a.x * c, a.y * c, a.z * c, a.w * c);
            }
        }
        l += pj;
        s_p[lane_pos * H + lane_h] = pj;
        arrived();         // V of the tile; and s_p is written
        auto add = [&](int pos) {
            const float4 vv = ld_shared_f4(va + pos * ROWB + (lane % LPP) * 16);
            float pv[H];
            if constexpr (H >= 4) {
#pragma unroll
                for (int h = 0; h < H; h += 4) *reinterpret_cast<float4*>(&pv[h]) = ld_shared_f4(pa + (pos * H + h) * 4);
            } else {
#pragma unroll
                for (int h = 0; h < H; ++h) pv[h] = s_p[pos * H + h];
            }
#pragma unroll
            for (int h = 0; h < H; ++h) {
                acc[h].x = fmaf(pv[h], vv.x, acc[h].x);
                acc[h].y = fmaf(pv[h], vv.y, acc[h].y);
                acc[h].z = fmaf(pv[h], vv.z, acc[h].z);
                acc[h].w = fmaf(pv[h], vv.w, acc[h].w);
            }
        };
        if (np == kTilePos) {
#pragma unroll
            for (int t = 0; t < kTilePos; t += PPS) add(t + lane / LPP);
        } else {      // (rows that were not copied are left out, not multiplied by zero)
#pragma unroll 1
            for (int pos = lane / LPP; pos < np; pos += PPS) add(pos);
        }
        __syncwarp();   // every lane is done with V and s_p
        request(2 * i + 1 + NU);
    }

    // ---- the warps' states -> the CTA's ----
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 8);
    l += __shfl_xor_sync(0xffffffffu, l, 16);
    if (PPS == 2) {
#pragma unroll
        for (int h = 0; h < H; ++h) {
            acc[h].x += __shfl_xor_sync(0xffffffffu, acc[h].x, 16);
            acc[h].y += __shfl_xor_sync(0xffffffffu, acc[h].y, 16);
            acc[h].z += __shfl_xor_sync(0xffffffffu, acc[h].z, 16);
            acc[h].w += __shfl_xor_sync(0xffffffffu, acc[h].w, 16);
        }
    }
    __syncthreads();    // the rings are drained: their place is free
    float* s_part = reinterpret_cast<float*>(s_raw);     // [warp][gc][ROW]: weighted V, max, sum
#pragma unroll
    for (int h = 0; h < H; ++h)
        if (h < gc && lane < LPP) reinterpret_cast<float4*>(s_part + (warp * gc + h) * ROW)[lane] = acc[h];
    if (lane_h < gc && grp == 0) {       // (the lanes of a head agree)
        s_part[(warp * gc + lane_h) * ROW + HD] = m;
        s_part[(warp * gc + lane_h) * ROW + HD + 1] = l;
    }
    __syncthreads();
    if (warp < gc && lane < WARPS) {          // warp h merges the (max, sum) pairs of head h
        const float* s = s_part + (lane * gc + warp) * ROW + HD;
        const float mw = s[0], lw = s[1];
        float M = mw;
#pragma unroll
        for (int o = WARPS / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync((1u << WARPS) - 1u, M, o));
        const float e = expf(mw - M);
        float L = lw * e;
#pragma unroll
        for (int o = WARPS / 2; o > 0; o >>= 1) L += __shfl_xor_sync((1u << WARPS) - 1u, L, o);
        s_cw[warp][lane] = e;
        if (lane == 0) {
            s_cM[warp] = M;
            s_cL[warp] = L;
        }
    }
    __syncthreads();
    const int cols = gc * LPP, S = p.S;              // float4 columns of the CTA's output (at most 128)
    float4* s_o = reinterpret_cast<float4*>(s_raw + attn_o_off(HD, WARPS));
    float* all = p.part + ((int64_t)hkv * gridDim.z + gz) * S * (p.gs * ROW);
    float* out_part = all + (int64_t)split * (p.gs * ROW);
    if (tid < cols) {
        const int h = tid / LPP, c = tid - h * LPP;
        float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float4 a = reinterpret_cast<const float4*>(s_part + (w * gc + h) * ROW)[c];
            const float e = s_cw[h][w];
            O.x = fmaf(a.x, e, O.x);
            O.y = fmaf(a.y, e, O.y);
            O.z = fmaf(a.z, e, O.z);
            O.w = fmaf(a.w, e, O.w);
        }
        if (CL || S == 1) s_o[tid] = O;      // (without a cluster, the one slice's state is the result's)
        else slot_write(reinterpret_cast<float4*>(out_part + h * ROW) + c, O);
    }
    if constexpr (CL) {
        // The slices' states -> out, through distributed shared memory: a warp takes 32 neighbouring values of a head.
        attn_cluster_sync();
        const uint32_t o = smem_u32(s_o), m_at = smem_u32(s_cM), l_at = smem_u32(s_cL);
        for (int b = split + S * warp; b < gc * (HD / 32); b += S * WARPS) {
            const int e = b * 32 + lane, h = b / (HD / 32);
            float Os[kClusterMax], Ms[kClusterMax], Ls[kClusterMax], M = kNegInf, L = 0.f, O = 0.f;
#pragma unroll
            for (int k = 0; k < kClusterMax; ++k)
                if (k < S) {
                    Ms[k] = ld_cluster(m_at + h * 4, k);
                    Ls[k] = ld_cluster(l_at + h * 4, k);
                    Os[k] = ld_cluster(o + e * 4, k);
                }
#pragma unroll
            for (int k = 0; k < kClusterMax; ++k)
                if (k < S) M = fmaxf(M, Ms[k]);
#pragma unroll
            for (int k = 0; k < kClusterMax; ++k)
                if (k < S) {
                    const float w = expf(Ms[k] - M);
                    L = fmaf(Ls[k], w, L);
                    O = fmaf(Os[k], w, O);
                }
            attn_store(p, (int64_t)(hkv * p.group + g0) * HD + e, O * (1.0f / L), lane);
        }
        attn_cluster_sync();   // nobody leaves while its shared memory is read
        return;
    }
    int groups = 1;
    if (S == 1) {
        if (tid < gc) s_L[tid] = 1.0f / s_cL[tid];
    } else {
        if (tid < gc) slot_write(reinterpret_cast<float2*>(out_part + tid * ROW + HD), make_float2(s_cM[tid], s_cL[tid]));
        if (split != S - 1) return;
        // ---- the slices' states -> out: the CTA of the last slice ----
        // What it reads lies a trip to L2 away, so it is requested kHold float4 per thread at a time (slices g, g + groups,
        // ...).  The code is run once and cold: short loops rather than unrolled ones.
        // At least kSlotsPerThread slices each: with one (and the rest of what it holds read for nothing) the addition of up to 32
        // groups' partial outputs took longer than it saved (2 / 2 heads x 1600 of 64 elements 8.0 -> 7.4 us, 32 / 16 x 2000
        // 10.5 -> 10.1).
        constexpr int kHold = 10, kSlotsPerThread = 4;
        groups = min(THREADS / cols, (S + kSlotsPerThread - 1) / kSlotsPerThread);
        const int g = tid / cols, c = tid - g * cols, ch = c / LPP, pitch = p.gs * ROW;
        float* s_w = reinterpret_cast<float*>(s_raw + attn_w_off(HD, WARPS));     // [gc][S]: maxima, then weights
        float4* col = reinterpret_cast<float4*>(all + ch * ROW) + (c - ch * LPP);
        float4 held[kHold];
        auto hold = [&](int from) {       // (beyond the last slice that one again, without a branch: it is not looked at)
#pragma unroll
            for (int k = 0; k < kHold; ++k) held[k] = slot_read4(col + min(from + k * groups, S - 1) * (pitch / 4));
        };
        unsigned long long t0 = 0;
        uint32_t polls = 0;
        bool ok = true;
        auto patience = [&]() {           // (the timer is slow to read: not while there is hope)
            if ((++polls & 255u) != 0) return true;
            const unsigned long long now = gtime_ns();
            if (t0 == 0) t0 = now;
            if (!*abort_flag && now - t0 <= kWaitLimitNs) return true;
            *abort_flag = 1;
            return ok = false;
        };
        if (warp < gc) {
            float M = kNegInf, L = 0.f, ls[kMaxSlices / 32];
#pragma unroll
            for (int k = 0; k < kMaxSlices / 32; ++k) {
                const int sl = lane + 32 * k;
                ls[k] = 0.f;
                if (sl < S) {
                    float2* at = reinterpret_cast<float2*>(all + sl * pitch + warp * ROW + HD);
                    float2 v;
                    do v = slot_read2(at);
                    while (!slot_full(v) && patience());
                    *at = make_float2(__uint_as_float(kEmpty), __uint_as_float(kEmpty));
                    s_w[warp * S + sl] = v.x;
                    ls[k] = v.y;
                    M = fmaxf(M, v.x);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
            for (int k = 0; k < kMaxSlices / 32; ++k) {
                const int sl = lane + 32 * k;
                if (sl < S) {
                    const float e = expf(s_w[warp * S + sl] - M);
                    s_w[warp * S + sl] = e;
                    L = fmaf(ls[k], e, L);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
            if (lane == 0) s_L[warp] = 1.0f / L;
        }
        __syncthreads();
        if (g < groups) {
            const float* w = s_w + ch * S;
            float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (int from = g; from < S; from += kHold * groups) {
                hold(from);
                for (;;) {
                    bool full = true;
#pragma unroll
                    for (int k = 0; k < kHold; ++k) full &= from + k * groups >= S || slot_full(held[k]);
                    if (full || !patience()) break;
                    hold(from);
                }
#pragma unroll
                for (int k = 0; k < kHold; ++k) {
                    const int sl = from + k * groups;
                    if (sl < S) {
                        col[sl * (pitch / 4)] = slot_empty4();
                        const float e = w[sl];
                        O.x = fmaf(held[k].x, e, O.x);
                        O.y = fmaf(held[k].y, e, O.y);
                        O.z = fmaf(held[k].z, e, O.z);
                        O.w = fmaf(held[k].w, e, O.w);
                    }
                }
            }
            s_o[tid] = O;     // [group][column]
        }
        if (!ok) atomicExch(p.status, 2);
    }
    __syncthreads();
    // the groups' partial outputs, [group][gc * HD], added up
    const float* o = reinterpret_cast<const float*>(s_o);
#pragma unroll 1
    for (int i = tid; i < gc * HD; i += THREADS) {
        float v = o[i];
#pragma unroll 1
        for (int g = 1; g < groups; ++g) v += o[g * gc * HD + i];
        attn_store(p, (int64_t)(hkv * p.group + g0) * HD + i, v * s_L[i / HD], lane);
    }
}

// cluster: thread blocks along y that are one
template <typename K, typename... Args>
static cudaError_t launch_attn_cluster(K kernel, dim3 grid, dim3 block, size_t smem, const DeviceState& ds, unsigned cluster, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ds.stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (ds.pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = attr[n].val.clusterDim.z = 1;
        attr[n++].val.clusterDim.y = cluster;
    }
    cfg.attrs = attr;
    cfg.numAttrs = (unsigned)n;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename K, typename... Args>
static cudaError_t launch_attn(K kernel, dim3 grid, dim3 block, size_t smem, const DeviceState& ds, Args... args) {
    return launch_attn_cluster(kernel, grid, block, smem, ds, 1u, args...);
}

template <int HD, int H>
static int32_t attn_attrs() {
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    RSTQ_CUDA(cudaFuncSetAttribute((gqa_decode_stream_kernel<HD, H, false, kStreamWarps>), attr, attn_smem(HD, kStreamWarps)));
    RSTQ_CUDA(cudaFuncSetAttribute((gqa_decode_stream_kernel<HD, H, true, kStreamWarps>), attr, attn_smem(HD, kStreamWarps)));
    RSTQ_CUDA(cudaFuncSetAttribute((gqa_decode_stream_kernel<HD, H, true, kNarrowWarps>), attr, attn_smem(HD, kNarrowWarps)));
    return RSTQ_OK;
}
// how many clusters of each size the device holds at once (148 SMs, 16 warps: 74, 45, 33, 26, 22, 15, 15)
template <int WARPS>
static int32_t attn_count_clusters(int (&count)[kClusterMax + 1]) {
    for (int c = 2; c <= kClusterMax; ++c) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, (unsigned)c);
        cfg.blockDim = dim3(WARPS * 32);
        cfg.dynamicSmemBytes = attn_smem(128, WARPS);
        cudaLaunchAttribute a[1];
        a[0].id = cudaLaunchAttributeClusterDimension;
        a[0].val.clusterDim.x = a[0].val.clusterDim.z = 1;
        a[0].val.clusterDim.y = (unsigned)c;
        cfg.attrs = a;
        cfg.numAttrs = 1;
        RSTQ_CUDA(cudaOccupancyMaxActiveClusters(&count[c], (gqa_decode_stream_kernel<128, 4, true, WARPS>), &cfg));
    }
    return RSTQ_OK;
}
// Scratch of both kernels, the most that a call can need (0.3 and 2.5 MB): a call under capture needs no call before it,
// and a recorded launch and rstq_sync's reset always mean the same blocks.  Slices that meet through slots are at most as
// many in all as the device has SMs (attention_impl's S; clusters need none), those of the general kernel twice as many.
static int32_t attn_reserve(DeviceState& ds) {
    const int64_t slots = (int64_t)ds.sm_count * kStreamHeads * (128 + 4) * 4;
    RSTQ_CUDA(cudaMalloc(&ds.attn_slots, (size_t)slots));
    ds.attn_slots_bytes = slots;
    RSTQ_CUDA(cudaMemsetAsync(ds.attn_slots, 0xFF, (size_t)slots, ds.stream));
    const int64_t states = 2ll * ds.sm_count * kAttnGroup * (128 * kAttnVec + 4) * 4;
    RSTQ_CUDA(cudaMalloc(&ds.attn_scratch, (size_t)(kAttnCounters * 4 + states)));
    RSTQ_CUDA(cudaMemsetAsync(ds.attn_scratch, 0, kAttnCounters * 4, ds.stream));
    return RSTQ_OK;
}
int32_t attn_configure(DeviceState& ds) {
    int32_t rc = attn_reserve(ds);
    if (rc == RSTQ_OK) rc = attn_attrs<64, 1>();
    if (rc == RSTQ_OK) rc = attn_attrs<64, 2>();
    if (rc == RSTQ_OK) rc = attn_attrs<64, 4>();
    if (rc == RSTQ_OK) rc = attn_attrs<128, 1>();
    if (rc == RSTQ_OK) rc = attn_attrs<128, 2>();
    if (rc == RSTQ_OK) rc = attn_attrs<128, 4>();
    if (rc == RSTQ_OK) rc = attn_count_clusters<kStreamWarps>(ds.attn_clusters);
    if (rc == RSTQ_OK) rc = attn_count_clusters<kNarrowWarps>(ds.attn_narrow_clusters);
    return rc;
}

}  // namespace rstq

using namespace rstq;

static bool attn_buf(const rstq_buf* b, const rstq_ctx* ctx, int64_t bytes) {
    return b && b->magic == kBufMagic && b->ctx == ctx && b->bytes >= bytes && ((uintptr_t)b->ptr & 15) == 0;
}

extern "C" {

int32_t rstq_rope_pos(rstq_ctx* ctx, rstq_buf* x, rstq_buf* out, rstq_buf* posbuf, int64_t heads,
                      int64_t head_dim, double theta, int64_t pos) {
    RSTQ_REQUIRE(ctx && ctx->magic == kCtxMagic, RSTQ_E_INVALID, "invalid context handle");
    RSTQ_REQUIRE(heads >= 1 && head_dim >= 2 && head_dim % 2 == 0 && theta > 0.0 && (posbuf || pos >= 0), RSTQ_E_SHAPE,
                 "heads = %lld, head_dim = %lld (even), theta = %g, pos = %lld", (long long)heads,
                 (long long)head_dim, theta, (long long)pos);
    const int64_t n = heads * head_dim;
    RSTQ_REQUIRE(attn_buf(x, ctx, n * 4) && attn_buf(out, ctx, n * 4) && (!posbuf || attn_buf(posbuf, ctx, 8)),
                 RSTQ_E_INVALID, "invalid, unaligned or too small buffer");
    RSTQ_REQUIRE(x->dev == out->dev && (!posbuf || posbuf->dev == x->dev), RSTQ_E_DEVICE,
                 "buffers live on different devices");
    DeviceState& ds = ctx->devs[x->dev];
    int32_t rc = use_dev(ctx, x->dev);
    if (rc != RSTQ_OK) return rc;
    const int64_t items = heads * (head_dim / 2);
    RSTQ_CUDA(launch_attn(rope_pos_kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, ds,
                          (const float*)x->ptr, (float*)out->ptr, heads, head_dim, log(theta), pos,
                          posbuf ? (const int64_t*)posbuf->ptr : (const int64_t*)nullptr));
    ctx->launches++;
    return RSTQ_OK;
}

int32_t rstq_kv_append(rstq_ctx* ctx, rstq_buf* src, rstq_buf* cache, rstq_buf* posbuf, int64_t kvrow,
                       int64_t pos, int64_t maxpos) {
    RSTQ_REQUIRE(ctx && ctx->magic == kCtxMagic, RSTQ_E_INVALID, "invalid context handle");
    RSTQ_REQUIRE(kvrow >= 1 && maxpos >= 1 && (posbuf || (pos >= 0 && pos < maxpos)), RSTQ_E_SHAPE,
                 "kvrow = %lld, pos = %lld of %lld", (long long)kvrow, (long long)pos, (long long)maxpos);
    RSTQ_REQUIRE(attn_buf(src, ctx, kvrow * 4) && attn_buf(cache, ctx, maxpos * kvrow * 4) &&
                     (!posbuf || attn_buf(posbuf, ctx, 8)),
                 RSTQ_E_INVALID, "invalid, unaligned or too small buffer (the cache holds maxpos rows)");
    RSTQ_REQUIRE(src->dev == cache->dev && (!posbuf || posbuf->dev == src->dev), RSTQ_E_DEVICE,
                 "buffers live on different devices");
    DeviceState& ds = ctx->devs[src->dev];
    int32_t rc = use_dev(ctx, src->dev);
    if (rc != RSTQ_OK) return rc;
    int64_t ctas = (kvrow + 255) / 256;
    if (ctas > ds.sm_count * 4) ctas = ds.sm_count * 4;
    RSTQ_CUDA(launch_attn(kv_append_kernel, dim3((unsigned)ctas), dim3(256), 0, ds, (const float*)src->ptr,
                          (float*)cache->ptr, kvrow, pos, posbuf ? (const int64_t*)posbuf->ptr : (const int64_t*)nullptr));
    ctx->launches++;
    return RSTQ_OK;
}

int32_t rstq_rope_append(rstq_ctx* ctx, rstq_buf* q, rstq_buf* k, rstq_buf* v, rstq_buf* kcache,
                         rstq_buf* vcache, rstq_buf* posbuf, int64_t n_q, int64_t n_kv, int64_t head_dim,
                         double theta, int64_t pos, int64_t maxpos) {
    RSTQ_REQUIRE(ctx && ctx->magic == kCtxMagic, RSTQ_E_INVALID, "invalid context handle");
    RSTQ_REQUIRE(n_q >= 1 && n_kv >= 1 && head_dim >= 2 && head_dim % 2 == 0 && theta > 0.0 && maxpos >= 1 &&
                     (posbuf || (pos >= 0 && pos < maxpos)),
                 RSTQ_E_SHAPE, "n_q = %lld, n_kv = %lld, head_dim = %lld (even), pos = %lld of %lld", (long long)n_q,
                 (long long)n_kv, (long long)head_dim, (long long)pos, (long long)maxpos);
    const int64_t kvrow = n_kv * head_dim;
    RSTQ_REQUIRE(attn_buf(q, ctx, n_q * head_dim * 4) && attn_buf(k, ctx, kvrow * 4) && attn_buf(v, ctx, kvrow * 4) &&
                     attn_buf(kcache, ctx, maxpos * kvrow * 4) && attn_buf(vcache, ctx, maxpos * kvrow * 4) &&
                     (!posbuf || attn_buf(posbuf, ctx, 8)),
                 RSTQ_E_INVALID, "invalid, unaligned or too small buffer (the caches hold maxpos rows)");
    RSTQ_REQUIRE(q->dev == k->dev && q->dev == v->dev && q->dev == kcache->dev && q->dev == vcache->dev &&
                     (!posbuf || posbuf->dev == q->dev),
                 RSTQ_E_DEVICE, "buffers live on different devices");
    DeviceState& ds = ctx->devs[q->dev];
    int32_t rc = use_dev(ctx, q->dev);
    if (rc != RSTQ_OK) return rc;
    const int64_t items = (n_q + 2 * n_kv) * (head_dim / 2);
    RSTQ_CUDA(launch_attn(rope_append_kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, ds, (float*)q->ptr,
                          (float*)k->ptr, (const float*)v->ptr, (float*)kcache->ptr, (float*)vcache->ptr, n_q, n_kv,
                          head_dim, log(theta), pos, posbuf ? (const int64_t*)posbuf->ptr : (const int64_t*)nullptr));
    ctx->launches++;
    return RSTQ_OK;
}

static int32_t attention_impl(rstq_ctx* ctx, rstq_buf* q, rstq_buf* k, rstq_buf* v, rstq_buf* out,
                              int64_t cache_len, rstq_buf* clenbuf, int64_t n_q, int64_t group, int64_t n_kv,
                              int64_t head_dim, int64_t maxpos, double scale, rstq_buf* xq, rstq_buf* xs,
                              rstq_buf* xsum) {
    RSTQ_REQUIRE(ctx && ctx->magic == kCtxMagic, RSTQ_E_INVALID, "invalid context handle");
    RSTQ_REQUIRE(n_q >= 1 && group >= 1 && n_kv >= 1 && n_q == group * n_kv, RSTQ_E_SHAPE,
                 "n_q = %lld must be group (%lld) x n_kv (%lld)", (long long)n_q, (long long)group, (long long)n_kv);
    RSTQ_REQUIRE(head_dim >= 4 && head_dim % 4 == 0 && head_dim <= 128 * kAttnVec, RSTQ_E_SHAPE,
                 "head_dim = %lld (a multiple of 4, at most %d)", (long long)head_dim, 128 * kAttnVec);
    RSTQ_REQUIRE(maxpos >= 1 && (clenbuf || (cache_len >= 1 && cache_len <= maxpos)), RSTQ_E_SHAPE,
                 "cache_len = %lld of maxpos = %lld", (long long)cache_len, (long long)maxpos);
    const int64_t kvbytes = maxpos * n_kv * head_dim * 4;
    RSTQ_REQUIRE(attn_buf(q, ctx, n_q * head_dim * 4) && attn_buf(out, ctx, n_q * head_dim * 4) &&
                     attn_buf(k, ctx, kvbytes) && attn_buf(v, ctx, kvbytes) && (!clenbuf || attn_buf(clenbuf, ctx, 8)),
                 RSTQ_E_INVALID, "invalid, unaligned or too small buffer (the caches hold maxpos rows)");
    RSTQ_REQUIRE(q->dev == k->dev && q->dev == v->dev && q->dev == out->dev && (!clenbuf || clenbuf->dev == q->dev),
                 RSTQ_E_DEVICE, "buffers live on different devices");
    DeviceState& ds = ctx->devs[q->dev];
    int32_t rc = use_dev(ctx, q->dev);
    if (rc != RSTQ_OK) return rc;
    const bool fast = head_dim == 64 || head_dim == 128;
    // query heads per CTA of the stream kernel: four (eight, in two passes over a tile, were slower)
    const int64_t gmax = fast ? kStreamHeads : kAttnGroup;
    const int64_t gs = group < gmax ? group : gmax, gz = (group + gs - 1) / gs;
    const int64_t per = !fast ? kAttnGroup : (group >= 2 ? 2 : 1);      // (the limit of the entry point, not of the grid)
    RSTQ_REQUIRE(n_kv * ((group + per - 1) / per) <= kAttnCounters, RSTQ_E_LIMIT, "n_kv x ceil(group / %d) = %lld exceeds %d", (int)per,
                 (long long)(n_kv * ((group + per - 1) / per)), kAttnCounters);
    // slices of the cache: one wave of CTAs, at least 64 positions each; sized from the
    // capacity when the length lives on the device, so that one captured launch serves every length
    const int64_t span = clenbuf ? maxpos : cache_len;
    int64_t S = (fast ? 1 : 2) * (int64_t)ds.sm_count / (n_kv * gz);
    if (S > (span + 63) / 64) S = (span + 63) / 64;
    const int64_t row = head_dim + 4;
    if (!fast && S > 8 * row - 1) S = 8 * row - 1;   // the general kernel's merge keeps S weights + 1 sum per head in the states' place
    if (fast && S > kMaxSlices) S = kMaxSlices;
    if (S > 512) S = 512;
    if (S < 1) S = 1;
    // Up to eight slices may be one cluster and meet in distributed shared memory, which saves 0.3 - 1.5 us of the tail (against
    // slots: 32 / 32 heads x 1000 10.3 -> 9.7 us, 32 / 8 x 200 6.8 -> 5.3, four 7B layers 204.5 -> 195.6), as long as all clusters
    // are resident together: 16 of eight took two waves, 32 / 16 x 2000 16.1 us against 10.4.  Fewer, longer slices are taken
    // for it where each grows by less than attn_cluster_extra (slots -> cluster: 32 / 16 x 500, nine -> six, 7.6 -> 6.3; x 1200 9.8 -> 8.4, x
    // 1700 9.7 / 10.1; 2 / 2 x 1600 of 64 elements 7.4 -> 6.1; 32 / 8 x 1150, four heads, 7.7 / 8.4, x 1250 8.2 / 8.5).
    // With more KV heads than half the SMs there is one block of 16 warps for each, and where these leave a third of the SMs
    // without one, or two fifths in several rounds, blocks of four warps share the work more evenly: four per SM, as many
    // slices (a cluster) as all fit at once, with a little to spare (112 clusters of five, of 112 that fit, took two rounds).
    // Their merge takes longer, so a short cache of one round stays with 16 warps, and one of 64 positions for four query
    // heads; else in several rounds a short cache is mostly the start and end of each, which four blocks per SM overlap.
    // us, 16 warps -> four: 80 / 80 heads x 250 7.2 / 8.0, x 500 10.7 -> 9.6, x 2000 33.9 -> 28.4, 90 x 1000 19.3 -> 17.5 (112 x 2000: 38.9 /
    // 39.6), 160 x 100 8.6 -> 8.1, x 2000 62.5 -> 52.9, 256 x 500 25.0 -> 23.2 (x 2000: 78.3 / 84.5), 640 / 160 x 64 8.8 / 10.5.
    const int64_t heads = n_kv * gz, rounds = (heads + ds.sm_count - 1) / ds.sm_count;
    const bool narrow = fast && (rounds == 1 ? 2 * heads > ds.sm_count && 3 * heads <= 2 * ds.sm_count && span >= 384
                                             : (gs < kStreamHeads || span > 64) && (5 * heads < 3 * rounds * ds.sm_count || span < 768));
    bool clustered = narrow;
    if (narrow) {
        S = std::max<int64_t>(1, std::min({4 * ds.sm_count / heads, (span + 63) / 64, (int64_t)kClusterMax}));
        while (S > 1 && 32 * heads > 31 * ds.attn_narrow_clusters[S]) --S;
    }
    for (int64_t c = fast ? (S < kClusterMax ? S : kClusterMax) : 0; c > 1 && !clustered; --c) {
        if (n_kv * gz > ds.attn_clusters[c]) continue;
        if ((span / c - span / S) * head_dim * 8 > attn_cluster_extra(gs)) break;
        S = c;
        clustered = true;
    }
    if (xq) {
        RSTQ_REQUIRE(fast, RSTQ_E_SHAPE, "the quantized output needs head_dim 64 or 128, got %lld", (long long)head_dim);
        const int64_t n = n_q * head_dim;
        RSTQ_REQUIRE(attn_buf(xq, ctx, n) && attn_buf(xs, ctx, n / 32 * 4) && (!xsum || attn_buf(xsum, ctx, n / 32 * 4)),
                     RSTQ_E_INVALID, "invalid, unaligned or too small quantizer buffer");
        RSTQ_REQUIRE(xq->dev == q->dev && xs->dev == q->dev && (!xsum || xsum->dev == q->dev), RSTQ_E_DEVICE,
                     "buffers live on different devices");
    }
    AttnParams p;
    p.q = (const float*)q->ptr;
    p.k = (const float*)k->ptr;
    p.v = (const float*)v->ptr;
    p.out = (float*)out->ptr;
    p.counters = fast ? nullptr : (int*)ds.attn_scratch;
    p.part = fast ? (float*)ds.attn_slots : (float*)((char*)ds.attn_scratch + kAttnCounters * 4);
    p.clenbuf = clenbuf ? (const int64_t*)clenbuf->ptr : nullptr;
    p.cache_len = cache_len;
    p.n_q = (int)n_q;
    p.group = (int)group;
    p.n_kv = (int)n_kv;
    p.head_dim = (int)head_dim;
    p.S = (int)S;
    p.scale = (float)scale;
    p.gs = (int)gs;
    p.maxpos = maxpos;
    p.status = ds.status;
    p.xq = xq ? (int8_t*)xq->ptr : nullptr;
    p.xs = xq ? (float*)xs->ptr : nullptr;
    p.xsum = xq && xsum ? (int32_t*)xsum->ptr : nullptr;
    const dim3 grid((unsigned)n_kv, (unsigned)S, (unsigned)gz);
    if (fast) {
        auto launch = [&](auto kernel, int warps) {
            return launch_attn_cluster(kernel, grid, dim3((unsigned)warps * 32), (size_t)attn_smem((int)head_dim, warps), ds,
                                       clustered ? (unsigned)S : 1u, p);
        };
#define RSTQ_ATTN(HD, CL, WARPS)                                                  \
    (gs == 1   ? launch(gqa_decode_stream_kernel<HD, 1, CL, WARPS>, WARPS)       \
     : gs == 2 ? launch(gqa_decode_stream_kernel<HD, 2, CL, WARPS>, WARPS)       \
               : launch(gqa_decode_stream_kernel<HD, 4, CL, WARPS>, WARPS))
        if (narrow) RSTQ_CUDA(head_dim == 64 ? RSTQ_ATTN(64, true, kNarrowWarps) : RSTQ_ATTN(128, true, kNarrowWarps));
        else if (clustered) RSTQ_CUDA(head_dim == 64 ? RSTQ_ATTN(64, true, kStreamWarps) : RSTQ_ATTN(128, true, kStreamWarps));
        else RSTQ_CUDA(head_dim == 64 ? RSTQ_ATTN(64, false, kStreamWarps) : RSTQ_ATTN(128, false, kStreamWarps));
#undef RSTQ_ATTN
    } else {
        const size_t smem = (size_t)(kAttnWarps * gs * row * 4);
        if (smem > 48 * 1024)
            RSTQ_CUDA(cudaFuncSetAttribute(gqa_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        RSTQ_CUDA(launch_attn(gqa_decode_kernel, grid, dim3(kAttnWarps * 32), smem, ds, p));
    }
    ctx->launches++;
    return RSTQ_OK;
}

int32_t rstq_gqa_decode_attention(rstq_ctx* ctx, rstq_buf* q, rstq_buf* k, rstq_buf* v, rstq_buf* out,
                                  rstq_buf* clenbuf, int64_t cache_len, int64_t n_q, int64_t group,
                                  int64_t n_kv, int64_t head_dim, int64_t maxpos, double scale) {
    return attention_impl(ctx, q, k, v, out, cache_len, clenbuf, n_q, group, n_kv, head_dim, maxpos, scale, nullptr,
                          nullptr, nullptr);
}

int32_t rstq_gqa_decode_attention_quant_act(rstq_ctx* ctx, rstq_buf* q, rstq_buf* k, rstq_buf* v, rstq_buf* out,
                                            rstq_buf* xq, rstq_buf* xs, rstq_buf* xsum, rstq_buf* clenbuf,
                                            int64_t cache_len, int64_t n_q, int64_t group, int64_t n_kv,
                                            int64_t head_dim, int64_t maxpos, double scale) {
    RSTQ_REQUIRE(xq && xs, RSTQ_E_INVALID, "null quantizer buffer");
    return attention_impl(ctx, q, k, v, out, cache_len, clenbuf, n_q, group, n_kv, head_dim, maxpos, scale, xq, xs, xsum);
}

}  // extern "C"
