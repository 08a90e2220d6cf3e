// Prompt-pass attention on the 5th-generation tensor cores: exec_grouped_query_attention
// (crates/yscv-onnx/src/runner/linear.rs:552-646) over the KV cache for many query positions per
// sequence, fp32 results from fp16 tensor-core products.
//
// Precision. An fp32 operand x, scaled by a power of two so that the largest magnitude of its block (a
// 64-key tile of one KV head, or one query row) lies in [2^13, 2^14), is split into hi = fp16(x) and
// lo = fp16(x - hi): 22 significant bits, and an absolute error below 2^-39 of the block's maximum for
// its small elements. A product is three MMAs, hi hi + hi lo + lo hi (the dropped lo lo term is 2^-22 of
// the product), with fp32 accumulators. The tensor core adds into its accumulator by truncation, so no
// accumulator outlives one 64-key tile: scores are complete after D products, and every tile's weighted
// value sum is drained into fp32 registers with rounded adds. Tiles that two terms cannot hold are marked when
// they are split, and a CTA that meets one works in fp32 FMAs (at_fp32_tile).
//
// Two kernels. kv_split_kernel converts the cached keys and values of a layer once (they would otherwise
// be converted by every query tile: 128 times for a 2048-token prompt) into the shared-memory images
// the second kernel wants, keys [64][D] and values transposed [D][64], both K-major with the 128-byte
// swizzle, hi and lo, so that a stage is two plain bulk copies. gqa_prefill_tc_kernel takes a tile of 128
// (position, query head) pairs of one KV head per CTA:
//   warp 0      producer: bulk copies of the key and value images, STAGES deep
//   warp 1      TMEM allocation; MMAs: S = Q K^T (M 128, N 64), O_tile = P V (A = P from TMEM, N = D)
//   warps 4-7   softmax, a thread per pair: S from TMEM, running maximum and exp-sum, the weights (times
//               2^10, so that small ones stay clear of fp16 subnormals) split and stored to TMEM as the
//               A operand of the second product; the rescale factor goes through shared memory
//   warps 8-11  drain, a thread per pair: o = o * alpha + O_tile * 2^-s
// S, P and O_tile are double-buffered in TMEM, so the products of tile i + 1 run under the softmax of
// tile i. All warps convert the query tile first. CTAs with the longest key ranges start first.
//
// Bound: the tensor pipe. 3 x (64 D + 64 D) x 128 MACs per tile: 1536 cycles at the nominal rate for
// D = 128, against about 700 issue slots of the softmax warps and 400 of the drain warps per scheduler.
// The fp32 FMA kernel this replaces needed 2.97 ms per layer for a 2048-token prompt at the Llama-3-70B
// head shape (64 / 8 heads of 128).
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.cuh"
#include "tma.cuh"

namespace yscv {

constexpr int AT_ROWS = 128;      // (position, head) pairs per CTA
constexpr int AT_KT = 64;         // keys per tile
constexpr int AT_THREADS = 384;

__device__ __forceinline__ void at_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void at_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// K-major operand with the 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t at_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)2 << 61;
}
__device__ __forceinline__ void at_mma_ss(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void at_mma_ts(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void at_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void at_ld32(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
          "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void at_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void at_st32(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};\n" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
        "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ float at_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// Power of two that brings a block maximum into [2^13, 2^14) (1 for zero, subnormal and non-finite
// maxima), and its inverse.
__device__ __forceinline__ void at_scale(float amax, float &up, float &down) {
    const uint32_t e = (__float_as_uint(amax) >> 23) & 255u;
    uint32_t u = 267u - e;                      // biased exponent of 2^(13 - (e - 127))
    u = (e == 0u || e == 255u) ? 127u : (u > 253u ? 253u : u);
    up = __uint_as_float(u << 23);
    down = __uint_as_float((254u - u) << 23);   // (u >= 13, so the inverse stays normal)
}
// two scaled values -> fp16 pair of the leading terms, fp16 pair of the remainders
__device__ __forceinline__ void at_split(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

// ---- keys and values of one layer -> fp16 hi / lo images ---------------------------------------
// Block (tile of 64 keys, KV head, sequence). Image of a tile: keys {hi, lo} x [D / 64][64 rows][128 B],
// values {hi, lo} x [D rows][128 B]; rows past the last key in use are zeros. inv_scales: the inverse scales
// {keys, values} of the tile; 0 for the keys says that the tile cannot be had in two terms:
//   - a row with an infinity or NaN (it would reach, as 0 x NaN, positions that do not attend to its key),
//   - a row whose largest magnitude is below 2^-12 of the tile's (its absolute error, 2^-39 of the tile's
//     maximum, would come near 2^-24 of the row's own, which is what an fp32 operand has),
//   - a tile maximum outside [2^-50, 2^50] (the product of the inverse scales would leave the fp32 range).
constexpr float AT_ROW_RANGE = 1.0f / 4096.0f, AT_LEAST = 8.8817842e-16f, AT_MOST = 1.1258999e15f;
__device__ __forceinline__ bool at_in_range(float amax) { return (amax == 0.0f) | ((amax >= AT_LEAST) & (amax <= AT_MOST)); }
template <int D> struct ATImage {
    static constexpr int K_TERM = AT_KT * D * 2;          // one term of the keys, in bytes
    static constexpr int V_TERM = AT_KT * D * 2;
    static constexpr int K_BYTES = 2 * K_TERM, V_BYTES = 2 * V_TERM;
    static constexpr int BYTES = K_BYTES + V_BYTES;
};

// What both kernels know of a call. A (sequence, KV head) pair is b * n_kv + head.
template <typename KV> struct ATCall {
    const float *q;
    int q_stride, q_vec, seq_q, n_q, n_kv, max_seq, causal;
    const KV *kc, *vc;
    const float *kscale, *vscale;
    const int32_t *pos;
    float *out;
    int QB;                       // query positions per CTA
    int n_tiles;                  // key tiles of max_seq
    int pair0, pairs;             // pairs of this launch
    unsigned char *images;        // [pairs][n_tiles]; null: no scratch, every CTA takes the fp32 path
    float *inv_scales;            // [pairs][n_tiles][2]
};

// Block (pair, tile), then every gridDim.y-th tile of the pair up to the last key in use
template <typename KV, int D>
__global__ void __launch_bounds__(256, 2) kv_split_kernel(const __grid_constant__ ATCall<KV> a) {
    pdl_wait();
    pdl_trigger();
    constexpr bool I8 = sizeof(KV) == 1;
    constexpr int CPR = D / 8;                    // groups of 8 elements per row
    constexpr int ITEMS = AT_KT * CPR / 256;      // such groups per thread
    __shared__ float vt[AT_KT][D + 1];
    __shared__ float red[2][8];
    const int b = (a.pair0 + blockIdx.x) / a.n_kv, h = (a.pair0 + blockIdx.x) % a.n_kv, tid = threadIdx.x;
    const int limit = min(*a.pos + a.seq_q, a.max_seq);
    const size_t row_elems = (size_t)a.n_kv * D;
    for (int tile = blockIdx.y; tile * AT_KT < limit; tile += gridDim.y) {
        const int k0 = tile * AT_KT;
        const size_t row0 = (size_t)b * a.max_seq + k0;
        const KV *kb = a.kc + row0 * row_elems + (size_t)h * D, *vb = a.vc + row0 * row_elems + (size_t)h * D;
        float k[ITEMS][8], v[ITEMS][8];
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const int idx = tid + it * 256, r = idx / CPR, c = (idx % CPR) * 8;
            const bool live = k0 + r < limit;
            if constexpr (I8) {
                const float rk = live ? a.kscale[row0 + r] : 0.0f, rv = live ? a.vscale[row0 + r] : 0.0f;
                uint2 kw = make_uint2(0u, 0u), vw = make_uint2(0u, 0u);
                if (live) {
                    kw = *reinterpret_cast<const uint2 *>(kb + r * row_elems + c);
                    vw = *reinterpret_cast<const uint2 *>(vb + r * row_elems + c);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t wk = j < 4 ? kw.x : kw.y, wv = j < 4 ? vw.x : vw.y;
                    k[it][j] = __fmul_rn((float)(int8_t)(wk >> (8 * (j & 3))), rk);
                    v[it][j] = __fmul_rn((float)(int8_t)(wv >> (8 * (j & 3))), rv);
                }
            } else {
                float4 ka = make_float4(0.f, 0.f, 0.f, 0.f), kd = ka, va = ka, vd = ka;
                if (live) {
                    const float4 *kp = reinterpret_cast<const float4 *>(kb + r * row_elems + c);
                    const float4 *vp = reinterpret_cast<const float4 *>(vb + r * row_elems + c);
                    ka = kp[0]; kd = kp[1]; va = vp[0]; vd = vp[1];
                }
                k[it][0] = ka.x; k[it][1] = ka.y; k[it][2] = ka.z; k[it][3] = ka.w;
                k[it][4] = kd.x; k[it][5] = kd.y; k[it][6] = kd.z; k[it][7] = kd.w;
                v[it][0] = va.x; v[it][1] = va.y; v[it][2] = va.z; v[it][3] = va.w;
                v[it][4] = vd.x; v[it][5] = vd.y; v[it][6] = vd.z; v[it][7] = vd.w;
            }
        }
        float km = 0.0f, vm = 0.0f, krow[ITEMS], vrow[ITEMS];   // of the tile, of this thread's rows (CPR lanes each)
        float nan = 0.0f;                                        // 0 x value, summed: NaN behind an infinity or NaN
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const int idx = tid + it * 256, r = idx / CPR, c = (idx % CPR) * 8;
            krow[it] = vrow[it] = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                krow[it] = fmaxf(krow[it], fabsf(k[it][j]));
                vrow[it] = fmaxf(vrow[it], fabsf(v[it][j]));
                nan = fmaf(k[it][j], 0.0f, fmaf(v[it][j], 0.0f, nan));
                vt[r][c + j] = v[it][j];
            }
#pragma unroll
            for (int o = CPR / 2; o > 0; o >>= 1) {
                krow[it] = fmaxf(krow[it], __shfl_xor_sync(0xffffffffu, krow[it], o));
                vrow[it] = fmaxf(vrow[it], __shfl_xor_sync(0xffffffffu, vrow[it], o));
            }
            km = fmaxf(km, krow[it]);
            vm = fmaxf(vm, vrow[it]);
        }
#pragma unroll
        for (int o = 16; o >= CPR; o >>= 1) {
            km = fmaxf(km, __shfl_xor_sync(0xffffffffu, km, o));
            vm = fmaxf(vm, __shfl_xor_sync(0xffffffffu, vm, o));
        }
        if ((tid & 31) == 0) { red[0][tid >> 5] = km; red[1][tid >> 5] = vm; }
        __syncthreads();
        for (int i = 0; i < 8; ++i) { km = fmaxf(km, red[0][i]); vm = fmaxf(vm, red[1][i]); }
        bool wide = (nan != 0.0f) | !at_in_range(km) | !at_in_range(vm);
#pragma unroll
        for (int it = 0; it < ITEMS; ++it)
            wide |= ((krow[it] > 0.0f) & (krow[it] < km * AT_ROW_RANGE)) | ((vrow[it] > 0.0f) & (vrow[it] < vm * AT_ROW_RANGE));
        wide = __syncthreads_or(wide);
        float kup, kdown, vup, vdown;
        at_scale(km, kup, kdown);
        at_scale(vm, vup, vdown);
        const size_t t_idx = (size_t)blockIdx.x * a.n_tiles + tile;
        unsigned char *img = a.images + t_idx * ATImage<D>::BYTES;
        if (tid == 0) { a.inv_scales[2 * t_idx] = wide ? 0.0f : kdown; a.inv_scales[2 * t_idx + 1] = vdown; }
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const int idx = tid + it * 256, r = idx / CPR, c8 = idx % CPR;
            uint4 hi, lo;
            at_split(k[it][0] * kup, k[it][1] * kup, hi.x, lo.x);
            at_split(k[it][2] * kup, k[it][3] * kup, hi.y, lo.y);
            at_split(k[it][4] * kup, k[it][5] * kup, hi.z, lo.z);
            at_split(k[it][6] * kup, k[it][7] * kup, hi.w, lo.w);
            // 16-byte chunk c of row r sits at chunk c ^ (r & 7) of its 64-element sub-tile
            unsigned char *dst = img + (c8 >> 3) * (AT_KT * 128) + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4 *>(dst) = hi;
            *reinterpret_cast<uint4 *>(dst + ATImage<D>::K_TERM) = lo;
        }
        unsigned char *vimg = img + ATImage<D>::K_BYTES;
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const int idx = tid + it * 256, d = idx % D, g = idx / D;   // element d of keys 8 g .. 8 g + 7
            uint4 hi, lo;
            at_split(vt[8 * g][d] * vup, vt[8 * g + 1][d] * vup, hi.x, lo.x);
            at_split(vt[8 * g + 2][d] * vup, vt[8 * g + 3][d] * vup, hi.y, lo.y);
            at_split(vt[8 * g + 4][d] * vup, vt[8 * g + 5][d] * vup, hi.z, lo.z);
            at_split(vt[8 * g + 6][d] * vup, vt[8 * g + 7][d] * vup, hi.w, lo.w);
            unsigned char *dst = vimg + d * 128 + ((g ^ (d & 7)) << 4);
            *reinterpret_cast<uint4 *>(dst) = hi;
            *reinterpret_cast<uint4 *>(dst + ATImage<D>::V_TERM) = lo;
        }
        __syncthreads();   // the next tile writes vt and red
    }
}

// ---- attention ----------------------------------------------------------------------------------
// What truncation takes from a tile's sums on average (1.2e-7 of the output, 0.5e-7 to 2.5e-7 by head size and data)
// is given back in the two factors that scale them anyway: log2(e) / sqrt(D), a little above its nearest float,
// and 1 + 2^-23. Relative error against float64 without and with, scores of std 0.8, 512 positions: heads of 64
// 2.44e-7 / 2.09e-7, of 128 2.72e-7 / 2.17e-7 (fp32 FMAs: 2.08e-7, 2.80e-7).
template <int D> constexpr float AT_SCORE = D == 64 ? (float)(1.4426950408889634 / 8.0 * (1.0 + 0.8e-7))
                                                    : (float)(1.4426950408889634 / 11.313708498984761 * (1.0 + 1.4e-7));
constexpr float AT_VALUE = 1.0f + 1.1920929e-7f;

template <int D> struct ATGeom {
    static constexpr int STAGES = D == 128 ? 2 : 4;
    static constexpr int Q_TERM = AT_ROWS * D * 2;
    static constexpr int RING = 2 * Q_TERM;
    static constexpr int TAIL = RING + STAGES * ATImage<D>::BYTES;      // floats: qinv[128], l[128], alpha[4][128]
    static constexpr int BARS = TAIL + 6 * 128 * 4;
    static constexpr int SMEM = BARS + 272;
};

// The query tile in fp32 throughout, for what two fp16 terms cannot hold (see kv_split_kernel) and for calls
// without scratch: FMAs over 64-key chunks staged in shared memory, four (position, head) pairs per warp. A key
// that a pair does not attend to is not multiplied at all. 2048 tokens, 64 / 8 heads of 128: 3.5 ms a layer
// against 0.28 on the tensor cores.
template <typename KV, int D>
__device__ __noinline__ void at_fp32_tile(const ATCall<KV> &a, float *sm, int b, int kv_h, int qt, int p0) {
    constexpr bool I8 = sizeof(KV) == 1;
    constexpr int KP = D + 4;   // key row pitch: a lane per key reads its row 16 bytes at a time without bank conflicts
    constexpr int KPAR = 32 / (D / 4), WARPS = AT_THREADS / 32, QH = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *ks = sm, *vs = ks + AT_KT * KP, *sc = vs + AT_KT * D + warp * QH * AT_KT;
    float *qs = vs + AT_KT * D + WARPS * QH * AT_KT + warp * QH * D;
    const int group = a.n_q / a.n_kv;
    const float scale = 1.0f / sqrtf((float)D);
    const int e4 = (lane % (D / 4)) * 4, kpar = lane / (D / 4);
    const size_t row_elems = (size_t)a.n_kv * D, seq_row = (size_t)b * a.max_seq;
    for (int r0 = 0; r0 < group * a.QB; r0 += WARPS * QH) {
        int sq[QH], qh[QH], lim[QH];
        bool live[QH];
        float4 acc[QH];
        float m[QH], l[QH];
        int warp_limit = 0;
#pragma unroll
        for (int j = 0; j < QH; ++j) {
            const int idx = r0 + warp * QH + j;
            sq[j] = qt * a.QB + idx / group;
            qh[j] = kv_h * group + idx % group;
            live[j] = idx < group * a.QB && sq[j] < a.seq_q;
            lim[j] = live[j] ? max(0, min(a.max_seq, p0 + (a.causal ? sq[j] + 1 : a.seq_q))) : 0;
            warp_limit = max(warp_limit, lim[j]);
            acc[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            m[j] = -INFINITY;
            l[j] = 0.0f;
            for (int i = lane; i < D; i += 32)
                qs[j * D + i] = live[j] ? a.q[((size_t)b * a.seq_q + sq[j]) * a.q_stride + (size_t)qh[j] * D + i] : 0.0f;
        }
        const int last = min(a.seq_q, qt * a.QB + (min(r0 + WARPS * QH, group * a.QB) - 1) / group + 1);
        const int block_limit = max(0, min(a.max_seq, p0 + (a.causal ? last : a.seq_q)));
        for (int c0 = 0; c0 < block_limit; c0 += AT_KT) {
            const int rows = min(AT_KT, block_limit - c0);
            __syncthreads();
            for (int idx = threadIdx.x; idx < rows * (D / 4); idx += AT_THREADS) {
                const int r = idx / (D / 4), c4 = (idx % (D / 4)) * 4;
                const size_t off = (seq_row + c0 + r) * row_elems + (size_t)kv_h * D + c4;
                float4 k4, v4;
                if constexpr (I8) {
                    const float rk = a.kscale[seq_row + c0 + r], rv = a.vscale[seq_row + c0 + r];
                    const char4 kw = *reinterpret_cast<const char4 *>(a.kc + off), vw = *reinterpret_cast<const char4 *>(a.vc + off);
                    k4 = make_float4(__fmul_rn((float)kw.x, rk), __fmul_rn((float)kw.y, rk), __fmul_rn((float)kw.z, rk), __fmul_rn((float)kw.w, rk));
                    v4 = make_float4(__fmul_rn((float)vw.x, rv), __fmul_rn((float)vw.y, rv), __fmul_rn((float)vw.z, rv), __fmul_rn((float)vw.w, rv));
                } else {
                    k4 = *reinterpret_cast<const float4 *>(a.kc + off);
                    v4 = *reinterpret_cast<const float4 *>(a.vc + off);
                }
                *reinterpret_cast<float4 *>(ks + r * KP + c4) = k4;
                *reinterpret_cast<float4 *>(vs + r * D + c4) = v4;
            }
            __syncthreads();
            const int nkw = min(rows, warp_limit - c0);   // keys of this chunk that any of the warp's pairs attends to
            if (nkw <= 0) continue;
            // scores: a lane per key (lane and lane + 32), each piece of a query read once for both
            float s[2][QH];
#pragma unroll
            for (int j = 0; j < QH; ++j) s[0][j] = s[1][j] = 0.0f;
            const float4 *kr = reinterpret_cast<const float4 *>(ks + lane * KP);
#pragma unroll 2
            for (int i = 0; i < D / 4; ++i) {
                const float4 k0 = kr[i], k1 = kr[i + 32 * KP / 4];
#pragma unroll
                for (int j = 0; j < QH; ++j) {
                    const float4 x = reinterpret_cast<const float4 *>(qs + j * D)[i];
                    s[0][j] = fmaf(x.w, k0.w, fmaf(x.z, k0.z, fmaf(x.y, k0.y, fmaf(x.x, k0.x, s[0][j]))));
                    s[1][j] = fmaf(x.w, k1.w, fmaf(x.z, k1.z, fmaf(x.y, k1.y, fmaf(x.x, k1.x, s[1][j]))));
                }
            }
#pragma unroll
            for (int j = 0; j < QH; ++j) {
                // (rows past the limit hold stale values)
                const float s0 = lane < lim[j] - c0 ? s[0][j] * scale : -INFINITY, s1 = lane + 32 < lim[j] - c0 ? s[1][j] * scale : -INFINITY;
                float cm = fmaxf(s0, s1);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
                const float m_new = fmaxf(m[j], cm);
                const float alpha = m_new == -INFINITY ? 1.0f : expf(m[j] - m_new);   // 0 for a pair's first chunk
                const float e0 = s0 == -INFINITY ? 0.0f : expf(s0 - m_new), e1 = s1 == -INFINITY ? 0.0f : expf(s1 - m_new);
                sc[j * AT_KT + lane] = e0;
                sc[j * AT_KT + lane + 32] = e1;
                float ps = e0 + e1;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
                l[j] = l[j] * alpha + ps;
                acc[j].x *= alpha; acc[j].y *= alpha; acc[j].z *= alpha; acc[j].w *= alpha;
                m[j] = m_new;
            }
            __syncwarp();
            // weighted values: a lane owns four columns (D = 64: the half warps take alternate keys)
            for (int k = kpar; k < nkw; k += KPAR) {
                const float4 v4 = *reinterpret_cast<const float4 *>(vs + k * D + e4);
#pragma unroll
                for (int j = 0; j < QH; ++j) {
                    if (k < lim[j] - c0) {
                        const float p = sc[j * AT_KT + k];
                        acc[j].x = fmaf(p, v4.x, acc[j].x);
                        acc[j].y = fmaf(p, v4.y, acc[j].y);
                        acc[j].z = fmaf(p, v4.z, acc[j].z);
                        acc[j].w = fmaf(p, v4.w, acc[j].w);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < QH; ++j) {
            if constexpr (KPAR == 2) {
                acc[j].x += __shfl_xor_sync(0xffffffffu, acc[j].x, 16);
                acc[j].y += __shfl_xor_sync(0xffffffffu, acc[j].y, 16);
                acc[j].z += __shfl_xor_sync(0xffffffffu, acc[j].z, 16);
                acc[j].w += __shfl_xor_sync(0xffffffffu, acc[j].w, 16);
            }
            if (live[j] && kpar == 0) {
                const float inv = l[j] == 0.0f ? 0.0f : 1.0f / l[j];
                float *row = a.out + ((size_t)b * a.seq_q + sq[j]) * (size_t)a.n_q * D + (size_t)qh[j] * D;
                *reinterpret_cast<float4 *>(row + e4) = make_float4(acc[j].x * inv, acc[j].y * inv, acc[j].z * inv, acc[j].w * inv);
            }
        }
        __syncthreads();   // the next pairs' queries
    }
}

template <typename KV, int D>
__global__ void __launch_bounds__(AT_THREADS, 1) gqa_prefill_tc_kernel(const __grid_constant__ ATCall<KV> a, int *__restrict__ status) {
    using G = ATGeom<D>;
    const int q_stride = a.q_stride, seq_q = a.seq_q, n_q = a.n_q, n_kv = a.n_kv, max_seq = a.max_seq, QB = a.QB;
    constexpr int STAGES = G::STAGES;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = smem_u32(smem);
    float *qinv_sm = reinterpret_cast<float *>(smem + G::TAIL), *l_sm = qinv_sm + 128, *alpha_sm = l_sm + 128;
    const uint32_t bars = base + G::BARS;
    const uint32_t kfull = bars, kempty = bars + 32, vfull = bars + 64, vempty = bars + 96;           // [STAGES]
    const uint32_t sfull = bars + 128, sfree = bars + 144, pfull = bars + 160, pfree = bars + 176;    // [2]
    const uint32_t ofull = bars + 192, ofree = bars + 208, afull = bars + 224;                        // [2], [2], [4]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + G::BARS + 256);
    const int group = n_q / n_kv;
    const int pair = blockIdx.x % a.pairs, kv_h = (a.pair0 + pair) % n_kv, b = (a.pair0 + pair) / n_kv;
    const int qt = (gridDim.x - 1 - blockIdx.x) / a.pairs;      // the longest key ranges first

    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(kfull + i * 8, 1);
            mbar_init(kempty + i * 8, 1);
            mbar_init(vfull + i * 8, 1);
            mbar_init(vempty + i * 8, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(sfull + i * 8, 1);
            mbar_init(sfree + i * 8, 4);
            mbar_init(pfull + i * 8, 4);
            mbar_init(pfree + i * 8, 1);
            mbar_init(ofull + i * 8, 1);
            mbar_init(ofree + i * 8, 4);
        }
        for (int i = 0; i < 4; ++i) mbar_init(afull + i * 8, 4);
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    pdl_wait();
    pdl_trigger();
    const int p0 = *a.pos;
    auto limit_of = [&](int s) {
        const int l = p0 + (a.causal ? s + 1 : seq_q);
        return l > max_seq ? max_seq : (l < 0 ? 0 : l);
    };
    const int block_limit = limit_of(min(seq_q, (qt + 1) * QB) - 1);   // limits do not decrease with the position
    const int n = (block_limit + AT_KT - 1) / AT_KT;                   // key tiles of this CTA
    const unsigned char *img = a.images + (size_t)pair * a.n_tiles * ATImage<D>::BYTES;
    const float *inv = a.inv_scales + (size_t)pair * a.n_tiles * 2;
    bool wide = a.images == nullptr;                                   // this CTA takes the fp32 path

    // ---- query tile: pair r -> head r % group of the group, position r / group of the tile ----
    {
        constexpr int LPR = D / 8;                // lanes per row (8 elements each)
        constexpr int RPW = 32 / LPR;             // rows per warp and step
        constexpr int STEPS = (AT_ROWS / RPW + 11) / 12;
        const int c8 = lane % LPR;
        float v[STEPS][8];
#pragma unroll
        for (int it = 0; it < STEPS; ++it) {
            const int r = (it * 12 + warp) * RPW + lane / LPR, s = qt * QB + r / group;
            const bool live = r < group * QB && s < seq_q;
#pragma unroll
            for (int j = 0; j < 8; ++j) v[it][j] = 0.0f;
            if (live) {
                const float *src = a.q + ((size_t)b * seq_q + s) * q_stride + (size_t)(kv_h * group + r % group) * D + c8 * 8;
                if (a.q_vec) {
                    const float4 c = __ldg(reinterpret_cast<const float4 *>(src)), d = __ldg(reinterpret_cast<const float4 *>(src) + 1);
                    v[it][0] = c.x; v[it][1] = c.y; v[it][2] = c.z; v[it][3] = c.w;
                    v[it][4] = d.x; v[it][5] = d.y; v[it][6] = d.z; v[it][7] = d.w;
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[it][j] = __ldg(src + j);
                }
            }
        }
        // (here the position, on which n hangs, is there as well: in front of the query loads this took 1 %)
        if (!wide)
            for (int i = tid; i < n; i += AT_THREADS) wide |= inv[2 * i] == 0.0f;
#pragma unroll
        for (int it = 0; it < STEPS; ++it) {
            const int r = (it * 12 + warp) * RPW + lane / LPR;
            float m = 0.0f, nan = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                m = fmaxf(m, fabsf(v[it][j]));
                nan = fmaf(v[it][j], 0.0f, nan);
            }
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (r < AT_ROWS) {
                float up, down;
                at_scale(m, up, down);
                wide |= (nan != 0.0f) | !at_in_range(m);
                if (c8 == 0) qinv_sm[r] = down;
                uint4 hi, lo;
                at_split(v[it][0] * up, v[it][1] * up, hi.x, lo.x);
                at_split(v[it][2] * up, v[it][3] * up, hi.y, lo.y);
                at_split(v[it][4] * up, v[it][5] * up, hi.z, lo.z);
                at_split(v[it][6] * up, v[it][7] * up, hi.w, lo.w);
                unsigned char *dst = smem + (c8 >> 3) * (AT_ROWS * 128) + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
                *reinterpret_cast<uint4 *>(dst) = hi;
                *reinterpret_cast<uint4 *>(dst + G::Q_TERM) = lo;
            }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    at_fence_before();
    wide = __syncthreads_or(wide);
    at_fence_after();
    const uint32_t tmem = *tmem_slot;
    // TMEM columns: scores [2] x 64, weights [2] x {hi 32, lo 32}, value sums [2] x 128
    const uint32_t t_s = tmem, t_p = tmem + 128, t_o = tmem + 256;

    if (wide) {
        at_fp32_tile<KV, D>(a, reinterpret_cast<float *>(smem), b, kv_h, qt, p0);
    } else if (warp == 0) {
        if (lane == 0) {
            uint32_t phase = 0;
            bool alive = true;
            int keys = 0, values = 0;   // tiles whose copies were issued
            for (int i = 0, st = 0; i < n && alive; ++i) {
                const uint32_t dst = base + G::RING + (uint32_t)st * ATImage<D>::BYTES;
                const unsigned char *src = img + (size_t)i * ATImage<D>::BYTES;
                alive = mbar_wait(kempty + st * 8, phase ^ 1u, status);
                if (!alive) break;
                mbar_expect_tx(kfull + st * 8, ATImage<D>::K_BYTES);
                bulk_load(dst, src, ATImage<D>::K_BYTES, kfull + st * 8);
                ++keys;
                alive = mbar_wait(vempty + st * 8, phase ^ 1u, status);
                if (!alive) break;
                mbar_expect_tx(vfull + st * 8, ATImage<D>::V_BYTES);
                bulk_load(dst + ATImage<D>::K_BYTES, src + ATImage<D>::K_BYTES, ATImage<D>::V_BYTES, vfull + st * 8);
                ++values;
                if (++st == STAGES) { st = 0; phase ^= 1u; }
            }
            // a consumer gave up: no copy may be in flight when the CTA leaves (bounded)
            if (!alive) {
                for (int i = max(0, keys - STAGES); i < keys; ++i) mbar_wait(kfull + i % STAGES * 8, (uint32_t)(i / STAGES) & 1u, nullptr);
                for (int i = max(0, values - STAGES); i < values; ++i) mbar_wait(vfull + i % STAGES * 8, (uint32_t)(i / STAGES) & 1u, nullptr);
            }
        }
    } else if (warp == 1) {
        {
            // D fp32, A and B fp16, both K-major, M = 128
            const uint32_t id_s = (1u << 4) | ((uint32_t)(AT_KT >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
            const uint32_t id_o = (1u << 4) | ((uint32_t)(D >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
            bool alive = true;
            auto scores = [&](int i) {
                const int st = i % STAGES, s = i & 1;
                alive = __all_sync(0xffffffffu, mbar_wait(kfull + st * 8, (uint32_t)(i / STAGES) & 1u, status) &&
                                                    mbar_wait(sfree + s * 8, ((uint32_t)(i >> 1) & 1u) ^ 1u, status));
                if (!alive) return;
                at_fence_after();
                const uint32_t ks = base + G::RING + (uint32_t)st * ATImage<D>::BYTES;
                if (elect_one()) {
                    uint32_t acc = 0;
#pragma unroll
                    for (int term = 0; term < 3; ++term) {      // lo hi, hi lo, hi hi
                        const uint32_t qa = base + (term == 0 ? G::Q_TERM : 0), kb = ks + (term == 1 ? ATImage<D>::K_TERM : 0);
#pragma unroll
                        for (int sub = 0; sub < D / 64; ++sub) {
                            const uint64_t da = at_desc(qa + sub * (AT_ROWS * 128)), db = at_desc(kb + sub * (AT_KT * 128));
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {     // K = 16 per instruction: +32 bytes
                                at_mma_ss(t_s + s * 64, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), id_s, acc);
                                acc = 1;
                            }
                        }
                    }
                    at_commit(kempty + st * 8);
                    at_commit(sfull + s * 8);
                }
                __syncwarp();
            };
            auto values = [&](int i) {
                const int st = i % STAGES, s = i & 1;
                const uint32_t par = (uint32_t)(i >> 1) & 1u;
                alive = __all_sync(0xffffffffu, mbar_wait(vfull + st * 8, (uint32_t)(i / STAGES) & 1u, status) &&
                                                    mbar_wait(pfull + s * 8, par, status) &&
                                                    mbar_wait(ofree + s * 8, par ^ 1u, status));
                if (!alive) return;
                at_fence_after();
                const uint32_t vs = base + G::RING + (uint32_t)st * ATImage<D>::BYTES + ATImage<D>::K_BYTES;
                if (elect_one()) {
                    uint32_t acc = 0;
#pragma unroll
                    for (int term = 0; term < 3; ++term) {
                        const uint32_t pa = t_p + s * 64 + (term == 0 ? 32 : 0);
                        const uint64_t db = at_desc(vs + (term == 1 ? ATImage<D>::V_TERM : 0));
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {         // 16 keys: 8 columns of the weights
                            at_mma_ts(t_o + s * 128, pa + kk * 8, db + (uint64_t)(kk * 2), id_o, acc);
                            acc = 1;
                        }
                    }
                    at_commit(vempty + st * 8);
                    at_commit(pfree + s * 8);
                    at_commit(ofull + s * 8);
                }
                __syncwarp();
            };
            for (int i = 0; i < n && alive; ++i) {
                scores(i);
                if (alive && i > 0) values(i - 1);
            }
            if (alive && n > 0) values(n - 1);
        }
    } else if (warp >= 4 && warp < 8) {
        // ---- softmax ----
        const int row = (warp & 3) * 32 + lane;
        const int s_pos = qt * QB + row / group;
        const int lim = (row < group * QB && s_pos < seq_q) ? limit_of(s_pos) : 0;
        const float to_log2 = qinv_sm[row] * AT_SCORE<D>;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        float m = -INFINITY, l = 0.0f;     // running maximum (log2 units), exp-sum (times 2^10)
        bool alive = true;
        float kinv = n > 0 ? inv[0] : 1.0f;
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            const uint32_t par = (uint32_t)(i >> 1) & 1u;
            const float c = to_log2 * kinv;
            if (i + 1 < n) kinv = inv[2 * (i + 1)];
            alive = mbar_wait(sfull + s * 8, par, status);
            if (!alive) break;
            at_fence_after();
            float v[64];
            at_ld32(t_s + lane_off + s * 64, reinterpret_cast<uint32_t *>(v));
            at_ld32(t_s + lane_off + s * 64 + 32, reinterpret_cast<uint32_t *>(v) + 32);
            at_wait_ld();
            at_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(sfree + s * 8);
            const int left = lim - i * AT_KT;      // keys of this tile the pair attends to
            if (__any_sync(0xffffffffu, left < AT_KT)) {
#pragma unroll
                for (int j = 0; j < 64; ++j)
                    if (j >= left) v[j] = -INFINITY;
            }
            float mx[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
            for (int j = 4; j < 64; ++j) mx[j & 3] = fmaxf(mx[j & 3], v[j]);
            const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c);
            // nothing to attend to yet: m_new stays -inf, every weight is 0
            const float alpha = m_new == -INFINITY ? 1.0f : at_exp2(m - m_new);
            const float off = m_new == -INFINITY ? 0.0f : 10.0f - m_new;
            float ps[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t hi[32], lo[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float a = at_exp2(fmaf(v[2 * j], c, off)), d = at_exp2(fmaf(v[2 * j + 1], c, off));
                ps[(2 * j) & 3] += a;
                ps[(2 * j + 1) & 3] += d;
                at_split(a, d, hi[j], lo[j]);
            }
            l = fmaf(l, alpha, (ps[0] + ps[1]) + (ps[2] + ps[3]));
            m = m_new;
            alive = mbar_wait(pfree + s * 8, par ^ 1u, status);
            if (!alive) break;
            at_fence_after();
            at_st32(t_p + lane_off + s * 64, hi);
            at_st32(t_p + lane_off + s * 64 + 32, lo);
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            // slot i & 3 was read by the drain of tile i - 4, which the products of tile i - 2 waited for
            alpha_sm[(i & 3) * 128 + row] = alpha;
            if (i == n - 1) l_sm[row] = l;
            at_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(afull + (i & 3) * 8);
                mbar_arrive(pfull + s * 8);
            }
        }
    } else if (warp >= 8) {
        // ---- drain ----
        const int row = (warp & 3) * 32 + lane;
        const int s_pos = qt * QB + row / group;
        const bool live = row < group * QB && s_pos < seq_q;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        float o[D];
#pragma unroll
        for (int j = 0; j < D; ++j) o[j] = 0.0f;
        bool alive = true;
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            const float vinv = inv[2 * i + 1] * AT_VALUE;
            alive = mbar_wait(afull + (i & 3) * 8, (uint32_t)(i >> 2) & 1u, status);
            if (!alive) break;
            const float alpha = alpha_sm[(i & 3) * 128 + row];
            alive = mbar_wait(ofull + s * 8, (uint32_t)(i >> 1) & 1u, status);
            if (!alive) break;
            at_fence_after();
#pragma unroll
            for (int j0 = 0; j0 < D; j0 += 32) {
                float t[32];
                at_ld32(t_o + lane_off + s * 128 + j0, reinterpret_cast<uint32_t *>(t));
                at_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; ++j) o[j0 + j] = fmaf(o[j0 + j], alpha, t[j] * vinv);
            }
            at_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ofree + s * 8);
        }
        if (live && alive) {
            const float l = n > 0 ? l_sm[row] : 0.0f;
            const float f = l > 0.0f ? 1.0f / l : 0.0f;
            float4 *dst = reinterpret_cast<float4 *>(a.out + ((size_t)b * seq_q + s_pos) * (size_t)n_q * D + (size_t)(kv_h * group + row % group) * D);
#pragma unroll
            for (int j = 0; j < D / 4; ++j) dst[j] = make_float4(o[4 * j] * f, o[4 * j + 1] * f, o[4 * j + 2] * f, o[4 * j + 3] * f);
        }
    }
    at_fence_before();
    __syncthreads();
    if (warp == 1) {
        at_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

template <typename KV, int D> static int prefill_tc_launch(yscv_cuda_ctx *ctx, size_t batch, ATCall<KV> a) {
    using G = ATGeom<D>;
    a.n_tiles = (a.max_seq + AT_KT - 1) / AT_KT;
    a.QB = AT_ROWS / (a.n_q / a.n_kv);
    // The images of as many (sequence, KV head) pairs at a time as fit 256 MB, but of a whole sequence up to
    // 1.25 GB where that much is free: one head after another takes 16 positions on an empty cache of 131072 x 8 x
    // 128 from 28 to 117 us.
    const size_t per_pair = (size_t)a.n_tiles * (ATImage<D>::BYTES + 2 * sizeof(float)), pairs = batch * a.n_kv;
    const size_t fit = (256u << 20) / per_pair > 1 ? (256u << 20) / per_pair : 1, all = (1280u << 20) / per_pair;
    size_t group = fit < (size_t)a.n_kv && all >= (size_t)a.n_kv ? a.n_kv : fit;
    if (group > pairs) group = pairs;
    bool split = ctx->scratch_attn.try_reserve(group * per_pair, ctx->stream);
    if (!split && fit < group) split = ctx->scratch_attn.try_reserve((group = fit) * per_pair, ctx->stream);
    if (split) {
        a.images = reinterpret_cast<unsigned char *>(ctx->scratch_attn.ptr);
        a.inv_scales = reinterpret_cast<float *>(a.images + group * a.n_tiles * ATImage<D>::BYTES);
    } else {
        group = pairs;
    }
    auto kern = gqa_prefill_tc_kernel<KV, D>;
    const int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kern), ctx->device, 227 * 1024);
    if (rc) return rc;
    const size_t q_tiles = ((size_t)a.seq_q + a.QB - 1) / a.QB;
    for (size_t p0 = 0; p0 < pairs; p0 += group) {
        a.pair0 = (int)p0;
        a.pairs = (int)(pairs - p0 < group ? pairs - p0 : group);
        if (split) {
            // blocks for two or three rounds of the SMs: a cache is mostly longer than the keys in use
            const int rounds = 16 * ctx->sm_count / a.pairs + 1;
            YSCV_CUDA_TRY(launch_pdl(kv_split_kernel<KV, D>, dim3((unsigned)a.pairs, (unsigned)(a.n_tiles < rounds ? a.n_tiles : rounds)),
                                     dim3(256), 0, ctx->stream, a));
            ctx->launches++;
        }
        YSCV_CUDA_TRY(launch_pdl(kern, dim3((unsigned)(a.pairs * q_tiles)), dim3(AT_THREADS), (size_t)G::SMEM, ctx->stream, a, ctx->d_status));
        ctx->launches++;
    }
    YSCV_CUDA_TRY(cudaGetLastError());
    return YSCV_CUDA_OK;
}

template <typename KV>
int gqa_prefill_tc(yscv_cuda_ctx *ctx, const float *q, size_t q_stride, size_t batch, size_t seq_q, size_t n_q, size_t n_kv,
                   size_t d_head, const KV *kc, const KV *vc, const float *kscale, const float *vscale, size_t max_seq,
                   const int32_t *pos, int causal, float *out) {
    ATCall<KV> a = {};
    a.q = q;
    a.q_stride = (int)q_stride;
    a.q_vec = (reinterpret_cast<uintptr_t>(q) & 15) == 0 && q_stride % 4 == 0;
    a.seq_q = (int)seq_q;
    a.n_q = (int)n_q;
    a.n_kv = (int)n_kv;
    a.max_seq = (int)max_seq;
    a.causal = causal;
    a.kc = kc;
    a.vc = vc;
    a.kscale = kscale;
    a.vscale = vscale;
    a.pos = pos;
    a.out = out;
    return d_head == 64 ? prefill_tc_launch<KV, 64>(ctx, batch, a) : prefill_tc_launch<KV, 128>(ctx, batch, a);
}
template int gqa_prefill_tc<float>(yscv_cuda_ctx *, const float *, size_t, size_t, size_t, size_t, size_t, size_t, const float *,
                                   const float *, const float *, const float *, size_t, const int32_t *, int, float *);
template int gqa_prefill_tc<int8_t>(yscv_cuda_ctx *, const float *, size_t, size_t, size_t, size_t, size_t, size_t, const int8_t *,
                                    const int8_t *, const float *, const float *, size_t, const int32_t *, int, float *);

}  // namespace yscv
