// The fp32 operators that sit between the quantized linears of a Llama-shape
// decoder step: embedding gather, RMSNorm (with the residual add fused in front),
// rotate-half RoPE fused with the KV-cache append, GQA attention over the cache,
// SwiGLU, the fp32 LM-head matmul and the greedy argmax.
//
// Semantics follow the reference's CPU operators
//   RMSNorm   crates/yscv-kernels/src/ops/norm.rs:1497-1518
//   RoPE      crates/yscv-kernels/src/ops/rope.rs:24-117 (rotate-half, pairs (i, i+d/2))
//   GQA       crates/yscv-onnx/src/runner/linear.rs:552-646 (kv head = q head / group,
//             max-subtracted softmax; causality is added here because the exported
//             graphs the reference runs carry it in their mask)
//   SiLU      crates/yscv-kernels/src/ops/simd/activation.rs:1000-1005
//   embedding crates/yscv-kernels/src/ops/embedding.rs:12
//   argmax    apps/llm-bench/src/main.rs:538-543 (LAST index among equal maxima)
//   KV cache  crates/yscv-onnx/src/runner/kv_cache.rs:118-254 (f32 storage)
// All of them are bandwidth-trivial next to the weight streams; they exist so that a
// whole decode step stays on the device and can be replayed as one CUDA graph: the
// sequence position and the token ids are read from device memory, never passed as
// kernel arguments.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace yscv {

__device__ __forceinline__ float block_sum(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[w] = v;
    __syncthreads();
    float t = 0.0f;
    for (int i = 0; i < nw; ++i) t += red[i];
    return t;
}

__device__ __forceinline__ float block_max(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[w] = v;
    __syncthreads();
    float t = -INFINITY;
    for (int i = 0; i < nw; ++i) t = fmaxf(t, red[i]);
    return t;
}

__global__ void embedding_kernel(const float *__restrict__ w, const int32_t *__restrict__ tokens,
                                 float *__restrict__ out, int vocab, int dim) {
    pdl_wait();
    pdl_trigger();
    const int row = blockIdx.x;
    int tok = tokens[row];
    tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
    const float4 *src = reinterpret_cast<const float4 *>(w + (size_t)tok * dim);
    float4 *dst = reinterpret_cast<float4 *>(out + (size_t)row * dim);
    for (int i = threadIdx.x; i < dim / 4; i += blockDim.x) dst[i] = src[i];
}

// Eight consecutive values that are the sum of `parts` arrays `pitch` floats apart, added in that order
__device__ __forceinline__ void load8(const float *p, int parts, size_t pitch, float (&v)[8]) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(p)), b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
#pragma unroll 4
    for (int s = 1; s < parts; ++s) {
        const float4 *q = reinterpret_cast<const float4 *>(p + s * pitch);
        const float4 c = __ldg(q), d = __ldg(q + 1);
        v[0] += c.x; v[1] += c.y; v[2] += c.z; v[3] += c.w;
        v[4] += d.x; v[5] += d.y; v[6] += d.z; v[7] += d.w;
    }
}

// Position of element e of a group of 8 in that order
__device__ __forceinline__ int gemm_order_pos(int e) { return ((e & 3) << 1) | (e >> 2); }

// x_out = x + delta (delta may be null), the row normalised, (x_out / sqrt(mean(x_out^2) + eps)) * gamma, as fp32 or as the
// bf16 activations of the matmul behind it. Input row of block b: row0 + b * row_step.
//
// Latency-bound for a few rows (a block per row), bandwidth-bound for many. A thread keeps its values in registers between
// the sum of squares and the scaling: one round trip with every load in flight, 128-bit accesses, eight consecutive values
// per lane where the form wants them, else four, so that an access of a warp is whole lines. The sum of squares goes through
// shared memory so that its order is that of the scalar kernel below (thread t: elements t, t + T, ...): the same result for every
// form and alignment. T = 256 up to 2048 values, else 1024 (hidden <= 8 T).
// FEW (up to two rows per SM, NORM_FEW): gamma is fetched before the reduction, a thread takes eight values. More: what counts
// is rows per SM, so gamma comes late (28 to 32 registers instead of 40, six and more blocks of 256) and blocks of 512 take 16 values
// per thread, two of them per SM in different phases. us, fp32 to fp32 / to bf16, warm caches: 1 x 2048 1.5 / 1.6, 1 x 8192 3.1 / 3.5,
// 1024 x 2048 4.6 / 5.5 (with FEW 4.6 / 5.3; 512 x 2048 3.0 / 3.4, FEW 3.1 / 4.4), 300 x 4096 5.2 / 5.5 (FEW 5.9 / 6.3), 128 x 4096 2.7 / 2.7 (FEW 2.7 /
// 2.8), 128 x 8192 from HBM 5.8 / 4.9 (FEW 5.1 / 4.5), 2048 x 8192 42.7 / 41.1 (4.9 TB/s of fp32 to bf16; FEW 49.9 / 46.9). The scalar
// kernel: 2.0, 3.7, 5.0, 8.2, 3.2, 5.9, 65. With a sum over parts left in for one part (72 registers) and blocks of 128 and 256
// for more than 512 rows, 40 registers and spills, this took 10.0 / 8.9 at 1024 x 2048 and 20.5 / 17.5 at 513 x 8192 (now 9.5 / 10.9).
constexpr size_t NORM_FEW = 2;
template <bool BF16, int T, bool FEW>
__global__ void __launch_bounds__(FEW || T == 256 ? T : T / 2, FEW ? 1 : T == 256 ? 6 : 2)
norm_rows_kernel(const float *x, const float *delta, const float *__restrict__ gamma, float eps, int hidden, size_t row0, size_t row_step,
                 float *x_out, ActOut o) {
    pdl_wait();
    pdl_trigger();
    constexpr int P = FEW || T == 256 ? 1 : 2, TH = T / P;                 // P eights of values per thread
    constexpr int W = BF16 ? 8 : 4, N = P * 8 / W, Q = W / 4;   // N accesses of W values
    __shared__ float red[32];
    __shared__ __align__(16) float sm[8 * T];
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const size_t base = (row0 + row * row_step) * hidden;
    float4 v[N * Q];
#pragma unroll
    for (int p = 0; p < N; ++p) {
        const int i = (tid + p * TH) * W;
        if (i < hidden) {   // (x not through the read-only path: x_out may be x)
#pragma unroll
            for (int h = 0; h < Q; ++h) v[p * Q + h] = *reinterpret_cast<const float4 *>(x + base + i + 4 * h);
        }
    }
    if (delta) {
#pragma unroll
        for (int p = 0; p < N; ++p) {
            const int i = (tid + p * TH) * W;
            if (i < hidden) {
#pragma unroll
                for (int h = 0; h < Q; ++h) {
                    const float4 d = __ldg(reinterpret_cast<const float4 *>(delta + base + i + 4 * h));
                    float4 &y = v[p * Q + h];
                    y.x += d.x; y.y += d.y; y.z += d.z; y.w += d.w;
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < N; ++p) {
        const int i = (tid + p * TH) * W;
        if (i < hidden) {
#pragma unroll
            for (int h = 0; h < Q; ++h) {
                *reinterpret_cast<float4 *>(sm + i + 4 * h) = v[p * Q + h];
                if (x_out) *reinterpret_cast<float4 *>(x_out + base + i + 4 * h) = v[p * Q + h];
            }
        }
    }
    float4 g[FEW ? N * Q : 1];
    if constexpr (FEW) {
#pragma unroll
        for (int p = 0; p < N; ++p) {
            const int i = (tid + p * TH) * W;
            if (i < hidden) {
#pragma unroll
                for (int h = 0; h < Q; ++h) g[p * Q + h] = __ldg(reinterpret_cast<const float4 *>(gamma + i + 4 * h));
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < P; ++p) {
        float ss = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = tid + p * TH + j * T;
            const float y = e < hidden ? sm[e] : 0.0f;
            ss = fmaf(y, y, ss);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
        if (lane == 0) red[(tid + p * TH) >> 5] = ss;
    }
    __syncthreads();
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < T / 32; ++w) total += red[w];
    const float inv = 1.0f / sqrtf(total / (float)hidden + eps);
#pragma unroll
    for (int p = 0; p < N; ++p) {
        const int i = (tid + p * TH) * W;
        if (i < hidden) {
            float n[W];
#pragma unroll
            for (int h = 0; h < Q; ++h) {
                const float4 y = P > 1 ? *reinterpret_cast<const float4 *>(sm + i + 4 * h) : v[p * Q + h];
                const float4 c = FEW ? g[p * Q + h] : __ldg(reinterpret_cast<const float4 *>(gamma + i + 4 * h));
                n[4 * h] = (y.x * inv) * c.x;
                n[4 * h + 1] = (y.y * inv) * c.y;
                n[4 * h + 2] = (y.z * inv) * c.z;
                n[4 * h + 3] = (y.w * inv) * c.w;
            }
            if constexpr (BF16) store_act<ACT_BF16>(o, n, row, i, true);
            else *reinterpret_cast<float4 *>(static_cast<float *>(o.ptr) + (size_t)row * o.k + i) = make_float4(n[0], n[1], n[2], n[3]);
        }
    }
}

// The same between two matmuls of a chain of few rows: delta the sum of `parts` arrays `pitch` floats apart, the row in any
// form (blocks past the rows of `o` write padding), eight consecutive values per thread. One part takes it too: what it has
// over the kernel above are registers, 72 for 40, which keep its blocks from moving in beside the CTAs of the matmul in front, on as
// many SMs as there are rows, where they would hold up the CTAs of the matmul behind, which fetch their first weights early (1B
// shape, us per step with this one / with the loop taken out: 4 sequences 967 / 1007, 9 1275 / 1360, 16 1286 / 1377, 64 1160 / 1233).
template <int FORM, int T>
__global__ void __launch_bounds__(T, 1)   // (without the 1 the compiler keeps to 44 registers)
norm_form_kernel(const float *x, const float *delta, int parts, size_t pitch, const float *__restrict__ gamma, float eps, int hidden,
                 size_t row0, size_t row_step, float *x_out, ActOut o) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[32];
    __shared__ __align__(16) float sm[8 * T];
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, i = tid * 8;
    const bool on = i < hidden;
    if (FORM == ACT_DIGITS && row >= o.rows) {
        store_act_padding(o, row, on ? i : 0, on);
        return;
    }
    const size_t base = (row0 + row * row_step) * hidden;
    float v[8] = {};
    if (on) {   // (x not through the read-only path: x_out may be x)
        const float4 a = *reinterpret_cast<const float4 *>(x + base + i), b = *reinterpret_cast<const float4 *>(x + base + i + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        if (delta) {
            float d[8];
            load8(delta + base + i, parts, pitch, d);
#pragma unroll
            for (int t = 0; t < 8; ++t) v[t] += d[t];
        }
        const float4 lo = make_float4(v[0], v[1], v[2], v[3]), hi = make_float4(v[4], v[5], v[6], v[7]);
        *reinterpret_cast<float4 *>(sm + i) = lo;
        *reinterpret_cast<float4 *>(sm + i + 4) = hi;
        if (x_out) {
            *reinterpret_cast<float4 *>(x_out + base + i) = lo;
            *reinterpret_cast<float4 *>(x_out + base + i + 4) = hi;
        }
    }
    float g[8] = {};
    if (on) load8(gamma + i, 1, 0, g);
    __syncthreads();
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int e = tid + j * T;
        const float y = e < hidden ? sm[e] : 0.0f;
        ss = fmaf(y, y, ss);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
    if (lane == 0) red[tid >> 5] = ss;
    __syncthreads();
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < T / 32; ++w) total += red[w];
    const float inv = 1.0f / sqrtf(total / (float)hidden + eps);
#pragma unroll
    for (int t = 0; t < 8; ++t) v[t] = (v[t] * inv) * g[t];
    store_act<FORM>(o, v, row, i, on);
}

// The same for operands that are not 16-byte aligned and rows that are no multiple of 8, up to 16384
template <bool ACT, int NE>
__global__ void __launch_bounds__(1024)
add_rms_norm_kernel(const float *x, const float *__restrict__ delta, const float *__restrict__ gamma, float eps,
                    int hidden, float *x_out, void *__restrict__ normed) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[32];
    const size_t base = (size_t)blockIdx.x * hidden;
    float v[NE], g[NE];
#pragma unroll
    for (int j = 0; j < NE; ++j) {
        const int i = threadIdx.x + j * blockDim.x;
        v[j] = i < hidden ? x[base + i] : 0.0f;
        g[j] = i < hidden ? __ldg(gamma + i) : 0.0f;
    }
    if (delta) {
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            const int i = threadIdx.x + j * blockDim.x;
            if (i < hidden) v[j] += __ldg(delta + base + i);
        }
    }
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < NE; ++j) ss = fmaf(v[j], v[j], ss);
    if (x_out) {
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            const int i = threadIdx.x + j * blockDim.x;
            if (i < hidden) x_out[base + i] = v[j];
        }
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)hidden + eps);
#pragma unroll
    for (int j = 0; j < NE; ++j) {
        const int i = threadIdx.x + j * blockDim.x;
        if (i < hidden) {
            const float n = (v[j] * inv) * g[j];
            if constexpr (ACT)
                static_cast<__nv_bfloat16 *>(normed)[base + (i & ~7) + gemm_order_pos(i & 7)] = __float2bfloat16_rn(n);
            else
                static_cast<float *>(normed)[base + i] = n;
        }
    }
}

// The same for rows longer than 16384: the row is walked in a loop and read again for the scaling
template <bool ACT>
__global__ void __launch_bounds__(1024)
add_rms_norm_long_kernel(const float *x, const float *__restrict__ delta, const float *__restrict__ gamma, float eps,
                         int hidden, float *x_out, void *__restrict__ normed) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[32];
    const size_t base = (size_t)blockIdx.x * hidden;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
        float v = x[base + i];
        if (delta) v += delta[base + i];
        if (x_out) x_out[base + i] = v;
        ss = fmaf(v, v, ss);
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)hidden + eps);
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
        // x_out may alias x (in-place residual update): read the sum back instead of adding twice; every
        // thread re-reads exactly the elements it wrote
        float v = x_out ? x_out[base + i] : x[base + i];
        if (!x_out && delta) v += delta[base + i];
        const float n = (v * inv) * gamma[i];
        if constexpr (ACT)
            static_cast<__nv_bfloat16 *>(normed)[base + (i & ~7) + gemm_order_pos(i & 7)] = __float2bfloat16_rn(n);
        else
            static_cast<float *>(normed)[base + i] = n;
    }
}

// gate_up rows: [gate (inter) | up (inter)] -> silu(gate) * up, as fp32 or (ACT) as the bf16 activations of
// the next prefill-shaped linear. Bandwidth-bound: eight values per thread and step, 128-bit accesses
// (inter % 8 == 0, 16-byte aligned operands; swiglu_any_kernel takes the rest).
__device__ __forceinline__ float swiglu_one(float g, float u) {
    const float s = 1.0f / (1.0f + expf(-g));
    return (g * s) * u;
}
template <bool ACT>
__global__ void __launch_bounds__(256)
swiglu_kernel(const float *__restrict__ gu, void *__restrict__ out, int rows, int inter) {
    pdl_wait();
    pdl_trigger();
    const int n8 = inter / 8;
    for (int r = blockIdx.y; r < rows; r += gridDim.y) {
        const float4 *grow = reinterpret_cast<const float4 *>(gu + (size_t)r * 2 * inter);
        for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n8; c += gridDim.x * blockDim.x) {
            const float4 ga = __ldg(grow + 2 * c), gb = __ldg(grow + 2 * c + 1);
            const float4 ua = __ldg(grow + 2 * (n8 + c)), ub = __ldg(grow + 2 * (n8 + c) + 1);
            const float n[8] = {swiglu_one(ga.x, ua.x), swiglu_one(ga.y, ua.y), swiglu_one(ga.z, ua.z), swiglu_one(ga.w, ua.w),
                                swiglu_one(gb.x, ub.x), swiglu_one(gb.y, ub.y), swiglu_one(gb.z, ub.z), swiglu_one(gb.w, ub.w)};
            if constexpr (ACT) {
                reinterpret_cast<uint4 *>(out)[(size_t)r * n8 + c] = pack_bf16_gemm_order(n);
            } else {
                float4 *o = reinterpret_cast<float4 *>(out) + 2 * ((size_t)r * n8 + c);
                o[0] = make_float4(n[0], n[1], n[2], n[3]);
                o[1] = make_float4(n[4], n[5], n[6], n[7]);
            }
        }
    }
}
// The same for partial sums and for the forms of up to 16 rows. (In the place of the kernel above, one part, fp32 or bf16 out: 1 x
// 28672 1.8 us for 1.66, 128 x 5632 2.8 for 2.2, 2048 x 1024 5.5 for 4.3, 2048 x 28672 to bf16 94 for 83; without the loop over
// parts still up to 18 % more, 128 x 14336 3.9 for 3.3: whole warps and the general store. Between two matmuls of few rows it stays all
// the same, as told at norm_form_kernel: a step of 40 sequences 1106 us, 1114 with the other.)
template <int FORM>
__global__ void __launch_bounds__(256)
swiglu_form_kernel(const float *__restrict__ gu, int parts, size_t pitch, int rows, int inter, ActOut o) {
    pdl_wait();
    pdl_trigger();
    const int n8 = inter / 8;
    for (int r = blockIdx.y; r < rows; r += gridDim.y) {
        for (int c0 = blockIdx.x * blockDim.x; c0 < n8; c0 += gridDim.x * blockDim.x) {   // (whole warps reach store_act)
            const int c = c0 + threadIdx.x;
            const bool on = c < n8;
            if (FORM == ACT_DIGITS && r >= o.rows) {
                store_act_padding(o, r, on ? c * 8 : 0, on);
                continue;
            }
            float g[8] = {}, u[8] = {}, n[8];
            if (on) {
                load8(gu + (size_t)r * 2 * inter + c * 8, parts, pitch, g);
                load8(gu + (size_t)r * 2 * inter + inter + c * 8, parts, pitch, u);
            }
#pragma unroll
            for (int t = 0; t < 8; ++t) n[t] = swiglu_one(g[t], u[t]);
            store_act<FORM>(o, n, r, c * 8, on);
        }
    }
}
// any inter (ACT: a multiple of 8), any alignment of gate_up
template <bool ACT>
__global__ void swiglu_any_kernel(const float *__restrict__ gu, void *__restrict__ out, size_t rows, int inter) {
    pdl_wait();
    pdl_trigger();
    constexpr int V = ACT ? 8 : 1;
    const size_t total = rows * (size_t)(inter / V);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / (inter / V);
        const int c = (int)(i % (inter / V)) * V;
        float n[V];
#pragma unroll
        for (int j = 0; j < V; ++j) n[j] = swiglu_one(gu[r * 2 * inter + c + j], gu[r * 2 * inter + inter + c + j]);
        if constexpr (ACT)
            reinterpret_cast<uint4 *>(out)[i] = pack_bf16_gemm_order(n);
        else
            static_cast<float *>(out)[i] = n[0];
    }
}

// Element access to a KV cache row: f32 storage, or per-row symmetric int8 with one f32
// scale per row (KvDtype::I8 of crates/yscv-onnx/src/runner/kv_cache.rs:8-90; a row is one
// token's n_kv*d values of one layer). Reads dequantise on the fly: (float)q * scale.
template <typename KV>
__device__ __forceinline__ float kv_get(const KV *row, int i, float scale);
template <>
__device__ __forceinline__ float kv_get<float>(const float *row, int i, float) { return row[i]; }
template <>
__device__ __forceinline__ float kv_get<int8_t>(const int8_t *row, int i, float scale) {
    return __fmul_rn((float)row[i], scale);
}

// qkv rows: [q (n_q*d) | k (n_kv*d) | v (n_kv*d)], row r = b*seq + s at position *pos + s.
// The rows are the sum of `parts` arrays `pitch` floats apart (SUM; the loop costs one array 3 to 13 %: 1 position of 64 / 8
// heads of 128, int8, 2.24 us without it, 2.46 with). Writes rotated q to q_out (which may be the q of qkv,
// in place), rotated k and v into the cache at [b][position][head][d]
// (f32), or quantised per row with their scales at [b][position] (int8). A position outside
// [0, max_seq) appends nothing and raises YSCV_DEV_POS_OVERFLOW in the status word.
//
// Latency-bound: block (row, part) takes one part of a row: 0 its keys, 1 its values, 2.. pieces of up to
// ROPE_ITEMS x V query pairs, so that a thread has all its loads in flight at once and a decode batch fills
// more SMs than it has rows (one block per row, scalar accesses: 29 us for 64 rows of 64 + 16 heads of 128,
// 10 us for 32 rows of 32 + 8 heads of 64). The frequencies need only theta and are formed while the
// predecessor drains. V = pairs per thread and access: 4 where d % 8 == 0 and the rows are 16-byte aligned.
//
// int8 rows are LayerStorage::append for KvDtype::I8 (kv_cache.rs:44-60): scale = abs_max / 127 (1.0 when
// abs_max <= f32::EPSILON), inv = 1 / scale, q = clamp(round_half_away(v * inv), -127, 127).
// Dynamic shared memory: d floats of rotary factors (+ n_kv*d floats of the row to quantise, int8).
constexpr int ROPE_THREADS = 256, ROPE_ITEMS = 1024;
template <int V> struct RopeVec;
template <> struct RopeVec<4> { using T = float4; };
template <> struct RopeVec<1> { using T = float; };
template <typename KV, int V, bool SUM>
__global__ void __launch_bounds__(ROPE_THREADS)
rope_kv_append_kernel(const float *qkv, int parts, size_t pitch, float *q_out, int q_out_stride, int seq, int n_q, int n_kv, int d, float theta,
                      const int32_t *__restrict__ pos, KV *__restrict__ kc, KV *__restrict__ vc,
                      float *__restrict__ kscale, float *__restrict__ vscale, int max_seq, int *__restrict__ status) {
    constexpr bool I8 = sizeof(KV) == 1;
    using VT = typename RopeVec<V>::T;
    extern __shared__ __align__(16) float rsm[];
    __shared__ float red[8];
    const int half = d / 2, hv = half / V;
    float *cs_tab = rsm, *sn_tab = rsm + half, *row_sm = rsm + d;
    const int part = blockIdx.y;
    if (part != 1)
        for (int i = threadIdx.x; i < half; i += blockDim.x) cs_tab[i] = 1.0f / powf(theta, 2.0f * (float)i / (float)d);
    pdl_wait();
    pdl_trigger();
    const int row = blockIdx.x, b = row / seq, s = row % seq;
    const int p = *pos + s;
    const bool in_range = p >= 0 && p < max_seq;
    if (!in_range && part == 0 && threadIdx.x == 0) *status = YSCV_DEV_POS_OVERFLOW;
    const float *r = qkv + (size_t)row * (n_q + 2 * n_kv) * d;
    const int kv_n = n_kv * d;
    auto load = [&](const float *v) {
        VT x = *reinterpret_cast<const VT *>(v);
        if constexpr (!SUM) return x;
        float *a = reinterpret_cast<float *>(&x);
#pragma unroll 4
        for (int s = 1; s < parts; ++s) {
            const VT y = *reinterpret_cast<const VT *>(v + s * pitch);
            const float *b = reinterpret_cast<const float *>(&y);
#pragma unroll
            for (int j = 0; j < V; ++j) a[j] += b[j];
        }
        return x;
    };
    const size_t slot = (size_t)b * max_seq + (in_range ? p : 0);
    if (part != 1) {
        // the angle of pair i is the same for every head: one table per block
        const float fp = (float)p;
        for (int i = threadIdx.x; i < half; i += blockDim.x) {
            const float a = cs_tab[i] * fp;
            sincosf(a, &sn_tab[i], &cs_tab[i]);
        }
        __syncthreads();
        const int first = part == 0 ? 0 : (part - 2) * ROPE_ITEMS;
        const int n_items = part == 0 ? n_kv * hv : min(n_q * hv - first, ROPE_ITEMS);
        const float *src = part == 0 ? r + (size_t)n_q * d : r;
        float *dst = part == 0 ? (I8 ? row_sm : reinterpret_cast<float *>(kc) + slot * kv_n) : q_out + (size_t)row * q_out_stride;
        for (int i0 = threadIdx.x; i0 < n_items; i0 += 4 * ROPE_THREADS) {
            VT x0[4], x1[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int idx = i0 + u * ROPE_THREADS + first;
                if (i0 + u * ROPE_THREADS < n_items) {
                    const float *v = src + (size_t)(idx / hv) * d + (idx % hv) * V;
                    x0[u] = load(v);
                    x1[u] = load(v + half);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int idx = i0 + u * ROPE_THREADS + first;
                if (i0 + u * ROPE_THREADS < n_items && (part != 0 || I8 || in_range)) {
                    const int i = (idx % hv) * V;
                    VT y0, y1;
                    const float *a0 = reinterpret_cast<const float *>(&x0[u]), *a1 = reinterpret_cast<const float *>(&x1[u]);
                    float *o0 = reinterpret_cast<float *>(&y0), *o1 = reinterpret_cast<float *>(&y1);
#pragma unroll
                    for (int j = 0; j < V; ++j) {
                        const float cs = cs_tab[i + j], sn = sn_tab[i + j];
                        // each product rounded, as the reference rounds it (rope.rs:24-117)
                        o0[j] = __fsub_rn(__fmul_rn(a0[j], cs), __fmul_rn(a1[j], sn));
                        o1[j] = __fadd_rn(__fmul_rn(a0[j], sn), __fmul_rn(a1[j], cs));
                    }
                    float *v = dst + (size_t)(idx / hv) * d + i;
                    *reinterpret_cast<VT *>(v) = y0;
                    *reinterpret_cast<VT *>(v + half) = y1;
                }
            }
        }
    }
    if (part > 1 || !in_range) return;   // (uniform across the block)
    const float *vsrc = r + (size_t)(n_q + n_kv) * d;
    if constexpr (I8) {
        if (part == 1)
            for (int i = threadIdx.x * V; i < kv_n; i += blockDim.x * V)
                *reinterpret_cast<VT *>(row_sm + i) = load(vsrc + i);
        __syncthreads();
        float amax = 0.0f;
        for (int i = threadIdx.x; i < kv_n; i += blockDim.x) amax = fmaxf(amax, fabsf(row_sm[i]));
        amax = block_max(amax, red);
        const float scale = (amax <= 1.1920929e-07f) ? 1.0f : __fdiv_rn(amax, 127.0f);
        const float inv = __fdiv_rn(1.0f, scale);
        if (threadIdx.x == 0) (part == 0 ? kscale : vscale)[slot] = scale;
        int8_t *dst = reinterpret_cast<int8_t *>(part == 0 ? kc : vc) + slot * kv_n;
        for (int i = threadIdx.x * V; i < kv_n; i += blockDim.x * V) {
            int8_t o[V];
#pragma unroll
            for (int j = 0; j < V; ++j) {
                const float x = __fmul_rn(row_sm[i + j], inv);
                // NaN -> 0, as Rust's saturating float-to-int cast does
                o[j] = (x != x) ? (int8_t)0 : (int8_t)(int)fminf(fmaxf(roundf(x), -127.0f), 127.0f);
            }
            if constexpr (V == 4)
                *reinterpret_cast<char4 *>(dst + i) = make_char4(o[0], o[1], o[2], o[3]);
            else
                dst[i] = o[0];
        }
    } else if (part == 1) {
        float *vdst = reinterpret_cast<float *>(vc) + slot * kv_n;
        for (int i = threadIdx.x * V; i < kv_n; i += blockDim.x * V)
            *reinterpret_cast<VT *>(vdst + i) = load(vsrc + i);
    }
}

// One block per (b, q head, sq). Keys 0 .. *pos + sq (causal) or *pos + seq_q - 1.
template <typename KV>
__global__ void __launch_bounds__(128)
gqa_attention_kernel(const float *__restrict__ q, int q_stride, int seq_q, int n_q, int n_kv, int d,
                     const KV *__restrict__ kc, const KV *__restrict__ vc,
                     const float *__restrict__ kscale, const float *__restrict__ vscale, int max_seq,
                     const int32_t *__restrict__ pos, int causal, float *__restrict__ out) {
    pdl_wait();
    pdl_trigger();
    constexpr bool I8 = sizeof(KV) == 1;
    extern __shared__ float sm[];
    float *scores = sm;           // max_seq
    float *qs = sm + max_seq;     // d
    __shared__ float red[4];
    const int sq = blockIdx.x, qh = blockIdx.y, b = blockIdx.z;
    const int kv_h = qh / (n_q / n_kv);
    int limit = *pos + (causal ? sq + 1 : seq_q);
    limit = limit > max_seq ? max_seq : (limit < 0 ? 0 : limit);
    const float scale = 1.0f / sqrtf((float)d);
    const float *qrow = q + ((size_t)b * seq_q + sq) * q_stride + (size_t)qh * d;
    for (int i = threadIdx.x; i < d; i += blockDim.x) qs[i] = qrow[i];
    __syncthreads();
    const KV *kb = kc + (size_t)b * max_seq * n_kv * d + (size_t)kv_h * d;
    const KV *vb = vc + (size_t)b * max_seq * n_kv * d + (size_t)kv_h * d;
    const float *ksc = I8 ? kscale + (size_t)b * max_seq : nullptr;
    const float *vsc = I8 ? vscale + (size_t)b * max_seq : nullptr;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float mx = -INFINITY;
    // a warp per key: lanes stride over d (coalesced), shuffle-reduce
    for (int sk = warp; sk < limit; sk += 4) {
        const KV *kr = kb + (size_t)sk * n_kv * d;
        const float rs = I8 ? ksc[sk] : 1.0f;
        float dot = 0.0f;
        for (int i = lane; i < d; i += 32) dot = fmaf(qs[i], kv_get<KV>(kr, i, rs), dot);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float sc = dot * scale;
        if (lane == 0) scores[sk] = sc;
        mx = fmaxf(mx, sc);
    }
    mx = block_max(mx, red);
    float se = 0.0f;
    for (int sk = threadIdx.x; sk < limit; sk += blockDim.x) {
        const float e = expf(scores[sk] - mx);
        scores[sk] = e;
        se += e;
    }
    se = block_sum(se, red);
    const float inv = se > 0.0f ? 1.0f / se : 0.0f;
    float *orow = out + ((size_t)b * seq_q + sq) * (size_t)n_q * d + (size_t)qh * d;
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        float acc = 0.0f;
        for (int sk = 0; sk < limit; ++sk)
            acc = fmaf(scores[sk] * inv, kv_get<KV>(vb + (size_t)sk * n_kv * d, i, I8 ? vsc[sk] : 1.0f), acc);
        orow[i] = acc;
    }
}

// Decode-shaped attention (one query position per sequence) with the keys split across
// blocks so that a long cache fills the machine: block (split, kv head, b) handles an equal share of
// the keys in use (dec_share) for ALL the query heads of its KV head's group from one pass over the
// share's key and value rows (a row is read once per group, not once per query head), leaves
// per query head an unnormalised partial output, its running max and its exp-sum in `part`;
// attention_combine_kernel merges the splits that have keys (the usual max-rescaling of a split softmax).
// Query heads are taken eight at a time. d % 16 == 0, d <= 128, 256 threads, n_splits * CH >= max_seq.
//
// Bound by the latency of its phases, not by the cache's bytes (32 sequences x 200 keys of the 1B head
// shape are 13 MB). So the whole share is brought to shared memory by asynchronous copies issued at once
// (keys and values: one memory latency), and the softmax takes one warp per head (two block barriers in
// all; one block-wide maximum and sum per head were 32): 25.6 -> 11.0 us for that shape.
constexpr int DEC_HB = 8;
constexpr int DEC_THREADS = 256;
__device__ __forceinline__ int dec_limit(const int32_t *pos, int max_seq) { return max(0, min(max_seq, *pos + 1)); }
// Keys per split. A cache is mostly longer than the conversation in it, and a block costs about as much for a
// few keys as for CH: equal shares over as few splits as hold the keys in use in shares of up to CH, or, while
// that is fewer than `want` (two blocks per SM), in shares of down to 64. 200 keys in a cache of 8192, 32
// sequences, 64 / 8 heads of 128, f32 / int8: 59 / 27 us, spread over all splits 318 / 139. A nearly full cache
// keeps all its splits (32 / 4 heads of 64, 8 sequences, 2049 keys: 16.1 us in 18 shares, 19.6 in 17).
template <int CH> __device__ __forceinline__ int dec_share(int limit, int n_splits, int want) {
    int used = max(1, max((limit + CH - 1) / CH, min(min((limit + 63) / 64, want), n_splits)));
    if (used * 8 >= n_splits * 7) used = n_splits;
    return (limit + used - 1) / used;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <typename KV> __host__ __device__ constexpr int dec_pitch(int d) { return d * (int)sizeof(KV) + 16; }   // bytes of a staged row
template <typename KV, int CH> __host__ __device__ constexpr int dec_k_bytes(int d) {
    // (the partial sums, 32 KB, take the keys' place)
    return CH * dec_pitch<KV>(d) > DEC_THREADS * 4 * DEC_HB * 4 ? CH * dec_pitch<KV>(d) : DEC_THREADS * 4 * DEC_HB * 4;
}
template <typename KV, int CH> constexpr size_t dec_smem(int d) {
    return (size_t)DEC_HB * d * 4 + DEC_HB * (CH + 4) * 4 + dec_k_bytes<KV, CH>(d) + (size_t)CH * dec_pitch<KV>(d);
}

// D = 64 or 128: the head size, known to the compiler (index arithmetic without divisions); 0: any
template <typename KV, int CH, int D>
__global__ void __launch_bounds__(DEC_THREADS, 3)
gqa_decode_split_kernel(const float *__restrict__ q, int q_stride, int n_q, int n_kv, int d_,
                        const KV *__restrict__ kc, const KV *__restrict__ vc,
                        const float *__restrict__ kscale, const float *__restrict__ vscale, int max_seq,
                        const int32_t *__restrict__ pos, int want, float *__restrict__ part) {
    pdl_wait();
    pdl_trigger();
    constexpr bool I8 = sizeof(KV) == 1;
    constexpr int HB = DEC_HB, WP = CH + 4;
    const int d = D ? D : d_;
    constexpr int HT = HB * CH / DEC_THREADS;      // heads per thread in the score phase
    extern __shared__ __align__(16) unsigned char dsm[];
    const int pitch = dec_pitch<KV>(d);
    float *qs = reinterpret_cast<float *>(dsm);    // [HB][d]
    float *wts = qs + HB * d;                      // [HB][WP]
    unsigned char *ks = reinterpret_cast<unsigned char *>(wts + HB * WP);   // [CH][pitch]
    unsigned char *vs = ks + dec_k_bytes<KV, CH>(d);                        // [CH][pitch]
    float *psum = reinterpret_cast<float *>(ks);   // [key groups][HB][d], after the scores
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int split = blockIdx.x, kv_h = blockIdx.y, b = blockIdx.z, n_splits = gridDim.x;
    const int grp = n_q / n_kv;
    const int limit = dec_limit(pos, max_seq), share = dec_share<CH>(limit, n_splits, want);
    const int k0 = split * share, nk = min(limit, k0 + share) - k0;
    if (nk <= 0) return;   // (the merge does not read this split)
    const float scale = 1.0f / sqrtf((float)d);
    const size_t row_bytes = (size_t)n_kv * d * sizeof(KV);
    const float *vsc = I8 ? vscale + (size_t)b * max_seq + k0 : nullptr;
    {
        const size_t first = (((size_t)b * max_seq + k0) * n_kv + kv_h) * d * sizeof(KV);
        const unsigned char *kb = reinterpret_cast<const unsigned char *>(kc) + first, *vb = reinterpret_cast<const unsigned char *>(vc) + first;
        const int pieces = d * (int)sizeof(KV) / 16;
        const uint32_t kd = (uint32_t)__cvta_generic_to_shared(ks), vd = (uint32_t)__cvta_generic_to_shared(vs);
        for (int i = tid; i < nk * pieces; i += DEC_THREADS) {
            const int row = i / pieces, c = (i - row * pieces) * 16;
            cp_async16(kd + row * pitch + c, kb + row * row_bytes + c);
        }
        cp_async_commit();
        for (int i = tid; i < nk * pieces; i += DEC_THREADS) {
            const int row = i / pieces, c = (i - row * pieces) * 16;
            cp_async16(vd + row * pitch + c, vb + row * row_bytes + c);
        }
        cp_async_commit();
    }
    const int quads = d / 4, kgroups = DEC_THREADS / quads;      // value phase: thread = (key group, 4 dims)
    const int vq = tid % quads, vg = tid / quads;
    for (int h0 = 0; h0 < grp; h0 += HB) {
        const int nh = min(HB, grp - h0);
        const int qh0 = kv_h * grp + h0;
        for (int i = tid; i < HB * d; i += DEC_THREADS)
            qs[i] = i < nh * d ? q[(size_t)b * q_stride + (size_t)qh0 * d + i] : 0.0f;
        if (h0 > 0) {
            // the partial sums of the pass before lie where the keys were
            __syncthreads();
            const unsigned char *kb = reinterpret_cast<const unsigned char *>(kc) + (((size_t)b * max_seq + k0) * n_kv + kv_h) * d * sizeof(KV);
            const int pieces = d * (int)sizeof(KV) / 16;
            const uint32_t kd = (uint32_t)__cvta_generic_to_shared(ks);
            for (int i = tid; i < nk * pieces; i += DEC_THREADS) {
                const int row = i / pieces, c = (i - row * pieces) * 16;
                cp_async16(kd + row * pitch + c, kb + row * row_bytes + c);
            }
            cp_async_commit();
            cp_async_wait<0>();
        } else {
            cp_async_wait<1>();
        }
        __syncthreads();
        // ---- scores: thread = (key, HT heads) ----
        const int key = tid % CH, hs = tid / CH * HT;
        if (key < nk) {
            float dot[HT];
#pragma unroll
            for (int h = 0; h < HT; ++h) dot[h] = 0.0f;
            const unsigned char *kr = ks + key * pitch;
            const float rs = I8 ? kscale[(size_t)b * max_seq + k0 + key] : 1.0f;
#pragma unroll 2
            for (int c = 0; c < d; c += 16) {
                float kv[16];
                if constexpr (I8) {
                    const int4 w = *reinterpret_cast<const int4 *>(kr + c);
                    const int ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int t = 0; t < 16; ++t)
                        kv[t] = __fmul_rn((float)(int8_t)((ww[t >> 2] >> (8 * (t & 3))) & 255), rs);
                } else {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const float4 f = *reinterpret_cast<const float4 *>(kr + c * 4 + t * 16);
                        kv[4 * t] = f.x; kv[4 * t + 1] = f.y; kv[4 * t + 2] = f.z; kv[4 * t + 3] = f.w;
                    }
                }
#pragma unroll
                for (int h = 0; h < HT; ++h) {
                    const float4 *qh = reinterpret_cast<const float4 *>(qs + (hs + h) * d + c);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const float4 f = qh[t];
                        dot[h] = fmaf(f.x, kv[4 * t], dot[h]);
                        dot[h] = fmaf(f.y, kv[4 * t + 1], dot[h]);
                        dot[h] = fmaf(f.z, kv[4 * t + 2], dot[h]);
                        dot[h] = fmaf(f.w, kv[4 * t + 3], dot[h]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < HT; ++h) wts[(hs + h) * WP + key] = dot[h] * scale;
        }
        __syncthreads();
        // ---- softmax over the share: warp = head ----
        if (warp < nh) {
            float e[CH / 32], mx = -INFINITY, se = 0.0f;
#pragma unroll
            for (int i = 0; i < CH / 32; ++i) {
                const int j = lane + i * 32;
                e[i] = j < nk ? wts[warp * WP + j] : -INFINITY;
                mx = fmaxf(mx, e[i]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float ref = mx == -INFINITY ? 0.0f : mx;   // a share of -inf scores weighs nothing (and is no -inf + inf)
#pragma unroll
            for (int i = 0; i < CH / 32; ++i) {
                const int j = lane + i * 32;
                e[i] = j < nk ? expf(e[i] - ref) : 0.0f;
                se += e[i];
                // int8 values: fold the row scale of the value row into its weight once
                if (j < nk) wts[warp * WP + j] = I8 ? e[i] * vsc[j] : e[i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
            if (lane == 0) {
                float *po = part + (((size_t)b * n_q + qh0 + warp) * n_splits + split) * (d + 2);
                po[d] = mx;
                po[d + 1] = se;
            }
        }
        cp_async_wait<0>();
        __syncthreads();
        // ---- weighted values: thread (key group vg, dims 4*vq..): a value row quad serves every head ----
        if (vg < kgroups) {
            float acc[HB][4];
#pragma unroll
            for (int h = 0; h < HB; ++h) acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.0f;
#pragma unroll 2
            for (int j = vg; j < nk; j += kgroups) {
                float v4[4];
                if constexpr (I8) {
                    const int w = *reinterpret_cast<const int *>(vs + j * pitch + vq * 4);
                    v4[0] = (float)(int8_t)(w & 255); v4[1] = (float)(int8_t)((w >> 8) & 255);
                    v4[2] = (float)(int8_t)((w >> 16) & 255); v4[3] = (float)(int8_t)((w >> 24) & 255);
                } else {
                    const float4 f = *reinterpret_cast<const float4 *>(vs + j * pitch + vq * 16);
                    v4[0] = f.x; v4[1] = f.y; v4[2] = f.z; v4[3] = f.w;
                }
#pragma unroll
                for (int h = 0; h < HB; ++h) {
                    if (h < nh) {
                        const float w = wts[h * WP + j];
                        acc[h][0] = fmaf(w, v4[0], acc[h][0]);
                        acc[h][1] = fmaf(w, v4[1], acc[h][1]);
                        acc[h][2] = fmaf(w, v4[2], acc[h][2]);
                        acc[h][3] = fmaf(w, v4[3], acc[h][3]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < HB; ++h)
                if (h < nh)
                    *reinterpret_cast<float4 *>(psum + ((size_t)vg * HB + h) * d + 4 * vq) =
                        make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
        }
        __syncthreads();
        for (int i = tid; i < nh * d; i += DEC_THREADS) {
            const int h = i / d, dd = i - h * d;
            float v = 0.0f;
            for (int g = 0; g < kgroups; ++g) v += psum[((size_t)g * HB + h) * d + dd];
            part[(((size_t)b * n_q + qh0 + h) * n_splits + split) * (d + 2) + dd] = v;
        }
        __syncthreads();   // the next pass writes the shared arrays
    }
}

// ---- decode attention over an int8 cache on the tensor cores ------------------------------
//
// Same work split and the same `part` records as gqa_decode_split_kernel (one block per key chunk
// of 128, KV head and sequence, eight query heads of the group per pass), but both contractions
// run as mma.sync.m16n8k16 on fp16 operands with fp32 accumulators: an int8 cache entry is exact
// in fp16 (0x6400 | (q ^ 0x80) is 1024 + q + 128, minus 1152), the rotated query and the softmax
// weights are split into two fp16 terms (hi + lo, error below 2^-21 relative), so the result
// differs from the fp32 loop only in summation order.
//   scores^T [16 keys x 8 heads] = K tile [16 keys x d] (A, straight from the staged rows) x
//                                  Q^T [d x 8 heads] (B, two terms)
//   out [8 heads x d]            = P [8 (of 16 rows) x 128 keys] (A, two terms) x V [128 keys x d]
//                                  (B, four value rows' words transposed in registers)
// The k order inside an MMA is free as long as both operands agree: a thread takes 4 consecutive
// d (or keys) for the four k slots it owns, so its K bytes are one 16-byte read per 64 d and its V
// bytes four 32-bit reads per 16 keys and 32 columns. d is 64 or 128, a template argument: the kernel is bound by
// the instructions it issues (2.7 per cycle), and index divisions by a run-time d were a quarter of them: 64 x 2049
// keys, 64 / 8 heads of 128: 144 us with transposed byte stores, 119 without, 95 with d known (its bytes: 41).
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// four int8 -> two fp16 pairs {x0, x1}, {x2, x3}, exact
__device__ __forceinline__ void s8x4_to_h2x2(uint32_t w, uint32_t &lo, uint32_t &hi) {
    const uint32_t x = w ^ 0x80808080u;
    const __half2 bias = __floats2half2_rn(1152.0f, 1152.0f);
    uint32_t p0 = __byte_perm(x, 0x64646464u, 0x4140), p1 = __byte_perm(x, 0x64646464u, 0x4342);
    __half2 h0 = __hsub2(*reinterpret_cast<__half2 *>(&p0), bias), h1 = __hsub2(*reinterpret_cast<__half2 *>(&p1), bias);
    lo = *reinterpret_cast<uint32_t *>(&h0);
    hi = *reinterpret_cast<uint32_t *>(&h1);
}
// two floats -> fp16 pair of their leading terms and fp16 pair of the remainders
__device__ __forceinline__ void split_h2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
    const __half la = __float2half_rn(a - __half2float(ha)), lb = __float2half_rn(b - __half2float(hb));
    const __half2 h = __halves2half2(ha, hb), l = __halves2half2(la, lb);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

template <int D>
__global__ void __launch_bounds__(128)
gqa_decode_split_tc_kernel(const float *__restrict__ q, int q_stride, int n_q, int n_kv,
                           const int8_t *__restrict__ kc, const int8_t *__restrict__ vc,
                           const float *__restrict__ kscale, const float *__restrict__ vscale, int max_seq,
                           const int32_t *__restrict__ pos, int want, float *__restrict__ part) {
    pdl_wait();
    pdl_trigger();
    constexpr int CH = 128, HB = 8, d = D;
    constexpr int SP = CH + 4;            // scores row pitch (floats)
    constexpr int PP = CH + 8;            // weight row pitch (halves)
    extern __shared__ __align__(16) unsigned char tsm[];
    // rows of d bytes, keys and values alike. Keys: for d = 128 the 16-byte piece c of row r sits at piece
    // c ^ ((r & 1) * 4): the eight lanes of a read phase (two rows x four pieces) then touch eight different
    // bank groups. Values: piece c ^ (((r >> 2) & (d / 32 - 1)) * 2): the four lanes of a quad read 32-bit
    // words of rows four apart, the eight quads 32 consecutive bytes.
    constexpr int ksw = d == 128 ? 4 : 0, vmask = d / 32 - 1;
    unsigned char *Ks = tsm;                                         // [CH][d]
    unsigned char *Vs = Ks + CH * d;                                 // [CH][d]
    float *Ssm = reinterpret_cast<float *>(Vs + CH * d);             // [HB][SP]
    __half *Ph = reinterpret_cast<__half *>(Ssm + HB * SP);          // [HB][PP] leading terms
    __half *Pl = Ph + HB * PP;                                       // [HB][PP] remainders
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int split = blockIdx.x, kv_h = blockIdx.y, b = blockIdx.z, n_splits = gridDim.x;
    const int grp = n_q / n_kv;
    const int limit = dec_limit(pos, max_seq), share = dec_share<CH>(limit, n_splits, want);
    const int k0 = split * share, nk = min(limit, k0 + share) - k0;
    if (nk <= 0) return;   // (the merge does not read this split)
    const float scale = 1.0f / sqrtf((float)d);
    const int8_t *kb = kc + (size_t)b * max_seq * n_kv * d + (size_t)kv_h * d;
    const int8_t *vb = vc + (size_t)b * max_seq * n_kv * d + (size_t)kv_h * d;
    const float *ksc = kscale + (size_t)b * max_seq, *vsc = vscale + (size_t)b * max_seq;

    // ---- stage the share by asynchronous copies, all in flight at once; rows past nk are zeros ----
    {
        constexpr int pieces = d / 16;    // 16-byte pieces per row
        const uint32_t kd = (uint32_t)__cvta_generic_to_shared(Ks), vd = (uint32_t)__cvta_generic_to_shared(Vs);
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            // (piece and swizzle of a thread stay the same from step to step: rows advance by 128 / pieces)
#pragma unroll
            for (int i0 = 0; i0 < CH * pieces; i0 += 128) {
                const int i = i0 + tid, row = i / pieces, pc = i % pieces;
                const int at = pc ^ (which == 0 ? (row & 1) * ksw : ((row >> 2) & vmask) * 2);
                const int8_t *src = (which == 0 ? kb : vb) + (size_t)(k0 + min(row, nk - 1)) * n_kv * d + pc * 16;
                const int live = row < nk ? 16 : 0;   // 0 source bytes: the piece is filled with zeros
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((which == 0 ? kd : vd) + row * d + (at << 4)),
                             "l"(src), "r"(live) : "memory");
            }
            cp_async_commit();
        }
    }
    // what else a thread reads from memory travels with them: the scales of its four keys in the scores
    // (rows 32 warp + 16 i + g and + 8) and of its four in the weights, and (below) the query operands
    float ks4[4], vs4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int key = warp * 32 + (i >> 1) * 16 + (i & 1) * 8 + g;
        ks4[i] = key < nk ? __ldg(ksc + k0 + key) * scale : 0.0f;
        vs4[i] = 4 * lane + i < nk ? __ldg(vsc + k0 + 4 * lane + i) : 0.0f;
    }

    for (int h0 = 0; h0 < grp; h0 += HB) {
        const int nh = min(HB, grp - h0);
        const int qh0 = kv_h * grp + h0;
        // ---- this thread's query operands: head g, for the k step (64-block B, quarter s4) the
        // four d = 64 B + 16 t + 4 s4 .. + 3, as leading terms and remainders ----
        uint32_t qh[8][2], ql[8][2];      // [k step][b0, b1]
        {
            const float *qr = q + (size_t)b * q_stride + (size_t)(qh0 + (g < nh ? g : 0)) * d;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (ks * 16 < d && g < nh) v = __ldg(reinterpret_cast<const float4 *>(qr + (ks >> 2) * 64 + 16 * t + 4 * (ks & 3)));
                split_h2(v.x, v.y, qh[ks][0], ql[ks][0]);
                split_h2(v.z, v.w, qh[ks][1], ql[ks][1]);
            }
        }
        if (h0 == 0) {
            cp_async_wait<1>();
            __syncthreads();
        }
        // ---- scores^T: warp w takes keys 32 w .. 32 w + 31 as two tiles of 16 ----
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const int keyA = warp * 32 + mt * 16 + g, keyB = keyA + 8;
            float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int blk = 0; blk < 2; ++blk) {
                if (blk * 64 < d) {
                    // (keyA and keyB = keyA + 8 have the same parity, hence the same swizzle)
                    const int pc = (blk * 4 + t) ^ ((keyA & 1) * ksw);
                    const uint4 wa = *reinterpret_cast<const uint4 *>(Ks + keyA * d + (pc << 4));
                    const uint4 wb = *reinterpret_cast<const uint4 *>(Ks + keyB * d + (pc << 4));
                    const uint32_t xa[4] = {wa.x, wa.y, wa.z, wa.w}, xb[4] = {wb.x, wb.y, wb.z, wb.w};
#pragma unroll
                    for (int s4 = 0; s4 < 4; ++s4) {
                        uint32_t a0, a2, a1, a3;
                        s8x4_to_h2x2(xa[s4], a0, a2);
                        s8x4_to_h2x2(xb[s4], a1, a3);
                        const int ks = blk * 4 + s4;
                        mma_f16(c, a0, a1, a2, a3, ql[ks][0], ql[ks][1]);
                        mma_f16(c, a0, a1, a2, a3, qh[ks][0], qh[ks][1]);
                    }
                }
            }
            // c0, c1 = (keyA, heads 2t, 2t+1); c2, c3 = (keyB, same heads)
            const float sa = ks4[mt * 2], sb = ks4[mt * 2 + 1];
            Ssm[(2 * t) * SP + keyA] = keyA < nk ? c[0] * sa : -INFINITY;
            Ssm[(2 * t + 1) * SP + keyA] = keyA < nk ? c[1] * sa : -INFINITY;
            Ssm[(2 * t) * SP + keyB] = keyB < nk ? c[2] * sb : -INFINITY;
            Ssm[(2 * t + 1) * SP + keyB] = keyB < nk ? c[3] * sb : -INFINITY;
        }
        __syncthreads();
        // ---- softmax over the chunk: warp w takes heads 2 w and 2 w + 1, a lane four keys ----
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int h = 2 * warp + hh;
            const float4 sv = *reinterpret_cast<const float4 *>(Ssm + h * SP + 4 * lane);
            float mx = fmaxf(fmaxf(sv.x, sv.y), fmaxf(sv.z, sv.w));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const int key = 4 * lane;
            float e[4] = {sv.x, sv.y, sv.z, sv.w};
            float se = 0.0f;
            const float ref = mx == -INFINITY ? 0.0f : mx;   // (as above)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                e[i] = (key + i < nk && h < nh) ? expf(e[i] - ref) : 0.0f;
                se += e[i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
            if (lane == 0 && h < nh) {
                float *po = part + (((size_t)b * n_q + qh0 + h) * n_splits + split) * (d + 2);
                po[d] = mx;
                po[d + 1] = se;
            }
            // the value row's scale is folded into its weight; two fp16 terms per weight
            uint32_t hi01, lo01, hi23, lo23;
            split_h2(e[0] * vs4[0], e[1] * vs4[1], hi01, lo01);
            split_h2(e[2] * vs4[2], e[3] * vs4[3], hi23, lo23);
            *reinterpret_cast<uint2 *>(Ph + h * PP + key) = make_uint2(hi01, hi23);
            *reinterpret_cast<uint2 *>(Pl + h * PP + key) = make_uint2(lo01, lo23);
        }
        cp_async_wait<0>();
        __syncthreads();
        // ---- out = P x V, rows 8..15 of P zero: a warp takes 32 columns as four n tiles, tile j the columns
        // 4 g + j, so that a 32-bit word of a value row holds one column of each tile and four rows' words
        // transpose in registers (a transposed copy in shared memory took 128 byte stores per thread).
        // d = 64: two warps per column block, half the keys each ----
        {
            constexpr int blocks = d / 32, steps = CH / 16 * blocks / 4;
            const int cb = warp % blocks, part_k = warp / blocks;
            float o[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0f;
#pragma unroll
            for (int k_ = 0; k_ < steps; ++k_) {
                const int key0 = (part_k * steps + k_) * 16 + 4 * t;
                const uint2 ah = *reinterpret_cast<const uint2 *>(Ph + g * PP + key0);
                const uint2 al = *reinterpret_cast<const uint2 *>(Pl + g * PP + key0);
                // (rows key0 .. key0 + 3 share the piece swizzle)
                const unsigned char *vr = Vs + key0 * d + (((cb * 2 + (g >> 2)) ^ (((key0 >> 2) & vmask) * 2)) << 4) + (g & 3) * 4;
                const uint32_t w0 = *reinterpret_cast<const uint32_t *>(vr), w1 = *reinterpret_cast<const uint32_t *>(vr + d);
                const uint32_t w2 = *reinterpret_cast<const uint32_t *>(vr + 2 * d), w3 = *reinterpret_cast<const uint32_t *>(vr + 3 * d);
                uint32_t b0[4], b1[4];
                s8x4_to_h2x2(__byte_perm(w0, w1, 0x5140), b0[0], b0[1]);
                s8x4_to_h2x2(__byte_perm(w0, w1, 0x7362), b0[2], b0[3]);
                s8x4_to_h2x2(__byte_perm(w2, w3, 0x5140), b1[0], b1[1]);
                s8x4_to_h2x2(__byte_perm(w2, w3, 0x7362), b1[2], b1[3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    mma_f16(o[j], al.x, 0u, al.y, 0u, b0[j], b1[j]);
                    mma_f16(o[j], ah.x, 0u, ah.y, 0u, b0[j], b1[j]);
                }
            }
            // o[j][0], o[j][1] = head g, columns 32 cb + 4 * (2t) + j and 4 * (2t + 1) + j
            if (blocks == 2) {
                float *half = Ssm;   // [2 column blocks][32 lanes][8]; the scores are used up
                if (part_k == 1) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        half[(cb * 32 + lane) * 9 + 2 * j] = o[j][0];
                        half[(cb * 32 + lane) * 9 + 2 * j + 1] = o[j][1];
                    }
                }
                __syncthreads();
                if (part_k == 0) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        o[j][0] += half[(cb * 32 + lane) * 9 + 2 * j];
                        o[j][1] += half[(cb * 32 + lane) * 9 + 2 * j + 1];
                    }
                }
            }
            if (part_k == 0 && g < nh) {
                // (records start at multiples of d + 2 floats: 8-byte aligned)
                float *po = part + (((size_t)b * n_q + qh0 + g) * n_splits + split) * (d + 2) + cb * 32 + 8 * t;
                *reinterpret_cast<float2 *>(po) = make_float2(o[0][0], o[1][0]);
                *reinterpret_cast<float2 *>(po + 2) = make_float2(o[2][0], o[3][0]);
                *reinterpret_cast<float2 *>(po + 4) = make_float2(o[0][1], o[1][1]);
                *reinterpret_cast<float2 *>(po + 6) = make_float2(o[2][1], o[3][1]);
            }
        }
        __syncthreads();   // the score and weight arrays are reused by the next pass
    }
}

// Merges the splits: block per (q head, b), 128 threads; out row [b][n_q*d]. The splits' weights are
// worked out once per block, a thread per split, then a thread per column adds with its loads in flight
// (a serial walk that evaluated every weight in every thread: 27 us for 64 x 64 heads x 18 splits).
// PRE: loads of a column in flight, BLOCKS: per SM. Sixteen and ten behind the f32 kernel (8 sequences, 64 / 8 heads of
// 128, 2049 keys in 2178: 62.4 us both kernels, with eight and sixteen 65.2), eight and sixteen behind the int8
// kernels, which leave it half the time (32 sequences, 32 / 4 heads of 64, 200 keys in 330: 8.0 us, the other way 12.2).
constexpr int COMBINE_BATCH = 128;
// The row goes out in the form of the matmul behind it; rows past those of `o` are its padding.
template <int CH, int PRE, int BLOCKS, int FORM>
__global__ void __launch_bounds__(128, BLOCKS)
attention_combine_kernel(const float *__restrict__ part, int n_splits, int d, int max_seq, const int32_t *__restrict__ pos,
                         int want, ActOut o) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[4], wt[COMBINE_BATCH];
    const int tid = threadIdx.x;
    if (FORM == ACT_DIGITS && (int)blockIdx.y >= o.rows) {
        if (tid < 32) store_act_padding(o, blockIdx.y, blockIdx.x * d + (tid * 8 < d ? tid * 8 : 0), tid * 8 < d);
        return;
    }
    const size_t hb = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
    const float *p = part + hb * n_splits * (d + 2);
    // what the first splits left is fetched while the position, which says how many count, is on its way
    float v[PRE];
    const float m0 = tid < n_splits ? p[(size_t)tid * (d + 2) + d] : -INFINITY, l0 = tid < n_splits ? p[(size_t)tid * (d + 2) + d + 1] : 0.0f;
#pragma unroll
    for (int u = 0; u < PRE; ++u) v[u] = tid < d && u < n_splits ? p[(size_t)u * (d + 2) + tid] : 0.0f;
    const int limit = dec_limit(pos, max_seq), share = dec_share<CH>(limit, n_splits, want);
    const int used = limit > 0 ? (limit + share - 1) / share : 0;
    float M = tid < used ? m0 : -INFINITY;
    for (int s = tid + 128; s < used; s += 128) M = fmaxf(M, p[(size_t)s * (d + 2) + d]);
    M = block_max(M, red);
    float L = 0.0f, acc = 0.0f;
    for (int s0 = 0; s0 < used; s0 += COMBINE_BATCH) {
        const int s = s0 + tid, ns = min(COMBINE_BATCH, used - s0);
        float w = 0.0f;
        if (s < used) {
            const float m = s0 == 0 ? m0 : p[(size_t)s * (d + 2) + d];
            if (m > -INFINITY) w = expf(m - M);
            if (w > 0.0f) L += w * (s0 == 0 ? l0 : p[(size_t)s * (d + 2) + d + 1]);
        }
        __syncthreads();
        wt[tid] = w;
        __syncthreads();
        if (tid < d) {
            for (int i = 0; i < ns; i += PRE) {
                if (s0 + i > 0) {
#pragma unroll
                    for (int u = 0; u < PRE; ++u) v[u] = i + u < ns ? p[(size_t)(s0 + i + u) * (d + 2) + tid] : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < PRE; ++u)
                    if (i + u < ns) acc = fmaf(wt[i + u], v[u], acc);
            }
        }
    }
    L = block_sum(L, red);
    const float inv = L > 0.0f ? 1.0f / L : 0.0f;
    if constexpr (FORM == ACT_F32) {
        if (tid < d) static_cast<float *>(o.ptr)[hb * d + tid] = acc * inv;
    } else {
        __shared__ __align__(16) float row[128];
        row[tid] = acc * inv;
        __syncthreads();
        if (tid < 32) {
            float v[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) v[t] = row[tid * 8 < d ? tid * 8 + t : 0];
            store_act<FORM>(o, v, blockIdx.y, blockIdx.x * d + tid * 8, tid * 8 < d);
        }
    }
}

// out[m][n] = sum_k x[m][k] * w[n][k]; one warp per weight row, up to MT x rows per pass. For few weight rows, where what
// counts is how many warps share the weights: with two and four rows per warp (the kernel below, which takes over where the
// rows fill the SMs; its sums are the same) 3 x 300 x 512 takes 2.9 us and here 1.9, 4 x 1000 x 4096 12.7 and 7.3, 8 x 1000 x 4096
// 20.1 and 14.5, from HBM 1 x 3000 x 4096 15.6 and 12.6, 3 x 3000 x 4096 23.8 and 16.2; the other way 1 x 4096 x 4096 17.1 and
// 21.9, 4 x 4096 x 4096 24.3 and 28.0, 8 x 3000 x 4096 30.1 and 32.4, 5 x 6000 x 1024 10.6 and 15.9.
template <int MT>
__global__ void __launch_bounds__(256)
f32_matmul_rows_kernel(const float *__restrict__ w, const float *__restrict__ x, float *__restrict__ out, int m0, int M, int N, int K) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int mt = min(MT, M - m0);
    for (int n = blockIdx.x * wpb + (threadIdx.x >> 5); n < N; n += gridDim.x * wpb) {
        const float4 *wr = reinterpret_cast<const float4 *>(w + (size_t)n * K);
        float acc[MT];
#pragma unroll
        for (int i = 0; i < MT; ++i) acc[i] = 0.0f;
#pragma unroll 4
        for (int c = lane; c < K / 4; c += 32) {
            const float4 wv = __ldg(wr + c);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                if (i < mt) {
                    const float4 xv = __ldg(reinterpret_cast<const float4 *>(x + (size_t)(m0 + i) * K) + c);
                    acc[i] = fmaf(wv.x, xv.x, acc[i]);
                    acc[i] = fmaf(wv.y, xv.y, acc[i]);
                    acc[i] = fmaf(wv.z, xv.z, acc[i]);
                    acc[i] = fmaf(wv.w, xv.w, acc[i]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            float v = acc[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0 && i < mt) out[(size_t)(m0 + i) * N + n] = v;
        }
    }
}

// out[m][n] = sum_k x[m][k] * w[n][k] for m <= MT: one warp per R weight rows, which share the x rows it reads.
// Bound by the weights' HBM stream: enough loads in flight per warp (R rows, unrolled) and one pass whatever m.
// The weights skip L1, which holds the x rows. With a row per warp, four loads in flight and a pass per 4 x rows
// 32000 x 2048 took 54.1 / 57.3 / 119 us at 1 / 4 / 8 x rows, now 41.2 / 49 / 67 (6.4, 5.3 and 3.9 TB/s; from five rows
// on the x rows' L1 reads bound it); 128256 x 8192 at one row 770 -> 600 us.
__device__ __forceinline__ float4 ldg_stream(const float4 *p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
template <int MT, int R, int UNROLL>
__global__ void __launch_bounds__(256)
f32_matmul_kernel(const float *__restrict__ w, const float *__restrict__ x, float *__restrict__ out, int M, int N, int K) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5, K4 = K / 4;
    for (int n = (blockIdx.x * wpb + (threadIdx.x >> 5)) * R; n < N; n += gridDim.x * wpb * R) {
        const float4 *wr[R];
#pragma unroll
        for (int j = 0; j < R; ++j) wr[j] = reinterpret_cast<const float4 *>(w + (size_t)min(n + j, N - 1) * K);
        float acc[R][MT];
#pragma unroll
        for (int j = 0; j < R; ++j)
#pragma unroll
            for (int i = 0; i < MT; ++i) acc[j][i] = 0.0f;
        // (no branch on i: x rows past M repeat the last one, so that a step's loads are issued together)
        auto step = [&](const float4 (&wv)[R], int c) {
            float4 xv[MT];
#pragma unroll
            for (int i = 0; i < MT; ++i) xv[i] = __ldg(reinterpret_cast<const float4 *>(x + (size_t)min(i, M - 1) * K) + c);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    acc[j][i] = fmaf(wv[j].x, xv[i].x, acc[j][i]);
                    acc[j][i] = fmaf(wv[j].y, xv[i].y, acc[j][i]);
                    acc[j][i] = fmaf(wv[j].z, xv[i].z, acc[j][i]);
                    acc[j][i] = fmaf(wv[j].w, xv[i].w, acc[j][i]);
                }
            }
        };
        int c = lane;
        for (; c + (UNROLL - 1) * 32 < K4; c += UNROLL * 32) {
            float4 wv[UNROLL][R];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u)
#pragma unroll
                for (int j = 0; j < R; ++j) wv[u][j] = ldg_stream(wr[j] + c + u * 32);
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) step(wv[u], c + u * 32);
        }
        for (; c < K4; c += 32) {
            float4 wv[R];
#pragma unroll
            for (int j = 0; j < R; ++j) wv[j] = ldg_stream(wr[j] + c);
            step(wv, c);
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                float v = acc[j][i];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0 && i < M && n + j < N) out[(size_t)i * N + n + j] = v;
            }
        }
    }
}

// The same product for a wide batch (m > 8): a shared-memory tiled SGEMM, 128 weight rows x 64
// activation rows per block, K walked 32 at a time, every thread an 8 x 4 block of outputs.
// The weights are read once from HBM per 64 activation rows.
constexpr int FM_BN = 128, FM_BM = 64, FM_BK = 32;
__global__ void __launch_bounds__(256)
f32_matmul_tiled_kernel(const float *__restrict__ w, const float *__restrict__ x, float *__restrict__ out,
                        int M, int N, int K) {
    pdl_wait();
    pdl_trigger();
    __shared__ float ws[FM_BK][FM_BN + 4];
    __shared__ float xs[FM_BK][FM_BM + 4];
    const int tid = threadIdx.x;
    const int n0 = blockIdx.x * FM_BN, m0 = blockIdx.y * FM_BM;
    const int tn = tid % 16, tm = tid / 16;      // outputs n0 + tn*8 .. +7, m0 + tm*4 .. +3
    float acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += FM_BK) {
        // stage the tiles transposed: [k][row]; rows / k past the edge are zero
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int idx = tid + it * 256, r = idx / 8, c = (idx % 8) * 4;   // 128 rows x 8 float4
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (n0 + r < N && k0 + c < K) v = __ldg(reinterpret_cast<const float4 *>(w + (size_t)(n0 + r) * K + k0 + c));
            ws[c][r] = v.x; ws[c + 1][r] = v.y; ws[c + 2][r] = v.z; ws[c + 3][r] = v.w;
        }
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            const int idx = tid + it * 256, r = idx / 8, c = (idx % 8) * 4;   // 64 rows x 8 float4
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (m0 + r < M && k0 + c < K) v = __ldg(reinterpret_cast<const float4 *>(x + (size_t)(m0 + r) * K + k0 + c));
            xs[c][r] = v.x; xs[c + 1][r] = v.y; xs[c + 2][r] = v.z; xs[c + 3][r] = v.w;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < FM_BK; ++kk) {
            const float4 wa = *reinterpret_cast<const float4 *>(&ws[kk][tn * 8]);
            const float4 wb = *reinterpret_cast<const float4 *>(&ws[kk][tn * 8 + 4]);
            const float4 xa = *reinterpret_cast<const float4 *>(&xs[kk][tm * 4]);
            const float wv[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
            const float xv[4] = {xa.x, xa.y, xa.z, xa.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + tm * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + tn * 8 + j;
            if (n < N) out[(size_t)m * N + n] = acc[i][j];
        }
    }
}

// greedy token per row: the LAST index among equal maxima (Iterator::max_by)
__global__ void __launch_bounds__(256)
argmax_last_kernel(const float *__restrict__ logits, int vocab, int32_t *__restrict__ out) {
    pdl_wait();
    pdl_trigger();
    __shared__ float bv[256];
    __shared__ int bi[256];
    const float *row = logits + (size_t)blockIdx.x * vocab;
    float best = -INFINITY;
    int idx = -1;
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
        const float v = row[i];
        if (idx < 0 || !(v < best)) {  // v >= best (or NaN): later index wins ties
            best = v;
            idx = i;
        }
    }
    bv[threadIdx.x] = best;
    bi[threadIdx.x] = idx;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            const float a = bv[threadIdx.x], b = bv[threadIdx.x + s];
            const int ia = bi[threadIdx.x], ib = bi[threadIdx.x + s];
            const bool take_b = ib >= 0 && (ia < 0 || b > a || (b == a && ib > ia));
            if (take_b) {
                bv[threadIdx.x] = b;
                bi[threadIdx.x] = ib;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = bi[0] < 0 ? 0 : bi[0];
}

// two-stage variant for wide vocabularies: 64 blocks per row leave (value, index) partials,
// the single-block kernel above then reduces those (indices carried along)
__global__ void __launch_bounds__(256)
argmax_partial_kernel(const float *__restrict__ logits, int vocab, float *__restrict__ pv,
                      int32_t *__restrict__ pi) {
    pdl_wait();
    pdl_trigger();
    __shared__ float bv[256];
    __shared__ int bi[256];
    const int row = blockIdx.y, nb = gridDim.x;
    const int per = (vocab + nb - 1) / nb;
    const int lo = blockIdx.x * per, hi = min(vocab, lo + per);
    const float *r = logits + (size_t)row * vocab;
    float best = -INFINITY;
    int idx = -1;
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        const float v = r[i];
        if (idx < 0 || !(v < best)) { best = v; idx = i; }
    }
    bv[threadIdx.x] = best;
    bi[threadIdx.x] = idx;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            const float a = bv[threadIdx.x], b = bv[threadIdx.x + s];
            const int ia = bi[threadIdx.x], ib = bi[threadIdx.x + s];
            if (ib >= 0 && (ia < 0 || b > a || (b == a && ib > ia))) { bv[threadIdx.x] = b; bi[threadIdx.x] = ib; }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) { pv[row * nb + blockIdx.x] = bv[0]; pi[row * nb + blockIdx.x] = bi[0]; }
}

__global__ void __launch_bounds__(64)
argmax_final_kernel(const float *__restrict__ pv, const int32_t *__restrict__ pi, int nb,
                    int32_t *__restrict__ out) {
    pdl_wait();
    pdl_trigger();
    // partials are in increasing index order: scan them in order, later wins ties (staged first: a scan that
    // loads as it goes waits for L2 again and again)
    __shared__ float sv[64];
    __shared__ int32_t si[64];
    const int row = blockIdx.x;
    if (threadIdx.x < nb) {
        sv[threadIdx.x] = pv[row * nb + threadIdx.x];
        si[threadIdx.x] = pi[row * nb + threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    float best = -INFINITY;
    int idx = -1;
#pragma unroll 8
    for (int j = 0; j < nb; ++j) {
        const int i = si[j];
        const float v = sv[j];
        if (i >= 0 && (idx < 0 || !(v < best))) { best = v; idx = i; }
    }
    out[row] = idx < 0 ? 0 : idx;
}

__global__ void advance_pos_kernel(int32_t *pos, int by) {
    pdl_wait();  // the predecessor may still read *pos, and its own predecessors must be covered
    pdl_trigger();
    *pos += by;
}

}  // namespace yscv

using namespace yscv;

#define DEC_PROLOGUE(ctx)                                                    \
    if (!(ctx)) return fail(YSCV_CUDA_ERR_BAD_ARG, "ctx is null");           \
    YSCV_CUDA_TRY(cudaSetDevice((ctx)->device))
#define DEC_EPILOGUE(ctx, name)                  \
    YSCV_CUDA_TRY(cudaGetLastError());           \
    (ctx)->launches++;                           \
    (ctx)->last_kernel = name;                   \
    return YSCV_CUDA_OK

extern "C" {

int yscv_cuda_embedding_dev(yscv_cuda_ctx *ctx, const float *d_weight, size_t vocab, size_t dim,
                            const int32_t *d_tokens, size_t rows, float *d_out) {
    DEC_PROLOGUE(ctx);
    if (!d_weight || !d_tokens || !d_out) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (dim % 4 != 0) return fail(YSCV_CUDA_ERR_UNSUPPORTED, "embedding dim must be a multiple of 4");
    if ((reinterpret_cast<uintptr_t>(d_weight) | reinterpret_cast<uintptr_t>(d_out)) & 15)
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "embedding table and output must be 16-byte aligned");
    if (rows == 0) return YSCV_CUDA_OK;
    YSCV_CUDA_TRY(launch_pdl(embedding_kernel, dim3((unsigned)rows), dim3(128), 0, ctx->stream, d_weight, d_tokens, d_out, (int)vocab, (int)dim));
    DEC_EPILOGUE(ctx, "embedding");
}

}  // extern "C"

namespace yscv {
// Name of an operator by the form it writes
static const char *form_name(int form, const char *f32, const char *bf16, const char *digits, const char *terms) {
    return form == ACT_BF16 ? bf16 : form == ACT_DIGITS ? digits : form == ACT_TERMS ? terms : f32;
}

// hidden % 8 == 0 and at most 8192, operands (and `pitch` floats) 16-byte aligned
int norm_form(yscv_cuda_ctx *ctx, const float *x, const float *delta, int parts, size_t pitch, const float *gamma, float eps,
              size_t rows, size_t row0, size_t row_step, size_t hidden, float *x_out, const ActOut &out, bool between) {
    const bool small = hidden <= 2048, few = rows <= NORM_FEW * ctx->sm_count;
    const char *name = form_name(out.form, "add_rms_norm", "add_rms_norm(bf16 activations out)", "add_rms_norm(digit planes out)", "add_rms_norm(fp16 terms out)");
    if (parts == 1 && (out.form == ACT_F32 || out.form == ACT_BF16) && !(between && few)) {
        auto pick = [&](auto bf16) {
            constexpr bool B = decltype(bf16)::value;
            return few ? (small ? norm_rows_kernel<B, 256, true> : norm_rows_kernel<B, 1024, true>)
                       : (small ? norm_rows_kernel<B, 256, false> : norm_rows_kernel<B, 1024, false>);
        };
        auto kern = out.form == ACT_BF16 ? pick(std::true_type()) : pick(std::false_type());
        YSCV_CUDA_TRY(launch_pdl(kern, dim3((unsigned)rows), dim3(small ? 256u : few ? 1024u : 512u), 0, ctx->stream, x, delta, gamma, eps, (int)hidden,
                                 row0, row_step, x_out, out));
        DEC_EPILOGUE(ctx, name);
    }
    auto pick = [&](auto form) {
        constexpr int F = decltype(form)::value;
        return small ? norm_form_kernel<F, 256> : norm_form_kernel<F, 1024>;
    };
    auto kern = out.form == ACT_BF16     ? pick(std::integral_constant<int, ACT_BF16>())
                : out.form == ACT_DIGITS ? pick(std::integral_constant<int, ACT_DIGITS>())
                : out.form == ACT_TERMS  ? pick(std::integral_constant<int, ACT_TERMS>())
                                         : pick(std::integral_constant<int, ACT_F32>());
    YSCV_CUDA_TRY(launch_pdl(kern, dim3((unsigned)out.slots()), dim3(small ? 256u : 1024u), 0, ctx->stream, x, delta, parts, pitch, gamma, eps,
                             (int)hidden, row0, row_step, x_out, out));
    DEC_EPILOGUE(ctx, name);
}
}  // namespace yscv

template <bool ACT>
static int add_rms_norm_impl(yscv_cuda_ctx *ctx, const float *x, const float *delta, const float *gamma, float eps,
                             size_t rows, size_t hidden, float *x_out, void *normed) {
    if (rows == 0) return YSCV_CUDA_OK;
    const uintptr_t ptrs = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(gamma) |
                           reinterpret_cast<uintptr_t>(x_out) | reinterpret_cast<uintptr_t>(normed);
    if (hidden % 8 == 0 && hidden <= 8192 && (ptrs & 15) == 0)
        return norm_form(ctx, x, delta, 1, 0, gamma, eps, rows, 0, 1, hidden, x_out, act_out(ACT ? ACT_BF16 : ACT_F32, rows, hidden, normed), false);
    // eight elements per thread: 256 threads are enough up to 2048, 1024 up to 8192; sixteen up to 16384
    const unsigned threads = hidden <= 2048 ? 256u : 1024u;
    auto kern = hidden <= 8192 ? add_rms_norm_kernel<ACT, 8> : hidden <= 16384 ? add_rms_norm_kernel<ACT, 16> : add_rms_norm_long_kernel<ACT>;
    YSCV_CUDA_TRY(launch_pdl(kern, dim3((unsigned)rows), dim3(threads), 0, ctx->stream, x, delta, gamma, eps, (int)hidden, x_out, normed));
    DEC_EPILOGUE(ctx, ACT ? "add_rms_norm(bf16 activations out)" : "add_rms_norm");
}

extern "C" {

int yscv_cuda_add_rms_norm_dev(yscv_cuda_ctx *ctx, const float *d_x, const float *d_delta,
                               const float *d_gamma, float eps, size_t rows, size_t hidden,
                               float *d_x_out, float *d_normed) {
    DEC_PROLOGUE(ctx);
    if (!d_x || !d_gamma || !d_normed) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    return add_rms_norm_impl<false>(ctx, d_x, d_delta, d_gamma, eps, rows, hidden, d_x_out, d_normed);
}

}  // extern "C"

namespace yscv {
template <typename KV>
int rope_append_form(yscv_cuda_ctx *ctx, const float *qkv, int parts, size_t pitch, float *q_out, size_t q_out_stride, size_t batch,
                     size_t seq, size_t n_q, size_t n_kv, size_t d_head, float theta, const int32_t *d_pos, KV *kcache, KV *vcache,
                     float *kscale, float *vscale, size_t max_seq) {
    const size_t smem = (d_head + (sizeof(KV) == 1 ? n_kv * d_head : 0)) * sizeof(float);
    if (smem > 48 * 1024)
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "RoPE tables for d_head=%zu, n_kv=%zu do not fit shared memory", d_head, n_kv);
    const uintptr_t ptrs = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(kcache) |
                           reinterpret_cast<uintptr_t>(vcache);
    const bool vec = d_head % 8 == 0 && (ptrs & 15) == 0 && pitch % 4 == 0 && q_out_stride % 4 == 0;
    const size_t q_items = n_q * (d_head / 2) / (vec ? 4 : 1);
    const dim3 grid((unsigned)(batch * seq), (unsigned)(2 + (q_items + ROPE_ITEMS - 1) / ROPE_ITEMS));
    auto kern = parts > 1 ? (vec ? rope_kv_append_kernel<KV, 4, true> : rope_kv_append_kernel<KV, 1, true>)
                          : (vec ? rope_kv_append_kernel<KV, 4, false> : rope_kv_append_kernel<KV, 1, false>);
    YSCV_CUDA_TRY(launch_pdl(kern, grid, dim3(ROPE_THREADS), smem, ctx->stream, qkv, parts, pitch, q_out, (int)q_out_stride, (int)seq,
                             (int)n_q, (int)n_kv, (int)d_head, theta, d_pos, kcache, vcache, kscale, vscale, (int)max_seq, ctx->d_status));
    DEC_EPILOGUE(ctx, sizeof(KV) == 1 ? "rope_kv_append(int8 cache)" : "rope_kv_append");
}
template int rope_append_form<float>(yscv_cuda_ctx *, const float *, int, size_t, float *, size_t, size_t, size_t, size_t, size_t, size_t,
                                     float, const int32_t *, float *, float *, float *, float *, size_t);
template int rope_append_form<int8_t>(yscv_cuda_ctx *, const float *, int, size_t, float *, size_t, size_t, size_t, size_t, size_t, size_t,
                                      float, const int32_t *, int8_t *, int8_t *, float *, float *, size_t);
}  // namespace yscv

template <typename KV>
static int rope_kv_append_impl(yscv_cuda_ctx *ctx, float *d_qkv, size_t batch, size_t seq, size_t n_q,
                               size_t n_kv, size_t d_head, float theta, const int32_t *d_pos,
                               KV *d_kcache, KV *d_vcache, float *d_kscale, float *d_vscale,
                               size_t max_seq) {
    DEC_PROLOGUE(ctx);
    if (!d_qkv || !d_pos || !d_kcache || !d_vcache) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (sizeof(KV) == 1 && (!d_kscale || !d_vscale)) return fail(YSCV_CUDA_ERR_BAD_ARG, "null scale table");
    if (d_head == 0 || d_head % 2 != 0) return fail(YSCV_CUDA_ERR_BAD_ARG, "d_head must be even for RoPE");
    if (n_kv == 0 || max_seq == 0) return fail(YSCV_CUDA_ERR_BAD_ARG, "n_kv and max_seq must be positive");
    if (batch * seq == 0) return YSCV_CUDA_OK;
    return rope_append_form(ctx, d_qkv, 1, 0, d_qkv, (n_q + 2 * n_kv) * d_head, batch, seq, n_q, n_kv, d_head, theta, d_pos, d_kcache, d_vcache,
                            d_kscale, d_vscale, max_seq);
}

extern "C" {

int yscv_cuda_rope_kv_append_dev(yscv_cuda_ctx *ctx, float *d_qkv, size_t batch, size_t seq, size_t n_q,
                                 size_t n_kv, size_t d_head, float theta, const int32_t *d_pos,
                                 float *d_kcache, float *d_vcache, size_t max_seq) {
    return rope_kv_append_impl<float>(ctx, d_qkv, batch, seq, n_q, n_kv, d_head, theta, d_pos, d_kcache, d_vcache,
                                      nullptr, nullptr, max_seq);
}

int yscv_cuda_rope_kv_append_i8_dev(yscv_cuda_ctx *ctx, float *d_qkv, size_t batch, size_t seq, size_t n_q,
                                    size_t n_kv, size_t d_head, float theta, const int32_t *d_pos,
                                    int8_t *d_kcache, float *d_kscale, int8_t *d_vcache, float *d_vscale,
                                    size_t max_seq) {
    return rope_kv_append_impl<int8_t>(ctx, d_qkv, batch, seq, n_q, n_kv, d_head, theta, d_pos, d_kcache, d_vcache,
                                       d_kscale, d_vscale, max_seq);
}

}  // extern "C"

namespace yscv {
static bool decode_attention(size_t seq_q, int causal, size_t max_seq) { return seq_q == 1 && causal && max_seq > 128; }
bool gqa_attention_writes(int form, size_t seq_q, size_t d_head, size_t max_seq) {
    return (form == ACT_BF16 || (form == ACT_DIGITS && d_head % 32 == 0)) && decode_attention(seq_q, 1, max_seq);
}

// Merge of the splits, in the form of `out`
template <int CH, int PRE, int BLOCKS>
static int launch_combine(yscv_cuda_ctx *ctx, const float *part, int n_splits, size_t n_q, size_t d_head, size_t max_seq, const int32_t *d_pos,
                          int want, const ActOut &out) {
    auto kern = out.form == ACT_BF16     ? attention_combine_kernel<CH, PRE, BLOCKS, ACT_BF16>
                : out.form == ACT_DIGITS ? attention_combine_kernel<CH, PRE, BLOCKS, ACT_DIGITS>
                                         : attention_combine_kernel<CH, PRE, BLOCKS, ACT_F32>;
    YSCV_CUDA_TRY(launch_pdl(kern, dim3((unsigned)n_q, (unsigned)out.slots()), dim3(128), 0, ctx->stream, part, n_splits, (int)d_head, (int)max_seq,
                             d_pos, want, out));
    return YSCV_CUDA_OK;
}

template <typename KV>
int gqa_attention_form(yscv_cuda_ctx *ctx, const float *d_q, size_t q_stride, size_t batch, size_t seq_q, size_t n_q, size_t n_kv,
                       size_t d_head, const KV *d_kcache, const KV *d_vcache, const float *d_kscale, const float *d_vscale,
                       size_t max_seq, const int32_t *d_pos, int causal, const ActOut &out) {
    float *d_out = static_cast<float *>(out.ptr);   // (ACT_F32 everywhere but behind the merge)
    if (decode_attention(seq_q, causal, max_seq)) {
        // decode over a long cache: split the keys across blocks, then merge
        if (d_head % 16 != 0 || d_head > 128)
            return fail(YSCV_CUDA_ERR_UNSUPPORTED, "d_head %zu not supported by the decode attention", d_head);
        // key and value rows are read with 128-bit loads
        if (((reinterpret_cast<uintptr_t>(d_kcache) | reinterpret_cast<uintptr_t>(d_vcache)) & 15) != 0)
            return fail(YSCV_CUDA_ERR_UNSUPPORTED, "the key and value caches must be 16-byte aligned");
        const int chunk = sizeof(KV) == 4 && d_head > 64 ? 64 : 128;   // (what fits shared memory twice)
        const int n_splits = (int)((max_seq + chunk - 1) / chunk);
        const int want = (2 * ctx->sm_count + (int)(batch * n_kv) - 1) / (int)(batch * n_kv);
        const size_t need = batch * n_q * (size_t)n_splits * (d_head + 2) * sizeof(float);
        int rc = ctx->scratch_attn.reserve(need, ctx->stream);
        if (rc) return rc;
        float *part = reinterpret_cast<float *>(ctx->scratch_attn.ptr);
        // one block per (key chunk, KV head, sequence): it serves every query head of the group
        dim3 grid((unsigned)n_splits, (unsigned)n_kv, (unsigned)batch);
        if constexpr (sizeof(KV) == 1) {
            // int8 caches with head sizes of 64 or 128: both contractions on the tensor cores
            if ((d_head == 64 || d_head == 128) && ctx->attn_tensor_cores) {
                const size_t tc_smem = 2 * 128 * d_head + 8 * (128 + 4) * sizeof(float) +
                                       2 * 8 * (128 + 8) * sizeof(uint16_t);
                auto kern = d_head == 128 ? gqa_decode_split_tc_kernel<128> : gqa_decode_split_tc_kernel<64>;
                YSCV_CUDA_TRY(launch_pdl(kern, dim3(grid), dim3(128), tc_smem, ctx->stream, d_q, (int)q_stride, (int)n_q, (int)n_kv,
                                         reinterpret_cast<const int8_t *>(d_kcache), reinterpret_cast<const int8_t *>(d_vcache),
                                         d_kscale, d_vscale, (int)max_seq, d_pos, want, part));
                YSCV_CUDA_TRY(cudaGetLastError());
                ctx->launches++;
                if ((rc = launch_combine<128, 8, 16>(ctx, part, n_splits, n_q, d_head, max_seq, d_pos, want, out))) return rc;
                DEC_EPILOGUE(ctx, "gqa_attention(split-k,int8 cache,mma)");
            }
        }
        auto kern = d_head == 64 ? gqa_decode_split_kernel<KV, 128, 64> : gqa_decode_split_kernel<KV, 128, 0>;
        size_t split_smem = dec_smem<KV, 128>((int)d_head);
        if constexpr (sizeof(KV) == 4) {
            if (chunk == 64) {
                kern = d_head == 128 ? gqa_decode_split_kernel<KV, 64, 128> : gqa_decode_split_kernel<KV, 64, 0>;
                split_smem = dec_smem<KV, 64>((int)d_head);
            }
        }
        if ((rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kern), ctx->device, 80 * 1024))) return rc;
        YSCV_CUDA_TRY(launch_pdl(kern, dim3(grid), dim3(DEC_THREADS), split_smem, ctx->stream, d_q, (int)q_stride, (int)n_q, (int)n_kv,
                                 (int)d_head, d_kcache, d_vcache, d_kscale, d_vscale, (int)max_seq, d_pos, want, part));
        YSCV_CUDA_TRY(cudaGetLastError());
        ctx->launches++;
        rc = sizeof(KV) == 1 ? launch_combine<128, 8, 16>(ctx, part, n_splits, n_q, d_head, max_seq, d_pos, want, out)
             : chunk == 64   ? launch_combine<64, 16, 10>(ctx, part, n_splits, n_q, d_head, max_seq, d_pos, want, out)
                             : launch_combine<128, 16, 10>(ctx, part, n_splits, n_q, d_head, max_seq, d_pos, want, out);
        if (rc) return rc;
        DEC_EPILOGUE(ctx, sizeof(KV) == 1 ? "gqa_attention(split-k,int8 cache)" : "gqa_attention(split-k)");
    }
    // a prompt pass: tiles of 128 (position, head) pairs on the tensor cores
    const size_t group = n_q / n_kv;
    const uintptr_t vec_ptrs = reinterpret_cast<uintptr_t>(d_kcache) | reinterpret_cast<uintptr_t>(d_vcache) | reinterpret_cast<uintptr_t>(d_out);
    if (seq_q >= 16 && (d_head == 64 || d_head == 128) && group <= 128 && (vec_ptrs & 15) == 0) {
        const int rc = gqa_prefill_tc<KV>(ctx, d_q, q_stride, batch, seq_q, n_q, n_kv, d_head, d_kcache, d_vcache, d_kscale, d_vscale,
                                          max_seq, d_pos, causal, d_out);
        if (rc) return rc;
        ctx->last_kernel = sizeof(KV) == 1 ? "gqa_attention(prompt tiles,tcgen05,int8 cache)" : "gqa_attention(prompt tiles,tcgen05)";
        return YSCV_CUDA_OK;
    }
    const size_t smem = (max_seq + d_head) * sizeof(float);
    if (smem > 200 * 1024) return fail(YSCV_CUDA_ERR_UNSUPPORTED, "max_seq %zu too long for the attention kernel", max_seq);
    if (smem > 48 * 1024) {
        int arc = ensure_dynamic_smem(reinterpret_cast<const void *>(gqa_attention_kernel<KV>), ctx->device, 200 * 1024);
        if (arc) return arc;
    }
    dim3 grid((unsigned)seq_q, (unsigned)n_q, (unsigned)batch);
    YSCV_CUDA_TRY(launch_pdl(gqa_attention_kernel<KV>, dim3(grid), dim3(128), smem, ctx->stream, d_q, (int)q_stride, (int)seq_q,
                             (int)n_q, (int)n_kv, (int)d_head, d_kcache, d_vcache, d_kscale, d_vscale, (int)max_seq,
                             d_pos, causal, d_out));
    DEC_EPILOGUE(ctx, sizeof(KV) == 1 ? "gqa_attention(int8 cache)" : "gqa_attention");
}
template int gqa_attention_form<float>(yscv_cuda_ctx *, const float *, size_t, size_t, size_t, size_t, size_t, size_t, const float *,
                                       const float *, const float *, const float *, size_t, const int32_t *, int, const ActOut &);
template int gqa_attention_form<int8_t>(yscv_cuda_ctx *, const float *, size_t, size_t, size_t, size_t, size_t, size_t, const int8_t *,
                                        const int8_t *, const float *, const float *, size_t, const int32_t *, int, const ActOut &);
}  // namespace yscv

template <typename KV>
static int gqa_attention_impl(yscv_cuda_ctx *ctx, const float *d_q, size_t q_stride, size_t batch,
                              size_t seq_q, size_t n_q, size_t n_kv, size_t d_head, const KV *d_kcache,
                              const KV *d_vcache, const float *d_kscale, const float *d_vscale,
                              size_t max_seq, const int32_t *d_pos, int causal, float *d_out) {
    DEC_PROLOGUE(ctx);
    if (!d_q || !d_kcache || !d_vcache || !d_pos || !d_out) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (sizeof(KV) == 1 && (!d_kscale || !d_vscale)) return fail(YSCV_CUDA_ERR_BAD_ARG, "null scale table");
    if (n_kv == 0 || n_q % n_kv != 0) return fail(YSCV_CUDA_ERR_BAD_ARG, "n_q must be a multiple of n_kv");
    if (batch * seq_q == 0) return YSCV_CUDA_OK;
    return gqa_attention_form(ctx, d_q, q_stride, batch, seq_q, n_q, n_kv, d_head, d_kcache, d_vcache, d_kscale, d_vscale, max_seq, d_pos,
                              causal, act_out(ACT_F32, batch * seq_q, n_q * d_head, d_out));
}

extern "C" {

int yscv_cuda_gqa_attention_dev(yscv_cuda_ctx *ctx, const float *d_q, size_t q_stride, size_t batch,
                                size_t seq_q, size_t n_q, size_t n_kv, size_t d_head,
                                const float *d_kcache, const float *d_vcache, size_t max_seq,
                                const int32_t *d_pos, int causal, float *d_out) {
    return gqa_attention_impl<float>(ctx, d_q, q_stride, batch, seq_q, n_q, n_kv, d_head, d_kcache, d_vcache, nullptr,
                                     nullptr, max_seq, d_pos, causal, d_out);
}

int yscv_cuda_gqa_attention_i8_dev(yscv_cuda_ctx *ctx, const float *d_q, size_t q_stride, size_t batch,
                                   size_t seq_q, size_t n_q, size_t n_kv, size_t d_head,
                                   const int8_t *d_kcache, const float *d_kscale, const int8_t *d_vcache,
                                   const float *d_vscale, size_t max_seq, const int32_t *d_pos, int causal,
                                   float *d_out) {
    return gqa_attention_impl<int8_t>(ctx, d_q, q_stride, batch, seq_q, n_q, n_kv, d_head, d_kcache, d_vcache, d_kscale,
                                      d_vscale, max_seq, d_pos, causal, d_out);
}

}  // extern "C"

namespace yscv {
// inter % 8 == 0, operands (and `pitch` floats) 16-byte aligned
int swiglu_form(yscv_cuda_ctx *ctx, const float *gate_up, int parts, size_t pitch, size_t rows, size_t inter, const ActOut &out, bool between) {
    const size_t visit = out.slots();
    const dim3 grid((unsigned)((inter / 8 + 255) / 256), (unsigned)(visit < 32768 ? visit : 32768));
    const char *name = form_name(out.form, "swiglu", "swiglu(bf16 activations out)", "swiglu(digit planes out)", "swiglu(fp16 terms out)");
    if (parts == 1 && (out.form == ACT_F32 || out.form == ACT_BF16) && !(between && rows <= NORM_FEW * ctx->sm_count)) {
        auto plain = out.form == ACT_BF16 ? swiglu_kernel<true> : swiglu_kernel<false>;
        YSCV_CUDA_TRY(launch_pdl(plain, grid, dim3(256), 0, ctx->stream, gate_up, out.ptr, (int)rows, (int)inter));
        DEC_EPILOGUE(ctx, name);
    }
    auto kern = out.form == ACT_BF16     ? swiglu_form_kernel<ACT_BF16>
                : out.form == ACT_DIGITS ? swiglu_form_kernel<ACT_DIGITS>
                : out.form == ACT_TERMS  ? swiglu_form_kernel<ACT_TERMS>
                                         : swiglu_form_kernel<ACT_F32>;
    YSCV_CUDA_TRY(launch_pdl(kern, grid, dim3(256), 0, ctx->stream, gate_up, parts, pitch, (int)visit, (int)inter, out));
    DEC_EPILOGUE(ctx, name);
}
}  // namespace yscv

template <bool ACT>
static int swiglu_impl(yscv_cuda_ctx *ctx, const float *gate_up, size_t rows, size_t inter, void *out) {
    if (rows * inter == 0) return YSCV_CUDA_OK;
    if (inter % 8 == 0 && ((reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
        return swiglu_form(ctx, gate_up, 1, 0, rows, inter, act_out(ACT ? ACT_BF16 : ACT_F32, rows, inter, out), false);
    } else {
        const size_t total = rows * (inter / (ACT ? 8 : 1));
        const unsigned blocks = (unsigned)((total + 255) / 256 < 65535 ? (total + 255) / 256 : 65535);
        YSCV_CUDA_TRY(launch_pdl(swiglu_any_kernel<ACT>, dim3(blocks), dim3(256), 0, ctx->stream, gate_up, out, rows, (int)inter));
    }
    DEC_EPILOGUE(ctx, ACT ? "swiglu(bf16 activations out)" : "swiglu");
}

extern "C" {

int yscv_cuda_swiglu_dev(yscv_cuda_ctx *ctx, const float *d_gate_up, size_t rows, size_t inter,
                         float *d_out) {
    DEC_PROLOGUE(ctx);
    if (!d_gate_up || !d_out) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    return swiglu_impl<false>(ctx, d_gate_up, rows, inter, d_out);
}

int yscv_cuda_add_rms_norm_act_dev(yscv_cuda_ctx *ctx, const float *d_x, const float *d_delta, const float *d_gamma,
                                   float eps, size_t rows, size_t hidden, float *d_x_out, void *d_normed_act) {
    DEC_PROLOGUE(ctx);
    if (!d_x || !d_gamma || !d_normed_act) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (hidden % 8 != 0 || (reinterpret_cast<uintptr_t>(d_normed_act) & 15))
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "hidden must be a multiple of 8 and the activation buffer 16-byte aligned");
    return add_rms_norm_impl<true>(ctx, d_x, d_delta, d_gamma, eps, rows, hidden, d_x_out, d_normed_act);
}

int yscv_cuda_swiglu_act_dev(yscv_cuda_ctx *ctx, const float *d_gate_up, size_t rows, size_t inter, void *d_out_act) {
    DEC_PROLOGUE(ctx);
    if (!d_gate_up || !d_out_act) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (inter % 8 != 0 || (reinterpret_cast<uintptr_t>(d_out_act) & 15))
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "inter must be a multiple of 8 and the activation buffer 16-byte aligned");
    return swiglu_impl<true>(ctx, d_gate_up, rows, inter, d_out_act);
}

int yscv_cuda_f32_matmul_dev(yscv_cuda_ctx *ctx, const float *d_w, const float *d_x, size_t m, size_t n,
                             size_t k, float *d_out) {
    DEC_PROLOGUE(ctx);
    if (!d_w || !d_x || !d_out) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (k % 4 != 0) return fail(YSCV_CUDA_ERR_UNSUPPORTED, "k must be a multiple of 4");
    if ((reinterpret_cast<uintptr_t>(d_w) | reinterpret_cast<uintptr_t>(d_x)) & 15)
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "weights and activations must be 16-byte aligned");
    if (m * n == 0) return YSCV_CUDA_OK;
    if (m > 8 && ctx->f32_tensor_cores && f32_gemm_tc_supported(d_w, d_x, m, n, k)) {
        // wide batch: three TF32 products per fp32 product on the tensor cores, weights read once
        int rc = ctx->scratch.reserve(f32_gemm_tc_scratch_bytes(m, k), ctx->stream);
        if (rc) return rc;
        rc = f32_gemm_tc(ctx, d_w, d_x, m, n, k, d_out, ctx->scratch.ptr);
        if (rc) return rc;
        ctx->last_kernel = "f32_matmul(tcgen05,3xtf32)";
        return YSCV_CUDA_OK;
    }
    if (m > 8) {
        // wide batch without the tensor-core form (k not a multiple of 32): tiled SGEMM, the weights
        // cross HBM once per 64 activation rows
        dim3 grid((unsigned)((n + FM_BN - 1) / FM_BN), (unsigned)((m + FM_BM - 1) / FM_BM));
        YSCV_CUDA_TRY(launch_pdl(f32_matmul_tiled_kernel, grid, dim3(256), 0, ctx->stream, d_w, d_x, d_out, (int)m, (int)n, (int)k));
        YSCV_CUDA_TRY(cudaGetLastError());
        ctx->launches++;
        ctx->last_kernel = "f32_matmul(tiled)";
        return YSCV_CUDA_OK;
    }
    if (n < (m <= 4 ? 4096u : 2500u)) {
        const unsigned blocks = (unsigned)((n + 7) / 8);
        for (size_t m0 = 0; m0 < m; m0 += 4) {
            YSCV_CUDA_TRY(launch_pdl(f32_matmul_rows_kernel<4>, dim3(blocks), dim3(256), 0, ctx->stream, d_w, d_x, d_out, (int)m0, (int)m, (int)n, (int)k));
            YSCV_CUDA_TRY(cudaGetLastError());
            ctx->launches++;
        }
        ctx->last_kernel = "f32_matmul";
        return YSCV_CUDA_OK;
    }
    // one pass over the weights: rows per warp and unroll with enough loads in flight for the registers that m takes
    auto kern = m == 1 ? f32_matmul_kernel<1, 2, 4> : m == 2 ? f32_matmul_kernel<2, 2, 4> : m <= 4 ? f32_matmul_kernel<4, 4, 2> : f32_matmul_kernel<8, 4, 1>;
    const size_t rows = m <= 2 ? 2 : 4, need = (n + 8 * rows - 1) / (8 * rows), most = (size_t)16 * ctx->sm_count;
    const unsigned blocks = (unsigned)(need < most ? need : most);
    YSCV_CUDA_TRY(launch_pdl(kern, dim3(blocks), dim3(256), 0, ctx->stream, d_w, d_x, d_out, (int)m, (int)n, (int)k));
    YSCV_CUDA_TRY(cudaGetLastError());
    ctx->launches++;
    ctx->last_kernel = "f32_matmul";
    return YSCV_CUDA_OK;
}

int yscv_cuda_argmax_last_dev(yscv_cuda_ctx *ctx, const float *d_logits, size_t rows, size_t vocab,
                              int32_t *d_out) {
    DEC_PROLOGUE(ctx);
    if (!d_logits || !d_out) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (rows == 0) return YSCV_CUDA_OK;
    if (vocab == 0) return fail(YSCV_CUDA_ERR_BAD_ARG, "empty vocabulary");
    if (vocab >= 8192) {
        const int nb = 64;
        int rc = ctx->scratch_attn.reserve(rows * nb * 8, ctx->stream);
        if (rc) return rc;
        float *pv = reinterpret_cast<float *>(ctx->scratch_attn.ptr);
        int32_t *pi = reinterpret_cast<int32_t *>(pv + rows * nb);
        YSCV_CUDA_TRY(launch_pdl(argmax_partial_kernel, dim3(dim3(nb, (unsigned)rows)), dim3(256), 0, ctx->stream, d_logits, (int)vocab, pv, pi));
        YSCV_CUDA_TRY(cudaGetLastError());
        ctx->launches++;
        YSCV_CUDA_TRY(launch_pdl(argmax_final_kernel, dim3((unsigned)rows), dim3(64), 0, ctx->stream, pv, pi, nb, d_out));
        DEC_EPILOGUE(ctx, "argmax_last(two-stage)");
    }
    YSCV_CUDA_TRY(launch_pdl(argmax_last_kernel, dim3((unsigned)rows), dim3(256), 0, ctx->stream, d_logits, (int)vocab, d_out));
    DEC_EPILOGUE(ctx, "argmax_last");
}

int yscv_cuda_advance_pos_dev(yscv_cuda_ctx *ctx, int32_t *d_pos, int by) {
    DEC_PROLOGUE(ctx);
    if (!d_pos) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    YSCV_CUDA_TRY(launch_pdl(advance_pos_kernel, dim3(1), dim3(1), 0, ctx->stream, d_pos, by));
    DEC_EPILOGUE(ctx, "advance_pos");
}

}  // extern "C"
