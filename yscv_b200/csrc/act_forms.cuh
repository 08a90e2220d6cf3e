// The forms in which a packed-int4 matmul takes its activations, so that the operator in front of it can write
// them itself (the fusion of docs/int4-quant-pipeline-plan.md:45-51) instead of leaving a conversion pass between
// the two. Every writer holds eight consecutive values of a row per lane, a warp's lanes on consecutive eights.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "int4_digits.cuh"

namespace yscv {

enum ActForm : int {
    ACT_F32 = 0,      // fp32 rows
    ACT_BF16 = 1,     // bf16 rows, k order 0,4,1,5,2,6,3,7 of every group of 8 (17 rows and more)
    ACT_DIGITS = 2,   // digit planes (int4_digits.cuh)
    ACT_TERMS = 3,    // two fp16 terms per value and inverse scales per row and 256 k (int4_batch_gemm.cu)
};

struct ActOut {
    int form = ACT_F32;
    int rows = 0, k = 0;       // rows of the matmul, row length
    void *ptr = nullptr;
    float *inv = nullptr;      // ACT_TERMS: [256-k block][16]
    QuantLayout q = {};        // ACT_DIGITS
    // rows a writer visits: digit planes have padding rows, which are zero
    int slots() const { return form == ACT_DIGITS ? quant_slots(q) : rows; }
};

// Eight fp32 values -> bf16 in the order the packed-int4 GEMM consumes its activations: k = 0,4,1,5,2,6,3,7 of
// every group of 8 (what its nibble unpack produces), round to nearest even.
__device__ __forceinline__ uint4 pack_bf16_gemm_order(const float (&v)[8]) {
    const __nv_bfloat162 p[4] = {__floats2bfloat162_rn(v[0], v[4]), __floats2bfloat162_rn(v[1], v[5]),
                                 __floats2bfloat162_rn(v[2], v[6]), __floats2bfloat162_rn(v[3], v[7])};
    return make_uint4(*reinterpret_cast<const uint32_t *>(&p[0]), *reinterpret_cast<const uint32_t *>(&p[1]),
                      *reinterpret_cast<const uint32_t *>(&p[2]), *reinterpret_cast<const uint32_t *>(&p[3]));
}

// Eight values of row m from k on (k % 8 == 0) as fp16 terms [hi: 16 rows][K], [lo: 16 rows][K], k order as above,
// and the inverse scale of the 256-k block. A warp holds one block; lanes past the row's end pass valid = false.
__device__ __forceinline__ void store_terms(const float (&a)[8], __half *terms, float *inv, int K, int m, int k, bool valid) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = valid ? a[(i >> 1) | (i & 1) << 2] : 0.0f;
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    // power of two that brings the block's maximum into [2^13, 2^14) (2^126 at most), and its inverse. A block with
    // an infinity keeps its scale of 1 and its infinities, whose remainder is 0 (not inf - inf); what else it holds
    // only has to stay finite, since the row's sums no longer are.
    const uint32_t e = (__float_as_uint(mx) >> 23) & 255u;
    const bool inf = e == 255u;
    const uint32_t s = inf ? 127u : min(267u - e, 253u);
    const float up = __uint_as_float(s << 23);
    if (inf) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (fabsf(v[i]) < INFINITY) v[i] = fminf(fmaxf(v[i], -65504.0f), 65504.0f);
    }
    uint4 hi, lo;
    uint32_t *h = &hi.x, *l = &lo.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float x = v[2 * i] * up, y = v[2 * i + 1] * up;
        const __half2 hh = __floats2half2_rn(x, y);
        const float2 f = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(inf && f.x == x ? 0.0f : x - f.x, inf && f.y == y ? 0.0f : y - f.y);
        h[i] = *reinterpret_cast<const uint32_t *>(&hh);
        l[i] = *reinterpret_cast<const uint32_t *>(&ll);
    }
    if (valid) {
        *reinterpret_cast<uint4 *>(terms + (size_t)m * K + k) = hi;
        *reinterpret_cast<uint4 *>(terms + (size_t)(16 + m) * K + k) = lo;
        if (k % 256 == 0) inv[k / 256 * 16 + m] = __uint_as_float((254u - s) << 23);
    }
}

// Eight values of row m from k on, in the form of `o`. All lanes of the warp call it together.
template <int FORM>
__device__ __forceinline__ void store_act(const ActOut &o, const float (&v)[8], int m, int k, bool valid) {
    if constexpr (FORM == ACT_F32) {
        if (!valid) return;
        float4 *p = reinterpret_cast<float4 *>(static_cast<float *>(o.ptr) + (size_t)m * o.k + k);
        p[0] = make_float4(v[0], v[1], v[2], v[3]);
        p[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else if constexpr (FORM == ACT_BF16) {
        if (valid) *reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(o.ptr) + (size_t)m * o.k + k) = pack_bf16_gemm_order(v);
    } else if constexpr (FORM == ACT_DIGITS) {
        quantize_group_values(v, static_cast<unsigned char *>(o.ptr), o.q, k / 32, m, (k / 8) & 3, valid);
    } else {
        store_terms(v, static_cast<__half *>(o.ptr), o.inv, o.k, m, k, valid);
    }
}
// A padding row's eight values (digit planes only)
__device__ __forceinline__ void store_act_padding(const ActOut &o, int m, int k, bool valid) {
    quantize_group(nullptr, static_cast<unsigned char *>(o.ptr), o.q, k / 32, m, (k / 8) & 3, valid);
}

}  // namespace yscv
