// Decode attention of the layer chain (decoder_layers.cu): RoPE of the new position's query and key, the cache append
// and grouped-query attention over the cache in one kernel, the result in the form the output projection takes. The
// arithmetic of rope_kv_append_kernel, gqa_decode_split_kernel and attention_combine_kernel (decoder_ops.cu; the
// reference's files are named there), with the splits of a sequence merged through distributed shared memory.
//
// A decode step of a server batch is bound by launches and by the latency chain inside each: three kernels of 1.8 to 3.4,
// 4.7 to 8.5 and 2.8 to 4.0 us for 8 to 32 sequences at 200 keys, whose bytes take 2. Here the cached rows, which only
// earlier steps wrote, are on their way before the matmul in front has finished, and a cluster of C CTAs per
// (sequence, KV head) shares its keys, so that no partial result goes through memory: 6 us for 8 sequences, 10 for 32.
// What is left are the phases' latencies and shared memory's bandwidth.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "tma.cuh"

namespace yscv {

constexpr int DF_THREADS = 256, DF_HB = 8;   // query heads of a group (at most)

constexpr int DF_CH = 64;                        // keys staged at a time: a thread per key and quarter of its dimensions
template <typename KV, int D> struct DFGeom {
    // bytes of a staged row; keys: two rows' quarters (64 bytes f32, 16 int8) fall on different banks
    static constexpr int KP = sizeof(KV) == 4 ? D * 4 + 64 : D + 16, VP = D * (int)sizeof(KV);
    static constexpr int KVB = DF_CH * (KP + VP) > 32 * 1024 ? DF_CH * (KP + VP) : 32 * 1024;   // keys, values; at the end partial sums
    static constexpr int FLOATS = DF_HB * D + DF_CH * DF_HB + D + 2 * D + DF_HB * D + 3 * DF_HB + 8 * DF_HB;
    static constexpr int SMEM = FLOATS * 4 + KVB;
};

__device__ __forceinline__ void df_put(uint32_t cluster_addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(cluster_addr), "f"(v) : "memory");
}
__device__ __forceinline__ void df_cp16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

struct DFParams {
    const float *qkv;          // rows [q | k | v], the sum of `parts` arrays `pitch` floats apart
    int parts;
    size_t pitch;
    void *kc, *vc;             // [batch][max_seq][n_kv][D]
    float *kscale, *vscale;    // int8: [batch][max_seq]
    const int32_t *pos;
    int n_q, n_kv, max_seq;
    float theta;
    int *status;
    ActOut out;
};

// grid (C, n_kv, rows of `out` with padding), cluster (C, 1, 1)
template <typename KV, int D, int FORM>
__global__ void __launch_bounds__(DF_THREADS, 3)
gqa_decode_fused_kernel(DFParams p) {
    using G = DFGeom<KV, D>;
    constexpr bool I8 = sizeof(KV) == 1;
    constexpr int CH = DF_CH, KP = G::KP, VP = G::VP, HALF = D / 2;
    constexpr int PIECES = D * (int)sizeof(KV) / 16;
    extern __shared__ __align__(16) unsigned char dsm[];
    float *const qs = reinterpret_cast<float *>(dsm);          // [HB][D] rotated queries
    float *const wts = qs + DF_HB * D;                         // [CH][HB] weights
    float *const rope = wts + CH * DF_HB;                      // [D/2] cos, [D/2] sin
    float *const fresh = rope + D;                             // the new position's key and value as the cache holds them
    float *const res = fresh + 2 * D;                          // [HB][D] weighted sums that this CTA merges
    float *const res_m = res + DF_HB * D, *const res_l = res_m + DF_HB, *const resc = res_l + DF_HB;
    float *const red = resc + DF_HB;                           // [8 warps][HB]
    unsigned char *const ks = reinterpret_cast<unsigned char *>(red + 8 * DF_HB), *const vs = ks + CH * KP;
    float *const psum = reinterpret_cast<float *>(ks);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = gridDim.x, rank = blockIdx.x, kv_h = blockIdx.y, b = blockIdx.z, grp = p.n_q / p.n_kv;
    if (FORM == ACT_DIGITS && b >= p.out.rows) {               // (the whole cluster)
        pdl_wait();
        pdl_trigger();
        for (int h = rank * 8 + warp; h < grp; h += C * 8) {
            const int k = (kv_h * grp + h) * D + (lane * 8 < D ? lane * 8 : 0);
            store_act_padding(p.out, b, k, lane * 8 < D);
        }
        return;
    }
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");   // waited for before the first store to a peer
    // ---- before the predecessor is done: the position and the cached rows are from earlier steps ----
    const int pos = *p.pos, limit = max(0, min(p.max_seq, pos + 1)), share = (limit + C - 1) / C;
    const bool in_range = pos >= 0 && pos < p.max_seq;
    const int k0 = min(limit, rank * share), k1 = min(limit, k0 + share);
    const bool has_new = in_range && pos >= k0 && pos < k1;    // the CTA of the last keys
    const size_t row_bytes = (size_t)p.n_kv * D * sizeof(KV), first = (((size_t)b * p.max_seq) * p.n_kv + kv_h) * D * sizeof(KV);
    unsigned char *const kb = static_cast<unsigned char *>(p.kc) + first, *const vb = static_cast<unsigned char *>(p.vc) + first;
    auto fetch = [&](uint32_t dst, int pitch, const unsigned char *src, int c0) {   // keys c0 .. of the share, not the new one
        const int n = min(CH, k1 - c0);
        for (int i = tid; i < n * PIECES; i += DF_THREADS) {
            const int row = i / PIECES, c = (i - row * PIECES) * 16;
            if (c0 + row != pos) df_cp16(dst + row * pitch + c, src + (size_t)(c0 + row) * row_bytes + c);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const uint32_t ks_a = smem_u32(ks), vs_a = smem_u32(vs);
    fetch(ks_a, KP, kb, k0);
    fetch(vs_a, VP, vb, k0);
    if (tid < HALF) {
        const float a = 1.0f / powf(p.theta, 2.0f * (float)tid / (float)D) * (float)pos;
        sincosf(a, &rope[HALF + tid], &rope[tid]);
    }
    __syncthreads();
    pdl_wait();
    pdl_trigger();

    // ---- queries, new key and value ----
    const float *const row = p.qkv + (size_t)b * (p.n_q + 2 * p.n_kv) * D;
    auto load = [&](int i) {   // every part's load in flight
        float4 y[INT4_MAX_PARTS];
#pragma unroll
        for (int t = 0; t < INT4_MAX_PARTS; ++t) y[t] = t < p.parts ? *reinterpret_cast<const float4 *>(row + t * p.pitch + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 x = y[0];
#pragma unroll
        for (int t = 1; t < INT4_MAX_PARTS; ++t)
            if (t < p.parts) { x.x += y[t].x; x.y += y[t].y; x.z += y[t].z; x.w += y[t].w; }
        return x;
    };
    // Half of four rotary pairs (i, i + D/2) of one head by two neighbouring lanes (`up`: the second half); each product
    // rounded, as the reference rounds it (rope.rs:24-117). All lanes of a warp call it together.
    auto rotate = [&](int head, int i, bool up, float *dst, bool on) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (on) x = load(head * D + i + (up ? HALF : 0));
        float y[4], m = 0.0f;
        const float *a = &x.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float o = __shfl_xor_sync(0xffffffffu, a[j], 1), cs = rope[i + j], sn = rope[HALF + i + j];
            y[j] = up ? __fadd_rn(__fmul_rn(o, sn), __fmul_rn(a[j], cs)) : __fsub_rn(__fmul_rn(a[j], cs), __fmul_rn(o, sn));
            m = fmaxf(m, fabsf(y[j]));
        }
        if (on) *reinterpret_cast<float4 *>(dst + i + (up ? HALF : 0)) = make_float4(y[0], y[1], y[2], y[3]);
        return on ? m : 0.0f;
    };
    constexpr int HV = HALF / 4;
    const int qh0 = kv_h * grp;
    // item = (head, four pairs, half); rounds are the same for all lanes
    auto rotate_heads = [&](int head0, int n, float *dst) {
        float m = 0.0f;
        for (int r = 0; r < n * HV * 2; r += DF_THREADS) {
            const int i = r + tid, h = min(i / (HV * 2), n - 1);
            m = fmaxf(m, rotate(head0 + h, (i >> 1) % HV * 4, i & 1, dst + h * D, i < n * HV * 2));
        }
        return m;
    };
    rotate_heads(qh0, grp, qs);
    for (int i = grp * D + tid; i < DF_HB * D; i += DF_THREADS) qs[i] = 0.0f;   // (heads past the group)
    if (!in_range && rank == 0 && kv_h == 0 && tid == 0) *p.status = YSCV_DEV_POS_OVERFLOW;
    float new_ks = 1.0f, new_vs = 1.0f;
    if (has_new) {
        if constexpr (I8) {
            // one scale per row of n_kv * D values: every KV head's CTA forms the whole row's maximum
            float *const tmp = reinterpret_cast<float *>(ks + G::KVB);     // [2][n_kv * D]
            float km = rotate_heads(p.n_q, p.n_kv, tmp), vm = 0.0f;
            for (int i = tid * 4; i < p.n_kv * D; i += DF_THREADS * 4) {
                const float4 v = load((p.n_q + p.n_kv) * D + i);
                *reinterpret_cast<float4 *>(tmp + p.n_kv * D + i) = v;
                vm = fmaxf(vm, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                km = fmaxf(km, __shfl_xor_sync(0xffffffffu, km, o));
                vm = fmaxf(vm, __shfl_xor_sync(0xffffffffu, vm, o));
            }
            if (lane == 0) { red[warp] = km; red[8 + warp] = vm; }
            __syncthreads();
#pragma unroll
            for (int w = 0; w < DF_THREADS / 32; ++w) { km = fmaxf(km, red[w]); vm = fmaxf(vm, red[8 + w]); }
            new_ks = km <= 1.1920929e-07f ? 1.0f : __fdiv_rn(km, 127.0f);
            new_vs = vm <= 1.1920929e-07f ? 1.0f : __fdiv_rn(vm, 127.0f);
            if (kv_h == 0 && tid == 0) {
                p.kscale[(size_t)b * p.max_seq + pos] = new_ks;
                p.vscale[(size_t)b * p.max_seq + pos] = new_vs;
            }
            if (tid < 2 * D) {
                const bool is_v = tid >= D;
                const int i = is_v ? tid - D : tid;
                const float x = __fmul_rn(tmp[(is_v ? p.n_kv * D : 0) + kv_h * D + i], __fdiv_rn(1.0f, is_v ? new_vs : new_ks));
                // NaN -> 0, as Rust's saturating float-to-int cast does
                const int8_t q = (x != x) ? (int8_t)0 : (int8_t)(int)fminf(fmaxf(roundf(x), -127.0f), 127.0f);
                ((is_v ? vb : kb) + (size_t)pos * row_bytes)[i] = (unsigned char)q;
                reinterpret_cast<int8_t *>(fresh)[tid] = q;
            }
        } else {
            if (warp == 0) {
                const int i = (lane >> 1) % HV * 4 + (lane & 1 ? HALF : 0);
                rotate(p.n_q + kv_h, (lane >> 1) % HV * 4, lane & 1, fresh, lane < 2 * HV);
                if (lane < 2 * HV)
                    *reinterpret_cast<float4 *>(reinterpret_cast<float *>(kb + (size_t)pos * row_bytes) + i) = *reinterpret_cast<const float4 *>(fresh + i);
            } else if (tid >= 32 && tid < 32 + D / 4) {
                const int i = (tid - 32) * 4;
                const float4 v = load((p.n_q + p.n_kv + kv_h) * D + i);
                *reinterpret_cast<float4 *>(fresh + D + i) = v;
                *reinterpret_cast<float4 *>(reinterpret_cast<float *>(vb + (size_t)pos * row_bytes) + i) = v;
            }
        }
    }
    __syncthreads();

    // ---- chunks of the share: scores, online softmax, weighted values in registers ----
    // Scores: thread = (key, quarter of the dimensions: 4 of every 16) for all eight heads, so that a key is read once;
    // the quarters' lanes then share the heads out, two each. Values: thread = (key group, 4 dims) for all heads. (With a
    // thread per key and two heads, keys read four times and weights one by one, shared memory held both back by half.)
    constexpr int QUADS = D / 4, KG = DF_THREADS / QUADS;
    const int vq = tid % QUADS, vg = tid / QUADS, key = tid >> 2, qt = tid & 3;
    const float scale = 1.0f / sqrtf((float)D);
    const float *const ksc = I8 ? p.kscale + (size_t)b * p.max_seq : nullptr, *const vsc = I8 ? p.vscale + (size_t)b * p.max_seq : nullptr;
    float acc[DF_HB][4];
#pragma unroll
    for (int h = 0; h < DF_HB; ++h) acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.0f;
    float run_m[2] = {-INFINITY, -INFINITY}, run_l[2] = {0.0f, 0.0f};   // of heads 2 qt, 2 qt + 1; exp-sums of this thread's keys
    for (int c0 = k0; c0 < k1; c0 += CH) {
        const int nk = min(CH, k1 - c0);
        const bool new_here = has_new && pos >= c0 && pos < c0 + CH;
        if (new_here) {   // the new row joins the staged ones
            if constexpr (I8) {
                if (tid < 2 * D / 4)
                    reinterpret_cast<int *>(tid < D / 4 ? ks + (pos - c0) * KP : vs + (pos - c0) * VP)[tid % (D / 4)] = reinterpret_cast<const int *>(fresh)[tid];
            } else if (tid < 2 * D / 4) {
                reinterpret_cast<float4 *>(tid < D / 4 ? ks + (pos - c0) * KP : vs + (pos - c0) * VP)[tid % (D / 4)] = reinterpret_cast<const float4 *>(fresh)[tid];
            }
        }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        float sc[2] = {-INFINITY, -INFINITY};
        if (warp * 8 < nk) {
            float dot[DF_HB];
#pragma unroll
            for (int h = 0; h < DF_HB; ++h) dot[h] = 0.0f;
            const unsigned char *kr = ks + key * KP + qt * 4 * (int)sizeof(KV);
            const float rs = I8 && key < nk ? (new_here && c0 + key == pos ? new_ks : ksc[c0 + key]) : 1.0f;
#pragma unroll
            for (int i = 0; i < D / 16; ++i) {
                float4 kv;
                if constexpr (I8) {
                    const int w = *reinterpret_cast<const int *>(kr + i * 16);
                    kv = make_float4(__fmul_rn((float)(int8_t)(w & 255), rs), __fmul_rn((float)(int8_t)((w >> 8) & 255), rs),
                                     __fmul_rn((float)(int8_t)((w >> 16) & 255), rs), __fmul_rn((float)(int8_t)((w >> 24) & 255), rs));
                } else {
                    kv = *reinterpret_cast<const float4 *>(kr + i * 64);
                }
#pragma unroll
                for (int h = 0; h < DF_HB; ++h) {
                    const float4 f = *reinterpret_cast<const float4 *>(qs + h * D + i * 16 + qt * 4);
                    dot[h] = fmaf(f.x, kv.x, dot[h]);
                    dot[h] = fmaf(f.y, kv.y, dot[h]);
                    dot[h] = fmaf(f.z, kv.z, dot[h]);
                    dot[h] = fmaf(f.w, kv.w, dot[h]);
                }
            }
            float four[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) four[j] = (qt & 2 ? dot[4 + j] : dot[j]) + __shfl_xor_sync(0xffffffffu, qt & 2 ? dot[j] : dot[4 + j], 2);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float d2 = (qt & 1 ? four[2 + j] : four[j]) + __shfl_xor_sync(0xffffffffu, qt & 1 ? four[j] : four[2 + j], 1);
                if (key < nk) sc[j] = d2 * scale;
            }
        }
        float mx[2] = {sc[0], sc[1]};
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1) {
            mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], o));
            mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], o));
        }
        if (lane < 4) *reinterpret_cast<float2 *>(red + warp * DF_HB + 2 * qt) = make_float2(mx[0], mx[1]);
        __syncthreads();
        const bool more = c0 + CH < k1;
        if (more) fetch(ks_a, KP, kb, c0 + CH);
        mx[0] = run_m[0];
        mx[1] = run_m[1];
#pragma unroll
        for (int w = 0; w < DF_THREADS / 32; ++w) {
            const float2 m = *reinterpret_cast<const float2 *>(red + w * DF_HB + 2 * qt);
            mx[0] = fmaxf(mx[0], m.x);
            mx[1] = fmaxf(mx[1], m.y);
        }
        float2 wt;
        float *const wo = &wt.x;
        const float fold = I8 && key < nk ? (new_here && c0 + key == pos ? new_vs : vsc[c0 + key]) : 1.0f;   // the value row's scale
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float ref = mx[j] == -INFINITY ? 0.0f : mx[j];   // -inf scores weigh nothing (and are no -inf + inf)
            const float keep = run_m[j] == -INFINITY ? 0.0f : expf(run_m[j] - ref), e = key < nk ? expf(sc[j] - ref) : 0.0f;
            run_l[j] = fmaf(run_l[j], keep, e);
            run_m[j] = mx[j];
            wo[j] = I8 ? e * fold : e;
            if (tid < 4) resc[2 * qt + j] = keep;
        }
        *reinterpret_cast<float2 *>(wts + key * DF_HB + 2 * qt) = wt;
        if (more) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        if (c0 > k0) {
#pragma unroll
            for (int h = 0; h < DF_HB; ++h) {
                const float f = resc[h];
                acc[h][0] *= f; acc[h][1] *= f; acc[h][2] *= f; acc[h][3] *= f;
            }
        }
#pragma unroll 2
        for (int j = vg; j < nk; j += KG) {
            float v4[4], w8[DF_HB];
            *reinterpret_cast<float4 *>(w8) = *reinterpret_cast<const float4 *>(wts + j * DF_HB);
            *reinterpret_cast<float4 *>(w8 + 4) = *reinterpret_cast<const float4 *>(wts + j * DF_HB + 4);
            if constexpr (I8) {
                const int w = *reinterpret_cast<const int *>(vs + j * VP + vq * 4);
                v4[0] = (float)(int8_t)(w & 255); v4[1] = (float)(int8_t)((w >> 8) & 255);
                v4[2] = (float)(int8_t)((w >> 16) & 255); v4[3] = (float)(int8_t)((w >> 24) & 255);
            } else {
                const float4 f = *reinterpret_cast<const float4 *>(vs + j * VP + vq * 16);
                v4[0] = f.x; v4[1] = f.y; v4[2] = f.z; v4[3] = f.w;
            }
#pragma unroll
            for (int h = 0; h < DF_HB; ++h) {
                acc[h][0] = fmaf(w8[h], v4[0], acc[h][0]);
                acc[h][1] = fmaf(w8[h], v4[1], acc[h][1]);
                acc[h][2] = fmaf(w8[h], v4[2], acc[h][2]);
                acc[h][3] = fmaf(w8[h], v4[3], acc[h][3]);
            }
        }
        __syncthreads();   // the values' place and the weights are used again
        if (more) fetch(vs_a, VP, vb, c0 + CH);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    // ---- the CTA's sums ----
    __syncthreads();   // (a CTA without keys: its queries' writes; cp.async of an empty chunk)
#pragma unroll
    for (int h = 0; h < DF_HB; ++h) *reinterpret_cast<float4 *>(psum + ((size_t)vg * DF_HB + h) * D + 4 * vq) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) {
        run_l[0] += __shfl_xor_sync(0xffffffffu, run_l[0], o);
        run_l[1] += __shfl_xor_sync(0xffffffffu, run_l[1], o);
    }
    if (lane < 4) *reinterpret_cast<float2 *>(red + warp * DF_HB + 2 * qt) = make_float2(run_l[0], run_l[1]);
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");   // (the peers run)
    // head h is merged by CTA h % C, which gets every CTA's part: [CTA][h / C][D] sums, [CTA][h / C] maxima and exp-sums
    const int lc = 31 - __clz(C), hpo = DF_HB >> lc;
    if (tid < 4) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int h = 2 * qt + j, at = rank * hpo + (h >> lc);
            float l = 0.0f;
#pragma unroll
            for (int w = 0; w < DF_THREADS / 32; ++w) l += red[w * DF_HB + h];
            df_put(map_to_cta(smem_u32(res_m + at), h & (C - 1)), run_m[j]);
            df_put(map_to_cta(smem_u32(res_l + at), h & (C - 1)), l);
        }
    }
    for (int i = tid; i < grp * D; i += DF_THREADS) {
        float v = 0.0f;
#pragma unroll
        for (int g = 0; g < KG; ++g) v += psum[g * DF_HB * D + i];
        const int h = i / D;
        df_put(map_to_cta(smem_u32(res + (rank * hpo + (h >> lc)) * D + i % D), h & (C - 1)), v);
    }
    cluster_sync_all();
    // ---- merge (the usual max-rescaling of a split softmax): warp = head, lanes (group of CTAs, eight values) ----
    constexpr int VL = D / 8, LG = 32 / VL;
    const int h = warp * C + rank;
    if (warp < hpo && h < grp) {
        const float m = lane < C ? res_m[lane * hpo + warp] : -INFINITY;
        float M = m;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        M = __shfl_sync(0xffffffffu, M, 0);
        const float w = m > -INFINITY ? expf(m - M) : 0.0f;
        float L = lane < C ? res_l[lane * hpo + warp] * w : 0.0f;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        L = __shfl_sync(0xffffffffu, L, 0);
        const float inv = L > 0.0f ? 1.0f / L : (L == L ? 0.0f : L);
        const int vl = lane % VL;
        float v[8] = {};
#pragma unroll
        for (int c0 = 0; c0 < 8; c0 += LG) {
            const int c = c0 + lane / VL;
            const float wc = __shfl_sync(0xffffffffu, w, c);
            if (c < C) {
                const float4 *src = reinterpret_cast<const float4 *>(res + (c * hpo + warp) * D + vl * 8);
                const float4 x = src[0], y = src[1];
                v[0] = fmaf(wc, x.x, v[0]); v[1] = fmaf(wc, x.y, v[1]); v[2] = fmaf(wc, x.z, v[2]); v[3] = fmaf(wc, x.w, v[3]);
                v[4] = fmaf(wc, y.x, v[4]); v[5] = fmaf(wc, y.y, v[5]); v[6] = fmaf(wc, y.z, v[6]); v[7] = fmaf(wc, y.w, v[7]);
            }
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) {
#pragma unroll
            for (int o = VL; o < 32; o <<= 1) v[t] += __shfl_xor_sync(0xffffffffu, v[t], o);
            v[t] *= inv;
        }
        store_act<FORM>(p.out, v, b, (qh0 + h) * D + vl * 8, lane < VL);
    }
}

// CTAs per (sequence, KV head): a power of two up to 8 that keeps the grid within two CTAs per SM. us per step, 1B shape, with
// 1 / 2 / 4 / 8: 8 sequences, 200 keys 1233 / 1072 / 994 / 977; 16, 300 keys 1569 / 1362 / 1267 / 1344; 32, 200 keys 1155 / 1012 /
// 1083 / 1199; 64, 50 keys 1089 / 1181 / 1296 / 1652
static int df_ctas(const yscv_cuda_ctx *ctx, size_t pairs) {
    int C = 1;
    while (C < 8 && pairs * C * 2 <= (size_t)2 * ctx->sm_count) C *= 2;
    return C;
}
// The longest cache that this kernel takes. A CTA walks its share of the keys chunk after chunk, where the three kernels spread long
// ones over the machine and read int8 rows on the tensor cores; the host knows the cache's length and not the position, so the line lies
// where a full cache is even. It depends on the CTAs that share a sequence's keys, on how much of the machine's two CTAs per
// SM the grid fills (the three kernels gain by what it leaves empty), and on the heads of a group (eight are computed whatever
// there are). us per layer of a step, full cache, this / three kernels (about 5000 points, 1 to 148 sequences, caches of 130 to 8192):
//   f32, 32 / 4 heads of 64: 2 sequences 600 keys 37.7 / 37.1, 1600 45.9 / 37.6; 8: 200 34.9 / 37.2, 1200 43.6 / 44.1, 2100 51.2 / 48.6; 12: 400 48.4 /
//   49.7, 1200 60.9 / 56.3; 16: 800 55.7 / 56.0; 24: 300 43.9 / 46.4, 600 53.2 / 50.6; 32: 600 53.9 / 54.0, 1200 73.0 / 65.5; 48: 200 49.9 / 49.6, 400
//   62.1 / 56.6; 64: 400 63.4 / 63.5. 16 / 16 heads of 64, 8 sequences: 200 34.9 / 35.0, 400 42.8 / 40.0.
//   f32, 64 / 8 heads of 128: 4: 400 57.2 / 55.1 (clusters of eight, 82 KB a CTA: a grid of more than 200 does not fit at once), 8192 190 / 148;
//   8: 8192 209 / 240; 9: 1200 116 / 100; 19: 400 77.8 / 78.7, 2100 211 / 164; 37: 2100 216 / 267; 40: 800 181 / 156; 64: 2100 389 / 425.
//   32 / 8: 16: 1600 114 / 117; 64: 600 143 / 142, 2100 376 / 345. 32 / 32, 8: 400 83.0 / 83.0, 2100 216 / 190.
//   int8: 32 / 4 heads of 64, 8: 300 35.9 / 35.8, 800 40.5 / 37.3; 32: 130 39.7 / 42.3, 300 46.2 / 44.2; 64 / 8 of 128, 2: 200 44.0 / 44.5, 600 50.5 / 44.6;
//   64: 130 80.1 / 70.3.
static size_t df_longest(const yscv_cuda_ctx *ctx, bool kv_int8, size_t pairs, size_t group, size_t d_head) {
    const size_t C = df_ctas(ctx, pairs), ctas = pairs * C, slots = (size_t)2 * ctx->sm_count, waves = (ctas + slots - 1) / slots;
    const size_t fill = 100 * ctas / (slots * waves);   // % of the slots of its waves
    if (kv_int8) {
        if (d_head == 128) return group == 1 ? 0 : C == 8 ? 200 : C == 4 ? 130 : 0;
        return C == 8 ? 300 : C == 4 ? 200 : C == 2 || (group >= 3 && waves == 1) ? 130 : 0;
    }
    if (d_head == 64) {
        const bool full = fill >= 80;
        if (group >= 4) return waves > 2 ? 0 : waves == 2 ? 400 : (C == 8 ? 600 : C == 4 ? 400 : C == 2 ? 300 : 200) * (full ? 2 : 1);
        if (waves > 1 || (C == 1 && group == 1)) return 0;
        return C == 8 ? (full ? 600 : 400) : C == 4 ? (full ? 400 : 200) : full ? 200 : 130;
    }
    if (C == 8) return ctas <= 64 ? 400 : ctas <= 128 ? 600 : ctas <= 200 ? (group >= 4 ? 1200 : 600) : 0;
    if (C == 4 && ctas > 256) return 200;
    if (waves > 2 || (waves == 2 && group < 4)) return 0;
    if (group >= 8) return fill >= 85 ? (size_t)-1 : fill >= 75 ? 2000 : waves == 2 ? 200 : fill >= 60 ? 600 : 400;
    if (group >= 4) return waves == 2 ? (fill >= 85 ? 600 : fill >= 75 ? 300 : 130) : fill >= 85 ? 1600 : fill >= 75 ? 800 : fill >= 60 ? 400 : 300;
    return fill >= 85 ? (group > 1 ? 600 : 200) : fill >= 75 ? 200 : 130;
}
bool gqa_decode_fused_wins(const yscv_cuda_ctx *ctx, int form, bool kv_int8, size_t batch, size_t n_q, size_t n_kv, size_t d_head, size_t max_seq) {
    if ((d_head != 64 && d_head != 128) || n_q / n_kv > DF_HB || n_kv * d_head > 4096 || n_kv > 65535 || batch > 65000 || form == ACT_TERMS) return false;
    return max_seq <= df_longest(ctx, kv_int8, batch * n_kv, n_q / n_kv, d_head);
}

template <typename KV>
int gqa_decode_fused(yscv_cuda_ctx *ctx, const float *qkv, int parts, size_t pitch, size_t batch, size_t n_q, size_t n_kv, size_t d_head,
                     float theta, const int32_t *d_pos, KV *kcache, KV *vcache, float *kscale, float *vscale, size_t max_seq, const ActOut &out) {
    if (parts > INT4_MAX_PARTS) return fail(YSCV_CUDA_ERR_BAD_ARG, "%d partial sums, at most %d", parts, INT4_MAX_PARTS);
    DFParams p = {qkv, parts, pitch, kcache, vcache, kscale, vscale, d_pos, (int)n_q, (int)n_kv, (int)max_seq, theta, ctx->d_status, out};
    auto pick = [&](auto dim) {
        constexpr int D = decltype(dim)::value;
        return out.form == ACT_BF16     ? gqa_decode_fused_kernel<KV, D, ACT_BF16>
               : out.form == ACT_DIGITS ? gqa_decode_fused_kernel<KV, D, ACT_DIGITS>
                                        : gqa_decode_fused_kernel<KV, D, ACT_F32>;
    };
    auto kern = d_head == 64 ? pick(std::integral_constant<int, 64>()) : pick(std::integral_constant<int, 128>());
    const size_t smem = (d_head == 64 ? DFGeom<KV, 64>::SMEM : DFGeom<KV, 128>::SMEM) + (sizeof(KV) == 1 ? 2 * n_kv * d_head * sizeof(float) : 0);
    int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kern), ctx->device, 100 * 1024);
    if (rc) return rc;
    const int C = df_ctas(ctx, batch * n_kv);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)C, (unsigned)n_kv, (unsigned)out.slots());
    cfg.blockDim = dim3(DF_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim = {(unsigned)C, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    YSCV_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
    ctx->launches++;
    ctx->last_kernel = sizeof(KV) == 1 ? "gqa_decode(rope,append,int8 cache)" : "gqa_decode(rope,append)";
    return YSCV_CUDA_OK;
}
template int gqa_decode_fused<float>(yscv_cuda_ctx *, const float *, int, size_t, size_t, size_t, size_t, size_t, float, const int32_t *, float *,
                                     float *, float *, float *, size_t, const ActOut &);
template int gqa_decode_fused<int8_t>(yscv_cuda_ctx *, const float *, int, size_t, size_t, size_t, size_t, size_t, float, const int32_t *, int8_t *,
                                      int8_t *, float *, float *, size_t, const ActOut &);

}  // namespace yscv
