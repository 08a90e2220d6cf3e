// fp32 x fp32 matmul for a wide decode batch (the fp32 LM head of the decoder,
// out[m][n] = sum_k x[m][k] * w[n][k], m > 8) on the 5th-generation tensor cores, keeping fp32
// accuracy: every operand is split into a TF32 part and a remainder,
//     x = x_hi + x_lo,   w = w_hi + w_lo,   x_hi = x with the low 13 mantissa bits cleared,
// and the product is accumulated in fp32 (TMEM) as w_hi*x_hi + w_hi*x_lo + w_lo*x_hi by
// tcgen05.mma.kind::tf32. The parts with cleared bits are exact TF32 values whatever the
// hardware does with the bits it does not use; the remainders keep 11 of their 13 significant
// bits: the relative error of a product is ~2^-21, that of the dropped w_lo*x_lo term 2^-22.
//
// Same orientation as the packed-int4 GEMMs: the weight rows are the MMA's M side (128 per tile half, one or
// two halves per CTA), the batch rows its N side (BT <= 128 per pass). A ring stage is 32 k: TMA brings the
// weight rows and the two activation tiles [BT][32] (x_hi, x_lo come from a small pre-pass over the
// activations). The thread that owns a weight row reads its 32 values, splits them in registers and writes
// both parts to TMEM (tcgen05.st), where the MMA reads its A operand. The weights are read from HBM once.
//
// What bounds it: the weights' HBM stream, with shared memory next. With the parts written back to shared
// memory a 16 KB weight block cost 128 bytes x 1088 cycles there (TMA 128, split 384, MMA operands 576), which
// held 128256 x 8192 at 64 rows at 1265 us (3.3 TB/s); through TMEM it is 576, or 512 with two halves sharing
// the activation tiles: 775 us (5.4 TB/s), at 32 rows 974 -> 644 us (the copy rate); 32000 x 2048 at 32 / 64 / 128
// rows 78 / 96 / 106 -> 59 / 64 / 95 us.
//
// The tensor core adds into its fp32 accumulator by truncation, so a long chain of accumulations
// drifts toward zero: one accumulator over K = 2048 (768 MMAs) came out with a relative error of
// 1.8e-5, over K = 8192 with 6e-5, ten to thirty times what fp32 FMAs leave. So an accumulator
// only ever collects one unit of 64 k (24 MMAs); the drain warps add it to fp32 registers
// with ordinary rounded adds while the MMAs fill the other buffer, and store once per tile. That
// bounds the drift by the chunk length, whatever K is (measured ~1e-6).
//
// Work split: the units (tile, 64 k) are numbered through and every CTA takes an equal contiguous range
// (501 tiles of 256 rows on 148 SMs would be 4 rounds for 3.4). The parts of a tile that several CTAs share go
// to a workspace as fp32 sums and a second kernel adds them in CTA order, so the result does not depend on
// timing. Persistent CTAs, all waits bounded.
#include "common.cuh"
#include "kernels.cuh"
#include "tma.cuh"

namespace yscv {

constexpr int FT_BM = 128;       // weight rows per tile half
constexpr int FT_BK = 32;        // k per ring stage: fp32 per 128-byte swizzle row
constexpr int FT_UNIT = 64;      // k per accumulator and unit of work: two stages
constexpr int FT_BT_MAX = 128;   // batch rows per pass (one tile half; 64 with two)
constexpr int FT_W_BYTES = FT_BM * FT_BK * 4;   // 16 KB
constexpr int FT_SLOTS = 4;      // A slots in TMEM: 32 columns of leading parts, 32 of remainders
constexpr int FT_MAX_STAGES = 8;
// warps 0..7 drain (their TMEM lanes are 32 * (warp % 4)), 8..15 split, 16 TMA producer, 17 (and 18) MMA issuers
constexpr int FT_SPLIT0 = 8, FT_PRODUCER = 16, FT_ISSUE0 = 17;
constexpr int FT_THREADS = 19 * 32;

struct FTParams {
    int M, N, K;
    int BT;                 // batch rows per pass (multiple of 16)
    int t_chunks;           // passes; tile = weight tile * t_chunks + pass
    int kb, units;          // units per tile, units in all
    int stages, stage_bytes;
    float *ws;              // [CTA][2: part with its tile's last unit, part without][NA][BT][128]; null: CTAs take whole tiles
};

__device__ __forceinline__ void ft_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void ft_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// K-major tile, 128-byte swizzle, rows 128 bytes apart, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t ft_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// A operand in TMEM
__device__ __forceinline__ void ft_mma_tf32(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void ft_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void ft_tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void ft_tmem_st(uint32_t taddr, const uint32_t (&r)[32]) {
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

__device__ __forceinline__ void ft_tmem_st(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};\n" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
        : "memory");
}

constexpr uint32_t FT_HI_MASK = 0xFFFFE000u;   // sign, exponent, 10 mantissa bits

// activations -> x_hi (low 13 mantissa bits cleared) and x_lo = x - x_hi (exact)
__global__ void __launch_bounds__(256) ft_split_act_kernel(const float4 *__restrict__ x, float4 *__restrict__ hi,
                                                           float4 *__restrict__ lo, size_t n4) {
    pdl_wait();
    pdl_trigger();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        const float4 v = x[i];
        float4 h;
        h.x = __uint_as_float(__float_as_uint(v.x) & FT_HI_MASK);
        h.y = __uint_as_float(__float_as_uint(v.y) & FT_HI_MASK);
        h.z = __uint_as_float(__float_as_uint(v.z) & FT_HI_MASK);
        h.w = __uint_as_float(__float_as_uint(v.w) & FT_HI_MASK);
        hi[i] = h;
        lo[i] = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
    }
}

// First unit of CTA c's range (of `grid` CTAs); without a workspace the ranges end where tiles do
__host__ __device__ inline int ft_first_unit(const FTParams &p, int c, int grid) {
    const int u = (int)((long long)c * p.units / grid);
    return p.ws ? u : (u + p.kb - 1) / p.kb * p.kb;
}
// One CTA's walk over its units, last one first: every call yields a tile and its range of k units.
struct FTWalk {
    int end, first, kb;
    __device__ FTWalk(const FTParams &p)
        : end(ft_first_unit(p, blockIdx.x + 1, gridDim.x)), first(ft_first_unit(p, blockIdx.x, gridDim.x)), kb(p.kb) {}
    __device__ bool next(int &tile, int &k0, int &k1) {
        if (end <= first) return false;
        tile = (end - 1) / kb;
        const int start = max(first, tile * kb);
        k0 = start - tile * kb;
        k1 = end - tile * kb;
        end = start;
        return true;
    }
};

// NA = 128-row halves per tile. Two share the activation tiles of a stage (with 64 batch rows as many bytes as
// a half's weights); their accumulators leave room for up to 64 batch rows.
template <int NA>
__global__ void __launch_bounds__(FT_THREADS, 1)
f32_gemm_tf32x3_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_xh,
                       const __grid_constant__ CUtensorMap tm_xl, float *__restrict__ out, FTParams p,
                       int *__restrict__ status) {
    constexpr int RING = FT_SLOTS / NA;          // A slots per half
    constexpr int ACC = FT_BT_MAX / NA;          // columns of an accumulator
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = smem_u32(smem);
    // stage: [NA][128 rows][128 B of weights] [x_hi: BT rows][128 B] [x_lo: BT rows][128 B]
    const int x_bytes = p.BT * 128;
    const uint32_t bars = base + (uint32_t)p.stages * p.stage_bytes;
    const uint32_t full = bars, empty = bars + 64, afull = bars + 128, mdone = bars + 160, tfull = bars + 192, tempty = bars + 208;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + (size_t)p.stages * p.stage_bytes + 224);

    if (tid == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(full + i * 8, 1);
            mbar_init(empty + i * 8, 8 + NA);   // the splitting warps have read the weights, the MMAs the activations
        }
        for (int i = 0; i < FT_SLOTS; ++i) {
            mbar_init(afull + i * 8, 8 / NA);
            mbar_init(mdone + i * 8, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(tfull + i * 8, NA);
            mbar_init(tempty + i * 8, 8);
        }
        mbar_fence_init();
    }
    if (warp == FT_ISSUE0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    ft_fence_before();
    __syncthreads();
    ft_fence_after();
    const uint32_t tmem = *tmem_slot;            // columns 0..255: accumulators [buffer][half], 256..511: A slots
    const uint32_t t_a = tmem + 256;
    // the activation parts come from the pre-pass, the output may still be read by a predecessor
    pdl_wait();
    pdl_trigger();

    FTWalk walk(p);
    const int stages_k = p.K / FT_BK;            // (odd: the last unit is one stage)
    int tile, k0, k1;
    bool alive = true;
    if (warp == FT_PRODUCER) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 0;
            while (alive && walk.next(tile, k0, k1)) {
                const int nt = tile / p.t_chunks, tc = tile - nt * p.t_chunks;
                for (int s = 2 * k0; s < min(2 * k1, stages_k); ++s) {
                    alive = mbar_wait(empty + st * 8, ph ^ 1u, status);
                    if (!alive) break;
                    const uint32_t dst = base + (uint32_t)st * p.stage_bytes, bar = full + st * 8;
                    mbar_expect_tx(bar, (uint32_t)(NA * FT_W_BYTES + 2 * x_bytes));
#pragma unroll
                    for (int a = 0; a < NA; ++a) tma_load_2d(dst + a * FT_W_BYTES, &tm_w, s * FT_BK, (nt * NA + a) * FT_BM, bar);
                    tma_load_2d(dst + NA * FT_W_BYTES, &tm_xh, s * FT_BK, tc * p.BT, bar);
                    tma_load_2d(dst + NA * FT_W_BYTES + x_bytes, &tm_xl, s * FT_BK, tc * p.BT, bar);
                    if (++st == p.stages) { st = 0; ph ^= 1u; }
                }
            }
            // a consumer gave up: no stage's copies may be in flight when the CTA leaves (bounded)
            if (!alive)
                for (int i = 0; i < p.stages; ++i) mbar_wait(full + i * 8, i < st ? ph : ph ^ 1u, nullptr);
        }
        __syncwarp();
    } else if (warp >= FT_ISSUE0 && warp < FT_ISSUE0 + NA) {
        // ---------------- MMA issuer of half a ----------------
        const int a = warp - FT_ISSUE0;
        // D fp32, A (TMEM) and B TF32, K-major, N = BT, M = 128
        const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(p.BT >> 3) << 17) | ((uint32_t)(FT_BM >> 4) << 24);
        int st = 0, ring = 0, buf = 0;
        uint32_t ph = 0, rph = 0, bph = 0;
        while (alive && walk.next(tile, k0, k1)) {
            for (int s = 2 * k0; s < min(2 * k1, stages_k); ++s) {
                const bool first = (s & 1) == 0, last = !first || s + 1 == stages_k;   // a unit's first stage starts an accumulator
                const int slot = a * RING + ring;
                alive = __all_sync(0xffffffffu, (!first || mbar_wait(tempty + buf * 8, bph ^ 1u, status)) &&
                                                    mbar_wait(full + st * 8, ph, status) && mbar_wait(afull + slot * 8, rph, status));
                if (!alive) break;
                ft_fence_after();
                if (elect_one()) {
                    const uint32_t acc = tmem + (buf * NA + a) * ACC, whi = t_a + slot * 64, wlo = whi + 32;
                    const uint64_t d_xhi = ft_desc_sw128(base + (uint32_t)st * p.stage_bytes + NA * FT_W_BYTES);
                    const uint64_t d_xlo = d_xhi + (uint64_t)(x_bytes >> 4);
#pragma unroll
                    for (int kk = 0; kk < FT_BK / 8; ++kk) {   // K = 8 per instruction: 8 columns of A, 32 bytes of B
                        ft_mma_tf32(acc, wlo + kk * 8, d_xhi + (uint64_t)(kk * 2), idesc, (!first || kk > 0) ? 1u : 0u);
                        ft_mma_tf32(acc, whi + kk * 8, d_xlo + (uint64_t)(kk * 2), idesc, 1u);
                        ft_mma_tf32(acc, whi + kk * 8, d_xhi + (uint64_t)(kk * 2), idesc, 1u);
                    }
                    ft_commit(empty + st * 8);
                    ft_commit(mdone + slot * 8);
                    if (last) ft_commit(tfull + buf * 8);
                }
                __syncwarp();
                if (++st == p.stages) { st = 0; ph ^= 1u; }
                if (++ring == RING) { ring = 0; rph ^= 1u; }
                if (last && ++buf == 2) { buf = 0; bph ^= 1u; }
            }
        }
    } else if (warp >= FT_SPLIT0 && warp < FT_PRODUCER) {
        // ---- split: thread = weight row r of a half. Two halves: group g of four warps takes half g; one:
        // every thread 16 of the 32 k (both groups visit every stage: a barrier whose phases a waiter skips
        // could not tell one round from the next but one) ----
        constexpr int CH = NA == 2 ? 8 : 4;          // 16-byte pieces per thread
        const int g = (warp - FT_SPLIT0) >> 2, r = (warp & 3) * 32 + lane;
        const int a = NA == 2 ? g : 0, c0 = NA == 2 ? 0 : g * CH;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        int st = 0, ring = 0;
        uint32_t ph = 0, rph = 0;
        while (alive && walk.next(tile, k0, k1)) {
            for (int s = 2 * k0; s < min(2 * k1, stages_k); ++s) {
                const int slot = a * RING + ring;
                alive = mbar_wait(full + st * 8, ph, status);
                if (!alive) break;
                const unsigned char *row = smem + (size_t)st * p.stage_bytes + a * FT_W_BYTES + r * 128;
                uint32_t hi[CH * 4], lo[CH * 4];
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    // 16-byte piece c of row r sits at piece c ^ (r & 7) (128-byte swizzle)
                    const uint4 v = *reinterpret_cast<const uint4 *>(row + (((c0 + c) ^ (r & 7)) << 4));
                    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        hi[c * 4 + j] = x[j] & FT_HI_MASK;
                        lo[c * 4 + j] = __float_as_uint(__uint_as_float(x[j]) - __uint_as_float(hi[c * 4 + j]));
                    }
                }
                alive = mbar_wait(mdone + slot * 8, rph ^ 1u, status);
                if (!alive) break;
                ft_fence_after();
                ft_tmem_st(t_a + slot * 64 + c0 * 4 + lane_base, hi);
                ft_tmem_st(t_a + slot * 64 + 32 + c0 * 4 + lane_base, lo);
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                ft_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(empty + st * 8);
                    mbar_arrive(afull + slot * 8);
                }
                if (++st == p.stages) { st = 0; ph ^= 1u; }
                if (++ring == RING) { ring = 0; rph ^= 1u; }
            }
        }
    } else if (warp < FT_SPLIT0) {
        // ---- drain: eight warps, TMEM lanes 32 * (warp % 4); two halves: warps 4..7 the second; one: columns 64.. ----
        const int a = NA == 2 ? warp >> 2 : 0, r = (warp & 3) * 32 + lane;
        const int col_base = NA == 2 ? 0 : (warp >> 2) * 64;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        int buf = 0;
        uint32_t bph = 0;
        while (alive && walk.next(tile, k0, k1)) {
            float acc[4][16];
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c][j] = 0.0f;
            for (int u = k0; u < k1; ++u) {
                alive = mbar_wait(tfull + buf * 8, bph, status);
                if (!alive) break;
                ft_fence_after();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (col_base + c * 16 < p.BT) {   // the same for the whole warp
                        uint32_t d[16];
                        ft_tmem_ld16(tmem + (buf * NA + a) * ACC + col_base + c * 16 + lane_base, d);
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c][j] += __uint_as_float(d[j]);
                    }
                }
                ft_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty + buf * 8);
                if (++buf == 2) { buf = 0; bph ^= 1u; }
            }
            if (!alive) break;
            const int nt = tile / p.t_chunks, tc = tile - nt * p.t_chunks;
            const int n = (nt * NA + a) * FT_BM + r;   // output column (weight row) of this lane
            if (k0 > 0 || k1 < p.kb) {
                float *mine = p.ws + ((size_t)(2 * blockIdx.x + (k1 == p.kb ? 0 : 1)) * NA + a) * p.BT * FT_BM + r;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (col_base + c * 16 < p.BT) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) mine[(size_t)(col_base + c * 16 + j) * FT_BM] = acc[c][j];
                    }
                }
            } else if (n < p.N) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int col = col_base + c * 16 + j, row = tc * p.BT + col;
                        if (col < p.BT && row < p.M) out[(size_t)row * p.N + n] = acc[c][j];
                    }
                }
            }
        }
    }

    ft_fence_before();
    __syncthreads();
    if (warp == FT_ISSUE0) {
        ft_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

// The tiles that several CTAs share: their parts added in CTA order. Block (tile half, 8 batch rows).
__global__ void __launch_bounds__(128) ft_join_kernel(FTParams p, int NA, int grid, float *__restrict__ out) {
    pdl_wait();
    pdl_trigger();
    const int tile = blockIdx.x / NA, a = blockIdx.x - tile * NA, t0 = blockIdx.y * 8, r = threadIdx.x;
    const long long u0 = (long long)tile * p.kb;
    const int c0 = (int)(((u0 + 1) * grid - 1) / p.units), c1 = (int)(((u0 + p.kb) * grid - 1) / p.units);   // CTAs of the first and last unit
    if (c0 == c1) return;
    float sum[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) sum[t] = 0.0f;
#pragma unroll 4
    for (int c = c0; c <= c1; ++c) {
        const float *part = p.ws + ((size_t)(2 * c + (c == c1 ? 0 : 1)) * NA + a) * p.BT * FT_BM + (size_t)t0 * FT_BM + r;
#pragma unroll
        for (int t = 0; t < 8; ++t) sum[t] += __ldcg(part + t * FT_BM);
    }
    const int nt = tile / p.t_chunks, row0 = (tile - nt * p.t_chunks) * p.BT + t0, n = (nt * NA + a) * FT_BM + r;
    if (n >= p.N) return;
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (row0 + t < p.M) out[(size_t)(row0 + t) * p.N + n] = sum[t];
}

bool f32_gemm_tc_supported(const float *d_w, const float *d_x, size_t m, size_t n, size_t k) {
    return tensor_map_encoder() != nullptr && m > 8 && n >= 1 && k >= FT_BK && k % FT_BK == 0 &&
           ((reinterpret_cast<uintptr_t>(d_w) | reinterpret_cast<uintptr_t>(d_x)) & 15) == 0 &&
           m < (1u << 30) && n < (1u << 30) && k < (1u << 30);
}

size_t f32_gemm_tc_scratch_bytes(size_t m, size_t k) { return 2 * m * k * sizeof(float) + 256; }

// d_w [n][k], d_x [m][k], d_out [m][n]; scratch: f32_gemm_tc_scratch_bytes(m, k)
int f32_gemm_tc(yscv_cuda_ctx *ctx, const float *d_w, const float *d_x, size_t m, size_t n, size_t k,
                float *d_out, void *scratch) {
    FTParams p = {};
    p.M = (int)m;
    p.N = (int)n;
    p.K = (int)k;
    const int m16 = (int)((m + 15) / 16 * 16), sms = ctx->sm_count;
    p.BT = m16 <= FT_BT_MAX ? m16 : FT_BT_MAX;
    p.t_chunks = (p.M + p.BT - 1) / p.BT;
    p.kb = (p.K + FT_UNIT - 1) / FT_UNIT;
    const int tiles1 = (p.N + FT_BM - 1) / FT_BM * p.t_chunks, tiles2 = (p.N + 2 * FT_BM - 1) / (2 * FT_BM) * p.t_chunks;
    const int NA = p.BT <= FT_BT_MAX / 2 && (long long)tiles2 * p.kb >= 8ll * sms ? 2 : 1;
    const int tiles = NA == 2 ? tiles2 : tiles1;
    if ((long long)tiles * p.kb >= (1ll << 31))
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "fp32 matmul too large: m=%zu n=%zu k=%zu", m, n, k);
    p.units = tiles * p.kb;
    p.stage_bytes = NA * FT_W_BYTES + 2 * p.BT * 128;
    p.stages = (227 * 1024 - 1024) / p.stage_bytes;
    if (p.stages > FT_MAX_STAGES) p.stages = FT_MAX_STAGES;
    const int smem = p.stages * p.stage_bytes + 256;
    // parts of shared tiles, up to 19 MB of the batch GEMM's workspace; where it cannot be had (a first call
    // inside a capture, no memory), or K < 1024, where the second launch costs more than the balance gains
    // (17 x 130 x 96: 12.9 us with it, 9.5 without), every CTA takes whole tiles
    int grid = p.units < sms ? p.units : sms;
    if (grid > tiles * 4) grid = tiles * 4;
    if (p.kb >= 16 && int4_batch_ready(ctx)) p.ws = reinterpret_cast<float *>(ctx->batch_ws.ptr);

    float *x_hi = reinterpret_cast<float *>(scratch), *x_lo = x_hi + m * k;
    const size_t n4 = m * k / 4;
    const unsigned sb = (unsigned)((n4 + 255) / 256 < 2368 ? (n4 + 255) / 256 : 2368);
    YSCV_CUDA_TRY(launch_pdl(ft_split_act_kernel, dim3(sb), dim3(256), 0, ctx->stream,
                             reinterpret_cast<const float4 *>(d_x), reinterpret_cast<float4 *>(x_hi),
                             reinterpret_cast<float4 *>(x_lo), n4));
    ctx->launches++;

    CUtensorMap tm_w, tm_xh, tm_xl;
    int rc = encode_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d_w, n, k, k * 4, FT_BM, FT_BK, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = encode_2d(&tm_xh, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, x_hi, m, k, k * 4, (uint32_t)p.BT, FT_BK, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = encode_2d(&tm_xl, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, x_lo, m, k, k * 4, (uint32_t)p.BT, FT_BK, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    auto kern = NA == 2 ? f32_gemm_tf32x3_kernel<2> : f32_gemm_tf32x3_kernel<1>;
    rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kern), ctx->device, 227 * 1024);
    if (rc) return rc;
    YSCV_CUDA_TRY(launch_pdl(kern, dim3(grid), dim3(FT_THREADS), (size_t)smem, ctx->stream, tm_w, tm_xh, tm_xl, d_out, p,
                             ctx->d_status));
    ctx->launches++;
    bool shared = false;
    for (int c = 1; c < grid && !shared; ++c) shared = ft_first_unit(p, c, grid) % p.kb != 0;
    if (shared) {
        YSCV_CUDA_TRY(launch_pdl(ft_join_kernel, dim3((unsigned)(tiles * NA), (unsigned)(p.BT / 8)), dim3(128), 0, ctx->stream, p, NA, grid, d_out));
        ctx->launches++;
    }
    return YSCV_CUDA_OK;
}

}  // namespace yscv
