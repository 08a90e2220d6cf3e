// Packed-int4 x fp32 matmul for a batch of 3..128 activation rows on the 5th-generation tensor cores,
// dequantised weights through tensor memory: packed_int4_gemm_dispatch
// (crates/yscv-kernels/src/ops/int4_matmul.rs:387-435, 548-605) between the few-row GEMV and the
// prompt-sized GEMM. The weight rows are the MMA's M side (128 per tile), the activation rows its N side.
//
// Two forms of one kernel:
//   bf16   17..128 rows: weights q * scale and activations rounded to bf16, fp32 accumulators (the
//          contract and the products of int4_prefill_gemm.cu)
//   exact  3..16 rows: the int4 values themselves as fp16 (exact), activations as two fp16 terms
//          hi + lo of the value scaled by a power of two per row and 256 k (22 significant bits, absolute
//          error below 2^-38 of that block's maximum). One accumulator holds one group of 32 k (the
//          tensor core adds by truncation: nothing accumulates longer), and the drain multiplies it by
//          the fp32 group scale and adds in fp32 registers, rounded. Relative error against float64
//          1.2e-7 (the integer-MMA GEMV's 21-bit blocks: 5.4e-7; with outliers of 10^4: 1.2e-7 and 1.2e-6).
//
// What bounds it: the weights' HBM stream (0.625 B per weight). A dequantised tile that goes through
// shared memory costs 4 B of shared-memory traffic per weight and a round trip; here the thread that
// owns a weight row writes its values to TMEM (tcgen05.st), where the MMA reads its A operand. A stage
// is 256 k (128 contiguous bytes of every row), so that DRAM sees whole lines.
//
// Work split, large matrices: the units (tile, 256 k) are numbered through and every CTA takes an equal contiguous
// range, so that no tile count leaves SMs idle. The parts of a tile whose units lie in several CTAs go
// to a workspace as fp32 partial sums; a second kernel adds them in CTA order (the same result every time).
// Smaller ones (bf16, SLICED): a CTA takes whole items (tile, slice of k) and stores the slice's sums as
// [slice][M][N] rows, which add_kslices_kernel adds in slice order; nothing to add with one slice.
// bg_split chooses.
//
// A small call is a chain of latencies: launch, weights from HBM, dequantisation, activations, MMA, drain, and the
// next kernel's wait. So a stage has a barrier for its weights and one for its activations, and the weights are
// fetched and dequantised into the A slots while the predecessor still runs; no more stages than a CTA has units, so
// that its blocks fit beside it; the drain steps one pointer (with an address and two bounds per element it took 1.1
// us for 32 columns, now 0.35). us per call with its activation pass, 32 / 64 / 128 rows, against
// int4_prefill_gemm_kernel with K slices: 2560 x 2048 8.0 / 8.6 / 9.8 (9.7 / 12.5 / 16.5), 11264 x 2048 12.2 / 12.9 / 15.3
// (15.4 / 15.4 / 17.3), 2048 x 5632 10.1 / 10.7 / 12.2 (11.8 / 13.4 / 23.5), 4096 x 4096 10.8 / 11.6 / 13.2 (12.7 / 13.6 /
// 20.3). The drain alone: 57344 x 8192 at 64 rows 90 -> 84.
//
// Warps: 0 TMA producer, 1 (and 2) MMA issuer of tile half 0 (and 1), 4..11 dequantise (two groups of
// four warps: a tile half each, or every other slot), 12.. drain and store. A hand-over between the
// roles costs about 330 cycles of barrier traffic whatever it carries and an MMA here 40 to 60, so a
// slot (one hand-over) is 128 rows x 128 k and the two halves have an issuer each: with 64-k slots and
// one issuer 57344 x 8192 at 64 rows took 126 us, without any work in the roles still 72.
#include "common.cuh"
#include "kernels.cuh"
#include "tma.cuh"

namespace yscv {

constexpr int BG_UNIT = 256;                       // k per stage and unit of work
constexpr int BG_W = 128 * 128;                    // packed nibbles of a tile and unit
constexpr int BG_S = 128 * 32;                     // scales of a tile and unit
constexpr int BG_SLOTS = 4;                        // A slots in TMEM, 128 k (64 columns) each
constexpr int BG_DEQ0 = 4, BG_EPI0 = 12;
constexpr int BG_MAX_STAGES = 8;
constexpr int BG_INV = 1024;                       // exact form: inverse scales of the unit's rows (64 bytes used)

template <int NA, bool EXACT> constexpr int bg_threads() { return (BG_EPI0 + (EXACT ? 4 * NA : 4)) * 32; }

struct BGParams {
    int M, N, K;
    int BT;                 // activation rows of the MMA (multiple of 16); exact: 16
    int kb, units;          // units per tile, units in all
    int per, rest;          // units / CTAs, units % CTAs
    int slices, tiles;      // sliced form: k slices per tile, tiles
    int stages, stage_bytes;
    int acc_bufs;           // bf16: accumulator sets in TMEM
    float *ws;              // [CTA][2: part with its tile's last unit, part without][NA][BT][128]
    const float *inv;       // exact: [kb][16]
};

__device__ __forceinline__ void bg_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void bg_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// K-major operand with the 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t bg_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)2 << 61;
}
__device__ __forceinline__ void bg_mma(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void bg_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bg_ld32(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
          "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void bg_st32(uint32_t taddr, const uint32_t *r) {
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
// First unit of CTA c: c * units / CTAs without the 64-bit division (a third of a small call's set-up)
__host__ __device__ inline int bg_first_unit(const BGParams &p, int c, int grid) { return c * p.per + c * p.rest / grid; }
// One CTA's walk: every call yields a tile and its range of k units. Equal ranges of the units, last one first, or
// (SLICED) the items (slice, tile) CTA by CTA.
template <bool SLICED> struct BGWalk {
    int end, first, kb, slice;
    __device__ BGWalk(const BGParams &p)
        : end(SLICED ? (int)blockIdx.x : bg_first_unit(p, blockIdx.x + 1, gridDim.x)), first(SLICED ? p.tiles : bg_first_unit(p, blockIdx.x, gridDim.x)),
          kb(p.kb), slice(SLICED ? p.slices : 0) {}
    __device__ bool next(int &tile, int &k0, int &k1, int &sl) {
        if (SLICED) {
            if (end >= first * slice) return false;
            sl = end / first;
            tile = end - sl * first;
            k0 = sl * kb / slice;
            k1 = (sl + 1) * kb / slice;
            end += gridDim.x;
            return true;
        }
        if (end <= first) return false;
        tile = (end - 1) / kb;
        const int start = max(first, tile * kb);
        k0 = start - tile * kb;
        k1 = end - tile * kb;
        end = start;
        sl = 0;
        return true;
    }
};

template <int NA, bool EXACT, bool SLICED>
__global__ void __launch_bounds__(bg_threads<NA, EXACT>(), 1)
int4_batch_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_s,
                       const __grid_constant__ CUtensorMap tm_a, float *__restrict__ out, BGParams p, int *__restrict__ status) {
    constexpr int EPI_WARPS = EXACT ? 4 * NA : 4;
    constexpr int RING = BG_SLOTS / NA;              // A slots per tile half
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = smem_u32(smem);
    // stage: [NA][128 rows][128 B nibbles] [NA][128 rows][8 scales] [4][BT rows][64 k] (exact: + inverse scales)
    const int act_rows = EXACT ? 32 : p.BT;
    constexpr int S_OFF = NA * BG_W, A_OFF = NA * (BG_W + BG_S);
    const uint32_t bars = base + (uint32_t)p.stages * p.stage_bytes;
    const uint32_t wfull = bars, xfull = bars + 64, empty = bars + 128, afull = bars + 192, mdone = bars + 224, dempty = bars + 256;
    const uint32_t tfull = bars + 288, tempty = bars + 304;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + (size_t)p.stages * p.stage_bytes + 320);

    if (tid == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(wfull + i * 8, 1);   // nibbles and scales have landed
            mbar_init(xfull + i * 8, 1);   // activations (and inverse scales) have landed
            mbar_init(empty + i * 8, NA + (EXACT ? EPI_WARPS : 0));
        }
        for (int i = 0; i < BG_SLOTS; ++i) {
            mbar_init(afull + i * 8, 4);
            mbar_init(mdone + i * 8, 1);
            mbar_init(dempty + i * 8, 4);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(tfull + i * 8, NA);
            mbar_init(tempty + i * 8, 4);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    bg_fence_before();
    __syncthreads();
    bg_fence_after();
    pdl_trigger();
    const uint32_t tmem = *tmem_slot;
    const uint32_t t_a = tmem + 256;                 // columns 0..255: accumulators, 256..511: A slots
    BGWalk<SLICED> walk(p);
    int tile, k0, k1, sl;
    bool alive = true;
    // The weights are the caller's constants (the kernels that pack them are ordinary launches, complete
    // before a dependent one starts): the first stages' are fetched, and dequantised into the A slots, while the
    // predecessor drains. The producer waits before it fetches activations, which may be its output, the drain
    // before it writes the workspace and `out`, which may still be in its use.

    if (warp == 0) {
        if (lane == 0) {
            auto weights = [&](int st, int tl, int u) {
                const uint32_t dst = base + (uint32_t)st * p.stage_bytes, bar = wfull + st * 8;
                mbar_expect_tx(bar, NA * (BG_W + BG_S));
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    tma_load_2d(dst + a * BG_W, &tm_w, u * (BG_UNIT / 2), (tl * NA + a) * 128, bar);
                    tma_load_2d(dst + S_OFF + a * BG_S, &tm_s, u * (BG_UNIT / 32), (tl * NA + a) * 128, bar);
                }
            };
            BGWalk<SLICED> ahead(p);
            int early = 0;
            while (early < p.stages && ahead.next(tile, k0, k1, sl))
                for (int u = k0; u < k1 && early < p.stages; ++u) weights(early++, tile, u);
            pdl_wait();
            int st = 0, cnt = 0;
            uint32_t ph = 0;
            while (alive && walk.next(tile, k0, k1, sl)) {
                for (int u = k0; u < k1; ++u) {
                    if (cnt++ >= early) {
                        alive = mbar_wait(empty + st * 8, ph ^ 1u, status);
                        if (!alive) break;
                        weights(st, tile, u);
                    }
                    const uint32_t dst = base + (uint32_t)st * p.stage_bytes, bar = xfull + st * 8;
                    mbar_expect_tx(bar, 4 * act_rows * 128 + (EXACT ? 64 : 0));
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        tma_load_2d(dst + A_OFF + s * act_rows * 128, &tm_a, u * BG_UNIT + s * 64, 0, bar);
                    if (EXACT) bulk_load(dst + A_OFF + 4 * 32 * 128, p.inv + u * 16, 64, bar);
                    if (++st == p.stages) { st = 0; ph ^= 1u; }
                }
            }
            // a consumer gave up: no stage's copies may be in flight when the CTA leaves (bounded)
            if (!alive)
                for (int i = 0; i < p.stages; ++i) {
                    mbar_wait(wfull + i * 8, i < st ? ph : ph ^ 1u, nullptr);
                    mbar_wait(xfull + i * 8, i < st ? ph : ph ^ 1u, nullptr);
                }
        }
        __syncwarp();
    } else if (warp <= NA) {
        // ---- MMA issuer of tile half a ----
        const int a = warp - 1;
        // D fp32, A (TMEM) and B both bf16 or both fp16, K-major, M = 128
        const uint32_t idesc = (1u << 4) | (EXACT ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)((EXACT ? 16 : p.BT) >> 3) << 17) |
                               ((uint32_t)(128 >> 4) << 24);
        int st = 0, ring = 0, buf = 0;
        uint32_t ph = 0, rph = 0, bph = 0;
        while (alive && walk.next(tile, k0, k1, sl)) {
            if (!EXACT) {
                alive = __all_sync(0xffffffffu, mbar_wait(tempty + buf * 8, bph ^ 1u, status));
                if (!alive) break;
            }
            const uint32_t acc = tmem + (buf * NA + a) * p.BT;
            for (int u = k0; u < k1 && alive; ++u) {
                alive = __all_sync(0xffffffffu, mbar_wait(xfull + st * 8, ph, status));
                if (!alive) break;
                const uint32_t act = base + (uint32_t)st * p.stage_bytes + A_OFF;
#pragma unroll
                for (int half = 0; half < 2; ++half) {       // 128 k: two 64-k activation tiles
                    const int slot = a * RING + ring;
                    alive = __all_sync(0xffffffffu, mbar_wait(afull + slot * 8, rph, status) &&
                                                        (!EXACT || mbar_wait(dempty + slot * 8, rph ^ 1u, status)));
                    if (!alive) break;
                    bg_fence_after();
                    const uint32_t ta = t_a + slot * 64;
                    const uint64_t db = bg_desc(act + half * 2 * act_rows * 128);
                    const uint64_t sub_step = (uint64_t)(act_rows * 128 >> 4);
                    if (elect_one()) {
                        if constexpr (EXACT) {
                            // rows 16..31 of an activation tile are the low terms (16 x 128 bytes further on);
                            // group g of 32 k: columns g * 16 of A, its own accumulator of 16 columns
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const int kk = (g & 1) * 2 + (i & 1);
                                    bg_mma(tmem + slot * 64 + g * 16, ta + g * 16 + (i & 1) * 8,
                                           db + (uint64_t)(g >> 1) * sub_step + (uint64_t)(kk * 2 + (i < 2 ? 128 : 0)), idesc, i > 0);
                                }
                            }
                        } else {
#pragma unroll
                            for (int kk = 0; kk < 8; ++kk)
                                bg_mma(acc, ta + kk * 8, db + (uint64_t)(kk >> 2) * sub_step + (uint64_t)((kk & 3) * 2), idesc,
                                       (u > k0 || half > 0 || kk > 0) ? 1u : 0u);
                        }
                        bg_commit(mdone + slot * 8);
                        if (half == 1) bg_commit(empty + st * 8);
                        if (!EXACT && half == 1 && u + 1 == k1) bg_commit(tfull + buf * 8);
                    }
                    __syncwarp();
                    if (++ring == RING) { ring = 0; rph ^= 1u; }
                }
                if (++st == p.stages) { st = 0; ph ^= 1u; }
            }
            if (++buf == p.acc_bufs) { buf = 0; bph ^= 1u; }
        }
    } else if (warp >= BG_DEQ0 && warp < BG_EPI0) {
        // ---- dequantise: thread = weight row r; a slot is 128 k = 64 columns. Two tile halves: group g
        // takes half g; one: group g takes every other slot ----
        const int g = (warp - BG_DEQ0) >> 2, r = (warp & 3) * 32 + lane;
        const int a = NA == 2 ? g : 0;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        int st = 0, ring = NA == 2 ? 0 : g;
        uint32_t ph = 0, rph = 0;
        while (alive && walk.next(tile, k0, k1, sl)) {
            for (int u = k0; u < k1 && alive; ++u) {
                alive = mbar_wait(wfull + st * 8, ph, status);
                if (!alive) break;
                const unsigned char *stage = smem + (size_t)st * p.stage_bytes;
                const unsigned char *row = stage + a * BG_W + r * 128;
#pragma unroll 1
                for (int half = NA == 2 ? 0 : g; half < 2; half += NA == 2 ? 1 : 2) {
                    const int slot = a * RING + ring;
                    // 16-byte chunk c of scale row r sits at chunk c ^ ((r >> 2) & 1) (32-byte swizzle)
                    const float4 sc4 = *reinterpret_cast<const float4 *>(stage + S_OFF + a * BG_S + r * 32 + ((half ^ ((r >> 2) & 1)) << 4));
                    const float sc[4] = {sc4.x, sc4.y, sc4.z, sc4.w};
#pragma unroll
                    for (int sub = 0; sub < 2; ++sub) {
                        const int c = half * 4 + sub * 2;
                        const uint4 wa = *reinterpret_cast<const uint4 *>(row + ((c ^ (r & 7)) << 4));
                        const uint4 wb = *reinterpret_cast<const uint4 *>(row + (((c + 1) ^ (r & 7)) << 4));
                        const uint32_t words[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
                        uint32_t o[32];
                        if constexpr (EXACT) {
                            // 0x6400 | (nibble ^ 8) is the fp16 value 1032 + q, 0x6400 | (nibble ^ 8) << 4 is 1152 + 16 q
                            const __half2 c0 = __float2half2_rn(1032.0f), c1 = __float2half2_rn(-72.0f), sixteenth = __float2half2_rn(0.0625f);
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                uint32_t x[4];
                                const uint32_t w8 = words[i] >> 8;
                                asm("lop3.b32 %0, %1, 0x000f000f, 0x64086408, 0x6a;\n" : "=r"(x[0]) : "r"(words[i]));
                                asm("lop3.b32 %0, %1, 0x00f000f0, 0x64806480, 0x6a;\n" : "=r"(x[1]) : "r"(words[i]));
                                asm("lop3.b32 %0, %1, 0x000f000f, 0x64086408, 0x6a;\n" : "=r"(x[2]) : "r"(w8));
                                asm("lop3.b32 %0, %1, 0x00f000f0, 0x64806480, 0x6a;\n" : "=r"(x[3]) : "r"(w8));
#pragma unroll
                                for (int h = 0; h < 4; ++h) {
                                    __half2 v = *reinterpret_cast<__half2 *>(&x[h]);
                                    v = (h & 1) ? __hfma2(v, sixteenth, c1) : __hsub2(v, c0);
                                    o[i * 4 + h] = *reinterpret_cast<uint32_t *>(&v);
                                }
                            }
                        } else {
                            const __nv_bfloat162 bias = __float2bfloat162_rn(136.0f);
                            const __nv_bfloat162 s2[2] = {__float2bfloat162_rn(sc[sub * 2]), __float2bfloat162_rn(sc[sub * 2 + 1])};
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const uint32_t w = words[i];
                                uint32_t x[4];
                                // 0x4300 | (nibble ^ 8) is the bf16 value 136 + q, exactly
                                asm("lop3.b32 %0, %1, 0x000f000f, 0x43084308, 0x6a;\n" : "=r"(x[0]) : "r"(w));
                                asm("lop3.b32 %0, %1, 0x000f000f, 0x43084308, 0x6a;\n" : "=r"(x[1]) : "r"(w >> 4));
                                asm("lop3.b32 %0, %1, 0x000f000f, 0x43084308, 0x6a;\n" : "=r"(x[2]) : "r"(w >> 8));
                                asm("lop3.b32 %0, %1, 0x000f000f, 0x43084308, 0x6a;\n" : "=r"(x[3]) : "r"(w >> 12));
#pragma unroll
                                for (int h = 0; h < 4; ++h) {
                                    __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162 *>(&x[h]);
                                    v = __hmul2(__hsub2(v, bias), s2[i >> 2]);
                                    o[i * 4 + h] = *reinterpret_cast<uint32_t *>(&v);
                                }
                            }
                        }
                        if (sub == 0) {
                            alive = mbar_wait(mdone + slot * 8, rph ^ 1u, status);
                            if (!alive) break;
                            bg_fence_after();
                        }
                        bg_st32(t_a + slot * 64 + sub * 32 + lane_base, o);
                    }
                    if (!alive) break;
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    bg_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(afull + slot * 8);
                    ring += NA == 2 ? 1 : 2;
                    if (ring >= RING) { ring -= RING; rph ^= 1u; }
                }
                if (++st == p.stages) { st = 0; ph ^= 1u; }
            }
        }
    } else if (warp >= BG_EPI0) {
        const int w = warp - BG_EPI0, r = (w & 3) * 32 + lane;
        const uint32_t lane_base = (uint32_t)((w & 3) * 32) << 16;
        int st = 0, buf = 0, ring = 0;
        uint32_t ph = 0, bph = 0, rph = 0;
        pdl_wait();
        while (alive && walk.next(tile, k0, k1, sl)) {
            const bool whole = SLICED || (k0 == 0 && k1 == p.kb);
            float *const mine = p.ws + (size_t)(2 * blockIdx.x + (k1 == p.kb ? 0 : 1)) * NA * p.BT * 128 + r;
            if constexpr (EXACT) {
                const int a = w >> 2;
                float acc[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) acc[t] = 0.0f;
                for (int u = k0; u < k1 && alive; ++u) {
                    const unsigned char *stage = smem + (size_t)st * p.stage_bytes;
                    alive = mbar_wait(wfull + st * 8, ph, status) && mbar_wait(xfull + st * 8, ph, status);
                    if (!alive) break;
                    const unsigned char *srow = stage + S_OFF + a * BG_S + r * 32;
                    float part[16];
#pragma unroll
                    for (int t = 0; t < 16; ++t) part[t] = 0.0f;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int slot = a * RING + ring;
                        const float4 s4 = *reinterpret_cast<const float4 *>(srow + ((half ^ ((r >> 2) & 1)) << 4));
                        alive = alive && mbar_wait(mdone + slot * 8, rph, status);
                        if (!alive) break;
                        bg_fence_after();
                        const float sc[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                        for (int pair = 0; pair < 2; ++pair) {
                            uint32_t d[32];
                            bg_ld32(tmem + slot * 64 + pair * 32 + lane_base, d);
                            if (pair == 1) {
                                bg_fence_before();
                                __syncwarp();
                                if (lane == 0) mbar_arrive(dempty + slot * 8);
                            }
#pragma unroll
                            for (int t = 0; t < 16; ++t) {
                                part[t] = fmaf(__uint_as_float(d[t]), sc[pair * 2], part[t]);
                                part[t] = fmaf(__uint_as_float(d[16 + t]), sc[pair * 2 + 1], part[t]);
                            }
                        }
                        if (++ring == RING) { ring = 0; rph ^= 1u; }
                    }
                    const float4 *inv = reinterpret_cast<const float4 *>(stage + A_OFF + 4 * 32 * 128);
#pragma unroll
                    for (int t4 = 0; t4 < 4; ++t4) {
                        const float4 iv = inv[t4];
                        acc[t4 * 4] = fmaf(part[t4 * 4], iv.x, acc[t4 * 4]);
                        acc[t4 * 4 + 1] = fmaf(part[t4 * 4 + 1], iv.y, acc[t4 * 4 + 1]);
                        acc[t4 * 4 + 2] = fmaf(part[t4 * 4 + 2], iv.z, acc[t4 * 4 + 2]);
                        acc[t4 * 4 + 3] = fmaf(part[t4 * 4 + 3], iv.w, acc[t4 * 4 + 3]);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty + st * 8);
                    if (++st == p.stages) { st = 0; ph ^= 1u; }
                }
                if (!alive) break;
                const int n = (tile * NA + a) * 128 + r;
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    if (!whole) mine[((size_t)a * 16 + t) * 128] = acc[t];
                    else if (n < p.N && t < p.M) out[(size_t)t * p.N + n] = acc[t];
                }
            } else {
                alive = mbar_wait(tfull + buf * 8, bph, status);
                if (!alive) break;
                bg_fence_after();
#pragma unroll 1
                for (int a = 0; a < NA; ++a) {
                    const int n = (tile * NA + a) * 128 + r;
                    // a column of the result, or of this CTA's part of the tile
                    float *o = whole ? out + (size_t)sl * p.M * p.N + n : mine + (size_t)a * p.BT * 128;
                    const size_t pitch = whole ? p.N : 128;
                    const int rows = whole ? (n < p.N ? p.M : 0) : p.BT;
#pragma unroll 1
                    for (int t0 = 0; t0 < p.BT; t0 += 32) {
                        uint32_t d[32];
                        bg_ld32(tmem + (buf * NA + a) * p.BT + t0 + lane_base, d);
#pragma unroll
                        for (int t = 0; t < 32; ++t) {
                            if (t0 + t < rows) *o = __uint_as_float(d[t]);
                            o += pitch;
                        }
                    }
                }
                bg_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty + buf * 8);
                if (++buf == p.acc_bufs) { buf = 0; bph ^= 1u; }
            }
        }
    }

    bg_fence_before();
    __syncthreads();
    if (warp == 1) {
        bg_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

// The tiles that several CTAs share: their parts added in CTA order. Block (128-row tile half, 8
// activation rows); `grid` is the GEMM's. Parts are at most 2 x grid x NA x BT x 512 B and in L2.
__global__ void __launch_bounds__(128)
bg_join_kernel(BGParams p, int NA, int grid, float *__restrict__ out) {
    pdl_wait();
    pdl_trigger();
    const int tile = blockIdx.x / NA, a = blockIdx.x - tile * NA, t0 = blockIdx.y * 8, r = threadIdx.x;
    const long long u0 = (long long)tile * p.kb;
    const int c0 = (int)(((u0 + 1) * grid - 1) / p.units), c1 = (int)(((u0 + p.kb) * grid - 1) / p.units);   // CTAs of the first and last unit
    if (c0 == c1) return;
    const int n = (tile * NA + a) * 128 + r;
    float sum[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) sum[t] = 0.0f;
#pragma unroll 4
    for (int c = c0; c <= c1; ++c) {
        const float *part = p.ws + ((size_t)(2 * c + (c == c1 ? 0 : 1)) * NA + a) * p.BT * 128 + (size_t)t0 * 128 + r;
#pragma unroll
        for (int t = 0; t < 8; ++t) sum[t] += __ldcg(part + t * 128);
    }
    if (n < p.N) {
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (t0 + t < p.M) out[(size_t)(t0 + t) * p.N + n] = sum[t];
    }
}

// fp32 activations -> the exact form's fp16 terms (store_terms). A warp takes one row and 256 k.
__global__ void __launch_bounds__(128)
act_split16_kernel(const float *__restrict__ act, int M, int K, int kb, __half *__restrict__ terms, float *__restrict__ inv) {
    pdl_wait();
    pdl_trigger();
    const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= M * kb) return;
    const int m = item / kb, u = item - m * kb, k = u * BG_UNIT + lane * 8;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (k < K) {
        const float4 *src = reinterpret_cast<const float4 *>(act + (size_t)m * K + k);
        a = __ldg(src);
        b = __ldg(src + 1);
    }
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    store_terms(v, terms, inv, K, m, k, k < K);
}

// 39 MB, whatever the shape. Where it cannot be had (a first call inside a capture, no memory) the call takes the
// kernel that it took before there was this one.
static size_t bg_ws_bytes(const yscv_cuda_ctx *ctx) { return (size_t)ctx->sm_count * 2 * 2 * 128 * 128 * sizeof(float); }
bool int4_batch_ready(yscv_cuda_ctx *ctx) { return ctx->batch_ws.try_reserve(bg_ws_bytes(ctx), ctx->stream); }
static size_t bg_inv_offset(size_t k) { return (32 * k * 2 + 255) / 256 * 256; }   // of the inverse scales behind the terms
size_t int4_batch_exact_scratch_bytes(size_t k) { return bg_inv_offset(k) + (k + BG_UNIT - 1) / BG_UNIT * 64 + 256; }

size_t act_bytes(int form, size_t m, size_t k) {
    if (form == ACT_DIGITS) return int4_gemv_scratch_bytes(m, k);
    if (form == ACT_TERMS) return int4_batch_exact_scratch_bytes(k);
    return m * k * (form == ACT_BF16 ? 2 : 4);
}
ActOut act_out(int form, size_t m, size_t k, void *buffer) {
    ActOut o;
    o.form = form;
    o.rows = (int)m;
    o.k = (int)k;
    o.ptr = buffer;
    if (form == ACT_DIGITS) o.q = int4_gemv_layout(m, k);
    if (form == ACT_TERMS) o.inv = reinterpret_cast<float *>(static_cast<unsigned char *>(buffer) + bg_inv_offset(k));
    return o;
}

// k % 128: the scale rows (k / 32 floats) are TMA rows, whose pitch must be a multiple of 16 bytes.
static bool bg_shape(size_t n, size_t k, size_t gs) {
    return tensor_map_encoder() != nullptr && gs == 32 && k % 128 == 0 && k >= 128 && n >= 1 && n < (1u << 22) && k < (1u << 22);
}

// Which calls gain.
//   bf16: every one of 17..128 rows, against int4_prefill_gemm_kernel (figures at the top; large ones, 32 / 64 / 128
//   rows: 57344 x 8192 77 / 148, 84 / 173, 130 / 194; 8192 x 28672 50 / 76, 52 / 81, 68 / 89; 10240 x 8192 26 / 33, 29 / 36,
//   35 / 42; 14336 x 4096 20 / 27, 21 / 26, 26 / 29; the closest 16384 x 2048 at 128 rows 15.9 / 18.0)
bool int4_batch_bf16_wins(size_t m, size_t n, size_t k, size_t gs) { return m > 16 && m <= 128 && bg_shape(n, k, gs); }
//   exact, against the integer-MMA GEMV, 4 / 8 / 16 rows: 57344 x 8192 79 / 85, 80 / 95, 78 / 143; 8192 x 28672
//   49 / 49, 50 / 60, 50 / 83; 28672 x 8192 47 / 46, 47 / 51, 47 / 74; 22016 x 4096 27 / 29, 27 / 28, 27 / 41; 10240 x
//   8192 25 / 24, 25.1 / 26.5, 25 / 39; 14336 x 4096 22 / 18, 23 / 16, 23 / 22; 2 rows: everywhere behind. Depths that
//   are no multiple of 256 would take the fp32 FMA kernel, several times slower: earlier lines.
bool int4_batch_exact_wins(size_t m, size_t n, size_t k, size_t gs) {
    const size_t weights = n * k;
    const bool gemv = k % 256 == 0;
    return m > 2 && m <= 16 && bg_shape(n, k, gs) && weights >= (m > 8 ? 64000000u : m > 4 ? (gemv ? 80000000u : 64000000u) : gemv ? 350000000u : 200000000u);
}

template <int NA, bool EXACT, bool SLICED>
static int launch_batch(yscv_cuda_ctx *ctx, const CUtensorMap &tm_w, const CUtensorMap &tm_s, const CUtensorMap &tm_a, float *out,
                        BGParams p, int grid) {
    const int act = EXACT ? 4 * 32 * 128 + BG_INV : 4 * p.BT * 128;
    p.stage_bytes = NA * (BG_W + BG_S) + act;
    p.stages = (227 * 1024 - 1024) / p.stage_bytes;
    if (p.stages > BG_MAX_STAGES) p.stages = BG_MAX_STAGES;
    const int longest = SLICED ? (p.tiles * p.slices + grid - 1) / grid * ((p.kb + p.slices - 1) / p.slices) : (p.units + grid - 1) / grid;
    if (p.stages > longest) p.stages = longest;   // units of a CTA
    const int smem = p.stages * p.stage_bytes + 512;
    auto kern = int4_batch_gemm_kernel<NA, EXACT, SLICED>;
    p.per = p.units / grid;
    p.rest = p.units % grid;
    int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kern), ctx->device, 227 * 1024);
    if (rc) return rc;
    ctx->prof_begin();
    YSCV_CUDA_TRY(launch_pdl(kern, dim3(grid), dim3(bg_threads<NA, EXACT>()), (size_t)smem, ctx->stream, tm_w, tm_s, tm_a, out, p,
                             ctx->d_status));
    ctx->prof_end();
    YSCV_CUDA_TRY(cudaGetLastError());
    ctx->launches++;
    bool shared = false;
    for (int c = 1; c < grid && !shared && !SLICED; ++c) shared = bg_first_unit(p, c, grid) % p.kb != 0;
    if (shared) {
        YSCV_CUDA_TRY(launch_pdl(bg_join_kernel, dim3((unsigned)(p.units / p.kb * NA), (unsigned)(p.BT / 8)), dim3(128), 0, ctx->stream, p,
                                 NA, grid, out));
        ctx->launches++;
    }
    const int splits = SLICED ? p.slices : (grid + (p.units / p.kb) - 1) / (p.units / p.kb);
    if (EXACT) {
        snprintf(ctx->report_int4, sizeof(ctx->report_int4),
                 "int4_fast m=%d n=%d k=%d: tcgen05 fp16 two-term, CTA tile %d rows x 16, 256 k per stage, %d stages, %d units on %d CTAs",
                 p.M, p.N, p.K, NA * 128, p.stages, p.units, grid);
        ctx->last_kernel = "int4_fast(tcgen05,fp16x2,tmem)";
    } else {
        snprintf(ctx->report_int4, sizeof(ctx->report_int4),
                 "int4_prefill_gemm m=%d n=%d k=%d: tcgen05 bf16, weights through TMEM, CTA tile %d rows x %d tokens, 2 x 128 k per stage, "
                 "%d stages, %d K slice(s), %d units on %d CTAs", p.M, p.N, p.K, NA * 128, p.BT, p.stages, splits, p.units, grid);
        ctx->last_kernel = "int4_prefill_gemm(tcgen05,bf16,tmem)";
    }
    return YSCV_CUDA_OK;
}

// K slices of the sliced form, or 0 for equal ranges over the CTAs, by the modelled time in us: units one after another
// in a CTA, a round's drain, the launch that adds slices and their traffic; equal ranges cost a second drain and the
// join. The constants are a fit to 24 shapes from 512 x 2048 to 8192 x 28672 at 20 / 32 / 64 / 128 rows with every
// choice forced in turn; its choice is 0.15 % behind the best of them on average and 3 % at worst. left_apart: the
// caller's next kernel adds the slices, which costs it their reads.
static int bg_split(const BGParams &p, int NA, int grid, int sms, bool slices_ok, size_t ws_bytes, bool left_apart) {
    const double unit = 0.64 + 0.002 * p.BT, mb = 0.07e-6;
    double best = 3.2 + (p.units + grid - 1) / grid * unit * (NA == 2 ? 1.75 : 1.0) + 2.0 * grid * NA * 128 * p.BT * 4 * mb;
    int slices = 0;
    const int tiles = (p.N + 127) / 128;
    for (int s = 1; s <= INT4_MAX_PARTS && s <= p.kb; ++s) {
        const double bytes = (double)s * p.M * p.N * 4;
        if (s > 1 && (!slices_ok || bytes > (double)ws_bytes)) break;
        const double rounds = (int)(((long long)tiles * s + sms - 1) / sms);
        const double cost = rounds * ((p.kb + s - 1) / s * unit + 0.55) + (s == 1 ? 0.0 : left_apart ? 0.1 * s + bytes * mb / 2 : 0.97 + 0.022 * s + bytes * mb);
        if (cost < best) { best = cost; slices = s; }
    }
    return slices;
}

struct BGPlan {
    BGParams p;
    int NA, grid;
};
static BGPlan bg_plan(yscv_cuda_ctx *ctx, size_t m, size_t n, size_t k, bool exact, bool slices_ok, bool left_apart) {
    BGParams p = {};
    p.M = (int)m;
    p.N = (int)n;
    p.K = (int)k;
    p.BT = (int)((m + 15) / 16 * 16);
    p.kb = (p.K + BG_UNIT - 1) / BG_UNIT;
    p.ws = reinterpret_cast<float *>(ctx->batch_ws.ptr);
    const int sms = ctx->sm_count;
    const int tiles1 = (p.N + 127) / 128, tiles2 = (p.N + 255) / 256;
    // two tile halves share a unit's activations, but halve the number of units: 10240 x 8192 at 128 rows
    // 40 us with one, 50 with two; 8192 x 28672 at 32 rows 55 and 50 (the exact form, whose unit is
    // longer: 14336 x 4096 26 and 23)
    const int NA = exact || (long long)tiles2 * p.kb >= 20ll * sms ? 2 : 1;
    const int tiles = NA == 2 ? tiles2 : tiles1;
    p.units = tiles * p.kb;
    // at most four parts to a tile on average: 2048 x 2048 at 32 rows 11.2 us against 13.0 with eight
    int grid = p.units < sms ? p.units : sms;
    if (grid > tiles * 4) grid = tiles * 4;
    p.acc_bufs = NA * p.BT > 128 ? 1 : 2;
    if (!exact) p.slices = bg_split(p, NA, grid, sms, slices_ok, bg_ws_bytes(ctx), left_apart);
    if (p.slices > 0) {
        p.tiles = tiles1;
        p.units = tiles1 * p.kb;
        p.acc_bufs = 2;
        const int items = tiles1 * p.slices;
        return {p, 1, items < sms ? items : sms};
    }
    return {p, NA, grid};
}
int int4_batch_parts(yscv_cuda_ctx *ctx, size_t m, size_t n, size_t k) {
    const int s = bg_plan(ctx, m, n, k, false, true, true).p.slices;
    return s > 1 ? s : 1;
}

// exact: act = fp32 rows (null: terms and inverse scales are in `scratch`), scratch of int4_batch_exact_scratch_bytes(k).
// Otherwise act_bf16 = bf16 rows in the permuted k order.
int int4_batch_gemm(yscv_cuda_ctx *ctx, const uint8_t *wq, const float *scales, const float *act, const void *act_bf16, float *out,
                    size_t m, size_t n, size_t k, void *scratch, int *parts) {
    const bool exact = act_bf16 == nullptr;
    // (add_kslices reads 16 bytes at a time)
    const bool join_ok = (m * n) % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    bool left_apart = parts && *parts > 1;
    BGPlan plan = bg_plan(ctx, m, n, k, exact, left_apart || join_ok, left_apart);
    if (left_apart && plan.p.slices > *parts) {
        left_apart = false;
        plan = bg_plan(ctx, m, n, k, exact, join_ok, false);
    }
    BGParams p = plan.p;
    const int NA = plan.NA, grid = plan.grid;
    if (parts) *parts = left_apart && p.slices > 1 ? p.slices : 1;

    CUtensorMap tm_w, tm_s, tm_a;
    int rc = encode_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wq, n, k / 2, k / 2, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = encode_2d(&tm_s, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, scales, n, k / 32, k / 8, 128, 8, CU_TENSOR_MAP_SWIZZLE_32B);
    if (rc) return rc;
    if (exact) {
        __half *terms = reinterpret_cast<__half *>(scratch);
        float *inv = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(scratch) + bg_inv_offset(k));
        p.inv = inv;
        if (act) {
            const unsigned blocks = (unsigned)((m * p.kb + 3) / 4);
            YSCV_CUDA_TRY(launch_pdl(act_split16_kernel, dim3(blocks), dim3(128), 0, ctx->stream, act, p.M, p.K, p.kb, terms, inv));
            ctx->launches++;
        }
        rc = encode_2d(&tm_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, terms, 32, k, k * 2, 32, 64, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
        return launch_batch<2, true, false>(ctx, tm_w, tm_s, tm_a, out, p, grid);
    }
    rc = encode_2d(&tm_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, act_bf16, m, k, k * 2, (uint32_t)p.BT, 64, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    if (p.slices > 0) {
        const bool join = p.slices > 1 && !left_apart;
        rc = launch_batch<1, false, true>(ctx, tm_w, tm_s, tm_a, join ? p.ws : out, p, grid);
        return rc || !join ? rc : add_kslices(ctx, p.ws, out, m * n, p.slices);
    }
    return NA == 2 ? launch_batch<2, false, false>(ctx, tm_w, tm_s, tm_a, out, p, grid) : launch_batch<1, false, false>(ctx, tm_w, tm_s, tm_a, out, p, grid);
}

}  // namespace yscv
