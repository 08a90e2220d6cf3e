// Internal launch wrappers shared between the kernel files and the C ABI.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "act_forms.cuh"

struct yscv_cuda_ctx;
struct yscv_cuda_i8b;
struct yscv_cuda_int4_weight;

namespace yscv {

// int4_gemv.cu
bool int4_gemv_fast_supported(size_t m, size_t n, size_t k, size_t gs);
size_t int4_gemv_scratch_bytes(size_t m, size_t k);
bool int4_gemv_uses_scratch(const yscv_cuda_ctx *ctx, size_t m, size_t n, size_t k);
bool int4_gemv_wants_digits(const yscv_cuda_ctx *ctx, size_t m, size_t n, size_t k);
bool int4_gemv_can_do_without_scratch(size_t m, size_t k);   // scratch == nullptr then
// fp32 matmul out[m][n] = sum_k x[m][k] w[n][k] for m > 8 as three TF32 products per fp32 product
// on the tensor cores (f32_gemm_tf32x3.cu)
bool f32_gemm_tc_supported(const float *d_w, const float *d_x, size_t m, size_t n, size_t k);
size_t f32_gemm_tc_scratch_bytes(size_t m, size_t k);
int f32_gemm_tc(yscv_cuda_ctx *ctx, const float *d_w, const float *d_x, size_t m, size_t n, size_t k,
                float *d_out, void *scratch);
int int4_gemv_fast(yscv_cuda_ctx *ctx, const uint8_t *wq, const float *scales, const float *act,
                   float *out, size_t m, size_t n, size_t k, void *scratch);
// the same with digit planes that the caller wrote (ActForm ACT_DIGITS, act_out())
int int4_gemv_digits(yscv_cuda_ctx *ctx, const uint8_t *wq, const float *scales, const void *digits, float *out, size_t m, size_t n, size_t k);
QuantLayout int4_gemv_layout(size_t m, size_t k);
bool int4_gemv_digits_whole(size_t m, size_t k);
int int4_gemv_generic(yscv_cuda_ctx *ctx, const uint8_t *wq, const float *scales,
                      const float *act, float *out, size_t m, size_t n, size_t k, size_t gs);

// int4_prefill_gemm.cu
bool int4_prefill_supported(size_t m, size_t n, size_t k, size_t gs);
size_t int4_prefill_scratch_bytes(size_t m, size_t k);
int int4_prefill_gemm(yscv_cuda_ctx *ctx, const uint8_t *wq, const float *scales, const float *act,
                      float *out, size_t m, size_t n, size_t k, void *scratch, const void *act_bf16 = nullptr, int *parts = nullptr);

constexpr int INT4_MAX_PARTS = 8;   // k slices of a matmul, and the parts that a kernel which adds them holds in registers
int add_kslices(yscv_cuda_ctx *ctx, const float *parts, float *out, size_t elements, int slices);

// int4_batch_gemm.cu: 3..128 activation rows, k % 128 == 0, 16-byte aligned operands. act_bf16 == nullptr:
// at most 16 rows, fp32-exact, `act` fp32 and scratch of int4_batch_exact_scratch_bytes(k); otherwise bf16
// activations in the prefill GEMM's k order. The two predicates say where each form is the faster kernel.
size_t int4_batch_exact_scratch_bytes(size_t k);
bool int4_batch_bf16_wins(size_t m, size_t n, size_t k, size_t gs);
bool int4_batch_exact_wins(size_t m, size_t n, size_t k, size_t gs);
bool int4_batch_ready(yscv_cuda_ctx *ctx);   // its workspace is there, or could be allocated now
// With *parts > 1 (bf16 form; int4_batch_parts() says how many are wanted) `out` has room for so many partial sums
// [part][m][n], whose sum in that order is the result; *parts then says how many there are. act == nullptr: `scratch` holds the exact form's terms already.
int int4_batch_gemm(yscv_cuda_ctx *ctx, const uint8_t *wq, const float *scales, const float *act, const void *act_bf16, float *out,
                    size_t m, size_t n, size_t k, void *scratch, int *parts = nullptr);
int int4_batch_parts(yscv_cuda_ctx *ctx, size_t m, size_t n, size_t k);

// A matmul's activations in the form it takes them best, written by the operator in front of it (act_forms.cuh).
int int4_act_form(yscv_cuda_ctx *ctx, const yscv_cuda_int4_weight *w, size_t m);
size_t act_bytes(int form, size_t m, size_t k);
ActOut act_out(int form, size_t m, size_t k, void *buffer);
// Partial sums that int4_matmul_form leaves where there is room for them (1: the result itself); its `parts` is
// the room, and then what there is.
int int4_form_parts(yscv_cuda_ctx *ctx, const yscv_cuda_int4_weight *w, int form, size_t m);
int int4_matmul_form(yscv_cuda_ctx *ctx, const yscv_cuda_int4_weight *w, const ActOut &act, float *out, int *parts);

// decoder_ops.cu, the operators between the matmuls. Inputs that are `parts` partial sums lie `pitch` floats apart.
int norm_form(yscv_cuda_ctx *ctx, const float *x, const float *delta, int parts, size_t pitch, const float *gamma, float eps,
              size_t rows, size_t row0, size_t row_step, size_t hidden, float *x_out, const ActOut &out, bool between);
int swiglu_form(yscv_cuda_ctx *ctx, const float *gate_up, int parts, size_t pitch, size_t rows, size_t inter, const ActOut &out, bool between);
template <typename KV>
int rope_append_form(yscv_cuda_ctx *ctx, const float *qkv, int parts, size_t pitch, float *q_out, size_t q_out_stride, size_t batch,
                     size_t seq, size_t n_q, size_t n_kv, size_t d_head, float theta, const int32_t *d_pos, KV *kcache, KV *vcache,
                     float *kscale, float *vscale, size_t max_seq);
template <typename KV>
int gqa_attention_form(yscv_cuda_ctx *ctx, const float *d_q, size_t q_stride, size_t batch, size_t seq_q, size_t n_q, size_t n_kv,
                       size_t d_head, const KV *d_kcache, const KV *d_vcache, const float *d_kscale, const float *d_vscale,
                       size_t max_seq, const int32_t *d_pos, int causal, const ActOut &out);
// gqa_decode_fused.cu: RoPE, cache append and attention of one position per sequence, for a chain in which nothing
// between the two kernels in front of it and the end of the step before touches the caches or the position
bool gqa_decode_fused_wins(const yscv_cuda_ctx *ctx, int form, bool kv_int8, size_t batch, size_t n_q, size_t n_kv, size_t d_head, size_t max_seq);
template <typename KV>
int gqa_decode_fused(yscv_cuda_ctx *ctx, const float *qkv, int parts, size_t pitch, size_t batch, size_t n_q, size_t n_kv, size_t d_head,
                     float theta, const int32_t *d_pos, KV *kcache, KV *vcache, float *kscale, float *vscale, size_t max_seq, const ActOut &out);
bool gqa_attention_writes(int form, size_t seq_q, size_t d_head, size_t max_seq);   // forms other than ACT_F32

// gqa_prefill_tc.cu: attention of seq_q >= 16 query positions per sequence over a cache (KV = float or
// int8_t), head size 64 or 128, at most 128 query heads per KV head, 16-byte aligned caches and output
template <typename KV>
int gqa_prefill_tc(yscv_cuda_ctx *ctx, const float *q, size_t q_stride, size_t batch, size_t seq_q, size_t n_q, size_t n_kv,
                   size_t d_head, const KV *kc, const KV *vc, const float *kscale, const float *vscale, size_t max_seq,
                   const int32_t *pos, int causal, float *out);

// int4_pack.cu
int pack_int4(yscv_cuda_ctx *ctx, const float *d_weights, size_t m_w, size_t k, size_t gs,
              uint8_t *d_packed, float *d_scales);

int int4_from_matmulnbits(yscv_cuda_ctx *ctx, const uint8_t *d_src, uint8_t *d_dst, size_t bytes);

// int8_gemm.cu
int pack_i8_b(yscv_cuda_ctx *ctx, const int8_t *d_b, size_t k, size_t n, int8_t *d_bt,
              int32_t *d_colsum, size_t kp);
int int8_gemm(yscv_cuda_ctx *ctx, const void *d_a, const yscv_cuda_i8b *b, size_t m, void *d_out,
              int a_unsigned, int a_zp, int mode, float composite, float y_zp, int qmin, int qmax,
              int round_mode, const int32_t *d_corr = nullptr, const float *d_comp_pc = nullptr,
              int relu = 0);

}  // namespace yscv
