//! Raw declarations of libyscv_cuda.so (include/yscv_cuda.h). Generated by
//! bindings/rust/gen_sys.py from the header: edit the header, not this file.
#![allow(non_camel_case_types)]

use core::ffi::{c_char, c_int, c_void};

#[repr(C)]
pub struct yscv_cuda_ctx {
    _private: [u8; 0],
}

#[repr(C)]
pub struct yscv_cuda_int4_weight {
    _private: [u8; 0],
}

#[repr(C)]
pub struct yscv_cuda_i8b {
    _private: [u8; 0],
}

#[repr(C)]
pub struct yscv_cuda_registry {
    _private: [u8; 0],
}

#[repr(C)]
pub struct yscv_cuda_decode_plan {
    _private: [u8; 0],
}

#[repr(C)]
pub struct yscv_cuda_tp_comm {
    _private: [u8; 0],
}

#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct yscv_cuda_quant_stats {
    pub int4_gemv_calls: u64,
    pub int4_gemm_calls: u64,
    pub int4_generic_calls: u64,
    pub int8_gemm_calls: u64,
    pub qlinear_matmul_calls: u64,
    pub matmul_integer_calls: u64,
    pub requant_calls: u64,
    pub decode_step_calls: u64,
    pub cpu_fallbacks: u64,
}

#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct yscv_cuda_requant {
    pub a_is_unsigned: c_int,
    pub a_zero_point: i32,
    pub composite: f32,
    pub y_zero_point: f32,
    pub qmin: i32,
    pub qmax: i32,
    pub round_mode: c_int,
}

#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct yscv_cuda_decode_layer {
    pub qkv: *const yscv_cuda_int4_weight,
    pub o: *const yscv_cuda_int4_weight,
    pub gate_up: *const yscv_cuda_int4_weight,
    pub down: *const yscv_cuda_int4_weight,
    pub d_gamma_attn: *const f32,
    pub d_gamma_mlp: *const f32,
    pub d_kcache: *mut c_void,
    pub d_vcache: *mut c_void,
    pub d_kscale: *mut f32,
    pub d_vscale: *mut f32,
}

#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct yscv_cuda_decode_options {
    pub variant: c_int,
    pub max_tiles: c_int,
    pub k_chunk: c_int,
    pub attention_form: c_int,
    pub spin_limit: c_int,
    pub tp: *const yscv_cuda_tp_comm,
    pub kv_int8: c_int,
    pub batch: c_int,
}

pub const YSCV_CUDA_OK: c_int = 0;
pub const YSCV_CUDA_ERR_BAD_ARG: c_int = -1;
pub const YSCV_CUDA_ERR_CUDA: c_int = -2;
pub const YSCV_CUDA_ERR_UNSUPPORTED: c_int = -3;
pub const YSCV_CUDA_ERR_TIMEOUT: c_int = -4;
pub const YSCV_CUDA_ERR_NO_DEVICE: c_int = -5;
pub const YSCV_CUDA_WEIGHT_MATMUL_KN: c_int = 0;
pub const YSCV_CUDA_WEIGHT_GEMM_NK: c_int = 1;
pub const YSCV_CUDA_WEIGHT_GEMM_KN: c_int = 2;
pub const YSCV_CUDA_TP_HANDLE_BYTES: usize = 64;

extern "C" {
    pub fn yscv_cuda_ctx_create(device: c_int, out: *mut *mut yscv_cuda_ctx) -> c_int;
    pub fn yscv_cuda_ctx_create_on_stream(device: c_int, cuda_stream: *mut c_void, out: *mut *mut yscv_cuda_ctx) -> c_int;
    pub fn yscv_cuda_ctx_destroy(ctx: *mut yscv_cuda_ctx);
    pub fn yscv_cuda_ctx_synchronize(ctx: *mut yscv_cuda_ctx) -> c_int;
    pub fn yscv_cuda_ctx_device_status(ctx: *mut yscv_cuda_ctx, status: *mut c_int) -> c_int;
    pub fn yscv_cuda_last_error() -> *const c_char;
    pub fn yscv_cuda_last_kernel(ctx: *const yscv_cuda_ctx) -> *const c_char;
    pub fn yscv_cuda_ctx_launch_count(ctx: *const yscv_cuda_ctx) -> u64;
    pub fn yscv_cuda_dispatch_report(ctx: *const yscv_cuda_ctx) -> *const c_char;
    pub fn yscv_cuda_quant_stats_read(out: *mut yscv_cuda_quant_stats);
    pub fn yscv_cuda_quant_stats_reset();
    pub fn yscv_cuda_ctx_set_int4_prefill_exact(ctx: *mut yscv_cuda_ctx, exact: c_int) -> c_int;
    pub fn yscv_cuda_ctx_set_int4_prefill_cta_pairs(ctx: *mut yscv_cuda_ctx, enable: c_int) -> c_int;
    pub fn yscv_cuda_ctx_set_int8_cta_pairs(ctx: *mut yscv_cuda_ctx, mode: c_int) -> c_int;
    pub fn yscv_cuda_ctx_set_int8_tail_split(ctx: *mut yscv_cuda_ctx, enable: c_int) -> c_int;
    pub fn yscv_cuda_ctx_set_attention_tensor_cores(ctx: *mut yscv_cuda_ctx, enable: c_int) -> c_int;
    pub fn yscv_cuda_ctx_set_f32_tensor_cores(ctx: *mut yscv_cuda_ctx, enable: c_int) -> c_int;
    pub fn yscv_cuda_ctx_profile_enable(ctx: *mut yscv_cuda_ctx, enable: c_int) -> c_int;
    pub fn yscv_cuda_ctx_profile_read(ctx: *mut yscv_cuda_ctx, launches: *mut u64, total_ms: *mut f64) -> c_int;
    pub fn yscv_cuda_packed_int4_gemv(ctx: *mut yscv_cuda_ctx, weight_packed: *const u8, scales: *const f32, activation: *const f32, output: *mut f32, m_w: usize, k: usize, group_size: usize) -> c_int;
    pub fn yscv_cuda_packed_int4_gemm(ctx: *mut yscv_cuda_ctx, weight_packed: *const u8, scales: *const f32, activation: *const f32, output: *mut f32, m: usize, n: usize, k: usize, group_size: usize) -> c_int;
    pub fn yscv_cuda_pack_int4_symmetric_per_group(ctx: *mut yscv_cuda_ctx, weights: *const f32, m_w: usize, k: usize, group_size: usize, packed: *mut u8, scales: *mut f32) -> c_int;
    pub fn yscv_cuda_int4_weight_upload(ctx: *mut yscv_cuda_ctx, packed: *const u8, scales: *const f32, m_w: usize, k: usize, group_size: usize, out: *mut *mut yscv_cuda_int4_weight) -> c_int;
    pub fn yscv_cuda_int4_weight_wrap(d_packed: *const u8, d_scales: *const f32, m_w: usize, k: usize, group_size: usize, out: *mut *mut yscv_cuda_int4_weight) -> c_int;
    pub fn yscv_cuda_int4_weight_free(w: *mut yscv_cuda_int4_weight);
    pub fn yscv_cuda_int4_matmul_dev(ctx: *mut yscv_cuda_ctx, w: *const yscv_cuda_int4_weight, d_activation: *const f32, d_output: *mut f32, m: usize) -> c_int;
    pub fn yscv_cuda_int4_matmul_act_dev(ctx: *mut yscv_cuda_ctx, w: *const yscv_cuda_int4_weight, d_activation_bf16: *const c_void, d_output: *mut f32, m: usize) -> c_int;
    pub fn yscv_cuda_int4_matmul(ctx: *mut yscv_cuda_ctx, w: *const yscv_cuda_int4_weight, activation: *const f32, output: *mut f32, m: usize) -> c_int;
    pub fn yscv_cuda_int4_matmul_dev_static(ctx: *mut yscv_cuda_ctx, d_packed: *const u8, d_scales: *const f32, n: usize, k: usize, group_size: usize, d_activation: *const f32, d_output: *mut f32, m: usize) -> c_int;
    pub fn yscv_cuda_int4_from_matmulnbits(src: *const u8, dst: *mut u8, bytes: usize) -> c_int;
    pub fn yscv_cuda_int4_from_matmulnbits_dev(ctx: *mut yscv_cuda_ctx, d_src: *const u8, d_dst: *mut u8, bytes: usize) -> c_int;
    pub fn yscv_cuda_int4_to_matmulnbits(src: *const u8, dst: *mut u8, bytes: usize) -> c_int;
    pub fn yscv_cuda_int4_weight_from_f32(ctx: *mut yscv_cuda_ctx, weight: *const f32, dim0: usize, dim1: usize, layout: c_int, group_size: usize, out: *mut *mut yscv_cuda_int4_weight) -> c_int;
    pub fn yscv_cuda_int4_weight_rows(w: *const yscv_cuda_int4_weight) -> usize;
    pub fn yscv_cuda_int4_weight_k(w: *const yscv_cuda_int4_weight) -> usize;
    pub fn yscv_cuda_int4_weight_group_size(w: *const yscv_cuda_int4_weight) -> usize;
    pub fn yscv_cuda_int4_weight_download(ctx: *mut yscv_cuda_ctx, w: *const yscv_cuda_int4_weight, packed: *mut u8, scales: *mut f32) -> c_int;
    pub fn yscv_cuda_int4_container_size(m_w: usize, k: usize, group_size: usize) -> usize;
    pub fn yscv_cuda_int4_container_write(packed: *const u8, scales: *const f32, m_w: usize, k: usize, group_size: usize, dst: *mut u8, capacity: usize, written: *mut usize) -> c_int;
    pub fn yscv_cuda_int4_container_read(src: *const u8, len: usize, m_w: *mut usize, k: *mut usize, group_size: *mut usize, packed: *mut *const u8, scales: *mut *const f32) -> c_int;
    pub fn yscv_cuda_int4_weight_from_container(ctx: *mut yscv_cuda_ctx, src: *const u8, len: usize, out: *mut *mut yscv_cuda_int4_weight) -> c_int;
    pub fn yscv_cuda_pack_int4_dev(ctx: *mut yscv_cuda_ctx, d_weights: *const f32, m_w: usize, k: usize, group_size: usize, d_packed: *mut u8, d_scales: *mut f32) -> c_int;
    pub fn yscv_cuda_int8_matmul(ctx: *mut yscv_cuda_ctx, a: *const i8, b: *const i8, m: usize, k: usize, n: usize, out: *mut i32) -> c_int;
    pub fn yscv_cuda_pack_i8_b_for_matmul(ctx: *mut yscv_cuda_ctx, b: *const i8, k: usize, n: usize, out: *mut *mut yscv_cuda_i8b) -> c_int;
    pub fn yscv_cuda_pack_i8_b_dev(ctx: *mut yscv_cuda_ctx, d_b: *const i8, k: usize, n: usize, out: *mut *mut yscv_cuda_i8b) -> c_int;
    pub fn yscv_cuda_i8b_free(b: *mut yscv_cuda_i8b);
    pub fn yscv_cuda_i8b_set_zero_point(b: *mut yscv_cuda_i8b, b_zero_point: i32) -> c_int;
    pub fn yscv_cuda_i8b_k(b: *const yscv_cuda_i8b) -> usize;
    pub fn yscv_cuda_i8b_n(b: *const yscv_cuda_i8b) -> usize;
    pub fn yscv_cuda_int8_matmul_prepacked(ctx: *mut yscv_cuda_ctx, a: *const i8, b: *const yscv_cuda_i8b, m: usize, out: *mut i32) -> c_int;
    pub fn yscv_cuda_int8_matmul_prepacked_dev(ctx: *mut yscv_cuda_ctx, d_a: *const i8, b: *const yscv_cuda_i8b, m: usize, d_out: *mut i32) -> c_int;
    pub fn yscv_cuda_qlinear_matmul(ctx: *mut yscv_cuda_ctx, a: *const c_void, b: *const yscv_cuda_i8b, m: usize, rq: *const yscv_cuda_requant, out: *mut c_void) -> c_int;
    pub fn yscv_cuda_qlinear_matmul_dev(ctx: *mut yscv_cuda_ctx, d_a: *const c_void, b: *const yscv_cuda_i8b, m: usize, rq: *const yscv_cuda_requant, d_out: *mut c_void) -> c_int;
    pub fn yscv_cuda_matmul_integer(ctx: *mut yscv_cuda_ctx, a: *const c_void, a_is_unsigned: c_int, a_zero_point: i32, b: *const yscv_cuda_i8b, m: usize, out: *mut i32) -> c_int;
    pub fn yscv_cuda_matmul_integer_dev(ctx: *mut yscv_cuda_ctx, d_a: *const c_void, a_is_unsigned: c_int, a_zero_point: i32, b: *const yscv_cuda_i8b, m: usize, d_out: *mut i32) -> c_int;
    pub fn yscv_cuda_requant_i32_row_to_i8(ctx: *mut yscv_cuda_ctx, acc: *const i32, bias: *const i32, composite: f32, y_zero_point: f32, relu: c_int, out: *mut i8, len: usize, c: usize) -> c_int;
    pub fn yscv_cuda_requant_i32_row_to_i8_dev(ctx: *mut yscv_cuda_ctx, d_acc: *const i32, d_bias: *const i32, composite: f32, y_zero_point: f32, relu: c_int, d_out: *mut i8, len: usize, c: usize) -> c_int;
    pub fn yscv_cuda_registry_create(out: *mut *mut yscv_cuda_registry) -> c_int;
    pub fn yscv_cuda_registry_destroy(reg: *mut yscv_cuda_registry);
    pub fn yscv_cuda_registry_put_int4(reg: *mut yscv_cuda_registry, name: *const c_char, w: *mut yscv_cuda_int4_weight) -> c_int;
    pub fn yscv_cuda_registry_put_i8b(reg: *mut yscv_cuda_registry, name: *const c_char, b: *mut yscv_cuda_i8b) -> c_int;
    pub fn yscv_cuda_registry_get_int4(reg: *const yscv_cuda_registry, name: *const c_char) -> *const yscv_cuda_int4_weight;
    pub fn yscv_cuda_registry_get_i8b(reg: *const yscv_cuda_registry, name: *const c_char) -> *const yscv_cuda_i8b;
    pub fn yscv_cuda_registry_len(reg: *const yscv_cuda_registry) -> usize;
    pub fn yscv_cuda_registry_register_matmul_weight(ctx: *mut yscv_cuda_ctx, reg: *mut yscv_cuda_registry, name: *const c_char, weight: *const f32, dim0: usize, dim1: usize, layout: c_int, group_size: usize, packed: *mut c_int) -> c_int;
    pub fn yscv_cuda_registry_register_i8_weight(ctx: *mut yscv_cuda_ctx, reg: *mut yscv_cuda_registry, name: *const c_char, b: *const i8, k: usize, n: usize, prepacked: *mut c_int) -> c_int;
    pub fn yscv_cuda_should_prepack_i8_b(k: usize, n: usize) -> c_int;
    pub fn yscv_cuda_should_use_prepacked_i8_b(m: usize, k: usize, n: usize) -> c_int;
    pub fn yscv_cuda_embedding_dev(ctx: *mut yscv_cuda_ctx, d_weight: *const f32, vocab: usize, dim: usize, d_tokens: *const i32, rows: usize, d_out: *mut f32) -> c_int;
    pub fn yscv_cuda_add_rms_norm_dev(ctx: *mut yscv_cuda_ctx, d_x: *const f32, d_delta: *const f32, d_gamma: *const f32, eps: f32, rows: usize, hidden: usize, d_x_out: *mut f32, d_normed: *mut f32) -> c_int;
    pub fn yscv_cuda_add_rms_norm_act_dev(ctx: *mut yscv_cuda_ctx, d_x: *const f32, d_delta: *const f32, d_gamma: *const f32, eps: f32, rows: usize, hidden: usize, d_x_out: *mut f32, d_normed_act: *mut c_void) -> c_int;
    pub fn yscv_cuda_rope_kv_append_dev(ctx: *mut yscv_cuda_ctx, d_qkv: *mut f32, batch: usize, seq: usize, n_q: usize, n_kv: usize, d_head: usize, theta: f32, d_pos: *const i32, d_kcache: *mut f32, d_vcache: *mut f32, max_seq: usize) -> c_int;
    pub fn yscv_cuda_gqa_attention_dev(ctx: *mut yscv_cuda_ctx, d_q: *const f32, q_stride: usize, batch: usize, seq_q: usize, n_q: usize, n_kv: usize, d_head: usize, d_kcache: *const f32, d_vcache: *const f32, max_seq: usize, d_pos: *const i32, causal: c_int, d_out: *mut f32) -> c_int;
    pub fn yscv_cuda_rope_kv_append_i8_dev(ctx: *mut yscv_cuda_ctx, d_qkv: *mut f32, batch: usize, seq: usize, n_q: usize, n_kv: usize, d_head: usize, theta: f32, d_pos: *const i32, d_kcache: *mut i8, d_kscale: *mut f32, d_vcache: *mut i8, d_vscale: *mut f32, max_seq: usize) -> c_int;
    pub fn yscv_cuda_gqa_attention_i8_dev(ctx: *mut yscv_cuda_ctx, d_q: *const f32, q_stride: usize, batch: usize, seq_q: usize, n_q: usize, n_kv: usize, d_head: usize, d_kcache: *const i8, d_kscale: *const f32, d_vcache: *const i8, d_vscale: *const f32, max_seq: usize, d_pos: *const i32, causal: c_int, d_out: *mut f32) -> c_int;
    pub fn yscv_cuda_swiglu_dev(ctx: *mut yscv_cuda_ctx, d_gate_up: *const f32, rows: usize, inter: usize, d_out: *mut f32) -> c_int;
    pub fn yscv_cuda_swiglu_act_dev(ctx: *mut yscv_cuda_ctx, d_gate_up: *const f32, rows: usize, inter: usize, d_out_act: *mut c_void) -> c_int;
    pub fn yscv_cuda_f32_matmul_dev(ctx: *mut yscv_cuda_ctx, d_w: *const f32, d_x: *const f32, m: usize, n: usize, k: usize, d_out: *mut f32) -> c_int;
    pub fn yscv_cuda_argmax_last_dev(ctx: *mut yscv_cuda_ctx, d_logits: *const f32, rows: usize, vocab: usize, d_out: *mut i32) -> c_int;
    pub fn yscv_cuda_advance_pos_dev(ctx: *mut yscv_cuda_ctx, d_pos: *mut i32, by: c_int) -> c_int;
    pub fn yscv_cuda_int8_matmul_requant_per_channel_dev(ctx: *mut yscv_cuda_ctx, d_a: *const i8, b: *const yscv_cuda_i8b, m: usize, d_corr: *const i32, d_composite: *const f32, y_zero_point: f32, d_out: *mut i8) -> c_int;
    pub fn yscv_cuda_int8_matmul_requant_per_channel(ctx: *mut yscv_cuda_ctx, a: *const i8, b: *const yscv_cuda_i8b, m: usize, corr: *const i32, composite: *const f32, y_zero_point: f32, out: *mut i8) -> c_int;
    pub fn yscv_cuda_int8_matmul_requant_i8_dev(ctx: *mut yscv_cuda_ctx, d_a: *const i8, b: *const yscv_cuda_i8b, m: usize, d_bias: *const i32, composite: f32, y_zero_point: f32, relu: c_int, d_out: *mut i8) -> c_int;
    pub fn yscv_cuda_int8_matmul_requant_i8(ctx: *mut yscv_cuda_ctx, a: *const i8, b: *const yscv_cuda_i8b, m: usize, bias: *const i32, composite: f32, y_zero_point: f32, relu: c_int, out: *mut i8) -> c_int;
    pub fn yscv_cuda_decode_plan_create(ctx: *mut yscv_cuda_ctx, layers: *const yscv_cuda_decode_layer, n_layers: usize, hidden: usize, inter: usize, n_q: usize, n_kv: usize, d_head: usize, max_seq: usize, eps: f32, rope_theta: f32, out: *mut *mut yscv_cuda_decode_plan) -> c_int;
    pub fn yscv_cuda_tp_comm_create(ctx: *mut yscv_cuda_ctx, rank: c_int, world: c_int, max_rows: usize, out: *mut *mut yscv_cuda_tp_comm, handle_out: *mut u8) -> c_int;
    pub fn yscv_cuda_tp_comm_connect(comm: *mut yscv_cuda_tp_comm, handles: *const u8) -> c_int;
    pub fn yscv_cuda_tp_comm_destroy(comm: *mut yscv_cuda_tp_comm);
    pub fn yscv_cuda_tp_comm_connect_unanswered(comm: *mut yscv_cuda_tp_comm) -> c_int;
    pub fn yscv_cuda_decode_plan_create_ex(ctx: *mut yscv_cuda_ctx, layers: *const yscv_cuda_decode_layer, n_layers: usize, hidden: usize, inter: usize, n_q: usize, n_kv: usize, d_head: usize, max_seq: usize, eps: f32, rope_theta: f32, opt: *const yscv_cuda_decode_options, out: *mut *mut yscv_cuda_decode_plan) -> c_int;
    pub fn yscv_cuda_decode_plan_check(ctx: *mut yscv_cuda_ctx, plan: *mut yscv_cuda_decode_plan) -> c_int;
    pub fn yscv_cuda_decode_plan_step_dev(ctx: *mut yscv_cuda_ctx, plan: *const yscv_cuda_decode_plan, d_embedding: *const f32, vocab: usize, d_token: *const i32, d_pos: *const i32, d_x: *mut f32) -> c_int;
    pub fn yscv_cuda_decode_plan_step_token_dev(ctx: *mut yscv_cuda_ctx, plan: *const yscv_cuda_decode_plan, d_embedding: *const f32, vocab: usize, d_token: *mut i32, d_pos: *mut i32, d_final_gamma: *const f32, d_lm_head: *const f32, d_x: *mut f32, d_logits: *mut f32) -> c_int;
    pub fn yscv_cuda_decode_plan_step_token_shard_dev(ctx: *mut yscv_cuda_ctx, plan: *const yscv_cuda_decode_plan, d_embedding: *const f32, vocab: usize, d_token: *mut i32, d_pos: *mut i32, d_final_gamma: *const f32, d_lm_head_rows: *const f32, lm_row0: usize, lm_rows: usize, d_x: *mut f32, d_logits: *mut f32) -> c_int;
    pub fn yscv_cuda_decode_plan_free(plan: *mut yscv_cuda_decode_plan);
    pub fn yscv_cuda_decoder_layers_workspace(ctx: *mut yscv_cuda_ctx, layers: *const yscv_cuda_decode_layer, n_layers: usize, hidden: usize, inter: usize, n_q: usize, n_kv: usize, d_head: usize, batch: usize, seq: usize, bytes: *mut usize) -> c_int;
    pub fn yscv_cuda_decoder_layers_dev(ctx: *mut yscv_cuda_ctx, layers: *const yscv_cuda_decode_layer, n_layers: usize, hidden: usize, inter: usize, n_q: usize, n_kv: usize, d_head: usize, max_seq: usize, eps: f32, rope_theta: f32, kv_int8: c_int, batch: usize, seq: usize, d_pos: *const i32, d_x: *mut f32, d_final_gamma: *const f32, d_last: *mut f32, d_workspace: *mut c_void, workspace_bytes: usize) -> c_int;
}
