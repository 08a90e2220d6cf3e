// The layers of a Llama-shape int4 decoder as a chain of the library's kernels, for any number of sequences and
// positions (a decode step, a prompt pass). The same operators as the stand-alone entry points, in the order of the
// reference's exported graph (apps/llm-bench/src/main.rs:491-561); what one call over the layers can do and
// single calls cannot is hand results over as they are: an operator writes the activations in the form that the
// matmul behind it takes (act_forms.cuh), and a matmul whose k was cut into slices leaves them for the operator behind
// it to add. A launch of a small decode batch is 1.5 to 2 us of latency whatever it does: 32 sequences at the 1B shape
// (22 layers) had 15 launches per layer, 8 sequences 13; now 8: norm, QKV, attention, output, norm, gate/up, SwiGLU, down
// (10 with RoPE, split and merge apart over long caches, and one more behind a matmul whose tiles several CTAs share).
#include "common.cuh"
#include "kernels.cuh"

using namespace yscv;

namespace {

struct Shape {
    size_t hidden, inter, n_q, n_kv, d, batch, seq;
    size_t rows() const { return batch * seq; }
    size_t qkv() const { return (n_q + 2 * n_kv) * d; }
};

// Byte offsets of the buffers of a pass, and the room for partial sums of each matmul
struct Layout {
    size_t act, qkv, q, down, gu, total;
    int parts_qkv, parts_o, parts_gu, parts_down;
};

// What the form of a weight's activations depends on besides its shape, which check() makes the same in every layer
bool alike(const yscv_cuda_int4_weight *a, const yscv_cuda_int4_weight *b) {
    auto skew = [](const yscv_cuda_int4_weight *w) { return ((reinterpret_cast<uintptr_t>(w->d_packed) | reinterpret_cast<uintptr_t>(w->d_scales)) & 15) != 0; };
    return a->group_size == b->group_size && skew(a) == skew(b);
}

// Room for the activations in every layer's form, and for the partial sums of the layer that leaves most
Layout layout(yscv_cuda_ctx *ctx, const yscv_cuda_decode_layer *layers, size_t n_layers, const Shape &s, bool apart) {
    const size_t m = s.rows();
    Layout o = {};
    size_t at = 0, act = 0;
    auto take = [&](size_t bytes) {
        const size_t p = at;
        at += (bytes + 255) / 256 * 256;
        return p;
    };
    auto fit = [&](const yscv_cuda_int4_weight *w, int &parts) {
        const int form = int4_act_form(ctx, w, m);
        act = std::max(act, std::max(act_bytes(ACT_F32, m, w->k), act_bytes(form, m, w->k)));
        // (run() may find the library's workspace there that was not to be had a moment ago)
        if (int4_batch_exact_wins(m, w->m_w, w->k, w->group_size)) act = std::max(act, act_bytes(ACT_TERMS, m, w->k));
        parts = std::max(parts, apart ? int4_form_parts(ctx, w, form, m) : 1);
    };
    const yscv_cuda_decode_layer &l0 = layers[0];
    for (size_t i = 0; i < n_layers; ++i) {
        const yscv_cuda_decode_layer &l = layers[i];
        if (i > 0 && alike(l.qkv, l0.qkv) && alike(l.o, l0.o) && alike(l.gate_up, l0.gate_up) && alike(l.down, l0.down)) continue;
        fit(l.qkv, o.parts_qkv);
        fit(l.o, o.parts_o);
        fit(l.gate_up, o.parts_gu);
        fit(l.down, o.parts_down);
    }
    o.act = take(act);
    o.qkv = take(o.parts_qkv * m * s.qkv() * sizeof(float));
    o.q = take(o.parts_qkv > 1 ? m * s.n_q * s.d * sizeof(float) : 0);
    // (the output projection's sums are used up before the down projection's are written)
    o.down = take(std::max(o.parts_o, o.parts_down) * m * s.hidden * sizeof(float));
    o.gu = take(o.parts_gu * m * 2 * s.inter * sizeof(float));
    o.total = at;
    return o;
}

int check(yscv_cuda_ctx *ctx, const yscv_cuda_decode_layer *layers, size_t n_layers, const Shape &s, int kv_int8) {
    if (!ctx || !layers) return fail(YSCV_CUDA_ERR_BAD_ARG, "null argument");
    if (n_layers == 0 || s.n_kv == 0 || s.n_q % s.n_kv != 0 || s.d == 0 || s.d % 2 != 0)
        return fail(YSCV_CUDA_ERR_BAD_ARG, "bad decoder shape: %zu layers, %zu / %zu heads of %zu", n_layers, s.n_q, s.n_kv, s.d);
    if (s.hidden == 0 || s.inter == 0 || s.hidden % 8 != 0 || s.inter % 8 != 0 || s.d % 8 != 0 || s.hidden > 8192)
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "hidden=%zu, inter=%zu and d_head=%zu must be multiples of 8, hidden at most 8192", s.hidden, s.inter, s.d);
    for (size_t i = 0; i < n_layers; ++i) {
        const yscv_cuda_decode_layer &l = layers[i];
        if (!l.qkv || !l.o || !l.gate_up || !l.down || !l.d_gamma_attn || !l.d_gamma_mlp || !l.d_kcache || !l.d_vcache ||
            (kv_int8 && (!l.d_kscale || !l.d_vscale)))
            return fail(YSCV_CUDA_ERR_BAD_ARG, "layer %zu has a null member", i);
        if (l.qkv->m_w != s.qkv() || l.qkv->k != s.hidden || l.o->m_w != s.hidden || l.o->k != s.n_q * s.d || l.gate_up->m_w != 2 * s.inter ||
            l.gate_up->k != s.hidden || l.down->m_w != s.hidden || l.down->k != s.inter)
            return fail(YSCV_CUDA_ERR_BAD_ARG, "the weights of layer %zu do not have the decoder's shape", i);
        if ((reinterpret_cast<uintptr_t>(l.d_gamma_attn) | reinterpret_cast<uintptr_t>(l.d_gamma_mlp)) & 15)
            return fail(YSCV_CUDA_ERR_UNSUPPORTED, "the gammas of layer %zu must be 16-byte aligned", i);
    }
    return YSCV_CUDA_OK;
}

bool caches_aligned(const yscv_cuda_decode_layer &l) {
    return ((reinterpret_cast<uintptr_t>(l.d_kcache) | reinterpret_cast<uintptr_t>(l.d_vcache)) & 15) == 0;
}

template <typename KV>
int run(yscv_cuda_ctx *ctx, const yscv_cuda_decode_layer *layers, size_t n_layers, const Shape &s, const Layout &o, size_t max_seq, float eps,
        float theta, const int32_t *pos, float *x, const float *final_gamma, float *last, unsigned char *ws) {
    const size_t m = s.rows(), H = s.hidden, nq = s.n_q * s.d;
    float *const qkv = reinterpret_cast<float *>(ws + o.qkv), *const gu = reinterpret_cast<float *>(ws + o.gu);
    float *const down = reinterpret_cast<float *>(ws + o.down);
    void *const act = ws + o.act;
    const float *delta = nullptr;
    int parts = 1, rc;
    for (size_t i = 0; i < n_layers; ++i) {
        const yscv_cuda_decode_layer &l = layers[i];
        KV *kc = static_cast<KV *>(l.d_kcache), *vc = static_cast<KV *>(l.d_vcache);
        ActOut a = act_out(int4_act_form(ctx, l.qkv, m), m, H, act);
        if ((rc = norm_form(ctx, x, delta, parts, m * H, l.d_gamma_attn, eps, m, 0, 1, H, x, a, true))) return rc;
        parts = o.parts_qkv;
        if ((rc = int4_matmul_form(ctx, l.qkv, a, qkv, &parts))) return rc;
        const int form = int4_act_form(ctx, l.o, m);
        const int own = form == ACT_TERMS ? (int)ACT_F32 : form;   // (a block of terms spans heads)
        if (s.seq == 1 && caches_aligned(l) && gqa_decode_fused_wins(ctx, own, sizeof(KV) == 1, s.batch, s.n_q, s.n_kv, s.d, max_seq)) {
            a = act_out(own, m, nq, act);
            if ((rc = gqa_decode_fused<KV>(ctx, qkv, parts, m * s.qkv(), s.batch, s.n_q, s.n_kv, s.d, theta, pos, kc, vc, l.d_kscale, l.d_vscale, max_seq, a)))
                return rc;
        } else {
            float *const q = parts > 1 ? reinterpret_cast<float *>(ws + o.q) : qkv;
            const size_t q_stride = parts > 1 ? nq : s.qkv();
            if ((rc = rope_append_form<KV>(ctx, qkv, parts, m * s.qkv(), q, q_stride, s.batch, s.seq, s.n_q, s.n_kv, s.d, theta, pos, kc, vc,
                                           l.d_kscale, l.d_vscale, max_seq)))
                return rc;
            a = act_out(gqa_attention_writes(form, s.seq, s.d, max_seq) ? form : (int)ACT_F32, m, nq, act);
            if ((rc = gqa_attention_form<KV>(ctx, q, q_stride, s.batch, s.seq, s.n_q, s.n_kv, s.d, kc, vc, l.d_kscale, l.d_vscale, max_seq, pos, 1, a)))
                return rc;
        }
        parts = o.parts_o;
        if ((rc = int4_matmul_form(ctx, l.o, a, down, &parts))) return rc;
        a = act_out(int4_act_form(ctx, l.gate_up, m), m, H, act);
        if ((rc = norm_form(ctx, x, down, parts, m * H, l.d_gamma_mlp, eps, m, 0, 1, H, x, a, true))) return rc;
        parts = o.parts_gu;
        if ((rc = int4_matmul_form(ctx, l.gate_up, a, gu, &parts))) return rc;
        a = act_out(int4_act_form(ctx, l.down, m), m, s.inter, act);
        if ((rc = swiglu_form(ctx, gu, parts, m * 2 * s.inter, m, s.inter, a, true))) return rc;
        parts = o.parts_down;
        if ((rc = int4_matmul_form(ctx, l.down, a, down, &parts))) return rc;
        delta = down;
    }
    // the final norm of the last position of every sequence
    return norm_form(ctx, x, delta, parts, m * H, final_gamma, eps, s.batch, s.seq - 1, s.seq, H, nullptr, act_out(ACT_F32, s.batch, H, last), true);
}

}  // namespace

extern "C" {

int yscv_cuda_decoder_layers_workspace(yscv_cuda_ctx *ctx, const yscv_cuda_decode_layer *layers, size_t n_layers, size_t hidden, size_t inter,
                                       size_t n_q, size_t n_kv, size_t d_head, size_t batch, size_t seq, size_t *bytes) {
    const Shape s = {hidden, inter, n_q, n_kv, d_head, batch, seq};
    if (!bytes) return fail(YSCV_CUDA_ERR_BAD_ARG, "null argument");
    const int rc = check(ctx, layers, n_layers, s, 0);
    if (rc) return rc;
    YSCV_CUDA_TRY(cudaSetDevice(ctx->device));
    *bytes = batch * seq == 0 ? 0 : layout(ctx, layers, n_layers, s, true).total;
    return YSCV_CUDA_OK;
}

int yscv_cuda_decoder_layers_dev(yscv_cuda_ctx *ctx, const yscv_cuda_decode_layer *layers, size_t n_layers, size_t hidden, size_t inter,
                                 size_t n_q, size_t n_kv, size_t d_head, size_t max_seq, float eps, float rope_theta, int kv_int8,
                                 size_t batch, size_t seq, const int32_t *d_pos, float *d_x, const float *d_final_gamma, float *d_last,
                                 void *d_workspace, size_t workspace_bytes) {
    const Shape s = {hidden, inter, n_q, n_kv, d_head, batch, seq};
    int rc = check(ctx, layers, n_layers, s, kv_int8);
    if (rc) return rc;
    if (!d_pos || !d_x || !d_final_gamma || !d_last) return fail(YSCV_CUDA_ERR_BAD_ARG, "null operand");
    if (max_seq == 0) return fail(YSCV_CUDA_ERR_BAD_ARG, "max_seq must be positive");
    if (batch * seq == 0) return YSCV_CUDA_OK;
    if (!d_workspace) return fail(YSCV_CUDA_ERR_BAD_ARG, "null workspace");
    if ((reinterpret_cast<uintptr_t>(d_x) | reinterpret_cast<uintptr_t>(d_final_gamma) | reinterpret_cast<uintptr_t>(d_last) |
         reinterpret_cast<uintptr_t>(d_workspace)) & 15)
        return fail(YSCV_CUDA_ERR_UNSUPPORTED, "d_x, d_final_gamma, d_last and the workspace must be 16-byte aligned");
    YSCV_CUDA_TRY(cudaSetDevice(ctx->device));
    Layout o = layout(ctx, layers, n_layers, s, true);
    // (room for partial sums is wanted only where the library can use its own workspace, which it may have got since)
    if (o.total > workspace_bytes) o = layout(ctx, layers, n_layers, s, false);
    if (o.total > workspace_bytes)
        return fail(YSCV_CUDA_ERR_BAD_ARG, "workspace of %zu bytes is too small: %zu needed", workspace_bytes, o.total);
    unsigned char *ws = static_cast<unsigned char *>(d_workspace);
    return kv_int8 ? run<int8_t>(ctx, layers, n_layers, s, o, max_seq, eps, rope_theta, d_pos, d_x, d_final_gamma, d_last, ws)
                   : run<float>(ctx, layers, n_layers, s, o, max_seq, eps, rope_theta, d_pos, d_x, d_final_gamma, d_last, ws);
}

}  // extern "C"
