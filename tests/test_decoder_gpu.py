"""The decoder operators one by one, and whole decoders (small, and TinyLlama-1.1B shape)
against the CPU oracle decoder: logits and greedy tokens."""
import numpy as np
import pytest

from yscv_b200 import synth
from yscv_b200.decoder import DecoderConfig, Int4Decoder, TINYLLAMA_1B

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tctx():
    import torch
    import yscv_b200
    s = torch.cuda.Stream()
    c = yscv_b200.Context(0, stream=s.cuda_stream)
    yield c, s
    c.close()


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_operators(tctx, oracle):
    import torch
    ctx, s = tctx
    with torch.cuda.stream(s):
        # RMSNorm with the residual add in front
        x = synth.normal(1, 0, 3 * 512, 1.0).reshape(3, 512)
        dl = synth.normal(1, 1, 3 * 512, 1.0).reshape(3, 512)
        gm = synth.normal(1, 2, 512, 1.0)
        dx, dd, dg = dev(x), dev(dl), dev(gm)
        xo, nm = torch.empty_like(dx), torch.empty_like(dx)
        ctx.add_rms_norm_dev(dx.data_ptr(), dd.data_ptr(), dg.data_ptr(), 1e-5, 3, 512, xo.data_ptr(), nm.data_ptr())
        s.synchronize()
        assert np.array_equal(xo.cpu().numpy(), x + dl)
        assert np.max(np.abs(nm.cpu().numpy() - oracle.rms_norm(x + dl, gm, 1e-5))) < 1e-5
        # in place, as the decoder uses it
        ctx.add_rms_norm_dev(dx.data_ptr(), dd.data_ptr(), dg.data_ptr(), 1e-5, 3, 512, dx.data_ptr(), nm.data_ptr())
        s.synchronize()
        assert np.array_equal(dx.cpu().numpy(), x + dl)
        assert np.max(np.abs(nm.cpu().numpy() - oracle.rms_norm(x + dl, gm, 1e-5))) < 1e-5
        # RoPE + KV append, then attention over the cache, two calls (prefill 5, decode 1)
        B, nq, nkv, d, max_seq = 2, 4, 2, 64, 16
        kc = torch.zeros(B, max_seq, nkv, d, device="cuda")
        vc = torch.zeros_like(kc)
        pos = torch.zeros(1, dtype=torch.int32, device="cuda")
        hist_k = [np.zeros((0, nkv * d), np.float32) for _ in range(B)]
        hist_v = [np.zeros((0, nkv * d), np.float32) for _ in range(B)]
        p = 0
        for seq in (5, 1, 1):
            qkv = synth.normal(2 + p, 0, B * seq * (nq + 2 * nkv) * d, 1.0).reshape(B * seq, -1)
            dq = dev(qkv)
            out = torch.empty(B * seq, nq * d, device="cuda")
            ctx.rope_kv_append_dev(dq.data_ptr(), B, seq, nq, nkv, d, 10000.0, pos.data_ptr(), kc.data_ptr(),
                                   vc.data_ptr(), max_seq)
            ctx.gqa_attention_dev(dq.data_ptr(), (nq + 2 * nkv) * d, B, seq, nq, nkv, d, kc.data_ptr(), vc.data_ptr(),
                                  max_seq, pos.data_ptr(), True, out.data_ptr())
            ctx.advance_pos_dev(pos.data_ptr(), seq)
            s.synchronize()
            got = out.cpu().numpy()
            for b in range(B):
                rows = qkv[b * seq:(b + 1) * seq]
                q, k, v = rows[:, :nq * d], rows[:, nq * d:(nq + nkv) * d], rows[:, (nq + nkv) * d:]
                qr, kr = oracle.rope(q.ravel(), k.ravel(), nq, nkv, d, seq, p, 10000.0)
                hist_k[b] = np.concatenate([hist_k[b], kr.reshape(seq, -1)])
                hist_v[b] = np.concatenate([hist_v[b], v])
                want = oracle.gqa_attention(qr, hist_k[b].ravel(), hist_v[b].ravel(), 1, seq, hist_k[b].shape[0], nq,
                                            nkv, d, True).reshape(seq, -1)
                assert np.max(np.abs(got[b * seq:(b + 1) * seq] - want)) < 2e-5
                assert np.max(np.abs(kc[b, :hist_k[b].shape[0]].reshape(-1, nkv * d).cpu().numpy() - hist_k[b])) < 2e-5
            p += seq
        assert int(pos.item()) == 7
        # SwiGLU
        gu = synth.normal(5, 0, 4 * 2 * 96, 2.0).reshape(4, 192)
        o = torch.empty(4, 96, device="cuda")
        dgu = dev(gu)
        ctx.swiglu_dev(dgu.data_ptr(), 4, 96, o.data_ptr())
        s.synchronize()
        assert np.max(np.abs(o.cpu().numpy() - oracle.silu(gu[:, :96]) * gu[:, 96:])) < 1e-6
        # embedding, fp32 matmul, argmax-last (ties -> last index)
        emb = synth.normal(6, 0, 50 * 64, 1.0).reshape(50, 64)
        tok = np.array([3, 49, 0, 3], np.int32)
        e = torch.empty(4, 64, device="cuda")
        demb, dtok = dev(emb), dev(tok)
        ctx.embedding_dev(demb.data_ptr(), 50, 64, dtok.data_ptr(), 4, e.data_ptr())
        xs = synth.normal(6, 1, 6 * 64, 1.0).reshape(6, 64)
        lg = torch.empty(6, 50, device="cuda")
        dxs = dev(xs)
        ctx.f32_matmul_dev(demb.data_ptr(), dxs.data_ptr(), 6, 50, 64, lg.data_ptr())
        tie = np.zeros((3, 1000), np.float32)
        tie[0, [5, 700, 999]] = 2.0
        tie[1, :] = -1.0
        tie[2, 17] = 1.0
        am = torch.empty(3, dtype=torch.int32, device="cuda")
        dtie = dev(tie)
        ctx.argmax_last_dev(dtie.data_ptr(), 3, 1000, am.data_ptr())
        s.synchronize()
        assert np.array_equal(e.cpu().numpy(), emb[tok])
        assert np.max(np.abs(lg.cpu().numpy() - xs @ emb.T)) < 1e-4
        assert am.cpu().numpy().tolist() == [999, 999, 17]
        assert [oracle.argmax_last(tie[i]) for i in range(3)] == [999, 999, 17]
        wide = synth.normal(8, 0, 2 * 32000, 1.0).reshape(2, 32000)
        wide[0, [100, 31999]] = 9.0     # tie across partial blocks: the last index wins
        wide[1, [7, 15000, 15001]] = 9.0
        dwide = dev(wide)
        am2 = torch.empty(2, dtype=torch.int32, device="cuda")
        ctx.argmax_last_dev(dwide.data_ptr(), 2, 32000, am2.data_ptr())
        s.synchronize()
        assert am2.cpu().numpy().tolist() == [31999, 15001]


def test_split_attention_long_cache(tctx, oracle):
    """Decode attention over a long cache takes the split-key kernel; same result."""
    import torch
    ctx, s = tctx
    B, nq, nkv, d, max_seq, filled = 2, 8, 2, 128, 1500, 1203
    with torch.cuda.stream(s):
        k = synth.normal(31, 0, B * filled * nkv * d, 1.0).reshape(B, filled, nkv * d)
        v = synth.normal(31, 1, B * filled * nkv * d, 1.0).reshape(B, filled, nkv * d)
        kc = torch.zeros(B, max_seq, nkv * d, device="cuda")
        vc = torch.zeros_like(kc)
        kc[:, :filled] = dev(k)
        vc[:, :filled] = dev(v)
        q = synth.normal(31, 2, B * nq * d, 1.0).reshape(B, nq * d)
        dq = dev(q)
        pos = torch.full((1,), filled - 1, dtype=torch.int32, device="cuda")
        out = torch.empty(B, nq * d, device="cuda")
        ctx.gqa_attention_dev(dq.data_ptr(), nq * d, B, 1, nq, nkv, d, kc.data_ptr(), vc.data_ptr(), max_seq,
                              pos.data_ptr(), True, out.data_ptr())
        s.synchronize()
        assert "split" in ctx.last_kernel()
        got = out.cpu().numpy()
        for b in range(B):
            want = oracle.gqa_attention(q[b], k[b].ravel(), v[b].ravel(), 1, 1, filled, nq, nkv, d, True)
            assert np.max(np.abs(got[b] - want)) < 2e-5


def export_weights(dec):
    full = {}
    for l, w in dec.full.items():
        full[l] = {k: (p.cpu().numpy(), s.cpu().numpy()) for k, (p, s) in w.items()}
    return full


def run_parity(tctx, oracle, cfg, n_layers, batch, prompt_len, steps, seed, logit_tol, exact_prefill=True,
               fused_step=True, kv_int8=False, plan_options=None):
    """exact_prefill: the prompt pass uses the fp32-exact int4 kernel (tokens must then match the
    oracle except at rounding-level ties); otherwise the bf16 tensor-core GEMM, whose logits
    may differ by up to 2e-2 (relative Frobenius) and whose tokens may differ only where the
    oracle's own top-2 margin is inside that noise."""
    import torch
    ctx, s = tctx
    ctx.set_int4_prefill_exact(exact_prefill)
    flip_margin = 1e-4 if exact_prefill else 5e-2
    if kv_int8:
        # a cached value that sits on a rounding boundary of its row's int8 grid may land one
        # step (1/127 of the row maximum) apart on the two sides, whose fp32 sums differ in the
        # last bits: the logits then agree to that step's share, not to fp32 rounding
        flip_margin = 1e-2
    dec = Int4Decoder.with_full_weights(ctx, cfg, batch, prompt_len + steps + 1, s, seed=seed, layers=n_layers,
                                        fused_step=fused_step, kv_int8=kv_int8, plan_options=plan_options)
    dec.one_launch = dec.plan is not None   # the form that the caller asked for, also where the chain is the default
    assert (dec.plan is not None) == (fused_step and (batch == 1 or (batch <= 8 and not kv_int8 and cfg.hidden <= 2048)))
    from oracle_decoder import OracleDecoder
    ref = OracleDecoder(oracle, cfg, n_layers, export_weights(dec), dec.embedding.cpu().numpy(),
                        dec.lm_head.cpu().numpy(), batch, kv_int8=kv_int8)
    prompt = np.stack([synth.uniform_int(seed + b, 9, prompt_len, 0, cfg.vocab - 1) for b in range(batch)]).astype(np.int32)
    d_prompt = dev(prompt)
    logits = dec.prefill(d_prompt)
    s.synchronize()
    want_logits, want_next = ref.forward(prompt, prompt_len)
    got_logits = logits.cpu().numpy()
    rel = np.linalg.norm(got_logits - want_logits) / np.linalg.norm(want_logits)
    ctx.set_int4_prefill_exact(False)
    assert rel < logit_tol, rel
    if exact_prefill and not kv_int8:
        assert np.array_equal(dec.next_tokens.cpu().numpy(), want_next)  # token chosen by the prefill
    elif not exact_prefill:
        assert rel > 1e-6  # the prompt pass really took the bf16 path
    if not exact_prefill:
        # the KV cache now carries bf16-level noise: follow the GPU's tokens and require the
        # logits of every decode step to stay within the same bound
        toks = dec.next_tokens.cpu().numpy().astype(np.int32)
        for i in range(steps):
            with torch.cuda.stream(s):
                lg = dec.forward(dec.next_tokens, 1)
            s.synchronize()
            wl, _ = ref.forward(toks.reshape(batch, 1), 1)
            r = np.linalg.norm(lg.cpu().numpy() - wl) / np.linalg.norm(wl)
            assert r < 1.5 * logit_tol, (i, r)
            toks = dec.next_tokens.cpu().numpy().astype(np.int32)
        return rel
    dec.capture_decode_step()
    got = dec.decode(steps)                        # [steps, batch], enqueued on the decoder's stream
    s.synchronize()
    got = got.cpu().numpy()
    toks = dec.next_tokens.cpu().numpy().astype(np.int32) if not exact_prefill else want_next
    mism = 0
    for i in range(steps):
        lg, nxt = ref.forward(toks.reshape(batch, 1), 1)
        for b in range(batch):
            if got[i, b] != nxt[b]:
                # a flip is only acceptable when the oracle's own top-2 margin is at rounding level
                srt = np.sort(lg[b])
                assert srt[-1] - srt[-2] < flip_margin * max(1.0, abs(srt[-1])), (i, b, srt[-1] - srt[-2])
                mism += 1
        toks = got[i].astype(np.int32)  # follow the GPU's token so one tie cannot derail the rest
    assert mism <= (steps * batch // 4 if (kv_int8 or not exact_prefill) else 1)
    return rel


@pytest.mark.parametrize("fused", [True, False])
def test_small_decoder_matches_oracle(tctx, oracle, fused):
    """Two sequences: the batch form of the one-launch step (two key chunks per head, rows 2..7
    of the activation planes zero), and the operator chain."""
    cfg = DecoderConfig(layers=3, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    run_parity(tctx, oracle, cfg, 3, batch=2, prompt_len=20, steps=12, seed=3, logit_tol=1e-4, fused_step=fused)
    ctx, _ = tctx
    assert ctx.device_status() == 0


@pytest.mark.parametrize("batch,form", [(3, -1), (5, 1), (8, -1), (8, 1)])
def test_small_decoder_batch_step_matches_oracle(tctx, oracle, batch, form):
    """The batch form of the one-launch step at odd batch sizes and a full batch of 8, a shape
    whose down projection is walked in K chunks (mlp 2560 > one chunk of 2048) and whose prompt
    differs per sequence; attention per (sequence, query head, key chunk) (the default) and per
    (sequence, KV head, key chunk)."""
    cfg = DecoderConfig(layers=2, hidden=1024, mlp=2560, n_q=16, n_kv=4, head_dim=64, vocab=1200)
    run_parity(tctx, oracle, cfg, 2, batch=batch, prompt_len=24, steps=8, seed=9, logit_tol=1e-4,
               plan_options=dict(attention_form=form))
    ctx, _ = tctx
    assert "decode_step_batch" in ctx.last_kernel()
    assert ctx.device_status() == 0


def test_small_decoder_fused_step_matches_oracle(tctx, oracle):
    # batch 1: every decode step is one launch of the persistent step kernel
    cfg = DecoderConfig(layers=3, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    run_parity(tctx, oracle, cfg, 3, batch=1, prompt_len=20, steps=12, seed=4, logit_tol=1e-4)
    ctx, _ = tctx
    assert ctx.device_status() == 0


def test_fused_step_logits_match_operator_chain(tctx):
    """The one-launch step against the chain of separate operator launches, same weights, same
    cache contents: logits of every step within 1e-5 (relative), same tokens."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=1024, mlp=2560, n_q=16, n_kv=4, head_dim=64, vocab=2000)
    prompt = dev(synth.uniform_int(21, 9, 24, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    ctx.set_int4_prefill_exact(True)
    logs, toks = [], []
    for fused in (False, True):
        dec = Int4Decoder(ctx, cfg, 1, 64, s, seed=12, fused_step=fused)
        assert (dec.plan is not None) == fused
        dec.prefill(prompt)
        lg, tk = [], []
        for _ in range(10):
            with torch.cuda.stream(s):
                out = dec.forward(dec.next_tokens, 1)
            s.synchronize()
            lg.append(out.cpu().numpy().copy())
            tk.append(int(dec.next_tokens.cpu().numpy()[0]))
        logs.append(lg)
        toks.append(tk)
        dec.close()
    ctx.set_int4_prefill_exact(False)
    assert toks[0] == toks[1]
    for a, b in zip(*logs):
        assert np.linalg.norm(a - b) / np.linalg.norm(a) < 1e-5
    assert ctx.device_status() == 0


@pytest.mark.parametrize("opts", [
    dict(max_tiles=2, k_chunk=1024),                    # default variant
    dict(max_tiles=2, k_chunk=1024, variant=0),         # plain
    dict(max_tiles=4, k_chunk=1536, variant=5),
    dict(attention_form=1),                             # attention per KV head and key chunk + merge phase
    dict(attention_form=1, max_tiles=2),
])
def test_fused_step_row_blocks_and_k_chunks(tctx, opts):
    """Small shapes pushed through the paths large models take: several row blocks per CTA
    (gate/up) and a down projection longer than one K chunk, by shrinking the plan's limits."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=1024, mlp=2560, n_q=16, n_kv=4, head_dim=64, vocab=2000)
    prompt = dev(synth.uniform_int(23, 9, 40, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    ctx.set_int4_prefill_exact(True)
    logs, toks = [], []
    try:
        for fused in (False, True):
            dec = Int4Decoder(ctx, cfg, 1, 64, s, seed=15, fused_step=fused, plan_options=opts if fused else None)
            assert (dec.plan is not None) == fused
            dec.prefill(prompt)
            lg, tk = [], []
            for _ in range(6):
                with torch.cuda.stream(s):
                    out = dec.forward(dec.next_tokens, 1)
                s.synchronize()
                lg.append(out.cpu().numpy().copy())
                tk.append(int(dec.next_tokens.cpu().numpy()[0]))
            logs.append(lg)
            toks.append(tk)
            dec.close()
    finally:
        ctx.set_int4_prefill_exact(False)
    assert toks[0] == toks[1]
    for a, b in zip(*logs):
        assert np.linalg.norm(a - b) / np.linalg.norm(a) < 1e-5
    assert ctx.device_status() == 0


def test_decode_plan_step_without_tail(tctx):
    """yscv_cuda_decode_plan_step_dev (layers only) leaves the same residual stream as the
    full step, touches neither the token nor the position, and the operator tail on top of it
    gives the same logits."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=777)
    prompt = dev(synth.uniform_int(41, 9, 18, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    decs = [Int4Decoder(ctx, cfg, 1, 32, s, seed=19) for _ in range(2)]
    for d_ in decs:
        d_.prefill(prompt)
    a, b = decs
    with torch.cuda.stream(s):
        logits = a.forward(a.next_tokens, 1).clone()           # full step
        xa = a._buf("x", 1, cfg.hidden).clone()
        tok_before, pos_before = b.next_tokens.clone(), b.pos.clone()
        xb = torch.empty(1, cfg.hidden, device="cuda")
        b.plan.step_dev(b.embedding.data_ptr(), cfg.vocab, b.next_tokens.data_ptr(), b.pos.data_ptr(), xb.data_ptr())
        h = torch.empty_like(xb)
        lg = torch.empty(1, cfg.vocab, device="cuda")
        ctx.add_rms_norm_dev(xb.data_ptr(), 0, b.gamma.data_ptr(), cfg.eps, 1, cfg.hidden, xb.data_ptr(), h.data_ptr())
        ctx.f32_matmul_dev(b.lm_head.data_ptr(), h.data_ptr(), 1, cfg.vocab, cfg.hidden, lg.data_ptr())
    s.synchronize()
    assert torch.equal(xa, xb)
    assert torch.equal(b.next_tokens, tok_before) and torch.equal(b.pos, pos_before)
    assert int(a.pos.item()) == int(pos_before.item()) + 1
    rel = float(torch.linalg.norm(lg - logits) / torch.linalg.norm(logits))
    assert rel < 1e-5, rel
    mx = logits[0].max()
    assert float(logits[0, int(a.next_tokens.item())]) == float(mx)   # the greedy token is a maximum
    for d_ in decs:
        d_.close()
    assert ctx.device_status() == 0


def test_fused_step_grouped_attention_long_cache(tctx):
    """A cache long enough that the plan picks attention per KV head and key chunk by itself,
    with more than 128 keys per chunk (the passes past the prefetched rows)."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    P, steps = 4300, 3
    prompt = dev(synth.uniform_int(35, 9, P, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    logs = []
    for fused in (False, True):
        dec = Int4Decoder(ctx, cfg, 1, P + steps + 1, s, seed=17, fused_step=fused)
        assert (dec.plan is not None) == fused
        dec.prefill(prompt)
        lg = []
        for _ in range(steps):
            with torch.cuda.stream(s):
                out = dec.forward(dec.next_tokens, 1)
            s.synchronize()
            lg.append(out.cpu().numpy().copy())
        logs.append(lg)
        dec.close()
    for a, b in zip(*logs):
        assert np.linalg.norm(a - b) / np.linalg.norm(a) < 1e-5
    assert ctx.device_status() == 0


def test_fused_step_llama70b_layer_shape(tctx):
    """One layer of BASELINE config 5's shape (hidden 8192, MLP 28672, 64/8 heads of 128; small
    vocabulary): four row blocks in gate/up, a down projection of 3.5 K chunks, two CTAs per
    head. The one-launch step against the operator chain."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=1, hidden=8192, mlp=28672, n_q=64, n_kv=8, head_dim=128, vocab=4096,
                        rope_theta=500000.0)
    prompt = dev(synth.uniform_int(29, 9, 200, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    logs, toks = [], []
    for fused in (False, True):
        dec = Int4Decoder(ctx, cfg, 1, 256, s, seed=16, fused_step=fused)
        assert (dec.plan is not None) == fused
        dec.prefill(prompt)
        lg, tk = [], []
        for _ in range(3):
            with torch.cuda.stream(s):
                out = dec.forward(dec.next_tokens, 1)
            s.synchronize()
            lg.append(out.cpu().numpy().copy())
            tk.append(int(dec.next_tokens.cpu().numpy()[0]))
        logs.append(lg)
        toks.append(tk)
        dec.close()
    assert toks[0] == toks[1]
    for a, b in zip(*logs):
        assert np.linalg.norm(a - b) / np.linalg.norm(a) < 1e-5
    assert ctx.device_status() == 0


def test_fused_step_long_context_and_limits(tctx):
    """More than 128 keys per attention split (the loops past the prefetched rows), the last
    cache slot, and shapes the plan refuses."""
    import torch
    import yscv_b200
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    P, steps = 700, 4   # 148 // 8 -> 4 splits per head: 175+ keys each
    prompt = dev(synth.uniform_int(33, 9, P, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    logs = []
    for fused in (False, True, "grouped"):
        # "grouped": 32 chunks per KV head; the last step fills the cache
        dec = Int4Decoder(ctx, cfg, 1, P + steps, s, seed=14, fused_step=bool(fused),
                          plan_options=dict(attention_form=1) if fused == "grouped" else None)
        assert (dec.plan is not None) == bool(fused)
        dec.prefill(prompt)
        lg = []
        for _ in range(steps):
            with torch.cuda.stream(s):
                out = dec.forward(dec.next_tokens, 1)
            s.synchronize()
            lg.append(out.cpu().numpy().copy())
        logs.append(lg)
        dec.close()
    for a, b, c in zip(*logs):
        assert np.linalg.norm(a - b) / np.linalg.norm(a) < 1e-5
        assert np.linalg.norm(a - c) / np.linalg.norm(a) < 1e-5
    assert ctx.device_status() == 0
    # K not a multiple of 512, fewer rows than SMs, too many heads: refused when the plan is built
    for bad in (DecoderConfig(layers=1, hidden=768, mlp=1024, n_q=12, n_kv=4, head_dim=64, vocab=100),
                DecoderConfig(layers=1, hidden=512, mlp=1024, n_q=2, n_kv=1, head_dim=32, vocab=100),
                DecoderConfig(layers=1, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=100, group_size=64)):
        dec = Int4Decoder(ctx, bad, 1, 32, s, seed=1)
        assert dec.plan is None
        dec.close()


def test_tinyllama_shape_greedy_tokens(tctx, oracle):
    # BASELINE config 4 at full depth: 22 layers, prompt 128, seed 3, 32 greedy steps, every
    # decode step one launch of the step kernel, against the CPU oracle decoder
    run_parity(tctx, oracle, TINYLLAMA_1B, 22, batch=1, prompt_len=128, steps=32, seed=3, logit_tol=1e-4)


@pytest.mark.parametrize("fused", [True, False])
def test_tinyllama_shape_batch8(tctx, oracle, fused):
    # BASELINE config 4, batch 8 (independent sequences, prompt seed + b): the batch form of the
    # one-launch step, and the operator chain
    run_parity(tctx, oracle, TINYLLAMA_1B, 2, batch=8, prompt_len=32, steps=8, seed=3, logit_tol=1e-4,
               fused_step=fused)


LLAMA70B_LAYER = DecoderConfig(layers=2, hidden=8192, mlp=28672, n_q=64, n_kv=8, head_dim=128, vocab=16032,
                               rope_theta=500000.0)


@pytest.mark.parametrize("fused", [True, False])
def test_llama70b_shape_two_layers_match_oracle(tctx, oracle, fused):
    """BASELINE config 5's layer shape (hidden 8192, MLP 28672, 64/8 heads of 128, RoPE base
    5e5), truncated to 2 layers and an eighth of the vocabulary so that the CPU oracle finishes
    in seconds: logits of the prompt pass and 8 greedy tokens against the oracle decoder, for
    the one-launch step (four row blocks in gate/up, a K-chunked down projection, two CTAs
    per head) and for the operator chain."""
    run_parity(tctx, oracle, LLAMA70B_LAYER, 2, batch=1, prompt_len=24, steps=8, seed=4, logit_tol=1e-4,
               fused_step=fused)
    ctx, _ = tctx
    assert ctx.device_status() == 0


def test_int8_kv_cache_matches_oracle(tctx, oracle):
    """KvDtype::I8 (kv_cache.rs:8-90): rows quantised at append time, dequantised in the
    attention; logits and tokens against the oracle decoder with the same cache format, at
    batch 1 and 3, with a prompt pass (block per query) and decode steps (split keys)."""
    cfg = DecoderConfig(layers=3, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    run_parity(tctx, oracle, cfg, 3, batch=3, prompt_len=20, steps=10, seed=6, logit_tol=2e-3, kv_int8=True)
    cfg = DecoderConfig(layers=2, hidden=1024, mlp=2048, n_q=8, n_kv=2, head_dim=128, vocab=1500)
    run_parity(tctx, oracle, cfg, 2, batch=1, prompt_len=150, steps=6, seed=7, logit_tol=2e-3, kv_int8=True,
               fused_step=False)
    ctx, _ = tctx
    assert ctx.device_status() == 0


@pytest.mark.parametrize("form", [0, 1])
def test_int8_kv_cache_fused_step_matches_oracle(tctx, oracle, form):
    """The one-launch step over KvDtype::I8 caches: the step kernel quantises the new position's
    key and value rows (one scale over every KV head of the row) and dequantises the cached rows
    in both of its attention forms (CTAs per query head; CTAs per KV head and key chunk plus a
    merge), head sizes 64 and 128, against the oracle decoder with the same cache format. The
    cache bytes the kernel appended are compared with the oracle's rows as well."""
    opts = dict(attention_form=form)
    cfg = DecoderConfig(layers=3, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    run_parity(tctx, oracle, cfg, 3, batch=1, prompt_len=20, steps=10, seed=8, logit_tol=2e-3, kv_int8=True,
               plan_options=opts)
    cfg = DecoderConfig(layers=2, hidden=1024, mlp=2048, n_q=8, n_kv=2, head_dim=128, vocab=1500)
    run_parity(tctx, oracle, cfg, 2, batch=1, prompt_len=150, steps=6, seed=7, logit_tol=2e-3, kv_int8=True,
               plan_options=opts)
    ctx, _ = tctx
    assert ctx.device_status() == 0


def test_int8_kv_cache_fused_step_appends_the_same_rows_as_the_chain(tctx):
    """After the same prompt and the same decode steps the int8 caches and their scales written
    by the one-launch step equal those written by the operator chain, except where a value
    sits on a rounding boundary of its row's grid (at most one step apart, in a handful of
    places)."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=1024, mlp=2048, n_q=8, n_kv=2, head_dim=128, vocab=1500)
    prompt = dev(synth.uniform_int(5, 9, 40, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    caches = {}
    ctx.set_int4_prefill_exact(True)
    try:
        for fused in (False, True):
            dec = Int4Decoder(ctx, cfg, 1, 64, s, seed=11, fused_step=fused, kv_int8=True)
            assert (dec.plan is not None) == fused
            dec.prefill(prompt)
            toks = dec.decode(8)
            s.synchronize()
            caches[fused] = ([c[0, :48].cpu().numpy().astype(np.int32) for c in dec.kcache + dec.vcache],
                             [c[0, :48].cpu().numpy() for c in dec.kscale + dec.vscale], toks.cpu().numpy())
            dec.close()
    finally:
        ctx.set_int4_prefill_exact(False)
    assert np.array_equal(caches[False][2], caches[True][2])
    for a, b in zip(caches[False][0], caches[True][0]):
        assert np.abs(a - b).max() <= 1 and np.count_nonzero(a != b) <= a.size // 200
    for a, b in zip(caches[False][1], caches[True][1]):
        assert np.allclose(a, b, rtol=1e-5, atol=0)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("n_q,n_kv,d,pos", [(8, 2, 64, 300), (32, 4, 128, 129), (16, 1, 128, 1000), (8, 8, 64, 0)])
def test_int8_decode_attention_tensor_core_kernel(tctx, n_q, n_kv, d, pos):
    """Decode attention over an int8 cache: the fp16 tensor-core kernel (int8 entries exact in
    fp16, query and softmax weights as two fp16 terms, fp32 accumulation) against the fp32 loop
    on the same cache: groups of 4, 8, 16 and 1 query heads per KV head, both head sizes, a last
    chunk that is not full, a single cached position, three sequences at once."""
    import torch
    ctx, s = tctx
    B, max_seq = 3, 1100
    rng = np.random.default_rng(31)
    kc = dev(rng.integers(-127, 128, size=(B, max_seq, n_kv * d), dtype=np.int8))
    vc = dev(rng.integers(-127, 128, size=(B, max_seq, n_kv * d), dtype=np.int8))
    ks = dev((rng.random((B, max_seq), dtype=np.float32) * 0.02 + 0.001))
    vs = dev((rng.random((B, max_seq), dtype=np.float32) * 0.02 + 0.001))
    qkv_w = (n_q + 2 * n_kv) * d
    qkv = dev(rng.normal(0, 1.5, (B, qkv_w)).astype(np.float32))
    d_pos = dev(np.array([pos], np.int32))
    outs = {}
    try:
        for tc in (False, True):
            ctx.set_attention_tensor_cores(tc)
            out = torch.zeros(B, n_q * d, device="cuda")
            torch.cuda.synchronize()
            ctx.gqa_attention_i8_dev(qkv.data_ptr(), qkv_w, B, 1, n_q, n_kv, d, kc.data_ptr(), ks.data_ptr(),
                                     vc.data_ptr(), vs.data_ptr(), max_seq, d_pos.data_ptr(), True, out.data_ptr())
            ctx.synchronize()
            assert ("mma" in ctx.last_kernel()) == tc
            outs[tc] = out.cpu().numpy()
    finally:
        ctx.set_attention_tensor_cores(True)
    err = np.abs(outs[True] - outs[False]).max() / np.abs(outs[False]).max()
    assert err < 1e-4, err   # (summation order and two-term fp16 operands; the scores here reach +-30)
    assert ctx.device_status() == 0


def test_int8_kv_cache_bytes(tctx, oracle):
    """The cache rows themselves: int8 values and scales bit-identical to the reference's append."""
    import torch
    ctx, s = tctx
    B, seq, n_q, n_kv, d, max_seq = 2, 5, 4, 2, 64, 16
    rng = np.random.default_rng(12)
    qkv = rng.normal(0, 1, (B * seq, (n_q + 2 * n_kv) * d)).astype(np.float32)
    qkv[3, n_q * d:(n_q + n_kv) * d] = 0.0    # an all-zero key row: scale falls to 1.0
    d_qkv = dev(qkv.copy())
    kc = torch.zeros(B, max_seq, n_kv * d, dtype=torch.int8, device="cuda")
    vc = torch.zeros_like(kc)
    ks = torch.zeros(B, max_seq, device="cuda")
    vs = torch.zeros_like(ks)
    pos = dev(np.array([2], np.int32))
    with torch.cuda.stream(s):
        ctx.rope_kv_append_i8_dev(d_qkv.data_ptr(), B, seq, n_q, n_kv, d, 10000.0, pos.data_ptr(), kc.data_ptr(),
                                  ks.data_ptr(), vc.data_ptr(), vs.data_ptr(), max_seq)
    s.synchronize()
    for b in range(B):
        rows = qkv[b * seq:(b + 1) * seq]
        _, k_rot = oracle.rope(rows[:, :n_q * d].ravel(), rows[:, n_q * d:(n_q + n_kv) * d].ravel(), n_q, n_kv, d,
                               seq, 2, 10000.0)
        kq, ksc = oracle.kv_append_i8(k_rot.reshape(seq, -1))
        vq, vsc = oracle.kv_append_i8(rows[:, (n_q + n_kv) * d:])
        assert np.array_equal(vc[b, 2:2 + seq].cpu().numpy(), vq) and np.array_equal(vs[b, 2:2 + seq].cpu().numpy(), vsc)
        got_k, got_ks = kc[b, 2:2 + seq].cpu().numpy(), ks[b, 2:2 + seq].cpu().numpy()
        # the rotated keys come from sincosf on the GPU and libm on the CPU: a value on a rounding
        # boundary may land one step apart
        assert np.max(np.abs(got_k.astype(np.int32) - kq.astype(np.int32))) <= 1
        assert np.mean(got_k != kq) < 0.01
        np.testing.assert_allclose(got_ks, ksc, rtol=1e-6)
        assert not kc[b, :2].any() and not kc[b, 2 + seq:].any()
    assert ctx.device_status() == 0


def test_norm_and_swiglu_write_the_gemm_activations(tctx, oracle):
    """add_rms_norm_act / swiglu_act hand the tensor-core GEMM its bf16 activations: the linear that follows
    (int4_matmul_act_dev) gives the same output, bit for bit, as the fp32 operators followed by
    int4_matmul_dev with its own conversion pass; shapes the bf16 path does not take are refused."""
    import torch
    import yscv_b200
    ctx, s = tctx
    rows, H, inter, n = 40, 512, 320, 300
    rng = np.random.default_rng(91)
    x = rng.normal(0, 1, (rows, H)).astype(np.float32)
    dl = rng.normal(0, 1, (rows, H)).astype(np.float32)
    gm = rng.normal(1, 0.1, H).astype(np.float32)
    gu = rng.normal(0, 2, (rows, 2 * inter)).astype(np.float32)
    w1 = rng.normal(0, 0.02, (n, H)).astype(np.float32)
    w2 = rng.normal(0, 0.02, (n, inter)).astype(np.float32)
    p1, s1 = oracle.pack_int4(w1.ravel(), n, H, 32)
    p2, s2 = oracle.pack_int4(w2.ravel(), n, inter, 32)
    h1, h2 = ctx.int4_weight_upload(p1, s1, n, H, 32), ctx.int4_weight_upload(p2, s2, n, inter, 32)
    with torch.cuda.stream(s):
        dx, dd, dg, dgu = dev(x), dev(dl), dev(gm), dev(gu)
        xo_a, xo_b = torch.empty_like(dx), torch.empty_like(dx)
        nm = torch.empty_like(dx)
        nm16 = torch.empty(rows, H, dtype=torch.bfloat16, device="cuda")
        act = torch.empty(rows, inter, device="cuda")
        act16 = torch.empty(rows, inter, dtype=torch.bfloat16, device="cuda")
        o_a, o_b = torch.empty(rows, n, device="cuda"), torch.empty(rows, n, device="cuda")
        ctx.add_rms_norm_dev(dx.data_ptr(), dd.data_ptr(), dg.data_ptr(), 1e-5, rows, H, xo_a.data_ptr(), nm.data_ptr())
        ctx.int4_matmul_dev(h1, nm.data_ptr(), o_a.data_ptr(), rows)
        ctx.add_rms_norm_act_dev(dx.data_ptr(), dd.data_ptr(), dg.data_ptr(), 1e-5, rows, H, xo_b.data_ptr(), nm16.data_ptr())
        ctx.int4_matmul_act_dev(h1, nm16.data_ptr(), o_b.data_ptr(), rows)
        s.synchronize()
        assert "prefill" in ctx.last_kernel()
        assert torch.equal(xo_a, xo_b) and torch.equal(o_a, o_b)
        # in place, as the decoder uses it
        x_in = dx.clone()
        ctx.add_rms_norm_act_dev(x_in.data_ptr(), dd.data_ptr(), dg.data_ptr(), 1e-5, rows, H, x_in.data_ptr(), nm16.data_ptr())
        ctx.int4_matmul_act_dev(h1, nm16.data_ptr(), o_b.data_ptr(), rows)
        s.synchronize()
        assert torch.equal(x_in, xo_a) and torch.equal(o_a, o_b)
        ctx.swiglu_dev(dgu.data_ptr(), rows, inter, act.data_ptr())
        ctx.int4_matmul_dev(h2, act.data_ptr(), o_a.data_ptr(), rows)
        ctx.swiglu_act_dev(dgu.data_ptr(), rows, inter, act16.data_ptr())
        ctx.int4_matmul_act_dev(h2, act16.data_ptr(), o_b.data_ptr(), rows)
        s.synchronize()
        assert torch.equal(o_a, o_b)
        # refused: a decode-shaped call, and the fp32-exact prefill mode
        with pytest.raises(yscv_b200.YscvCudaError):
            ctx.int4_matmul_act_dev(h2, act16.data_ptr(), o_b.data_ptr(), 8)
        ctx.set_int4_prefill_exact(True)
        try:
            with pytest.raises(yscv_b200.YscvCudaError):
                ctx.int4_matmul_act_dev(h2, act16.data_ptr(), o_b.data_ptr(), rows)
        finally:
            ctx.set_int4_prefill_exact(False)
    assert ctx.device_status() == 0
    h1.free()
    h2.free()


@pytest.mark.parametrize("B,seq,p0,nq,nkv,d,causal,i8", [
    (2, 100, 0, 8, 2, 64, True, False),      # tiles of 4 positions x 4 heads, ragged last tile, two key chunks
    (1, 70, 37, 8, 1, 128, True, False),     # a prompt appended behind 37 cached positions, 8 heads per KV head
    (1, 33, 0, 6, 2, 64, False, False),      # not causal, 3 heads per KV head (5 positions per tile)
    (2, 130, 5, 16, 4, 128, True, True),     # int8 cache, three key chunks
])
def test_prompt_attention_in_tiles(tctx, oracle, B, seq, p0, nq, nkv, d, causal, i8):
    """The prompt-pass attention kernel (query positions in tiles, keys and values staged in shared memory
    once per tile, chunked softmax) against the oracle's attention over the same cache contents."""
    import torch
    ctx, s = tctx
    rng = np.random.default_rng(77)
    total = p0 + seq
    max_seq = total + 3
    q = rng.normal(0, 1, (B, seq, nq * d)).astype(np.float32)
    if i8:
        kq = rng.integers(-127, 128, (B, max_seq, nkv * d), dtype=np.int8)
        vq = rng.integers(-127, 128, (B, max_seq, nkv * d), dtype=np.int8)
        ksc = rng.uniform(0.005, 0.02, (B, max_seq)).astype(np.float32)
        vsc = rng.uniform(0.005, 0.02, (B, max_seq)).astype(np.float32)
        kf = (kq.astype(np.float32) * ksc[:, :, None]).astype(np.float32)
        vf = (vq.astype(np.float32) * vsc[:, :, None]).astype(np.float32)
    else:
        kf = rng.normal(0, 1, (B, max_seq, nkv * d)).astype(np.float32)
        vf = rng.normal(0, 1, (B, max_seq, nkv * d)).astype(np.float32)
    pos = dev(np.array([p0], np.int32))
    out = torch.full((B * seq, nq * d), float("nan"), device="cuda")
    d_q = dev(q.reshape(B * seq, -1))
    with torch.cuda.stream(s):
        if i8:
            d_k, d_v, d_ks, d_vs = dev(kq), dev(vq), dev(ksc), dev(vsc)
            ctx.gqa_attention_i8_dev(d_q.data_ptr(), nq * d, B, seq, nq, nkv, d, d_k.data_ptr(), d_ks.data_ptr(),
                                     d_v.data_ptr(), d_vs.data_ptr(), max_seq, pos.data_ptr(), causal, out.data_ptr())
        else:
            d_k, d_v = dev(kf), dev(vf)
            ctx.gqa_attention_dev(d_q.data_ptr(), nq * d, B, seq, nq, nkv, d, d_k.data_ptr(), d_v.data_ptr(), max_seq,
                                  pos.data_ptr(), causal, out.data_ptr())
    s.synchronize()
    assert "prompt tiles" in ctx.last_kernel(), ctx.last_kernel()
    got = out.cpu().numpy().reshape(B, seq, -1)
    for b in range(B):
        want = oracle.gqa_attention(q[b].ravel(), kf[b, :total].ravel(), vf[b, :total].ravel(), 1, seq, total, nq, nkv, d,
                                    causal).reshape(seq, -1)
        assert np.max(np.abs(got[b] - want)) < 2e-5, (b, float(np.max(np.abs(got[b] - want))))
    assert ctx.device_status() == 0


def test_f32_matmul_wide_batch(tctx):
    """The LM-head product for more than 8 rows against float64: the 3xTF32 tensor-core kernel (k a
    multiple of 32; ragged rows and columns, more than one pass of 256 rows, more tiles than CTAs) and
    the tiled FMA kernel (any k, or on request). Both keep fp32 accuracy."""
    import torch
    ctx, s = tctx
    rng = np.random.default_rng(31)
    for m, n, k, tc in [(9, 1000, 512, True), (32, 3207, 2048, True), (70, 130, 36, False), (64, 20000, 256, True),
                        (300, 515, 96, True), (33, 129, 32, True)]:
        w = rng.normal(0, 0.02, (n, k)).astype(np.float32)
        x = rng.normal(0, 1.0, (m, k)).astype(np.float32)
        d_w, d_x = dev(w), dev(x)
        want = x.astype(np.float64) @ w.astype(np.float64).T
        for allow in (True, False):
            out = torch.full((m, n), float("nan"), device="cuda")
            ctx.set_f32_tensor_cores(allow)
            try:
                with torch.cuda.stream(s):
                    ctx.f32_matmul_dev(d_w.data_ptr(), d_x.data_ptr(), m, n, k, out.data_ptr())
                s.synchronize()
            finally:
                ctx.set_f32_tensor_cores(True)
            assert ("3xtf32" in ctx.last_kernel()) == (allow and tc), ctx.last_kernel()
            assert ("tiled" in ctx.last_kernel()) == (not (allow and tc))
            got = out.cpu().numpy()
            assert np.max(np.abs(got - want)) / np.max(np.abs(want)) < 1e-5, (m, n, k, allow)
    assert ctx.device_status() == 0


def test_decode_attention_serves_whole_groups(tctx, oracle):
    """Split-key decode attention over a long cache, f32 and int8, batch 3, groups of 4 and of
    12 query heads per KV head (more than one pass of eight), a ragged last chunk."""
    import torch
    ctx, s = tctx
    rng = np.random.default_rng(32)
    for n_q, n_kv, d, seq in [(8, 2, 64, 300), (12, 1, 128, 131), (16, 2, 32, 257)]:
        B, max_seq = 3, seq + 5
        q = rng.normal(0, 1, (B, n_q * d)).astype(np.float32)
        kf = rng.normal(0, 1, (B, max_seq, n_kv * d)).astype(np.float32)
        vf = rng.normal(0, 1, (B, max_seq, n_kv * d)).astype(np.float32)
        pos = dev(np.array([seq - 1], np.int32))
        out = torch.empty(B, n_q * d, device="cuda")
        d_q, d_k, d_v = dev(q), dev(kf), dev(vf)
        with torch.cuda.stream(s):
            ctx.gqa_attention_dev(d_q.data_ptr(), n_q * d, B, 1, n_q, n_kv, d, d_k.data_ptr(), d_v.data_ptr(),
                                  max_seq, pos.data_ptr(), True, out.data_ptr())
        s.synchronize()
        assert "split-k" in ctx.last_kernel()
        for b in range(B):
            want = oracle.gqa_attention(q[b], kf[b, :seq].ravel(), vf[b, :seq].ravel(), 1, 1, seq, n_q, n_kv, d, False)
            assert np.max(np.abs(out[b].cpu().numpy() - want)) < 2e-5 * max(1.0, np.max(np.abs(want)))
        # the same cache quantised row by row
        kq = np.empty((B, max_seq, n_kv * d), np.int8)
        vq = np.empty_like(kq)
        ksc = np.empty((B, max_seq), np.float32)
        vsc = np.empty_like(ksc)
        for b in range(B):
            kq[b], ksc[b] = oracle.kv_append_i8(kf[b])
            vq[b], vsc[b] = oracle.kv_append_i8(vf[b])
        d_kq, d_ks, d_vq, d_vs = dev(kq), dev(ksc), dev(vq), dev(vsc)
        with torch.cuda.stream(s):
            ctx.gqa_attention_i8_dev(d_q.data_ptr(), n_q * d, B, 1, n_q, n_kv, d, d_kq.data_ptr(),
                                     d_ks.data_ptr(), d_vq.data_ptr(), d_vs.data_ptr(), max_seq,
                                     pos.data_ptr(), True, out.data_ptr())
        s.synchronize()
        for b in range(B):
            kd, vd = oracle.kv_dequantise_i8(kq[b, :seq], ksc[b, :seq]), oracle.kv_dequantise_i8(vq[b, :seq], vsc[b, :seq])
            want = oracle.gqa_attention(q[b], kd.ravel(), vd.ravel(), 1, 1, seq, n_q, n_kv, d, False)
            assert np.max(np.abs(out[b].cpu().numpy() - want)) < 2e-5 * max(1.0, np.max(np.abs(want)))
    assert ctx.device_status() == 0


def test_position_outside_the_cache_is_reported(tctx):
    """pos >= max_seq: both decode paths leave the caches alone and set status 3."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    prompt = dev(synth.uniform_int(35, 9, 8, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    for fused in (True, False):
        dec = Int4Decoder(ctx, cfg, 1, 9, s, seed=2, fused_step=fused)   # room for the prompt and one step
        dec.prefill(prompt)
        with torch.cuda.stream(s):
            dec.forward(dec.next_tokens, 1)          # position 8: the last slot
        s.synchronize()
        assert ctx.device_status() == 0
        before = [c.clone() for c in dec.kcache + dec.vcache]
        with torch.cuda.stream(s):
            dec.forward(dec.next_tokens, 1)          # position 9 == max_seq
        s.synchronize()
        assert ctx.device_status() == 3
        assert all(torch.equal(a, b) for a, b in zip(before, dec.kcache + dec.vcache))
        assert ctx.device_status() == 0              # reading cleared it
        dec.close()


def test_eager_steps_equal_graph_replay_wide_vocabulary(tctx):
    """Operator chain without a graph (kernels chained by programmatic dependent launch, the
    two-stage arg-max of a vocabulary >= 8192, the position bump) against the replayed graph."""
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=9000)
    prompt = dev(np.stack([synth.uniform_int(45 + b, 9, 12, 0, cfg.vocab - 1) for b in range(2)]).astype(np.int32))
    outs = []
    for use_graph in (False, True):
        dec = Int4Decoder(ctx, cfg, 2, 48, s, seed=21)
        dec.prefill(prompt)
        if use_graph:
            dec.capture_decode_step()
        toks = dec.decode(24, use_graph=use_graph)
        s.synchronize()
        outs.append(toks.cpu().numpy())
        assert int(dec.pos.cpu().numpy()[0]) == 12 + 24
        dec.close()
    assert np.array_equal(outs[0], outs[1])
    assert ctx.device_status() == 0


def test_bounded_wait_gives_up_and_the_context_survives(tctx):
    """The give-up path of the step kernel's waits, without hanging anything: a tensor-parallel
    plan of two ranks whose peer never answers (its exchange region is a stand-in nobody
    writes) and a short spin limit. The first wait for the peer runs out, the kernel raises its
    abort flag, falls through every later wait and returns; the status word says 2, the plan is
    poisoned, and a fresh plan on the same context works."""
    import torch
    import yscv_b200
    ctx, s = tctx
    full = DecoderConfig(layers=2, hidden=1024, mlp=2048, n_q=16, n_kv=4, head_dim=64, vocab=2000)
    dec = Int4Decoder(ctx, full, 1, 32, s, seed=8, fused_step=False)
    # rank 0's shards of a 2-rank group, cut from the unsharded decoder's weights
    from yscv_b200 import sharding
    comm = yscv_b200.TpComm(ctx, 0, 2, full.hidden)
    comm.connect_unanswered()
    g, d = full.group_size, full.head_dim
    keep, layers = [], []
    for l in range(2):
        def rows(w, r0, r1):
            return w.packed[r0:r1], w.scales[r0:r1]
        q, k, v = (full.n_q * d, full.n_kv * d, full.n_kv * d)
        parts = [rows(dec.wqkv[l], 0, q // 2), rows(dec.wqkv[l], q, q + k // 2), rows(dec.wqkv[l], q + k, q + k + v // 2)]
        qkv = (torch.cat([p for p, _ in parts]).contiguous(), torch.cat([sc for _, sc in parts]).contiguous())
        o = tuple(t.contiguous() for t in sharding.shard_cols(dec.wo[l].packed, dec.wo[l].scales, g, 0, 2))
        parts = [rows(dec.wgu[l], 0, full.mlp // 2), rows(dec.wgu[l], full.mlp, full.mlp + full.mlp // 2)]
        gu = (torch.cat([p for p, _ in parts]).contiguous(), torch.cat([sc for _, sc in parts]).contiguous())
        dn = tuple(t.contiguous() for t in sharding.shard_cols(dec.wdown[l].packed, dec.wdown[l].scales, g, 0, 2))
        keep += [qkv, o, gu, dn]
        hs = [ctx.int4_weight_wrap(p.data_ptr(), sc.data_ptr(), p.shape[0], p.shape[1] * 2, g) for p, sc in (qkv, o, gu, dn)]
        keep += hs
        kc = torch.zeros(32, full.n_kv // 2, d, device="cuda")
        vc = torch.zeros_like(kc)
        keep += [kc, vc]
        layers.append(dict(qkv=hs[0], o=hs[1], gate_up=hs[2], down=hs[3], gamma_attn=dec.gamma.data_ptr(),
                           gamma_mlp=dec.gamma.data_ptr(), kcache=kc.data_ptr(), vcache=vc.data_ptr()))
    plan = ctx.decode_plan(layers, full.hidden, full.mlp // 2, full.n_q // 2, full.n_kv // 2, d, 32, full.eps,
                           full.rope_theta, tp=comm, spin_limit=2000)
    tok = dev(np.array([5], np.int32))
    pos = dev(np.array([0], np.int32))
    x = torch.zeros(full.hidden, device="cuda")
    logits = torch.zeros(full.vocab, device="cuda")
    with torch.cuda.stream(s):
        plan.step_token_shard_dev(dec.embedding.data_ptr(), full.vocab, tok.data_ptr(), pos.data_ptr(),
                                  dec.gamma.data_ptr(), dec.lm_head.data_ptr(), 0, full.vocab // 2, x.data_ptr(),
                                  logits.data_ptr())
    s.synchronize()                                   # the kernel returned
    assert ctx.device_status() == 2                   # YSCV_DEV_FLAG_TIMEOUT
    with pytest.raises(yscv_b200.YscvCudaError) as e:
        plan.check()
    assert e.value.status == -4
    with pytest.raises(yscv_b200.YscvCudaError) as e:  # poisoned: refuses to launch again
        plan.step_dev(dec.embedding.data_ptr(), full.vocab, tok.data_ptr(), pos.data_ptr(), x.data_ptr())
    assert e.value.status == -4
    plan.free()
    comm.close()
    dec.close()
    # the context is intact: a fresh one-GPU plan runs and agrees with the operator chain
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    prompt = dev(synth.uniform_int(3, 0, 12, 0, cfg.vocab - 1).astype(np.int32).reshape(1, -1))
    logs = []
    for fused in (False, True):
        d2 = Int4Decoder(ctx, cfg, 1, 32, s, seed=3, fused_step=fused)
        d2.prefill(prompt)
        with torch.cuda.stream(s):
            lg = d2.forward(d2.next_tokens, 1)
        s.synchronize()
        logs.append(lg.cpu().numpy().copy())
        d2.close()
    assert np.linalg.norm(logs[0] - logs[1]) / np.linalg.norm(logs[0]) < 1e-5
    assert ctx.device_status() == 0


def test_tinyllama_shape_operator_chain(tctx, oracle):
    # the same comparison with the single-token steps as separate operator launches
    run_parity(tctx, oracle, TINYLLAMA_1B, 2, batch=1, prompt_len=64, steps=8, seed=3, logit_tol=1e-4,
               fused_step=False)


def test_tinyllama_shape_bf16_prefill(tctx, oracle):
    # same decoder with the prompt pass on the tensor-core GEMM: logits within 2e-2
    run_parity(tctx, oracle, TINYLLAMA_1B, 4, batch=1, prompt_len=128, steps=16, seed=3, logit_tol=2e-2,
               exact_prefill=False)


def test_graph_replay_equals_eager(tctx):
    import torch
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=8, n_kv=2, head_dim=64, vocab=1000)
    prompt = dev(np.stack([synth.uniform_int(5 + b, 9, 16, 0, 999) for b in range(3)]).astype(np.int32))
    outs = []
    for use_graph in (False, True):
        dec = Int4Decoder(ctx, cfg, 3, 64, s, seed=11)
        dec.prefill(prompt)
        if use_graph:
            dec.capture_decode_step()
        toks = dec.decode(10, use_graph=use_graph)
        s.synchronize()
        outs.append(toks.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    assert ctx.device_status() == 0
