"""The layers of a decoder in one call (decoder_layers_dev) against the same operators called one by one: every form of
handed-over activations, partial sums left apart and joined, steps and prompts, both cache formats."""
import numpy as np
import pytest
import torch

import yscv_b200
from yscv_b200 import synth
from yscv_b200.decoder import DecoderConfig, Int4Decoder, Int4Linear

pytestmark = pytest.mark.gpu

SMALL = DecoderConfig(layers=2, hidden=512, mlp=1280, n_q=8, n_kv=2, head_dim=64, vocab=600)
WIDE = DecoderConfig(layers=2, hidden=2304, mlp=2560, n_q=16, n_kv=4, head_dim=128, vocab=600)   # the 1024-thread norm
ODD = DecoderConfig(layers=2, hidden=640, mlp=1088, n_q=4, n_kv=4, head_dim=48, vocab=600)       # no depth is a multiple of 256
ONE_B = DecoderConfig(layers=2, hidden=2048, mlp=5632, n_q=32, n_kv=4, head_dim=64, vocab=600)   # both layouts of handed-over digit planes
DEEP = DecoderConfig(layers=1, hidden=1024, mlp=65536, n_q=8, n_kv=2, head_dim=64, vocab=600)    # fp16 terms from 9 rows on


@pytest.fixture(scope="module")
def tctx():
    s = torch.cuda.Stream()
    c = yscv_b200.Context(0, stream=s.cuda_stream)
    yield c, s
    c.close()


@pytest.mark.parametrize("cfg,batch,prompt,kv_int8", [
    *[(SMALL, b, 5, i8) for b in (1, 3, 4, 5, 8, 9, 16, 17, 40, 128, 129) for i8 in (False, True)],
    (WIDE, 8, 3, False), (WIDE, 33, 3, True), (ODD, 6, 4, False), (ODD, 24, 4, False),
    (SMALL, 2, 150, False), (SMALL, 1, 700, True), (WIDE, 1, 600, False), (DEEP, 12, 1, False),
    *[(ONE_B, b, 5, False) for b in (1, 2, 3, 4)],
])
def test_layers_against_single_operators(tctx, cfg, batch, prompt, kv_int8):
    """Up to 16 rows the prompt is the same sums in the same order: equal bits; a step's attention adds its keys in
    another order, about 2^-24 * sqrt(200 terms) = 1e-6 a layer, 1e-5 asked for (int8 caches: 2e-3, a value on a rounding
    boundary moves by a step, as in the parity tests). Above 16 rows k is cut into other slices and an fp32 sum that
    moves in its last bit can move an activation by one bf16 rounding (2^-8 of it): with every activation of the 4
    linears of 2 layers moved, 2^-8 * sqrt(8) = 1.1e-2."""
    ctx, s = tctx
    tokens = torch.from_numpy(np.stack([synth.uniform_int(b, 3, prompt, 0, cfg.vocab - 1) for b in range(batch)]).astype(np.int32)).cuda()
    torch.cuda.synchronize()
    out, filled = [], None
    for single in (False, True):
        dec = Int4Decoder(ctx, cfg, batch, max(prompt + 4, 140), s, seed=4, fused_step=False, kv_int8=kv_int8)
        assert dec.layers is not None
        if single:
            dec.layers = None
        with torch.cuda.stream(s):
            res = [dec.prefill(tokens).clone()]
            tables = dec.kscale + dec.vscale if kv_int8 else []
            res += [c[:, :prompt].clone() for c in tables or dec.kcache + dec.vcache]
            # the steps start from the same caches, so that they answer for themselves
            held = dec.kcache + dec.vcache + tables
            if filled is None:
                filled = [c.clone() for c in held]
            for dst, src in zip(held, filled):
                dst.copy_(src)
            n_prompt = len(res)
            for _ in range(2):
                dec.next_tokens.copy_(tokens[:, 0])
                res.append(dec.forward(dec.next_tokens, 1).clone())
            out.append(res + [c[:, prompt:prompt + 2].clone() for c in tables or dec.kcache + dec.vcache])
        s.synchronize()
        dec.close()
    assert ctx.device_status() == 0
    for i, (a, b) in enumerate(zip(*out)):
        rows = batch * prompt if i < n_prompt else batch
        if i == 0 and rows <= 16:
            assert torch.equal(a, b)
        elif rows <= 16:
            assert float((a - b).norm() / b.norm()) <= (2e-3 if kv_int8 else 1e-5), i
        else:
            assert float((a - b).norm() / b.norm()) <= 1.1e-2, i


@pytest.mark.parametrize("batch", [2, 20])
@pytest.mark.parametrize("kv_int8", [False, True])
def test_a_decoder_given_other_tensors(tctx, batch, kv_int8):
    """A pass reads the caches, gamma and weights that the decoder holds now, at an odd address of gamma too: equal bits
    to a decoder that runs operator by operator on the same (up to 16 rows; above, the bound given above)."""
    ctx, s = tctx
    tokens = torch.randint(0, SMALL.vocab, (batch, 3), dtype=torch.int32, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    torch.cuda.synchronize()
    one, other = (Int4Decoder(ctx, SMALL, batch, 140, s, seed=4, fused_step=False, kv_int8=kv_int8) for _ in range(2))
    donor = Int4Decoder(ctx, SMALL, batch, 140, s, seed=5, fused_step=False, kv_int8=kv_int8)
    other.layers = None
    kept = []   # what the decoders held before stays allocated
    with torch.cuda.stream(s):
        gammas = [torch.rand(SMALL.hidden, device="cuda") + 0.5, (torch.rand(SMALL.hidden + 1, device="cuda") + 0.5)[1:]]
        for step in ("nothing", "caches", "gamma", "weights", "odd gamma"):
            got = []
            for dec in (one, other):
                kept.append((dec.kcache, dec.vcache, dec.gamma, dec.wqkv, dec.wo, dec.wgu, dec.wdown, *([dec.kscale, dec.vscale] if kv_int8 else [])))
                if step == "caches":
                    dec.kcache, dec.vcache = ([torch.zeros_like(c) for c in cs] for cs in (dec.kcache, dec.vcache))
                    if kv_int8:
                        dec.kscale, dec.vscale = ([torch.zeros_like(c) for c in cs] for cs in (dec.kscale, dec.vscale))
                elif step == "weights":
                    dec.wqkv, dec.wo, dec.wgu, dec.wdown = donor.wqkv, list(reversed(donor.wo)), donor.wgu, donor.wdown
                elif "gamma" in step:
                    dec.gamma = gammas[step == "odd gamma"]
                dec.reset()
                lg = dec.prefill(tokens).clone()
                got.append([lg] + [c.clone() for c in (dec.kscale + dec.vscale if kv_int8 else dec.kcache + dec.vcache)])
            s.synchronize()
            for a, b in zip(*got):
                assert torch.equal(a, b) if batch == 2 else float((a - b).norm() / b.norm()) <= 1.1e-2, step
    assert ctx.device_status() == 0
    for dec in (one, other, donor):
        dec.close()


def _repack(ctx, dec, layer, group, seed):
    """Other random weights of the layer's shapes, packed in groups of `group`."""
    for lins in (dec.wqkv, dec.wo, dec.wgu, dec.wdown):
        n, k = lins[layer].n, lins[layer].k
        w = torch.randn(n, k, device="cuda", generator=torch.Generator("cuda").manual_seed(seed + n)) * 0.02
        packed, scales = torch.empty(n, k // 2, dtype=torch.uint8, device="cuda"), torch.empty(n, k // group, device="cuda")
        ctx.pack_int4_dev(w.data_ptr(), n, k, group, packed.data_ptr(), scales.data_ptr())
        lins[layer] = Int4Linear(ctx, packed, scales, n, k, group)


@pytest.mark.parametrize("mlp,batch", [(28672, 1), (8192, 2), (8192, 4), (5632, 9), (65536, 12), (5632, 24)])
@pytest.mark.parametrize("groups", [(64, 32, 32), (32, 64, 32)])
def test_layers_of_different_groups(tctx, mlp, batch, groups):
    """Groups of 64 take fp32 activations, groups of 32 digit planes, fp16 terms, bf16 with k slices: the workspace holds
    the largest form of any layer, nothing behind it is written, and the results are the single operators' (bound above; from
    17 rows on those run in fp32, and each of 12 linears rounds weights and activations to bf16: 2^-8 * sqrt(24) = 1.9e-2)."""
    ctx, s = tctx
    cfg = DecoderConfig(layers=3, hidden=1024, mlp=mlp, n_q=8, n_kv=2, head_dim=64, vocab=300)
    shape = (cfg.hidden, cfg.mlp, cfg.n_q, cfg.n_kv, cfg.head_dim)
    dec = Int4Decoder(ctx, cfg, batch, 140, s, seed=8, fused_step=False)
    largest = ctx.decoder_layers_workspace(dec.layers, *shape, batch, 1)
    with torch.cuda.stream(s):
        for l, group in enumerate(groups):
            _repack(ctx, dec, l, group, 10 * l)
        layers = ctx.decode_layers(dec._layers_of())
        need = ctx.decoder_layers_workspace(layers, *shape, batch, 1)
        assert need >= largest
        x0 = torch.randn(batch, cfg.hidden, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        x, last = x0.clone(), torch.empty(batch, cfg.hidden, device="cuda")
        ws = torch.full((need + 4096,), 77, dtype=torch.uint8, device="cuda")
        ctx.decoder_layers_dev(layers, *shape, 140, cfg.eps, cfg.rope_theta, False, batch, 1, dec.pos.data_ptr(), x.data_ptr(),
                               dec.gamma.data_ptr(), last.data_ptr(), ws.data_ptr(), need)
        assert bool((ws[need:] == 77).all())
        got = []
        tokens = torch.arange(batch, dtype=torch.int32, device="cuda")
        for form in (dec.layers, None):
            dec.layers = form
            ctx.set_int4_prefill_exact(form is None)
            dec.reset()
            got.append(dec.forward(tokens, 1).clone())
        # the direct call against the operators from the same residual rows
        dec.embedding[:batch].copy_(x0)
        dec.reset()
        dec.forward(tokens, 1)
        want = dec._buf("h", batch, cfg.hidden)
        ctx.set_int4_prefill_exact(False)
    s.synchronize()
    assert ctx.device_status() == 0
    tol = 1.9e-2 if batch > 16 else 1e-5
    assert float((got[0] - got[1]).norm() / got[1].norm()) <= tol
    assert float((last - want).norm() / want.norm()) <= tol
    dec.close()


HEADS = [  # n_q, n_kv, d: groups of 1 to 8 heads, both head sizes
    (8, 1, 64), (6, 6, 64), (12, 4, 64), (4, 2, 128), (8, 1, 128), (20, 4, 64)]


@pytest.mark.parametrize("n_q,n_kv,d", HEADS)
@pytest.mark.parametrize("batch", [2, 7, 40])
@pytest.mark.parametrize("kv_int8", [False, True])
@pytest.mark.parametrize("max_seq", [196, 126])   # the shorter one keeps one and two CTAs per sequence in the one kernel
def test_step_attention_positions(tctx, n_q, n_kv, d, batch, kv_int8, max_seq):
    """One step at positions around the chunks and the CTAs' shares of the one-kernel attention, against the three
    kernels; the appended rows; a sequence whose cache holds a NaN and an infinity; a position past the cache."""
    ctx, s = tctx
    cfg = DecoderConfig(layers=1, hidden=256, mlp=256, n_q=n_q, n_kv=n_kv, head_dim=d, vocab=300)
    dec = Int4Decoder(ctx, cfg, batch, max_seq, s, seed=6, fused_step=False, kv_int8=kv_int8)
    layers = dec.layers
    g = torch.Generator(device="cuda")
    g.manual_seed(d + n_q)
    with torch.cuda.stream(s):
        tokens = torch.randint(0, cfg.vocab, (batch,), dtype=torch.int32, device="cuda", generator=g)
        fill = []
        for c in dec.kcache + dec.vcache:
            fill.append(torch.randint(-127, 128, c.shape, dtype=torch.int8, device="cuda", generator=g) if kv_int8
                        else torch.randn(c.shape, device="cuda", generator=g))
        scales = [0.01 + 0.02 * torch.rand(batch, max_seq, device="cuda", generator=g) for _ in range(2)] if kv_int8 else []
        bad = fill[0] if not kv_int8 else scales[0]
        bad[batch - 1, 0].fill_(float("nan"))
        caches = dec.kcache + dec.vcache
        tables = dec.kscale + dec.vscale if kv_int8 else []
        for p in [q for q in (0, 1, 23, 24, 25, 63, 64, 65, 127, 128, 129) if q < max_seq - 1] + [max_seq - 1, max_seq]:
            res = []
            for form in (layers, None):
                dec.layers = form
                for dst, src in zip(caches + tables, fill + scales):
                    dst.copy_(src)
                dec.pos.fill_(p)
                lg = dec.forward(tokens, 1).clone()
                res.append([lg] + [c[:, min(p, max_seq - 1)].float().clone() for c in caches + tables])
            s.synchronize()
            assert ctx.device_status() == (3 if p == max_seq else 0)
            a, b = ([t[:batch - 1] for t in r] for r in res)
            tol = 1.1e-2 if batch > 16 else 1e-5   # bounds as above; one layer
            assert float((a[0] - b[0]).norm() / b[0].norm()) <= (max(tol, 2e-3) if kv_int8 else tol), p
            for x, y in zip(a[1:], b[1:]):
                assert float((x - y).norm()) <= (2e-3 if kv_int8 else 1e-6) * float(y.norm()), p
            if p > 0:
                assert not torch.isfinite(res[0][0][batch - 1]).any()
    dec.close()


@pytest.mark.parametrize("n_q,n_kv,d,batch,kv_int8,one,three", [
    # CTAs per sequence and KV head 8, 4, 2, 1, with a grid that fills the machine's two CTAs per SM or not
    (32, 4, 64, 2, False, 600, 640), (32, 4, 64, 8, False, 1200, 1240), (32, 4, 64, 12, False, 400, 440), (32, 4, 64, 24, False, 300, 340),
    (32, 4, 64, 40, False, 200, 240), (32, 4, 64, 64, False, 400, 440), (32, 4, 64, 2, True, 300, 340), (32, 4, 64, 48, True, 130, 170),
    (16, 16, 64, 8, False, 200, 240), (16, 2, 128, 10, False, 1200, 1240), (16, 2, 128, 40, False, 400, 440), (8, 2, 128, 95, False, 400, 440),
    (16, 2, 128, 16, True, 200, 240)])
def test_longest_cache_of_the_one_attention_kernel(tctx, n_q, n_kv, d, batch, kv_int8, one, three):
    """On both sides of the line: two launches more, and the same step over a nearly full cache within the bounds above."""
    ctx, s = tctx
    cfg = DecoderConfig(layers=1, hidden=256, mlp=256, n_q=n_q, n_kv=n_kv, head_dim=d, vocab=300)
    g = torch.Generator(device="cuda").manual_seed(batch)
    out, launches = [], []
    with torch.cuda.stream(s):
        tokens = torch.randint(0, cfg.vocab, (batch,), dtype=torch.int32, device="cuda", generator=g)
        shape = (batch, one, n_kv, d)
        fill = [torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=g) if kv_int8 else torch.randn(shape, device="cuda", generator=g)
                for _ in range(2)]
        scales = [0.005 + 0.01 * torch.rand(batch, one, device="cuda", generator=g) for _ in range(2)]
        for max_seq in (one, three):
            dec = Int4Decoder(ctx, cfg, batch, max_seq, s, seed=6, fused_step=False, kv_int8=kv_int8)
            for dst, src in zip(dec.kcache + dec.vcache + (dec.kscale + dec.vscale if kv_int8 else []), fill + scales):
                dst[:, :one].copy_(src)
            dec.pos.fill_(one - 1)
            before = ctx.launch_count()
            out.append(dec.forward(tokens, 1).clone())
            launches.append(ctx.launch_count() - before)
            s.synchronize()
            dec.close()
    assert launches[1] - launches[0] == 2
    assert ctx.device_status() == 0
    tol = 1.1e-2 if batch > 16 else 1e-5
    assert float((out[0] - out[1]).norm() / out[1].norm()) <= (max(tol, 2e-3) if kv_int8 else tol)


@pytest.mark.parametrize("n_q,n_kv", [(8, 2), (32, 4)])   # up to 16 and up to 4 key splits per head
@pytest.mark.parametrize("kv_int8", [False, True])
def test_one_launch_step_positions(tctx, n_q, n_kv, kv_int8):
    """The one-launch step against the chain at positions where one more key split comes into use (128 keys each), with
    the bounds above: the linears quantise their activations to 2^-22 of a group's maximum in both forms, but before or
    after the norm's row factor, a few 1e-7 a linear."""
    ctx, s = tctx
    cfg = DecoderConfig(layers=2, hidden=512, mlp=1024, n_q=n_q, n_kv=n_kv, head_dim=64, vocab=300)
    max_seq = 600
    dec = Int4Decoder(ctx, cfg, 1, max_seq, s, seed=7, kv_int8=kv_int8)
    assert dec.plan is not None and dec.layers is not None
    g = torch.Generator(device="cuda")
    g.manual_seed(n_q)
    with torch.cuda.stream(s):
        caches = dec.kcache + dec.vcache
        tables = dec.kscale + dec.vscale if kv_int8 else []
        fill = [torch.randint(-127, 128, c.shape, dtype=torch.int8, device="cuda", generator=g) if kv_int8
                else torch.randn(c.shape, device="cuda", generator=g) for c in caches]
        fill += [0.005 + 0.01 * torch.rand(t.shape, device="cuda", generator=g) for t in tables]
        for p in (0, 1, 127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 512, 513, max_seq - 1):
            res = []
            for one in (True, False):
                dec.one_launch = one
                for dst, src in zip(caches + tables, fill):
                    dst.copy_(src)
                dec.pos.fill_(p)
                dec.next_tokens.fill_(p % cfg.vocab)
                lg = dec.forward(dec.next_tokens, 1).clone()
                assert int(dec.pos.reshape(-1)[0]) == p + 1
                res.append([lg] + [c[:, p].float().clone() for c in caches + tables])
            s.synchronize()
            assert ctx.device_status() == 0
            a, b = res
            assert float((a[0] - b[0]).norm() / b[0].norm()) <= (2e-3 if kv_int8 else 1e-5), p
            for i, (x, y) in enumerate(zip(a[1:], b[1:])):
                if kv_int8 and i < len(caches):   # a value on a rounding boundary
                    assert float((x - y).abs().max()) <= 1, p
                else:
                    assert float((x - y).norm()) <= 1e-5 * float(y.norm()), p
    dec.close()


def test_workspace_of_another_size(tctx):
    """Without room for partial sums the matmuls join them; without room for the pass the call is refused."""
    ctx, s = tctx
    batch = 32
    dec = Int4Decoder(ctx, SMALL, batch, 140, s, seed=4, fused_step=False)
    shape = (SMALL.hidden, SMALL.mlp, SMALL.n_q, SMALL.n_kv, SMALL.head_dim)
    need = ctx.decoder_layers_workspace(dec.layers, *shape, batch, 1)
    plain = 4 * batch * (SMALL.mlp + (SMALL.n_q + 2 * SMALL.n_kv) * SMALL.head_dim + SMALL.hidden + 2 * SMALL.mlp) + 4 * 256
    assert plain < need
    res = []
    with torch.cuda.stream(s):
        x0 = torch.randn(batch, SMALL.hidden, device="cuda")
        for size in (need, plain):
            x, last = x0.clone(), torch.empty(batch, SMALL.hidden, device="cuda")
            ws = torch.full((size + 4096,), 77, dtype=torch.uint8, device="cuda")
            call = lambda n: ctx.decoder_layers_dev(dec.layers, *shape, 140, 1e-5, 1e4, False, batch, 1, dec.pos.data_ptr(), x.data_ptr(),
                                                    dec.gamma.data_ptr(), last.data_ptr(), ws.data_ptr(), n)
            call(size)
            res.append(last)
            assert bool((ws[size:] == 77).all())
        with pytest.raises(yscv_b200.YscvCudaError):
            call(plain // 2)
    s.synchronize()
    assert float((res[0] - res[1]).norm() / res[1].norm()) <= 1.1e-2
    dec.close()
