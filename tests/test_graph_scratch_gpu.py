"""Captured decode steps after later calls outgrew the scratch buffers whose addresses the graph holds."""
import numpy as np
import pytest
import torch

import yscv_b200
from yscv_b200 import synth
from yscv_b200.decoder import DecoderConfig, Int4Decoder

pytestmark = pytest.mark.gpu

CFG = DecoderConfig(layers=2, hidden=2048, mlp=5632, n_q=32, n_kv=4, head_dim=64, vocab=9000)


def _outgrow(ctx):
    """Calls that need more of every scratch buffer than a small decode step: activations and last-round parts
    of a large GEMM, partial outputs of a long decode attention."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    n, k, m = 10240, 8192, 2048
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    scales = torch.rand(n, k // 32, device="cuda", generator=g)
    x, out = torch.randn(m, k, device="cuda", generator=g), torch.empty(m, n, device="cuda")
    h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
    ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
    max_seq, n_q, d = 131072, 64, 128
    kc, vc = (torch.zeros(max_seq, d, device="cuda") for _ in range(2))
    q, o = torch.randn(n_q * d, device="cuda", generator=g), torch.empty(n_q * d, device="cuda")
    pos = torch.full((1,), 1000, dtype=torch.int32, device="cuda")
    ctx.gqa_attention_dev(q.data_ptr(), n_q * d, 1, 1, n_q, 1, d, kc.data_ptr(), vc.data_ptr(), max_seq, pos.data_ptr(),
                          True, o.data_ptr())
    ctx.synchronize()


@pytest.mark.parametrize("batch,kv_int8", [(2, False), (8, False), (8, True), (24, False)])
def test_replay_after_the_scratch_grew(batch, kv_int8):
    """The replayed steps equal the eager operator chain bit for bit, and memory that somebody else allocated
    in the meantime keeps its contents."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)

    def prompt(length):
        rows = [synth.uniform_int(60 + b, length, length, 0, CFG.vocab - 1) for b in range(batch)]
        return torch.from_numpy(np.stack(rows).astype(np.int32)).cuda()

    decs = [Int4Decoder(ctx, CFG, batch, 300, stream, seed=5, fused_step=f, kv_int8=kv_int8) for f in (True, False)]

    def both(steps):
        toks = [d.decode(steps, use_graph=i == 0) for i, d in enumerate(decs)]
        stream.synchronize()
        assert torch.equal(toks[0], toks[1])
        assert torch.equal(*[d._buf("logits", batch, CFG.vocab) for d in decs])

    first, second = prompt(9), prompt(200)
    for d in decs:
        d.prefill(first)
    decs[0].capture_decode_step()
    both(3)
    with torch.cuda.stream(stream):
        _outgrow(ctx)
        canaries = [torch.full((1 << s,), 0x5A, dtype=torch.uint8, device="cuda") for s in range(16, 28) for _ in range(3)]
    for d in decs:
        d.reset()
        d.prefill(second)
    both(6)
    assert all(bool((c == 0x5A).all()) for c in canaries)
    assert ctx.device_status() == 0
    for d in decs:
        d.close()
    ctx.close()


@pytest.mark.parametrize("m,k", [(1, 4608), (1, 6912), (1, 8192), (1, 8960), (2, 4352), (3, 2048), (4, 2304)])
@pytest.mark.parametrize("n", [2048, 14336])
def test_few_rows_in_a_graph_hold_no_scratch(m, k, n):
    """Digit planes that fit a CTA: a captured call is one launch that quantises for itself, so that its replays are
    independent of what other calls leave in the context's scratch, and its bits are those of the eager call."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(k)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    scales = torch.rand(n, k // 32, device="cuda", generator=g)
    x, eager, replayed = torch.randn(m, k, device="cuda", generator=g), torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
    torch.cuda.synchronize()
    h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
    ctx.int4_matmul_dev(h, x.data_ptr(), eager.data_ptr(), m)
    stream.synchronize()
    before = ctx.launch_count()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        ctx.int4_matmul_dev(h, x.data_ptr(), replayed.data_ptr(), m)
    assert ctx.launch_count() - before == 1 and "fused-quant" in ctx.last_kernel()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(eager, replayed)
    assert ctx.device_status() == 0
    del graph
    ctx.close()


def test_outgrown_buffers_are_given_back():
    """Without a graph nothing is kept: the memory in use after a call that outgrew the scratch is that of a
    context which made the larger call first; destroying a context returns what graphs made it keep."""
    used = []
    for small_first in (True, False):
        ctx = yscv_b200.Context(0)
        n, k = 512, 8192
        packed, scales = torch.zeros(n, k // 2, dtype=torch.uint8, device="cuda"), torch.zeros(n, k // 32, device="cuda")
        h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        x, out = torch.zeros(8192, k, device="cuda"), torch.empty(8192, n, device="cuda")
        torch.cuda.synchronize()
        if small_first:
            for m in (2048, 4096):
                ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), 8192)
        ctx.synchronize()
        used.append(torch.cuda.mem_get_info()[0])
        ctx.close()
        del x, out
    assert abs(used[0] - used[1]) <= 8 << 20, used


@pytest.mark.parametrize("hidden,batch,launches", [(512, 1, 1), (512, 4, 1), (1024, 4, None), (2048, 1, 1), (2048, 2, None),
                                                    (2048, 8, None)])
def test_eager_and_replayed_steps_take_the_same_form(hidden, batch, launches):
    """Bit for bit the same logits and tokens, whichever form (one launch, or None: the operator chain) the
    shape takes; a program that chooses the other form gets it in both."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    cfg = DecoderConfig(layers=2, hidden=hidden, mlp=2 * hidden, n_q=hidden // 64, n_kv=4, head_dim=64, vocab=9000)
    rows = [synth.uniform_int(80 + b, 7, 20, 0, cfg.vocab - 1) for b in range(batch)]
    prompt = torch.from_numpy(np.stack(rows).astype(np.int32)).cuda()
    for other in (False, True):
        want = not other if launches else other
        got = []
        for graph in (False, True):
            dec = Int4Decoder(ctx, cfg, batch, 64, stream, seed=6)
            assert dec.plan is not None and dec.one_launch == (launches is not None)
            dec.one_launch = want
            dec.prefill(prompt)
            if graph:
                dec.capture_decode_step()
            before = ctx.launch_count()
            toks = dec.decode(5, use_graph=graph)
            stream.synchronize()
            if not graph:
                assert (ctx.launch_count() - before == 5) == want
            got.append((toks, dec._buf("logits", batch, cfg.vocab).clone()))
            dec.close()
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert ctx.device_status() == 0
    ctx.close()
