"""The layers of a decoder in one call (decoder_layers_dev) against the same operators called one by one: every form of
handed-over activations, partial sums left apart and joined, steps and prompts, both cache formats."""
import numpy as np
import pytest
import torch

import yscv_b200
from yscv_b200 import synth
from yscv_b200.decoder import DecoderConfig, Int4Decoder

pytestmark = pytest.mark.gpu

SMALL = DecoderConfig(layers=2, hidden=512, mlp=1280, n_q=8, n_kv=2, head_dim=64, vocab=600)
WIDE = DecoderConfig(layers=2, hidden=2304, mlp=2560, n_q=16, n_kv=4, head_dim=128, vocab=600)   # the 1024-thread norm
ODD = DecoderConfig(layers=2, hidden=640, mlp=1088, n_q=4, n_kv=4, head_dim=48, vocab=600)       # no depth is a multiple of 256
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
])
def test_layers_against_single_operators(tctx, cfg, batch, prompt, kv_int8):
    """Up to 16 rows the same sums in the same order: equal bits. Above, k is cut into other slices and an fp32 sum that
    moves in its last bit can move an activation by one bf16 rounding (2^-8 of it): with every activation of the 4
    linears of 2 layers moved, 2^-8 * sqrt(8) = 1.1e-2."""
    ctx, s = tctx
    tokens = torch.from_numpy(np.stack([synth.uniform_int(b, 3, prompt, 0, cfg.vocab - 1) for b in range(batch)]).astype(np.int32)).cuda()
    torch.cuda.synchronize()
    out = []
    for single in (False, True):
        dec = Int4Decoder(ctx, cfg, batch, max(prompt + 4, 140), s, seed=4, fused_step=False, kv_int8=kv_int8)
        assert dec.layers is not None
        if single:
            dec.layers = None
        with torch.cuda.stream(s):
            res = [dec.prefill(tokens).clone()]
            for _ in range(2):
                dec.next_tokens.copy_(tokens[:, 0])
                res.append(dec.forward(dec.next_tokens, 1).clone())
            caches = dec.kscale + dec.vscale if kv_int8 else dec.kcache + dec.vcache
            out.append(res + [c[:, :prompt + 2].clone() for c in caches])
        s.synchronize()
        dec.close()
    assert ctx.device_status() == 0
    for a, b in zip(*out):
        if batch * prompt <= 16:
            assert torch.equal(a, b)
        else:
            assert float((a - b).norm() / b.norm()) <= 1.1e-2


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
