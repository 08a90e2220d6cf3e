"""The decoder operators at the edges of their kernels' ranges: row lengths around the register forms of
the norm, head sizes and operands the vector forms of RoPE and SwiGLU cannot take."""
import numpy as np
import pytest

from yscv_b200 import synth

pytestmark = pytest.mark.gpu

# bf16 position of element e of a group of 8 in the prefill GEMM's activation order
ORDER = [0, 4, 1, 5, 2, 6, 3, 7]


@pytest.fixture(scope="module")
def tctx():
    import torch
    import yscv_b200
    s = torch.cuda.Stream()
    c = yscv_b200.Context(0, stream=s.cuda_stream)
    yield c, s
    c.close()


@pytest.mark.parametrize("hidden", [8, 511, 2048, 2056, 8192, 8200, 16384, 16392])
@pytest.mark.parametrize("in_place", [False, True])
def test_norm_row_lengths(tctx, hidden, in_place):
    import torch
    ctx, s = tctx
    rows = 3
    x = synth.normal(1, hidden, rows * hidden).reshape(rows, hidden)
    dl = synth.normal(2, hidden, rows * hidden).reshape(rows, hidden)
    gm = synth.normal(3, hidden, hidden)
    total = (x + dl).astype(np.float64)
    want = total / np.sqrt((total ** 2).mean(axis=1, keepdims=True) + 1e-5) * gm
    with torch.cuda.stream(s):
        d, g = (torch.from_numpy(a).cuda() for a in (dl, gm))
        dx = torch.from_numpy(x).cuda()
        xo = dx if in_place else torch.empty_like(dx)
        out = torch.empty_like(dx)
        ctx.add_rms_norm_dev(dx.data_ptr(), d.data_ptr(), g.data_ptr(), 1e-5, rows, hidden, xo.data_ptr(), out.data_ptr())
        # fp32 sum of `hidden` squares: relative error below 1e-6 here
        assert np.array_equal(xo.cpu().numpy(), x + dl)
        got = out.cpu().numpy()
        assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()
        if hidden % 8 == 0:
            act = torch.empty(rows, hidden, dtype=torch.bfloat16, device="cuda")
            ctx.add_rms_norm_act_dev(xo.data_ptr(), None, g.data_ptr(), 1e-5, rows, hidden, None, act.data_ptr())
            order = out.view(rows, hidden // 8, 8)[:, :, ORDER].reshape(rows, hidden).to(torch.bfloat16)
            assert torch.equal(act, order)


@pytest.mark.parametrize("inter,shift", [(1, 0), (7, 0), (8, 0), (8, 1), (2056, 0), (2056, 3)])
def test_swiglu_sizes_and_alignment(tctx, inter, shift):
    """shift: floats by which the gate_up rows are off a 16-byte boundary."""
    import torch
    ctx, s = tctx
    rows = 5
    gu = synth.normal(4, inter, rows * 2 * inter, 2.0)
    g, u = np.split(gu.reshape(rows, 2 * inter).astype(np.float64), 2, axis=1)
    want = g / (1 + np.exp(-g)) * u
    with torch.cuda.stream(s):
        buf = torch.zeros(gu.size + 8, device="cuda")
        buf[shift:shift + gu.size] = torch.from_numpy(gu).cuda()
        out = torch.empty(rows, inter, device="cuda")
        ctx.swiglu_dev(buf[shift:].data_ptr(), rows, inter, out.data_ptr())
        assert np.abs(out.cpu().numpy() - want).max() <= 1e-6 * max(1.0, np.abs(want).max())
        if inter % 8 == 0:
            act = torch.empty(rows, inter, dtype=torch.bfloat16, device="cuda")
            ctx.swiglu_act_dev(buf[shift:].data_ptr(), rows, inter, act.data_ptr())
            assert torch.equal(act, out.view(rows, inter // 8, 8)[:, :, ORDER].reshape(rows, inter).to(torch.bfloat16))


@pytest.mark.parametrize("n_q,n_kv,d,shift", [(4, 2, 6, 0), (64, 8, 128, 0), (64, 8, 128, 1), (130, 1, 64, 0)])
@pytest.mark.parametrize("i8", [False, True])
def test_rope_append_parts_and_alignment(tctx, oracle, n_q, n_kv, d, shift, i8):
    import torch
    ctx, s = tctx
    B, seq, p, max_seq = 2, 3, 7, 16
    w = (n_q + 2 * n_kv) * d
    qkv = synth.normal(5, n_q * d, B * seq * w)
    with torch.cuda.stream(s):
        buf = torch.zeros(qkv.size + 8, device="cuda")
        buf[shift:shift + qkv.size] = torch.from_numpy(qkv).cuda()
        kc, vc = (torch.zeros(B, max_seq, n_kv * d, dtype=torch.int8 if i8 else torch.float32, device="cuda") for _ in range(2))
        ks, vs = torch.zeros(B, max_seq, device="cuda"), torch.zeros(B, max_seq, device="cuda")
        pos = torch.full((1,), p, dtype=torch.int32, device="cuda")
        if i8:
            ctx.rope_kv_append_i8_dev(buf[shift:].data_ptr(), B, seq, n_q, n_kv, d, 10000.0, pos.data_ptr(), kc.data_ptr(),
                                      ks.data_ptr(), vc.data_ptr(), vs.data_ptr(), max_seq)
        else:
            ctx.rope_kv_append_dev(buf[shift:].data_ptr(), B, seq, n_q, n_kv, d, 10000.0, pos.data_ptr(), kc.data_ptr(),
                                   vc.data_ptr(), max_seq)
        got = buf[shift:shift + qkv.size].cpu().numpy().reshape(B, seq, w)
        rows = qkv.reshape(B, seq, w)
        for b in range(B):
            q, k, v = rows[b, :, :n_q * d], rows[b, :, n_q * d:(n_q + n_kv) * d], rows[b, :, (n_q + n_kv) * d:]
            qr, kr = oracle.rope(q.ravel(), k.ravel(), n_q, n_kv, d, seq, p, 10000.0)
            assert np.abs(got[b, :, :n_q * d] - qr.reshape(seq, -1)).max() < 2e-5
            for cache, scale, want in ((kc, ks, kr.reshape(seq, -1)), (vc, vs, v)):
                c = cache[b, p:p + seq].cpu().numpy().astype(np.float32)
                if i8:
                    c *= scale[b, p:p + seq].cpu().numpy()[:, None]
                    # half a step of a row's grid, and the rounding of sinf / cosf
                    assert (np.abs(c - want) <= 0.5001 * np.abs(want).max(axis=1, keepdims=True) / 127 + 2e-5).all()
                else:
                    assert np.abs(c - want).max() < 2e-5
            assert (cache[b, :p] == 0).all() and (cache[b, p + seq:] == 0).all()
        assert ctx.device_status() == 0


@pytest.mark.parametrize("hidden", [8, 2040, 2048, 2056, 4088, 8192])
@pytest.mark.parametrize("rows", [1, 2, 295, 296, 297, 600])
def test_norm_forms_are_the_scalar_kernel(tctx, rows, hidden):
    """Around two rows per SM and the sizes of the blocks: the bits of the kernel for operands at odd addresses, with and
    without a delta, in place and not, to fp32 and to the bf16 of a following matmul."""
    import torch
    ctx, s = tctx
    with torch.cuda.stream(s):
        gen = torch.Generator(device="cuda").manual_seed(hidden + rows)
        x, d = (torch.randn(rows * hidden, device="cuda", generator=gen) for _ in range(2))
        g = torch.rand(hidden + 1, device="cuda", generator=gen)
        for delta in (False, True):
            xo = [torch.empty(rows * hidden + 1, device="cuda") for _ in range(2)]
            no = [torch.empty(rows * hidden + 1, device="cuda") for _ in range(2)]
            n16 = torch.empty(rows * hidden, dtype=torch.bfloat16, device="cuda")
            inplace = x.clone()
            dp = d.data_ptr() if delta else 0
            g0 = g[1:].clone()
            ctx.add_rms_norm_dev(x.data_ptr(), dp, g0.data_ptr(), 1e-5, rows, hidden, xo[0].data_ptr(), no[0].data_ptr())
            ctx.add_rms_norm_dev(x.data_ptr(), dp, g[1:].data_ptr(), 1e-5, rows, hidden, xo[1].data_ptr() + 4, no[1].data_ptr() + 4)
            ctx.add_rms_norm_act_dev(inplace.data_ptr(), dp, g0.data_ptr(), 1e-5, rows, hidden, inplace.data_ptr(), n16.data_ptr())
            assert torch.equal(xo[0][:-1], xo[1][1:]) and torch.equal(no[0][:-1], no[1][1:])
            assert torch.equal(inplace, xo[0][:-1])
            assert torch.equal(n16.view(-1, 8), no[0][:-1].view(-1, 8)[:, ORDER].to(torch.bfloat16))
    s.synchronize()
    assert ctx.device_status() == 0
