"""Decode attention (one query per sequence, keys split across blocks) at the edges of its key shares, head
groups and head sizes, against float64."""
import math

import pytest
import torch

import yscv_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n_kv,group", [(16, 2, 3), (48, 1, 8), (64, 2, 12), (64, 3, 1), (80, 2, 5), (128, 2, 8), (128, 1, 17)])
@pytest.mark.parametrize("max_seq,cached", [(129, 0), (130, 129), (300, 127), (300, 128), (300, 256), (700, 699), (2100, 5), (9000, 63),
                                            (9000, 64), (9000, 200), (9000, 1300), (20000, 19000), (2178, 1999)])
@pytest.mark.parametrize("kv_int8", [False, True])
def test_decode_shares(d, n_kv, group, max_seq, cached, kv_int8):
    """Scores of a few units. f32: 32-bit products and sums leave 1e-6 of the output's norm; the bound is 4e-6.
    int8: a weight (exp times the value row's scale, here at least 0.005) is two fp16 terms, the second with an
    absolute error of up to 2^-25: 6e-6 of the largest weights, and with most of n keys far below the largest
    the error of all n meets the norm of the n / 50 that count, sqrt(50) times that; the bound is 4e-5."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(d * 1009 + max_seq + cached)
    batch, n_q, limit = 2, n_kv * group, cached + 1
    with torch.cuda.stream(stream):
        width = (n_q + 2 * n_kv) * d
        q = torch.randn(batch, width, device="cuda", generator=g)
        shape = (batch, max_seq, n_kv, d)
        pos = torch.full((1,), cached, dtype=torch.int32, device="cuda")
        out = torch.full((batch * n_q * d + 8,), 3.0, device="cuda")
        if kv_int8:
            k, v = (torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=g) for _ in range(2))
            ks, vs = (torch.rand(batch, max_seq, device="cuda", generator=g) * 0.03 + 0.005 for _ in range(2))
            kd, vd = k.double() * ks.double()[:, :, None, None], v.double() * vs.double()[:, :, None, None]
            ctx.gqa_attention_i8_dev(q.data_ptr(), width, batch, 1, n_q, n_kv, d, k.data_ptr(), ks.data_ptr(), v.data_ptr(),
                                     vs.data_ptr(), max_seq, pos.data_ptr(), True, out.data_ptr())
        else:
            k, v = (torch.randn(shape, device="cuda", generator=g) for _ in range(2))
            k[:, limit:], v[:, limit:] = float("nan"), float("nan")   # rows that no share may read
            kd, vd = k.double(), v.double()
            ctx.gqa_attention_dev(q.data_ptr(), width, batch, 1, n_q, n_kv, d, k.data_ptr(), v.data_ptr(), max_seq,
                                  pos.data_ptr(), True, out.data_ptr())
        assert "split" in ctx.last_kernel()
        qd = q[:, :n_q * d].double().reshape(batch, n_kv, group, d)
        p = torch.softmax(torch.einsum("bhgd,bshd->bhgs", qd, kd[:, :limit]) / math.sqrt(d), -1)
        want = torch.einsum("bhgs,bshd->bhgd", p, vd[:, :limit]).reshape(-1)
    stream.synchronize()
    got = out[:-8].double()
    assert torch.all(out[-8:] == 3.0)
    assert float((got - want).norm() / want.norm()) <= (4e-5 if kv_int8 else 4e-6)
    ctx.close()


@pytest.mark.parametrize("d", [48, 64, 128])
@pytest.mark.parametrize("kv_int8", [False, True])
def test_shares_of_infinite_scores(d, kv_int8):
    """A whole share of keys with scores of -inf weighs nothing in the merge; a NaN score reaches the output of
    its head and of no other."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    n_q, n_kv, max_seq, cached = 6, 2, 400, 390
    with torch.cuda.stream(stream):
        q = torch.rand(1, n_q * d, device="cuda", generator=g) + 0.1     # (positive: the sign of a score is its key's)
        shape = (1, max_seq, n_kv, d)
        pos = torch.full((1,), cached, dtype=torch.int32, device="cuda")
        out = torch.empty(n_q, d, device="cuda")
        if kv_int8:
            k, v = (torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=g) for _ in range(2))
            k[0, :200] = -torch.randint(1, 128, (200, n_kv, d), device="cuda", generator=g).to(torch.int8)
            ks, vs = (torch.rand(1, max_seq, device="cuda", generator=g) * 0.01 + 0.005 for _ in range(2))
            ks[0, :200] = float("inf")
        else:
            k, v = (torch.randn(shape, device="cuda", generator=g) for _ in range(2))
            k[0, :200, :, 0] = -float("inf")

        def call():
            if kv_int8:
                ctx.gqa_attention_i8_dev(q.data_ptr(), n_q * d, 1, 1, n_q, n_kv, d, k.data_ptr(), ks.data_ptr(), v.data_ptr(),
                                         vs.data_ptr(), max_seq, pos.data_ptr(), True, out.data_ptr())
            else:
                ctx.gqa_attention_dev(q.data_ptr(), n_q * d, 1, 1, n_q, n_kv, d, k.data_ptr(), v.data_ptr(), max_seq,
                                      pos.data_ptr(), True, out.data_ptr())
            return out.clone()

        got = call()
        kd, vd = (k * ks[:, :, None, None], v * vs[:, :, None, None]) if kv_int8 else (k, v)
        kd, vd = kd[0, 200:cached + 1].double(), vd[0, 200:cached + 1].double()
        p = torch.softmax(torch.einsum("hgd,shd->hgs", q.double().view(n_kv, -1, d), kd) / math.sqrt(d), -1)
        want = torch.einsum("hgs,shd->hgd", p, vd).reshape(n_q, d)
        q[0, 2 * d] = float("nan")
        poisoned = call()
    stream.synchronize()
    assert float((got.double() - want).norm() / want.norm()) <= (4e-5 if kv_int8 else 4e-6)
    assert torch.isnan(poisoned[2]).all()
    keep = [0, 1, 3, 4, 5]
    assert torch.equal(poisoned[keep], got[keep])
    ctx.close()
