"""Prompt-pass attention (tcgen05, fp32 operands as two scaled fp16 terms) at the edges of its tiles, rings and
number range, against float64."""
import math

import pytest
import torch

import yscv_b200

pytestmark = pytest.mark.gpu


def _context():
    stream = torch.cuda.Stream()
    return yscv_b200.Context(0, stream=stream.cuda_stream), stream


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _call(ctx, q, k, v, p0, causal=True, ks=None, vs=None, stride=None, shift=0):
    """q [B, seq, n_q, d], caches [B, max_seq, n_kv, d]; stride and shift: floats between query rows and in front
    of the first."""
    B, seq, n_q, d = q.shape
    max_seq, n_kv = k.shape[1:3]
    stride = stride or n_q * d
    buf = torch.zeros(B * seq * stride + shift, device="cuda")
    buf[shift:].view(B * seq, stride)[:, :n_q * d] = q.reshape(B * seq, n_q * d)
    out = torch.full((B * seq * n_q * d + 16,), 3.0, device="cuda")
    pos = torch.full((1,), p0, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    if ks is None:
        ctx.gqa_attention_dev(buf[shift:].data_ptr(), stride, B, seq, n_q, n_kv, d, k.data_ptr(), v.data_ptr(), max_seq,
                              pos.data_ptr(), causal, out.data_ptr())
    else:
        ctx.gqa_attention_i8_dev(buf[shift:].data_ptr(), stride, B, seq, n_q, n_kv, d, k.data_ptr(), ks.data_ptr(),
                                 v.data_ptr(), vs.data_ptr(), max_seq, pos.data_ptr(), causal, out.data_ptr())
    ctx.synchronize()
    assert "tcgen05" in ctx.last_kernel()
    assert ctx.device_status() == 0
    assert torch.all(out[-16:] == 3.0)
    return out[:-16].view(B, seq, n_q, d)


def _exact(q, k, v, p0, causal=True):
    B, seq, n_q, d = q.shape
    n_kv, total = k.shape[2], p0 + seq
    qd = q.double().view(B, seq, n_kv, n_q // n_kv, d)
    s = torch.einsum("bqhgd,bkhd->bhgqk", qd, k[:, :total].double()) / math.sqrt(d)
    if causal:
        hidden = torch.arange(total, device="cuda")[None, :] > p0 + torch.arange(seq, device="cuda")[:, None]
        s.masked_fill_(hidden, -math.inf)
    return torch.einsum("bhgqk,bkhd->bqhgd", torch.softmax(s, -1), v[:, :total].double()).reshape(B, seq, n_q, d)


def _check(got, want, overall=1e-6, row=1e-5):
    """Bounds for scores of a few units: operands of 22 bits (2^-23 each, two per product), about ten truncated
    sums of 2^-24 per tile, and the scores' absolute error (their size times the same) in the exponent: 3e-7 of
    the whole measured; a single row, whose weighted values may cancel to a tenth of their size, ten times that."""
    diff = got.double() - want
    assert float(diff.norm() / want.norm()) <= overall
    assert float((diff.norm(dim=-1) / want.norm(dim=-1)).max()) <= row


@pytest.mark.parametrize("B,seq,p0,n_q,n_kv,d,causal", [
    (1, 16, 0, 4, 4, 64, True),          # the fewest positions, one head per KV head
    (2, 17, 300, 17, 1, 64, True),       # 7 positions of 17 heads to a tile of 128; six key tiles: the ring of four wraps
    (1, 700, 0, 6, 2, 64, True),
    (3, 129, 64, 64, 1, 128, True),      # two positions to a tile
    (1, 40, 333, 128, 1, 128, True),     # one position to a tile
    (2, 515, 0, 16, 2, 128, True),       # nine key tiles: ring of two, four alpha slots
    (1, 100, 190, 8, 2, 64, False),
])
@pytest.mark.parametrize("stride,shift", [(0, 0), (4, 1), (3, 0)])
def test_shapes_and_query_alignment(B, seq, p0, n_q, n_kv, d, causal, stride, shift):
    ctx, _ = _context()
    g = _generator(seq * 7 + d)
    q = torch.randn(B, seq, n_q, d, device="cuda", generator=g)
    k, v = (torch.randn(B, p0 + seq + 70, n_kv, d, device="cuda", generator=g) for _ in range(2))
    k[:, p0 + seq:], v[:, p0 + seq:] = float("nan"), float("inf")     # rows behind the prompt are not read
    got = _call(ctx, q, k, v, p0, causal, stride=n_q * d + stride, shift=shift)
    _check(got, _exact(q, k, v, p0, causal))
    ctx.close()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("spread", [0.05, 6.0])
def test_flat_and_sharp_scores(d, spread):
    """Scores of std 6 (weights from 1 down to e^-50): their errors in the exponent are ten times larger."""
    ctx, _ = _context()
    g = _generator(d)
    q = torch.randn(1, 300, 8, d, device="cuda", generator=g) * spread
    k, v = (torch.randn(1, 300, 2, d, device="cuda", generator=g) for _ in range(2))
    _check(_call(ctx, q, k, v, 0), _exact(q, k, v, 0), *((1e-6, 1e-5) if spread < 1 else (3e-6, 5e-5)))
    ctx.close()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kv_int8", [False, True])
@pytest.mark.parametrize("what,value", [("v", math.nan), ("v", math.inf), ("k", math.nan), ("k", -math.inf), ("v", 1e6),
                                        ("k", 1e6), ("v", 1e30)])
def test_a_key_reaches_only_who_attends_to_it(d, kv_int8, what, value):
    """Row t of one KV head's keys or values is not finite, or far larger than its neighbours: the positions in
    front of it, and the other heads, keep their values and their precision."""
    ctx, _ = _context()
    g = _generator(d + kv_int8)
    seq, t, n_q, n_kv = 200, 90, 8, 2
    q = torch.randn(1, seq, n_q, d, device="cuda", generator=g)
    ks = vs = None
    if kv_int8:   # (a scale belongs to the row of all heads)
        k8, v8 = (torch.randint(-127, 128, (1, seq, n_kv, d), dtype=torch.int8, device="cuda", generator=g) for _ in range(2))
        ks, vs = (torch.rand(1, seq, device="cuda", generator=g) * 0.01 + 0.01 for _ in range(2))
        (ks if what == "k" else vs)[0, t] *= value
        k, v = k8.float() * ks[:, :, None, None], v8.float() * vs[:, :, None, None]
        got = _call(ctx, q, k8, v8, 0, ks=ks, vs=vs)
    else:
        k, v = (torch.randn(1, seq, n_kv, d, device="cuda", generator=g) for _ in range(2))
        (k if what == "k" else v)[0, t, 1] *= value
        got = _call(ctx, q, k, v, 0)
    want = _exact(q, k, v, 0)
    _check(got[:, :t], _exact(q[:, :t], k, v, 0))
    if not kv_int8:
        _check(got[:, :, :4], want[:, :, :4])
    if not math.isfinite(value):
        # (keys of -inf: scores of both signs, or no weight where the query's sign says so)
        assert what == "k" or not torch.isfinite(got[:, t:, 4:]).any()
        assert torch.isfinite(got[:, :t]).all()
    elif what == "v":
        _check(got, want)
    ctx.close()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("qs,ks,vs", [(1e-20, 1e-20, 1.0), (1e-30, 1.0, 1.0), (1.0, 1.0, 1e-35), (1.0, 1.0, 1e35), (1e-25, 1e25, 1.0),
                                      (1e25, 1e-25, 1e-20), (0.0, 1.0, 1.0), (1.0, 0.0, 1.0)])
def test_magnitudes(d, qs, ks, vs):
    ctx, _ = _context()
    g = _generator(d)
    q = torch.randn(1, 100, 4, d, device="cuda", generator=g) * qs
    k, v = (torch.randn(1, 100, 2, d, device="cuda", generator=g) for _ in range(2))
    k *= ks
    v *= vs
    _check(_call(ctx, q, k, v, 0), _exact(q, k, v, 0))
    ctx.close()


@pytest.mark.parametrize("d", [64, 128])
def test_a_query_row_stays_in_its_row(d):
    ctx, _ = _context()
    g = _generator(d)
    q = torch.randn(1, 60, 8, d, device="cuda", generator=g)
    q[0, 10, 3, 5], q[0, 41, 0, 0] = math.nan, math.inf
    k, v = (torch.randn(1, 60, 2, d, device="cuda", generator=g) for _ in range(2))
    got = _call(ctx, q, k, v, 0)
    bad = torch.zeros(1, 60, 8, dtype=torch.bool, device="cuda")
    bad[0, 10, 3] = bad[0, 41, 0] = True
    assert not torch.isfinite(got[bad]).any()
    want = _exact(torch.nan_to_num(q, nan=0.0, posinf=0.0), k, v, 0)
    _check(got[~bad], want[~bad])
    ctx.close()


@pytest.mark.parametrize("B,n_kv,max_seq,launches", [(3, 2, 80000, 4), (2, 3, 100000, 4), (3, 1, 100000, 4)])
def test_images_of_a_long_cache_in_groups(B, n_kv, max_seq, launches):
    """Caches whose images pass 256 MB: (sequence, KV head) pairs are taken in groups, here six in threes (the
    middle sequence in both), six in whole sequences of three, and two and one."""
    ctx, _ = _context()
    g = _generator(9)
    seq, p0, n_q, d = 20, 1000, 4 * n_kv, 128
    q = torch.randn(B, seq, n_q, d, device="cuda", generator=g)
    k, v = (torch.zeros(B, max_seq, n_kv, d, device="cuda") for _ in range(2))
    for t in (k, v):
        t[:, :p0 + seq] = torch.randn(B, p0 + seq, n_kv, d, device="cuda", generator=g)
    before = ctx.launch_count()
    got = _call(ctx, q, k, v, p0)
    assert ctx.launch_count() - before == launches
    _check(got, _exact(q, k, v, p0))
    ctx.close()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kv_int8", [False, True])
def test_first_call_inside_a_capture(d, kv_int8):
    """A context that has no scratch for the images yet and may not allocate: the call takes the fp32 path."""
    ctx, stream = _context()
    g = _generator(d)
    B, seq, p0, n_q, n_kv, max_seq = 2, 100, 70, 24, 4, 200
    q = torch.randn(B, seq, n_q, d, device="cuda", generator=g)
    pos = torch.full((1,), p0, dtype=torch.int32, device="cuda")
    out = torch.zeros(B, seq, n_q, d, device="cuda")
    if kv_int8:
        k8, v8 = (torch.randint(-127, 128, (B, max_seq, n_kv, d), dtype=torch.int8, device="cuda", generator=g) for _ in range(2))
        ks, vs = (torch.rand(B, max_seq, device="cuda", generator=g) * 0.01 + 0.01 for _ in range(2))
        k, v = k8.float() * ks[:, :, None, None], v8.float() * vs[:, :, None, None]
    else:
        k, v = (torch.randn(B, max_seq, n_kv, d, device="cuda", generator=g) for _ in range(2))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        if kv_int8:
            ctx.gqa_attention_i8_dev(q.data_ptr(), n_q * d, B, seq, n_q, n_kv, d, k8.data_ptr(), ks.data_ptr(), v8.data_ptr(),
                                     vs.data_ptr(), max_seq, pos.data_ptr(), True, out.data_ptr())
        else:
            ctx.gqa_attention_dev(q.data_ptr(), n_q * d, B, seq, n_q, n_kv, d, k.data_ptr(), v.data_ptr(), max_seq,
                                  pos.data_ptr(), True, out.data_ptr())
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        _check(out, _exact(q, k, v, p0))
    assert ctx.device_status() == 0
    del graph
    ctx.close()
