"""The fp32 matmul (LM head) at the edges of its kernels' tiles, units and row counts, against float64."""
import pytest
import torch

import yscv_b200

pytestmark = pytest.mark.gpu


@pytest.fixture()
def sctx():
    stream = torch.cuda.Stream()
    return yscv_b200.Context(0, stream=stream.cuda_stream), stream


def _operands(stream, m, n, k, seed=7):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    with torch.cuda.stream(stream):
        w, x = torch.randn(n, k, device="cuda", generator=g) * 0.02, torch.randn(m, k, device="cuda", generator=g)
        out = torch.full((m * n + 64,), 3.0, device="cuda")
    return w, x, out


def _check(got, w, x, bound):
    m, n = x.shape[0], w.shape[0]
    want = x.double() @ w.double().T
    assert torch.all(got[m * n:] == 3.0)
    err = (got[:m * n].view(m, n).double() - want).norm() / want.norm()
    assert err < bound, float(err)


# one or two 128-row halves per tile, tiles shared by several CTAs (K of 16 units and more) or not, a last unit of
# 32 k, more than one pass of batch rows
@pytest.mark.parametrize("m", [9, 16, 63, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("n,k", [(1, 32), (127, 992), (129, 1024), (257, 1056), (20000, 1024), (9999, 2080), (38000, 64)])
def test_wide_batch(sctx, m, n, k):
    """An accumulator takes 24 truncated additions (2^-23 each at most, half of that on average: 1.4e-6 of its
    partial sum, which is an eighth of the row's with 64 of 4096 k and all of it at k = 64); the two parts of an
    operand leave 2^-21, the chunks' rounded sums less. The bound is 2e-6."""
    ctx, stream = sctx
    w, x, out = _operands(stream, m, n, k)
    ctx.f32_matmul_dev(w.data_ptr(), x.data_ptr(), m, n, k, out.data_ptr())
    stream.synchronize()
    assert "3xtf32" in ctx.last_kernel()
    _check(out, w, x, 2e-6)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("n,k", [(1, 4), (3, 128), (17, 132), (33, 1020), (50, 1028), (40001, 256)])
def test_few_rows(sctx, m, n, k):
    """fp32 sums: a lane's k / 128 chained groups of four and five shuffles, 2^-24 per addition. A row of x with
    an infinity or a NaN leaves the others alone."""
    ctx, stream = sctx
    w, x, out = _operands(stream, m, n, k)
    ctx.f32_matmul_dev(w.data_ptr(), x.data_ptr(), m, n, k, out.data_ptr())
    stream.synchronize()
    bound = 2.0 ** -24 * (4 * (k // 128 + 1) + 5)
    _check(out, w, x, bound)
    if m > 1:
        bad = x.clone()
        bad[m - 1, 0], bad[m - 1, k - 1] = float("inf"), float("nan")
        torch.cuda.synchronize()
        again = out.clone()
        ctx.f32_matmul_dev(w.data_ptr(), bad.data_ptr(), m, n, k, again.data_ptr())
        stream.synchronize()
        assert torch.equal(again[:(m - 1) * n], out[:(m - 1) * n])
        assert not torch.any(torch.isfinite(again[(m - 1) * n:m * n]))


def test_capture_without_workspace(sctx):
    """Inside a capture without an earlier call of the size every CTA takes whole tiles."""
    ctx, stream = sctx
    m, n, k = 16, 20000, 2048
    w, x, out = _operands(stream, m, n, k)
    small_w, small_x, small_out = _operands(stream, 128, 128, 960)   # sizes the activation scratch, needs no parts
    ctx.f32_matmul_dev(small_w.data_ptr(), small_x.data_ptr(), 128, 128, 960, small_out.data_ptr())
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        ctx.f32_matmul_dev(w.data_ptr(), x.data_ptr(), m, n, k, out.data_ptr())
    graph.replay()
    stream.synchronize()
    _check(out, w, x, 2e-6)
    assert ctx.device_status() == 0


def test_argmax_over_partials(sctx):
    """The last index among equal maxima, wherever the blocks' partial results lie."""
    ctx, stream = sctx
    vocab = 32000
    with torch.cuda.stream(stream):
        logits = torch.zeros(5, vocab, device="cuda")
        logits[0, 17] = logits[0, 31999] = 1.0
        logits[1, 0] = 1.0
        logits[2, 12345] = logits[2, 12346] = 2.0
        logits[4] = float("-inf")
        out = torch.empty(5, dtype=torch.int32, device="cuda")
        ctx.argmax_last_dev(logits.data_ptr(), 5, vocab, out.data_ptr())
    stream.synchronize()
    assert out.tolist() == [31999, 0, 12346, 31999, 31999]


@pytest.mark.parametrize("n", [1, 9, 2499, 2500, 4095])
@pytest.mark.parametrize("k", [4, 132, 1028])
def test_few_weight_rows_are_the_same_sums(sctx, n, k):
    """Up to 8 activation rows: fewer weight rows than fill the SMs take a kernel of their own; its columns are the bits of
    those that the other kernel makes of the same rows in a larger matrix."""
    ctx, s = sctx
    with torch.cuda.stream(s):
        g = torch.Generator(device="cuda").manual_seed(n * k)
        w, x = torch.randn(4099, k, device="cuda", generator=g), torch.randn(8, k, device="cuda", generator=g)
        for m in range(1, 9):
            few, many = torch.full((m, n), float("nan"), device="cuda"), torch.empty(m, 4099, device="cuda")
            ctx.f32_matmul_dev(w.data_ptr(), x.data_ptr(), m, n, k, few.data_ptr())
            ctx.f32_matmul_dev(w.data_ptr(), x.data_ptr(), m, 4099, k, many.data_ptr())
            assert torch.equal(few, many[:, :n])
    s.synchronize()
    assert ctx.device_status() == 0
