"""The batched int4 matmul (3..128 activation rows, weights through tensor memory) at the edges of its tiles,
stages and work split, against float64."""
import numpy as np
import pytest
import torch

import yscv_b200

pytestmark = pytest.mark.gpu


def _weights(g, n, k):
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    scales = torch.rand(n, k // 32, device="cuda", generator=g) * 0.02 + 0.001
    q = torch.stack([packed & 15, packed >> 4], -1).reshape(n, k).to(torch.int16)
    q = torch.where(q > 7, q - 16, q).double()
    return packed, scales, q * scales.double().repeat_interleave(32, 1)


# (rows, outputs, depth): more work than the dispatch rule asks of each row count; n and k around the
# 128-row tiles, the 256-k units and the CTA ranges
CASES = [(m, n, k) for ms, shapes in [
    ((3, 4), [(43000, 8192), (25000, 8064)]),
    ((5, 8), [(20000, 4096), (2300, 29312), (60001, 1152), (600, 135168)]),
    ((11, 16), [(16400, 4096), (2300, 29312), (60001, 1152), (600, 110080)]),
    ((17, 31, 32), [(23000, 2176), (1650, 30080), (42000, 1152), (380000, 128)]),
    ((33, 48, 64), [(20000, 4096), (2800, 28928), (63000, 1280)]),
    ((65, 100, 128), [(20000, 4096), (2800, 28800), (10241, 8192)]),
    # slices of k: one tile and many, more slices than CTAs of a round, units that do not divide, an odd number of outputs
    ((17, 32, 33, 64, 97, 128), [(1, 128), (127, 384), (129, 256), (300, 16384), (1001, 1152), (2560, 2176), (2048, 5632), (11264, 2048)]),
] for m in ms for n, k in shapes]


@pytest.mark.parametrize("m,n,k", CASES)
def test_batch_rows(m, n, k):
    """Bounds: exact form (m <= 16) 22-bit operands (2^-23 each, relative) and fp32 sums, 1e-6; bf16 form three
    roundings of 2^-9 (uniform: 1.13e-3 each, 2e-3 together), 4e-3."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(m * 7919 + n + k)
    with torch.cuda.stream(stream):
        packed, scales, w = _weights(g, n, k)
        x = torch.randn(m, k, device="cuda", generator=g) * torch.exp(2 * torch.randn(1, k, device="cuda", generator=g))
        out = torch.full((m + 1, n), 7.0, device="cuda")
        h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        first = out.clone()
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        want = x.double() @ w.T
    stream.synchronize()
    assert ctx.device_status() == 0
    assert "tmem" in ctx.last_kernel(), ctx.last_kernel()
    assert torch.equal(first, out)
    assert torch.all(out[m] == 7.0)
    err = float((out[:m].double() - want).norm() / want.norm())
    assert err <= (1e-6 if m <= 16 else 4e-3), err
    if n >= 16:
        rows = (out[:m].double() - want).norm(dim=1) / want.norm(dim=1)
        assert float(rows.max()) <= (2e-6 if m <= 16 else 8e-3), int(rows.argmax())
    ctx.close()


def test_non_finite_rows_stay_in_their_row():
    ctx = yscv_b200.Context(0)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    n, k, m = 20000, 4096, 6
    packed, scales, w = _weights(g, n, k)
    x = torch.randn(m, k, device="cuda", generator=g)
    x[1, 700] = float("nan")
    x[3, 5] = float("inf")
    x[4] = 0.0
    out = torch.empty(m, n, device="cuda")
    torch.cuda.synchronize()
    h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
    ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
    ctx.synchronize()
    assert not torch.isfinite(out[1]).any() and not torch.isfinite(out[3]).any()
    assert torch.all(out[4] == 0.0)
    keep = [0, 2, 5]
    want = x[keep].double() @ w.T
    assert float((out[keep].double() - want).norm() / want.norm()) <= 1e-6
    ctx.close()


@pytest.mark.parametrize("m,n,k", [(300, 19456, 4096), (515, 13001, 2112), (400, 24000, 8192), (257, 19301, 4096)])
def test_split_last_round(m, n, k):
    """The CTA-pair GEMM with few tiles in its last round (their k blocks are cut over all pairs): ragged rows
    and tokens, both stage depths. Bound as above, for every 512-row column of tiles too."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    with torch.cuda.stream(stream):
        packed, scales, w = _weights(g, n, k)
        x = torch.randn(m, k, device="cuda", generator=g)
        out = torch.full((m + 1, n), 7.0, device="cuda")
        h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        report = ctx.dispatch_report()
        first = out.clone()
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        want = x.double() @ w.T
    stream.synchronize()
    assert ctx.device_status() == 0
    assert "split over k" in report and " 0 split over k" not in report, report
    assert torch.equal(first, out)
    assert torch.all(out[m] == 7.0)
    diff = out[:m].double() - want
    assert float(diff.norm() / want.norm()) <= 4e-3
    for n0 in range(0, n, 512):
        assert float(diff[:, n0:n0 + 512].norm() / want[:, n0:n0 + 512].norm()) <= 5e-3, n0
    ctx.close()


@pytest.mark.parametrize("m,n,k", [
    (2048, 14336, 4096), (257, 19301, 4096),                       # two tiles left, 64 k blocks for 74 pairs
    (200, 38400, 1792), (200, 38300, 4096),                        # one tile left, 14 and 32 k blocks
    (130, 38400, 9344), (130, 38400, 9472), (130, 38400, 9600),    # one tile left, 73, 74 and 75 k blocks
    (513, 13312, 2112),                                            # 78 tiles, four left, 64 k per stage
])
def test_split_last_round_reads_only_what_it_wrote(m, n, k):
    """The same GEMM with fewer left-over k blocks than CTA pairs (some pairs then have no part of the last
    round), behind a GEMM that left large values all over the workspace. Bound as above, column by column of
    tiles."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(k + m)
    with torch.cuda.stream(stream):
        packed, scales, _ = _weights(g, 10240, 8192)
        x = torch.full((2048, 8192), 1e6, device="cuda")
        out = torch.empty(2048, 10240, device="cuda")
        h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), 10240, 8192, 32)
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), 2048)
        report = ctx.dispatch_report()
        assert "split over k" in report and " 0 split over k" not in report, report
        packed, scales, w = _weights(g, n, k)
        x = torch.randn(m, k, device="cuda", generator=g)
        out = torch.full((m + 1, n), 7.0, device="cuda")
        h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        report = ctx.dispatch_report()
        want = x.double() @ w.T
    stream.synchronize()
    assert ctx.device_status() == 0
    assert "split over k" in report and " 0 split over k" not in report, report
    assert torch.all(out[m] == 7.0)
    diff = out[:m].double() - want
    for n0 in range(0, n, 512):
        assert float(diff[:, n0:n0 + 512].norm() / want[:, n0:n0 + 512].norm()) <= 5e-3, n0
    ctx.close()


def test_workspace_is_taken_by_the_first_call():
    """A context that runs no such call does not hold its 39 MB; inside a capture, where nothing may be allocated,
    a first call takes the kernel for smaller matrices."""
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    assert free - torch.cuda.mem_get_info()[0] <= 8 << 20
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    n, k, m = 20000, 4096, 8
    with torch.cuda.stream(stream):
        packed, scales, w = _weights(g, n, k)
        x = torch.randn(m, k, device="cuda", generator=g)
        out = torch.empty(m, n, device="cuda")
        small = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), 64, k, 32)
        large = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        ctx.int4_matmul_dev(small, x.data_ptr(), out.data_ptr(), m)     # sizes the scratch of this k
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            ctx.int4_matmul_dev(large, x.data_ptr(), out.data_ptr(), m)
        assert "tmem" not in ctx.last_kernel()
        want = x.double() @ w.T
        for again in range(2):
            out.zero_()
            graph.replay() if not again else ctx.int4_matmul_dev(large, x.data_ptr(), out.data_ptr(), m)
            stream.synchronize()
            assert float((out.double() - want).norm() / want.norm()) <= 2e-6
    assert "tmem" in ctx.last_kernel()
    assert ctx.device_status() == 0
    del graph
    ctx.close()


@pytest.mark.parametrize("n,k", [(20000, 4096), (16400, 4224)])
def test_infinite_and_tiny_activations(n, k):
    """Up to 16 rows, what a sum of fp32 products gives: an infinity times a weight of 0 is NaN, else the weight's
    sign says which infinity, whatever else the row holds; rows of 1e-30 and of subnormals keep their values
    (the bound for subnormals, which have 2^-149 as their last place: 1e-3)."""
    ctx = yscv_b200.Context(0)
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    packed, scales, w = _weights(g, n, k)
    x = torch.randn(5, k, device="cuda", generator=g)
    x[0, 700] = float("inf")
    x[0, 701] = -3e38
    x[1, k - 1] = -float("inf")
    x[2] *= 1e-30
    x[3] *= 1e-40
    out = torch.empty(5, n, device="cuda")
    torch.cuda.synchronize()
    h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
    ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), 5)
    ctx.synchronize()
    assert "tmem" in ctx.last_kernel()
    for row, col, sign in ((0, 700, 1.0), (1, k - 1, -1.0)):
        want = torch.where(w[:, col] == 0, torch.nan, torch.sign(w[:, col]) * sign * torch.inf).float()
        assert torch.equal(torch.nan_to_num(out[row], 7.0, 1.0, -1.0), torch.nan_to_num(want, 7.0, 1.0, -1.0))
    for row, bound in ((2, 1e-6), (3, 1e-3), (4, 1e-6)):
        want = x[row].double() @ w.T
        assert float((out[row].double() - want).norm() / want.norm()) <= bound, row
    ctx.close()


@pytest.mark.parametrize("m,n,k,form", [
    (129, 1000, 4096, "slices"), (200, 8192, 4096, "slices"), (300, 2048, 2112, "slices"), (700, 520, 8192, "slices"), (1000, 2048, 2048, "slices"),
    (257, 14336, 1088, "pairs"), (300, 14336, 4096, "pairs"), (700, 8200, 2048, "pairs"), (1000, 14336, 2112, "pairs"), (1001, 14335, 1024, "pairs"),
    (600, 57344, 1024, "pairs"), (1030, 38400, 2048, "pairs"),
])
def test_prompt_tiles(m, n, k, form):
    """Prompt matmuls that leave SMs idle with tiles of 256 tokens: k in slices (one or more tiles of tokens), CTA-pair tiles of
    fewer tokens, fewer pair tiles than pairs, a split last round of narrow tiles; bounds as above, row by row too."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(n + m)
    with torch.cuda.stream(stream):
        packed, scales, w = _weights(g, n, k)
        x = torch.randn(m, k, device="cuda", generator=g)
        out = torch.full((m + 1, n), 7.0, device="cuda")
        h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        report = ctx.dispatch_report()
        first = out.clone()
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        want = x.double() @ w.T
    stream.synchronize()
    assert ctx.device_status() == 0
    if form == "slices":
        assert "K slice(s)" in report and " 1 K slice(s)" not in report, report
    else:
        assert "cta_group::2" in report and "rows x 256 tokens" not in report, report
    assert torch.equal(first, out)
    assert torch.all(out[m] == 7.0)
    diff = out[:m].double() - want
    assert float(diff.norm() / want.norm()) <= 4e-3
    assert float((diff.norm(dim=1) / want.norm(dim=1)).max()) <= 8e-3
    for n0 in range(0, n, 512):
        assert float(diff[:, n0:n0 + 512].norm() / want[:, n0:n0 + 512].norm()) <= 8e-3, n0
    ctx.close()


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k", [(100, 256), (4736, 1280), (4800, 1536), (4737, 1792), (2048, 4352), (6000, 6912), (300, 8448), (4737, 6656),
                                 (2048, 2048), (2048, 2304), (2048, 2560), (2048, 3584), (2048, 4608), (2500, 4096), (19000, 3840)])
def test_few_rows_depths(m, n, k):
    """The few-row matmul where its last stage ends in half, and on both sides of the line between quantising the rows in the
    kernel and before it: 21-bit blocks of 32 values (2^-22 of the block's maximum each, about four times its rms) and fp32 sums, 2e-6."""
    stream = torch.cuda.Stream()
    ctx = yscv_b200.Context(0, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(n + k)
    with torch.cuda.stream(stream):
        packed, scales, w = _weights(g, n, k)
        x = torch.randn(m, k, device="cuda", generator=g)
        out = torch.full((m + 1, n), 7.0, device="cuda")
        h = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        ctx.int4_matmul_dev(h, x.data_ptr(), out.data_ptr(), m)
        want = x.double() @ w.T
    stream.synchronize()
    assert ctx.device_status() == 0 and "int4_gemv_fast" in ctx.last_kernel()
    assert torch.all(out[m] == 7.0)
    assert float((out[:m].double() - want).norm() / want.norm()) <= 2e-6
    ctx.close()
