"""tcgen05 grouped expert GEMM against a PyTorch FP32 reference: ragged expert sizes (including empty
experts, sizes that are no multiple of a tile's rows, aligned gaps), plain and SwiGLU epilogues."""

import pytest
import torch

from pcie_ep_b200.ops.grouped_ffn import grouped_gemm, grouped_gemm_reference, grouped_swiglu_ffn, quantize_weights_fp8
from pcie_ep_b200.quantization import quantize_fp8_reference

pytestmark = pytest.mark.gpu


def _layout(counts, alignment=1):
    counts = torch.tensor(counts, dtype=torch.int32)
    padded = (counts + alignment - 1) // alignment * alignment
    offsets = torch.zeros(len(counts) + 1, dtype=torch.int32)
    offsets[1:] = padded.cumsum(0)
    return offsets, counts


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("n", [384, 512])  # plain GEMM: a last tile with the channels of one CTA / whole tiles
@pytest.mark.parametrize("counts,alignment", [([128], 1), ([5, 0, 300, 129, 1, 0, 77, 256], 1), ([40, 130, 0, 9], 16)])
def test_grouped_gemm_matches_reference(ext, swiglu, n, counts, alignment):
    torch.manual_seed(0)
    k = 256
    offsets, cnts = _layout(counts, alignment)
    rows = int(offsets[-1]) + 37  # spare capacity behind the last expert
    a = (torch.randn(rows, k) * 0.5).to(torch.bfloat16).cuda()
    w = (torch.randn(len(counts), (2 if swiglu else 1) * n, k) * 0.05).to(torch.bfloat16).cuda()
    out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    grouped_gemm(a, w, offsets.cuda(), cnts.cuda(), swiglu=swiglu, out=out, status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    want = grouped_gemm_reference(a.cpu(), w.cpu(), offsets, cnts, swiglu)
    valid = torch.zeros(rows, dtype=torch.bool)
    for e, c in enumerate(counts):
        valid[int(offsets[e]):int(offsets[e]) + c] = True
    got = out.cpu().float()
    assert torch.allclose(got[valid], want[valid], rtol=2e-2, atol=2e-2), (got[valid] - want[valid]).abs().max()
    assert (got[~valid] == 7.0).all(), "rows outside every expert must not be written"


def test_swiglu_ffn_two_stage(ext):
    torch.manual_seed(1)
    hidden, inter = 512, 256
    offsets, cnts = _layout([200, 3, 0, 131])
    rows = int(offsets[-1])
    x = (torch.randn(rows, hidden) * 0.5).to(torch.bfloat16).cuda()
    w13 = (torch.randn(4, 2 * inter, hidden) * 0.03).to(torch.bfloat16).cuda()
    w2 = (torch.randn(4, hidden, inter) * 0.03).to(torch.bfloat16).cuda()
    y = grouped_swiglu_ffn(x, w13, w2, offsets.cuda(), cnts.cuda())
    torch.cuda.synchronize()
    h = grouped_gemm_reference(x.cpu(), w13.cpu(), offsets, cnts, True).to(torch.bfloat16)
    want = grouped_gemm_reference(h, w2.cpu(), offsets, cnts, False)
    assert torch.allclose(y.cpu().float(), want, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("swiglu", [False, True])
def test_grouped_gemm_fp8_matches_dequantised_reference(ext, swiglu):
    """E4M3 operands on kind::f8f6f4 with per-row / per-channel scales in the epilogue: exact w.r.t. the
    quantised operands up to FP32 accumulation order and the BF16 output rounding."""
    torch.manual_seed(2)
    k, n = 512, 256
    counts = [70, 0, 200, 129, 3]
    offsets, cnts = _layout(counts)
    rows = int(offsets[-1]) + 11
    a = torch.randn(rows, k) * 0.7
    a[5] *= 40.0  # an outlier row gets its own scale
    codes, a_scales = quantize_fp8_reference(a)
    a8 = codes.view(torch.float8_e4m3fn)
    w = torch.randn(len(counts), (2 if swiglu else 1) * n, k) * 0.05
    w8, w_scales = quantize_weights_fp8(w)
    out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    grouped_gemm(a8.cuda(), w8.cuda(), offsets.cuda(), cnts.cuda(), swiglu=swiglu, out=out, status=status,
                 a_scales=a_scales.cuda(), w_scales=w_scales.cuda())
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    want = grouped_gemm_reference(a8, w8, offsets, cnts, swiglu, a_scales, w_scales)
    valid = torch.zeros(rows, dtype=torch.bool)
    for e, c in enumerate(counts):
        valid[int(offsets[e]):int(offsets[e]) + c] = True
    got = out.cpu().float()
    scale = float(want[valid].abs().max())
    assert torch.allclose(got[valid], want[valid], rtol=2e-2, atol=1e-2 * scale), (got[valid] - want[valid]).abs().max()
    assert (got[~valid] == 7.0).all()


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("swiglu,n", [(True, 256), (False, 256), (False, 128)])
def test_last_tiles_at_the_box_heights(ext, fp8, swiglu, n):
    """Experts whose last tile ends at, before and behind steps of a tile's width (two activation boxes of 8 to 128 rows).  The
    rows around an expert's own hold NaN: what shares a box with it must not reach its results, nor be written."""
    counts = [31, 32, 33, 0, 63, 64, 65, 127, 128, 1, 128 + 32, 128 + 33, 128 + 64, 128 + 65]
    k, experts = 384, len(counts)
    offsets = torch.zeros(experts + 1, dtype=torch.int32)
    for e, c in enumerate(counts):
        offsets[e + 1] = offsets[e] + c + (1, 40, 0, 7)[e % 4]  # rows between the experts: none, few, more than a box
    rows = int(offsets[-1]) + 5
    gen = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(rows, k, device="cuda", generator=gen).to(torch.bfloat16)
    own = torch.zeros(rows, dtype=torch.bool, device="cuda")
    for e, c in enumerate(counts):
        own[int(offsets[e]):int(offsets[e]) + c] = True
    a[~own] = float("nan")
    w = (torch.randn(experts, (2 if swiglu else 1) * n, k, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
    scales = {}
    if fp8:
        a, w = a.to(torch.float8_e4m3fn), w.to(torch.float8_e4m3fn)
        scales = dict(a_scales=torch.rand(rows, device="cuda", generator=gen) + 0.5, w_scales=torch.rand(w.shape[:2], device="cuda", generator=gen) + 0.5)
    out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    grouped_gemm(a, w, offsets.cuda(), torch.tensor(counts, dtype=torch.int32, device="cuda"), swiglu=swiglu, out=out, status=status, **scales)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0] and bool((out[~own] == 7.0).all())
    for e, c in enumerate(counts):
        at = slice(int(offsets[e]), int(offsets[e]) + c)
        x, m = a[at].double(), w[e].double()
        if fp8:
            x, m = x * scales["a_scales"][at].double().unsqueeze(1), m * scales["w_scales"][e].double().unsqueeze(1)
        want = x @ m.t()
        # K products summed in 32 bits (and two scale factors): relative to the sum of their magnitudes
        error = (x.abs() @ m.abs().t()) * (k + 4) * 2.0 ** -24
        if swiglu:
            gate, up = want[:, :n], want[:, n:]
            silu = torch.nn.functional.silu(gate)
            # |silu'| < 1.1; the fast exponential is good to 2 + 1.2 |gate| units in the last of 24 bits
            error = 1.1 * error[:, :n] * up.abs() + silu.abs() * error[:, n:] + (silu * up).abs() * (8 + 2 * gate.abs()) * 2.0 ** -24
            want = silu * up
        assert bool(((out[at].double() - want).abs() <= error + (want.abs() + error) * 2.0 ** -8).all()), counts[e]


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("swiglu", [True, False])
@pytest.mark.parametrize("k", [128, 1152])
def test_tiles_of_every_width(ext, fp8, swiglu, k):
    """Tiles of 16 to 256 rows in steps of 16 (one expert each, and several chunks per expert), K shorter and longer than the ring
    of stages, and output columns that leave the second CTA of the last pair without channels."""
    _check_tiles([1, 17, 33, 49, 65, 81, 97, 113, 129, 145, 161, 177, 193, 209, 225, 256, 257, 0, 289, 511, 513, 770, 1025], 384, k, fp8, swiglu)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("swiglu", [True, False])
def test_more_row_chunks_than_a_group(ext, fp8, swiglu):
    """Tiles go by groups of eight row chunks: experts with exactly one group, one and two chunks more, two full groups and a part."""
    _check_tiles([2048, 2049, 3, 2304 + 1, 4096, 0, 4625], 640, 128, fp8, swiglu)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("swiglu", [True, False])
@pytest.mark.parametrize("widest", [16, 48, 80, 112, 144, 176, 224])
def test_rings_of_every_depth(ext, fp8, swiglu, widest):
    """The ring has as many stages as fit for the widest tile of the launch (ten for 16 rows, six for 224).  Twenty-five K blocks a
    tile and several tiles per pair of CTAs: the ring turns over many times, at another stage in every tile."""
    _check_tiles([widest if e % 5 == 0 else max(1, widest - 7 * (e % 9)) for e in range(24)], 2048, 25 * (128 if fp8 else 64), fp8, swiglu)


def _check_tiles(counts, n, k, fp8, swiglu):
    experts = len(counts)
    offsets, cnts = _layout(counts)
    rows = int(offsets[-1])
    gen = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(rows, k, device="cuda", generator=gen).to(torch.bfloat16)
    w = (torch.randn(experts, (2 if swiglu else 1) * n, k, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
    scales = {}
    if fp8:
        x, w = x.to(torch.float8_e4m3fn), w.to(torch.float8_e4m3fn)
        scales = dict(a_scales=torch.rand(rows, device="cuda", generator=gen) + 0.5, w_scales=torch.rand(w.shape[:2], device="cuda", generator=gen) + 0.5)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = grouped_gemm(x, w, offsets.cuda(), cnts.cuda(), swiglu=swiglu, status=status, **scales)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    for e, c in enumerate(counts):
        at = slice(int(offsets[e]), int(offsets[e]) + c)
        a, m = x[at].double(), w[e].double()
        if fp8:
            a, m = a * scales["a_scales"][at].double().unsqueeze(1), m * scales["w_scales"][e].double().unsqueeze(1)
        want = a @ m.t()
        # as in test_last_tiles_at_the_box_heights: K products summed in 32 bits, the fast exponential, one rounding to BF16
        error = (a.abs() @ m.abs().t()) * (k + 4) * 2.0 ** -24
        if swiglu:
            gate, up = want[:, :n], want[:, n:]
            silu = torch.nn.functional.silu(gate)
            error = 1.1 * error[:, :n] * up.abs() + silu.abs() * error[:, n:] + (silu * up).abs() * (8 + 2 * gate.abs()) * 2.0 ** -24
            want = silu * up
        assert bool(((out[at].double() - want).abs() <= error + (want.abs() + error) * 2.0 ** -8).all()), c


def test_swiglu_of_extreme_gates(ext):
    """gate / (1 + exp(-gate)) where the exponential over- or underflows, and of values that are no numbers."""
    gates = torch.tensor([0.0, -0.0, 1e-30, -1e-30, 20.0, -20.0, 80.0, -80.0, -87.0, -88.0, -88.5, -89.0, 89.0, -104.0, 3e38, -3e38, float("inf"),
                          -float("inf"), float("nan")] + [0.5 * i - 27.0 for i in range(109)]).to(torch.bfloat16)
    n, k = 128, 128
    assert gates.numel() == n
    w = torch.zeros(1, 2 * n, k, dtype=torch.bfloat16)
    w[0, :n, 0], w[0, n:, 0] = gates, 1.0
    x = torch.zeros(1, k, dtype=torch.bfloat16)
    x[0, 0] = 1.0
    got = grouped_gemm(x.cuda(), w.cuda(), torch.tensor([0, 1], dtype=torch.int32).cuda(), torch.tensor([1], dtype=torch.int32).cuda(), swiglu=True).cpu()[0]
    g = gates.float()
    want = (g.double() / (1.0 + torch.exp(-g.double()))).float()
    want[g == -float("inf")] = float("nan")
    assert torch.equal(got.isnan(), want.isnan())
    same = ~want.isnan()
    # a rounding to BF16; below -88 the 32-bit exponential is infinite and the quotient zero
    assert bool(((got.float() - want)[same].abs() <= want[same].abs() * 2.0 ** -8 + 1e-36).logical_or(got.float()[same] == want[same]).all())


def test_swiglu_division_in_32_bits(ext):
    """gate / (1 + exp(-gate)) before anything rounds it to BF16, and the division alone over all exponents, against 64 bits.  The
    bound: half a unit in the last place and 2^-20 of one, two units of the subnormal numbers (the remainder may be one), and |a| of
    them where the reciprocal of b is."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    gate = torch.cat([torch.randn(1 << 20, device="cuda", generator=gen) * 4, torch.linspace(-89, 89, 1 << 20, device="cuda"),
                      torch.linspace(-1e-3, 1e-3, 1 << 16, device="cuda")])
    mantissa = torch.rand(1 << 20, device="cuda", generator=gen) + 1.0
    exponent = torch.randint(0, 128, (1 << 20,), device="cuda", generator=gen)
    wide = torch.ldexp(torch.rand(1 << 20, device="cuda", generator=gen) * 2 - 1, torch.randint(-100, 127, (1 << 20,), device="cuda", generator=gen))
    a = torch.cat([gate, wide])
    b = torch.cat([1.0 + torch.exp(-gate), torch.ldexp(mantissa, exponent)])
    got, finite = ext.litmus_quotients(a, b), b.isfinite()
    want = a.double() / b.double()
    error = (got.double() - want).abs()
    bound = want.abs() * 2.0 ** -24 * (1 + 2.0 ** -20) + torch.where(b >= 2.0 ** 126, a.abs().double() + 2, 2.0) * 2.0 ** -149
    assert bool((error <= bound)[finite].all()), (error / bound)[finite].max()
    # an infinite sum, and operands that are no numbers: as the operator has it
    inf, nan = float("inf"), float("nan")
    a = torch.tensor([-88.9, -inf, inf, 0.0, -0.0, nan, 1.0, inf, 3e38, -3e38], device="cuda")
    b = torch.tensor([inf, inf, 1.0, 2.0, 2.0, inf, nan, inf, 1.0, inf], device="cuda")
    got, want = ext.litmus_quotients(a, b), a / b
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~want.isnan()], want[~want.isnan()])


@pytest.mark.parametrize("side_stream", [False, True])
def test_launches_that_start_early_see_what_the_ones_before_wrote(ext, side_stream):
    """The GEMM's CTAs come where those of the launch before have ended: its operands, counts and offsets are written by kernels
    directly in front of it and overwritten directly behind it, on the default stream and on another, eagerly and in a graph."""
    experts, rows, k, n = 8, 40, 1024, 512
    gen = torch.Generator(device="cuda").manual_seed(1)
    base = torch.randn(experts * rows, k, device="cuda", generator=gen).to(torch.bfloat16)
    up = (torch.randn(experts, n, k, device="cuda", generator=gen) * 0.05).to(torch.bfloat16)
    down = (torch.randn(experts, k, n, device="cuda", generator=gen) * 0.05).to(torch.bfloat16)
    offsets, counts = torch.arange(experts + 1, dtype=torch.int32, device="cuda") * rows, torch.full((experts,), rows, dtype=torch.int32, device="cuda")
    x, at, count = torch.zeros_like(base), torch.zeros_like(offsets), torch.zeros_like(counts)
    h = torch.zeros(experts * rows, n, dtype=torch.bfloat16, device="cuda")
    y, status = torch.zeros_like(base), torch.zeros(4, dtype=torch.int32, device="cuda")

    def layer(scale):
        at.copy_(offsets)
        count.copy_(counts)
        torch.mul(base, scale, out=x)
        grouped_gemm(x, up, at, count, out=h, status=status)
        grouped_gemm(h, down, at, count, out=y, status=status)
        got = y.clone()
        for t in (x, h, y, at, count):
            t.zero_()
        return got

    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        results = [layer(2.0 ** (i % 3)) for i in range(60)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = layer(2.0)
    for _ in range(20):
        graph.replay()
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    # scaling by two is exact all the way
    want = torch.cat([(base[e * rows:(e + 1) * rows].double() @ up[e].double().t()).to(torch.bfloat16).double() @ down[e].double().t() for e in range(experts)])
    assert float((results[0].double() - want).norm() / want.norm()) < 2.0 ** -8
    for i, got in enumerate(results):
        assert torch.equal(got, results[0] * 2.0 ** (i % 3)), i
    assert torch.equal(replayed, results[1])


@pytest.mark.parametrize("beyond", [-1, 0, 630])
def test_long_gate_up_launches_are_the_short_ones(ext, beyond):
    """Around the size from which MMAs keep a gap (rows x channels x K of 1.5e9 per SM): the same bits as in two launches of half as many
    rows, and a sample of rows against 64 bits."""
    n, k = 4096, 7168
    rows = -(-1500 * 10 ** 6 * (torch.cuda.get_device_properties(0).multi_processor_count // 2 * 2) // (n * k)) + beyond
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, k, device="cuda", generator=gen).to(torch.bfloat16)
    w = (torch.randn(1, 2 * n, k, device="cuda", generator=gen) * 0.02).to(torch.bfloat16)

    def gemm(first, count):
        out = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
        status = torch.zeros(4, dtype=torch.int32, device="cuda")
        grouped_gemm(x, w, torch.tensor([first, first + count], dtype=torch.int32, device="cuda"), torch.tensor([count], dtype=torch.int32, device="cuda"),
                     swiglu=True, out=out, status=status)
        assert status.tolist() == [0, 0, 0, 0]
        return out

    whole, half = gemm(0, rows), rows // 2
    assert torch.equal(whole[:half], gemm(0, half)[:half]) and torch.equal(whole[half:], gemm(half, rows - half)[half:])
    at = torch.tensor([0, 255, 256, rows // 2, rows - 1], device="cuda")
    both = x[at].double() @ w[0].double().t()
    size = (x[at].double().abs() @ w[0].double().abs().t()) * (k + 4) * 2.0 ** -24
    gate, up = both[:, :n], both[:, n:]
    silu = torch.nn.functional.silu(gate)
    # as in test_last_tiles_at_the_box_heights
    error = 1.1 * size[:, :n] * up.abs() + silu.abs() * size[:, n:] + (silu * up).abs() * (8 + 2 * gate.abs()) * 2.0 ** -24
    want = silu * up
    assert bool(((whole[at].double() - want).abs() <= error + (want.abs() + error) * 2.0 ** -8).all())


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("counts", [[1], [0, 0, 0], [40] * 24, [700, 3, 0, 55, 513, 16, 2100, 9], [256] * 90])
def test_linked_launches_are_the_unlinked_ones(ext, counts, fp8):
    """Gate/up and down projection of which the second starts on its experts while the first is at work: the same bits as one after
    the other, pass after pass on one set of counters, with other inputs in between, and the counters zero behind each pass."""
    hidden, inter = 512, 384  # three channel tiles of the first, two of the second, the last with one CTA's channels in both
    offsets, cnts = _layout(counts)
    rows = int(offsets[-1])
    gen = torch.Generator(device="cuda").manual_seed(len(counts))
    w13 = (torch.randn(len(counts), 2 * inter, hidden, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
    w2 = (torch.randn(len(counts), 128 * 3, inter, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
    offsets, cnts = offsets.cuda(), cnts.cuda()
    progress = torch.zeros(len(counts) + 1, dtype=torch.int32, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    h = torch.zeros(max(1, rows), inter, dtype=torch.bfloat16, device="cuda")
    for _ in range(4):
        x = torch.randn(max(1, rows), hidden, device="cuda", generator=gen).to(torch.bfloat16)
        scales = {}
        if fp8:
            scales = dict(a_scales=torch.rand(x.shape[0], device="cuda", generator=gen) + 0.5, w_scales=torch.rand(w13.shape[:2], device="cuda", generator=gen) + 0.5)
        operands = (x.to(torch.float8_e4m3fn), w13.to(torch.float8_e4m3fn)) if fp8 else (x, w13)
        outs = []
        for first, second in (((None, 0), (None, 0)), ((progress, 0), (progress, inter))):
            h.zero_()
            out = torch.zeros(h.shape[0], w2.shape[1], dtype=torch.bfloat16, device="cuda")
            grouped_gemm(*operands, offsets, cnts, swiglu=True, out=h, status=status, _link=first, **scales)
            grouped_gemm(h, w2, offsets, cnts, out=out, status=status, _link=second)
            outs.append(out)
        assert torch.equal(outs[0], outs[1]) and (rows == 0 or float(outs[0].float().abs().max()) > 0)
        assert int(progress.abs().max()) == 0
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("limit", [(), (300,)])
def test_a_second_launch_whose_rows_never_come_gives_up(ext, limit):
    """Linked to a first launch that was never made: the bounded wait runs out when it says, the status says so, nothing is written, and
    the counters are as a pass leaves them."""
    counts = torch.tensor([5, 7], dtype=torch.int32, device="cuda")
    offsets = torch.tensor([0, 5, 12], dtype=torch.int32, device="cuda")
    a, w = torch.ones(12, 64, dtype=torch.bfloat16, device="cuda"), torch.ones(2, 128, 64, dtype=torch.bfloat16, device="cuda")
    out, status = torch.full((12, 128), 7.0, dtype=torch.bfloat16, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    progress = torch.zeros(3, dtype=torch.int32, device="cuda")
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    begin.record()
    grouped_gemm(a, w, offsets, counts, out=out, status=status, _link=(progress, 64, *limit))
    end.record()
    torch.cuda.synchronize()
    # (three tenths of a second or two; not measured closer: the GPU's clock and its host are other things')
    assert (begin.elapsed_time(end) < 1000) == bool(limit) and begin.elapsed_time(end) > 250
    assert status.tolist()[0] == 1 and bool((out == 7.0).all()) and progress.tolist() == [0, 0, 0]
    for bad in ((progress[:2], 64), (progress.float(), 64), (progress, -1), (progress, 0)):  # (the last: a plain GEMM is no first launch)
        with pytest.raises(ValueError):
            grouped_gemm(a, w, offsets, counts, out=out, status=status, _link=bad)
    status.zero_()
    grouped_gemm(a, w, offsets, counts, out=out, status=status)
    assert bool((out == 64.0).all()) and status.tolist()[0] == 0
