"""A group of one rank: the kernels without the exchange protocol against the general dispatch kernel, field by field, and
the combine against a sum in 64 bits, where tiles, slices and chunks end."""

import os
import tempfile

import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def one_rank(ext):
    if not dist.is_initialized():
        store = dist.FileStore(os.path.join(tempfile.mkdtemp(prefix="local-store-"), "store"), 1)
        dist.init_process_group("gloo", store=store, rank=0, world_size=1)
    if dist.get_world_size() != 1:
        pytest.skip("needs a process group of one")
    return dist.group.WORLD


# tokens, capacity, experts, top-k, hidden, channels, FP8 rows, expand, alignment
CASES = [
    (0, 16, 8, 2, 64, 4, False, True, 1),            # nothing to send
    (1, 1, 1, 1, 8, 1, False, True, 256),            # one chunk per row, one expert
    (149, 149, 32, 4, 136, 32, False, True, 16),     # one CTA with two tokens, a row that is no multiple of 128 bytes
    (148 * 33, 148 * 33, 16, 2, 64, 128, False, True, 1),  # more than one 32-token chunk per CTA
    (77, 300, 600, 32, 1024, 3, False, True, 7),     # more experts than threads, widest top-k
    (300, 300, 40, 6, 2880, 64, True, True, 8),      # FP8 rows, several row buffers per warp
    (130, 256, 64, 8, 7168, 32, False, False, 1),    # a row per token, fewer row buffers than warps
    (200, 256, 64, 3, 1024, 128, True, False, 1),
    (148 * 49 + 5, 148 * 49 + 5, 16, 2, 64, 128, False, True, 1),  # more tokens than row buffers: the rest is claimed, with gaps
    (2400, 2500, 12, 3, 7168, 64, False, True, 8),   # the same with one row buffer per warp
    (2400, 2400, 8, 2, 7168, 100, True, False, 1),   # and with FP8 rows, a row per token
]
FIELDS = ["unique_count", "expanded_count", "expert_counts", "expert_offsets", "expert_prefix", "source_offsets", "source_expert_prefix",
          "recv_chan_counts"]


@pytest.mark.parametrize("tokens,capacity,experts,topk,hidden,channels,fp8,expand,alignment", CASES)
def test_local_dispatch_and_combine(one_rank, tokens, capacity, experts, topk, hidden, channels, fp8, expand, alignment):
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    gen = torch.Generator().manual_seed(tokens + topk)
    x = torch.randn(tokens, hidden, generator=gen).to(torch.bfloat16)
    idx = torch.rand(tokens, experts, generator=gen).topk(topk, dim=1).indices.to(torch.int64)
    idx[torch.rand(tokens, topk, generator=gen) < 0.2] = -1
    if tokens > 2:
        idx[tokens // 2] = -1  # a token that goes nowhere
    w = torch.rand(tokens, topk, generator=gen)
    wire = "fp8_e4m3" if fp8 else "bf16"
    config = HostStagedConfig(stage=7 if fp8 else 6, channels=channels, wire_dtype=wire, recv_dtype=wire, output_pool_size=4)
    options = dict(do_expand=expand, expert_alignment=alignment, do_zero_padding=expand)
    with HostStagedEPBuffer(one_rank, capacity, hidden, topk, experts, config) as buffer:
        args = (x.cuda(), idx.cuda(), w.cuda())
        assert buffer.runtime.dispatch_is_local()
        local = buffer.dispatch(*args, **options)
        buffer.runtime.set_test_prefix_delay_ns(1)  # a hook of the protocol: the general kernel takes the call
        assert not buffer.runtime.dispatch_is_local()
        general = buffer.dispatch(*args, **options)
        buffer.runtime.set_test_prefix_delay_ns(0)
        cached = buffer.dispatch(args[0], None, args[2], handle=buffer.cache_layout(general[3]), **options)
        for result in (general, cached, local):
            buffer.check_errors(result[3])
        rows = int(general[3].expert_offsets[-1]) if expand else int(general[3].unique_count[0])
        entries = (idx >= 0).any(1)
        per_channel = max(1, -(-tokens // channels))
        for got in (local, cached):
            for field in FIELDS:
                assert torch.equal(got[3]._result[field], general[3]._result[field]), field
            for mine, theirs in zip(got[:3], general[:3]):
                assert torch.equal(mine[:rows].view(torch.uint8), theirs[:rows].view(torch.uint8))
            assert torch.equal(got[3].source_meta[:rows], general[3].source_meta[:rows])
            if fp8:
                assert torch.equal(got[3]._result["recv_x_scales"][:rows], general[3]._result["recv_x_scales"][:rows])
            assert int(got[3].stats[6]) == int(entries.sum())
            # the combine map: token, rows, then (row, weight) pairs, for the entries that exist
            slots = got[3]._result["comb_map"].shape[0] // channels
            maps = [r[3]._result["comb_map"].cpu() for r in (got, general)]
            for channel in range(channels):
                first = channel * per_channel
                for j in range(int(entries[first:first + per_channel].sum())):
                    a, b = (m[channel * slots + j] for m in maps)
                    assert torch.equal(a[:2 + 2 * int(a[1])], b[:2 + 2 * int(b[1])])
        y = torch.randn(max(1, rows), hidden, generator=gen).to(torch.bfloat16)
        for result, weighted, num_sms in ((local, expand, 0), (cached, False, 3)):
            out = buffer.combine(y.cuda(), result[3], weighted=weighted, num_sms=num_sms)[0].cpu().double()
            meta = result[3].source_meta[:rows].cpu()
            used = meta[:, 1] >= 0
            token, slot = meta[used, 1], meta[used, 2].clamp_min(0)
            factor = w[token, slot].double() if weighted else torch.ones(int(used.sum()), dtype=torch.float64)
            terms = y[:rows][used].double() * factor.unsqueeze(1)
            want = torch.zeros(tokens, hidden, dtype=torch.float64).index_add_(0, token, terms)
            size = torch.zeros(tokens, hidden, dtype=torch.float64).index_add_(0, token, terms.abs())
            # one rounding to BF16 (half a unit in the last of 8 bits), and one FP32 rounding per added row
            assert bool(((out - want).abs() <= want.abs() * 2.0 ** -8 + size * topk * 2.0 ** -23).all())
            assert int(result[3]._result["combine_stats"][0]) == int(entries.sum())
            del out
        buffer.check_errors(local[3])
        del local, general, cached, result, got


@pytest.mark.parametrize("tokens,topk,hidden", [(148 * 4 - 1, 8, 2880), (148 * 5 + 3, 8, 2880), (148 * 12, 8, 2880), (148 * 12 + 1, 8, 2880), (148 * 13, 8, 2880),
                                                (148 * 11 + 5, 4, 3584), (148 * 16, 4, 3584), (148 * 16 + 1, 4, 3584), (148 * 17, 4, 3584)])
def test_combine_at_the_line_between_fixed_order_and_claims(one_rank, tokens, topk, hidden):
    """Units of more and of at most 32 KB, around 4, 12 and 16 of them per CTA, some entries missing: two passes (the counters of the
    first are the second's) against the sum in 64 bits."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    gen = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, hidden, generator=gen).to(torch.bfloat16).cuda()
    idx = torch.rand(tokens, 16, generator=gen).topk(topk, dim=1).indices.to(torch.int64)
    idx[torch.rand(tokens, generator=gen) < 0.1] = -1
    w = torch.rand(tokens, topk, generator=gen).cuda()
    with HostStagedEPBuffer(one_rank, tokens, hidden, topk, 16, HostStagedConfig(channels=16)) as buffer:
        recv_x, _, _, handle, _ = buffer.dispatch(x, idx.cuda(), w, do_expand=True)
        rows = int(handle.num_expanded_tokens)
        y = torch.randn(rows, hidden, generator=gen).to(torch.bfloat16).cuda()
        meta = handle.source_meta[:rows]
        terms = y.double() * w[meta[:, 1], meta[:, 2]].double().unsqueeze(1)
        want = torch.zeros(tokens, hidden, dtype=torch.float64, device="cuda").index_add_(0, meta[:, 1], terms)
        size = torch.zeros(tokens, hidden, dtype=torch.float64, device="cuda").index_add_(0, meta[:, 1], terms.abs())
        for _ in range(2):
            out = buffer.combine(y, handle)[0].double()
            # as above: one rounding to BF16, one FP32 rounding per added row
            assert bool(((out - want).abs() <= want.abs() * 2.0 ** -8 + size * topk * 2.0 ** -23).all())
        buffer.check_errors(handle)
        del recv_x, handle


@pytest.mark.parametrize("tokens,capacity,channels", [(300, 300, 7), (40, 300, 32), (30000, 30000, 1)])
def test_dispatch_beside_the_compute_stream_keeps_to_its_channels(one_rank, tokens, capacity, channels):
    """On the communication stream: as many CTAs as channels (or the general kernel where their tables would not fit)."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    with HostStagedEPBuffer(one_rank, capacity, 64, 4, 16, HostStagedConfig(channels=channels)) as buffer:
        x = torch.randn(tokens, 64).to(torch.bfloat16).cuda()
        idx = torch.rand(tokens, 16).topk(4, dim=1).indices.cuda()
        here = buffer.dispatch(x, idx, do_expand=True)
        there = buffer.dispatch(x, idx, do_expand=True, async_with_compute_stream=True)
        there[4].wait()
        buffer.check_errors(there[3])
        rows = tokens * 4
        assert torch.equal(here[0][:rows], there[0][:rows]) and torch.equal(here[3].source_meta[:rows], there[3].source_meta[:rows])
        assert torch.equal(here[3]._result["comb_map"], there[3]._result["comb_map"])
        assert torch.equal(here[0][:rows], x[here[3].source_meta[:rows, 1]])
        del here, there


@pytest.mark.parametrize("inference", [False, True])
def test_results_are_ordinary_tensors_over_the_pool(one_rank, inference):
    """What a dispatch and a combine hand out shares the pool's memory and version counter, also in inference mode."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    with HostStagedEPBuffer(one_rank, 32, 64, 2, 8, HostStagedConfig(channels=4)) as buffer:
        x = torch.randn(20, 64).to(torch.bfloat16).cuda()
        idx = torch.rand(20, 8).topk(2, dim=1).indices.cuda()
        with torch.inference_mode(inference):
            recv_x, recv_idx, recv_w, handle, _ = buffer.dispatch(x, idx, torch.ones(20, 2, device="cuda"), do_expand=True)
            out = buffer.combine(recv_x, handle)[0]
        buffer.check_errors(handle)
        assert torch.equal(out, 2 * x) and torch.equal(recv_x[:40], x[handle.source_meta[:40, 1]])
        for t in (recv_x, recv_idx, recv_w, out, handle.expert_counts):
            assert t.is_contiguous() and not t.is_inference() and not t.requires_grad
        version = recv_x._version
        recv_x[:1].zero_()
        assert recv_x._version == version + 1
        with pytest.raises(ValueError, match="expected dtype"):
            buffer.dispatch(x.float(), idx)
        with pytest.raises(TypeError, match="expected a torch.Tensor"):
            buffer.dispatch(x, [1])
        with pytest.raises(ValueError, match="contiguous"):
            buffer.combine(recv_x[:, :32], handle)


def test_combine_refuses_outputs_that_its_stores_do_not_fit(one_rank):
    """An output off the 16-byte boundary is an error of the call, and the buffer goes on after it, fused calls included."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    tokens, hidden, inter = 24, 256, 128
    with HostStagedEPBuffer(one_rank, tokens, hidden, 2, 4, HostStagedConfig(channels=4, fused_expert_combine=True)) as buffer:
        x = torch.randn(tokens, hidden).to(torch.bfloat16).cuda()
        idx = torch.rand(tokens, 4).topk(2, dim=1).indices.cuda()
        w = torch.rand(tokens, 2).cuda()
        recv_x, _, _, handle, _ = buffer.dispatch(x, idx, w, do_expand=True)
        hidden_rows = torch.randn(recv_x.shape[0], inter).to(torch.bfloat16).cuda()
        w_down = torch.randn(4, hidden, inter).to(torch.bfloat16).cuda()
        room = torch.empty(tokens * hidden + 8, dtype=torch.bfloat16, device="cuda")
        calls = [lambda out: buffer.combine(recv_x, handle, out=out), lambda out: buffer.fused_expert_combine(hidden_rows, w_down, handle, out=out)]
        for call in calls:
            for offset in (1, 4, 7):
                with pytest.raises(ValueError, match="16-byte boundary"):
                    call(room[offset:offset + tokens * hidden].view(tokens, hidden))
            with pytest.raises(ValueError, match=r"\[T, hidden\]"):
                call(room[:hidden].view(1, hidden))
            want = call(None)[0].clone()
            assert torch.equal(call(room[8:].view(tokens, hidden))[0], want) and float(want.float().abs().max()) > 0
        buffer.check_errors(handle)
        del recv_x, handle


def median_us(call, repeats=7, calls=5):
    times = []
    for _ in range(repeats):
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(2_000_000)  # the launches are queued behind it
        begin.record()
        for _ in range(calls):
            call()
        end.record()
        torch.cuda.synchronize()
        times.append(begin.elapsed_time(end) * 1000 / calls)
    return sorted(times)[repeats // 2]


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("tokens,alignment,fp8", [(3, 256, False), (64, 256, False), (1000, 128, True)])
def test_zeroing_padding_rows_is_spread_over_the_sms(one_rank, tokens, alignment, fp8, cached):
    """The rows between the experts' segments are zero, and zeroing them takes no longer than in the general kernel (a third
    on top for the spread between measurements; a few SMs doing it take three to six times as long)."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    wire = "fp8_e4m3" if fp8 else "bf16"
    config = HostStagedConfig(stage=7 if fp8 else 6, channels=32, wire_dtype=wire, recv_dtype=wire)
    with HostStagedEPBuffer(one_rank, tokens, 7168, 8, 32, config) as buffer:
        x = torch.randn(tokens, 7168).to(torch.bfloat16).cuda()
        idx = torch.rand(tokens, 32).topk(8, dim=1).indices.cuda()
        routes = dict(handle=buffer.cache_layout(buffer.dispatch(x, idx, do_expand=True, expert_alignment=alignment)[3])) if cached else dict(topk_idx=idx)

        def dispatch():
            return buffer.dispatch(x, do_expand=True, expert_alignment=alignment, do_zero_padding=True, **routes)

        for _ in range(config.output_pool_size):  # whatever set of results comes next holds no zeros
            dispatch()[0].view(torch.uint8).fill_(7)
        got = dispatch()
        buffer.check_errors(got[3])
        rows = int(got[3].expert_offsets[-1])
        padding = got[3].source_meta[:rows, 1] < 0
        assert int(padding.sum()) == rows - tokens * 8 and int(got[0][:rows][padding].view(torch.uint8).max()) == 0
        assert bool((got[1][:rows][padding] == -1).all()) and float(got[3]._result["recv_topk_weights"][:rows][padding].abs().max()) == 0.0
        del got
        local = median_us(dispatch)
        buffer.runtime.set_test_prefix_delay_ns(1)  # the general kernel takes the call
        general = median_us(dispatch)
        assert local <= general * 4 / 3, (local, general)


def assert_same_result(got, want, rows, channels, fp8):
    """Every field, the rows in use and the combine map's entries of two dispatch results."""
    for field in FIELDS:
        assert torch.equal(got[3]._result[field], want[3]._result[field]), field
    for mine, theirs in zip(got[:3], want[:3]):
        assert torch.equal(mine[:rows].view(torch.uint8), theirs[:rows].view(torch.uint8))
    assert torch.equal(got[3].source_meta[:rows], want[3].source_meta[:rows])
    if fp8:
        assert torch.equal(got[3]._result["recv_x_scales"][:rows], want[3]._result["recv_x_scales"][:rows])
    mine, theirs = (r[3]._result["comb_map"].view(channels, -1, r[3]._result["comb_map"].shape[1]) for r in (got, want))
    exists = torch.arange(theirs.shape[1], device="cuda") < want[3]._result["recv_chan_counts"].view(-1, 1)
    words = torch.arange(theirs.shape[2], device="cuda") < 2 + 2 * theirs[:, :, 1:2]
    assert torch.equal(mine[exists.unsqueeze(2) & words], theirs[exists.unsqueeze(2) & words])


@pytest.mark.parametrize("tokens,capacity,experts,topk,hidden,channels,fp8,expand,alignment", CASES)
def test_plans_of_both_kernels_are_the_same(one_rank, tokens, capacity, experts, topk, hidden, channels, fp8, expand, alignment):
    """A plan that either kernel has written gives the same results in either kernel when it is used again."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    gen = torch.Generator(device="cuda").manual_seed(tokens + topk)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    idx = torch.rand(tokens, experts, device="cuda", generator=gen).topk(topk, dim=1).indices
    idx[torch.rand(tokens, topk, device="cuda", generator=gen) < 0.2] = -1
    w = torch.rand(tokens, topk, device="cuda", generator=gen)
    wire = "fp8_e4m3" if fp8 else "bf16"
    config = HostStagedConfig(stage=7 if fp8 else 6, channels=channels, wire_dtype=wire, recv_dtype=wire, output_pool_size=5)
    options = dict(do_expand=expand, expert_alignment=alignment, do_zero_padding=expand)
    with HostStagedEPBuffer(one_rank, capacity, hidden, topk, experts, config) as buffer:
        def dispatch(general, *args, **more):
            buffer.runtime.set_test_prefix_delay_ns(1 if general else 0)  # a hook of the protocol: the general kernel takes the call
            assert buffer.runtime.dispatch_is_local() != general
            return buffer.dispatch(x, *args, topk_weights=w, **options, **more)

        want = dispatch(True, idx)
        buffer.check_errors(want[3])
        rows = int(want[3].expert_offsets[-1]) if expand else int(want[3].unique_count[0])
        for written_by_general in (False, True):
            fresh = dispatch(written_by_general, idx)
            plan = buffer.cache_layout(fresh[3])
            for used_by_general in (False, True):
                got = dispatch(used_by_general, handle=plan)
                buffer.check_errors(got[3])
                assert_same_result(got, want, rows, channels, fp8)
                del got
            del fresh, plan
        del want


# at the most pairs that every CTA counts by itself and one token beyond, pairs across words, the widest and the narrowest top-k,
# experts up to and beyond those that are counted with ballots
@pytest.mark.parametrize("tokens,topk,experts,channels", [(1, 1, 1, 1), (33, 3, 7, 4), (1003, 3, 9, 32), (2048, 8, 64, 128), (2049, 8, 64, 128), (700, 4, 65, 16),
                                                          (512, 32, 600, 20), (513, 32, 600, 20), (16384, 1, 5, 64), (16385, 1, 5, 64), (149, 32, 33, 3)])
@pytest.mark.parametrize("routes", ["some", "one expert", "none"])
def test_small_and_large_batches_lay_out_alike(one_rank, tokens, topk, experts, channels, routes):
    """Every CTA counts a small batch by itself, a large one is counted together behind a barrier: both as the general kernel,
    on the caller's stream and with fewer CTAs beside it, several times in a row."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    gen = torch.Generator(device="cuda").manual_seed(tokens + topk)
    x = torch.randn(tokens, 64, device="cuda", generator=gen).to(torch.bfloat16)
    idx = torch.rand(tokens, experts, device="cuda", generator=gen).topk(topk, dim=1).indices
    if routes == "some":
        idx[torch.rand(tokens, topk, device="cuda", generator=gen) < 0.3] = -1
    else:
        idx[:, 1:] = -1
        idx[:, 0] = experts - 1 if routes == "one expert" else -1
    w = torch.rand(tokens, topk, device="cuda", generator=gen)
    with HostStagedEPBuffer(one_rank, tokens, 64, topk, experts, HostStagedConfig(channels=channels, output_pool_size=4)) as buffer:
        def dispatch(general, **how):
            buffer.runtime.set_test_prefix_delay_ns(1 if general else 0)  # a hook of the protocol: the general kernel takes the call
            return buffer.dispatch(x, idx, w, do_expand=True, expert_alignment=4, do_zero_padding=True, **how)

        want = dispatch(True)
        buffer.check_errors(want[3])
        rows, epoch = int(want[3].expert_offsets[-1]), int(buffer.runtime.epochs()[0])
        for number, how in enumerate([{}, dict(async_with_compute_stream=True), {}]):
            got = dispatch(False, **how)
            got[4].wait()
            buffer.check_errors(got[3])
            assert_same_result(got, want, rows, channels, False)
            assert int(got[3].stats[6]) == int((idx >= 0).any(1).sum()) and int(buffer.runtime.epochs()[0]) == epoch + number + 1
            begin, end = got[3].transport_timestamps_ns.tolist()
            assert 0 < begin < end
            del got
        again = dispatch(True)  # the general kernel finds the epoch that the others left
        buffer.check_errors(again[3])
        assert_same_result(again, want, rows, channels, False)
        del again, want


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("tokens,hidden,experts", [(1, 7168, 32), (555, 7168, 32), (1184, 7168, 32), (2048, 7168, 32), (2000, 8192, 32), (700, 14336, 8)])
def test_batches_whose_tables_take_a_row_buffer_lay_out_alike(one_rank, tokens, hidden, experts, fp8):
    """Rows so long that the row buffers leave less than the counting tables need: with one of them given up as the general kernel,
    and beside the compute stream, where CTAs have more tokens than row buffers."""
    lay_out_alike(one_rank, tokens, 8, hidden, experts, fp8)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("tokens,topk,hidden,experts", [(1024, 8, 3584, 16), (4096, 2, 3584, 16), (148 * 30, 2, 3584, 16), (148 * 30 + 1, 2, 3584, 16),
                                                        (148 * 13, 8, 8192, 16), (148 * 13 + 1, 8, 8192, 16)])
def test_batches_that_just_fit_or_miss_the_rest_of_the_row_buffers_lay_out_alike(one_rank, tokens, topk, hidden, experts, fp8):
    """Two row buffers per warp, of which one warp's make room for the tables, and as many tokens as the other buffers hold or one more."""
    lay_out_alike(one_rank, tokens, topk, hidden, experts, fp8)


def lay_out_alike(one_rank, tokens, topk, hidden, experts, fp8):
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    idx = torch.rand(tokens, experts, device="cuda", generator=gen).topk(topk, dim=1).indices
    idx[torch.rand(tokens, topk, device="cuda", generator=gen) < 0.2] = -1
    w = torch.rand(tokens, topk, device="cuda", generator=gen)
    wire = "fp8_e4m3" if fp8 else "bf16"
    config = HostStagedConfig(stage=7 if fp8 else 6, channels=128, wire_dtype=wire, recv_dtype=wire, output_pool_size=3)
    with HostStagedEPBuffer(one_rank, tokens, hidden, topk, experts, config) as buffer:
        buffer.runtime.set_test_prefix_delay_ns(1)  # a hook of the protocol: the general kernel takes the call
        want = buffer.dispatch(x, idx, w, do_expand=True)
        buffer.runtime.set_test_prefix_delay_ns(0)
        rows = int((idx >= 0).sum())
        for how in ({}, dict(async_with_compute_stream=True), {}):
            got = buffer.dispatch(x, idx, w, do_expand=True, **how)
            got[4].wait()
            buffer.check_errors(got[3])
            assert_same_result(got, want, rows, 128, fp8)
            del got
        del want


@pytest.mark.parametrize("tokens,bad", [(40, 99), (40, -2), (5000, 99)])
def test_invalid_routes_are_an_error_whoever_counts_them(one_rank, tokens, bad):
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    with HostStagedEPBuffer(one_rank, tokens, 64, 8, 16, HostStagedConfig(channels=8)) as buffer:
        x = torch.randn(tokens, 64).to(torch.bfloat16).cuda()
        idx = torch.rand(tokens, 16).topk(8, dim=1).indices
        idx[tokens - 3, 5] = bad
        handle = buffer.dispatch(x, idx.cuda(), do_expand=True)[3]
        with pytest.raises(RuntimeError, match="EP dispatch GPU error"):
            buffer.check_errors(handle)
        assert handle.error.tolist()[1:3] == [tokens - 3, 5]
        del handle


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("fused", [False, True])
def test_linked_layers_are_the_unlinked_ones_and_keep_their_counters(one_rank, fused, fp8, monkeypatch):
    """Layers of which some passes link their GEMMs (the down projection scattered by its epilogue among them) and some do not, in turn:
    the bits of unlinked passes, with stale activations gone between them, on one set of counters that ends at zero."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer
    from pcie_ep_b200.models import moe_layer

    experts, topk, hidden, inter, capacity = 16, 4, 2048, 384, 1024  # more tiles than pairs of CTAs in the second launch, three channel tiles in the first
    line = moe_layer._LINKED_ROWS
    gen = torch.Generator(device="cuda").manual_seed(3)
    weights = ((torch.randn(experts, 2 * inter, hidden, device="cuda", generator=gen) * 0.05).to(torch.bfloat16),
               (torch.randn(experts, hidden, inter, device="cuda", generator=gen) * 0.05).to(torch.bfloat16))
    wire = "fp8_e4m3" if fp8 else "bf16"
    config = HostStagedConfig(stage=7 if fp8 else 6, channels=16, wire_dtype=wire, recv_dtype=wire, fused_expert_combine=fused)
    with HostStagedEPBuffer(one_rank, capacity, hidden, topk, experts, config) as buffer:
        layer = moe_layer.MoELayer(buffer, inter, with_router=False, weights=weights)
        counters = layer._progress.data_ptr()
        popularity = 1.0 / torch.arange(1, experts + 1, device="cuda") ** 2  # the last ones are often empty
        for tokens in (300, capacity, 300, 1, 17, line * experts // topk, line * experts // topk + 1, 40):
            x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
            scores = popularity.log() - (-torch.rand(tokens, experts, device="cuda", generator=gen).clamp(1e-6, 1 - 1e-6).log()).log()
            idx, w = scores.topk(topk, dim=1).indices.contiguous(), torch.rand(tokens, topk, device="cuda", generator=gen)
            outs = []
            for linked_rows in (-1, line, line):
                monkeypatch.setattr(moe_layer, "_LINKED_ROWS", linked_rows)
                if layer._hidden_rows is not None:
                    layer._hidden_rows.fill_(float("nan"))
                outs.append(layer(x, idx, w).clone())
                assert layer._progress is not None and layer._progress.data_ptr() == counters and int(layer._progress.abs().max()) == 0
            assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]) and float(outs[0].float().abs().max()) > 0
        layer.check_errors()


def test_a_layer_made_on_another_stream_waits_for_its_counters(one_rank):
    """The counters are zeroed on the stream that built the layer; a first pass elsewhere waits for that."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer
    from pcie_ep_b200.models.moe_layer import MoELayer

    with HostStagedEPBuffer(one_rank, 32, 256, 2, 4, HostStagedConfig(channels=4)) as buffer:
        x, idx, w = torch.randn(32, 256, device="cuda").to(torch.bfloat16), torch.rand(32, 4, device="cuda").topk(2, dim=1).indices, torch.rand(32, 2, device="cuda")
        weights = tuple((torch.randn(4, *shape, device="cuda") * 0.05).to(torch.bfloat16) for shape in ((256, 256), (256, 128)))
        want = MoELayer(buffer, 128, with_router=False, weights=weights)(x, idx, w).clone()
        torch.cuda.synchronize()
        junk = torch.full((4096,), 7, dtype=torch.int32, device="cuda")  # what the counters' memory may have held
        del junk
        torch.cuda._sleep(20_000_000)  # ten milliseconds, in front of the zeroing
        layer = MoELayer(buffer, 128, with_router=False, weights=weights)
        with torch.cuda.stream(torch.cuda.Stream()):
            got = layer(x, idx, w).clone()
        torch.cuda.synchronize()
        layer.check_errors()
        assert torch.equal(got, want) and int(layer._progress.abs().max()) == 0
