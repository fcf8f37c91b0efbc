"""What a group of one rank launches, from profiler traces: which kernel takes a call, with how many CTAs, and whether it fits
on an SM that an expert GEMM holds.  Sorted behind the other profiler test, whose trace lost launches in a process that had
already profiled some dozens of times."""

import json
import os
import tempfile
import time

import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def one_rank(ext):
    if not dist.is_initialized():
        store = dist.FileStore(os.path.join(tempfile.mkdtemp(prefix="launches-store-"), "store"), 1)
        dist.init_process_group("gloo", store=store, rank=0, world_size=1)
    if dist.get_world_size() != 1:
        pytest.skip("needs a process group of one")
    return dist.group.WORLD


def launches(call, count):
    """What ``call`` returns and the kernels that it launches, as a profiler saw them: name, CTAs, threads, shared memory and
    registers.  A trace that misses one of the ``count`` kernels is taken again."""
    for _ in range(3):
        result = None  # (the results of a call keep their pool busy)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            # well inside the profiler's window: launches close to its ends may be missing from the trace
            torch.cuda.synchronize()
            time.sleep(0.02)
            result = call()
            torch.cuda.synchronize()
            time.sleep(0.02)
        with tempfile.NamedTemporaryFile(suffix=".json") as file:
            prof.export_chrome_trace(file.name)
            events = json.load(open(file.name))["traceEvents"]
        kernels = sorted((e for e in events if e.get("cat") == "kernel" and "bep::" in e["name"]), key=lambda e: e["ts"])
        if len(kernels) >= count:
            break
    return result, [dict(name=e["name"], ctas=e["args"]["grid"][0], threads=e["args"]["block"][0], shared=e["args"]["shared memory"],
                         registers=e["args"]["registers per thread"]) for e in kernels]


def weighted_sum(y, idx, w, topk):
    """Expanded rows back to their tokens in 64 bits, and a bound on what 32-bit sums rounded to BF16 may differ by."""
    order = torch.argsort(idx.reshape(-1), stable=True)
    row_of = torch.empty_like(order)
    row_of[order] = torch.arange(order.numel(), device=order.device)
    terms = y[row_of].double().view(*idx.shape, -1) * w.double().unsqueeze(2)
    want = terms.sum(1)
    return want, want.abs() * 2.0 ** -8 + terms.abs().sum(1) * topk * 2.0 ** -23


# tokens per SM, tokens on top, hidden, top-k, whether whole rows are copied in bulk (at the lines of combine_local_pays)
KERNELS = [(8, 0, 512, 2, True), (8, 1, 512, 2, False), (14, 0, 1536, 2, True), (14, 0, 1528, 2, False), (14, 1, 1536, 2, False),
           (14, 1, 3584, 4, True), (14, 1, 3576, 4, False), (14, 1, 3584, 3, False), (14, 1, 5120, 1, True), (14, 1, 5112, 1, False)]


@pytest.mark.parametrize("per_sm,more,hidden,topk,bulk", KERNELS)
def test_combine_takes_the_faster_kernel_for_its_rows(one_rank, per_sm, more, hidden, topk, bulk):
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    tokens = torch.cuda.get_device_properties(0).multi_processor_count * per_sm + more
    with HostStagedEPBuffer(one_rank, tokens, hidden, topk, 16, HostStagedConfig(channels=64)) as buffer:
        gen = torch.Generator(device="cuda").manual_seed(hidden)
        x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
        idx = torch.rand(tokens, 16, device="cuda", generator=gen).topk(topk, dim=1).indices
        w = torch.rand(tokens, topk, device="cuda", generator=gen)
        y = torch.randn(tokens * topk, hidden, device="cuda", generator=gen).to(torch.bfloat16)
        handle = buffer.dispatch(x, idx, w, do_expand=True)[3]
        got, seen = launches(lambda: buffer.combine(y, handle)[0], 1)
        buffer.check_errors(handle)
        assert [("local_combine" in k["name"]) for k in seen if "combine" in k["name"]] == [bulk]
        want, bound = weighted_sum(y, idx, w, topk)
        assert bool(((got.double() - want).abs() <= bound).all())
        assert int(handle._result["combine_stats"][0]) == tokens
        del got, handle


def room_beside(*kernels):
    """Whether one CTA of each of these launches fits on one SM (a CTA's warps go round the four quarters of the SM, each with
    a quarter of the registers; 1 KB of shared memory per CTA is the system's)."""
    device = torch.cuda.get_device_properties(0)
    shared = sum(k["shared"] + 1024 for k in kernels)
    registers = sum(-(-k["threads"] // 128) * 32 * (-(-k["registers"] // 8) * 8) for k in kernels)
    return shared <= device.shared_memory_per_multiprocessor and registers <= device.regs_per_multiprocessor // 4


@pytest.mark.parametrize("swiglu,fp8", [(False, False), (True, False), (True, True)])
def test_expert_gemm_leaves_room_for_a_combine_reducer(one_rank, swiglu, fp8):
    """The reducers of the combine use no shared memory so that they can run on SMs which a persistent expert GEMM holds."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer
    from pcie_ep_b200.ops.grouped_ffn import grouped_gemm

    tokens = torch.cuda.get_device_properties(0).multi_processor_count * 8 + 1  # of short rows: the reducers take the call
    with HostStagedEPBuffer(one_rank, tokens, 512, 2, 16, HostStagedConfig(channels=64)) as buffer:
        x = torch.randn(tokens, 512).to(torch.bfloat16).cuda()
        idx = torch.rand(tokens, 16).topk(2, dim=1).indices.cuda()
        recv_x, _, _, handle, _ = buffer.dispatch(x, idx, do_expand=True)
        dtype = torch.float8_e4m3fn if fp8 else torch.bfloat16
        weights = torch.randn(16, 512 if swiglu else 256, 512).to(torch.bfloat16).cuda().to(dtype)
        scales = dict(a_scales=torch.ones(recv_x.shape[0], device="cuda"), w_scales=torch.ones(16, 512, device="cuda")) if fp8 else {}
        out = torch.empty(recv_x.shape[0], 256, dtype=torch.bfloat16, device="cuda")
        rows = recv_x.to(dtype)

        def call():
            grouped_gemm(rows, weights, handle.expert_offsets, handle.expert_counts, swiglu=swiglu, out=out, **scales)
            return buffer.combine(recv_x, handle)[0]

        got, seen = launches(call, 2)
        buffer.check_errors(handle)
        gemm, = (k for k in seen if "gemm" in k["name"])
        combine, = (k for k in seen if "combine" in k["name"])
        assert "local_combine" not in combine["name"] and room_beside(gemm, combine)
        assert torch.equal(got, 2 * x)
        del recv_x, handle, got


@pytest.mark.parametrize("how", ["async", "event", "side stream", "num_sms", "default"])
@pytest.mark.parametrize("tokens", [40, 600])
def test_combine_beside_other_work_fits_next_to_the_expert_gemm(one_rank, how, tokens):
    """On the communication stream, on a stream of the caller's own or limited to some SMs, a CTA of the combine finds room on
    an SM that a CTA of the persistent expert GEMM holds."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer
    from pcie_ep_b200.ops.grouped_ffn import grouped_gemm

    with HostStagedEPBuffer(one_rank, tokens, 1024, 2, 16, HostStagedConfig(channels=8)) as buffer:
        x = torch.randn(tokens, 1024).to(torch.bfloat16).cuda()
        idx = torch.rand(tokens, 16).topk(2, dim=1).indices.cuda()
        w = torch.rand(tokens, 2).cuda()
        y = torch.randn(2 * tokens, 1024).to(torch.bfloat16).cuda()
        handle = buffer.dispatch(x, idx, w, do_expand=True)[3]
        weights = torch.randn(16, 512, 1024).to(torch.bfloat16).cuda()
        gemm_out = torch.empty(2 * tokens, 256, dtype=torch.bfloat16, device="cuda")

        def call():
            grouped_gemm(y, weights, handle.expert_offsets, handle.expert_counts, swiglu=True, out=gemm_out)
            if how == "side stream":
                side = torch.cuda.Stream()
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    return buffer.combine(y, handle)[0]
            if how == "event":
                return buffer.combine(y, handle, previous_event=buffer.capture(), allocate_on_comm_stream=True)[0]
            return buffer.combine(y, handle, async_with_compute_stream=how == "async", num_sms=5 if how == "num_sms" else 0)[0]

        got, seen = launches(call, 2)
        buffer.check_errors(handle)
        gemm, = (k for k in seen if "gemm" in k["name"])
        combine, = (k for k in seen if "combine" in k["name"])
        assert ("local_combine" in combine["name"]) == (how == "default")
        assert how == "default" or room_beside(gemm, combine)
        assert how != "num_sms" or combine["ctas"] <= 2 * 5
        want, bound = weighted_sum(y, idx, w, 2)
        assert bool(((got.double() - want).abs() <= bound).all())
        del got, handle


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("tokens,channels", [(300, 7), (40, 300 // 4), (5, 32), (30000, 1)])
def test_dispatch_and_replay_launch_what_their_stream_allows(one_rank, tokens, channels, cached):
    """On the caller's stream every SM, on the communication stream as many CTAs as channels (the general kernel where the
    tables of so few CTAs would not fit); a captured dispatch follows the stream of the replay, not that of the capture."""
    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    with HostStagedEPBuffer(one_rank, tokens, 64, 4, 16, HostStagedConfig(channels=channels, enable_graph=True)) as buffer:
        x = torch.randn(tokens, 64).to(torch.bfloat16).cuda()
        idx = torch.rand(tokens, 16).topk(4, dim=1).indices.cuda()
        plan = buffer.cache_layout(buffer.dispatch(x, idx, do_expand=True)[3])
        routes = dict(handle=plan) if cached else dict(topk_idx=idx)
        graph = buffer.capture_dispatch(x, do_expand=True, **routes)
        beside = dict(async_with_compute_stream=True)

        def on_comm_stream(call):
            buffer.get_comm_stream().wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(buffer.get_comm_stream()):
                return call()

        def eager(**how):
            return buffer.dispatch(x, do_expand=True, **routes, **how)

        calls = [(eager, False), (lambda: eager(**beside), True), (lambda: on_comm_stream(eager), True), (graph.replay, False),
                 (lambda: graph.replay(**beside), True), (lambda: graph.replay(previous_event=buffer.capture()), True),
                 (lambda: on_comm_stream(graph.replay), True), (graph.replay, False)]
        for number, (call, few) in enumerate(calls):
            got, (seen,) = launches(call, 1)
            buffer.check_errors(got[3])
            fits = not (few and tokens == 30000)
            assert ("local_dispatch" in seen["name"]) == fits, number
            assert seen["ctas"] == (min(channels if few else sms, sms, tokens) if fits else channels), number
            rows = tokens * 4
            meta = got[3].source_meta[:rows]
            assert torch.equal(got[0][:rows], x[meta[:, 1]]) and torch.equal(got[3].expert_counts.long(), torch.bincount(idx.reshape(-1), minlength=16))
            del got, meta
        graph.close()
