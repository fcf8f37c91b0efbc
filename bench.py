"""Headline benchmark: dispatch + combine latency of one MoE exchange, device-timed, max over ranks.

Config: hidden 7168, 256 experts, top-8 distinct uniform expert ids, softmax weights,
BF16 tokens ~ N(0,1), T tokens per rank (default 4096; ``--tokens`` or ``--sweep`` for 128..8192),
``do_expand=True``, BF16 wire.  One "step" is one dispatch followed by one combine of the received
rows (identity experts), i.e. the full exchange a MoE layer performs around its expert FFN.

    python bench.py --gpus 1 --steps 20 --warmup 5
    python -m torch.distributed.run --nnodes=1 --nproc-per-node 8 --master-addr 127.0.0.1 \
        --master-port 29500 bench.py --gpus 8 --steps 20 --warmup 5
    python bench.py --impl reference ...     # the unmodified reference from baseline/_ref (dispatch only)

Rank 0 prints one JSON line.  ``value`` is microseconds per step (lower is better), the maximum over
ranks of a CUDA-event interval around exactly ``steps`` steps.  ``e2e`` is the same metric through the
public API including, every step, the host->device copy of that step's inputs from pinned memory and
a device->host read of a checksum of the combined output.
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

HIDDEN, EXPERTS, TOPK = 7168, 256, 8
VERIFY_ROUNDS = 3  # verified exchanges before (and after) the timed loops of every configuration

# both arms name the same model and shape in their result line
MODEL_NAME = "DeepSeek-V3-shaped MoE exchange (hidden 7168, 256 experts, top-%d)"


def source_fingerprint() -> str:
    """Hash of the native sources and flags the loaded library was built from (see benchmarks/source_manifest.py)."""
    from pcie_ep_b200 import _C

    return _C.source_fingerprint()[:16]


# reference dispatch-only latency on 8x H20D, ms (RESULTS_CONTROL_PROGRESS.md:31-40)
PUBLISHED_MS = {16: 0.260, 32: 0.282, 64: 0.405, 128: 0.647, 256: 1.033, 512: 1.950, 1024: 3.681, 2048: 7.079,
                4096: 13.558, 8192: 26.546}
METRIC = "dispatch+combine us (device, max over ranks), H=7168, E=256, top-%d"  # both arms print this string
INPUT_SETS = 4  # rotated every step: 4 x T x 14 KiB of tokens (> L2 at T >= 2304); see "l2" in config


def parse_args():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=20)
    p.add_argument("--warmup", type=int, default=5)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--tokens", type=int, default=4096)
    p.add_argument("--topk", type=int, default=TOPK)
    p.add_argument("--sweep", action="store_true", help="also time T in {128,256,1024,4096,8192} (device-timed only)")
    p.add_argument("--wire", default="bf16", choices=["bf16", "fp8_e4m3"])
    p.add_argument("--channels", type=int, default=0)
    p.add_argument("--engine", default="tma", choices=["tma", "vector"])
    p.add_argument("--transport", default="peer", choices=["peer", "host_staged"])
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--tx-warps", type=int, default=0, help="send warps per channel CTA (0: by rank count)")
    p.add_argument("--rx-warps", type=int, default=0, help="receive/expand warps per channel CTA (0: by rank count)")
    p.add_argument("--combine-reduce", default="auto", choices=["auto", "separate", "inline"])
    p.add_argument("--send-ctas", type=int, default=-1, help="dedicated sender CTAs (-1: by rank count)")
    p.add_argument("--stages", type=int, default=0, help="row buffers per send warp (0: tuned)")
    p.add_argument("--no-numa-bind", action="store_true", help="leave the process on whatever CPUs it was started on")
    return p.parse_args()


def init_distributed(args):
    import torch
    import torch.distributed as dist

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if world != args.gpus:
        raise SystemExit(f"--gpus {args.gpus} but WORLD_SIZE={world}: launch with torch.distributed.run --nproc-per-node {args.gpus}")
    torch.cuda.set_device(local_rank)
    if world == 1 and "MASTER_ADDR" not in os.environ:
        store = dist.FileStore(tempfile.mktemp(prefix="bench-store-"), 1)
        dist.init_process_group("gloo", store=store, rank=0, world_size=1)
    else:
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group("gloo", rank=rank, world_size=world)
    return rank, world, local_rank


def make_routes(tokens, experts, topk, rank, seed=20261024):
    """Distinct uniform expert ids, softmax weights (same generator recipe as the reference benchmark,
    benchmarks/benchmark.py:35-41)."""
    import torch

    g = torch.Generator().manual_seed(seed + rank * 104729 + tokens)
    idx = torch.rand(tokens, experts, generator=g).topk(topk, dim=1).indices.to(torch.int64)
    weights = torch.softmax(torch.randn(tokens, topk, generator=g), dim=1).to(torch.float32)
    return idx.contiguous(), weights.contiguous()


def roofline(idx, world, rank, tokens, topk, experts):
    """Lower bounds for one rank's dispatch and combine: the slower of its HBM traffic at the measured copy rate and
    its NVLink egress at the measured peer-copy rate (770 GB/s per direction).  Rows on the wire are the staged row
    (payload + metadata, 128-byte aligned) for dispatch and one BF16 row for combine."""
    local = experts // world
    ranks_hit = (idx // local)
    sent = 0
    for d in range(world):
        if d != rank:
            sent += int((ranks_hit == d).any(dim=1).sum())
    received = sent  # uniform routing: ingress equals egress on average
    expanded = tokens * topk  # rows this rank's experts receive, on average
    row_wire = ((HIDDEN * 2 + 16 + 12 * topk + 127) // 128) * 128
    row = HIDDEN * 2
    hbm = 6548.0e9
    try:
        hbm = float(json.loads((ROOT / "MEASURED_PEAKS.json").read_text())["hbm_gbs"]) * 1e9
    except Exception:  # noqa: BLE001
        pass
    nvlink = 770.0e9
    dispatch_hbm = tokens * row + 2 * received * row_wire + expanded * row
    combine_hbm = expanded * row + 2 * received * row + tokens * row
    out = {}
    for name, hbm_bytes, wire_bytes in (("dispatch", dispatch_hbm, sent * row_wire), ("combine", combine_hbm, sent * row)):
        t_hbm, t_link = hbm_bytes / hbm * 1e6, wire_bytes / nvlink * 1e6
        out[name + "_us"] = round(max(t_hbm, t_link), 1)
        out[name + "_bound"] = "nvlink" if t_link > t_hbm else "hbm"
    out["model"] = ("per rank: max(HBM bytes / measured copy rate, NVLink egress bytes / 770 GB/s); dispatch HBM = x read + staged "
                    "rows written and read + expanded rows written, combine HBM = expert rows read + partial rows written and "
                    "read + output written")
    return out


class ClockSampler:
    """SM clock and throttle reasons sampled every few milliseconds by a thread while the GPU works.

    Read-only NVML queries (no setting is changed).  Falls back to one nvidia-smi query per sample when
    the NVML binding is missing."""

    REASONS = {
        "hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40, "sw_power_cap": 0x4,
        "hw_power_brake_slowdown": 0x80,
    }

    def __init__(self, device_index):
        import threading

        self.device_index = device_index
        self.samples, self.max_clock, self.reasons = [], None, set()
        self.direct = 0  # samples taken by sample_now()
        self._stop = threading.Event()
        self._thread = None
        self._nvml = None
        self._handle = None
        try:
            import pynvml

            pynvml.nvmlInit()
            visible = os.environ.get("CUDA_VISIBLE_DEVICES")
            physical = device_index
            if visible:
                entries = [v.strip() for v in visible.split(",") if v.strip()]
                if device_index < len(entries) and entries[device_index].isdigit():
                    physical = int(entries[device_index])
            self._handle = pynvml.nvmlDeviceGetHandleByIndex(physical)
            self.max_clock = float(pynvml.nvmlDeviceGetMaxClockInfo(self._handle, pynvml.NVML_CLOCK_SM))
            self._nvml = pynvml
        except Exception:  # noqa: BLE001 - NVML binding unavailable: nvidia-smi fallback
            self._nvml = None

    def _sample_nvml(self):
        nv = self._nvml
        self.samples.append(float(nv.nvmlDeviceGetClockInfo(self._handle, nv.NVML_CLOCK_SM)))
        try:
            mask = int(nv.nvmlDeviceGetCurrentClocksEventReasons(self._handle))
        except Exception:  # noqa: BLE001 - older binding name
            mask = int(nv.nvmlDeviceGetCurrentClocksThrottleReasons(self._handle))
        for name, bit in self.REASONS.items():
            if mask & bit:
                self.reasons.add(name)

    def _sample_smi(self):
        query = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                 "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        out = subprocess.run(["nvidia-smi", f"--query-gpu={query}", "--format=csv,noheader,nounits", "-i",
                              str(self.device_index)], capture_output=True, text=True, timeout=10).stdout
        f = [v.strip() for v in out.strip().split(",")]
        if len(f) >= 6:
            self.samples.append(float(f[0]))
            self.max_clock = float(f[1])
            for name, value in zip(["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"], f[2:6]):
                if value.lower().startswith("active"):
                    self.reasons.add(name)

    def sample_now(self):
        """One sample on the calling thread.  The timed loops call it right after their last launch, while the GPU
        still works through the queue: the sampling thread has to win the interpreter lock from a main thread that is
        busy launching, and with several ranks querying NVML at once a query can take tens of milliseconds, so on its
        own it may see a short region only once.  Never inside an event pair."""
        try:
            if self._nvml is not None:
                self._sample_nvml()
            else:
                self._sample_smi()
            self.direct += 1
        except Exception:  # noqa: BLE001 - a failed sample is skipped
            pass

    def _run(self):
        while not self._stop.is_set():
            try:
                if self._nvml is not None:
                    self._sample_nvml()
                else:
                    self._sample_smi()
            except Exception:  # noqa: BLE001 - a failed sample is skipped
                pass
            self._stop.wait(0.001 if self._nvml is not None else 0.05)

    def start(self):
        import threading

        self._thread = threading.Thread(target=self._run, daemon=True)
        self._thread.start()

    def stop(self):
        self._stop.set()
        if self._thread is not None:
            self._thread.join(timeout=15)
        return {"sm_mhz": statistics.median(self.samples) if self.samples else None, "sm_max_mhz": self.max_clock,
                "samples": len(self.samples), "samples_after_last_launch": self.direct, "reasons": sorted(self.reasons),
                "how": ("NVML, a thread with about 1 ms period during the timed loop plus one query after the last launch of every "
                        "timed region, while the GPU works through the queue") if self._nvml is not None else "nvidia-smi per sample"}


def max_over_ranks(value):
    import torch
    import torch.distributed as dist

    t = torch.tensor([float(value)], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t[0])


REPEATS = 5  # the timed region (exactly --steps steps) is measured this many times; the median is reported


def timed_repeats(step, steps, repeats=REPEATS, sampler=None):
    """Time `steps` calls of step(i) `repeats` times, each bracketed by barrier + synchronize on both sides and a
    CUDA-event pair on the launching stream.  Returns the per-repeat microseconds per step, max over ranks.  A clock
    sampler, if given, is asked for one sample after the closing event has been recorded and before the host waits."""
    import torch
    import torch.distributed as dist

    samples = []
    for _ in range(repeats):
        dist.barrier()
        torch.cuda.synchronize()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for i in range(steps):
            step(i)
        end.record()
        if sampler is not None:
            sampler.sample_now()
        torch.cuda.synchronize()
        dist.barrier()
        samples.append(max_over_ranks(start.elapsed_time(end) * 1000.0 / steps))
    return samples


def summarise(samples):
    return {"median": round(statistics.median(samples), 2), "min": round(min(samples), 2), "max": round(max(samples), 2),
            "repeats": len(samples)}


def hashed_tokens(rank, tokens, hidden, device):
    """Token rows that any rank can regenerate from (source rank, token, column): small integers, exact in BF16."""
    import torch

    t = torch.arange(tokens, device=device, dtype=torch.int64).unsqueeze(1)
    c = torch.arange(hidden, device=device, dtype=torch.int64).unsqueeze(0)
    return (((rank * 131 + t * 7 + c * 3) % 251) - 125).to(torch.bfloat16)


def repeated_check(verify, all_gather, world, rounds=None):
    """``rounds`` verified exchanges (not timed), every rank in step: (this rank's last verdict, the verdicts of all
    ranks from the last round, whether every verdict of every round was fine).  Stops at the first round that any rank
    found wrong; an error raised by a check counts as that rank's verdict, so that all ranks keep making the same
    collective calls."""
    verdict, gathered = None, []
    for _ in range(VERIFY_ROUNDS if rounds is None else rounds):
        try:
            verdict = verify()
        except Exception as exc:  # noqa: BLE001 - an error word from the device (this buffer is finished) or anything else
            # that went wrong on this rank alone: it becomes this rank's verdict, so that every rank still reaches the gather
            verdict = {"ok": False, "rows_checked": 0, "elements_checked": 0, "problems": [f"{type(exc).__name__}: {exc}"[:200]]}
        gathered = [None] * world
        all_gather(gathered, verdict)
        if not all(v["ok"] for v in gathered):
            return verdict, gathered, False
    return verdict, gathered, True


FENCE_ENV = "PCIE_EP_B200_FENCE_EVERY_ROW"


def verified_buffer(make_buffer, check, world, environ=None):
    """A buffer whose exchange passed ``check`` (``repeated_check`` bound to the buffer), and the check's record.

    Should the exchange deliver a wrong row, the buffer is rebuilt once with one system-scope fence per row (the
    conservative way to publish a row; the runtime reads the setting from the environment when it is built) and the
    record says so under ``conservative_flags``; a second failure, or a failure where nothing is left to fall back
    to (one rank, or the conservative setting already in force), raises.  Every rank takes the same branch: ``check``
    returns the same verdict on all of them."""
    environ = os.environ if environ is None else environ
    buffer = make_buffer()
    payload_check, verdicts, fine = check(buffer)
    conservative = None
    if not fine and world > 1 and environ.get(FENCE_ENV) != "1":
        conservative = {"mode": "one system-scope fence per row", "after": [v["problems"] for v in verdicts if not v["ok"]][:2]}
        try:
            buffer.close()
        except Exception:  # noqa: BLE001 - a buffer that failed on the device may refuse an orderly close
            pass
        environ[FENCE_ENV] = "1"
        buffer = make_buffer()
        payload_check, verdicts, fine = check(buffer)
    if not fine:
        raise RuntimeError(f"payload check failed: {[v['problems'] for v in verdicts if not v['ok']]}")
    payload_check = dict(payload_check, elements_checked_all_ranks=sum(v["elements_checked"] for v in verdicts), rounds=VERIFY_ROUNDS)
    if conservative is not None:
        payload_check["conservative_flags"] = conservative
    return buffer, payload_check


def verify_exchange(buffer, rank, world, tokens, topk, idx_cpu, dev_idx, dev_w, device, wire="bf16"):
    """One dispatch + combine with regenerable payload: every received row is compared, on the GPU, with the row
    its (source rank, source token) metadata says it must be; dedup counters are compared with the route volume;
    the combined output is compared with the input (identity experts, weights sum to one).  Collective.

    With the FP8 wire a row from another rank must equal, bit for bit, the E4M3 round trip of its source (one scale per
    row); rows of the rank itself never take the wire format."""
    import torch

    from pcie_ep_b200.quantization import fp8_roundtrip_reference

    x = hashed_tokens(rank, tokens, HIDDEN, device)
    recv_x, recv_idx, _, handle, _ = buffer.dispatch(x, dev_idx, dev_w, do_expand=True)
    combined, _, _ = buffer.combine(recv_x, handle)
    torch.cuda.synchronize()
    buffer.check_errors()
    rows = int(handle.expanded_count)
    meta = handle.source_meta[:rows]
    problems, checked = [], 0
    cols = torch.arange(HIDDEN, device=device, dtype=torch.int64).unsqueeze(0)
    for lo in range(0, rows, 4096):
        part = meta[lo:lo + 4096]
        want = (((part[:, 0:1] * 131 + part[:, 1:2] * 7 + cols * 3) % 251) - 125).to(torch.bfloat16)
        if wire == "fp8_e4m3":
            want = torch.where(part[:, 0:1] == rank, want, fp8_roundtrip_reference(want).to(torch.bfloat16))
        if not torch.equal(recv_x[lo:lo + part.shape[0]], want):
            problems.append(f"rows {lo}..{lo + part.shape[0]} differ from their source")
            break
        checked += part.shape[0]
    local = EXPERTS // world
    ranks_hit = idx_cpu // local
    remote = ranks_hit != rank
    expect_sources = int(remote.any(dim=1).sum())
    expect_deliveries = sum(int((ranks_hit == d).any(dim=1).sum()) for d in range(world) if d != rank)
    stats = handle.stats.cpu().tolist()
    if stats[0] != expect_sources or stats[2] != expect_deliveries:
        problems.append(f"dedup counters {stats[:3]} != route volume ({expect_sources}, {expect_deliveries})")
    if rows != tokens * topk and world == 1:
        problems.append(f"expanded rows {rows} != {tokens * topk}")
    # (E4M3 keeps three mantissa bits: a quantised row is within 2^-4 of its source, relative, plus the subnormal floor)
    rtol, atol = (3e-2, 1.0) if wire == "bf16" else (8e-2, 2.0)
    if not torch.allclose(combined.float(), x.float(), rtol=rtol, atol=atol):
        problems.append("combined output differs from the input beyond the wire format's rounding")
    del recv_x, recv_idx, handle, combined
    return {"ok": not problems, "rows_checked": checked, "elements_checked": checked * HIDDEN, "problems": problems[:3]}


def run_ours(args, rank, world, local_rank):
    import torch
    import torch.distributed as dist

    from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer

    device = torch.device("cuda", local_rank)
    # pinned input buffers and the copy-issuing thread on the GPU's own NUMA node (8 ranks share two sockets)
    from pcie_ep_b200.utils.numa import bind_to_device_numa_node, bind_to_fastest_upload_node

    numa_node = None if args.no_numa_bind else bind_to_device_numa_node(local_rank)
    if numa_node is None and not args.no_numa_bind and not args.no_e2e:
        # the platform does not name the GPU's node: measure it, one rank at a time
        torch.cuda.set_device(device)
        for turn in range(world):
            if turn == rank:
                try:
                    numa_node = bind_to_fastest_upload_node(local_rank)
                except Exception as exc:  # noqa: BLE001 - placement is an optimisation, never a failure
                    numa_node = {"node": None, "error": f"{type(exc).__name__}: {exc}"[:160]}
            dist.barrier()

    def time_config(tokens, steps, warmup, want_e2e):
        tuned = HostStagedConfig.tuned(world, tokens)
        channels = args.channels or tuned.channels
        # send warps: with one rank every row is staged locally and the send role is latency-bound, four warps measured
        # best (dispatch 171 -> 161 us at T=4096); across NVLink two send and ten receive warps were best at 4 GPUs
        config = HostStagedConfig(channels=channels, stage=7 if args.wire != "bf16" else 6, wire_dtype=args.wire,
                                  copy_engine=args.engine, transport=args.transport, timeout_ms=20000,
                                  output_pool_size=2, tx_warps=args.tx_warps or tuned.tx_warps, rx_warps=args.rx_warps or tuned.rx_warps,
                                  combine_reduce=args.combine_reduce, send_ctas=args.send_ctas,
                                  pipeline_stages=args.stages or tuned.pipeline_stages)
        idx_cpu, w_cpu = make_routes(tokens, EXPERTS, args.topk, rank)
        dev_idx, dev_w = idx_cpu.to(device), w_cpu.to(device)

        def checked_exchanges(buf):
            return repeated_check(lambda: verify_exchange(buf, rank, world, tokens, args.topk, idx_cpu, dev_idx, dev_w, device, args.wire),
                                  dist.all_gather_object, world)

        # correctness evidence inside this very run: payload, dedup counters and the round trip (not timed)
        buffer, payload_check = verified_buffer(lambda: HostStagedEPBuffer(dist.group.WORLD, tokens, HIDDEN, args.topk, EXPERTS, config),
                                                checked_exchanges, world)
        g = torch.Generator().manual_seed(1234 + rank)
        host_x = [torch.randn(tokens, HIDDEN, generator=g).to(torch.bfloat16).pin_memory() for _ in range(INPUT_SETS)]
        host_idx, host_w = idx_cpu.pin_memory(), w_cpu.pin_memory()
        dev_x = [h.to(device) for h in host_x]

        def step(i):
            recv_x, _, _, handle, _ = buffer.dispatch(dev_x[i % INPUT_SETS], dev_idx, dev_w, do_expand=True)
            combined, _, _ = buffer.combine(recv_x, handle)
            return combined, handle

        for i in range(warmup):
            out, handle = step(i)
        torch.cuda.synchronize()
        buffer.check_errors()
        del out, handle

        def full_step(i):
            out, handle = step(i)
            del out, handle

        def dispatch_only(i):
            res = buffer.dispatch(dev_x[i % INPUT_SETS], dev_idx, dev_w, do_expand=True)
            del res

        sampler = ClockSampler(local_rank)
        sampler.start()
        total_samples = timed_repeats(full_step, steps, sampler=sampler)
        clocks = sampler.stop()
        dispatch_samples = timed_repeats(dispatch_only, steps, 3)
        buffer.check_errors()
        # dispatch and combine each with an event pair of their own, inside the full step (one extra pass)
        def split_pass():
            # in a function of its own: no name of this scope keeps a result pool referenced afterwards
            dist.barrier()
            torch.cuda.synchronize()
            marks = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(steps)]
            for i in range(steps):
                marks[i][0].record()
                recv_x, _, _, handle, event = buffer.dispatch(dev_x[i % INPUT_SETS], dev_idx, dev_w, do_expand=True)
                marks[i][1].record()
                combined, _, cevent = buffer.combine(recv_x, handle)
                marks[i][2].record()
                del recv_x, handle, combined, event, cevent
            torch.cuda.synchronize()
            return (max_over_ranks(sum(m[0].elapsed_time(m[1]) for m in marks) * 1000.0 / steps),
                    max_over_ranks(sum(m[1].elapsed_time(m[2]) for m in marks) * 1000.0 / steps))

        dispatch_in_step, combine_in_step = split_pass()
        # the dispatch kernel's own span (first CTA start to last CTA end, %globaltimer): separates
        # device time from host launch overhead at small T
        res = buffer.dispatch(dev_x[0], dev_idx, dev_w, do_expand=True)
        torch.cuda.synchronize()
        stamps = res[3].transport_timestamps_ns.cpu().tolist()
        kernel_us = (stamps[1] - stamps[0]) / 1000.0
        del res
        kernels = ["local_dispatch_kernel" if buffer.runtime.dispatch_is_local() else "dispatch_kernel"]
        if buffer.runtime.combine_is_inline():
            kernels.append("combine_kernel")
        else:
            kernels.append("local_combine_push_kernel" if buffer.runtime.combine_is_local() else "combine_push_kernel")
            if buffer.runtime.combine_is_split():
                kernels.append("fused_reduce_kernel")
        result = {
            "us_per_step": statistics.median(total_samples),
            "spread": summarise(total_samples),
            "dispatch_us": statistics.median(dispatch_samples),
            "dispatch_in_step_us": dispatch_in_step,
            "combine_us": combine_in_step,
            "dispatch_kernel_us": max_over_ranks(kernel_us),
            "clocks": clocks,
            "channels": channels,
            "kernels": kernels,
            "launches_per_step": len(kernels),
            "warps": (f"{buffer.runtime.send_ctas()} sender CTAs x {config.tx_warps} send warps, {channels} channel CTAs x "
                      f"(1 control + {config.rx_warps} receive/expand warps)" if buffer.runtime.send_ctas() else
                      f"1 control + {config.tx_warps} send + {config.rx_warps} receive/expand warps per channel CTA"),
            "roofline": roofline(idx_cpu, world, rank, tokens, args.topk, EXPERTS),
            "payload_check": payload_check,
        }
        if want_e2e:
            checksum_host = torch.zeros(1, dtype=torch.float32).pin_memory()
            h2d = host_x[0].numel() * 2 + host_idx.numel() * 8 + host_w.numel() * 4
            # A serving loop: two input buffers on the device, a copy stream that brings step i+1's inputs
            # from pinned host memory while step i computes, and a blocking read of every step's result.
            # Every step's host->device copy and device->host read are inside the timed region.
            copy_stream = torch.cuda.Stream()
            stages = [(torch.empty_like(dev_x[0]), torch.empty_like(dev_idx), torch.empty_like(dev_w)) for _ in range(2)]
            copied = [torch.cuda.Event() for _ in range(2)]
            consumed = [torch.cuda.Event() for _ in range(2)]

            def upload(i):
                slot = i % 2
                with torch.cuda.stream(copy_stream):
                    copy_stream.wait_event(consumed[slot])  # the kernels that read this buffer two steps ago are done
                    stages[slot][0].copy_(host_x[i % INPUT_SETS], non_blocking=True)
                    stages[slot][1].copy_(host_idx, non_blocking=True)
                    stages[slot][2].copy_(host_w, non_blocking=True)
                    copied[slot].record(copy_stream)

            def e2e_loop(count):
                compute = torch.cuda.current_stream()
                for slot in range(2):
                    consumed[slot].record(compute)
                upload(0)
                total = 0.0
                for i in range(count):
                    slot = i % 2
                    if i + 1 < count:
                        upload(i + 1)
                    compute.wait_event(copied[slot])
                    sx, si, sw = stages[slot]
                    recv_x, _, _, handle, _ = buffer.dispatch(sx, si, sw, do_expand=True)
                    combined, _, _ = buffer.combine(recv_x, handle)
                    consumed[slot].record(compute)
                    checksum_host.copy_(combined[:, :8].float().sum().reshape(1), non_blocking=True)
                    compute.synchronize()  # the step's result is read on the host
                    total += float(checksum_host[0])
                    del recv_x, handle, combined
                return total

            e2e_loop(min(3, warmup))
            e2e_samples = []
            for _ in range(3):
                dist.barrier()
                torch.cuda.synchronize()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                e2e_loop(steps)
                e1.record()
                torch.cuda.synchronize()
                e2e_samples.append(max_over_ranks(e0.elapsed_time(e1) * 1000.0 / steps))
            result["e2e"] = {"value": statistics.median(e2e_samples), "unit": "us/step", "spread": summarise(e2e_samples),
                             "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": 4,
                             "how": "inputs double-buffered: a copy stream uploads step i+1 from pinned memory while step i runs; every step ends with a blocking 4-byte read of its checksum",
                             "host_numa_node": numa_node}
            buffer.check_errors()
        # and once more after everything that was timed: the exchange still delivers what it should
        after, after_all, after_fine = checked_exchanges(buffer)
        result["payload_check_after"] = {"ok": after_fine, "problems": [v["problems"] for v in after_all if not v["ok"]][:2]}
        buffer.close()
        return result

    headline = time_config(args.tokens, args.steps, args.warmup, not args.no_e2e)
    sweep = {}
    if args.sweep:
        for tokens in (128, 256, 1024, 4096, 8192):
            if tokens == args.tokens:
                sweep[str(tokens)] = {"us_per_step": round(headline["us_per_step"], 2), "dispatch_us": round(headline["dispatch_us"], 2),
                                      "dispatch_kernel_us": round(headline["dispatch_kernel_us"], 2), "channels": headline["channels"]}
                continue
            r = time_config(tokens, args.steps, args.warmup, False)
            sweep[str(tokens)] = {"us_per_step": round(r["us_per_step"], 2), "dispatch_us": round(r["dispatch_us"], 2),
                                  "dispatch_kernel_us": round(r["dispatch_kernel_us"], 2), "channels": r["channels"]}
    if rank == 0:
        published = PUBLISHED_MS.get(args.tokens)
        value = headline["us_per_step"]
        line = {
            "metric": METRIC % args.topk,
            "value": round(value, 2),
            "unit": "us/step",
            "n_gpus": world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": round(value / 1000.0, 5),
            "higher_is_better": False,
            "scaling": "weak",
            "vs_baseline": round(value / (published * 1000.0), 5) if published else None,
            "baseline_note": "published number is the reference's dispatch-only latency at 8 ranks on 8xH20D PCIe5; "
                             "value here includes combine",
            "dtype": "bf16" if args.wire == "bf16" else "bf16 in/out, fp8_e4m3 wire",
            "data": "synthetic: x~N(0,1) bf16, distinct uniform top-k expert ids, softmax weights, random-init",
            "config": {
                "model": MODEL_NAME % args.topk,
                "tokens_per_rank": args.tokens,
                "global_batch": args.tokens * world,
                "seq_len": 1,
                "parallelism": f"ep{world}",
                "do_expand": True,
                "channels": headline["channels"],
                "warps": headline["warps"],
                "transport": args.transport,
                "copy_engine": args.engine,
                "l2": f"inputs rotate over {INPUT_SETS} token sets ({INPUT_SETS * args.tokens * HIDDEN * 2 >> 20} MiB) and each "
                      "step writes staging + expanded rows well beyond the 126 MB L2",
            },
            "timing": dict(headline["spread"], how=f"{REPEATS} timed regions of exactly --steps steps each, every one between "
                                                   "barrier + synchronize and a CUDA-event pair, max over ranks; value = median"),
            "dispatch_us": round(headline["dispatch_us"], 2),
            "dispatch_in_step_us": round(headline["dispatch_in_step_us"], 2),
            "dispatch_kernel_us": round(headline["dispatch_kernel_us"], 2),
            "combine_us": round(headline["combine_us"], 2),
            "split_how": "dispatch_us: dispatch-only loops (median of 3); dispatch_in_step_us and combine_us: an event pair "
                         "around each call inside full steps (one extra pass)",
            "clocks": headline["clocks"],
            "roofline": dict(headline["roofline"],
                             dispatch_fraction=round(headline["roofline"]["dispatch_us"] / headline["dispatch_us"], 3),
                             combine_fraction=round(headline["roofline"]["combine_us"] / max(headline["combine_us"], 1e-9), 3)),
            "gpu_launches": headline["launches_per_step"] * args.steps,
            "kernels_per_step": ", ".join(headline["kernels"]),
            "payload_check": headline["payload_check"],
            "payload_check_after": headline.get("payload_check_after"),
            "flag_publication": ("one system-scope fence per row" if os.environ.get(FENCE_ENV) == "1"
                                 else "READY flags of up to eight rows behind one system-scope fence"),
            "impl": "ours",
            "source_fingerprint": source_fingerprint(),
        }
        if "e2e" in headline:
            line["e2e"] = {k: (round(v, 2) if isinstance(v, float) else v) for k, v in headline["e2e"].items()}
        if sweep:
            line["sweep"] = sweep
        print(json.dumps(line), flush=True)


def run_reference(args, rank, world, local_rank):
    """The unmodified reference (copied to baseline/_ref) through its own public API: dispatch only."""
    import torch
    import torch.distributed as dist

    ref_root = ROOT / "baseline" / "_ref"
    if not (ref_root / "pcie_ep" / "__init__.py").exists():
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "baseline/_ref is missing (reference not installed)"}))
        return
    os.environ["TORCH_CUDA_ARCH_LIST"] = "10.0"
    os.environ.setdefault("TORCH_EXTENSIONS_DIR", str(ROOT / "baseline" / "_ref_build"))
    sys.path.insert(0, str(ref_root))
    try:
        from pcie_ep import HostStagedConfig, HostStagedEPBuffer

        device = torch.device("cuda", local_rank)
        tokens = args.tokens
        config = HostStagedConfig(timeout_ms=20000)
        buffer = HostStagedEPBuffer(dist.group.WORLD, tokens, HIDDEN, args.topk, EXPERTS, config)
        g = torch.Generator().manual_seed(1234 + rank)
        xs = [torch.randn(tokens, HIDDEN, generator=g).to(torch.bfloat16).to(device) for _ in range(INPUT_SETS)]
        idx_cpu, w_cpu = make_routes(tokens, EXPERTS, args.topk, rank)
        idx, w = idx_cpu.to(device), w_cpu.to(device)
        for i in range(args.warmup):
            res = buffer.dispatch(xs[i % INPUT_SETS], idx, w, do_expand=True)
            del res
        torch.cuda.synchronize()
        buffer.check_errors()
        def reference_step(i):
            res = buffer.dispatch(xs[i % INPUT_SETS], idx, w, do_expand=True)
            del res

        sampler = ClockSampler(local_rank)
        sampler.start()
        samples = timed_repeats(reference_step, args.steps, sampler=sampler)
        clocks = sampler.stop()
        buffer.check_errors()
        value = statistics.median(samples)
        e2e = None
        if not args.no_e2e:
            # the same serving loop as the other arm around the reference's dispatch: pinned host inputs uploaded
            # every step by a copy stream (double-buffered), a blocking device->host read of every step's result
            host_x = [x.cpu().pin_memory() for x in xs]
            host_idx, host_w = idx_cpu.pin_memory(), w_cpu.pin_memory()
            checksum_host = torch.zeros(1, dtype=torch.float32).pin_memory()
            h2d = host_x[0].numel() * 2 + host_idx.numel() * 8 + host_w.numel() * 4
            copy_stream = torch.cuda.Stream()
            stages = [(torch.empty_like(xs[0]), torch.empty_like(idx), torch.empty_like(w)) for _ in range(2)]
            copied = [torch.cuda.Event() for _ in range(2)]
            consumed = [torch.cuda.Event() for _ in range(2)]

            def upload(i):
                slot = i % 2
                with torch.cuda.stream(copy_stream):
                    copy_stream.wait_event(consumed[slot])
                    stages[slot][0].copy_(host_x[i % INPUT_SETS], non_blocking=True)
                    stages[slot][1].copy_(host_idx, non_blocking=True)
                    stages[slot][2].copy_(host_w, non_blocking=True)
                    copied[slot].record(copy_stream)

            def e2e_loop(count):
                compute = torch.cuda.current_stream()
                for slot in range(2):
                    consumed[slot].record(compute)
                upload(0)
                for i in range(count):
                    slot = i % 2
                    if i + 1 < count:
                        upload(i + 1)
                    compute.wait_event(copied[slot])
                    sx, si, sw = stages[slot]
                    res = buffer.dispatch(sx, si, sw, do_expand=True)
                    consumed[slot].record(compute)
                    checksum_host.copy_(res[0][:tokens, :8].float().sum().reshape(1), non_blocking=True)
                    compute.synchronize()
                    del res

            e2e_loop(min(3, args.warmup))
            e2e_samples = []
            for _ in range(3):
                dist.barrier()
                torch.cuda.synchronize()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                e2e_loop(args.steps)
                e1.record()
                torch.cuda.synchronize()
                e2e_samples.append(max_over_ranks(e0.elapsed_time(e1) * 1000.0 / args.steps))
            buffer.check_errors()
            e2e = {"value": round(statistics.median(e2e_samples), 2), "unit": "us/step", "spread": summarise(e2e_samples),
                   "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": 4,
                   "how": "same double-buffered upload loop as the other arm around the reference's dispatch (it has no combine)"}
        buffer.close()
    except Exception as exc:  # noqa: BLE001 - reported as unavailable
        reason = f"{type(exc).__name__}: {str(exc).splitlines()[0][:200] if str(exc) else ''}"
        failures = [None] * world
        try:
            dist.all_gather_object(failures, reason)
        except Exception:  # noqa: BLE001
            pass
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": reason}))
        return
    if rank == 0:
        published = PUBLISHED_MS.get(args.tokens)
        print(json.dumps({
            "impl": "reference",
            "metric": METRIC % args.topk,
            "reference_note": "dispatch only: the reference has no combine, so its value is a lower bound of what the "
                              "full exchange would cost it and any ratio against it is an under-estimate",
            "value": round(value, 2), "unit": "us/step", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": round(value / 1000.0, 5), "higher_is_better": False, "scaling": "weak",
            "vs_baseline": round(value / (published * 1000.0), 5) if published else None,
            "dtype": "bf16", "data": "synthetic, same generator as the other arm",
            "config": {"model": MODEL_NAME % args.topk, "tokens_per_rank": args.tokens,
                       "global_batch": args.tokens * world, "seq_len": 1, "parallelism": f"ep{world}",
                       "transport": "host_staged (reference default config)"},
            "timing": dict(summarise(samples), how=f"{REPEATS} timed regions of exactly --steps steps, median"),
            "dispatch_us": round(value, 2),
            "clocks": clocks, "gpu_launches": 8 * args.steps,
            **({"e2e": e2e} if e2e is not None else {}),
        }), flush=True)


def reexec_reference_with_system_libstdcxx():
    """The reference's extension uses std::ifstream.  In this image an extension built by
    torch.utils.cpp_extension does not record libstdc++ as a dependency, its iostream symbols then bind
    to copies inside other loaded libraries and the first ifstream use segfaults.  Preloading the
    system libstdc++ fixes the binding without touching the reference, so the reference arm runs in a
    child process started with LD_PRELOAD (every rank starts its own child; RANK/WORLD_SIZE/MASTER_* are
    inherited)."""
    import glob

    if os.environ.get("BENCH_REFERENCE_CHILD") == "1":
        return False
    candidates = sorted(glob.glob("/usr/lib/x86_64-linux-gnu/libstdc++.so.6") + glob.glob("/usr/lib64/libstdc++.so.6"))
    if not candidates:
        return False
    env = dict(os.environ)
    env["BENCH_REFERENCE_CHILD"] = "1"
    env["LD_PRELOAD"] = candidates[0] + (":" + env["LD_PRELOAD"] if env.get("LD_PRELOAD") else "")
    proc = subprocess.run([sys.executable, os.path.abspath(__file__), *sys.argv[1:]], env=env)
    if proc.returncode != 0 and int(os.environ.get("RANK", "0")) == 0:
        print(json.dumps({"impl": "reference", "unavailable": f"reference process exited with code {proc.returncode}"}), flush=True)
    return True


def main():
    args = parse_args()
    if args.impl == "reference" and reexec_reference_with_system_libstdcxx():
        return
    rank, world, local_rank = init_distributed(args)
    import torch.distributed as dist

    try:
        if args.impl == "reference":
            run_reference(args, rank, world, local_rank)
        else:
            run_ours(args, rank, world, local_rank)
    finally:
        if dist.is_initialized():
            dist.destroy_process_group()


if __name__ == "__main__":
    main()
