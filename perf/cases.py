"""The work that programs have this framework do on one GPU, as cases with sizes: MoE exchanges (dispatch and combine)
and whole MoE layers, from a few decode tokens to long prefill batches, through the public entry points.

A case is a dict of plain values.  ``listed()`` names the standing ones, ``draw(rng)`` makes another one of the same
ranges, ``prepare`` builds what a program holds before the call (the EP buffer, the inputs, the weights, a captured
graph), ``run`` makes one pass, ``work`` says what a pass cannot do without and ``tolerance`` how far two correct
implementations may be apart.

Kinds of case
    ``exchange``  ``buffer.dispatch`` then ``buffer.combine`` of the experts' output rows: what surrounds the expert FFN of
                  a layer.  ``expand`` picks rows per (token, expert) or per token.
    ``keep_fp8``  ``buffer.dispatch`` with rows that stay E4M3 at the receiver (codes and row scales for an FP8 GEMM).
    ``replay``    a captured dispatch with a cached layout, replayed, then the combine: a decode loop with fixed routes.
    ``layer``     ``MoELayer``: dispatch, grouped SwiGLU FFN, combine; ``fused`` merges the down projection with the
                  combine, ``fp8`` runs the gate/up GEMM on the E4M3 rows that the dispatch delivers.

One process, one GPU: the group has one rank, which owns every expert.  A buffer is built for ``capacity`` tokens and
called with ``tokens`` of them, as a server does whose batches vary.
"""

from __future__ import annotations

import math
import os
import tempfile

import torch
import torch.distributed as dist

from pcie_ep_b200 import HostStagedConfig, HostStagedEPBuffer
from pcie_ep_b200.models.moe_layer import MoELayer

#: share of the routing mass on the popular fifth of the experts, for ``profile="hotspot"``
HOT_EXPERTS, HOT_MASS = 0.2, 0.8


def _exchange(name, tokens, capacity, topk, *, hidden=7168, experts=256, profile="uniform", expand=True):
    return dict(name=name, kind="exchange", tokens=tokens, capacity=capacity, hidden=hidden, experts=experts, topk=topk,
                profile=profile, expand=expand)


def _layer(name, tokens, capacity, *, hidden=7168, inter=2048, experts=32, topk=8, profile="uniform", fp8=False, fused=False):
    return dict(name=name, kind="layer", tokens=tokens, capacity=capacity, hidden=hidden, inter=inter, experts=experts, topk=topk,
                profile=profile, fp8=fp8, fused=fused)


def listed():
    return [
        # one decode step of a small batch: nothing but latency and launches
        _exchange("exchange_t16", 16, 128, 8),
        # decode with a full batch
        _exchange("exchange_t128", 128, 128, 8),
        # a ragged chunk in a buffer built for 1024, another hidden size, skewed top-4 routes
        _exchange("exchange_t777_hot", 777, 1024, 4, hidden=4096, profile="hotspot"),
        # rows per token (not per expert): the layout for engines that gather inside their own GEMM
        _exchange("exchange_t2048_unique", 2048, 2048, 8, expand=False),
        # the headline exchange: one prefill chunk
        _exchange("exchange_t4096", 4096, 4096, 8),
        # the largest exchange, Zipf-popular experts, top-4
        _exchange("exchange_t8192_zipf", 8192, 8192, 4, profile="zipf"),
        # prefill chunk for an FP8 expert GEMM: quantise once, expand E4M3 rows
        dict(name="keep_fp8_t4096", kind="keep_fp8", tokens=4096, capacity=4096, hidden=7168, experts=256, topk=8, profile="uniform"),
        # decode loop with a captured dispatch
        dict(name="replay_t256", kind="replay", tokens=256, capacity=256, hidden=7168, experts=256, topk=8, profile="uniform"),
        # whole layers with the experts that one of eight ranks owns: a decode batch (weights dominate) ...
        _layer("layer_t64", 64, 128),
        # ... a ragged mixed batch with skewed experts, FP8 gate/up GEMM, in a buffer built for 1024 ...
        _layer("layer_t555_fp8_hot", 555, 1024, profile="hotspot", fp8=True),
        # ... a prefill chunk in BF16, down projection fused with the combine ...
        _layer("layer_t4096_fused", 4096, 4096, fused=True),
        # ... and one with the FP8 gate/up GEMM
        _layer("layer_t4096_fp8", 4096, 4096, fp8=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["exchange", "exchange", "exchange", "keep_fp8", "replay", "layer", "layer", "layer"])
    hidden = rng.choice([2048, 2880, 4096, 5120, 7168, 7168])
    topk = rng.choice([2, 4, 6, 8, 8])
    profile = rng.choice(["uniform", "hotspot", "zipf"])
    if kind == "layer":
        tokens = _log_int(rng, 16, 4096)
        case = dict(kind=kind, tokens=tokens, hidden=rng.choice([2048, 4096, 7168]), inter=rng.choice([768, 1024, 1536, 2048]),
                    experts=rng.choice([8, 16, 32]), topk=topk, profile=profile, fp8=rng.random() < 0.4, fused=rng.random() < 0.4)
    else:
        tokens = _log_int(rng, 16, 2048 if kind == "replay" else 8192)
        case = dict(kind=kind, tokens=tokens, hidden=hidden, experts=rng.choice([32, 64, 128, 256]), topk=topk, profile=profile)
        if kind == "keep_fp8":
            case["tokens"] = min(tokens, 4096)
        if kind == "exchange":
            case["expand"] = rng.random() < 0.75
    # a buffer is sized for the next power of two, or twice that
    case["capacity"] = max(128, min(8192 if kind == "exchange" else 4096, (1 << (case["tokens"] - 1).bit_length()) * rng.choice([1, 1, 2])))
    case["capacity"] = max(case["capacity"], case["tokens"])
    return case


# ---------------------------------------------------------------------------------------------------- inputs
def _group():
    """The process group of a single-process program (the data path never uses it)."""
    if not dist.is_initialized():
        store = dist.FileStore(os.path.join(tempfile.mkdtemp(prefix="ep-group-"), "store"), 1)
        dist.init_process_group("gloo", store=store, rank=0, world_size=1)
    return dist.group.WORLD


def _routes(case, gen):
    """Distinct expert ids per token (Gumbel top-k over the experts' popularity) and softmax weights."""
    tokens, experts, topk = case["tokens"], case["experts"], case["topk"]
    if case["profile"] == "zipf":
        popularity = 1.0 / torch.arange(1, experts + 1, device="cuda", dtype=torch.float32) ** 1.1
    elif case["profile"] == "hotspot":
        hot = max(1, int(experts * HOT_EXPERTS))
        popularity = torch.full((experts,), (1.0 - HOT_MASS) / (experts - hot), device="cuda")
        popularity[:hot] = HOT_MASS / hot
    else:
        popularity = torch.ones(experts, device="cuda")
    popularity = popularity[torch.randperm(experts, device="cuda", generator=gen)]
    uniform = torch.rand(tokens, experts, device="cuda", generator=gen).clamp_(1e-12, 1.0 - 1e-7)
    idx = (popularity.log() - (-uniform.log()).log()).topk(topk, dim=1).indices.to(torch.int64).contiguous()
    weights = torch.softmax(torch.randn(tokens, topk, device="cuda", generator=gen), dim=1).contiguous()
    return idx, weights


def _tokens(case, gen):
    x = torch.randn(case["tokens"], case["hidden"], device="cuda", generator=gen)
    if case["kind"] == "keep_fp8" or case.get("fp8"):
        # activations of real networks have a few large channels: one value in a hundred is fifty times as large
        x = torch.where(torch.rand(x.shape, device="cuda", generator=gen) < 0.01, x * 50.0, x)
    return x.to(torch.bfloat16)


def _config(case):
    fp8 = case["kind"] == "keep_fp8" or case.get("fp8", False)
    return HostStagedConfig.tuned(1, case["capacity"], stage=7 if fp8 else 6, wire_dtype="fp8_e4m3" if fp8 else "bf16",
                                  recv_dtype="fp8_e4m3" if fp8 else "bf16", enable_graph=case["kind"] == "replay",
                                  fused_expert_combine=case.get("fused", False))


class _State:
    """What the program holds; closes its buffer when dropped."""

    def __init__(self, case, buffer):
        self.case, self.buffer = case, buffer
        self.layer = self.graph = None

    def __del__(self):
        self.graph = self.layer = None
        self.buffer.close()


def prepare(case, seed):
    torch.cuda.set_device(0)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    group = _group()
    buffer = HostStagedEPBuffer(group, case["capacity"], case["hidden"], case["topk"], case["experts"], _config(case))
    state = _State(case, buffer)
    state.x = _tokens(case, gen)
    state.idx, state.weights = _routes(case, gen)
    if case["kind"] in ("exchange", "replay"):
        # what the experts hand to the combine
        state.y = torch.randn(_rows(case), case["hidden"], device="cuda", generator=gen, dtype=torch.bfloat16)
    if case["kind"] == "layer":
        experts, hidden, inter = case["experts"], case["hidden"], case["inter"]
        gate_up = torch.randn(experts, 2 * inter, hidden, device="cuda", generator=gen, dtype=torch.bfloat16) * 0.02
        down = torch.randn(experts, hidden, inter, device="cuda", generator=gen, dtype=torch.bfloat16) * 0.02
        state.layer = MoELayer(buffer, inter, with_router=False, weights=(gate_up, down))
    elif case["kind"] == "replay":
        _, _, _, handle, _ = buffer.dispatch(state.x, state.idx, state.weights, do_expand=True)
        layout = buffer.cache_layout(handle)
        del handle
        state.graph = buffer.capture_dispatch(state.x, None, state.weights, handle=layout, do_expand=True)
    return state


# ---------------------------------------------------------------------------------------------------- one pass
def _rows(case):
    """Rows that a dispatch fills on one rank (every token is routed to ``topk`` local experts); what lies behind them in
    the capacity-shaped results is spare room that nothing writes."""
    return case["tokens"] * (case["topk"] if case.get("expand", True) else 1)


def run(state):
    case, buffer = state.case, state.buffer
    if case["kind"] == "layer":
        return state.layer(state.x, state.idx, state.weights)
    expand = case.get("expand", True)
    if case["kind"] == "replay":
        recv_x, recv_idx, recv_w, handle, _ = state.graph.replay()
    else:
        recv_x, recv_idx, recv_w, handle, _ = buffer.dispatch(state.x, state.idx, state.weights, do_expand=expand)
    rows = _rows(case)
    out = dict(recv_x=recv_x[:rows], recv_idx=recv_idx[:rows], recv_w=recv_w[:rows], counts=handle.expert_counts,
               offsets=handle.expert_offsets)
    if case["kind"] == "keep_fp8":
        # the codes as bytes, and the scale of every row
        out["recv_x"], out["scales"] = recv_x.view(torch.uint8)[:rows], handle._result["recv_x_scales"][:rows]
        return out
    out["combined"], _, _ = buffer.combine(state.y, handle)
    return out


def _active_experts(case):
    """Experts that receive at least one row, on average (uniform routes; skewed ones leave some more idle)."""
    return case["experts"] * (1.0 - (1.0 - case["topk"] / case["experts"]) ** case["tokens"])


def work(case):
    tokens, hidden, topk = case["tokens"], case["hidden"], case["topk"]
    token_bytes, rows = tokens * hidden * 2, _rows(case)
    routes = tokens * topk * 12
    if case["kind"] == "layer":
        per_expert = case["inter"] * hidden * ((2 if case["fp8"] else 4) + 2)  # gate and up rows, down rows
        return {"bytes": 2 * token_bytes + routes + _active_experts(case) * per_expert,
                "flops": 2.0 * rows * hidden * case["inter"] * 3}
    if case["kind"] == "keep_fp8":
        return {"bytes": token_bytes + routes + rows * (hidden + 4), "flops": 0}
    return {"bytes": token_bytes + routes + 2 * rows * hidden * 2 + token_bytes, "flops": 2.0 * rows * hidden}


def tolerance(case):
    if case["kind"] == "keep_fp8":
        return "exact"
    if case["kind"] == "layer":
        # activations, expert outputs and the result are rounded to BF16: measured 2.9e-3 against the same layer in 64 bits
        return {"rel": 1.2e-2, "max": 0.08}
    # rows move unchanged; the weighted sum is taken in 32 bits and rounded to BF16 once: measured 1.7e-3 against 64 bits
    return {"rel": 6.6e-3, "max": 1.6e-2}


# ---------------------------------------------------------------------------------------------------- the values themselves
def _fp8_rows(rows):
    """Rows as the E4M3 codes of the wire format hold them (scale = largest magnitude / 448, one per row)."""
    rows = rows.float()
    peak = rows.abs().amax(dim=-1, keepdim=True)
    scale = torch.where(peak == 0, torch.ones_like(peak), (peak / 448.0).clamp_min(torch.finfo(torch.float32).tiny))
    return (rows * (1.0 / scale)).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double() * scale.double()


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits; ``None`` stands for rows and whole numbers that only move."""
    if case["kind"] == "keep_fp8":
        return None
    state = prepare(case, seed)
    x, idx, weights = state.x, state.idx, state.weights.double()
    if case["kind"] == "layer":
        fp8, inter = case["fp8"], case["inter"]
        rows = _fp8_rows(x) if fp8 else x.double()
        out = torch.zeros(x.shape, dtype=torch.float64, device=x.device)
        for expert in range(case["experts"]):
            token, slot = torch.nonzero(idx == expert, as_tuple=True)
            if token.numel() == 0:
                continue
            w = state.layer.w_gate_up[expert]
            gate_up = rows[token] @ (_fp8_rows(w) if fp8 else w.double()).t()
            hidden = torch.nn.functional.silu(gate_up[:, :inter]) * gate_up[:, inter:]
            out.index_add_(0, token, hidden @ state.layer.w_down[expert].double().t() * weights[token, slot].unsqueeze(1))
        return out
    result = dict(recv_x=None, recv_idx=None, recv_w=None, counts=None, offsets=None)
    if case.get("expand", True):
        # an expert's rows follow each other in token order, the experts in theirs
        order = torch.argsort(idx.reshape(-1), stable=True)
        row_of = torch.empty_like(order)
        row_of[order] = torch.arange(order.numel(), device=order.device)
        row_of = row_of.view(idx.shape)
        combined = torch.zeros(x.shape, dtype=torch.float64, device=x.device)
        for slot in range(case["topk"]):
            combined += state.y[row_of[:, slot]].double() * weights[:, slot:slot + 1]
        result["combined"] = combined
    else:
        result["combined"] = state.y.double()
    return result
