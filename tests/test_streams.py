"""The pool of CUDA events: which of them count as free (no GPU: an event that was never recorded is a plain object); and how the
kernels that may start before the launch in front of them has ended read their inputs."""

import re
import sys
from pathlib import Path

import pytest
import torch

from pcie_ep_b200.buffers import streams


class _Counts:
    """Stands in for ``sys``: an interpreter whose calls add another number of references than this one's."""

    def __init__(self, off):
        self.off = off

    def getrefcount(self, value):
        return sys.getrefcount(value) - 1 + self.off  # (-1: this call's own name)


def _pool(monkeypatch, getrefcount_of):
    monkeypatch.setattr(streams, "sys", getrefcount_of)
    monkeypatch.setattr(torch.cuda, "Event", type("Event", (), {}))
    policy = streams.StreamPolicy(0, False)
    return policy


@pytest.mark.parametrize("off", [-1, 0, 1])
def test_a_held_event_is_never_handed_out_again_whatever_the_interpreter_counts(monkeypatch, off):
    policy = _pool(monkeypatch, _Counts(off))
    held = [policy.event() for _ in range(5)]
    assert len({id(e) for e in held}) == 5
    kept = held[2]
    del held
    seen = {id(policy.event()) for _ in range(20)}
    assert id(kept) not in seen
    assert len(seen) == 4  # the others are used again


def test_no_pool_where_holders_do_not_show_in_the_count(monkeypatch):
    policy = _pool(monkeypatch, type("Constant", (), {"getrefcount": staticmethod(lambda value: 2)}))
    held = [policy.event() for _ in range(5)]
    assert len({id(e) for e in held}) == 5 and policy._events == []


def test_kernels_that_start_early_read_by_loads_that_stay_behind_the_wait():
    """A launch that may start before the one in front of it has ended reads what that one wrote: ld.global.nc (__ldg) promises
    memory that nobody writes while the kernel runs, so a compiler may move it in front of the wait."""
    kernels = Path(__file__).resolve().parents[1] / "csrc" / "kernels"
    early = [p for p in sorted(kernels.iterdir()) if p.name != "ptx.cuh" and "wait_for_launch_before" in p.read_text()]
    assert {p.name for p in early} == {"combine_local.cuh", "expert_gemm.cu"}
    for path in early:
        code = re.sub(r"//[^\n]*", "", path.read_text())
        assert "__ldg" not in code and "ld.global.nc" not in code, path.name
