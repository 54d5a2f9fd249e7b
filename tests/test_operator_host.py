"""Host side of a differentiable operator call, without a GPU: what it refuses, whether it keeps its phases."""
import types

import pytest
import torch
from torch._subclasses import FakeTensorMode

from aussm_b200 import ops

MB = 1 << 20


def _stats(reserved, active, fragments):
    return {k + "_bytes": {"all": {"current": v * MB}} for k, v in
            (("reserved", reserved), ("active", active), ("inactive_split", fragments))}


@pytest.fixture
def memory(monkeypatch):
    """memory(statistics or an exception, free megabytes) -> list that counts the questions to the driver"""
    def setup(stats, free_mb, total_mb=1500):
        asked = []

        def statistics(device=None):
            if isinstance(stats, Exception):
                raise stats
            return stats

        def driver(device=None):
            asked.append(device)
            return free_mb * MB, 180_000 * MB

        monkeypatch.setattr(torch.cuda.memory, "memory_stats_as_nested_dict", statistics)
        monkeypatch.setattr(torch.cuda, "mem_get_info", driver)
        monkeypatch.setattr(torch.cuda, "get_device_properties",
                            lambda device=None: types.SimpleNamespace(total_memory=total_mb * MB))
        return asked
    return setup


def test_whole_unused_segments_answer_for_a_small_buffer(memory):
    asked = memory(_stats(1000, 200, 300), 0)
    assert ops._fits_a_quarter(125 * MB, "cuda") and not asked          # a quarter of 500 MB
    assert not ops._fits_a_quarter(126 * MB, "cuda") and asked


def test_fragments_are_not_free_memory(memory):
    """A reserve in pieces serves no contiguous request and cannot be given back: the driver's answer stands."""
    asked = memory(_stats(100_000, 20_000, 79_990), 20)
    assert not ops._fits_a_quarter(50 * MB, "cuda") and asked


def test_fragments_serve_requests_of_the_shared_segments(memory):
    asked = memory(_stats(1000, 980, 20), 0)
    assert ops._fits_a_quarter(5 * MB, "cuda") and not asked
    assert not ops._fits_a_quarter(6 * MB, "cuda") and asked


def test_fragments_count_while_the_card_has_room_for_a_new_segment(memory):
    stats = _stats(1000, 600, 400)
    asked = memory(stats, 0, total_mb=2000)
    assert ops._fits_a_quarter(100 * MB, "cuda") and not asked
    assert not ops._fits_a_quarter(101 * MB, "cuda") and asked
    asked = memory(stats, 0, total_mb=1999)
    assert not ops._fits_a_quarter(100 * MB, "cuda") and asked


def test_a_large_buffer_asks_the_driver(memory):
    """Unused blocks of other streams and of graphs' pools are in the allocator's count too."""
    asked = memory(_stats(100_000, 0, 0), 500)
    assert not ops._fits_a_quarter(1024 * MB, "cuda") and asked
    memory(_stats(100_000, 0, 0), 4096)
    assert ops._fits_a_quarter(1024 * MB, "cuda")


@pytest.mark.parametrize("stats", [{}, RuntimeError("this allocator has no statistics")])
def test_an_allocator_without_statistics_asks_the_driver(memory, stats):
    asked = memory(stats, 100)
    assert ops._fits_a_quarter(25 * MB, "cuda") and not ops._fits_a_quarter(26 * MB, "cuda") and len(asked) == 2


def test_a_buffer_that_does_not_fit_after_all(monkeypatch):
    """The call falls back to recomputing the phases, unless keeping them was asked for."""
    def full(*args, **kwargs):
        raise torch.cuda.OutOfMemoryError("full")

    monkeypatch.setattr(torch, "empty", full)
    assert ops._keep_buffer(MB, "cuda") is None
    monkeypatch.setattr(ops, "keep_phases", True)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        ops._keep_buffer(MB, "cuda")


@pytest.mark.parametrize("given", [10, 11])
def test_half_of_a_state_is_refused(given):
    b, d, n, l = 2, 8, 4, 16
    with FakeTensorMode():
        shapes = [(b, d, l), (b, d, l), (d, n, d), (d, n)] + [(n,)] * 4 + [(d,), (b, d, l), None, None]
        shapes[given] = (b, d, n)
        inputs = [None if s is None else torch.empty(s, device="cuda") for s in shapes]
        with pytest.raises(RuntimeError, match="both"):
            ops._check_op_inputs(*inputs)
