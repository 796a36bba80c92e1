"""The multiply's workspaces: which calls share one (host logic, no kernel is launched)."""
import copy
import threading
import types

import pytest
import torch

LIKE = torch.empty(0)


@pytest.fixture
def scratch(pkg_host, monkeypatch):
    state = types.SimpleNamespace(capturing=False, counters=0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capturing)
    monkeypatch.setattr(pkg_host, "load_library", lambda: types.SimpleNamespace(nmspmm_gemm_counter_bytes=lambda desc: state.counters))
    s = pkg_host.Scratch()
    s.state = state
    return s


def test_one_workspace_per_stream_and_thread(scratch):
    first = scratch.get(1024, None, LIKE, 7)
    assert first[1] == 1024 and not first[2].any() and scratch.get(512, None, LIKE, 7) is first
    assert scratch.get(1024, None, LIKE, 8) is not first                  # another stream
    other = []
    thread = threading.Thread(target=lambda: other.append(scratch.get(1024, None, LIKE, 7)))
    thread.start()
    thread.join()
    assert other[0] is not first                                         # another thread on the same stream
    grown = scratch.get(4096, None, LIKE, 7)
    assert grown is not first and grown[1] == 4096 and scratch.get(1024, None, LIKE, 7) is grown


def test_kept_workspaces_are_bounded(scratch):
    for stream in range(50):
        scratch.get(256, None, LIKE, stream)
    assert len(scratch._kept) == scratch.SLOTS
    big = scratch.get(scratch.KEEP_BYTES + 1, None, LIKE, 99)
    assert all(kept[2] is not big[2] for kept in scratch._kept.values())


def test_captured_calls_get_memory_of_their_own(scratch):
    kept = scratch.get(1024, None, LIKE, 7)
    scratch.state.capturing, scratch.state.counters = True, 256
    captured = scratch.get(1024, None, LIKE, 7)
    assert captured[2] is not kept[2] and not captured[2][:256].any()
    assert scratch.get(1024, None, LIKE, 7)[2] is not captured[2]
    scratch.state.capturing = False
    assert scratch.get(1024, None, LIKE, 7) is kept


def test_a_copied_owner_starts_without_workspaces(scratch, pkg_host):
    scratch.get(1024, None, LIKE, 7)
    assert isinstance(copy.deepcopy(scratch), pkg_host.Scratch) and not copy.deepcopy(scratch)._kept
