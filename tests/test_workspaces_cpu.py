"""Workspaces of several threads (no GPU: a stand-in for what a workspace allocates)."""

import threading
import time

import pytest
import torch

from chunked_ep_moe_b200 import ChunkedMoEConfig
from chunked_ep_moe_b200.ops import fused

CFG = ChunkedMoEConfig(num_experts=4, top_k=2, slice_size=64, transport="nvshmem", expert_compute="fused", stripe_width=64)


class _Arena:
    def __init__(self):
        self.closed = 0

    def close(self):
        time.sleep(0.1)  # (the real one waits for the device)
        self.closed += 1


class _Rank:
    def release(self):
        pass


class _Workspace:
    made = []

    def __init__(self, cfg, group, hidden, ffn, tk_cap):
        time.sleep(0.05)  # (the real one allocates)
        self.world, self.tk_cap, self.arena, self.rank = 1, tk_cap, _Arena(), _Rank()
        _Workspace.made.append(self)


@pytest.fixture
def workspaces(monkeypatch):
    monkeypatch.setattr(fused, "FusedWorkspace", _Workspace)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(fused, "_workspaces", {})
    monkeypatch.setattr(fused, "_retired", [])
    monkeypatch.setattr(_Workspace, "made", [])


def _at_once(calls):
    got, start = [None] * len(calls), threading.Barrier(len(calls))

    def work(i):
        start.wait()
        got[i] = calls[i]()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return got


def test_threads_share_one_workspace(workspaces):
    """First calls at once make one workspace, calls that need more replace it once; all of them are found when they are released."""
    first = _at_once([lambda: fused.get_workspace(CFG, None, 256, 256, 100)] * 4)
    assert len(_Workspace.made) == 1 and all(ws is _Workspace.made[0] for ws in first)
    larger = _at_once([lambda: fused.get_workspace(CFG, None, 256, 256, 200)] * 4)
    assert len(_Workspace.made) == 2 and all(ws is _Workspace.made[1] for ws in larger)
    assert fused._retired == [_Workspace.made[0]] and not fused._making
    fused.release_workspaces()
    assert [ws.arena.closed for ws in _Workspace.made] == [1, 1]


def test_a_release_beside_first_calls_leaves_nothing_behind(workspaces):
    """A workspace that is being made while another thread releases those that there are: either released as well or there for the next call."""
    fused.get_workspace(CFG, None, 256, 256, 100)
    _at_once([lambda: fused.get_workspace(CFG, None, 512, 256, 100), fused.release_workspaces])
    assert len(_Workspace.made) == 2
    for ws in _Workspace.made:
        assert ws.arena.closed == (0 if ws in fused._workspaces.values() else 1)
