"""CPU: what threads share on the host side, with a stand-in for the library."""

import contextlib
import threading
import time
import types

import pytest
import torch

from sage_b200 import _lib, experts, ops


class Library:
    """Counts the calls that use a workspace at the same time."""

    def __init__(self):
        self.inside = self.most = 0

    def _use(self, *args):
        self.inside += 1
        self.most = max(self.most, self.inside)
        time.sleep(0.002)
        self.inside -= 1
        return 0

    sageb200_linear_grouped = sageb200_linear_grouped_fused = sageb200_experts = sageb200_expert_blocks = _use

    def _bytes(self, *args):
        return 4096

    sageb200_grouped_workspace_bytes = sageb200_fused_workspace_bytes = _bytes
    sageb200_experts_workspace_bytes = sageb200_expert_blocks_workspace_bytes = _bytes


@pytest.fixture
def library(monkeypatch):
    library = Library()
    monkeypatch.setattr(_lib, "load", lambda: library)
    monkeypatch.setattr(_lib, "check", lambda status: None)
    monkeypatch.setattr(ops, "_check_layout", lambda x, *packed: x.shape[-1])
    monkeypatch.setattr(ops, "_WORKSPACES", {})
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=0))
    return library


def grouped(library):
    x, packed = torch.zeros(2, 128, dtype=torch.float16), [torch.zeros(1, 64, 2, dtype=torch.float16)] * 5
    ops.sage_grouped([(x, *packed)], [16])


def fused(library):
    x, packed = torch.zeros(2, 128, dtype=torch.float16), [torch.zeros(1, 64, 2, dtype=torch.float16)] * 5
    ops.sage_grouped([(x, *packed)], [16], activation=(2, 0.0, x, x, None, None))


def slots(library):
    experts.SAGEExperts._run(None, library, 0, 0, (_lib.ExpertStack * 1)(), None, torch.zeros(1, dtype=torch.int32), 1, 0)


@pytest.mark.parametrize("call", [grouped, fused, slots])
def test_threads_take_turns_with_a_workspace(library, call):
    """A call is several launches through one buffer per stream: the next thread's comes behind all of them."""
    threads = [threading.Thread(target=lambda: [call(library) for _ in range(5)]) for _ in range(4)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert library.most == 1
