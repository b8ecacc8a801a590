"""Which scratch buffers ops.get_workspace keeps: the address of one that was handed out while its stream was captured is in a graph,
so it outlives its replacement.  (The native module and the streams are stand-ins here: no GPU.)"""
import pytest
import torch

from autogptq.tvm_b200 import ops

DEV = torch.device("cpu", 0)


class Host:
    """scratch_use, set_scratch and zeros_outside_capture as the native module has them; `capturing` is the stream's state."""

    def __init__(self):
        self.capturing, self.in_graph, self.outside = False, {}, 0

    def scratch_use(self, index, stream):
        key = (index, stream)
        if key in self.in_graph:
            self.in_graph[key] |= self.capturing
        return self.capturing, self.in_graph.get(key, False)

    def set_scratch(self, index, stream, tensor, size, in_graph):
        self.in_graph[index, stream] = in_graph

    def zeros_outside_capture(self, index, size):
        assert self.capturing
        self.outside += 1
        return torch.zeros(size, dtype=torch.uint8)


@pytest.fixture
def host(monkeypatch):
    h = Host()
    monkeypatch.setattr(ops._lib, "_host", h)
    monkeypatch.setattr(ops, "_stream", lambda device: 7)
    monkeypatch.setattr(ops, "_workspaces", {})
    monkeypatch.setattr(ops, "_held", {})
    return h


def test_scratch_that_a_graph_holds_is_kept(host):
    first = ops.get_workspace(DEV, 1 << 20)
    host.capturing = True
    assert ops.get_workspace(DEV, 1 << 20) is first          # the graph has its address now
    second = ops.get_workspace(DEV, (1 << 20) + 64)          # in the same capture, for a larger layer
    assert host.outside == 1 and ops._held[0, 7][0] is first
    host.capturing = False
    third = ops.get_workspace(DEV, second.numel() + 64)      # an ordinary call later on
    assert [w is k for w, k in zip(ops._held[0, 7], (first, second))] == [True, True] and host.outside == 1
    assert ops.get_workspace(DEV, 16) is third


def test_what_is_kept_is_smaller_than_the_scratch_in_use(host):
    host.capturing = True
    for n in range(1, 200):
        ws = ops.get_workspace(DEV, n * 100_000)
        assert sum(w.numel() for w in ops._held.get((0, 7), [])) < ws.numel() <= max(2 << 20, 2 * n * 100_000)


def test_scratch_that_no_graph_holds_is_given_back(host):
    first = ops.get_workspace(DEV, 1 << 20)
    first[16380:16384] = torch.tensor([1, 0, 0, 0], dtype=torch.uint8)      # the sticky status word
    second = ops.get_workspace(DEV, 2 << 20)
    assert not ops._held and second.numel() == 2 << 20 and second[16380] == 1
