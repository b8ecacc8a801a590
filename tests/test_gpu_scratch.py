"""Scratch under CUDA graphs: a graph that holds the address of a buffer can be replayed after a larger one has taken its place, and a
buffer that came with a capture serves other graphs at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from autogptq.tvm_b200 import ops, synth
    DEV = torch.device("cuda:0")


def test_graphs_outlive_the_growth_of_the_scratch():
    # the general kernel (explicit g_idx) counts and adds in the scratch
    layer = synth.make_layer(4, 2048, 1056, 64, True, seed=3, device=DEV)
    x = synth.make_x(3, 2048, seed=3, device=DEV)
    call = lambda: ops.gemv(x, layer.qweight, layer.qzeros, layer.scales, layer.g_idx, 4, 64)
    want = call()
    stream = torch.cuda.Stream(DEV)
    key = (0, stream.cuda_stream)
    base = len(ops._held.get(key, []))            # (streams come from a pool: an earlier test may have had this one)
    size = ops.get_workspace(DEV, 16).numel()
    with torch.cuda.stream(stream):
        size = max(size, ops.get_workspace(DEV, 16).numel())
    torch.cuda.synchronize()
    graphs, outs = [], []
    for grow in (0, size + 64, 0, 20 * size):     # in the second and the last capture the scratch grows between two calls
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=stream):
            a = call()
            if grow:
                ops.get_workspace(DEV, grow)
            b = call()
        graphs.append(g)
        outs.append((a, b))
    held = ops._held[key]
    assert len(held) == base + 2 and sum(w.numel() for w in held) < ops._workspaces[key].numel()
    torch.cuda.empty_cache()
    for i in (2, 3, 0, 1, 3):                     # first a graph that uses a buffer which came with another's capture
        for t in outs[i]:
            t.zero_()
        graphs[i].replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[i][0], want) and torch.equal(outs[i][1], want)
    for w in (*held, ops._workspaces[key]):
        assert not bool(w[:16384].any())
    ops.check_status(DEV)
