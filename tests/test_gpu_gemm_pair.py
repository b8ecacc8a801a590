"""The tensor-core kernel for pairs of SMs (more than 16 rows; 2 and 8 bits at any number) at the edges of its split: column
tiles with one CTA or part of one beyond the layer, cut k-tiles and units, one to four groups per unit, more tiles than pairs
(persistent), one and two sets of accumulators, and K split over pairs."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from autogptq.tvm_b200 import _lib, ops, synth
    DEV = torch.device("cuda:0")

CASES = [
    # bits, K, N, gs, M, gather
    (4, 32, 32, 32, 65, False),           # half a k-tile, one quarter of one CTA
    (4, 4128, 9632, 64, 700, False),      # odd number of k-tiles, several tiles per pair
    (3, 1184, 288, 96, 257, True),        # three-block groups, zero-point rows that start inside a 16-byte word
    (3, 2048, 19200, 128, 300, False),
    (2, 1056, 96, 32, 20, True),
    (2, 640, 4832, -1, 130, False),
    (8, 2080, 4128, 128, 9, False),
    (8, 96, 640, 32, 513, False),
    (4, 11008, 4096, 64, 77, False),      # four runs of K
    (8, 11008, 1056, 32, 128, True),
    (4, 992, 96, 32, 17, False),          # fewest rows of 3- and 4-bit layers
    (3, 4096, 4128, 128, 33, True),       # four runs, seventeen pairs of column tiles
    (4, 2048, 19232, -1, 64, False),      # a second tile for some pairs
    (3, 4064, 64, 32, 96, False),         # four runs above 64 rows
]


@pytest.mark.parametrize("bits,K,N,gs,M,gather", CASES)
def test_gemm_against_dequantised_product(bits, K, N, gs, M, gather):
    """The (bit-exact, separately tested) dequantised weights times x in fp32; twice, and with the groups as a g_idx, to the bit."""
    d = synth.make_layer(bits, K, N, gs, False, bias=True, seed=K + N, device=DEV)
    x = synth.make_x(M, K, seed=M, device=DEV)
    perm = torch.randperm(K, device=DEV).to(torch.int32) if gather else None
    run = lambda g: ops.gemm(x, d.qweight, d.qzeros, d.scales, g, bits, gs, bias=d.bias, x_perm=perm)
    y = run(None)
    _, W = ops.dequantize(d.qweight, d.qzeros, d.scales, d.g_idx, bits, gs, want_q=False)
    xg = (x if perm is None else x[:, perm.long()]).double()
    ref = xg @ W.double() + d.bias.double()
    # fp32 accumulation of K exact products (rounded or truncated: 2^-23 each) and one fp16 rounding
    bound = 2.0 ** -11 * ref.abs() + K * 2.0 ** -23 * (xg.abs() @ W.double().abs()) + 2.0 ** -24
    assert bool(((y.double() - ref).abs() <= bound).all())
    assert torch.equal(y, run(None)) and torch.equal(y, run(d.g_idx))
    ops.check_status(DEV)


@pytest.mark.parametrize("bits,K,N,gs,M,gather,runs", [
    (4, 11008, 4096, 64, 256, False, 2),      # runs over several tiles of rows
    (8, 8192, 2048, -1, 200, True, 4),
    (3, 8224, 2080, 32, 400, False, 2),       # a cut last unit, a part of a column tile, tiles of more than 96 rows
    (4, 8192, 2048, 128, 129, False, 4),      # fewest rows that are weighed
    (2, 8192, 2048, 128, 90, False, 4),       # rings smaller than the room that the sums need
    (2, 1056, 9472, 32, 130, False, 1),
])
def test_runs_of_k(bits, K, N, gs, M, gather, runs):
    assert ops.gemm_split(M, K, N, bits)[0] == runs
    test_gemm_against_dequantised_product(bits, K, N, gs, M, gather)


def test_split_of_the_cases_above():
    assert ops.gemm_split(77, 11008, 4096, 4)[0] == 4
    assert ops.gemm_split(128, 11008, 1056, 8)[0] == 4
    assert ops.gemm_split(33, 4096, 4128, 3) == (4, 1)
    assert ops.gemm_split(64, 2048, 19232, 4) == (1, 1)
    assert ops.gemm_split(96, 4064, 64, 3)[0] == 4


@pytest.mark.parametrize("K", [4096, 384])       # more units of K than there are stages, and fewer
def test_a_kernel_in_front_that_takes_longer_than_a_bounded_wait(K):
    """The kernel unpacks weights while the one in front of it still runs; the time it waits for that one is not its own.  In front: an
    all-reduce whose peer never comes, which gives up after 2.4e9 clocks (the GEMM's own waits end after 2e9)."""
    d = synth.make_layer(4, K, 1056, 128, False, seed=K, device=DEV)
    x = synth.make_x(77, K, seed=1, device=DEV)
    run = lambda: ops.gemm(x, d.qweight, d.qzeros, d.scales, None, 4, 128)
    want = run()
    buffers = [torch.zeros(int(_lib.lib.b200gptq_tp_buffer_bytes()), dtype=torch.uint8, device=DEV) for _ in range(2)]
    exchange = SimpleNamespace(rank=0, world=2, peer_table=(ctypes.c_void_p * 2)(*(b.data_ptr() for b in buffers)),
                               timeout_cycles=2_400_000_000)
    y = torch.zeros((1, 256), dtype=torch.float16, device=DEV)
    torch.cuda.synchronize()
    ops.tp_allreduce(y, exchange)
    got = run()
    torch.cuda.synchronize()
    assert int(buffers[0][:4].view(torch.int32)) == 2       # the all-reduce did run out of time
    assert torch.equal(got, want)
    ops.check_status(DEV)


def test_scratch_of_a_longer_prompt_serves_a_shorter_one():
    """More than 128 rows are taken with any scratch that holds the counters and a copy of x; without room for the sums of several runs
    of K there is one run."""
    bits, K, N, gs = 4, 8192, 2048, 128
    d = synth.make_layer(bits, K, N, gs, False, seed=4, device=DEV)
    x = synth.make_x(400, K, seed=5, device=DEV)
    need = lambda M: _lib.workspace_bytes(_lib.OP_GEMM, M, K, N, bits)
    assert ops.gemm_split(400, K, N, bits)[0] > 1 and need(1024) < need(400)
    _, W = ops.dequantize(d.qweight, d.qzeros, d.scales, d.g_idx, bits, gs, want_q=False)
    ref, size = x.double() @ W.double(), x.double().abs() @ W.double().abs()
    for nbytes in (need(400), need(1024), 16384 + 2 * 400 * K):
        ws = torch.zeros(nbytes, dtype=torch.uint8, device=DEV)
        y = ops.gemm(x, d.qweight, d.qzeros, d.scales, None, bits, gs, workspace=ws)
        assert bool(((y.double() - ref).abs() <= 2.0 ** -11 * ref.abs() + K * 2.0 ** -23 * size + 2.0 ** -24).all())
        assert not bool(ws[:16384].any())
    with pytest.raises((RuntimeError, ValueError)):
        ops.gemm(x, d.qweight, d.qzeros, d.scales, None, bits, gs, workspace=ws[:-16])
