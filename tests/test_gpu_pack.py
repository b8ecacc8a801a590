"""GPU packing (b200gptq_pack_fields and QuantLinear.pack on a CUDA device) against the reference's own
pack outputs (tests/golden/pack_*.npz, produced by auto_gptq/nn_modules/qlinear.py:77-175) and against the
CPU packer of the module, bit for bit."""
import os

import numpy as np
import pytest
import torch
import torch.nn as nn

from conftest import GOLDEN_DIR, golden_files

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from autogptq.tvm_b200 import QuantLinear, ops
    from autogptq.tvm_b200.qlinear import _pack_fields
    DEV = torch.device("cuda:0")


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("R,C", [(32, 32), (128, 96), (4096, 1000)])
def test_pack_fields_equals_the_cpu_packer(bits, R, C):
    gen = torch.Generator().manual_seed(bits * 1000 + R + C)
    vals = torch.randint(0, 1 << bits, (R, C), generator=gen, dtype=torch.int64)
    # a few values wider than the field, and negative ones: the reference does not mask, neither do we
    vals[0, 0] = (1 << bits) + 1
    vals[R - 1, C - 1] = -1
    vals[R // 2, C // 2] = 0x12345678
    want = _pack_fields(torch.from_numpy(vals.numpy().astype(np.uint32).astype(np.int64)), bits)
    as_i32 = torch.from_numpy(vals.numpy().astype(np.uint32).view(np.int32).copy())
    got = ops.pack_fields(as_i32.to(DEV), bits)
    assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("fname", golden_files("pack_"))
def test_module_pack_on_gpu_matches_reference_vectors(fname):
    g = np.load(os.path.join(GOLDEN_DIR, fname))
    bits, gs = int(g["bits"]), int(g["group_size"])
    N, K = g["weight"].shape
    lin = nn.Linear(K, N, bias=True)
    lin.weight.data = torch.from_numpy(g["weight"])
    lin.bias.data = torch.from_numpy(g["lin_bias"])
    lin = lin.to(DEV)
    m = QuantLinear(bits, gs, K, N, True).to(DEV)
    m.pack(lin, torch.from_numpy(g["scales_in"]).to(DEV), torch.from_numpy(g["zeros_in"]).to(DEV),
           torch.from_numpy(g["g_idx"]).to(DEV))
    assert m.qweight.is_cuda and m.qzeros.is_cuda
    assert np.array_equal(m.qweight.cpu().numpy(), g["qweight"])
    assert np.array_equal(m.qzeros.cpu().numpy(), g["qzeros"])
    assert np.array_equal(m.scales.cpu().numpy().view(np.uint16), g["scales"].view(np.uint16))
    # and the packed layer computes what the reference computed with it
    y = m(torch.from_numpy(g["x"]).to(DEV))
    ref = g["out"].astype(np.float32)
    assert np.allclose(y.float().cpu().numpy(), ref, rtol=2e-3, atol=2e-3 * np.abs(ref).max())


def test_module_pack_gpu_equals_cpu_at_layer_size():
    bits, gs, K, N = 4, 128, 1024, 512
    gen = torch.Generator().manual_seed(5)
    lin = nn.Linear(K, N, bias=False)
    lin.weight.data = torch.randn(N, K, generator=gen) * 0.05
    G = K // gs
    scales = torch.rand(N, G, generator=gen) * 0.02 + 1e-3
    zeros = torch.randint(1, 16, (N, G), generator=gen).float()
    a = QuantLinear(bits, gs, K, N, False)
    a.pack(lin, scales, zeros)
    b = QuantLinear(bits, gs, K, N, False).to(DEV)
    b.pack(lin.to(DEV), scales.to(DEV), zeros.to(DEV))
    assert torch.equal(a.qweight, b.qweight.cpu())
    assert torch.equal(a.qzeros, b.qzeros.cpu())
    assert torch.equal(a.scales, b.scales.cpu())


def test_pack_fields_rejects_bad_arguments():
    with pytest.raises(ValueError):
        ops.pack_fields(torch.zeros((31, 8), dtype=torch.int32, device=DEV), 4)
    with pytest.raises(ValueError):
        ops.pack_fields(torch.zeros((32, 8), dtype=torch.int32, device=DEV), 5)
    with pytest.raises(RuntimeError):
        ops.pack_fields(torch.zeros((32, 8), dtype=torch.int32), 4)


@pytest.mark.parametrize("bits,K,N,gs,dtype", [
    (2, 32, 32, 32, torch.float16),           # smallest layer
    (3, 1056, 64, 32, torch.float32),         # K is no multiple of the 256-row chunk
    (4, 544, 96, -1, torch.bfloat16),
    (8, 4128, 64, 8, torch.float16),          # 516 groups: the table does not fit, groups cut 32-row blocks
])
def test_one_launch_pack_equals_the_cpu_packer(bits, K, N, gs, dtype):
    """b200gptq_pack_linear rounds a product with 1 / scale and falls back to the division near a half: random weights
    (any fraction) and exact halves must give the words of the CPU route."""
    gen = torch.Generator().manual_seed(bits + K)
    size = gs if gs != -1 else K
    G = -(-K // size)
    scales = torch.rand(N, G, generator=gen) * 0.02 + 1e-3
    zeros = torch.randint(1, 2 ** bits, (N, G), generator=gen).float()
    g_idx = (torch.randperm(K, generator=gen) // size).to(torch.int32)
    sel = g_idx.long()
    W = (torch.rand(N, K, generator=gen) * (2 ** bits - 1) - zeros[:, sel]) * scales[:, sel]
    s16 = scales[:, sel].half().float()
    W[1] = ((torch.arange(K) % (2 ** bits - 1)).float() + 0.5) * s16[1] - (zeros * scales)[:, sel][1]
    lin = nn.Linear(K, N, bias=False)
    lin.weight.data = W.to(dtype)
    a, b = QuantLinear(bits, gs, K, N, False), QuantLinear(bits, gs, K, N, False).to(DEV)
    a.pack(lin, scales, zeros, g_idx)
    b.pack(lin.to(DEV), scales.to(DEV), zeros.to(DEV), g_idx.to(DEV))
    assert torch.equal(a.qweight, b.qweight.cpu())
    assert torch.equal(a.qzeros, b.qzeros.cpu())
    assert torch.equal(a.scales, b.scales.cpu())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("K,N,gs", [(288, 32, 32), (4480, 64, 32)])     # (140 groups: more than one tile of the zero-points)
def test_one_launch_pack_in_order_and_out_of_range(bits, K, N, gs, dtype):
    """Rows in group order take no table; fields outside 0..2^bits-1 spill into their neighbours as the CPU route has them."""
    gen = torch.Generator().manual_seed(bits + K)
    G = K // gs
    scales = 2.0 ** torch.randint(-8, -3, (N, G), generator=gen).float()
    zeros = torch.randint(1, 2 ** bits, (N, G), generator=gen).float()
    sel = torch.arange(K) // gs
    q = torch.randint(0, 2 ** bits, (N, K), generator=gen).float()
    for i, wrong in enumerate([-1., 2. ** bits, 300., -4194304., -9437184., 2.**24]):
        q[3 + i, 17 * i + 9] = wrong
    lin = nn.Linear(K, N, bias=False)
    W = (q - zeros[:, sel]) * scales[:, sel]
    lin.weight.data = W if dtype is torch.float32 else W.clamp(-6e4, 6e4).to(dtype)          # (finite)
    a, b = QuantLinear(bits, gs, K, N, False), QuantLinear(bits, gs, K, N, False).to(DEV)
    a.pack(lin, scales, zeros)
    b.pack(lin.to(DEV), scales.to(DEV), zeros.to(DEV))
    assert torch.equal(a.qweight, b.qweight.cpu())
    assert torch.equal(a.qzeros, b.qzeros.cpu())
    assert torch.equal(a.scales, b.scales.cpu())


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("K,N,gs", [(32, 32, 32), (288, 64, 16), (544, 32, -1), (4480, 96, 64), (16384, 32, 16)])
def test_fp16_weights_equal_the_cpu_packer(bits, K, N, gs):
    """fp16 weights of 2 to 4 bits are rounded in fp16 where that gives the quotient's integer for certain: any fraction, with quotients on
    both sides of the line (0.4375 from an integer) and of a half, zero-points and scales past the ones that fp16 takes (|zero * scale / s|
    > 32, 1 / s no normal number), negative scales, groups that cut 32-row blocks, more groups than the
    table holds (16384 rows in groups of 16)."""
    gen = torch.Generator().manual_seed(bits + K)
    size = gs if gs != -1 else K
    G, top = -(-K // size), 2 ** bits - 1
    scales = torch.rand(N, G, generator=gen) * 0.02 + 1e-3
    zeros = torch.randint(1, top + 2, (N, G), generator=gen).float()
    zeros[3::8], zeros[4::8] = 31.99, 33.0
    scales[5::8], scales[6::8], scales[7::8] = 2.0 ** -15.5, 20000.0, -scales[7::8]
    g_idx = (torch.randperm(K, generator=gen) // size).to(torch.int32)
    sel = g_idx.long()
    frac = torch.tensor([0.0, 0.43, 0.4375, 0.45, 0.4999, 0.5, 0.5001, -0.43, -0.4375, -0.45, -0.5, -0.5001])
    q = torch.randint(0, top + 1, (N, K), generator=gen) + frac[torch.randint(0, len(frac), (N, K), generator=gen)]
    q[0] = torch.rand(K, generator=gen) * (top + 2) - 1
    W = ((q - zeros[:, sel]) * scales[:, sel]).clamp(-6e4, 6e4).half()     # (finite: what an infinity becomes as an integer is nobody's)
    lin = nn.Linear(K, N, bias=False)
    lin.weight.data = W
    a, b = QuantLinear(bits, gs, K, N, False), QuantLinear(bits, gs, K, N, False).to(DEV)
    a.pack(lin, scales, zeros, g_idx)
    b.pack(lin.to(DEV), scales.to(DEV), zeros.to(DEV), g_idx.to(DEV))
    assert torch.equal(a.qweight, b.qweight.cpu())
    assert torch.equal(a.qzeros, b.qzeros.cpu())
    assert torch.equal(a.scales, b.scales.cpu())


@pytest.mark.parametrize("act", [False, True])
@pytest.mark.parametrize("wrong", [-1.0, "above", 300.0, "tiny scale", "huge scale", "zero-point"])
@pytest.mark.parametrize("bits", [2, 3, 4])
def test_fp16_columns_beside_one_that_is_redone(bits, wrong, act):
    """Columns c and c + 16 of a strip are packed in the two halves of a register.  Every field is an integer in the range, so that no block
    is redone, but for one field or one group's constants of columns c < 16 that send column c to the division: at each row of a block once, and
    in each group; column c + 16, which is not redone, must not notice."""
    K, N, gs = 1024, 96, 64
    gen = torch.Generator().manual_seed(bits)
    G, top = K // gs, 2 ** bits - 1
    scales = 2.0 ** torch.randint(-8, -3, (N, G), generator=gen).float()
    zeros = torch.randint(1, top + 1, (N, G), generator=gen).float()
    g_idx = torch.arange(K) // gs
    if act:
        g_idx = g_idx[torch.randperm(K, generator=gen)]
    q = torch.randint(0, top + 1, (N, K), generator=gen).float()
    bad = [(32 * (g % 2) + g % 16, g) for g in range(G)]                   # columns 0..15 and 32..47, a group each
    for n, g in bad:
        if wrong == "tiny scale":
            scales[n, g] = 2.0 ** -15.5
        elif wrong == "huge scale":
            scales[n, g], zeros[n, g] = 16384.0, 1.0
            q[n, g_idx == g] = q[n, g_idx == g].clamp(max=3)
        elif wrong == "zero-point":
            zeros[n, g] = 40.0
    if wrong not in ("tiny scale", "huge scale", "zero-point"):
        for j in range(K // 32):                                           # row j of block j
            q[32 * (j % 2) + j // 2, 32 * j + j] = top + 1.0 if wrong == "above" else wrong
    sel = g_idx.long()
    lin = nn.Linear(K, N, bias=False)
    lin.weight.data = ((q - zeros[:, sel]) * scales[:, sel]).half()
    a, b = QuantLinear(bits, gs, K, N, False), QuantLinear(bits, gs, K, N, False).to(DEV)
    a.pack(lin, scales, zeros, g_idx.to(torch.int32))
    b.pack(lin.to(DEV), scales.to(DEV), zeros.to(DEV), g_idx.to(torch.int32).to(DEV))
    differ = (a.qweight != b.qweight.cpu()).any(dim=0).nonzero().flatten().tolist()
    assert not differ, f"columns {differ}"
    assert torch.equal(a.qzeros, b.qzeros.cpu()) and torch.equal(a.scales, b.scales.cpu())


def test_pack_in_one_native_call_keeps_what_the_python_route_has():
    """The native call and the Python route (taken here because of a scale that is not contiguous, an int64 g_idx, a CPU g_idx) store the
    same buffers; the caller's g_idx is copied, the module's own kept where none is given, and hooks on buffers see every one."""
    K, N, gs = 256, 64, 64
    gen = torch.Generator().manual_seed(3)
    lin = nn.Linear(K, N, bias=True)
    lin.weight.data = torch.randn(N, K, generator=gen).half() * 0.05
    lin = lin.to(DEV)
    scales, zeros = (torch.rand(N, K // gs, generator=gen) * 0.02 + 1e-3).to(DEV), torch.randint(1, 16, (N, K // gs), generator=gen).float().to(DEV)
    g_idx = (torch.randperm(K, generator=gen) // gs).to(torch.int32).to(DEV)
    want = QuantLinear(4, gs, K, N, True).to(DEV)
    want.pack(lin, scales, zeros, g_idx)
    assert want.g_idx.data_ptr() != g_idx.data_ptr() and want.g_idx.dtype == torch.int32 and torch.equal(want.g_idx, g_idx)
    for kw in (dict(scales=scales.t().contiguous().t()), dict(g_idx=g_idx.long()), dict(g_idx=g_idx.cpu())):
        m = QuantLinear(4, gs, K, N, True).to(DEV)
        m.pack(lin, kw.get("scales", scales), zeros, kw.get("g_idx", g_idx))
        for name in ("qweight", "qzeros", "scales", "bias"):
            assert torch.equal(getattr(m, name), getattr(want, name)), name
        assert torch.equal(m.g_idx.to(DEV), g_idx.to(m.g_idx.dtype)) and m.g_idx.dtype == kw.get("g_idx", g_idx).dtype
    m = QuantLinear(4, gs, K, N, True).to(DEV)
    own = m.g_idx
    seen = []
    hook = torch.nn.modules.module.register_module_buffer_registration_hook(lambda mod, name, b: seen.append(name))
    try:
        m.pack(lin, scales, zeros)
    finally:
        hook.remove()
    assert m.g_idx is own and {"qweight", "qzeros", "scales"} <= set(seen)
    assert set(m.state_dict()) == {"qweight", "qzeros", "scales", "g_idx", "bias"}
    with pytest.raises(ValueError):
        m.pack(lin, scales[:, :2].contiguous(), zeros, g_idx)


@pytest.mark.parametrize("K,N,gs,dtype", [(10720, 320, -1, torch.float16), (9984, 256, -1, torch.float32)])
def test_the_copy_of_g_idx_costs_narrow_layers_little(K, N, gs, dtype):
    """A narrow layer has few CTAs for its constants; the copy took them up to half as long as the whole launch."""
    scales, zeros = torch.rand(N, 1, device=DEV) * 0.02 + 1e-3, torch.full((N, 1), 8.0, device=DEV)
    lin = nn.Linear(K, N, bias=False, device=DEV, dtype=dtype)
    lin.weight.data = (torch.randint(-8, 8, (N, K), device=DEV) * scales).to(dtype)
    g_idx, m = torch.zeros(K, dtype=torch.int32, device=DEV), QuantLinear(4, gs, K, N, False).to(DEV)

    def us(*given):
        m.pack(lin, scales, zeros, *given)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                m.pack(lin, scales, zeros, *given)
        times = []
        for _ in range(20):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record(), graph.replay(), ev[1].record()
            torch.cuda.synchronize()
            times.append(ev[0].elapsed_time(ev[1]))
        return min(times)
    assert us(g_idx) < 1.15 * us()
    assert torch.equal(m.g_idx, g_idx)
