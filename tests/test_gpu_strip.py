"""The decode GEMV for groups of whole 32-row blocks at the edges of its work split: all bit widths, groups inside and
across the 128-row units, a cut last unit, one strip of columns up to more strips than a pass, one row (byte planes, or fp16
where the row is long), two rows (planes) and more rows (fp16), with and without a gather."""
import numpy as np
import pytest
import torch

from oracle import gptq_oracle as O

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from autogptq.tvm_b200 import ops, synth
    DEV = torch.device("cuda:0")

CASES = [
    # bits, K, N, gs, gather
    (2, 32, 32, 32, False),            # a quarter of a unit, one strip
    (2, 1184, 4800, 96, True),         # groups of three steps, cut last unit, more strips than CTAs
    (2, 2048, 64, 128, False),
    (3, 160, 96, 32, False),
    (3, 1088, 5088, 64, True),
    (3, 4224, 288, 128, True),
    (3, 32768, 64, 128, False),        # planes of one row do not fit: fp16, the row kept whole
    (3, 69632, 32, 128, False),        # nor does the row
    (4, 49152, 64, 128, False),        # nor the row and its copy, one row included
    (2, 65536, 96, 64, False),
    (8, 40960, 32, 32, False),
    (4, 992, 96, 32, True),
    (4, 1056, 64, -1, False),          # one group, cut last unit
    (4, 640, 19008, 128, False),       # 594 strips: five per CTA, overlapping passes
    (4, 28672, 64, 1024, True),        # too long to gather from shared memory
    (8, 96, 32, 32, False),
    (8, 1152, 4832, 64, False),
    (8, 2560, 160, -1, True),
]


@pytest.mark.parametrize("bits,K,N,gs,gather", CASES)
@pytest.mark.parametrize("M", [1, 2, 3, 8])
def test_gemv_vs_oracle(bits, K, N, gs, gather, M):
    layer = synth.make_layer(bits, K, N, gs, False, bias=N % 96 == 0, seed=K + N + bits)
    _, _, W = O.dequantize(layer.qweight.numpy(), layer.qzeros.numpy(), layer.scales.numpy(), layer.g_idx.numpy(), bits)
    x = synth.make_x(M, K, seed=M)
    perm = torch.randperm(K, generator=torch.Generator().manual_seed(K)).to(torch.int32) if gather else None
    xg = x if perm is None else x[:, perm.long()]
    bias = None if layer.bias is None else layer.bias.numpy()
    d = layer.to(DEV)
    run = lambda **kw: ops.gemv(x.to(DEV), d.qweight, d.qzeros, d.scales, None, bits, gs, bias=d.bias,
                                x_perm=None if perm is None else perm.to(DEV), **kw)
    ref = O.forward_fp64(xg.numpy(), W, bias)
    # One fp16 rounding of the result, and the weights: the oracle rounds scale * (q - zero) to fp16, the kernel does not.  That
    # is up to 2^-11 |w| each with independent signs, a standard deviation of 2^-11 / sqrt(3) * norm(x) * rms(w); the largest
    # of 1e5 outputs is at 4.5 of them, and rms(w) is below a third of max |w| here: 2^-11 * norm(x) * max |w|.  The fp32
    # sums (2 and 3 bits subtract sums of powers of two up to 2^10 times the inputs) stay far below that.
    norm = np.linalg.norm(xg.numpy().astype(np.float64), axis=1, keepdims=True) * np.abs(W.astype(np.float64)).max()
    for y in (run(), run(tuning=(2, 1))):       # eight warps and sixteen
        err = np.abs(y.cpu().numpy().astype(np.float64) - ref)
        assert np.all(err <= 2.0 ** -10 * np.abs(ref) + 2.0 ** -11 * norm), err.max()
    ops.check_status(DEV)


@pytest.mark.parametrize("bits,K,N,gs,gather", [
    # planes with groups inside a unit (4 bits, from two strips per CTA and 16 units on): of one, two and three blocks, cut units
    (4, 992, 4832, 32, False), (4, 1120, 9632, 64, True), (4, 2080, 4832, 96, True), (4, 96, 4832, 32, True),
    (4, 2080, 4832, 32, False), (4, 2144, 9632, 64, True), (4, 2016, 9632, 96, False), (4, 3168, 4832, 32, True),
    # the last sizes that stay in fp16, and the first on planes
    (4, 2048, 4832, 128, True), (2, 2080, 4832, 128, False), (3, 2048, 9632, 128, False), (3, 2080, 9632, 128, True),
    (4, 1920, 9632, 128, False), (4, 4128, 4832, 32, False), (3, 4128, 19008, 128, True), (3, 1056, 19008, -1, False),
    # planes of one strip per CTA: one long row, rows with a gather
    (4, 8224, 96, 128, True), (4, 4128, 64, 128, True), (4, 4096, 4096, 128, False),
    # more pairs of units than one per warp, rows picked one by one
    (2, 5152, 9632, 128, True), (3, 9248, 14432, 128, True), (3, 4128, 14432, -1, False), (2, 4128, 4832, 160, False),
])
@pytest.mark.parametrize("M", [1, 2])
def test_byte_planes_vs_oracle(bits, K, N, gs, gather, M):
    """(test_gemv_vs_oracle's bound)"""
    test_gemv_vs_oracle(bits, K, N, gs, gather, M)


def _bound_of_planes(bits, x, w, a, rows):
    """What fixed point per `rows` rows of x and fp32 sums may be off by, for x [M, K], exact weights w and a = scale * (field + zero):
    X is rounded at 2^-26 of a power of two above the largest |x| (4 bits; 2^-22 for 2 and 3), uniformly, seven standard deviations
    for 1e5 outputs; every unit's sums are rounded half a dozen times and added over up to 16 units and 16 warps (2^-24 each)."""
    M, K = x.shape
    var, top = 0.0, 0.0
    for k in range(0, K, rows):
        m = np.abs(x[:, k:k + rows]).max(axis=1, keepdims=True)
        e = np.where(m > 0, np.floor(np.log2(np.maximum(m, 2.0 ** -24))) + 1, -30.0)
        step = 2.0 ** (e - (26 if bits == 4 else 22))
        var = var + step ** 2 / 12 * (w[k:k + rows] ** 2).sum(axis=0, keepdims=True)
        top = top + np.abs(x[:, k:k + rows]) @ a[k:k + rows]
    return 7 * np.sqrt(var) + 38 * 2.0 ** -24 * top


def _run_and_exact(layer, x):
    """The kernel's result, and the result, weights and scale * (field + zero) in 64 bits (no rounding of the weights)."""
    q, z, _ = O.dequantize(layer.qweight.numpy(), layer.qzeros.numpy(), layer.scales.numpy(), layer.g_idx.numpy(), layer.bits)
    g = layer.g_idx.numpy().astype(np.int64)
    s, q, z = layer.scales.numpy().astype(np.float64)[g], q.astype(np.float64), z.astype(np.float64)[g]
    w = s * (q - z)
    d = layer.to(DEV)
    y = ops.gemv(x.to(DEV), d.qweight, d.qzeros, d.scales, None, layer.bits, layer.group_size).cpu().numpy().astype(np.float64)
    ops.check_status(DEV)
    return y, x.numpy().astype(np.float64) @ w, w, s * (q + z)


@pytest.mark.parametrize("bits,K,N,gs", [(4, 4128, 9632, 32), (4, 4160, 9632, 64), (4, 4128, 9632, 96), (4, 4224, 9632, 128),
                                         (3, 4224, 9632, 128), (2, 4224, 9632, 128)])
@pytest.mark.parametrize("M", [1, 2])
def test_groups_of_other_magnitudes_keep_their_bits(bits, K, N, gs, M):
    """Neighbouring groups whose x differs by up to 2^23 and whose scales make up for it, on byte planes: the small ones count as much
    as the large ones.  (A fixed point shared by groups that are scaled apart loses them.)"""
    layer = synth.make_layer(bits, K, N, gs, False, seed=K + bits)
    G = layer.scales.shape[0]
    mag = 2.0 ** torch.tensor([[-10, 13, -9, 4, 0, -8][g % 6] for g in range(G)], dtype=torch.float64)
    gen = torch.Generator().manual_seed(5)
    layer.scales = ((1 + torch.rand((G, N), generator=gen)) / mag[:, None]).half()
    x = torch.randn((M, K), generator=gen).double() * mag[layer.g_idx.long()]
    x[:, 128:256] = 0.0                                    # a unit of zeros
    x[:, 300:416:3] = 0.0
    x = x.clamp(-60000, 60000).half()
    y, ref, w, a = _run_and_exact(layer, x)
    bound = _bound_of_planes(bits, x.numpy().astype(np.float64), w, a, 32 if gs % 128 else 128) + 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    assert np.all(np.abs(y - ref) <= bound), (np.abs(y - ref) / bound).max()


@pytest.mark.parametrize("M", [1, 2])
def test_small_values_beside_outliers_keep_their_bits(M):
    """4 bits, every 128 rows with two values 4e6 times the others that cancel exactly (rows of equal weights): what is left shows in
    how many bits the others were held."""
    K, N = 4096, 9632
    layer = synth.make_layer(4, K, N, 128, False, seed=9)
    first = layer.qweight[0::16]
    layer.qweight[0::16] = (first & ~0xf0) | ((first & 0xf) << 4)          # row 1 of every unit like row 0
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(6)) * 2.0 ** -7
    x[:, 0::128], x[:, 1::128] = 30000.0, -30000.0
    x = x.half()
    y, ref, w, a = _run_and_exact(layer, x)
    rest = np.abs(x.numpy().astype(np.float64))
    rest[:, 0::128] = rest[:, 1::128] = 0.0
    xs = x.numpy().astype(np.float64)
    w[0::128] = w[1::128] = 0.0                            # (exact in fixed point: integers of 11 bits)
    a[0::128] = a[1::128] = 0.0
    bound = _bound_of_planes(4, xs, w, a, 128) + 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    assert np.all(np.abs(y - ref) <= bound), (np.abs(y - ref) / bound).max()


@pytest.mark.parametrize("bits,K,N,gs,gather", [(2, 544, 96, 32, True), (3, 1152, 4832, 128, False), (3, 1184, 64, 64, True),
                                                (4, 4096, 4800, 128, True), (4, 992, 32, 32, False), (8, 288, 9632, -1, False),
                                                # x does not fit: places in turn, three and four of them, several passes
                                                (3, 6144, 9632, 128, False), (4, 12288, 4832, 128, False)])
@pytest.mark.parametrize("M", [9, 16])
def test_plan_of_nine_to_sixteen_rows_vs_oracle(bits, K, N, gs, gather, M):
    layer = synth.make_layer(bits, K, N, gs, False, bias=True, seed=K + N + bits)
    _, _, W = O.dequantize(layer.qweight.numpy(), layer.qzeros.numpy(), layer.scales.numpy(), layer.g_idx.numpy(), bits)
    x = synth.make_x(M, K, seed=M)
    perm = torch.randperm(K, generator=torch.Generator().manual_seed(K)).to(torch.int32) if gather else None
    xg = x if perm is None else x[:, perm.long()]
    d = layer.to(DEV)
    plan = ops.GemvPlan(d.qweight, d.qzeros, d.scales, None, None if perm is None else perm.to(DEV), d.bias, M, bits, gs)
    ref = O.forward_fp64(xg.numpy(), W, layer.bias.numpy())
    norm = np.linalg.norm(xg.numpy().astype(np.float64), axis=1, keepdims=True) * np.abs(W.astype(np.float64)).max()
    err = np.abs(plan.run(x.to(DEV)).cpu().numpy().astype(np.float64) - ref)
    assert np.all(err <= 2.0 ** -10 * np.abs(ref) + 2.0 ** -11 * norm), err.max()
    ops.check_status(DEV)


@pytest.mark.parametrize("bits,K", [(4, 1024), (4, 4096), (3, 4096), (4, 57344)])     # fp16, planes, the row kept, and too long for that
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("M", [1, 3])
def test_folded_activation_equals_the_kernel_in_front(bits, K, gated, M):
    layer = synth.make_layer(bits, K, 4832, 128, False, seed=K, device=DEV)
    u = synth.make_x(M, 2 * K if gated else K, seed=M, device=DEV)
    a = ops.act(u, torch.empty((M, K), dtype=torch.float16, device=DEV), K, gated)
    args = (layer.qweight, layer.qzeros, layer.scales, None, bits, 128)
    assert torch.equal(ops.gemv(u, *args, input_act=1 if gated else 2), ops.gemv(a, *args))
    ops.check_status(DEV)


@pytest.mark.parametrize("bits,K,N,gs,gather,M", [
    # four CTAs per strip (up to 33 strips on 148 SMs): the shortest K of one row and of sixteen; units that do not divide; a cut last unit
    (4, 4864, 32, 128, False, 1), (4, 8032, 1184, 32, False, 2), (3, 8064, 1024, 128, True, 8), (2, 11008, 1024, 128, False, 16),
    (8, 10496, 1152, 128, False, 5), (4, 2176, 1024, 128, False, 16), (4, 2208, 992, 96, True, 9), (3, 10272, 64, -1, False, 3),
    # two CTAs (up to 74 strips); the largest and smallest number of them
    (4, 9856, 1856, 64, False, 2), (4, 11008, 2368, 128, False, 8), (3, 8992, 1216, 128, True, 1), (8, 7168, 2304, 128, False, 12),
    (2, 8192, 1536, 64, False, 4), (4, 40960, 1536, 128, False, 1),
    # one strip more, or a little less K: unsplit
    (4, 11008, 2400, 128, False, 8), (4, 4608, 1024, 128, False, 1), (4, 11008, 1824, 128, True, 4),
])
def test_layers_of_few_strips_vs_oracle(bits, K, N, gs, gather, M):
    """Clusters of CTAs that share a strip, against the oracle (test_gemv_vs_oracle's bound), and the same bits every time."""
    layer = synth.make_layer(bits, K, N, gs, False, bias=N % 96 == 0, seed=K + N + bits)
    _, _, W = O.dequantize(layer.qweight.numpy(), layer.qzeros.numpy(), layer.scales.numpy(), layer.g_idx.numpy(), bits)
    x = synth.make_x(M, K, seed=M)
    perm = torch.randperm(K, generator=torch.Generator().manual_seed(K)).to(torch.int32) if gather else None
    xg = x if perm is None else x[:, perm.long()]
    d = layer.to(DEV)
    plan = ops.GemvPlan(d.qweight, d.qzeros, d.scales, None, None if perm is None else perm.to(DEV), d.bias, M, bits,
                        gs if gs != -1 else K, None, 0)
    y = plan.run(x.to(DEV))
    assert torch.equal(y, plan.run(x.to(DEV)))
    ops.check_status(DEV)
    ref = O.forward_fp64(xg.numpy(), W, None if layer.bias is None else layer.bias.numpy())
    err = np.abs(y.cpu().numpy().astype(np.float64) - ref)
    bound = 2.0 ** -11 * np.abs(ref) + 2.0 ** -11 * np.linalg.norm(xg.numpy().astype(np.float64), axis=1)[:, None] * np.abs(W.astype(np.float64)).max()
    assert np.all(err <= bound), (err / bound).max()


@pytest.mark.parametrize("K,M", [(4096, 8), (8192, 1), (11008, 16)])
def test_clusters_that_share_a_strip_run_in_one_wave(K, M):
    """34 to 37 strips by four CTAs each are no more CTAs than the GPU has SMs, but not all of their clusters run at once: two waves took 1.3 to
    1.6 times what the next larger layers took, which two CTAs each share."""
    def us(strips):
        N = 32 * strips
        d = [synth.make_layer(4, K, N, 128, False, seed=i, device=DEV) for i in range(4)]
        plans = [ops.GemvPlan(l.qweight, l.qzeros, l.scales, None, None, None, M, 4, 128, None, 0) for l in d]
        x = synth.make_x(M, K, device=DEV)
        [p.run(x) for p in plans]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for i in range(40):
                plans[i % 4].run(x)
        times = []
        for _ in range(20):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record(); graph.replay(); ev[1].record()
            torch.cuda.synchronize()
            times.append(ev[0].elapsed_time(ev[1]))
        return min(times)
    assert max(us(n) for n in (34, 35, 36, 37)) < 1.15 * us(38)


@pytest.mark.parametrize("K,N,gs,gather", [
    (2080, 32, 32, False), (2208, 96, 96, True), (3104, 2048, 64, False), (11008, 4096, 32, True),      # one strip per CTA, the shortest K; cut units
    (2048, 4096, 32, True),                                                                              # a little less: fp16
    (928, 9632, 32, False), (1024, 4832, 64, True), (1056, 14432, 96, False), (2144, 19008, 32, True),   # more strips; seven units: fp16
    (8192, 1024, 32, False), (7968, 1536, 64, True),                                                     # in clusters
])
def test_two_groups_to_a_product_vs_64_bits(K, N, gs, gather):
    """One row, 4 bits, groups scaled apart: within the rounding of the result and what fixed point per 32 rows and fp32 sums may be off by,
    where neighbouring groups differ by up to 2^23 in x and the scales make up for it (so that no group counts less than another, and
    one that met the other's scale, zero-point or factor would show)."""
    layer = synth.make_layer(4, K, N, gs, False, seed=K + N)
    G = layer.scales.shape[0]
    mag = 2.0 ** torch.tensor([[-10, 13, -9, 4, 0, -8, 7][g % 7] for g in range(G)], dtype=torch.float64)
    gen = torch.Generator().manual_seed(6)
    layer.scales = ((1 + torch.rand((G, N), generator=gen)) / mag[:, None]).half()
    xs = (torch.randn((1, K), generator=gen).double() * mag[layer.g_idx.long()]).clamp(-60000, 60000).half()
    perm = torch.randperm(K, generator=gen).to(torch.int32) if gather else None
    x = xs.clone()
    if gather:
        x[:, perm.long()] = xs                              # row k of the layer multiplies x[perm[k]]
    q, z, _ = O.dequantize(layer.qweight.numpy(), layer.qzeros.numpy(), layer.scales.numpy(), layer.g_idx.numpy(), 4)
    g = layer.g_idx.numpy().astype(np.int64)
    s, q, z = layer.scales.numpy().astype(np.float64)[g], q.astype(np.float64), z.astype(np.float64)[g]
    d = layer.to(DEV)
    plan = ops.GemvPlan(d.qweight, d.qzeros, d.scales, None, None if perm is None else perm.to(DEV), None, 1, 4, gs, None, 0)
    y = plan.run(x.to(DEV))
    assert torch.equal(y, plan.run(x.to(DEV)))
    ops.check_status(DEV)
    x64 = xs.numpy().astype(np.float64)
    ref = x64 @ (s * (q - z))
    bound = _bound_of_planes(4, x64, s * (q - z), s * (q + z), 32) + 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    err = np.abs(y.cpu().numpy().astype(np.float64) - ref)
    assert np.all(err <= bound), (err / bound).max()
