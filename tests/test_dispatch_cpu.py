"""Host-side dispatch of QuantLinear.forward (no GPU): which entry point a given number of rows
reaches.  The reference dispatches on M in TVMHandler.__call__ (tvm_untils/pycuda_warpper.py:138-189:
m == 1 -> GEMV kernel, otherwise the padded GEMM buckets); here up to 16 rows (8 where groups cut 32-row blocks or a
g_idx is kept) go to the GEMV, more rows to the tensor-core GEMM for every bit width, or, where it does not take the layout, to
GEMV passes of 8 rows and from 65 rows on to one dequantisation and a dense product."""
import pytest
import torch

from autogptq.tvm_b200 import qlinear as ql


class _FakeCuda(torch.Tensor):
    """A CPU tensor that claims to live on a GPU, so that forward() gets as far as its dispatch."""
    is_cuda = property(lambda self: True)


def _layer(bits, groupsize=128, g_idx=None):
    m = ql.QuantLinear(bits, groupsize, 256, 64, False)
    m._ready = lambda: True
    m._qweight_run, m._g_idx_run, m._x_perm = m.qweight, g_idx, None
    uniform = g_idx is None or bool((g_idx.view(-1, 32) == g_idx.view(-1, 32)[:, :1]).all())
    m._settled = m._constants()
    m._gemm_ok, m._gemv_rows = ql.row_rules(256, m.groupsize, g_idx is not None, uniform)      # as post_init() has it
    return m


BLOCKS = (torch.arange(256) // 32 * 3 % 8).to(torch.int32)      # one group per 32-row block, not k // group_size
CUT = (torch.arange(256) // 16 * 3 % 16).to(torch.int32)        # groups that cut the blocks


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("groupsize,g_idx,M,want", [
    (128, None, 1, ["plan:1"]), (128, None, 8, ["plan:8"]), (128, None, 9, ["plan:9"]), (128, None, 16, ["plan:16"]),
    (128, None, 17, ["gemm:17"]), (128, None, 2048, ["gemm:2048"]),
    (32, None, 16, ["plan:16"]), (32, None, 17, ["gemm:17"]), (-1, None, 16, ["plan:16"]), (-1, None, 17, ["gemm:17"]),
    # a stored g_idx: the general kernel up to 8 rows, the tensor-core kernel with one group per block
    (32, BLOCKS, 8, ["plan:8"]), (32, BLOCKS, 9, ["gemm:9"]), (32, BLOCKS, 65, ["gemm:65"]),
    # groups that cut through 32-row blocks cannot use it
    (16, None, 8, ["plan:8"]), (16, None, 9, ["gemv:8", "gemv:1"]), (16, None, 16, ["gemv:8", "gemv:8"]),
    (16, None, 64, ["gemv:8"] * 8), (16, None, 65, ["dequantize"]), (16, CUT, 20, ["gemv:8", "gemv:8", "gemv:4"]), (16, CUT, 65, ["dequantize"]),
])
def test_rows_decide_the_entry_point(monkeypatch, bits, groupsize, g_idx, M, want):
    calls = []

    def fake(name):
        def f(x, *args, out=None, **kw):
            calls.append(f"{name}:{x.shape[0]}")
            return out if out is not None else torch.zeros((x.shape[0], 64), dtype=torch.float16)
        return f

    def fake_dequantize(*args, **kw):
        calls.append("dequantize")
        return None, torch.zeros((256, 64), dtype=torch.float16)

    class FakePlan:   # up to 16 rows go through a prepared launch (ops.GemvPlan)
        def __init__(self, *a, **k):
            pass

        def run(self, x, out=None):
            return fake("plan")(x, out=out)

    monkeypatch.setattr(ql.ops, "GemvPlan", FakePlan)
    monkeypatch.setattr(ql.ops, "gemv", fake("gemv"))
    monkeypatch.setattr(ql.ops, "gemm", fake("gemm"))
    monkeypatch.setattr(ql.ops, "dequantize", fake_dequantize)
    monkeypatch.setattr(torch.cuda, "device", lambda d: __import__("contextlib").nullcontext())
    monkeypatch.setattr(torch, "empty", lambda *a, device=None, **k: torch.zeros(*a, **k))
    x = torch.zeros((M, 256), dtype=torch.float16).as_subclass(_FakeCuda)
    y = _layer(bits, groupsize, g_idx).forward(x)
    assert calls == want
    assert tuple(y.shape) == (M, 64)


def test_decode_positions_are_checked_on_the_host():
    from autogptq.tvm_b200.decoder import check_positions
    check_positions(512, 256, 768)
    with pytest.raises(ValueError):
        check_positions(512, 257, 768)
    with pytest.raises(ValueError):
        check_positions(-1, 1, 768)


def test_registered_operator_has_a_shape_rule():
    """torch.ops.b200gptq.quant_matmul is registered with a fake (meta) implementation: tracing tools can infer the
    output of a QuantLinear without running it (the reference module is not traceable at all: it calls pycuda)."""
    import torch
    from autogptq.tvm_b200 import torch_ops  # noqa: F401  (registers the operator)
    op = torch.ops.b200gptq.quant_matmul
    K, N, bits = 256, 96, 4
    x = torch.empty((5, K), dtype=torch.float16, device="meta")
    qweight = torch.empty((K // 32 * bits, N), dtype=torch.int32, device="meta")
    qzeros = torch.empty((2, N // 32 * bits), dtype=torch.int32, device="meta")
    scales = torch.empty((2, N), dtype=torch.float16, device="meta")
    y = op(x, qweight, qzeros, scales, None, None, None, bits, 128, True)
    assert y.shape == (5, N) and y.dtype == torch.float16 and y.device.type == "meta"
    import pytest
    with pytest.raises(Exception):
        op(torch.empty((5, K + 32), dtype=torch.float16, device="meta"), qweight, qzeros, scales, None, None, None,
           bits, 128, True)


def test_gemm_work_split_rule():
    """b200gptq_gemm_split is host-only (without a device it plans for 148 SMs): K is split for up to 128 rows
    while every run keeps 16 k-tiles (40 above 96 rows; from 65 rows on into no fewer than three), above that where it saves unpacking
    the weights for another tile of rows; more than 16 rows, and 2 and
    8 bits, run on pairs of SMs, one CTA each; the second CTA per SM comes only below that and only where it shortens waves x
    k-tiles."""
    from autogptq.tvm_b200 import ops
    assert ops.gemm_split(16, 4096, 4096, 4) == (4, 1)        # 32 column tiles on 148 SMs: four runs of 16 k-tiles
    assert ops.gemm_split(128, 4096, 4096, 4) == (1, 1)       # 16 k-tiles per run would be too few above 96 rows
    assert ops.gemm_split(96, 4096, 4096, 4) == (4, 1)        # 16 pairs of column tiles on 74 pairs of SMs: four runs
    assert ops.gemm_split(96, 2048, 4096, 4) == (1, 1)        # two runs would be too few above 64 rows
    assert ops.gemm_split(128, 11008, 4096, 4) == (4, 1)      # 172 k-tiles: four runs of 43
    assert ops.gemm_split(16, 4096, 12288, 4) == (3, 2)       # 96 tiles: three runs, two CTAs per SM
    assert ops.gemm_split(64, 9216, 27648, 3) == (1, 1)       # 108 pairs of column tiles: never two CTAs of a pair kernel per SM
    assert ops.gemm_split(16, 9216, 27648, 3) == (1, 2)       # 216 tiles: one wave of two per SM instead of two waves
    assert ops.gemm_split(16, 4096, 12288, 8)[1] == 1         # 8 bits: pairs at any number of rows
    assert ops.gemm_split(16, 9216, 9216, 3)[0] > 1
    assert ops.gemm_split(256, 4096, 4096, 4) == (1, 1)       # more than one row tile: split where pairs of SMs stand idle
    assert ops.gemm_split(256, 11008, 4096, 4) == (2, 1)
    assert ops.gemm_split(129, 8192, 2048, 4) == (4, 1)
    assert ops.gemm_split(2048, 4096, 12288, 4) == (1, 1)
    with pytest.raises(ValueError):
        ops.gemm_split(16, 4095, 4096, 4)


def test_runs_of_a_long_prompt_fit_their_pairs_and_their_scratch():
    """Above 128 rows a split product has a tile per pair of SMs (the kernel's sum over runs takes one), runs of eight units of 128 rows or
    more, and room for the sums of every run in the scratch; without runs only the counters and a copy of x are asked for."""
    from autogptq.tvm_b200 import _lib, ops
    split = 0
    for K in (1024, 2048, 2080, 4096, 8192, 11008):
        for N in (32, 1024, 2048, 4096, 6176, 12288):
            for M in (129, 160, 200, 256, 257, 300, 448, 512, 700, 1024, 2048):
                runs, per_sm = ops.gemm_split(M, K, N, 4)
                base = 16384 + -(-2 * M * K // 256) * 256
                extra = _lib.workspace_bytes(_lib.OP_GEMM, M, K, N, 4) - base
                assert per_sm == 1 and 1 <= runs <= 4
                if runs == 1:
                    assert extra == 0
                    continue
                split += 1
                rows = extra // (runs * N * 4)             # padded to whole tiles
                assert extra == runs * rows * N * 4 and M <= rows < M + 256 and rows % 32 == 0
                assert -(-K // 128) // runs >= 8
                # the fewest tiles that so many padded rows can be (256 rows each) fit, with all their runs
                assert -(-N // 256) * -(-rows // 256) * runs <= 74
    assert split > 20
