"""The shared library loads on a machine without a GPU and exports every symbol that
include/b200gptq.h declares (no kernel is launched here)."""
import ctypes
import os
import re

from conftest import ROOT


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "b200gptq.h")).read()
    return sorted(set(re.findall(r"B200GPTQ_API\s+[\w\s\*]+?\b(b200gptq_\w+)\s*\(", text)))


def test_header_declares_the_expected_entry_points():
    names = _declared_symbols()
    for must in ("b200gptq_gemv", "b200gptq_gemm", "b200gptq_dequant", "b200gptq_sort_rows",
                 "b200gptq_workspace_bytes", "b200gptq_strerror"):
        assert must in names


def test_library_exports_every_declared_symbol():
    from autogptq.tvm_b200 import build
    path = build.build()  # no-op when the library is newer than its sources
    lib = ctypes.CDLL(path)
    for name in _declared_symbols():
        assert hasattr(lib, name), f"{name} is declared in the header but not exported"


def test_status_strings_and_host_side_queries():
    from autogptq.tvm_b200 import _lib
    lib = _lib.lib
    assert lib.b200gptq_abi_version() >= 1
    assert lib.b200gptq_strerror(0) == b"ok"
    for code in range(-8, 0):
        assert lib.b200gptq_strerror(code) not in (b"", b"unknown status")
    assert lib.b200gptq_strerror(-99) == b"unknown status"
    # argument validation happens on the host before anything touches the device
    assert lib.b200gptq_gemv(None, None, None, None, None, None, None, None, 1, 4096, 4096, 4, 128, None, 0, None) == -1
    assert lib.b200gptq_dequant(None, None, None, None, 4096, 4096, 4, 128, None, None, None) == -1


def test_quantlinear_refuses_cpu_tensors_and_bad_bits():
    import pytest
    import torch
    from autogptq.tvm_b200 import QuantLinear
    with pytest.raises(NotImplementedError):
        QuantLinear(5, 128, 256, 64, False)
    with pytest.raises(ValueError):
        QuantLinear(4, 128, 100, 64, False)
    layer = QuantLinear(4, 128, 256, 64, True)
    assert layer.qweight.shape == (32, 64) and layer.qzeros.shape == (2, 8) and layer.scales.shape == (2, 64)
    assert layer.g_idx.tolist()[:3] == [0, 0, 0] and int(layer.g_idx[-1]) == 1
    with pytest.raises(RuntimeError):
        layer(torch.zeros(1, 256))


def test_a_prepared_module_can_be_copied_and_saved():
    """The native call object and the plans stay behind (they hold addresses); everything else travels."""
    import copy
    import io
    import torch
    from autogptq.tvm_b200 import QuantLinear, _lib
    m = QuantLinear(4, 128, 256, 64, True)
    m.bias.normal_()
    m._native = _lib._host.Layer(256, 64, 4, 128, 0, m.__dict__, True, 16, m.qweight, None, None)
    m._native_state, m._native_tuning = m._constants(), None
    m._plans = {(1, None, 0): (ctypes.c_void_p(1), m._constants())}
    m._ready_for = m._stored()
    f = io.BytesIO()
    torch.save(m, f)
    f.seek(0)
    for c in (copy.deepcopy(m), torch.load(f, weights_only=False)):
        assert c._native is None and c._plans == {} and not c._ready()
        assert torch.equal(c.bias, m.bias) and torch.equal(c.g_idx, m.g_idx) and c.groupsize == 128
    assert m._native is not None and m._ready()


def test_attention_refuses_caches_that_are_not_aligned():
    """Keys and values are read 16 bytes at a time; the check comes before anything is launched (the addresses are made up)."""
    from autogptq.tvm_b200 import _lib
    a, off = 0x100000, 0x100008
    for k, v in ((off, a), (a, off)):
        for hd in (64, 128):
            assert _lib.lib.b200gptq_attn_decode(a, k, v, a, a, 1, 8, hd, 256, 1.0, None) == -4
            assert _lib.lib.b200gptq_attn_step(a, a, a, a, k, v, a, 1, 8, hd, 256, 1, 1.0, None) == -4
