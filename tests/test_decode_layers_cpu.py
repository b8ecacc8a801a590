"""Which shapes the one-launch decode step takes: decided on the host, before anything is launched."""
import ctypes

import pytest


@pytest.mark.parametrize("change,takes", [
    ({}, True), (dict(batch=2), False), (dict(bits=8), False), (dict(bits=2), True), (dict(hidden=4160, heads=65), False),
    (dict(hidden=4096, heads=128), False), (dict(inter=11040), False), (dict(group_size=64), False), (dict(group_size=256), True),
    (dict(group_size=1 << 20), True), (dict(hidden=6144, heads=48), True), (dict(hidden=6272, heads=49), False),
    (dict(layers=0), False), (dict(max_seq=0), False), (dict(bits=3, inter=128), True)])
def test_shapes(change, takes):
    from autogptq.tvm_b200 import _lib
    base = dict(layers=32, batch=1, hidden=4096, heads=32, inter=11008, max_seq=768, bits=4, group_size=128, gated=1, rms=1, rope=1)
    shape = _lib.StepShape(**dict(base, **change))
    assert (_lib.lib.b200gptq_step_plan_bytes(ctypes.byref(shape)) > 0) == takes


def test_missing_tensors_are_refused():
    from autogptq.tvm_b200 import _lib
    shape = _lib.StepShape(1, 1, 256, 2, 512, 64, 4, 128, 1, 1, 1, 1e-6, 0.1, 256, 256, 256)
    layers, table, plan = (_lib.StepLayer * 1)(), ctypes.create_string_buffer(_lib.lib.b200gptq_step_table_bytes(1)), ctypes.c_void_p()
    assert _lib.lib.b200gptq_step_plan_create(ctypes.byref(shape), layers, table, None) == -1
    assert _lib.lib.b200gptq_step_plan_run(None, None, None, None, None) == -1


@pytest.mark.parametrize("bits,hidden,max_seq,pays", [
    (4, 4096, 768, True), (4, 4096, 4096, True), (4, 4096, 4097, False), (2, 3712, 8192, False), (4, 3584, 8192, True), (4, 4352, 8192, True),
    (4, 4736, 768, True), (4, 4864, 768, False), (2, 6144, 768, False), (3, 6144, 32768, True), (4, 256, 32768, True)])
def test_where_one_launch_pays(bits, hidden, max_seq, pays):
    from autogptq.tvm_b200.decoder import one_launch_pays
    assert one_launch_pays(bits, hidden, max_seq, 148) == pays
