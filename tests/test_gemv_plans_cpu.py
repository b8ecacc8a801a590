"""Every product that the decode GEMV says it takes gets a plan (no GPU: a plan is chosen on the host, and what would need
the device comes after the choice).  The limits of shared memory are met at long K, where x of a CTA grows with it."""
import ctypes

import pytest

from autogptq.tvm_b200 import _lib

TOO_LARGE = -8
ADDRESS = 0x100000      # aligned; nothing on the host reads it


def _create(M, K, N, bits, group, perm, ctas, act):
    plan = ctypes.c_void_p(0)
    st = _lib.lib.b200gptq_gemv_plan_create_ex(ctypes.byref(plan), ADDRESS, ADDRESS, ADDRESS, None,
                                               ADDRESS if perm else None, None, M, K, N, bits, group, 0, ctas, act)
    if plan:
        _lib.lib.b200gptq_gemv_plan_destroy(plan)
    return st


def test_the_status_this_file_looks_for():
    assert b"exceeds a fixed capacity" in _lib.lib.b200gptq_strerror(TOO_LARGE)


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("group", [32, 96, 128, -1])
def test_every_long_row_has_a_plan(bits, group):
    """One row: all K up to 10 000, then every seventh 32-row block up to 140 000 and the lengths around which x stops
    fitting; with a gather and without; eight warps, sixteen and the default."""
    lengths = list(range(32, 10000, 32)) + list(range(10016, 140000, 7 * 32)) + [40960, 49152, 53248, 57344, 65536, 65568]
    for K in lengths:
        for N in (32, 8192):
            for perm in (False, True):
                for ctas in (0, 1, 2) if K > 10000 else (0,):
                    assert _create(1, K, N, bits, group, perm, ctas, 0) != TOO_LARGE, (K, N, perm, ctas)


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("M", [2, 3, 8, 9, 16])
def test_every_batch_has_a_plan(bits, M):
    for K in list(range(32, 4096, 32)) + list(range(4096, 140000, 13 * 32)):
        for N in (32, 5120, 36864):
            for group in (32, 128):
                assert _create(M, K, N, bits, group, K % 64 == 0, 0, 0) != TOO_LARGE, (K, N, group)


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("act", [_lib.ACT_SWIGLU, _lib.ACT_RELU])
def test_every_folded_activation_has_a_plan(bits, act):
    for M in (1, 2, 8):
        for K in list(range(128, 20000, 1280)) + list(range(20480, 140000, 2560)):
            assert _create(M, K, 8192, bits, 128, False, 0, act) != TOO_LARGE, (M, K)


def test_the_query_for_folding_and_the_library_agree():
    """ops.can_fold_act says what b200gptq_gemv_plan_create_ex refuses (with the shape's status) and what it does not."""
    from autogptq.tvm_b200 import ops
    refused = 0
    for M in (1, 3, 8):
        for K in (128, 96, 256, 4096, 4128):
            for bits in (2, 3, 4, 8):
                for group in (32, 64, 128, 256, -1):
                    for perm in (False, True):
                        for act in (_lib.ACT_SWIGLU, _lib.ACT_RELU):
                            folds = ops.can_fold_act(M, K, 96, bits, group, False, perm, act)
                            assert (_create(M, K, 96, bits, group, perm, 0, act) != -3) == folds, (M, K, bits, group, perm, act)
                            refused += not folds
    assert refused


def test_the_path_query_names_the_kernel():
    for bits in (2, 3, 4, 8):
        for K, group, streams in ((256, 32, True), (256, 64, True), (256, 128, True), (256, -1, True), (96, -1, True), (256, 16, False),
                                  (288, 48, False)):
            want = _lib.PATH_STREAM if streams else _lib.PATH_GENERIC
            assert _lib.gemv_path(1, K, 96, bits, group, False) == want
            assert _lib.gemv_path(8, K, 96, bits, group, True) == _lib.PATH_GENERIC
