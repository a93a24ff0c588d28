"""The linear kernel that keeps a projection.s weights waiting in shared memory (up to eight rows) against the CPU oracle: one row and
eight, remainders of K (blocks of 128 bytes) and of N (16 channels a tile), one warp and sixteen along K.
The standalone entry point runs it when use_tensor_cores is 3."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_parity import gpu_linear, linear_case_inputs, oracle_linear

pytestmark = pytest.mark.gpu

CASES = [(1536, 2048, m) for m in (1, 2, 7, 8)] + [
    (16, 1, 1), (48, 77, 3), (64, 16, 8), (80, 17, 5), (144, 129, 7), (1040, 33, 8),
    (896, 1152, 1), (896, 9728, 8), (4864, 896, 1), (4864, 896, 8),
    (1536, 17920, 1), (1536, 17920, 5), (1536, 17920, 8), (8960, 1536, 1), (8960, 1536, 8), (11008, 2048, 2), (11008, 100, 2),
]


@pytest.mark.parametrize("K,N,M", CASES)
def test_layer_with_its_weights_waiting_matches_the_oracle(gpu_lib, K, N, M):
    x, w, fold, in_scales = linear_case_inputs(K, N, M)
    site = (1090717716, -44)
    want = oracle_linear(x, w, fold, in_scales, site)
    f = gpu_lib.dll.sslm_b200_tc_variant_counts
    f.argtypes = [C.c_void_p, C.c_int32]
    counts = np.zeros((2, 6), dtype=np.uint64)
    assert f(counts[0].ctypes.data, 6) == 0
    got = gpu_linear(gpu_lib, x, w, fold, in_scales, site, 3)
    assert f(counts[1].ctypes.data, 6) == 0
    assert list(counts[1] - counts[0]) == [0, 0, 0, 0, 0, 1]
    for a, b, what in zip(got, want, ("folded", "codes", "scales", "status")):
        assert (np.asarray(a, dtype=np.int64) == np.asarray(b, dtype=np.int64)).all(), what


def test_request_that_never_comes(gpu_lib):
    """one box of weights is not asked for: its wait runs out, every row says so, and the next call is right"""
    K, N, M = 1536, 300, 3
    x, w, fold, in_scales = linear_case_inputs(K, N, M)
    site = (1090717716, -44)
    arm = gpu_lib.dll.sslm_b200_debug_withhold_tc_load
    arm.argtypes = [C.c_int32]
    assert arm(1) == 0
    try:
        got = gpu_linear(gpu_lib, x, w, fold, in_scales, site, 3)
    finally:
        arm(0)
    assert (got[3] == 100).all()
    want, got = oracle_linear(x, w, fold, in_scales, site), gpu_linear(gpu_lib, x, w, fold, in_scales, site, 3)
    for a, b in zip(got, want):
        assert (np.asarray(a, dtype=np.int64) == np.asarray(b, dtype=np.int64)).all()


def test_its_launches_are_in_the_process_wide_count(gpu_lib):
    from tests.test_gpu_parity import tc_launches
    x, w, fold, in_scales = linear_case_inputs(144, 129, 7)
    before = tc_launches(gpu_lib)
    gpu_linear(gpu_lib, x, w, fold, in_scales, (1090717716, -44), 3)
    assert tc_launches(gpu_lib) - before == 1
