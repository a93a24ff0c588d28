"""The weights-first tensor-core linear kernel (up to 256 rows) against the CPU oracle: every padded row
count and its edges, ragged channel counts, short and long K, K cut over clusters and not, and which of the two
tensor-core kernels each case ran on. The standalone entry points run it when use_tensor_cores is 2."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_parity import cpu_gemm, gpu_linear, linear_case_inputs, oracle_linear, tc_launches

pytestmark = pytest.mark.gpu

CASES = [(1536, 2048, m) for m in (1, 2, 16, 17, 32, 33, 64, 65, 128, 129, 256)] + [
    (16, 1, 1), (48, 77, 7), (128, 128, 9), (144, 129, 31), (256, 300, 20), (896, 9728, 21), (4864, 896, 5),      # remainders of K and N
    (8960, 1536, 3), (8960, 1536, 200), (1536, 17920, 45), (1536, 17920, 130), (2048, 4000, 100), (11008, 2048, 1),
] + [(k, n, m) for k, n in ((1536, 1536), (8960, 1536), (1536, 17920)) for m in (65, 100, 128)]      # 128 padded rows, clustered and not


def runs_weights_first(K, N, M, sms=148):
    """the kernel's rule: where K would be cut over a cluster, only up to 64 rows, or 128 with up to 14 tiles"""
    tiles, kblocks, splits = -(-N // 128), -(-K // 128), 1
    while splits < 8 and tiles * splits * 2 <= sms and splits * 2 <= kblocks:
        splits *= 2
    return splits == 1 or M <= 64 or (M <= 128 and tiles <= 14)


def variants(lib):
    f = lib.dll.sslm_b200_tc_variant_counts
    f.argtypes = [C.c_void_p, C.c_int32]
    counts = np.zeros(5, dtype=np.uint64)
    assert f(counts.ctypes.data, 5) == 0
    return counts.astype(np.int64)


@pytest.mark.parametrize("K,N,M", CASES)
def test_weights_first_layer_matches_the_oracle(gpu_lib, K, N, M):
    x, w, fold, in_scales = linear_case_inputs(K, N, M)
    site = (1090717716, -44)
    want = oracle_linear(x, w, fold, in_scales, site)
    before, kinds = tc_launches(gpu_lib), variants(gpu_lib)
    got = gpu_linear(gpu_lib, x, w, fold, in_scales, site, 2)
    assert tc_launches(gpu_lib) - before == 1
    ran = variants(gpu_lib) - kinds
    assert ran.sum() == 1 and (ran[4] == 1) == runs_weights_first(K, N, M)
    for a, b, what in zip(got, want, ("folded", "codes", "scales", "status")):
        assert (np.asarray(a, dtype=np.int64) == np.asarray(b, dtype=np.int64)).all(), what


@pytest.mark.parametrize("N,M", [(1000, 1), (4097, 8), (40000, 40), (300, 256)])
def test_weights_first_head_keeps_the_lowest_index(gpu_lib, N, M):
    K = 256
    rng = np.random.default_rng(N + M)
    x = rng.integers(-127, 128, (M, K)).astype(np.int8)
    w = rng.integers(-127, 128, (N, K)).astype(np.int8)
    w[N - 1] = w[5] = np.where(x[0] >= 0, 127, -127)      # row 0's maximum, twice: channel 5 wins
    f = gpu_lib.dll.sslm_b200_logits
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_int32, C.c_int32, C.c_int32, C.c_void_p, C.c_void_p]
    rows, toks = np.zeros((M, N), dtype=np.int32), np.zeros(M, dtype=np.int32)
    only = np.zeros(M, dtype=np.int32)
    assert f(x.ctypes.data, w.ctypes.data, M, N, K, 2, rows.ctypes.data, toks.ctypes.data) == 0
    assert f(x.ctypes.data, w.ctypes.data, M, N, K, 2, None, only.ctypes.data) == 0
    acc = np.asarray(cpu_gemm(x, w)).astype(np.int64)
    assert (rows == acc).all()
    assert (toks == np.argmax(acc, axis=1)).all() and (only == toks).all() and toks[0] == 5
