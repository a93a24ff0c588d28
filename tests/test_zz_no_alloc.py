"""sslm_b200_linear_resident: the linear layer on device-resident operands with its scratch in
a fixed device array. Checked against sslm_b200_linear (the existing entry point, which stages
host buffers and allocates) on two calls in a row, so that a scratch slot left non-zero by the
first call would show in the second. Named to be collected last; passes alone too."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SITE = (1090717716, -44)


def reference_entry(lib, x, w, fold, in_scales):
    f = lib.dll.sslm_b200_linear
    f.argtypes = [C.c_void_p] * 3 + [C.c_int32] * 3 + [C.c_void_p, C.c_int64, C.c_int64, C.c_int32] + [C.c_void_p] * 4
    M, K = x.shape
    N = w.shape[0]
    folded = np.zeros((M, N), dtype=np.int32)
    codes = np.zeros((M, N), dtype=np.int8)
    scales = np.zeros((M, 2), dtype=np.int64)
    status = np.zeros(M, dtype=np.int32)
    assert f(x.ctypes.data, w.ctypes.data, fold.ctypes.data, M, N, K, in_scales.ctypes.data, SITE[0], SITE[1], 0,
             folded.ctypes.data, codes.ctypes.data, scales.ctypes.data, status.ctypes.data) == 0
    return folded, codes, scales, status


def resident_entry(lib, torch, x, w, fold, in_scales):
    f = lib.dll.sslm_b200_linear_resident
    f.restype = C.c_int32
    f.argtypes = [C.c_void_p] * 3 + [C.c_int32] * 3 + [C.c_void_p, C.c_int64, C.c_int64] + [C.c_void_p] * 5
    M, K = x.shape
    N = w.shape[0]
    dev = torch.device("cuda:0")
    dx, dw = torch.from_numpy(x).to(dev), torch.from_numpy(w).to(dev)
    dfold, dsc = torch.from_numpy(fold).to(dev), torch.from_numpy(in_scales).to(dev)
    # outputs pre-filled with junk: the entry must write every element it reports
    folded = torch.full((M, N), 0x5A5A5A5A, dtype=torch.int32, device=dev)
    codes = torch.full((M, N), 0x5A, dtype=torch.int8, device=dev)
    scales = torch.full((M, 2), -1, dtype=torch.int64, device=dev)
    status = torch.full((M,), 77, dtype=torch.int32, device=dev)
    torch.cuda.synchronize()
    st = f(dx.data_ptr(), dw.data_ptr(), dfold.data_ptr(), M, N, K, dsc.data_ptr(), SITE[0], SITE[1],
           folded.data_ptr(), codes.data_ptr(), scales.data_ptr(), status.data_ptr(), None)
    assert st == 0
    torch.cuda.synchronize()
    return folded.cpu().numpy(), codes.cpu().numpy(), scales.cpu().numpy(), status.cpu().numpy()


def make_case(seed, M, N, K, amplitude):
    rng = np.random.default_rng(seed)
    x = rng.integers(-amplitude, amplitude + 1, (M, K)).astype(np.int8)
    w = rng.integers(-127, 128, (N, K)).astype(np.int8)
    fold = np.zeros((N, 3), dtype=np.int32)
    fold[:, 1] = rng.integers(1 << 30, 1 << 31, N)
    fold[:, 2] = rng.integers(8, 21, N)
    fold[::5, 0] = 1
    in_scales = np.stack([rng.integers(1 << 30, 1 << 31, M), np.full(M, -37)], axis=1).astype(np.int64)
    return x, w, fold, in_scales


def test_resident_linear_matches_the_allocating_entry_twice_in_a_row(gpu_lib):
    torch = pytest.importorskip("torch")
    assert torch.cuda.is_available()
    torch.cuda.set_device(0)
    # the second call has fewer rows and much smaller magnitudes than the first: a row peak
    # surviving from call one would change its scales and codes
    for seed, (M, N, K, amp) in enumerate([(37, 777, 1536, 127), (21, 300, 512, 3)]):
        x, w, fold, in_scales = make_case(seed, M, N, K, amp)
        want = reference_entry(gpu_lib, x, w, fold, in_scales)
        got = resident_entry(gpu_lib, torch, x, w, fold, in_scales)
        for a, b, what in zip(got, want, ("folded", "codes", "scales", "status")):
            assert (a == b).all(), (what, seed)
        # (the other entry point runs the streaming kernel here; both are held to the CPU oracle)
        from tests.test_gpu_parity import oracle_linear
        cpu = oracle_linear(x, w, fold, in_scales, SITE)
        for a, b, what in zip(got, cpu, ("folded", "codes", "scales", "status")):
            assert (np.asarray(a, dtype=np.int64) == np.asarray(b, dtype=np.int64)).all(), ("oracle", what, seed)


def test_resident_linear_refuses_more_rows_than_its_scratch_holds(gpu_lib):
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    f = gpu_lib.dll.sslm_b200_linear_resident
    f.restype = C.c_int32
    f.argtypes = [C.c_void_p] * 3 + [C.c_int32] * 3 + [C.c_void_p, C.c_int64, C.c_int64] + [C.c_void_p] * 5
    buf = torch.zeros(1 << 16, dtype=torch.int32, device="cuda:0")
    p = buf.data_ptr()
    assert f(p, p, p, 257, 16, 16, p, SITE[0], SITE[1], p, None, None, None, None) == 1     # SSLM_INVALID_ARGUMENT
    assert f(p, p, p, 4, 16, 16400, p, SITE[0], SITE[1], p, None, None, None, None) == 1
    torch.cuda.synchronize()


def check_resident(lib, torch, seed, M, N, K):
    from tests.test_gpu_parity import oracle_linear
    x, w, fold, in_scales = make_case(seed, M, N, K, 127)
    got, want = resident_entry(lib, torch, x, w, fold, in_scales), oracle_linear(x, w, fold, in_scales, SITE)
    for a, b, what in zip(got, want, ("folded", "codes", "scales", "status")):
        assert (np.asarray(a, dtype=np.int64) == np.asarray(b, dtype=np.int64)).all(), what


@pytest.mark.parametrize("M,N,K", [(1, 300, 512), (2, 2048, 1536), (8, 1152, 896), (16, 77, 48), (17, 1536, 4864), (33, 900, 896),
                                   (64, 1536, 1536), (65, 1536, 1536), (128, 1536, 1536), (100, 4000, 1536), (129, 2048, 1536),
                                   (130, 17920, 256), (256, 2048, 896), (256, 9728, 896)])
def test_resident_linear_on_every_kernel(gpu_lib, M, N, K):
    """one row (streaming), each row padding of the weights-first kernel, clustered and not, and the activation-major one"""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    check_resident(gpu_lib, torch, M, M, N, K)


@pytest.mark.parametrize("M,N,K,given_up", [(40, 1536, 1536, 40), (40, 20000, 256, 40), (200, 2048, 1536, 128)])
def test_resident_linear_reports_a_wait_that_ran_out(gpu_lib, M, N, K, given_up):
    """the weights-first kernel, clustered and not, and the activation-major one (rows of the abandoned tile); there is
    no status array for the projection to write, so it travels as the row maximum"""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    arm = gpu_lib.dll.sslm_b200_debug_withhold_tc_load
    arm.argtypes = [C.c_int32]
    x, w, fold, in_scales = make_case(5, M, N, K, 127)
    assert arm(1) == 0
    try:
        status = resident_entry(gpu_lib, torch, x, w, fold, in_scales)[3]
    finally:
        arm(0)
    assert (status[:given_up] == 100).all() and (status[given_up:] == 0).all()
    check_resident(gpu_lib, torch, 6, M, N, K)      # nothing of it is left in the fixed array


@pytest.mark.parametrize("K,N,M,kind", [(896, 9728, 5, 4), (1536, 4096, 2, 4), (1024, 9728, 3, 4), (1280, 6144, 8, 5), (1280, 6128, 3, 4),
                                        (2048, 9728, 2, 5), (1536, 17920, 8, 5), (11008, 2048, 2, 5), (896, 1152, 8, 5)])
def test_which_kernel_serves_a_few_rows(gpu_lib, K, N, M, kind):
    """weights waiting in shared memory (5) where its blocks have a multiprocessor each or the projection is large, else weights
    first (4): kinds as sslm_b200_tc_variant_counts orders them"""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    from tests.test_gpu_parity import oracle_linear
    f = gpu_lib.dll.sslm_b200_tc_variant_counts
    f.argtypes = [C.c_void_p, C.c_int32]
    counts = np.zeros((2, 6), dtype=np.uint64)
    x, w, fold, in_scales = make_case(K + N + M, M, N, K, 127)
    assert f(counts[0].ctypes.data, 6) == 0
    got = resident_entry(gpu_lib, torch, x, w, fold, in_scales)
    assert f(counts[1].ctypes.data, 6) == 0
    assert list(counts[1] - counts[0]) == [int(i == kind) for i in range(6)]
    for a, b, what in zip(got, oracle_linear(x, w, fold, in_scales, SITE), ("folded", "codes", "scales", "status")):
        assert (np.asarray(a, dtype=np.int64) == np.asarray(b, dtype=np.int64)).all(), what
