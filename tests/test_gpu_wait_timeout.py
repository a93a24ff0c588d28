"""A bounded device wait that runs out, made to happen on purpose.

Every mbarrier wait of the kernels has a limit. The tensor-core linear kernel's producer is told
(test-only hook sslm_b200_debug_withhold_tc_load) to arm the barrier of its first weight tile without
requesting the tile; the wait on it gives up after the limit (a second or less), the tile's rows end
with the internal status 100, and the verb that launched the kernel returns SSLM_ALLOCATION_FAILED.
Nothing faults, nothing spins without a limit, the context stays usable, and the same call then
succeeds and gives the oracle's results. The exchanges between the blocks of a cluster likewise: one
block waits for four bytes more than its peers send (sslm_b200_debug_withhold_exchange). (The failure is injected on the host side of the launch:
a request that is never made. No kernel is made to trap or to loop.)
"""
import ctypes as C
import time

import numpy as np
import pytest

import failure_cases as F
from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import gpu_linear, linear_case_inputs, oracle_linear, run_port, tc_launches

pytestmark = pytest.mark.gpu
WAIT_TIMEOUT = 100


def hook(lib):
    f = lib.dll.sslm_b200_debug_withhold_tc_load
    f.argtypes = [C.c_int32]
    return f


def test_standalone_layer_reports_the_rows_of_the_abandoned_tile(gpu_lib):
    K, N, M = 1536, 512, 200
    x, w, fold, in_scales = linear_case_inputs(K, N, M)
    site = (1090717716, -44)
    want = oracle_linear(x, w, fold, in_scales, site)
    arm = hook(gpu_lib)
    assert arm(17) != 0 and arm(1) == 0
    try:
        before = tc_launches(gpu_lib)
        got = gpu_linear(gpu_lib, x, w, fold, in_scales, site, 1)
        assert tc_launches(gpu_lib) - before == 1
    finally:
        arm(0)
    # block 0's first tile starts at row 0: its 128 rows carry the internal status, the others finished
    assert (got[3][:128] == WAIT_TIMEOUT).all()
    assert (got[3][128:] == want[3][128:]).all()
    # the hook is spent: the same call now gives the oracle's rows
    got = gpu_linear(gpu_lib, x, w, fold, in_scales, site, 1)
    for k in range(4):
        assert (np.asarray(got[k]).astype(np.int64) == np.asarray(want[k]).astype(np.int64)).all(), k


def test_prefill_fails_cleanly_and_the_next_call_succeeds(gpu_lib):
    sh = A.SHAPES["mini1.5b"]
    art = A.build_synthetic_model("mini1.5b", 0x7100, 96)
    prompt = A.stream_uniform(0x7100, "prompt", 40, 0, sh.vocab - 1)
    want_toks, ps = run_port(art, prompt, 3)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=64)
    arm = hook(gpu_lib)
    try:
        s = eng.new_seq()
        fresh = F._state_digest(gpu_lib, s.handle, sh, 96)
        toks = np.ascontiguousarray(prompt, dtype=np.int32)
        consumed = C.c_int32(-1)
        assert arm(1) == 0
        before = tc_launches(gpu_lib)
        st = gpu_lib.sslm_prefill(eng.model, s.handle, toks.ctypes.data_as(C.POINTER(C.c_int32)), toks.size, 64, 0, eng.ws,
                                  C.byref(consumed))
        assert tc_launches(gpu_lib) > before                 # the chunk did run on the tensor-core kernel
        assert st == abi.ST["SSLM_ALLOCATION_FAILED"] and consumed.value == 0
        assert F._state_digest(gpu_lib, s.handle, sh, 96) == fresh      # nothing of the chunk was kept
        arm(0)
        assert s.prefill(prompt, 64) == len(prompt)
        assert s.decode(3, sh.layers) == want_toks
        blob = abi.parse_save_blob(s.save(), sh.hidden)
        assert blob["kv"] == ps.kv.tobytes()
    finally:
        arm(0)
        eng.close()


# kernel and exchange, shape, prompt, and the call whose wait runs out: the prefill or the decode step behind it
EXCHANGES = [(0, 0, "mini1.5b", 40, "prefill"), (1, 0, "mini1.5b", 300, "decode"), (1, 1, "mini1.5b", 300, "decode"),
             (1, 2, "mini1.5b", 300, "decode"), (1, 3, "mini1.5b", 300, "decode"),
             (2, 0, "tiny", 700, "prefill"), (2, 1, "tiny", 700, "prefill"), (2, 2, "tiny", 700, "prefill"), (3, 0, "mini1.5b", 40, "decode")]


@pytest.mark.parametrize("kernel,exchange,shape,n,call", EXCHANGES)
def test_exchange_that_runs_out(gpu_lib, kernel, exchange, shape, n, call):
    sh = A.SHAPES[shape]
    art = A.build_synthetic_model(shape, 0x7200 + n, n + 16)
    prompt = A.stream_uniform(0x7200 + n, "prompt", n, 0, sh.vocab - 1)
    want_toks, ps = run_port(art, prompt, 3)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=n)
    arm = gpu_lib.dll.sslm_b200_debug_withhold_exchange
    arm.argtypes = [C.c_int32, C.c_int32]
    assert arm(kernel, 4) == arm(4, 0) == abi.ST["SSLM_INVALID_ARGUMENT"]
    failed = abi.ST["SSLM_ALLOCATION_FAILED"]
    try:
        s = eng.new_seq()
        toks = np.ascontiguousarray(prompt, dtype=np.int32)
        consumed = C.c_int32(-1)
        t = time.perf_counter()
        if call == "prefill":
            assert arm(kernel, exchange) == 0
            assert gpu_lib.sslm_prefill(eng.model, s.handle, toks.ctypes.data_as(C.POINTER(C.c_int32)), n, n, 0, eng.ws,
                                        C.byref(consumed)) == failed
            assert consumed.value == 0
            took = time.perf_counter() - t
        assert s.prefill(prompt, n) == n
        assert s.decode(1, sh.layers) == want_toks[:1]
        if call == "decode":
            assert arm(kernel, exchange) == 0
            t = time.perf_counter()
            assert eng.decode_step([s], sh.layers)[0] == failed
            took = time.perf_counter() - t
        assert 0.2 < took < 5.0      # waits of a quarter of a second: four exchanges and six times that on the way out
        assert s.decode(2, sh.layers) == want_toks[1:]
        assert abi.parse_save_blob(s.save(), sh.hidden)["kv"] == ps.kv.tobytes()
    finally:
        arm(-1, 0)
        eng.close()


# batches whose q/k/v site runs inside the attention cluster: (shape, adapted, bias_bits, prompts, kernel and exchange). Clusters of 16
# blocks (up to six rows), of 8, and of 2; with biases there is a fifth exchange.
SITE = (5, 0)
SITE_EXCHANGES = [("mini1.5b", False, 0, (300, 40), (1, x)) for x in range(4)] + \
                 [("mini0.5b", False, 30, (300, 40, 5), x) for x in ((1, 0), (1, 1), (1, 2), (1, 3), SITE)] + \
                 [("tiny", True, 36, (200, 30), SITE), ("tiny", True, 0, (200, 30), (1, 1)),
                  ("small", False, 36, (70, 5, 30, 64, 1, 20, 9, 16), SITE), ("small", False, 30, (20, 5), SITE),
                  ("small", False, 30, (20, 5), (1, 0))]


@pytest.mark.parametrize("shape,adapted,bias_bits,lengths,exchange", SITE_EXCHANGES)
def test_exchange_of_a_batch_that_runs_out(gpu_lib, shape, adapted, bias_bits, lengths, exchange):
    """Row 0 of a batch gives up inside its cluster in the first layer: the call fails, no sequence moves, and the next calls give
    the oracle's tokens, K/V bytes and saturation counts (the failed call's own landings stay counted, as any refused call's)."""
    sh = A.SHAPES[shape]
    art = A.build_synthetic_model(shape, 0x7280, 320, bias_bits=bias_bits)
    adp = A.build_synthetic_adapter(art, 0x7281, 16, A.PEFT_ORDER) if adapted else None
    eng = abi.Engine(gpu_lib, art, blocks=len(lengths), max_batch=len(lengths), max_chunk=320)

    def holds(s):      # the positions that count, their K/V, where the sequence stands, its saturation count
        b = abi.parse_save_blob(s.save(), sh.hidden)
        kv = np.frombuffer(b["kv"], dtype=np.int8).reshape(sh.layers, 2, sh.kv_heads, 320, sh.head_dim)
        return kv[:, :, :, :b["context_length"]].tobytes(), b["context_length"], b["layer_index"], b["kv_saturation_count"]

    arm = gpu_lib.dll.sslm_b200_debug_withhold_exchange
    arm.argtypes = [C.c_int32, C.c_int32]
    try:
        handle = eng.map_adapter(adp) if adapted else None
        seqs, want = [], []
        for i, n in enumerate(lengths):
            prompt = A.stream_uniform(0x7290 + i, "prompt", n, 0, sh.vocab - 1)
            want.append(run_port(art, prompt, 4, adp))
            s = eng.new_seq()
            if adapted:
                s.set_adapter(handle)
            assert s.prefill(prompt, 320) == n
            seqs.append(s)
        got = [eng.decode_step(seqs, sh.layers)]
        before = [holds(s) for s in seqs]
        assert arm(*exchange) == 0
        t = time.perf_counter()
        assert eng.decode_step(seqs, sh.layers)[0] == abi.ST["SSLM_ALLOCATION_FAILED"]
        assert 0.2 < time.perf_counter() - t < 5.0
        after = [holds(s) for s in seqs]
        assert [a[:3] for a in after] == [b[:3] for b in before] and [a[3] for a in after[1:]] == [b[3] for b in before[1:]]
        again = after[0][3] - before[0][3]
        assert 0 <= again <= 2 * sh.kv_hidden
        got += [eng.decode_step(seqs, sh.layers) for _ in range(3)]
        assert [status for status, _ in got] == [0] * 4
        for i, (s, (tokens, ps)) in enumerate(zip(seqs, want)):
            assert [step[i] for _, step in got] == tokens
            blob = abi.parse_save_blob(s.save(), sh.hidden)
            assert blob["kv"] == ps.kv.tobytes()
            assert blob["kv_saturation_count"] == ps.s.kv_saturation_count + (again if i == 0 else 0)
    finally:
        arm(-1, 0)
        eng.close()


def test_the_next_sequence_finds_the_workspace_clean(gpu_lib):
    """The activation site of a sequence's last layer gives up with the row's gate and up maxima still in place;
    another sequence's row then takes the same place in the workspace, with maxima that may be smaller."""
    sh = A.SHAPES["tiny"]
    art = A.build_synthetic_model("tiny", 0x7300, 64)
    eng = abi.Engine(gpu_lib, art, blocks=2, max_chunk=16)
    arm = gpu_lib.dll.sslm_b200_debug_withhold_exchange
    arm.argtypes = [C.c_int32, C.c_int32]
    try:
        for i in range(6):
            a, b = eng.new_seq(), eng.new_seq()
            for s, salt in ((a, 2 * i), (b, 2 * i + 1)):
                assert s.prefill(A.stream_uniform(0x7300 + salt, "prompt", 9, 0, sh.vocab - 1), 9) == 9
                s.decode(1, sh.layers)
            want, ps = run_port(art, A.stream_uniform(0x7300 + 2 * i + 1, "prompt", 9, 0, sh.vocab - 1), 3)
            assert sh.layers == 2 and eng.decode_step([a], 1) == (0, [-1])
            assert arm(3, 0) == 0
            assert eng.decode_step([a], 1)[0] == abi.ST["SSLM_ALLOCATION_FAILED"]
            assert b.decode(2, sh.layers) == want[1:]
            assert abi.parse_save_blob(b.save(), sh.hidden)["kv"] == ps.kv.tobytes(), i
            a.release()
            b.release()
    finally:
        arm(-1, 0)
        eng.close()
