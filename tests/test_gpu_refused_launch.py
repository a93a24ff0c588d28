"""A call whose first kernel the runtime refuses (sslm_b200_debug_refuse_launch): the verb fails, nothing behind the
refused kernel runs, and what the call had prepared on the host -- K/V pages drawn for positions that were then
not written -- does not stand in the way of the calls that follow."""
import ctypes as C

import numpy as np
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu
FAILED = abi.ST["SSLM_ALLOCATION_FAILED"]


@pytest.mark.parametrize("call", ["prefill", "decode", "head"])
def test_calls_after_a_refused_one(gpu_lib, call):
    sh = A.SHAPES["tiny"]
    art = A.build_synthetic_model("tiny", 0x7400, 96)
    prompt = A.stream_uniform(0x7400, "prompt", 10, 0, sh.vocab - 1)
    want, ps = run_port(art, prompt, 60)      # five pages of positions
    eng = abi.Engine(gpu_lib, art, blocks=2, max_chunk=64)
    refuse = gpu_lib.dll.sslm_b200_debug_refuse_launch
    refuse.argtypes = [C.c_int32]
    assert refuse(17) != 0
    try:
        s, other = eng.new_seq(), eng.new_seq()      # (the other's pages lie between)
        assert s.prefill(prompt, 10) == 10 and other.prefill(prompt, 10) == 10
        if call == "prefill":
            more = np.ascontiguousarray(A.stream_uniform(1, "more", 60, 0, sh.vocab - 1), dtype=np.int32)
            consumed = C.c_int32(-1)
            assert refuse(1) == 0
            assert gpu_lib.sslm_prefill(eng.model, s.handle, more.ctypes.data_as(C.POINTER(C.c_int32)), 60, 60, 0, eng.ws,
                                        C.byref(consumed)) == FAILED
            assert consumed.value == 0
        elif call == "head":
            assert refuse(1) == 0
            assert eng.decode_step([s], sh.layers)[0] == FAILED
        got = []
        for i in range(60):
            if call == "decode" and i in (6, 7, 22):      # (positions 16 and 32 open pages)
                assert refuse(1) == 0
                assert eng.decode_step([s, other], 1)[0] == FAILED
            got += s.decode(1, sh.layers)
            other.decode(1, sh.layers)
        assert got == want
        assert abi.parse_save_blob(s.save(), sh.hidden)["kv"] == ps.kv.tobytes()
    finally:
        refuse(0)
        eng.close()


@pytest.mark.parametrize("call", ["prefill", "decode"])
def test_time_of_the_last_completed_call(gpu_lib, call):
    """A refused call has no device time: the one before it keeps its own, whether or not it was asked for by then."""
    sh = A.SHAPES["tiny"]
    art = A.build_synthetic_model("tiny", 0x7480, 700)
    prompt = A.stream_uniform(0x7480, "prompt", 600, 0, sh.vocab - 1)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=600)
    refuse = gpu_lib.dll.sslm_b200_debug_refuse_launch
    refuse.argtypes = [C.c_int32]
    f = gpu_lib.dll.sslm_b200_last_call_ms
    f.argtypes = [C.c_void_p, C.POINTER(C.c_float), C.POINTER(C.c_uint64)]

    def last_ms():
        ms = C.c_float(-1.0)
        assert f(eng.ws, C.byref(ms), None) == 0
        return ms.value

    toks = np.ascontiguousarray(prompt[:20], dtype=np.int32)
    try:
        s = eng.new_seq()
        assert s.prefill(prompt, 600) == 600
        asked = last_ms()
        for ask in (True, False):
            s.reset()
            assert s.prefill(prompt, 600) == 600
            if ask:
                asked = last_ms()
            assert refuse(1) == 0
            if call == "prefill":
                consumed = C.c_int32(-1)
                assert gpu_lib.sslm_prefill(eng.model, s.handle, toks.ctypes.data_as(C.POINTER(C.c_int32)), 20, 20, 0, eng.ws,
                                            C.byref(consumed)) == FAILED
            else:
                assert eng.decode_step([s], sh.layers)[0] == FAILED
            # (not asked before the refusal: the time of a pass over the same 600 tokens)
            assert last_ms() == asked if ask else asked / 4 < last_ms() < 4 * asked
            assert len(s.decode(2, sh.layers)) == 2 and last_ms() > 0
    finally:
        refuse(0)
        eng.close()
