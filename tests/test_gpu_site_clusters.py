"""Decode batches whose q/k/v site runs inside the attention cluster, on clusters of every size, against the CPU oracle. The number of
kernels a step launches tells that the site ran there."""
import ctypes as C

import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu

# clusters of 16 blocks, eight slices per kv head (short rows leave all but the first empty); one kv head; sixteen; clusters of eight
# blocks; the largest batch that keeps its clusters
WIDE = [
    (A.Shape("x128", 512, 2, 4, 2, 128, 256, 256), (1000, 640, 129, 513, 65), 0, False),
    (A.Shape("x128", 512, 2, 4, 2, 128, 256, 256), (897, 1, 450), 36, True),
    (A.Shape("one_kv", 512, 2, 8, 1, 64, 256, 256), (700, 70), 30, False),
    (A.Shape("sixteen_kv", 512, 2, 16, 16, 32, 256, 256), (100, 17), 30, True),
    (A.SHAPES["small"], (700, 5, 64, 256, 65, 300, 16, 1, 40), 30, True),
    (A.SHAPES["tiny"], (300, 20, 64) * 12 + (150,), 0, False),
]


def launches(lib, eng):
    n = C.c_uint64(0)
    f = lib.dll.sslm_b200_last_call_ms
    f.argtypes = [C.c_void_p, C.c_void_p, C.POINTER(C.c_uint64)]
    assert f(eng.ws, None, C.byref(n)) == 0
    return n.value


def check_batch(gpu_lib, sh, lengths, bias_bits, adapted, cap):
    art = A.build_synthetic_model(sh, 0x7A00, cap, bias_bits=bias_bits)
    adp = A.build_synthetic_adapter(art, 0x7A01, 16, A.PEFT_ORDER) if adapted else None
    rows = len(lengths)
    eng = abi.Engine(gpu_lib, art, blocks=rows, max_batch=rows, max_chunk=cap)
    try:
        handle = eng.map_adapter(adp) if adapted else None
        seqs, want, known = [], [], {}
        for i, n in enumerate(lengths):
            prompt = A.stream_uniform(0x7A02 + (i if rows <= 9 else n), "prompt", n, 0, sh.vocab - 1)
            mine = adp if adapted and i != 1 else None      # (one row without)
            key = (tuple(prompt), mine is None)
            if key not in known:
                known[key] = run_port(art, prompt, 4, mine)
            want.append(known[key])
            s = eng.new_seq()
            if mine is not None:
                s.set_adapter(handle)
            assert s.prefill(prompt, cap) == n
            seqs.append(s)
        got, count = [], [launches(gpu_lib, eng)]
        for _ in range(4):
            status, tokens = eng.decode_step(seqs, sh.layers)
            assert status == 0
            got.append(tokens)
            count.append(launches(gpu_lib, eng))
        for i, (s, (tokens, ps)) in enumerate(zip(seqs, want)):
            assert [step[i] for step in got] == tokens
            blob = abi.parse_save_blob(s.save(), sh.hidden)
            assert blob["kv"] == ps.kv.tobytes() and blob["kv_saturation_count"] == ps.s.kv_saturation_count
        # (one row runs the site in a kernel of its own: one more a layer)
        at = launches(gpu_lib, eng)
        seqs[0].decode(1, sh.layers)
        assert launches(gpu_lib, eng) - at == count[-1] - count[-2] + sh.layers
    finally:
        eng.close()


@pytest.mark.parametrize("shape,lengths,bias_bits,adapted", WIDE)
def test_clusters_of_every_size(gpu_lib, shape, lengths, bias_bits, adapted):
    check_batch(gpu_lib, shape, lengths, bias_bits, adapted, 1024)
