"""The widest activation row the kernels hold runs and matches the CPU oracle; a model with a wider one is refused when
it is mapped, not in its first call."""
import ctypes as C

import numpy as np
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu
WIDEST = 8 * 352 * 5 * 4      # blocks of a row, threads, quads per thread, elements per quad


def shape(inter):
    return A.Shape("wide%d" % inter, 128, 1, 4, 2, 32, inter, 512)


@pytest.mark.parametrize("rows", [1, 5, 40])
def test_widest_row_matches_the_oracle(gpu_lib, rows, monkeypatch):
    sh = shape(WIDEST)
    monkeypatch.setitem(A.SHAPES, sh.name, sh)
    art = A.build_synthetic_model(sh.name, 0x7500, 64)
    prompt = A.stream_uniform(0x7500, "prompt", rows, 0, sh.vocab - 1)
    want, ps = run_port(art, prompt, 2)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=64)
    try:
        s = eng.new_seq()
        assert s.prefill(prompt, 64) == rows
        assert s.decode(2, 1) == want
        assert abi.parse_save_blob(s.save(), sh.hidden)["kv"] == ps.kv.tobytes()
    finally:
        eng.close()


def test_wider_row_is_refused_when_mapped(gpu_lib, monkeypatch):
    sh = shape(WIDEST + 16)
    monkeypatch.setitem(A.SHAPES, sh.name, sh)
    art = np.frombuffer(A.build_synthetic_model(sh.name, 0x7500, 64), dtype=np.uint8)
    h = abi._H()
    assert gpu_lib.sslm_model_map(art.ctypes.data, art.size, C.byref(h)) == abi.ST["SSLM_ARTIFACT_REJECTED"]
    assert not h.value
