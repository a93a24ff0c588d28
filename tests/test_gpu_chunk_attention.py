"""Attention of prefill chunks in tiles of 32 query rows, against the CPU oracle: chunks around the tile and
step sizes and the sizes where it takes over, one block per tile and tiles split over clusters, prefixes of
earlier chunks, head dimensions 32 and 64 with the real models' group sizes. (Head dimension 128 and widths
up to 32,768 are held to records of the reference by test_gpu_configs.py.)"""
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu

CASES = [("tiny", [512]), ("tiny", [448, 64, 65]), ("tiny", [500, 127, 129]), ("tiny", [513]), ("tiny", [700, 64, 300]),
         ("tiny", [1300]), ("tiny", [1, 640]), ("tiny", [1599, 65]), ("tiny", [1600, 130]), ("small", [520, 200]),
         ("mini0.5b", [530])]


@pytest.mark.parametrize("shape,chunks", CASES)
def test_chunks_match_the_oracle(gpu_lib, shape, chunks):
    sh = A.SHAPES[shape]
    n = sum(chunks)
    art = A.build_synthetic_model(shape, 0x5100 + n, n + 16)
    prompt = A.stream_uniform(0x5100 + n, "prompt", n, 0, sh.vocab - 1)
    want, ps = run_port(art, prompt, 2)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=max(chunks))
    try:
        s = eng.new_seq()
        at = 0
        for c in chunks:
            assert s.prefill(prompt[at:at + c], c) == c
            at += c
        assert s.decode(2, sh.layers) == want
        assert abi.parse_save_blob(s.save(), sh.hidden)["kv"] == ps.kv.tobytes()
    finally:
        eng.close()
