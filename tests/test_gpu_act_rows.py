"""The activation site of prefill chunks with many rows, against the CPU oracle. Persistent blocks: around the
row count where they take over, rows shorter and longer than a block is wide with and without a remainder, and
one, two and more rows per block. Below: either side of the line to the form with one more block per multiprocessor,
at the two widths that have one."""
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu

CASES = [("tiny", 511), ("tiny", 512), ("tiny", 741), ("tiny", 3100), ("small", 800), ("mini0.5b", 515),
         ("mini1.5b", 222), ("mini1.5b", 223), ("mini3b", 148), ("mini3b", 149)]


@pytest.mark.parametrize("shape,n", CASES)
def test_rows_match_the_oracle(gpu_lib, shape, n):
    sh = A.SHAPES[shape]
    art = A.build_synthetic_model(shape, 0xAC70 + n, n + 16)
    prompt = A.stream_uniform(0xAC70 + n, "prompt", n, 0, sh.vocab - 1)
    want, ps = run_port(art, prompt, 2)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=n)
    try:
        s = eng.new_seq()
        assert s.prefill(prompt, n) == n
        assert s.decode(2, sh.layers) == want
        assert abi.parse_save_blob(s.save(), sh.hidden)["kv"] == ps.kv.tobytes()
    finally:
        eng.close()
