"""Adapters of every form of rank (multiples of sixteen, of four, of neither) on all seven projections, against the CPU
oracle: prompts beyond 256 rows (activation-major tensor-core kernel), up to 256 (weights-first) and decode rows."""
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [1, 4, 6, 8, 12, 16, 20, 32, 48, 64])
@pytest.mark.parametrize("rows", [300, 40])
def test_rank(gpu_lib, rank, rows):
    sh = A.SHAPES["small"]
    art = A.build_synthetic_model("small", 0x7700, 320)
    adp = A.build_synthetic_adapter(art, 0x7700 + rank, rank, A.PEFT_ORDER)
    prompt = A.stream_uniform(0x7700, "prompt", rows, 0, sh.vocab - 1)
    want, ps = run_port(art, prompt, 2, adp)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=rows)
    try:
        s = eng.new_seq()
        s.set_adapter(eng.map_adapter(adp))
        assert s.prefill(prompt, rows) == rows
        assert s.decode(2, sh.layers) == want
        blob = abi.parse_save_blob(s.save(), sh.hidden)
        assert blob["kv"] == ps.kv.tobytes() and blob["kv_saturation_count"] == ps.s.kv_saturation_count
    finally:
        eng.close()
