"""A model keeps working after a narrower one has been mapped beside it."""
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide,narrow", [("mini1.5b", "tiny"), ("mini0.5b", "small")])
def test_wide_model_after_a_narrow_one(gpu_lib, wide, narrow):
    art, prompt = A.build_synthetic_model(wide, 0x2A, 64), A.stream_uniform(0x2A, "prompt", 24, 0, A.SHAPES[wide].vocab - 1)
    want, _ = run_port(art, prompt, 2)
    eng = abi.Engine(gpu_lib, art, blocks=1, max_chunk=24)
    other = abi.Engine(gpu_lib, A.build_synthetic_model(narrow, 0x2B, 64), blocks=1, max_chunk=24)
    try:
        s = eng.new_seq()
        assert s.prefill(prompt, 24) == 24
        assert s.decode(2, A.SHAPES[wide].layers) == want
    finally:
        other.close()
        eng.close()
