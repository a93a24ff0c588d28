"""Decode batches of a few rows, whose q/k/v site runs inside the attention cluster, against the CPU oracle: every head
dimension, biases (saturating ones too) and adapters (64-bit rows) or none, rows that end a page, begin one, end and begin a
64-position group, and rows cut into slices."""
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu

LENGTHS = (1, 15, 16, 63, 64, 130)


@pytest.mark.parametrize("shape,rows", [("tiny", 2), ("small", 6), ("mini0.5b", 3), ("mini1.5b", 2), ("mini3b", 2)])
@pytest.mark.parametrize("bias_bits,adapted", [(0, False), (30, False), (0, True), (36, True)])
def test_batch_matches_the_oracle_row_by_row(gpu_lib, shape, rows, bias_bits, adapted):
    sh = A.SHAPES[shape]
    art = A.build_synthetic_model(shape, 0x7A00, 192, bias_bits=bias_bits)
    adp = A.build_synthetic_adapter(art, 0x7A01, 16, A.PEFT_ORDER) if adapted else None
    eng = abi.Engine(gpu_lib, art, blocks=rows, max_batch=rows, max_chunk=192)
    try:
        handle = eng.map_adapter(adp) if adapted else None
        seqs, want = [], []
        for i in range(rows):
            n = LENGTHS[(i + rows) % len(LENGTHS)]
            prompt = A.stream_uniform(0x7A02 + i, "prompt", n, 0, sh.vocab - 1)
            mine = adp if adapted and i != 1 else None      # (one row without)
            want.append(run_port(art, prompt, 4, mine))
            s = eng.new_seq()
            if mine is not None:
                s.set_adapter(handle)
            assert s.prefill(prompt, n) == n
            seqs.append(s)
        got = []
        for _ in range(4):
            status, tokens = eng.decode_step(seqs, sh.layers)
            assert status == 0
            got.append(tokens)
        for i, (s, (tokens, ps)) in enumerate(zip(seqs, want)):
            assert [step[i] for step in got] == tokens
            blob = abi.parse_save_blob(s.save(), sh.hidden)
            assert blob["kv"] == ps.kv.tobytes() and blob["kv_saturation_count"] == ps.s.kv_saturation_count
    finally:
        eng.close()
