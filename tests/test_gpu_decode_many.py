"""Decode batches too large for attention clusters, at each head dimension and with either block size (by the rule of
launch_attn), against the CPU oracle: rows of five widths, every row held to its prompt's tokens and K/V bytes."""
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_parity import run_port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,rows,bias_bits", [("tiny", 45, 0), ("small", 45, 30), ("mini0.5b", 40, 30), ("mini1.5b", 45, 0), ("mini1.5b", 100, 0)])
def test_every_row_matches_the_oracle(gpu_lib, shape, rows, bias_bits):
    sh = A.SHAPES[shape]
    art = A.build_synthetic_model(shape, 0x7B00, 160, bias_bits=bias_bits)
    prompts = [A.stream_uniform(0x7B01 + i, "prompt", n, 0, sh.vocab - 1) for i, n in enumerate((1, 16, 63, 64, 140))]
    want = [run_port(art, p, 3) for p in prompts]
    eng = abi.Engine(gpu_lib, art, blocks=rows, max_batch=rows, max_chunk=160)
    try:
        seqs = []
        for i in range(rows):
            seqs.append(eng.new_seq())
            assert seqs[i].prefill(prompts[i % 5], 160) == len(prompts[i % 5])
        got = []
        for _ in range(3):
            status, tokens = eng.decode_step(seqs, sh.layers)
            assert status == 0
            got.append(tokens)
        for i, s in enumerate(seqs):
            tokens, ps = want[i % 5]
            assert [step[i] for step in got] == tokens, i
            if i < 5 or i >= rows - 5:
                assert abi.parse_save_blob(s.save(), sh.hidden)["kv"] == ps.kv.tobytes(), i
    finally:
        eng.close()


@pytest.mark.parametrize("shape,rows", [("mini1.5b", 17), ("mini1.5b", 32), ("mini3b", 24), ("mini0.5b", 33), ("small", 64), ("tiny", 100)])
def test_adapted_rows_match_the_oracle(gpu_lib, shape, rows):
    """64-bit rows in every width of the weights-first kernel from 32 columns on; one row in three has no adapter"""
    sh = A.SHAPES[shape]
    art = A.build_synthetic_model(shape, 0x7B80, 64)
    adp = A.build_synthetic_adapter(art, 0x7B81, 16, A.PEFT_ORDER)
    prompts = [A.stream_uniform(0x7B82 + i, "prompt", n, 0, sh.vocab - 1) for i, n in enumerate((1, 40, 16))]
    want = [run_port(art, p, 3, adp if i != 2 else None) for i, p in enumerate(prompts)]
    eng = abi.Engine(gpu_lib, art, blocks=rows, max_batch=rows, max_chunk=64)
    try:
        handle, seqs = eng.map_adapter(adp), []
        for i in range(rows):
            seqs.append(eng.new_seq())
            if i % 3 != 2:
                seqs[i].set_adapter(handle)
            assert seqs[i].prefill(prompts[i % 3], 64) == len(prompts[i % 3])
        got = [eng.decode_step(seqs, sh.layers) for _ in range(3)]
        assert [status for status, _ in got] == [0] * 3
        for i, s in enumerate(seqs):
            tokens, ps = want[i % 3]
            assert [step[i] for _, step in got] == tokens, i
            if i < 3 or i >= rows - 3:
                assert abi.parse_save_blob(s.save(), sh.hidden)["kv"] == ps.kv.tobytes(), i
    finally:
        eng.close()
