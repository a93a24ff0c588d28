"""Save and restore of sequences whose K/V travels in several pieces of whole planes (16 MiB each, two places in
turn): against the same positions saved in one piece, round trips, and small sequences before and after in the same
staging blocks."""
import numpy as np
import pytest

from superslm_b200 import abi, artifact as A

pytestmark = pytest.mark.gpu
CAP = 16384


@pytest.fixture(scope="module")
def engine(gpu_lib):
    sh = A.Shape("planes", 256, 6, 2, 2, 128, 256, 512)      # 24 planes of up to 2 MiB: three pieces
    mp = pytest.MonkeyPatch()
    mp.setitem(A.SHAPES, sh.name, sh)
    eng = abi.Engine(gpu_lib, A.build_synthetic_model(sh.name, 0x7600, CAP), blocks=4, max_chunk=4096)
    mp.undo()
    yield eng, sh
    eng.close()


def planes(blob, sh):
    return np.frombuffer(abi.parse_save_blob(blob, sh.hidden)["kv"], dtype=np.int8).reshape(sh.layers * 2 * sh.kv_heads, CAP, 128)


@pytest.mark.parametrize("n,steps", [(16300, 0), (16001, 1), (8192, 7), (5461, 0), (17, 1)])
def test_pieces_are_the_sequence(engine, n, steps):
    """steps of one layer each behind a whole token: 0 and 6 rest between tokens, the others inside one."""
    eng, sh = engine
    prompt = A.stream_uniform(0x7600, "prompt", n, 0, sh.vocab - 1)
    short = eng.new_seq()
    assert short.prefill(prompt[:300], 300) == min(300, n)
    s = eng.new_seq()
    assert s.prefill(prompt, 4096) == n
    s.decode(1, sh.layers)
    for _ in range(steps):
        assert eng.decode_step([s], 1)[0] == 0
    blob = s.save()
    kv, head = planes(blob, sh), planes(short.save(), sh)
    m = min(n, 300)
    assert (kv[:, :m] == head[:, :m]).all() and not head[:, m:].any() and not kv[:, n + 2:].any()
    assert all(kv[i, :n].any() for i in range(kv.shape[0]))
    back = abi.Sequence.restore(eng, blob)
    assert back.save() == blob
    again = abi.Sequence.restore(eng, short.save())
    assert again.save() == short.save()
    assert back.decode(3, sh.layers) == s.decode(3, sh.layers)
    assert back.save() == s.save()
    for q in (s, short, back, again):
        q.release()
