"""Adoption of a prefix returns while its kernel may still run: what follows at once -- release of the prefix, save,
reset or release of the adopter, another adoption, other sequences in the freed pages, other threads -- must find
the state it would have found behind it."""
import ctypes as C
import threading

import numpy as np
import pytest

from superslm_b200 import abi, artifact as A
from tests.test_gpu_prefix import Prefix

pytestmark = pytest.mark.gpu
SHAPE, CAP = "small", 112


@pytest.fixture(scope="module")
def art():
    return A.build_synthetic_model(SHAPE, seed=0xADD, context_cap=CAP)


def toks(n, salt):
    return A.stream_uniform(700 + salt, "adopt_tokens", n, 0, A.SHAPES[SHAPE].vocab - 1).astype(np.int32)


def alone(lib, art, n, salt, ndec):
    """tokens and blobs (before and after decoding) of a sequence that prefilled the prompt itself"""
    eng = abi.Engine(lib, art, blocks=1, max_chunk=CAP)
    try:
        s = eng.new_seq()
        assert s.prefill(toks(n, salt), CAP) == n
        before = s.save()
        return before, s.decode(ndec, A.SHAPES[SHAPE].layers), s.save()
    finally:
        eng.close()


@pytest.mark.parametrize("n", [37, 48, 5])
def test_what_follows_at_once(gpu_lib, art, n):
    layers = A.SHAPES[SHAPE].layers
    want = alone(gpu_lib, art, n, 0, 4)
    other = alone(gpu_lib, art, 90, 1, 4)
    eng = abi.Engine(gpu_lib, art, blocks=3, max_batch=2, max_chunk=CAP)
    lib = gpu_lib
    try:
        for turn in range(3):
            px = Prefix(lib, eng)
            assert px.prefill(toks(n, 0), CAP) == 0
            px.freeze()
            a, b = eng.new_seq(), eng.new_seq()
            adopt = lambda s: lib.sslm_seq_adopt_prefix(s.handle, px.h)
            # a save reads what the adoption writes
            assert adopt(a) == 0
            assert a.save() == want[0]
            # another adoption, a reset and a prompt of one's own over one that may still run
            assert adopt(a) == 0 and adopt(a) == 0
            a.reset()
            assert a.prefill(toks(90, 1), CAP) == 90
            assert (a.decode(4, layers), a.save()) == (other[1], other[2])
            # the adopter leaves; its slot and its pages go to the next sequence
            assert adopt(a) == 0
            a.release()
            c = eng.new_seq()
            assert c.prefill(toks(90, 1), CAP) == 90
            assert (c.decode(4, layers), c.save()) == (other[1], other[2])
            c.release()
            # the prefix leaves; a sequence takes its slot and the page that was not shared
            assert adopt(b) == 0
            px.release()
            d = eng.new_seq()
            assert d.prefill(toks(90, 1), CAP) == 90
            assert (b.decode(4, layers), b.save()) == (want[1], want[2])
            assert (d.decode(4, layers), d.save()) == (other[1], other[2])
            b.release()
            d.release()
    finally:
        eng.close()


def test_several_threads(gpu_lib, art):
    layers = A.SHAPES[SHAPE].layers
    lengths = [37, 16, 90, 64]
    want = [alone(gpu_lib, art, n, i, 3) for i, n in enumerate(lengths)]
    eng = abi.Engine(gpu_lib, art, blocks=2 * len(lengths), max_chunk=CAP)
    wrong = []

    def work(i, px, s):
        params, out, arr = abi.SslmDecodeParams(layer_budget=layers), (C.c_int32 * 1)(), (abi._H * 1)(s.handle)
        for _ in range(25):
            got = []
            if gpu_lib.sslm_seq_adopt_prefix(s.handle, px.h) != 0:
                wrong.append((i, "adopt"))
            for _ in range(3):      # (no workspace given: the model's own, one call at a time)
                if gpu_lib.sslm_decode_step(eng.model, arr, 1, C.byref(params), None, out) != 0:
                    wrong.append((i, "decode"))
                got.append(out[0])
            if got != want[i][1] or s.save() != want[i][2]:
                wrong.append((i, got))
            s.reset()

    try:
        pxs = []
        for i, n in enumerate(lengths):
            px = Prefix(gpu_lib, eng)
            assert px.prefill(toks(n, i), CAP) == 0
            px.freeze()
            pxs.append((px, eng.new_seq()))
        threads = [threading.Thread(target=work, args=(i, px, s)) for i, (px, s) in enumerate(pxs)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong, wrong[:4]
        for px, _ in pxs:
            px.release()
    finally:
        eng.close()
