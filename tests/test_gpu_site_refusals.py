"""Refusals inside the attention cluster, where the q/k/v site of two decode rows and more runs: softmax constants, the q funnel, and
what biases can leave (their exponent's domain, the product's), with biases on q, k and v or on k alone. A conversation begun
on a healthy artifact is taken up on a hostile one with the same weights (its blob is given the other model's hash), so that a decode
batch meets the refusal behind a prompt. Status, committed layers, K/V bytes and saturation counts as the CPU oracle has them, and as
one row (whose site is a kernel of its own) leaves them."""
import struct

import numpy as np
import pytest

from oracle import harness as H
from superslm_b200 import abi, artifact as A

pytestmark = pytest.mark.gpu

CAP, CANON = 96, 1 << 30
SOFTMAX_KERNEL_REFUSED = 20
LENGTHS = (70, 9, 33)
# the healthy artifact's bias bits, what the hostile one overrides, its biases (projection -> factor; None: as they were), and
# whether the rows carry an adapter (64-bit rows)
CASES = {
    "constants_out_of_domain": (0, {"layer1.softmax_khead1": (CANON, -80)}, None, False),
    "kernel_refused": (0, {"layer2.softmax_khead0": (CANON, -3)}, None, False),
    "kernel_refused_adapted": (0, {"layer1.softmax_khead1": (CANON, -3)}, None, True),
    "kernel_refused_by_the_q_scale": (0, {"layer1.q_proj": ((1 << 31) - 1, 7)}, None, False),
    "constants_behind_saturating_landings": (33, {"layer1.softmax_khead0": (CANON, -80)}, None, False),
    "kernel_refused_behind_saturating_landings": (33, {"layer1.q_proj": ((1 << 31) - 1, 7)}, None, False),
    "biased_q_funnel": (30, {}, {"q": 1 << 32, "k": 1, "v": 1}, False),
    "bias_exponent": (30, {"layer1.attn_norm": (CANON, 7)}, None, False),
    "bias_exponent_of_k": (30, {"layer1.attn_norm": (CANON, 7)}, {"k": 1}, False),
    "q_product": (30, {"layer1.attn_norm": (CANON, -80)}, {"q": 1 << 32, "k": 1, "v": 1}, False),
    "k_product": (30, {"layer1.attn_norm": (CANON, -80)}, {"k": 1 << 32}, False),
    "v_product": (30, {"layer1.attn_norm": (CANON, -80)}, {"q": 0, "v": 1 << 32}, False),
    "v_product_adapted": (30, {"layer1.attn_norm": (CANON, -80)}, {"q": 0, "v": 1 << 32}, True),
}


def artifacts(name):
    bits, overrides, factors, _ = CASES[name]
    seed = 0x7C00 + sorted(CASES).index(name)
    healthy = A.build_synthetic_model("small", seed, CAP, bias_bits=bits)
    hostile = A.build_synthetic_model("small", seed, CAP, bias_bits=bits, const_overrides=overrides)
    if factors is not None:
        v = A.parse_artifact(hostile)
        # (gains of one lower the normed row's scale as far as the product's domain asks for)
        weights = [(k, np.ones_like(t) if k == "layer1.attn_norm.gain" and "product" in name else t)
                   for k, t in v.tensors(A.SEC_WEIGHTS, np.int8).items()]
        old = v.tensors(A.SEC_BIASES, np.int64)
        new = [(k, t * factors[k.split(".")[1][0]] if k.startswith("layer1.") else t) for k, t in old.items()
               if not k.startswith("layer1.") or k.split(".")[1][0] in factors]
        swap = {A.SEC_BIASES: A.tensor_manifest(b"BIA1", 8, new), A.SEC_WEIGHTS: A.tensor_manifest(b"WGT1", 1, weights)}
        sections = [(t, swap.get(t, bytes(raw))) for t, raw in v.sections.items()]
        hostile = A.build_container(sections)
    return healthy, hostile


def begin(lib, art, adp, sh):
    """(blob, oracle state) of every conversation behind its prompt and first token, on the healthy artifact"""
    out = []
    eng = abi.Engine(lib, art, blocks=len(LENGTHS), max_chunk=CAP) if lib is not None else None
    try:
        pm = H.PortModel(art)
        for i, n in enumerate(LENGTHS):
            prompt = A.stream_uniform(0x7C80 + i, "prompt", n, 0, sh.vocab - 1)
            ps = H.PortSeq(pm)
            assert ps.prefill(prompt) == 0
            want = ps.decode(1, sh.layers)
            blob = None
            if eng is not None:
                s = eng.new_seq()
                assert s.prefill(prompt, CAP) == n
                assert s.decode(1, sh.layers) == want
                blob = s.save()
            out.append((blob, ps))
        return out
    finally:
        if eng is not None:
            eng.close()


def refused(ps, pm, lora, sh):
    """the oracle's status of the next token on the hostile model, and what the sequence holds then"""
    q = H.PortSeq(pm)
    q.hidden[:], q.kv[:] = ps.hidden, ps.kv
    q.s.hidden_scale, q.s.context_length, q.s.kv_saturation_count = ps.s.hidden_scale, ps.s.context_length, ps.s.kv_saturation_count
    q.current_token, q.lora = ps.current_token, lora
    status = q.decode_step(sh.layers)[0]
    assert status != 0
    return status, q


def holds(blob, sh):
    """what a sequence observably holds: K/V of the positions that count, the stream of a token in flight, the counters"""
    b = abi.parse_save_blob(blob, sh.hidden)
    kv = np.frombuffer(b["kv"], dtype=np.int8).reshape(sh.layers, 2, sh.kv_heads, CAP, sh.head_dim).copy()
    for layer in range(sh.layers):
        kv[layer, :, :, b["context_length"] + (1 if layer < b["layer_index"] else 0):] = 0
    return kv.tobytes(), b["residual"], b["context_length"], b["layer_index"], b["kv_saturation_count"], \
        b["hidden_scale"] if b["layer_index"] else None


def oracle_holds(q, sh):
    kv = q.kv.reshape(sh.layers, 2, sh.kv_heads, CAP, sh.head_dim).copy()
    for layer in range(sh.layers):
        kv[layer, :, :, q.s.context_length + (1 if layer < q.s.layer_index else 0):] = 0
    li = q.s.layer_index
    return kv.tobytes(), q.hidden.tobytes() if li else b"", q.s.context_length, li, q.s.kv_saturation_count, \
        (q.s.hidden_scale.m, q.s.hidden_scale.e) if li else None


@pytest.mark.parametrize("name", sorted(CASES))
def test_refused_rows(gpu_lib, name):
    sh = A.SHAPES["small"]
    healthy, hostile = artifacts(name)
    adapted = CASES[name][3]
    begun = begin(gpu_lib, healthy, None, sh)
    pm = H.PortModel(hostile)
    adp = A.build_synthetic_adapter(hostile, 0x7CF0, 16, A.PEFT_ORDER) if adapted else None
    lora = pm.lora(adp) if adapted else None
    eng = abi.Engine(gpu_lib, hostile, blocks=len(LENGTHS), max_batch=len(LENGTHS), max_chunk=CAP)
    try:
        handle = eng.map_adapter(adp) if adapted else None
        probe = eng.new_seq()
        own = probe.save()[4:36]      # (the hostile model's hash)
        probe.release()
        for order in ((0,), (0, 1), (1, 0), (2, 1, 0)):      # (one row alone as well)
            seqs = []
            for i in order:
                blob = begun[i][0]
                s = abi.Sequence.restore(eng, blob[:4] + own + blob[36:])
                if adapted:
                    s.set_adapter(handle)
                seqs.append(s)
            before = [holds(s.save(), sh) for s in seqs]
            status, q = refused(begun[order[0]][1], pm, lora, sh)
            got, _ = eng.decode_step(seqs, sh.layers)
            want = "SSLM_NUMERIC_STEP_REFUSED" if status == SOFTMAX_KERNEL_REFUSED else "SSLM_ARTIFACT_REJECTED"
            assert got == abi.ST[want], (order, status)
            after = [holds(s.save(), sh) for s in seqs]
            assert after[0] == oracle_holds(q, sh), order
            assert after[1:] == before[1:], order
            for s in seqs:
                s.release()
    finally:
        eng.close()
