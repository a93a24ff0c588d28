"""Performance cases: the work a program that serves models through the `sslm_*` C ABI has it do.

Such a program maps a model once, keeps one workspace for it, and per conversation runs prefill and
decode calls on sequences of a KV pool. A case is one of

  reply    `n` conversations with cached prompts of `lo`..`hi` tokens (one frozen prefix each) each
           generate `tokens` tokens in one batch: reset, adopt the prefix, decode step by step
  prompt   a fresh prompt is prefilled in chunks and its first `tokens` tokens are decoded
  adapter  the same with a rank-16 adapter attached to the sequence, decoded a few layers per call
  session  a conversation is prefilled, parked (sslm_seq_save), resumed (sslm_seq_restore), continued
  layer    the standalone int8 linear layer on tensors in GPU memory (sslm_b200_linear_resident)

on the full 0.5B and 1.5B shapes of superslm_b200.artifact.SHAPES, or (adapters) four layers at the
3B widths. The 0.5B model carries q/k/v biases and a decode schema. Weights are seeded random values
with the constants that keep a random model inside every integer domain gate; they are the same for
every seed, as a served model is. Prompts, and the layer's operands, are made from the seed. All
results are integers and must be the same to the last bit.
"""
import ctypes as C
import math
import random
from fractions import Fraction

import numpy as np
import torch

from superslm_b200 import abi, artifact as A, build

CONTEXT_CAP = 2304
MAX_BATCH = 256
MAX_CHUNK = 2048
SITE = (1090717716, -44)      # site constant of the standalone layer's funnel


# ------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one projection on the caller's own tensors, between two steps of its own program
        dict(name="layer_45_rows", kind="layer", m=45, k=1536, n=8960),
        # the smallest call: a short exchange with the small model, latency is all that counts
        dict(name="reply_small_short", kind="reply", model="0.5b", n=1, lo=19, hi=19, tokens=4, budget=24, schema=False),
        # one user, long conversation
        dict(name="reply_one_long", kind="reply", model="1.5b", n=1, lo=2011, hi=2011, tokens=16, budget=28, schema=False),
        # a handful of users
        dict(name="reply_five", kind="reply", model="1.5b", n=5, lo=90, hi=700, tokens=16, budget=28, schema=False),
        # structured output: a batch whose tokens a schema constrains
        dict(name="reply_small_schema", kind="reply", model="0.5b", n=21, lo=64, hi=512, tokens=16, budget=24, schema=True),
        # a busy server, and a full one (the benchmark's batch)
        dict(name="reply_64", kind="reply", model="1.5b", n=64, lo=128, hi=1024, tokens=16, budget=28, schema=False),
        dict(name="reply_256", kind="reply", model="1.5b", n=256, lo=128, hi=1024, tokens=32, budget=28, schema=False),
        # time to first token: a short turn, a page of text, a long document
        dict(name="prompt_short", kind="prompt", model="1.5b", length=37, chunk=2048, tokens=1),
        dict(name="prompt_small_512", kind="prompt", model="0.5b", length=512, chunk=512, tokens=2),
        dict(name="prompt_long", kind="prompt", model="1.5b", length=2047, chunk=2048, tokens=2),
        # a character with its own adapter, decoded within a frame budget of one layer per call
        dict(name="adapter_sliced", kind="adapter", model="3b4l", length=901, chunk=512, tokens=8, budget=1),
        # a conversation that is parked and taken up again
        dict(name="session_parked", kind="session", model="0.5b", length=300, chunk=128, tokens=4),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choices(["reply", "prompt", "adapter", "session", "layer"], [9, 5, 2, 2, 2])[0]
    model = rng.choice(["0.5b", "1.5b"])
    if kind == "reply":
        n = _log_int(rng, 1, MAX_BATCH)
        ends = sorted(_log_int(rng, 8, 2047 if n <= 64 else 1024) for _ in range(2))
        layers = A.SHAPES[model].layers
        budget = layers if rng.random() < 0.7 else rng.randint(layers // 4, layers - 1)
        return dict(kind=kind, model=model, n=n, lo=ends[0], hi=ends[1], tokens=rng.randint(3, 16), budget=budget,
                    schema=model == "0.5b" and rng.random() < 0.4)
    length = _log_int(rng, 8, 2047)
    chunk = rng.choice([c for c in (64, 128, 256, 512, 1024, 2048) if length <= 16 * c])
    if kind == "prompt":
        return dict(kind=kind, model=model, length=length, chunk=chunk, tokens=rng.randint(1, 3))
    if kind == "adapter":
        return dict(kind=kind, model="3b4l", length=length, chunk=chunk, tokens=rng.randint(2, 12), budget=rng.randint(1, 4))
    if kind == "session":
        return dict(kind=kind, model=model, length=length, chunk=chunk, tokens=rng.randint(1, 6))
    k, n = rng.choice([(896, 1152), (896, 9728), (4864, 896), (1536, 2048), (1536, 17920), (8960, 1536), (2048, 2048), (11008, 2048)])
    return dict(kind=kind, m=_log_int(rng, 1, 256), k=k, n=n)


# ------------------------------------------------------------------------------------- models
def _json_like_schema(vocab):
    """A DFA of 12 states over the vocabulary, each allowing about 1,000 tokens and leading on."""
    g = np.random.default_rng(17)
    rows = []
    for st in range(12):
        toks = np.unique(g.integers(0, vocab, 1000))
        rows.append([(int(t), int(s)) for t, s in zip(toks, g.integers(0, 12, toks.size))])
    return [{"name": "record", "accepting": [0], "rows": rows}]


def _artifact(shape, seed, biases, schema):
    """A loadable artifact of the shape, as A.build_synthetic_model lays it out, with its large
    tensors drawn on the GPU."""
    sh = A.SHAPES[shape]
    H, I, KV = sh.hidden, sh.inter, sh.kv_hidden
    g = torch.Generator(device="cuda").manual_seed(seed)

    def ints(lo, hi, count, dtype):
        return torch.randint(lo, hi, (count,), dtype=dtype, device="cuda", generator=g).cpu().numpy()

    inv127, s_kh, s_in = Fraction(1, 127), Fraction(1, 30), Fraction(2.0 ** 8.5 / (73.3 * math.sqrt(H) * 0.58))
    s_o, s_down = (Fraction(2.0 ** 8.5 / (73.3 * math.sqrt(k) * 0.35)) for k in (H, I))
    c = {"norm": inv127 / (1 << 16) / 127, "proj": s_in / 127, "o_proj": s_o / 127, "down_proj": s_down / 127,
         "attn_ctx": s_kh / (1 << 15) / 127, "mlp_act": Fraction(1, (1 << 15) * 127), "residual": inv127,
         "khead": Fraction(float(s_kh) / math.sqrt(sh.head_dim)), "embed": inv127 / 127, "kv": s_kh}
    c = {k: A.canonical_scale(v) for k, v in c.items()}
    m_t, e_t = A.canonical_scale(s_kh / s_in)
    recip = (m_t, e_t, A.dynamic_scale_reciprocal(m_t))

    weights = [("embed", ints(-127, 128, sh.vocab * H, torch.int8).reshape(sh.vocab, H)),
               ("final_norm.gain", ints(-127, 128, H, torch.int8))]
    folds, bias, consts, kv_scales, kv_recips = [], [], [("embed", c["embed"]), ("final_norm", c["norm"])], [], []
    for l in range(sh.layers):
        p = "layer%d." % l
        for proj, rows, cols in (("q_proj", H, H), ("k_proj", KV, H), ("v_proj", KV, H), ("o_proj", H, H),
                                 ("gate_proj", I, H), ("up_proj", I, H), ("down_proj", H, I)):
            weights.append((p + proj, ints(-127, 128, rows * cols, torch.int8).reshape(rows, cols)))
            f = np.zeros((rows, 3), dtype=np.int32)
            f[:, 1] = ints(1 << 30, (1 << 31) - 1, rows, torch.int32)
            f[:, 2] = ints(8, 21, rows, torch.int32)
            folds.append((p + proj, f))
            if biases and proj in ("q_proj", "k_proj", "v_proj"):
                bias.append((p + proj, ints(-(1 << 29), 1 << 29, rows, torch.int64)))
        for norm in ("attn_norm", "mlp_norm"):
            weights.append((p + norm + ".gain", ints(-127, 128, H, torch.int8)))
            consts.append((p + norm, c["norm"]))
        ctx = np.zeros((sh.heads, 3), dtype=np.int32)
        ctx[:, 0] = 1
        folds.append((p + "ctx_fold", ctx))
        consts += [(p + q, c["proj"]) for q in ("q_proj", "gate_proj", "up_proj")]
        consts += [(p + q, c[q]) for q in ("o_proj", "down_proj", "attn_ctx", "mlp_act")]
        consts += [(p + q, c["residual"]) for q in ("attn_residual", "mlp_residual")]
        for h in range(sh.kv_heads):
            consts.append((p + "softmax_khead%d" % h, c["khead"]))
            for kv in ("k", "v"):
                kv_scales.append((p + "%s_head%d" % (kv, h), c["kv"]))
                kv_recips.append((p + "%s_head%d" % (kv, h), recip))
    cos, sin = A.rope_tables(CONTEXT_CAP, sh.head_dim, 1e6)
    sections = [
        (A.SEC_CONFIG, A.cfg1(H, sh.layers, sh.heads, sh.kv_heads, sh.head_dim, I, sh.vocab, CONTEXT_CAP)),
        (A.SEC_SIGMOID_LUT, A.sil1()),
        (A.SEC_WEIGHTS, A.tensor_manifest(b"WGT1", 1, weights)),
        (A.SEC_WEIGHT_SCALES, A.tensor_manifest(b"WSC1", 4, folds)),
        (A.SEC_ROPE, A.tensor_manifest(b"ROP1", 8, [("cos", cos), ("sin", sin)])),
        (A.SEC_COMPOSITION, A.keyed_constants(consts, 2)),
        (A.SEC_KV_SCALES, A.keyed_constants(kv_scales, 2)),
        (A.SEC_KV_RECIP, A.keyed_constants(kv_recips, 3)),
    ]
    if bias:
        sections.insert(3, (A.SEC_BIASES, A.tensor_manifest(b"BIA1", 8, bias)))
    if schema:
        sections.append((A.SEC_SCHEMA_MASKS, A.schema_masks(sh.vocab, _json_like_schema(sh.vocab))))
    return A.build_container(sections)


def _check(status, what):
    if status != abi.SSLM_OK:
        raise abi.SslmError(what, status)


class _Model:
    """What a serving program holds for a model from its start on: the mapped model and a workspace."""

    def __init__(self, lib, shape):
        self.lib = lib
        art = _artifact(shape, 20 + len(shape), biases=shape == "0.5b", schema=shape == "0.5b")
        self.eng = abi.Engine(lib, art, blocks=1, max_batch=MAX_BATCH, max_chunk=MAX_CHUNK)
        self.handle, self.ws, self.vocab = self.eng.model, self.eng.ws, A.SHAPES[shape].vocab
        self.layers = A.SHAPES[shape].layers
        self.adapter = self.eng.map_adapter(A.build_synthetic_adapter(art, 7)) if shape == "3b4l" else None
        self.schema = abi._H()
        if shape == "0.5b":
            _check(lib.sslm_schema_lookup(self.handle, b"record", C.byref(self.schema)), "sslm_schema_lookup")


_LIB = []
_MODELS = {}


def _lib():
    if not _LIB:
        _LIB.append(abi.SslmLib(build.LIB))
    return _LIB[0]


def _model(shape):
    if shape not in _MODELS:
        _MODELS[shape] = _Model(_lib(), shape)
    return _MODELS[shape]


class _Conversations:
    """Sequences (and the frozen prefixes they start from) in a KV pool of their own."""

    def __init__(self, model, count, prefixes, spare=0):
        self.model, self.lib = model, model.lib
        blocks = count + prefixes + spare
        need = model.eng.block_size * blocks + self.lib.sslm_kv_pool_overhead_size(model.handle, blocks)
        self._room = np.empty(need + 64, dtype=np.uint8)      # the caller's reservation; never touched
        at = self._room.ctypes.data
        self.pool, self.seqs, self.prefixes = abi._H(), (abi._H * count)(), [abi._H() for _ in range(prefixes)]
        _check(self.lib.sslm_kv_pool_create(model.handle, C.c_void_p(at + (-at) % 64), need, blocks, C.byref(self.pool)),
               "sslm_kv_pool_create")
        for i in range(count):
            s = abi._H()
            _check(self.lib.sslm_seq_create(model.handle, C.byref(self.pool), C.byref(s)), "sslm_seq_create")
            self.seqs[i] = s

    def __del__(self):
        for i in range(len(self.seqs)):
            if self.seqs[i]:
                self.lib.sslm_seq_release(self.seqs[i])
        for p in self.prefixes:
            if p:
                self.lib.sslm_prefix_release(p)
        if self.pool:
            self.lib.sslm_kv_pool_destroy(self.pool)

    def prefill(self, verb, handle, tokens, chunk):
        done = 0
        while done < tokens.size:
            took = C.c_int32(0)
            _check(verb(self.model.handle, handle, tokens[done:].ctypes.data_as(C.POINTER(C.c_int32)), tokens.size - done,
                        chunk, 0, self.model.ws, C.byref(took)), "prefill")
            done += took.value

    def decode(self, seqs, tokens, budget):
        """`tokens` greedy tokens of every sequence, [tokens, n]; a call advances `budget` layers."""
        n = len(seqs)
        out, params, got = (C.c_int32 * n)(), abi.SslmDecodeParams(layer_budget=budget), []
        while len(got) < tokens:
            _check(self.lib.sslm_decode_step(self.model.handle, seqs, n, C.byref(params), self.model.ws, out), "sslm_decode_step")
            if out[0] != -1:      # all sequences started on the same layer, so all finish a token together
                got.append(np.ctypeslib.as_array(out).copy())
        return np.stack(got)


# ------------------------------------------------------------------------------------- interface
def prepare(case, seed):
    g = np.random.default_rng(seed)
    if case["kind"] == "layer":
        m, n, k = case["m"], case["n"], case["k"]
        gt = torch.Generator(device="cuda").manual_seed(seed)

        def ints(lo, hi, size, dtype):
            return torch.randint(lo, hi, size, dtype=dtype, device="cuda", generator=gt)

        fold = torch.zeros((n, 3), dtype=torch.int32, device="cuda")
        fold[:, 1] = ints(1 << 30, (1 << 31) - 1, (n,), torch.int32)
        fold[:, 2] = ints(8, 21, (n,), torch.int32)
        scales = torch.full((m, 2), -37, dtype=torch.int64, device="cuda")
        scales[:, 0] = ints(1 << 30, (1 << 31) - 1, (m,), torch.int64)
        call = _lib().dll.sslm_b200_linear_resident
        call.restype = C.c_int32
        call.argtypes = [C.c_void_p] * 3 + [C.c_int32] * 3 + [C.c_void_p, C.c_int64, C.c_int64] + [C.c_void_p] * 5
        return dict(case=case, call=call, x=ints(-127, 128, (m, k), torch.int8), w=ints(-127, 128, (n, k), torch.int8),
                    fold=fold, scales=scales, folded=torch.empty((m, n), dtype=torch.int32, device="cuda"),
                    codes=torch.empty((m, n), dtype=torch.int8, device="cuda"),
                    out_scales=torch.empty((m, 2), dtype=torch.int64, device="cuda"),
                    status=torch.empty(m, dtype=torch.int32, device="cuda"))
    model = _model(case["model"])
    if case["kind"] == "reply":
        conv = _Conversations(model, case["n"], case["n"])
        for i in range(case["n"]):
            tokens = g.integers(0, model.vocab, int(g.integers(case["lo"], case["hi"] + 1))).astype(np.int32)
            _check(model.lib.sslm_prefix_begin(model.handle, C.byref(conv.pool), C.byref(conv.prefixes[i])), "sslm_prefix_begin")
            conv.prefill(model.lib.sslm_prefix_prefill, conv.prefixes[i], tokens, MAX_CHUNK)
            _check(model.lib.sslm_prefix_freeze(conv.prefixes[i]), "sslm_prefix_freeze")
            if case["schema"]:
                _check(model.lib.sslm_seq_set_schema(conv.seqs[i], model.schema), "sslm_seq_set_schema")
        return dict(case=case, conv=conv)
    conv = _Conversations(model, 1, 0, spare=1)
    if case["kind"] == "adapter":
        _check(model.lib.sslm_seq_set_adapter(conv.seqs[0], model.adapter), "sslm_seq_set_adapter")
    return dict(case=case, conv=conv, prompt=g.integers(0, model.vocab, case["length"]).astype(np.int32))


def run(state):
    case = state["case"]
    if case["kind"] == "layer":
        s = state
        _check(s["call"](s["x"].data_ptr(), s["w"].data_ptr(), s["fold"].data_ptr(), case["m"], case["n"], case["k"],
                         s["scales"].data_ptr(), SITE[0], SITE[1], s["folded"].data_ptr(), s["codes"].data_ptr(),
                         s["out_scales"].data_ptr(), s["status"].data_ptr(), torch.cuda.current_stream().cuda_stream),
               "sslm_b200_linear_resident")
        return dict(folded=s["folded"], codes=s["codes"], scales=s["out_scales"], status=s["status"])
    conv = state["conv"]
    lib, seqs, layers = conv.lib, conv.seqs, conv.model.layers
    for i in range(len(seqs)):
        _check(lib.sslm_seq_reset(seqs[i]), "sslm_seq_reset")
    if case["kind"] == "reply":
        for i in range(len(seqs)):
            _check(lib.sslm_seq_adopt_prefix(seqs[i], conv.prefixes[i]), "sslm_seq_adopt_prefix")
        return conv.decode(seqs, case["tokens"], case["budget"])
    conv.prefill(lib.sslm_prefill, seqs[0], state["prompt"], case["chunk"])
    if case["kind"] != "session":
        return conv.decode(seqs, case["tokens"], case.get("budget", layers))
    size = C.c_size_t(0)
    lib.sslm_seq_save(seqs[0], None, C.byref(size))
    blob = np.empty(size.value, dtype=np.uint8)
    _check(lib.sslm_seq_save(seqs[0], blob.ctypes.data, C.byref(size)), "sslm_seq_save")
    resumed = (abi._H * 1)()
    h = abi._H()
    _check(lib.sslm_seq_restore(conv.model.handle, C.byref(conv.pool), blob.ctypes.data, blob.size, C.byref(h)), "sslm_seq_restore")
    resumed[0] = h
    try:
        tokens = conv.decode(resumed, case["tokens"], layers)
    finally:
        lib.sslm_seq_release(h)
    return dict(blob=blob, tokens=tokens)


def work(case):
    if case["kind"] == "layer":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=n * k + 12 * n + m * (k + 5 * n + 36), flops=2 * m * n * k)
    sh = A.SHAPES[case["model"]]
    H, I, KV, L = sh.hidden, sh.inter, sh.kv_hidden, sh.layers
    mats = L * (2 * H * H + 2 * H * KV + 3 * H * I)            # weights of all layers, one byte each
    layers = mats + L * 12 * (2 * H + 2 * KV + 2 * I + sh.heads)     # and their folds
    head = sh.vocab * H
    if case["kind"] == "reply":
        # the first token comes from the prompt's last state (the head alone), the others from full steps
        n, steps, width = case["n"], case["tokens"] - 1, (case["lo"] + case["hi"]) / 2 + case["tokens"] / 2
        return dict(bytes=case["tokens"] * head + steps * layers + steps * n * L * 2 * KV * width,
                    flops=2 * n * (case["tokens"] * head + steps * mats) + steps * n * L * 4 * H * width)
    p, steps = case["length"], case["tokens"] - 1
    chunks = -(-p // case["chunk"])
    kv = L * 2 * KV * p
    b = chunks * layers + kv * (1 + (chunks - 1) / 2) + steps * (layers + kv) + case["tokens"] * head
    f = 2 * mats * p + L * 2 * H * p * p + steps * (2 * mats + L * 4 * H * p) + 2 * case["tokens"] * head
    if case["kind"] == "adapter":
        b += (chunks + steps) * L * 16 * (8 * H)
        f += 2 * (p + steps) * L * 16 * (6 * H + 2 * KV)
    if case["kind"] == "session":
        b += 2 * kv + L * 2 * KV * CONTEXT_CAP
    return dict(bytes=b, flops=f)


def tolerance(case):
    return "exact"
