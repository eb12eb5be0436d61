"""What the speed of this engine is measured on: the calls that a program serving the model makes.

The model is the released architecture (`full_size_config`: hidden 4096, 288 experts, vocabulary
154880) cut to its first eight layers - three dense KDA layers, then MLA + MoE, three KDA + MoE, MLA +
MoE - with random weights generated in HBM, as the tests and the benchmark cut it; the layer calls run
on one layer of it. A program loads a model once and sends it many inputs, so the states of one case
share an engine (it is released with the last of them), and a case's seed makes the inputs: prompts,
tokens, activations. Sessions that are already deep start from synthetic caches
(`synth_session`), not from a prompt.

Kinds of case
  moe      one MoE layer on host activations (`op_moe`): `tokens` rows
  kda      one KDA attention layer (`op_kda`): `tokens` consecutive positions, `heads` heads
  mla      one MLA attention layer with its indexer (`op_mla`) after `context` positions
  step     one token through the model, logits back to the host (`forward`): a host-side sampling loop
  greedy   `new` tokens decoded on the device (`decode_greedy`) after `context` positions
  sampled  the same with temperature and nucleus (`decode_sampled`)
  chat     a new session: `tokens` of prompt, then `new` greedy tokens
  prompt   a new session: a prompt of `tokens`, logits of its last position
  batch    one token for each of `sequences` sequences at `context` positions (`decode_batch`)
"bf16" says that the MLA latent cache is kept in BF16 (option latent_bf16); FP32 is the engine's default.
"""
import functools
import importlib.util
import os
import sys
import weakref

import numpy as np

LAYERS = 8                  # of the released architecture's 45
MAX_CONTEXT = 24576         # drawn sessions are at most this deep; the cache holds 32768 positions
CAP = 32768
SESSIONS = 8                # sequences of the engine that the states of a single-session case take in turn
WEIGHTS_SEED = 3


def listed():
    return [
        # one token through one MoE layer from host buffers: the smallest call, the benchmark's headline
        {"name": "moe_1", "kind": "moe", "tokens": 1},
        # a small batch of sequences in one MoE layer
        {"name": "moe_8", "kind": "moe", "tokens": 8},
        # the largest batch a layer call takes in one pass
        {"name": "moe_64", "kind": "moe", "tokens": 64},
        # one decode step of one KDA layer, the benchmark's 32-head configuration
        {"name": "kda_1", "kind": "kda", "tokens": 1, "heads": 32},
        # one decode step of one MLA layer at the deepest benchmarked context
        {"name": "mla_32768", "kind": "mla", "tokens": 1, "context": 32767, "bf16": True},
        # a chat service that samples on the host: one token in, logits out
        {"name": "step_4096", "kind": "step", "context": 4096, "bf16": True},
        # a short question answered greedily with the engine's default options (18 tokens in, as in the benchmark)
        {"name": "chat_18", "kind": "chat", "tokens": 18, "new": 24, "bf16": False},
        # sampled generation on the device in the middle of a conversation
        {"name": "sampled_1000", "kind": "sampled", "context": 1000, "new": 12, "bf16": True},
        # a few users at odd depth, logits for each
        {"name": "batch_7", "kind": "batch", "sequences": 7, "context": 601, "logits": True, "bf16": True},
        # a full batch of the serving benchmark: 64 sequences at 4096 positions
        {"name": "batch_64", "kind": "batch", "sequences": 64, "context": 4096, "logits": False, "bf16": True},
        # a document of a few pages, ragged length
        {"name": "prompt_333", "kind": "prompt", "tokens": 333, "bf16": False},
        # the prefill benchmark
        {"name": "prompt_2048", "kind": "prompt", "tokens": 2048, "bf16": True},
    ]


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("moe", "moe", "kda", "mla", "step", "greedy", "sampled", "chat", "prompt", "prompt", "batch", "batch"))
    bf16 = rng.random() < 0.75
    if kind == "moe":
        return {"kind": kind, "tokens": _log_int(rng, 1, 200)}
    if kind == "kda":
        return {"kind": kind, "tokens": _log_int(rng, 1, 200), "heads": rng.choice((32, 64))}
    if kind == "mla":
        return {"kind": kind, "tokens": _log_int(rng, 1, 40), "context": _log_int(rng, 64, 32000), "bf16": bf16}
    if kind == "step":
        return {"kind": kind, "context": _log_int(rng, 16, MAX_CONTEXT), "bf16": bf16}
    if kind in ("greedy", "sampled"):
        return {"kind": kind, "context": _log_int(rng, 16, MAX_CONTEXT), "new": _log_int(rng, 1, 24), "bf16": bf16}
    if kind == "chat":
        return {"kind": kind, "tokens": _log_int(rng, 2, 300), "new": _log_int(rng, 1, 24), "bf16": bf16}
    if kind == "prompt":
        return {"kind": kind, "tokens": _log_int(rng, 2, 2000), "bf16": bf16}
    return {"kind": kind, "sequences": _log_int(rng, 2, 64), "context": _log_int(rng, 16, 4096), "logits": rng.random() < 0.5, "bf16": True}


# ------------------------------------------------------------------ the engine of a case ----
@functools.lru_cache(None)
def _package():
    """The package of the tree in the working folder (its directory name is not an identifier)."""
    path = os.path.join(os.getcwd(), "glm-5.3-flash-in-c_b200")
    spec = importlib.util.spec_from_file_location("glm53f_b200", os.path.join(path, "__init__.py"), submodule_search_locations=[path])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["glm53f_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


BF16, FP8 = 1, 2


def _matrices(c, mla, dense, parts):
    """[(name, rows, cols, dtype)] of a layer's matrices, routed experts excluded."""
    E, MIX = c.hidden, (2 + c.hc_mult) * c.hc_mult
    t = [("hc_attn_fn", MIX, c.hc_mult * E, BF16), ("hc_ffn_fn", MIX, c.hc_mult * E, BF16)] if parts == "all" else []
    if parts in ("all", "attention"):
        if mla:
            H = c.mla_heads
            a = [("q_a_proj.weight", c.q_lora, E, FP8), ("q_b_proj.weight", H * c.qk_nope, c.q_lora, FP8),
                 ("kv_a_proj_with_mqa.weight", c.kv_lora, E, FP8), ("kv_b_proj.weight", H * (c.qk_nope + c.v_head), c.kv_lora, BF16),
                 ("o_proj.weight", E, H * c.v_head, FP8), ("indexer.wq_b.weight", c.index_heads * c.index_dim, c.q_lora, BF16),
                 ("indexer.wk.weight", c.index_dim, E, BF16), ("indexer.weights_proj.weight", c.index_heads, E, BF16),
                 ("indexer.index_kpool_compress_gate", c.index_dim, E, BF16)]
        else:
            D, P = c.kda_head_dim, c.kda_heads * c.kda_head_dim
            a = [(n + "_proj.weight", P, E, BF16) for n in "qkv"]
            a += [(n + "_a_proj.weight", D, E, BF16) for n in "fg"] + [(n + "_b_proj.weight", P, D, BF16) for n in "fg"]
            a += [("b_proj.weight", c.kda_heads, E, BF16), ("o_proj.weight", E, P, BF16)]
        t += [("self_attn." + n, r, k, d) for n, r, k, d in a]
    if parts in ("all", "moe"):
        if dense:
            t += [("mlp.gate_proj.weight", c.dense_inter, E, FP8), ("mlp.up_proj.weight", c.dense_inter, E, FP8), ("mlp.down_proj.weight", E, c.dense_inter, FP8)]
        else:
            I, s = c.moe_inter, "mlp.shared_experts."
            t += [("mlp.gate.weight", c.n_experts, E, BF16), (s + "gate_proj.weight", I, E, FP8), (s + "up_proj.weight", I, E, FP8), (s + "down_proj.weight", E, I, FP8)]
    return t


def _vectors(c, mla, dense, parts):
    """[(name, length, mean, deviation)] of a layer's vectors."""
    E, MIX = c.hidden, (2 + c.hc_mult) * c.hc_mult
    t = []
    if parts == "all":
        t += [("input_layernorm.weight", E, 1.0, 0.02), ("post_attention_layernorm.weight", E, 1.0, 0.02)]
        for site in ("attn", "ffn"):
            t += [("hc_%s_base" % site, MIX, 0.0, 0.02), ("hc_%s_scale" % site, 3, 1.0, 0.0)]
    if parts in ("all", "attention"):
        if mla:
            a = [("q_a_layernorm.weight", c.q_lora, 1.0, 0.02), ("kv_a_layernorm.weight", c.kv_lora, 1.0, 0.02), ("indexer.k_norm.weight", c.index_dim, 1.0, 0.02),
                 ("indexer.k_norm.bias", c.index_dim, 0.0, 0.02), ("indexer.index_kpool_compress_ape", c.index_kpool * c.index_dim, 0.0, 0.02)]
        else:
            D, P = c.kda_head_dim, c.kda_heads * c.kda_head_dim
            a = [(n + "_conv1d.weight", P * c.conv_k, 0.0, 0.3) for n in "qkv"]
            a += [("A_log", c.kda_heads, 0.0, 0.02), ("dt_bias", P, 0.0, 0.02), ("o_norm.weight", D, 1.0, 0.02)]
        t += [("self_attn." + n, k, m, d) for n, k, m, d in a]
    if parts in ("all", "moe") and not dense:
        t.append(("mlp.gate.e_score_correction_bias", c.n_experts, 0.0, 0.1))
    return t


def _layers(parts, n_layers, mla):
    """(is_mla, is_dense) flags of the engine's layers."""
    if parts != "all":
        return [int(mla)], [0]
    return [int(i % 4 == 3) for i in range(n_layers)], [int(i < 3) for i in range(n_layers)]


def _config(parts, heads=64):
    c = _package().full_size_config()
    c.n_layers = LAYERS if parts == "all" else 1
    c.kda_heads = heads
    return c


def _build(parts, mla=False, heads=64, cap=CAP, bf16=False, sequences=1, context=0):
    """An engine with random weights: matrices ~ N(0, 0.02) generated in HBM (FP8: uniform codes whose block
    scales give the same magnitude), norms near 1, router bias ~ N(0, 0.1)."""
    pkg, c = _package(), _config(parts, heads)
    is_mla, is_dense = _layers(parts, c.n_layers, mla)
    eng = pkg.Engine(c, is_mla, is_dense, cap)
    for k, v in (("allow_partial", int(parts != "all")), ("latent_bf16", int(bf16)), ("sequences", sequences)):
        eng.set_option(k, v)
    rng = np.random.default_rng(WEIGHTS_SEED)
    unit, blocks = 1.0 / 37837.2, (c.fp8_block_r, c.fp8_block_c)
    scales = lambda *n: (0.02 / 100.058 * np.exp2(2.0 * rng.random(n) - 1.0)).astype(np.float32)  # noqa: E731

    def matrix(name, rows, cols, dt):
        if dt == BF16:
            eng.fill_matrix(name, BF16, WEIGHTS_SEED, rows, mul=0.02 * unit)
        else:
            eng.fill_matrix(name, FP8, WEIGHTS_SEED, rows, scale_inv=scales(-(-rows // blocks[0]), -(-cols // blocks[1])))

    def vector(name, n, mean, dev):
        eng.load(name, (mean + dev * rng.standard_normal((n, 1))).astype(np.float32), pkg.DT_F32)

    if parts == "all":
        matrix("embed_tokens.weight", c.vocab, c.hidden, BF16)
        matrix("lm_head.weight", c.vocab, c.hidden, BF16)
        vector("norm.weight", c.hidden, 1.0, 0.02)
    for i in range(c.n_layers):
        p = "layers.%d." % i
        for name, rows, cols, dt in _matrices(c, is_mla[i], is_dense[i], parts):
            matrix(p + name, rows, cols, dt)
        for name, n, mean, dev in _vectors(c, is_mla[i], is_dense[i], parts):
            vector(p + name, n, mean, dev)
        if parts in ("all", "moe") and not is_dense[i]:
            grid = scales(c.n_experts, 3, (c.moe_inter // blocks[0]) * (c.hidden // blocks[1]))
            for x in range(c.n_experts):
                eng.fill_expert(i, x, WEIGHTS_SEED, *grid[x])
    eng.finalize()
    if parts != "moe":
        eng.synth_session(WEIGHTS_SEED, context)
    return eng


_engines = weakref.WeakValueDictionary()


class _Shared:
    """An engine and what its states share: which sequence the next one takes."""

    def __init__(self, eng):
        self.eng, self.taken = eng, 0


def _shared(**how):
    key = tuple(sorted(how.items()))
    got = _engines.get(key)
    if got is None:
        got = _Shared(_build(**how))
        _engines[key] = got
    return got


# ------------------------------------------------------------------------- the contract ----
def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng([seed, 17])
    bf16 = bool(case.get("bf16"))
    s = dict(case, seed=seed)
    rows = lambda n: rng.standard_normal((n, 4096)).astype(np.float32)  # noqa: E731
    if kind == "moe":
        s["on"] = _shared(parts="moe", cap=64)
        s["x"] = rows(case["tokens"])
    elif kind == "kda":
        s["on"] = _shared(parts="attention", heads=case["heads"], cap=64)
        s["x"] = rows(case["tokens"])
    elif kind == "mla":
        s["on"] = _shared(parts="attention", mla=True, cap=CAP, bf16=bf16)
        s["x"] = rows(case["tokens"])
    else:
        vocab = _config("all").vocab
        if kind == "batch":
            s["on"] = _shared(parts="all", cap=8192, bf16=bf16, sequences=case["sequences"], context=case["context"])
        elif kind in ("prompt", "chat"):
            s["on"] = _shared(parts="all", cap=4096, bf16=bf16)
        else:
            s["on"] = _shared(parts="all", cap=CAP, bf16=bf16, sequences=SESSIONS, context=case["context"])
            s["sequence"] = s["on"].taken % SESSIONS
            s["on"].taken += 1
        s["ids"] = rng.integers(0, vocab, case.get("tokens", case.get("sequences", 1))).astype(np.int32)
    s["engine"] = s["on"].eng
    return s


def _room(s, n):
    """A session that is full starts over at its context."""
    eng = s["engine"]
    if eng.cached + n > (8192 if s["kind"] == "batch" else CAP):
        eng.synth_session(WEIGHTS_SEED, s["context"])


def run(s):
    eng, kind = s["engine"], s["kind"]
    if kind == "moe":
        return eng.op_moe(0, s["x"])
    if kind == "kda":
        return eng.op_kda(0, s["x"])
    if kind == "mla":
        out, sel = eng.op_mla(0, s["x"], s["context"])
        return [out] if sel is None else [out, sel]
    if kind == "prompt":
        eng.reset()
        return eng.forward(s["ids"])[0]
    if kind == "chat":
        eng.reset()
        logits, _ = eng.forward(s["ids"])
        return [logits, eng.decode_greedy(int(logits.argmax()), s["new"])]
    if kind == "batch":
        _room(s, 1)
        logits, tokens = eng.decode_batch(s["ids"], want_logits=s["logits"])
        return [logits, tokens] if s["logits"] else tokens
    eng.use_sequence(s["sequence"])
    _room(s, s.get("new", 1))
    if kind == "step":
        return eng.forward(s["ids"])[0]
    if kind == "greedy":
        return eng.decode_greedy(int(s["ids"][0]), s["new"])
    return eng.decode_sampled(int(s["ids"][0]), s["new"], 0.8, 0.95, s["seed"])


@functools.lru_cache(None)
def _distinct_experts(tokens):
    """Experts that `tokens` tokens reach in one layer, for router scores and bias of these weights' distribution."""
    c = _package().full_size_config()
    rng = np.random.default_rng(1)
    bias = 0.1 * rng.standard_normal(c.n_experts)
    z = 0.02 * np.sqrt(c.hidden) * rng.standard_normal((tokens, c.n_experts))
    top = np.argpartition(-(1.0 / (1.0 + np.exp(-z)) + bias), c.topk, axis=1)[:, :c.topk]
    return len(np.unique(top))


def work(case):
    """Every weight that the pass uses read once (once per token where tokens follow from each other), session
    state read and written, two operations per weight and token."""
    kind = case["kind"]
    parts = {"moe": "moe", "kda": "attention", "mla": "attention"}.get(kind, "all")
    c = _config(parts, case.get("heads", 64))
    is_mla, is_dense = _layers(parts, c.n_layers, kind == "mla")
    expert = 3 * c.moe_inter * c.hidden * (1 + 4 / (c.fp8_block_r * c.fp8_block_c))
    lat = 2 if case.get("bf16") else 4

    def one_pass(tokens, sessions, depth, heads_out):
        """`tokens` positions in all, `sessions` sessions that hold `depth` positions each."""
        size = flops = 0.0
        for i in range(c.n_layers):
            for _, rows, cols, dt in _matrices(c, is_mla[i], is_dense[i], parts):
                size += rows * cols * (2 if dt == BF16 else 1 + 4 / (c.fp8_block_r * c.fp8_block_c))
                flops += 2.0 * rows * cols * tokens
            if parts in ("all", "moe") and not is_dense[i]:
                size += _distinct_experts(tokens) * expert
                flops += 2.0 * c.topk * 3 * c.moe_inter * c.hidden * tokens
            if parts != "moe":
                new = tokens / sessions
                if is_mla[i]:
                    seen = min(c.index_topk + c.index_kpool - 1, depth + (new + 1) / 2)
                    size += sessions * (min(depth + new, new * seen) * c.kv_lora * lat)
                    flops += 4.0 * tokens * seen * c.kv_lora * c.mla_heads
                    if depth + new > c.index_topk + c.index_kpool:
                        pools = (depth + new) / c.index_kpool
                        size += sessions * pools * c.index_dim * 4
                        flops += 2.0 * tokens * pools * c.index_dim * c.index_heads
                else:
                    size += sessions * 8.0 * c.kda_heads * c.kda_head_dim ** 2
                    flops += 7.0 * tokens * c.kda_heads * c.kda_head_dim ** 2
        if parts == "all":
            size += 2.0 * c.vocab * c.hidden
            flops += 2.0 * c.vocab * c.hidden * heads_out
        else:
            size += 8.0 * tokens * c.hidden
        return size, flops

    if kind in ("moe", "kda"):
        size, flops = one_pass(case["tokens"], 1, 0, 0)
    elif kind == "mla":
        size, flops = one_pass(case["tokens"], 1, case["context"], 0)
    elif kind == "batch":
        size, flops = one_pass(case["sequences"], case["sequences"], case["context"], case["sequences"])
        size += 4.0 * c.vocab * case["sequences"] * case["logits"]
    else:
        size = flops = 0.0
        if kind in ("prompt", "chat"):
            size, flops = one_pass(case["tokens"], 1, 0, 1)
            size += 4.0 * c.vocab
        if kind != "prompt":
            n = case.get("new", 1)
            a, b = one_pass(1, 1, case.get("context", case.get("tokens")), 1)
            size, flops = size + n * a, flops + n * b
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """One layer: sums of a few thousand terms in 32 bits. The model: the 1e-3 on logits that the tests ask for (a
    BF16 cache entry or an expert choice on the edge can fall the other way); decoded tokens are the same."""
    kind = case["kind"]
    if kind == "moe":
        return {"rel": 1e-5}
    if kind == "kda":
        return {"rel": 2e-5}
    if kind == "mla":
        return {"rel": 1e-4 if case["bf16"] else 2e-5, "differ": 0.01}
    return {"rel": 1e-3, "differ": 0.01}
