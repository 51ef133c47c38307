"""The work whose speed is watched: whole calls of the Llama-style model and single layers of the
engine's designs, through the entry points that a program calls (``ModelRunner.step``, a part's
``forward``, ``Sampler.sample``).

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a
program has in hand before the call, ``run`` is one pass, ``work`` what the pass cannot do without,
``tolerance`` how far two correct implementations of the same precision may lie apart, and ``exact``
the same outputs from plain torch in 64 bits.

Sizes: Llama-3-8B and Llama-3.2-1B (``bench.py --sizes``) and the two layer sizes of ``bench.py
--compare`` (width 2,048 and 4,096).
"""

from __future__ import annotations

import math

import torch

from scratch_llm_b200.cache import CacheManager
from scratch_llm_b200.config import config_from_dict
from scratch_llm_b200.config.spec import PartSpec
from scratch_llm_b200.engine import ModelRunner, RowInput, build_model
from scratch_llm_b200.engine.batch import BatchStager, build_batch
from scratch_llm_b200.kernels import ops
from scratch_llm_b200.parts import (FEED_FORWARDS, MIXERS, POSITION_ENCODINGS, BuildContext,
                                    CacheView, make)
from scratch_llm_b200.sampling import Sampler, SamplingParams

DEV = "cuda"
PAGE = 64
MAX_POSITION = 8192
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

LLAMA_1B = dict(hidden_size=2048, num_hidden_layers=16, num_attention_heads=32,
                num_key_value_heads=8, head_dim=64, intermediate_size=8192, vocab_size=128256,
                rope_theta=500000.0, rms_norm_eps=1e-5, tie_word_embeddings=True,
                max_position_embeddings=MAX_POSITION)
#: layer sizes by width: attention heads / kv heads / head size, the delta rule's heads / key
#: heads, the width of a routed expert, the query latent
LAYER = {2048: dict(heads=32, kv=8, dim=64, delta=(16, 8), expert=2048, q_rank=1536),
         4096: dict(heads=32, kv=8, dim=128, delta=(32, 16), expert=3584, q_rank=3072)}
DELTA_DIM, CONV, RANK = 128, 4, 64
GENERAL_DIM = 64
KV_RANK, ROT = 192, 64
EXPERTS = 16
THETA = 500000.0
EPS = 1e-5


def _case(kind, width=0, rows=1, tokens=1, ragged=False, dtype="bfloat16", **more):
    return dict(kind=kind, width=width, rows=rows, tokens=tokens, ragged=ragged, dtype=dtype, **more)


def listed():
    return [
        # one user, a short question, the first tokens of the answer: latency and launches count
        dict(_case("generate", 2048, 1, 33), steps=8, name="generate_one_short"),
        # a small server: eight prompts of mixed lengths in one step, then decoding side by side
        dict(_case("generate", 2048, 8, 1023, True), steps=12, name="generate_eight_ragged"),
        # a prompt's attention layer, the long products and the causal attention
        dict(_case("attention", 4096, 1, 2048), name="attention_prompt"),
        # a decode step's attention layer in a busy server: long contexts of mixed lengths
        dict(_case("attention_decode", 4096, 64, 4000, True), name="attention_decode_64"),
        # the 32-bit mode, in which a model is checked against its training code
        dict(_case("attention", 2048, 1, 777, dtype="float32"), name="attention_prompt_32bit"),
        # recurrent layers with a delta rule, a prompt: one decay per head,
        dict(_case("delta", 2048, 1, 2048), name="delta_prompt"),
        # one decay per key channel, several prompts of mixed lengths in one step,
        dict(_case("delta_channels", 2048, 4, 1201, True), name="delta_channels_prompts"),
        # the generalized rule
        dict(_case("general_delta", 2048, 1, 2048), name="general_delta_prompt"),
        # recurrent decoding: eight tokens each for many requests that continue one state
        dict(_case("delta_decode", 4096, 48, 8), name="delta_decode_48"),
        # a mixture of experts on a prompt step
        dict(_case("routed", 2048, 1, 2048, top=3), name="routed_prompt"),
        # attention through latents, two prompts
        dict(_case("latent", 2048, 2, 1500, True), name="latent_prompts"),
        # the choice of the next tokens of a large batch, nucleus and temperature beside greedy rows
        dict(_case("sample", 0, 64, 1), vocab=128256, name="sample_64"),
    ]


def _between(rng, low, high):
    """A whole number, spread evenly over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["generate", "attention", "attention_decode", "attention_32", "delta",
                       "delta_channels", "general_delta", "delta_decode", "routed", "latent",
                       "sample"])
    rows = _between(rng, 1, 8)
    ragged = rng.random() < 0.6
    if kind == "generate":
        return dict(_case("generate", 2048, rows, _between(rng, 9, 1023), ragged),
                    steps=rng.randint(2, 12))
    if kind == "sample":
        return dict(_case("sample", 0, _between(rng, 1, 64), 1), vocab=_between(rng, 30000, 128256))
    if kind == "attention_32":
        return _case("attention", 2048, min(rows, 3), _between(rng, 5, 777) // min(rows, 3) + 1,
                     ragged, "float32")
    width = rng.choice([2048, 4096])
    if kind == "attention_decode":
        return _case(kind, width, _between(rng, 1, 64), _between(rng, 60, 4000), ragged)
    if kind == "delta_decode":
        return _case(kind, width, _between(rng, 1, 48), rng.randint(2, 8))
    tokens = max(2, _between(rng, 17, 2400) // rows + 1)
    dtype = "float32" if kind.endswith(("delta", "channels")) and width == 2048 \
        and rng.random() < 0.25 else "bfloat16"
    if dtype == "float32":
        tokens = min(tokens, max(2, 600 // rows))
    if kind == "routed":
        return dict(_case("routed", width, 1, tokens * rows), top=rng.randint(1, 4))
    return _case(kind, width, rows, tokens, ragged, dtype)


def _lengths(case):
    """Tokens of each row (of its context, for attention_decode): the longest first; ragged rows
    go down to about a third of it."""
    n, t = case["rows"], case["tokens"]
    return [max(1, t - (i * t * 2) // (3 * n)) if case["ragged"] else t for i in range(n)]


# ------------------------------------------------------------------------------------- inputs

def _generator(case, seed, what):
    g = torch.Generator(device=DEV)
    g.manual_seed((seed * 1000003 + sum(ord(c) * 31 ** i for i, c in enumerate(what))) % (1 << 62))
    return g


def _randn(case, seed, what, *shape, scale=1.0, dtype=None):
    x = torch.randn(*shape, generator=_generator(case, seed, what), device=DEV)
    return x.mul_(scale).to(dtype or DTYPES[case["dtype"]])


def _uniform(case, seed, what, *shape, low=0.0, high=1.0):
    x = torch.rand(*shape, generator=_generator(case, seed, what), device=DEV)
    return x.mul_(high - low).add_(low)


def _matrix(case, seed, what, n, k):
    return _randn(case, seed, what, n, k, scale=k ** -0.5)


def _gain(case, seed, what, *shape):
    return _randn(case, seed, what, *shape, scale=0.1, dtype=torch.float32) + 1.0


def _input(case, seed):
    """The layer's normed input."""
    n = case["rows"] if case["kind"] == "attention_decode" else sum(_lengths(case))
    if case["kind"] == "delta_decode":
        return _randn(case, seed, "x", case["tokens"], case["rows"], case["width"])
    return _randn(case, seed, "x", n, case["width"])


def _tables(dim):
    """cos and sin of 32-bit angles, as checkpoints are trained with."""
    inv = 1.0 / (THETA ** (torch.arange(0, dim, 2).float() / dim))
    a = torch.outer(torch.arange(MAX_POSITION).float(), inv)
    return a.cos(), a.sin()


def _attention_tensors(case, seed):
    s = LAYER[case["width"]]
    d, H, G, hd = case["width"], s["heads"], s["kv"], s["dim"]
    return {"q_proj.weight": _matrix(case, seed, "q", H * hd, d),
            "k_proj.weight": _matrix(case, seed, "k", G * hd, d),
            "v_proj.weight": _matrix(case, seed, "v", G * hd, d),
            "o_proj.weight": _matrix(case, seed, "o", d, H * hd)}


def _delta_tensors(case, seed):
    d = case["width"]
    H, G = LAYER[d]["delta"]
    D, V = DELTA_DIM, DELTA_DIM
    t = {"q": _matrix(case, seed, "q", G * D, d), "k": _matrix(case, seed, "k", G * D, d),
         "v": _matrix(case, seed, "v", H * V, d), "o": _matrix(case, seed, "o", d, H * V),
         "b": _matrix(case, seed, "b", H, d),
         "q.conv": _randn(case, seed, "qc", G * D, CONV, scale=0.5, dtype=torch.float32),
         "k.conv": _randn(case, seed, "kc", G * D, CONV, scale=0.5, dtype=torch.float32),
         "v.conv": _randn(case, seed, "vc", H * V, CONV, scale=0.5, dtype=torch.float32),
         # rates of 1 to 16 and step sizes of 0.001 to 0.1, evenly over the logarithm
         "A_log": _uniform(case, seed, "A", H, low=0.0, high=math.log(16.0)),
         "norm": _gain(case, seed, "norm", V)}
    n = H if case["kind"] != "delta_channels" else H * D
    step = _uniform(case, seed, "dt", n, low=math.log(1e-3), high=math.log(1e-1)).exp()
    t["dt_bias"] = torch.log(torch.expm1(step))
    if case["kind"] == "delta_channels":
        t["a1"], t["a2"] = _matrix(case, seed, "a1", RANK, d), _matrix(case, seed, "a2", H * D, RANK)
        t["g1"], t["g2"] = _matrix(case, seed, "g1", RANK, d), _matrix(case, seed, "g2", H * V, RANK)
    else:
        t["a"], t["g"] = _matrix(case, seed, "a", H, d), _matrix(case, seed, "g", H * V, d)
    return t


def _general_tensors(case, seed):
    d = case["width"]
    t = {n: _matrix(case, seed, n, d, d) for n in "rkvgoa"}
    t["a.b"] = _randn(case, seed, "ab", d, dtype=torch.float32)
    t["w1"], t["w2"] = _matrix(case, seed, "w1", RANK, d), _matrix(case, seed, "w2", d, RANK)
    # from decays of 0.56 to nearly 1
    t["w0"] = _uniform(case, seed, "w0", d, low=-6.0, high=1.0)
    t["norm"] = _gain(case, seed, "norm", d)
    return t


def _routed_tensors(case, seed):
    d, f = case["width"], LAYER[case["width"]]["expert"]
    t = {"router": _matrix(case, seed, "router", EXPERTS, d), "shared.sg": _matrix(case, seed, "sg", 1, d)}
    for p in [f"e{i}" for i in range(EXPERTS)] + ["shared"]:
        t[p + ".gate"] = _matrix(case, seed, p + "g", f, d)
        t[p + ".up"] = _matrix(case, seed, p + "u", f, d)
        t[p + ".down"] = _matrix(case, seed, p + "d", d, f)
    return t


def _latent_tensors(case, seed):
    s = LAYER[case["width"]]
    d, H, dim, Q = case["width"], s["heads"], s["dim"], s["q_rank"]
    return {"dq": _matrix(case, seed, "dq", Q, d), "dq.norm": _gain(case, seed, "dqn", Q),
            "uq": _matrix(case, seed, "uq", H * (dim + ROT), Q),
            "dkv": _matrix(case, seed, "dkv", KV_RANK + ROT, d),
            "dkv.norm": _gain(case, seed, "dkvn", KV_RANK),
            "uk": _matrix(case, seed, "uk", H * dim, KV_RANK),
            "uv": _matrix(case, seed, "uv", H * dim, KV_RANK),
            "g": _matrix(case, seed, "g", H, d), "o": _matrix(case, seed, "o", d, H * dim)}


def _llama_tensors(case, seed):
    c = LLAMA_1B
    d, f, hd = c["hidden_size"], c["intermediate_size"], c["head_dim"]
    H, G = c["num_attention_heads"], c["num_key_value_heads"]
    t = {"model.embed_tokens.weight": _randn(case, seed, "embed", c["vocab_size"], d, scale=0.02),
         "model.norm.weight": _gain(case, seed, "norm", d)}
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, n, k in (("self_attn.q_proj", H * hd, d), ("self_attn.k_proj", G * hd, d),
                           ("self_attn.v_proj", G * hd, d), ("self_attn.o_proj", d, H * hd),
                           ("mlp.gate_proj", f, d), ("mlp.up_proj", f, d), ("mlp.down_proj", d, f)):
            t[p + name + ".weight"] = _matrix(case, seed, p + name, n, k)
        for name in ("input_layernorm", "post_attention_layernorm"):
            t[p + name + ".weight"] = _gain(case, seed, p + name, d)
    return t


def _prompts(case, seed):
    """Per request: the prompt's tokens and the tokens that are fed after it."""
    g = torch.Generator().manual_seed(seed * 7919 + 1)
    return [torch.randint(0, LLAMA_1B["vocab_size"], (n + case["steps"],), generator=g).tolist()
            for n in _lengths(case)]


def _decode_context(case, seed):
    """The keys and values that earlier steps have left, per request [2, kv heads, context, dim]."""
    s = LAYER[case["width"]]
    return [_randn(case, seed, f"ctx{i}", 2, s["kv"], n, s["dim"])
            for i, n in enumerate(_lengths(case))]


def _sampling(case, seed):
    n = case["rows"]
    logits = _randn(case, seed, "logits", n, case["vocab"], scale=3.0, dtype=torch.float32)
    kinds = [SamplingParams(temperature=0.8, top_p=0.9), SamplingParams(temperature=1.0, top_p=0.95),
             SamplingParams(temperature=0.7), SamplingParams(temperature=0.0)]
    return logits, [kinds[i % 4] for i in range(n)], [seed * 64 + i for i in range(n)]


# ------------------------------------------------------------------------------------ prepare

def _rows_of(case, lengths, kv, state):
    """A cache with the case's requests admitted, and the batch of one step that brings each its
    next tokens."""
    pages = sum(-(-(n + 1) // PAGE) for n in lengths) + 1
    cache = CacheManager([kv], [state], PAGE, pages, case["rows"], dtype=DTYPES[case["dtype"]],
                         device=DEV)
    decode = case["kind"] in ("attention_decode", "delta_decode")
    for i, n in enumerate(lengths):
        cache.admit(i)
        if case["kind"] == "attention_decode":
            cache.reserve(i, n)
            cache.commit(i, n)
        cache.reserve(i, 1 if decode else n)
    batch = build_batch(cache, BatchStager(torch.device(DEV)),
                        [RowInput(i, [0] * (1 if decode else n)) for i, n in enumerate(lengths)],
                        2, MAX_POSITION)
    paged, group = cache.entry_pages(0)
    view = CacheView(pages=paged, page_size=PAGE, state=cache.states[0],
                     block_table=None if group is None else batch.block_tables[group])
    return cache, batch, view


def _mixer_spec(case):
    d, kind = case["width"], case["kind"]
    s = LAYER[d]
    if kind.startswith("attention"):
        return PartSpec("gqa_attention", dict(hidden_size=d, n_heads=s["heads"],
                                              n_kv_heads=s["kv"], head_dim=s["dim"],
                                              scale=s["dim"] ** -0.5)), s["dim"]
    if kind == "latent":
        return PartSpec("latent_attention", dict(
            hidden_size=d, n_heads=s["heads"], dim=s["dim"], rot_dim=ROT, value_dim=s["dim"],
            q_rank=s["q_rank"], kv_rank=KV_RANK, scale=(s["dim"] + ROT) ** -0.5, eps=EPS)), ROT
    if kind == "general_delta":
        return PartSpec("general_delta", dict(hidden_size=d, n_heads=d // GENERAL_DIM,
                                              key_dim=GENERAL_DIM, eps=EPS, decay_rank=RANK)), 0
    more = dict(decay_rank=RANK, gate_rank=RANK, gate_activation="sigmoid") \
        if kind == "delta_channels" else {}
    return PartSpec("gated_delta_rule", dict(
        hidden_size=d, n_heads=s["delta"][0], n_kv_heads=s["delta"][1], key_dim=DELTA_DIM,
        value_dim=DELTA_DIM, conv_taps=CONV, eps=EPS, **more)), 0


def _mixer_tensors(case, seed):
    kind = case["kind"]
    make_them = _attention_tensors if kind.startswith("attention") else _latent_tensors \
        if kind == "latent" else _general_tensors if kind == "general_delta" else _delta_tensors
    return make_them(case, seed)


def prepare(case, seed):
    kind = case["kind"]
    dtype = DTYPES[case["dtype"]]
    context = BuildContext(dtype=dtype, device=torch.device(DEV))
    with torch.no_grad():
        if kind == "sample":
            logits, params, seeds = _sampling(case, seed)
            ops.prepare([], verbose=False)
            return dict(case=case, logits=logits, params=params, seeds=seeds,
                        sampler=Sampler(torch.device(DEV)))
        if kind == "generate":
            cfg = config_from_dict({**LLAMA_1B, "architectures": ["LlamaForCausalLM"]})
            model = build_model(cfg)
            ops.prepare(model.head_dims(), verbose=False)
            model.load(_llama_tensors(case, seed), context)
            prompts = _prompts(case, seed)
            pages = sum(-(-(len(p) + 1) // PAGE) for p in prompts) + 8
            return dict(case=case, runner=ModelRunner(model, PAGE, pages, case["rows"]),
                        prompts=prompts)
        if kind == "routed":
            d = case["width"]
            part = make(FEED_FORWARDS, "feed_forward", PartSpec("routed_experts", dict(
                hidden_size=d, expert_size=LAYER[d]["expert"], experts=EXPERTS, top=case["top"],
                correction=False, shared_size=LAYER[d]["expert"], shared_gate=True)))
            ops.prepare([], verbose=False)
            ops.prepare_jobs(part.kernel_jobs(dtype), verbose=False)
            part.load(_routed_tensors(case, seed), context)
            return dict(case=case, part=part, x=_input(case, seed))
        spec, rotated = _mixer_spec(case)
        part = make(MIXERS, "mixer", spec)
        jobs = part.kernel_jobs(dtype) if hasattr(part, "kernel_jobs") else None
        ops.prepare([] if jobs else [part.head_dim], verbose=False)
        ops.prepare_jobs(jobs or [], verbose=False)
        part.load(_mixer_tensors(case, seed), context)
        position = None
        if rotated:
            position = make(POSITION_ENCODINGS, "position", PartSpec("rotary", dict(
                head_dim=rotated, theta=THETA, max_position=MAX_POSITION, interleaved=False)))
            position.load({}, context)
        lengths = _lengths(case)
        cache, batch, view = _rows_of(case, lengths, part.kv_spec(), part.state_spec())
        state = dict(case=case, part=part, x=_input(case, seed), cache=cache, batch=batch,
                     view=view, position=position)
        if kind == "attention_decode":
            for i, kv in enumerate(_decode_context(case, seed)):
                table = torch.tensor(cache.table_of(i, 0), device=DEV)
                pad = len(table) * PAGE - kv.shape[2]
                kv = torch.nn.functional.pad(kv, (0, 0, 0, pad))
                view.pages[table] = kv.unflatten(2, (len(table), PAGE)).permute(2, 0, 1, 3, 4)
        if kind == "delta_decode":
            state["start"] = _randn(case, seed, "S", *view.state[0].shape, dtype=torch.float32)
        return state


# ---------------------------------------------------------------------------------------- run

def _generate(state):
    """Prompts in one step, then one given token per request and step (the tokens are given, so
    that every pass does the same work); the logits after every request's last prompt token and
    after each given one."""
    runner, prompts, steps = state["runner"], state["prompts"], state["case"]["steps"]
    for i in range(len(prompts)):
        runner.admit(i)
    out = [runner.step([RowInput(i, p[:-steps], [len(p) - steps - 1])
                        for i, p in enumerate(prompts)])]
    for s in range(steps):
        out.append(runner.step([RowInput(i, [p[len(p) - steps + s]], [0])
                                for i, p in enumerate(prompts)]))
    for i in range(len(prompts)):
        runner.release(i)
    return torch.stack(out)


@torch.no_grad()
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "generate":
        return _generate(state)
    if kind == "sample":
        n = case["rows"]
        tokens, _ = state["sampler"].sample(state["logits"], state["params"], state["seeds"],
                                            [5] * n)
        return torch.tensor(tokens)
    if kind == "routed":
        return state["part"].forward(state["x"])
    part, x, batch, view = state["part"], state["x"], state["batch"], state["view"]
    if kind in ("attention", "attention_decode", "latent"):
        return part.forward(x, batch, view, True, state["position"])
    if kind == "delta_decode":
        # several continuations of stored states: put back, then a few tokens each
        view.state[0].copy_(state["start"])
        view.state[1].zero_()
        out = torch.stack([part.forward(x[t], batch, view, True, None) for t in range(len(x))])
        return [out, *view.state]
    # a prompt is fed to a request that has just been admitted, with clean states
    cache = state["cache"]
    for i in reversed(range(case["rows"])):
        cache.release(i)
    for i in range(case["rows"]):
        cache.admit(i)
    out = part.forward(x, batch, view, True, None)
    states = view.state if isinstance(view.state, tuple) else (view.state,)
    return [out, *states]


# --------------------------------------------------------------------------------------- work

def work(case):
    kind, d, lengths = case["kind"], case["width"], _lengths(case)
    size = 4 if case["dtype"] == "float32" else 2
    n = sum(lengths)
    if kind == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"] + 4 * case["rows"], "flops": 0}
    if kind == "generate":
        c = LLAMA_1B
        H, G, hd, L = (c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"],
                       c["num_hidden_layers"])
        layer = d * (2 * H + 2 * G) * hd + 3 * d * c["intermediate_size"]
        head = c["vocab_size"] * d
        steps, rows = case["steps"], case["rows"]
        seen = sum(t + s + 1 for t in lengths for s in range(steps))   # keys that decoding reads
        pairs = sum(t * (t + 1) / 2 for t in lengths) + seen
        return {"bytes": 2.0 * (L * layer + head) * (steps + 1)
                + L * 4.0 * G * hd * (seen + n) + 4.0 * c["vocab_size"] * rows * (steps + 1),
                "flops": 2.0 * L * layer * (n + rows * steps) + 2.0 * head * rows * (steps + 1)
                + 4.0 * L * H * hd * pairs}
    s = LAYER[d]
    if kind == "routed":
        f, pairs = s["expert"], n * case["top"]
        used = min(EXPERTS, pairs)
        return {"bytes": 2.0 * (3 * d * f * (used + 1) + 2 * n * d),
                "flops": 6.0 * d * f * (pairs + n) + 2.0 * n * d * EXPERTS}
    if kind in ("attention", "attention_decode"):
        H, G, hd = s["heads"], s["kv"], s["dim"]
        decode = kind == "attention_decode"
        m = case["rows"] if decode else n
        pairs = sum(t + 1 for t in lengths) if decode else sum(t * (t + 1) / 2 for t in lengths)
        weights = d * (2 * H + 2 * G) * hd
        stored = 2 * G * hd * (pairs if decode else n)     # keys and values read (or written)
        return {"bytes": size * (weights + 2.0 * m * d + stored),
                "flops": 2.0 * m * weights + 4.0 * H * hd * pairs}
    if kind == "latent":
        H, dim, Q, R = s["heads"], s["dim"], s["q_rank"], KV_RANK
        weights = d * (Q + R + ROT + H) + Q * H * (dim + ROT) + H * dim * d
        absorbed = 2 * H * dim * R
        pairs = sum(t * (t + 1) / 2 for t in lengths)
        # attention in whichever form needs less: over the latents, or with keys and values per head
        latents = 2.0 * H * (2 * R + ROT) * pairs
        heads = 2.0 * H * (2 * dim + ROT) * pairs
        return {"bytes": 2.0 * (weights + absorbed + 2 * n * d + n * (R + ROT)),
                "flops": 2.0 * n * weights + 2.0 * n * absorbed + min(latents, heads)}
    if kind == "general_delta":
        weights = 6.0 * d * d + 2 * RANK * d
        S = case["rows"] * d * GENERAL_DIM
        return {"bytes": size * (weights + 2.0 * n * d) + 8.0 * S,
                "flops": 2.0 * n * weights + 8.0 * n * d * GENERAL_DIM}
    H, G = s["delta"]
    D = DELTA_DIM
    low = kind == "delta_channels"
    weights = d * (2 * G * D + (2 if low else 3) * H * D + 2 * H)
    weights += 2 * RANK * (d + H * D) if low else 0
    S = case["rows"] * H * D * D
    steps = case["tokens"] if kind == "delta_decode" else 1
    m = case["rows"] * steps if kind == "delta_decode" else n
    return {"bytes": steps * (size * weights + 8.0 * S) + size * 2.0 * m * d,
            "flops": 2.0 * m * weights + 6.0 * m * H * D * D}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return {"rel": 0.0, "differ": 0.04}      # (a draw on the edge of the nucleus or of a token)
    if kind == "generate":
        return {"rel": 5e-2}                     # bfloat16 through sixteen layers
    if case["dtype"] == "float32":               # (a recurrence carries its roundings along)
        return {"rel": 6e-6 if kind == "attention" else 2e-5}
    return {"rel": 2e-2}


# -------------------------------------------------------------------------------------- exact

def _rms(x, gain):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + EPS) * gain


def _rotate(x, cos, sin, adjacent=False):
    """``x`` [tokens, heads, dim], tables [tokens, dim / 2]."""
    c, s = cos[:, None], sin[:, None]
    if adjacent:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _causal(q, k, v, scale):
    """``q`` [tokens, heads, dim], ``k`` and ``v`` [keys, kv heads, dim]; the queries are the last."""
    per = q.shape[1] // k.shape[1]
    n, m = q.shape[0], k.shape[0]
    hidden = torch.ones(n, m, dtype=torch.bool, device=q.device).triu(m - n + 1)
    out = torch.empty(n, q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // per].T * scale).masked_fill(hidden, -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, h // per]
    return out.flatten(1)


def _wide(tensors):
    return {k: v.double() for k, v in tensors.items()}


def _exact_attention(case, seed):
    s = LAYER[case["width"]]
    H, G, hd = s["heads"], s["kv"], s["dim"]
    w, x = _wide(_attention_tensors(case, seed)), _input(case, seed).double()
    cos, sin = (t.double().to(DEV) for t in _tables(hd))
    decode = case["kind"] == "attention_decode"
    context = _decode_context(case, seed) if decode else None
    out, a = [], 0
    for i, n in enumerate(_lengths(case)):
        m, p0 = (1, n) if decode else (n, 0)
        row = x[a:a + m]
        q, k, v = ((row @ w[p + "_proj.weight"].T).view(m, -1, hd) for p in "qkv")
        c, z = cos[p0:p0 + m], sin[p0:p0 + m]
        q, k = _rotate(q, c, z), _rotate(k, c, z)
        if decode:
            old = context[i].double().transpose(1, 2)
            k, v = torch.cat([old[0], k]), torch.cat([old[1], v])
        out.append(_causal(q, k, v, hd ** -0.5))
        a += m
    return torch.cat(out) @ w["o_proj.weight"].T


def _exact_latent(case, seed):
    s = LAYER[case["width"]]
    H, dim = s["heads"], s["dim"]
    w, x = _wide(_latent_tensors(case, seed)), _input(case, seed).double()
    cos, sin = (t.double().to(DEV) for t in _tables(ROT))
    out, a = [], 0
    for n in _lengths(case):
        row = x[a:a + n]
        q = (_rms(row @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(n, H, dim + ROT)
        kv = row @ w["dkv"].T
        c = _rms(kv[:, :KV_RANK], w["dkv.norm"])
        kr = _rotate(kv[:, None, KV_RANK:], cos[:n], sin[:n]).expand(n, H, ROT)
        k = torch.cat([(c @ w["uk"].T).view(n, H, dim), kr], -1)
        q = torch.cat([q[..., :dim], _rotate(q[..., dim:], cos[:n], sin[:n])], -1)
        o = _causal(q, k, (c @ w["uv"].T).view(n, H, dim), (dim + ROT) ** -0.5)
        out.append((o.view(n, H, dim) * torch.sigmoid(row @ w["g"].T)[..., None]).flatten(1))
        a += n
    return torch.cat(out) @ w["o"].T


def _unit(x):
    return x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)


def _delta_row(w, x, case, S, carried):
    """One request's tokens [n, d] from state S [H, V, D] and the convolution's last inputs."""
    H, G = LAYER[case["width"]]["delta"]
    D, n = DELTA_DIM, x.shape[0]
    raw = torch.cat([carried, x @ torch.cat([w["q"], w["k"], w["v"]]).T])
    taps = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]])
    act = torch.nn.functional.silu(sum(raw[j:j + n] * taps[:, j] for j in range(CONV)))
    q, k, v = act.split([G * D, G * D, H * D], 1)
    q = _unit(q.view(n, G, D)).repeat_interleave(H // G, 1) * D ** -0.5
    k = _unit(k.view(n, G, D)).repeat_interleave(H // G, 1)
    v = v.view(n, H, D)
    beta = torch.sigmoid(x @ w["b"].T)
    soft = torch.nn.functional.softplus
    if case["kind"] == "delta_channels":
        rate = soft(x @ w["a1"].T @ w["a2"].T + w["dt_bias"]).view(n, H, D)
        g = torch.exp(-torch.exp(w["A_log"])[:, None] * rate)
        gate = torch.sigmoid(x @ w["g1"].T @ w["g2"].T)
    else:
        g = torch.exp(-torch.exp(w["A_log"]) * soft(x @ w["a"].T + w["dt_bias"]))[..., None]
        gate = torch.nn.functional.silu(x @ w["g"].T)
    out = torch.empty_like(v)
    for t in range(n):
        S = S * g[t][:, None]
        u = beta[t][:, None] * (v[t] - (S @ k[t][..., None])[..., 0])
        S = S + u[..., None] * k[t][:, None]
        out[t] = (S @ q[t][..., None])[..., 0]
    o = _rms(out, w["norm"]).flatten(1) * gate
    return o @ w["o"].T, S, raw[n:]


def _exact_delta(case, seed):
    w, x = _wide(_delta_tensors(case, seed)), _input(case, seed).double()
    H, G = LAYER[case["width"]]["delta"]
    D = DELTA_DIM
    zero = torch.zeros(CONV - 1, (2 * G + H) * D, dtype=torch.float64, device=DEV)
    outs, states, carried, a = [], [], [], 0
    decode = case["kind"] == "delta_decode"
    if decode:
        start = _randn(case, seed, "S", case["rows"], H, D, D, dtype=torch.float32).double()
    for i, n in enumerate(_lengths(case)):
        row = x[:, i] if decode else x[a:a + n]
        # (requests are admitted in order and slots are handed out from the first one on)
        S = start[i] if decode else torch.zeros(H, D, D, dtype=torch.float64, device=DEV)
        o, S, c = _delta_row(w, row, case, S, zero)
        outs.append(o)
        states.append(S)
        carried.append(c)
        a += n
    out = torch.stack(outs, 1) if decode else torch.cat(outs)
    return [out, torch.stack(states), torch.stack(carried)]


def _exact_general(case, seed):
    w, x = _wide(_general_tensors(case, seed)), _input(case, seed).double()
    D, d = GENERAL_DIM, case["width"]
    H = d // D
    outs, states, a = [], [], 0
    for n in _lengths(case):
        row = x[a:a + n]
        r, k, v = ((row @ w[p].T).view(n, H, D) for p in "rkv")
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(row @ w["w1"].T) @ w["w2"].T
                                                          + w["w0"])).view(n, H, D)
        u = _unit(k)
        au = torch.sigmoid(row @ w["a"].T + w["a.b"]).view(n, H, D) * u
        S = torch.zeros(H, D, D, dtype=torch.float64, device=DEV)     # [value, key]
        o = torch.empty_like(v)
        for t in range(n):
            S = S * decay[t][:, None] - (S @ u[t][..., None]) * au[t][:, None] \
                + v[t][..., None] * k[t][:, None]
            o[t] = (S @ r[t][..., None])[..., 0]
        o = _rms(o, w["norm"].view(H, D)).flatten(1) * torch.sigmoid(row @ w["g"].T)
        outs.append(o @ w["o"].T)
        states.append(S)
        a += n
    return [torch.cat(outs), torch.stack(states)]


def _exact_routed(case, seed):
    w, x = _routed_tensors(case, seed), _input(case, seed).double()

    def expert(p, h):
        g, u, dn = (w[p + n].double() for n in (".gate", ".up", ".down"))
        return (torch.nn.functional.silu(h @ g.T) * (h @ u.T)) @ dn.T

    score = torch.softmax(x @ w["router"].double().T, -1)
    best, ids = score.topk(case["top"], -1)
    best = best / best.sum(-1, keepdim=True)
    out = torch.sigmoid(x @ w["shared.sg"].double().T) * expert("shared", x)
    for e in range(EXPERTS):
        at, place = (ids == e).nonzero(as_tuple=True)
        out.index_add_(0, at, expert(f"e{e}", x[at]) * best[at, place][:, None])
    return out


def _exact_generate(case, seed):
    c = LLAMA_1B
    w = _llama_tensors(case, seed)
    hd, steps = c["head_dim"], case["steps"]
    cos, sin = (t.double().to(DEV) for t in _tables(hd))
    embed = w["model.embed_tokens.weight"].double()
    outs = []
    for p in _prompts(case, seed):
        n = len(p)
        x = embed[torch.tensor(p, device=DEV)]
        for i in range(c["num_hidden_layers"]):
            t = lambda name: w[f"model.layers.{i}.{name}.weight"].double()  # noqa: E731
            h = _rms(x, t("input_layernorm"))
            q, k, v = ((h @ t(f"self_attn.{m}_proj").T).view(n, -1, hd) for m in "qkv")
            q, k = (_rotate(m, cos[:n], sin[:n], adjacent=True) for m in (q, k))
            x = x + _causal(q, k, v, hd ** -0.5) @ t("self_attn.o_proj").T
            h = _rms(x, t("post_attention_layernorm"))
            x = x + (torch.nn.functional.silu(h @ t("mlp.gate_proj").T)
                     * (h @ t("mlp.up_proj").T)) @ t("mlp.down_proj").T
        outs.append(_rms(x[n - steps - 1:], w["model.norm.weight"].double()) @ embed.T)
    return torch.stack(outs, 1)


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None                    # (draws: whole numbers that no formula gives in 64 bits)
    if kind == "generate":
        return _exact_generate(case, seed)
    if kind in ("attention", "attention_decode"):
        return _exact_attention(case, seed)
    if kind == "latent":
        return _exact_latent(case, seed)
    if kind == "routed":
        return _exact_routed(case, seed)
    if kind == "general_delta":
        return _exact_general(case, seed)
    return _exact_delta(case, seed)
