"""The work this engine is measured on: whole calls of the step function and the layers they are made of.

A case names a `kind` and its sizes:

    engine      requests through `ModelRunner.step` as the replay tool and the scheduler drive it: prompts in one step, then
                single tokens from captured steps, the logits of every wanted place returned
    gqa         grouped-query attention with rotary positions (the Llama layers)
    mlp         the gated feed-forward
    experts     routed experts beside a shared one
    bias        attention with a learned bias by distance and a gate a head
    gla         gated linear attention, a decay a key channel
    delta       the delta rule, a decay a key channel
    retention   linear attention with one fixed decay a head
    mamba2      the state-space mixer

Layers run through their registered part (`MIXERS`, `FEED_FORWARDS`) on a `StepContext`, as a block calls them.  Prompts run
eagerly, steps of single tokens from a CUDA graph, as the engine runs both.  Sizes are those of `bench.py`'s configurations;
weights are N(0, 0.02) as in the random-weights mode, with the decays and biases a trained layer would have.  A recurrence
starts from the state of a request in the middle of its text and leaves it updated, so that a pass is the next portion.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import rustinfer_b200.models.decoder  # noqa: F401  (registers the built-in parts)
from rustinfer_b200.engine.runner import ModelRunner, StepEntry
from rustinfer_b200.parts.base import (FEED_FORWARDS, MIXERS, BuildContext, FixedState, GroupStep, PagedKV,
                                       PagedLayerCache, StateLayerCache, StepContext, StepShape)
from rustinfer_b200.parts.spec import PartSpec
from rustinfer_b200.weights.random_init import write_random_model

STD = 0.02
PAGE = 16
VOCAB = 16384
LLAMA_ROPE = dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0, original_max_position_embeddings=8192)


def listed():
    return [
        # one conversation: a short prompt, then one token at a time; launches and latency decide
        dict(name="llama one request", kind="engine", family="llama", requests=1, prompt=32, tokens=24),
        # a batch of requests through layers without a fused chain: many small products a step
        dict(name="fotulix sixteen requests", kind="engine", family="fotulix", requests=16, prompt=300, tokens=16),
        # the prompt of the headline benchmark, attention layer of the 8B sizes
        dict(name="attention prompt 2048", kind="gqa", size="8b", dtype="bfloat16", requests=1, tokens=2048, past=0),
        # the headline decode: eight requests at 4,096 keys, 1B sizes
        dict(name="attention 8 tokens", kind="gqa", size="1b", dtype="bfloat16", requests=8, tokens=1, past=4095),
        # the 32-bit engine, which logits are checked against
        dict(name="attention fp32 prompt 300", kind="gqa", size="1b", dtype="float32", requests=1, tokens=300, past=0),
        # a feed-forward over a prompt
        dict(name="mlp prompt 2048", kind="mlp", size="1b", dtype="bfloat16", requests=1, tokens=2048, past=0),
        # experts in a decode step
        dict(name="experts 8 tokens", kind="experts", size="w1024", dtype="bfloat16", requests=8, tokens=1, past=0),
        # a family's attention over a prompt, with the bias by distance
        dict(name="biased attention prompt 2048", kind="bias", size="w2048", dtype="bfloat16", requests=1, tokens=2048, past=0),
        # recurrences over prompts: one long one, ragged ones side by side, two, one
        dict(name="gated linear prompt 2048", kind="gla", size="w2048", dtype="bfloat16", requests=1, tokens=2048, past=0),
        dict(name="delta rule ragged prompts", kind="delta", size="w2048", dtype="bfloat16", requests=4, tokens=611, past=0),
        dict(name="retention two prompts", kind="retention", size="w2048", dtype="bfloat16", requests=2, tokens=1000, past=0),
        dict(name="state space prompt 2048", kind="mamba2", size="w1024", dtype="bfloat16", requests=1, tokens=2048, past=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["engine", "engine", "gqa", "gqa", "mlp", "experts", "bias", "gla", "delta", "retention", "mamba2"])
    if kind == "engine":
        requests, family = _log(rng, 1, 24), rng.choice(["llama", "fotulix"])
        return dict(kind=kind, family=family, requests=requests, tokens=rng.randint(4, 24),
                    prompt=_log(rng, 1, min(1500, (1400 if family == "llama" else 4000) // requests)))
    size = rng.choice(["1b", "8b"]) if kind in ("gqa", "mlp") else rng.choice(["w1024", "w2048"])
    if rng.random() < 0.3:                                   # a step of single tokens
        return dict(kind=kind, size=size, dtype="bfloat16", requests=_log(rng, 1, 64), tokens=1,
                    past=_log(rng, 16, 4095) if kind in ("gqa", "bias") else 0)
    if rng.random() < 0.12:                                  # the 32-bit engine
        return dict(kind=kind, size="1b" if kind in ("gqa", "mlp") else "w1024", dtype="float32", requests=rng.randint(1, 3),
                    tokens=_log(rng, 2, 100), past=0)
    requests = rng.choice([1, 1, 2, 3, 5])
    tokens = _log(rng, 2, (1200 if kind == "mlp" and size == "8b" else 2048) // requests)
    past = rng.choice([0, 0, _log(rng, 16, 1024)]) if kind in ("gqa", "bias") else 0
    return dict(kind=kind, size=size, dtype="bfloat16", requests=requests, tokens=tokens, past=past)


# ------------------------------------------------------------------------------------------------- sizes
_GQA = {"1b": (2048, 32, 8, 64), "8b": (4096, 32, 8, 128)}                       # hidden, heads, kv heads, head size
_MLP = {"1b": (2048, 8192), "8b": (4096, 14336)}
_EXPERTS = {"w1024": (1024, 768, 1024), "w2048": (2048, 1536, 2048)}             # width, expert, shared
_BIAS = {"w1024": (1024, 16, 4, 64), "w2048": (2048, 32, 8, 64)}
_GLA = {"w1024": (1024, 4, 128, 256), "w2048": (2048, 8, 128, 256)}              # width, heads, key, value
_DELTA = {"w1024": (1024, 8, 128), "w2048": (2048, 16, 128)}
_RETENTION = {"w1024": (1024, 8, 128), "w2048": (2048, 16, 128)}
_MAMBA = {"w1024": (1024, 32, 64, 128, 4, 4), "w2048": (2048, 64, 64, 128, 8, 8)}  # width, heads, value, state, groups, norm parts
RANK, TAPS, EXPERTS, TOP, GROUPS, KEEP, BUCKETS, FAR = 16, 4, 32, 4, 8, 4, 32, 128.0


def _lengths(case):
    """Tokens of every request: a few more or less than `tokens` each where there are several prompts."""
    n, t = case["requests"], case["tokens"]
    if t == 1 or n == 1:
        return [t] * n
    return [max(1, t + (i - n // 2) * (t // (2 * n)) - i % 2) for i in range(n)]


def _spec(case):
    kind, size = case["kind"], case["size"]
    if kind == "gqa":
        d, h, g, hd = _GQA[size]
        return PartSpec("gqa_attention", dict(hidden_size=d, num_heads=h, num_kv_heads=g, head_dim=hd, scale=hd ** -0.5, window=None,
                                              position=PartSpec("rope", dict(head_dim=hd, rotary_dim=hd, theta=500000.0, scaling=LLAMA_ROPE))))
    if kind == "mlp":
        d, ff = _MLP[size]
        return PartSpec("swiglu", dict(hidden_size=d, intermediate_size=ff))
    if kind == "experts":
        d, ff, shared = _EXPERTS[size]
        return PartSpec("routed_experts", dict(hidden_size=d, expert_ff=ff, experts=EXPERTS, top=TOP, groups_count=GROUPS, groups_keep=KEEP,
                                               shared_ff=shared, score="softmax", group_score="max", shared_gate=True, renormalize=True))
    if kind == "bias":
        d, h, g, hd = _BIAS[size]
        return PartSpec("distance_bias_attention", dict(hidden_size=d, num_heads=h, num_kv_heads=g, head_dim=hd, scale=hd ** -0.5,
                                                        bias="buckets", bias_far=FAR, head_gate=True))
    if kind == "gla":
        d, h, dk, dv = _GLA[size]
        return PartSpec("gated_linear_attention", dict(hidden_size=d, num_heads=h, key_dim=dk, value_dim=dv, tau=16.0, norm_eps=1e-6, decay_rank=RANK))
    if kind == "delta":
        d, h, dk = _DELTA[size]
        return PartSpec("delta_rule", dict(hidden_size=d, num_heads=h, key_dim=dk, norm_eps=1e-6, decay_rank=RANK))
    if kind == "retention":
        d, h, dk = _RETENTION[size]
        return PartSpec("retention", dict(hidden_size=d, num_heads=h, key_dim=dk, decay=_fixed_decays(h), norm_eps=1e-6,
                                          position=PartSpec("rope", dict(head_dim=dk, rotary_dim=dk, theta=10000.0, scaling=None))))
    d, h, vd, n, g, parts = _MAMBA[size]
    return PartSpec("mamba2", dict(hidden_size=d, num_heads=h, value_dim=vd, state_dim=n, groups=g, conv_taps=TAPS, norm_groups=parts, norm_eps=1e-6))


def _fixed_decays(heads):
    return [1.0 - 2.0 ** (-5.0 - 7.0 * i / max(1, heads - 1)) for i in range(heads)]


def _weights(part, case, gen):
    """The part's tensors on the GPU, in the engine's dtype."""
    dev, dt = torch.device("cuda:0"), getattr(torch, case["dtype"])
    rnd = lambda shape: torch.randn(shape, generator=gen, device=dev)
    uni = lambda shape, lo, hi: torch.rand(shape, generator=gen, device=dev) * (hi - lo) + lo
    out = {}
    for name, decl in part.param_decls().items():
        shape = tuple(BUCKETS if n == -1 else n for n in decl.shape)
        if name == "rel":
            t = rnd(shape)
        elif name == "conv":
            t = rnd(shape) * 0.4
        elif name == "a2.b":
            t = uni(shape, 0.0, 5.0)                         # decays of 0.957 to 0.9996 a token
        elif name == "w0":
            t = uni(shape, -6.0, 0.0)
        elif name == "dt_bias":
            t = torch.log(torch.expm1(torch.exp(uni(shape, math.log(1e-3), math.log(0.1)))))
        elif name == "A_log":
            t = torch.log(uni(shape, 1.0, 16.0))
        elif decl.init == "ones":
            t = 1.0 + 0.1 * rnd(shape)
        elif decl.init == "zeros":
            t = 0.1 * rnd(shape)
        else:
            t = rnd(shape) * STD
        out[name] = t.to(dt)
    return out


# ------------------------------------------------------------------------------------------------- engine
_FOLDERS = {}


def _folder(family):
    if family not in _FOLDERS:
        if family == "llama":
            cfg = dict(architectures=["LlamaForCausalLM"], model_type="llama", num_hidden_layers=2, hidden_size=2048, num_attention_heads=32,
                       num_key_value_heads=8, head_dim=64, intermediate_size=8192, vocab_size=VOCAB, rope_theta=500000.0, rope_scaling=LLAMA_ROPE,
                       rms_norm_eps=1e-5, tie_word_embeddings=True, max_position_embeddings=131072)
        else:
            attn = {"type": "attention", "mlp": {"kind": "dense", "ff": 4096},
                    "mixer": {"heads": 16, "kv_heads": 4, "dim": 64, "vdim": 64, "scale": 0.125, "bias_max": 128, "q_temp": {"coef": 0.1, "every": 1024}}}
            latent = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 4096},
                      "mixer": {"heads": 16, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 128, "scale": 96 ** -0.5, "mask": {"size": 1024},
                                "rot": {"dims": 32, "base": 10000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
            rotary = {"type": "attention_2", "mlp": {"kind": "dense", "ff": 4096},
                      "mixer": {"heads": 8, "kv_heads": 2, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": {
                          "dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
            cfg = {"architecture": "Fotulix", "width": 1024, "vocab": VOCAB, "norm": {"eps": 1e-6}, "residual_mult": 0.5,
                   "embedding": {"scale": 1.0, "bigram": {"buckets": 8191, "mul_prev": 40503, "mul_cur": 9973}}, "token_side": {"dim": 128},
                   "layers": [attn, latent, rotary]}
        place = tempfile.TemporaryDirectory(prefix=f"cases_{family}_")
        write_random_model(os.path.join(place.name, "model"), cfg, seed=2, std=STD, dtype="bfloat16")
        _FOLDERS[family] = place
    return os.path.join(_FOLDERS[family].name, "model")


def _replay(runner, prompts, later):
    """Prompts in one step, then the given tokens one step at a time: fp32 logits [steps, requests, vocab]."""
    n = len(prompts)
    for i in range(n):
        runner.open(i)
    logits = [runner.step([StepEntry(i, prompts[i], (len(prompts[i]) - 1,)) for i in range(n)])]
    for row in later:
        logits.append(runner.step([StepEntry(i, (row[i],), (0,)) for i in range(n)]))
    for i in range(n):
        runner.close(i)
    return torch.stack(logits)


# ------------------------------------------------------------------------------------------------- a layer and its step
def _context(case, part, gen):
    dev, dt = torch.device("cuda:0"), getattr(torch, case["dtype"])
    lens, past, n = np.array(_lengths(case)), case["past"], case["requests"]
    pos0 = np.full(n, past, dtype=np.int64)
    cu = np.concatenate([[0], np.cumsum(lens)])
    T = int(cu[-1])
    pages = -(-(past + int(lens.max())) // PAGE)
    entry = np.repeat(np.arange(n), lens)
    positions = np.arange(T) - cu[entry] + past
    table = torch.randperm(n * pages, generator=torch.Generator().manual_seed(int(T))).numpy().reshape(n, pages)
    slots = np.arange(n)[::-1].copy()
    i32 = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.int32, device=dev)
    shape = StepShape(lens, pos0, cu, pos0 + lens, slots)
    indices = {need.key: tuple(i32(a) for a in need.build(shape)) for need in (part.step_indices() if hasattr(part, "step_indices") else ())}
    group = GroupStep(i32(table), i32(table[entry, positions // PAGE] * PAGE + positions % PAGE))
    step = StepContext(T, n, i32(np.zeros(T)), i32(positions), i32(cu), i32(pos0 + lens), i32(slots), [group], [], int(lens.max()),
                       past + int(lens.max()), bool((lens == 1).all()), indices)
    caches = []
    needs = part.cache_need() if hasattr(part, "cache_need") else None
    for need in needs if isinstance(needs, tuple) else (needs,) if needs is not None else ():
        if isinstance(need, PagedKV):
            kv = torch.randn((n * pages, 2, need.num_kv_heads, PAGE, need.head_dim), generator=gen, device=dev).to(dt)
            caches.append(PagedLayerCache(kv, 0, True))
        elif isinstance(need, FixedState):
            caches.append(StateLayerCache(0.3 * torch.randn((n,) + tuple(need.shape), generator=gen, device=dev)))
    cache = caches[0] if len(caches) == 1 else tuple(caches) if caches else None
    return step, cache, table, slots


def _build(case, seed):
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + 13)
    registry = FEED_FORWARDS if case["kind"] in ("mlp", "experts") else MIXERS
    part = registry.build(_spec(case))
    longest = case["past"] + max(_lengths(case))
    part.prepare(BuildContext(dev, getattr(torch, case["dtype"]), -(-longest // PAGE) * PAGE, PAGE, max_batch_seqs=max(4, case["requests"])))
    weights = _weights(part, case, gen)
    part.load(weights)
    step, cache, table, slots = _context(case, part, gen)
    x = torch.randn((step.num_tokens, part.hidden), generator=gen, device=dev).to(getattr(torch, case["dtype"]))
    return dict(part=part, weights=weights, step=step, cache=cache, table=table, slots=slots, x=x)


def _forward(s):
    if s["cache"] is None:
        return s["part"].forward(s["x"], s["step"])
    return s["part"].forward(s["x"], s["step"], s["cache"])


def prepare(case, seed):
    if case["kind"] == "engine":
        longest = case["prompt"] + case["tokens"] + 1
        rng = np.random.RandomState(seed % (1 << 31))
        runner = ModelRunner(_folder(case["family"]), dtype="bfloat16", max_model_len=-(-longest // PAGE) * PAGE, page_size=PAGE,
                             max_batch_seqs=case["requests"], max_batch_tokens=max(512, case["requests"] * case["prompt"]),
                             num_pages=case["requests"] * -(-longest // PAGE), capture_sizes=[case["requests"]])
        ids = lambda n: [int(t) for t in rng.randint(0, VOCAB, n)]
        s = dict(runner=runner, prompts=[ids(case["prompt"]) for _ in range(case["requests"])], later=[ids(case["requests"]) for _ in range(case["tokens"])])
        _replay(runner, [p[:2] for p in s["prompts"]], s["later"][:1])   # the step is captured before requests come
        return s
    s = _build(case, seed)
    if case["tokens"] == 1:                                  # a step of single tokens: captured once, then replayed
        states = [c.state for c in _caches(s) if isinstance(c, StateLayerCache)]
        kept = [t.clone() for t in states]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _forward(s)
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = _forward(s)
        for t, was in zip(states, kept):
            t.copy_(was)
    s.pop("weights")
    return s


def _caches(s):
    c = s["cache"]
    return c if isinstance(c, tuple) else () if c is None else (c,)


def run(state):
    if "runner" in state:
        return _replay(state["runner"], state["prompts"], state["later"])
    if "graph" in state:
        state["graph"].replay()
        out = state["out"]
    else:
        out = _forward(state)
    return [out] + [c.state for c in _caches(state) if isinstance(c, StateLayerCache)]


# ------------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "engine":
        n, p, t = case["requests"], case["prompt"], case["tokens"]
        if case["family"] == "llama":
            layer = 2048 * (3072 + 2048) + 3 * 2048 * 8192
            weights, head, kv, att = 2 * layer, 2048 * VOCAB, 2 * 2 * 512, 2 * 2048 * 2
        else:
            mixers = 1024 * (1536 + 16 + 1024) + 1024 * (1536 + 160 + 16) + 2 * 16 * 64 * 128 + 1024 * 1024 + 1024 * (1536 + 8 + 1024)
            weights, head, kv, att = mixers + 3 * (3 * 1024 * 4096 + 2 * 128 * 1024), 1024 * VOCAB, 512 + 512 + 160, 2 * 1024 * 2 + 16 * 288
        keys = n * (p * p / 2 + sum(p + i + 1 for i in range(t)))
        flops = 2.0 * weights * n * (p + t) + 2.0 * head * n * (t + 1) + 2.0 * att * keys
        moved = (t + 1) * 2.0 * (weights + head) + 2.0 * kv * n * (2 * p + sum(p + i + 1 for i in range(t))) + 8.0 * n * (t + 1) * VOCAB
        return dict(bytes=moved, flops=flops)
    e = 2 if case["dtype"] == "bfloat16" else 4
    lens, past = _lengths(case), case["past"]
    T = sum(lens)
    pairs = sum(l * past + l * (l + 1) / 2 for l in lens)    # (query, key) pairs
    if kind == "gqa" or kind == "bias":
        d, h, g, hd = (_GQA if kind == "gqa" else _BIAS)[case["size"]]
        rows = (h + 2 * g) * hd + (h if kind == "bias" else 0)
        w = d * rows + d * h * hd
        moved = e * (w + T * d + 2 * g * hd * (sum(lens) + case["requests"] * past + T)) + (e if kind == "gqa" else 4) * T * d
        return dict(bytes=float(moved), flops=2.0 * w * T + 4.0 * h * hd * pairs)
    if kind == "mlp":
        d, ff = _MLP[case["size"]]
        return dict(bytes=float(e * (3 * d * ff + 2 * T * d)), flops=6.0 * d * ff * T)
    if kind == "experts":
        d, ff, shared = _EXPERTS[case["size"]]
        used = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** T)
        return dict(bytes=float(e * 3 * d * (ff * used + shared) + 4 * d * (EXPERTS + 1) + T * d * (e + 4)),
                    flops=6.0 * T * d * (TOP * ff + shared) + 2.0 * T * d * (EXPERTS + 1))
    if kind == "mamba2":
        d, h, vd, n, g, _ = _MAMBA[case["size"]]
        w = d * (2 * h * vd + 2 * g * n + h) + d * h * vd
        state, walk = h * vd * n, 4.0 * h * vd * n
    elif kind == "gla":
        d, h, dk, dv = _GLA[case["size"]]
        w = d * (2 * h * dk + 2 * h * dv) + RANK * (d + h * dk) + d * h * dv
        state, walk = h * dk * dv, 4.0 * h * dk * dv
    else:
        d, h, dk = (_DELTA if kind == "delta" else _RETENTION)[case["size"]]
        w = d * h * dk * (6 if kind == "delta" else 5) + (RANK * (d + h * dk) if kind == "delta" else 0)
        state, walk = h * dk * dk, (8.0 if kind == "delta" else 4.0) * h * dk * dk
    out = 4 if kind in ("mamba2", "retention") else e
    return dict(bytes=float(e * w + T * d * (e + out) + 8 * state * case["requests"]), flops=2.0 * w * T + walk * T)


def tolerance(case):
    """Relative error between two correct orders of the sums: bf16 roundings of activations that fall the other way in a
    layer, and in the engine the same carried through its layers (a split sum met in another order moved the logits by up
    to 2.5e-3); 32-bit sums in the 32-bit engine, whose recurrences add up hundreds of terms of either sign."""
    if case["kind"] == "engine":
        return {"rel": 1e-2, "max": 0.2}
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 8e-3, "max": 0.3}


# ------------------------------------------------------------------------------------------------- in 64 bits
def _rotate(x, positions, scaling, theta):
    """Pairs (i, i + half) of the last axis turned by position * frequency; llama3's bands where scaling is given."""
    hd = x.shape[-1]
    half = hd // 2
    f = theta ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / hd)
    if scaling:
        wave = 2.0 * math.pi / f
        long_wave, short_wave = scaling["original_max_position_embeddings"] / scaling["low_freq_factor"], scaling["original_max_position_embeddings"] / scaling["high_freq_factor"]
        blend = (scaling["original_max_position_embeddings"] / wave - scaling["low_freq_factor"]) / (scaling["high_freq_factor"] - scaling["low_freq_factor"])
        mixed = (1.0 - blend) * f / scaling["factor"] + blend * f
        f = torch.where(wave < short_wave, f, torch.where(wave > long_wave, f / scaling["factor"], mixed))
    angle = positions.double()[:, None, None] * f
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


def _bucket(distance, rows, far):
    """Distances below half of the rows have a row each; beyond, rows are equal steps of the logarithm up to `far`."""
    near = rows // 2
    d = distance.double().clamp(min=near)
    # as the mixer's table is defined: near + floor(log(d / near) / log(far / near) * (rows - near)), at most the last
    step = torch.floor(torch.log(d / near) / math.log(far / near) * (rows - near) + 1e-12).long() + near
    return torch.where(distance < near, distance, step.clamp(max=rows - 1))


def _attend(s, case, w, q, k, v, h, g, hd, bias=None, gate=None):
    """q [T, h, hd], k, v [T, g, hd] of this step over the cache's earlier keys; [T, h, hd]."""
    out, at, past = torch.empty_like(q), 0, case["past"]
    kv = s["cache"].kv
    for i, n in enumerate(_lengths(case)):
        kk, vv = k[at: at + n], v[at: at + n]
        if past:
            pages = torch.as_tensor(s["table"][i], device=q.device)
            old = kv[pages].double().permute(1, 2, 0, 3, 4).reshape(2, g, -1, hd)[:, :, :past].transpose(1, 2)
            kk, vv = torch.cat([old[0], kk]), torch.cat([old[1], vv])
        far = torch.arange(past, past + n, device=q.device)[:, None] - torch.arange(past + n, device=q.device)[None]
        for head in range(h):
            sc = q[at: at + n, head] @ kk[:, head // (h // g)].T * hd ** -0.5
            if bias is not None:
                sc = sc + bias[_bucket(far.clamp(min=0), bias.shape[0], FAR), head]
            o = torch.softmax(sc.masked_fill(far < 0, -math.inf), dim=-1) @ vv[:, head // (h // g)]
            out[at: at + n, head] = o if gate is None else o * torch.sigmoid(gate[at: at + n, head, None])
        at += n
    return out


def _head_rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _walk(case, s, which, H, dk, dv, token):
    """The recurrence of every request from the state it has; `token(S, t) -> (S, o)`; (o [T, H, dv], states as stored)."""
    cache = _caches(s)[which]
    state, outs, at = cache.state.double(), [], 0
    for i, n in enumerate(_lengths(case)):
        slot = int(s["slots"][i])
        S = state[slot, :, :, :dk].transpose(1, 2).clone()   # [H, dk, dv]
        for t in range(at, at + n):
            S, o = token(S, t)
            outs.append(o)
        state[slot, :, :, :dk] = S.transpose(1, 2)
        at += n
    return torch.stack(outs), state


def exact(case, seed):
    kind = case["kind"]
    if kind == "engine":
        return None
    s = _build(case, seed)
    W = {k: t.double() for k, t in s["weights"].items()}
    x = s["x"].double()
    T = x.shape[0]
    pos = s["step"].positions
    silu = torch.nn.functional.silu
    if kind == "gqa":
        d, h, g, hd = _GQA[case["size"]]
        q, k, v = (x @ W[n + "_proj.weight"].T for n in "qkv")
        q = _rotate(q.view(T, h, hd), pos, LLAMA_ROPE, 500000.0)
        k = _rotate(k.view(T, g, hd), pos, LLAMA_ROPE, 500000.0)
        return [_attend(s, case, W, q, k, v.view(T, g, hd), h, g, hd).reshape(T, -1) @ W["o_proj.weight"].T]
    if kind == "bias":
        d, h, g, hd = _BIAS[case["size"]]
        q, k, v, gate = (x @ W[n].T for n in ("q", "k", "v", "g"))
        o = _attend(s, case, W, q.view(T, h, hd), k.view(T, g, hd), v.view(T, g, hd), h, g, hd, bias=W["rel"], gate=gate)
        return [o.reshape(T, -1) @ W["o"].T]
    if kind == "mlp":
        return [(silu(x @ W["gate_proj.weight"].T) * (x @ W["up_proj.weight"].T)) @ W["down_proj.weight"].T]
    if kind == "experts":
        score = torch.softmax(x @ W["router"].T, dim=-1)
        groups = score.view(T, GROUPS, -1)
        best = groups.max(-1).values.topk(KEEP, dim=-1).indices
        allowed = torch.zeros(T, GROUPS, dtype=torch.bool, device=x.device).scatter_(1, best, True)
        score = score * allowed[:, :, None].expand_as(groups).reshape(T, -1)
        weight, ids = score.topk(TOP, dim=-1)
        weight = weight / weight.sum(-1, keepdim=True)
        ffn = lambda rows, p: (silu(rows @ W[p + "gate"].T) * (rows @ W[p + "up"].T)) @ W[p + "down"].T
        y = torch.sigmoid(x @ W["shared.sg"].T) * ffn(x, "shared.")
        for e in range(EXPERTS):
            row, choice = torch.nonzero(ids == e, as_tuple=True)
            if row.numel():
                y[row] += weight[row, choice, None] * ffn(x[row], f"e{e}.")
        return [y]
    if kind == "gla":
        d, H, dk, dv = _GLA[case["size"]]
        q, k, v, g = (x @ W[n].T for n in "qkvg")
        a = torch.sigmoid((x @ W["a1"].T) @ W["a2"].T + W["a2.b"]).view(T, H, dk) ** (1.0 / 16.0)
        q, k, v = q.view(T, H, dk) * dk ** -0.5, k.view(T, H, dk), v.view(T, H, dv)

        def token(S, t):
            S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
            return S, (S * q[t][:, :, None]).sum(1)
        o, state = _walk(case, s, 0, H, dk, dv, token)
        y = _head_rms(o, 1e-6) * W["norm"] * silu(g.view(T, H, dv))
        return [y.reshape(T, -1) @ W["o"].T, state]
    if kind == "delta":
        d, H, dk = _DELTA[case["size"]]
        r, k, v, g, a = ((x @ W[n].T).view(T, H, dk) for n in "rkvga")
        rate = torch.sigmoid(a + W["a.b"].view(H, dk))
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(x @ W["w1"].T) @ W["w2"].T + W["w0"])).view(T, H, dk)
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)

        def token(S, t):
            dot = (S * u[t][:, :, None]).sum(1)
            S = decay[t][:, :, None] * S - (rate[t] * u[t])[:, :, None] * dot[:, None] + k[t][:, :, None] * v[t][:, None]
            return S, (S * r[t][:, :, None]).sum(1)
        o, state = _walk(case, s, 0, H, dk, dk, token)
        y = _head_rms(o, 1e-6) * W["norm"].view(H, dk) * torch.sigmoid(g)
        return [y.reshape(T, -1) @ W["o"].T, state]
    if kind == "retention":
        d, H, dk = _RETENTION[case["size"]]
        q, k, v, g = ((x @ W[n].T).view(T, H, dk) for n in "qkvg")
        q, k = _rotate(q, pos, None, 10000.0) * dk ** -0.5, _rotate(k, pos, None, 10000.0)
        a = torch.tensor(_fixed_decays(H), dtype=torch.float64, device=x.device)[:, None, None]

        def token(S, t):
            S = a * S + k[t][:, :, None] * v[t][:, None]
            return S, (S * q[t][:, :, None]).sum(1)
        o, state = _walk(case, s, 0, H, dk, dk, token)
        return [(_head_rms(o, 1e-6) * silu(g)).reshape(T, -1) @ W["o"].T, state]
    d, H, vd, N, G, parts = _MAMBA[case["size"]]
    I, C = H * vd, H * vd + 2 * G * N
    proj = x @ W["in"].T
    z, raw, dt = proj[:, :I], proj[:, I: I + C], proj[:, I + C:]
    before, conv, at = s["cache"][0].state.double(), torch.empty_like(raw), 0
    for i, n in enumerate(_lengths(case)):
        slot = int(s["slots"][i])
        rows = torch.cat([before[slot], raw[at: at + n]])
        conv[at: at + n] = sum(rows[j: j + n] * W["conv"][:, j] for j in range(TAPS)) + W["conv.b"]
        before[slot] = rows[-(TAPS - 1):]
        at += n
    conv = silu(conv)
    xs, B, Cq = conv[:, :I].view(T, H, vd), conv[:, I: I + G * N].view(T, G, N), conv[:, I + G * N:].view(T, G, N)
    B, Cq = B.repeat_interleave(H // G, 1), Cq.repeat_interleave(H // G, 1)
    size = torch.nn.functional.softplus(dt + W["dt_bias"])
    a = torch.exp(-torch.exp(W["A_log"]) * size)

    def token(S, t):
        S = a[t][:, None, None] * S + B[t][:, :, None] * (size[t][:, None] * xs[t])[:, None]
        return S, (S * Cq[t][:, :, None]).sum(1)
    o, state = _walk(case, s, 1, H, N, vd, token)
    y = (o + W["D"][:, None] * xs).reshape(T, I) * silu(z)
    y = _head_rms(y.view(T, parts, -1), 1e-6).reshape(T, I) * W["norm"]
    return [y @ W["o"].T, before, state]
