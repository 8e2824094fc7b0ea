"""The work that programs have this framework do, as cases that can be timed and checked.

Most cases are single parts of a model (an attention layer, a recurrent mixer, a routed feed-forward), built from their
spec records and called as the generic model calls them; two are whole calls of the engine (prompts and decode steps);
one is the selection of tokens.  Steps that bring one token per sequence are replayed from a CUDA graph, as the engine
replays them.  Sizes are those of the benchmark's models (``bench.py``) and generic ones.

``exact`` is the same arithmetic in plain torch in float64, from the same inputs.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

from rust_inference_b200 import Engine, Entry, Model, ops
from rust_inference_b200.cache import Cache
from rust_inference_b200.config.registry import config_from_dict
from rust_inference_b200.config.specs import (AttentionSpec, GatedDeltaSpec, GatedFFSpec, GLASpec, LatentAttentionSpec,
                                              MoESpec, RMSNormSpec, RopePairsSpec, RopeSpec)
from rust_inference_b200.engine.model import expected_tensors
from rust_inference_b200.parts import BuildEnv, StepContext, build_part, part_class

DEV = "cuda:0"
PAGE = 32
EPS = 1e-6
THETA = 1e6
LATENT_THETA = 500000.0
GLA_TAU = 16.0
MOE_LIMIT, MOE_ALPHA = 7.0, 1.702

# what the attention and the recurrent mixers of the benchmark's models share
ATTENTION = dict(kind="attention", dtype="bfloat16", hidden=4096, heads=32, kv_heads=8, head_dim=128, ragged=False)
LATENT = dict(kind="latent", dtype="bfloat16", hidden=4096, heads=32, dim=128, rot=64, vdim=128, rank=192, window=4096, sink=False,
              gate="head", ragged=False)
DELTA = dict(kind="delta", dtype="bfloat16", hidden=4096, heads=16, qk_heads=8, dim=128, vdim=128, conv=4, decay_rank=64,
             gate_rank=64, ragged=False)
GLA = dict(kind="gla", dtype="bfloat16", hidden=4096, heads=32, dim=64, vdim=128, decay_rank=16, ragged=False)
MOE = dict(kind="moe", dtype="bfloat16", hidden=4096, experts=16, identity=2, top=4, inter=1376, shared=2752)
QWEN3_8B = dict(hidden=4096, inter=12288, heads=32, kv_heads=8, head_dim=128, vocab=151936)


def listed():
    return [
        # one short request on a small model, all steps of it: latency, launches and the host's share
        dict(name="generate_small_b1", kind="generate", dtype="bfloat16", layers=4, hidden=1024, inter=3072, heads=16, kv_heads=8,
             head_dim=128, vocab=32000, batch=1, prompt=24, steps=24),
        # eight requests through two layers and the head of the 8B shapes: a prompt step, then decode steps
        dict(QWEN3_8B, name="generate_8b_layers_b8", kind="generate", dtype="bfloat16", layers=2, batch=8, prompt=256, steps=16),
        # the attention layer of the 8B shapes: a prompt, and one token for each of eight long sequences
        dict(ATTENTION, name="attention_prompt_2048", batch=1, new=2048, past=0),
        dict(ATTENTION, name="attention_decode_b8_ctx4096", batch=8, new=1, past=4095),
        # the same layer in true 32-bit arithmetic
        dict(ATTENTION, name="attention_float32_prompt_512", dtype="float32", batch=1, new=512, past=0),
        # latent attention over a prompt
        dict(LATENT, name="latent_prompt_2048", batch=1, new=2048, past=0),
        # the gated delta rule over a prompt, and one token for each of eight sequences
        dict(DELTA, name="delta_prompt_2048", batch=1, new=2048, past=0),
        dict(DELTA, name="delta_decode_b8", batch=8, new=1, past=1),
        # gated linear attention over three prompts of unequal lengths
        dict(GLA, name="gla_prompts_ragged_b3", batch=3, new=1023, past=0, ragged=True),
        # the routed feed-forward: the tokens of a prompt step, and of a decode step
        dict(MOE, name="moe_prompt_2048", tokens=2048),
        dict(MOE, name="moe_decode_b8", tokens=8),
        # the next tokens of eight sequences, drawn with temperature, top-k and top-p
        dict(name="sample_b8", kind="sample", rows=8, vocab=151936, top_k=50, top_p=0.9),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["generate", "attention", "attention", "latent", "latent", "delta", "delta", "gla", "gla", "moe", "moe",
                       "sample"])
    if kind == "generate":
        return dict(kind="generate", dtype="bfloat16", layers=rng.choice([2, 4]), hidden=1024, inter=3072, heads=16, kv_heads=8,
                    head_dim=rng.choice([64, 128]), vocab=32000, batch=rng.choice([1, 2, 3, 5, 8, 16, 24]),
                    prompt=_log_int(rng, 5, 300), steps=rng.randint(8, 20))
    if kind == "sample":
        return dict(kind="sample", rows=_log_int(rng, 1, 32), vocab=rng.choice([32000, 32768, 100003, 151936]),
                    top_k=rng.choice([0, 40]), top_p=rng.choice([1.0, 0.8, 0.95]))
    dtype = "float32" if rng.random() < 0.2 else "bfloat16"
    most = 300 if dtype == "float32" else 2048
    small = rng.random() < 0.5
    width = dict(hidden=2048) if small else dict(hidden=4096)
    if kind == "moe":
        return dict(MOE, dtype=dtype, tokens=_log_int(rng, 1, most), experts=rng.choice([8, 16, 32]), top=rng.choice([1, 2, 4]),
                    identity=rng.choice([0, 2]), inter=rng.choice([704, 1376]), shared=rng.choice([0, 1408]), **width)
    # tokens of a step: one each for a batch of sequences, or prompts and pieces of prompts
    if rng.random() < 0.3:
        step = dict(batch=_log_int(rng, 1, 24), new=1, past=_log_int(rng, 1, 4000), ragged=rng.random() < 0.7)
    else:
        batch = rng.choice([1, 1, 2, 4])
        step = dict(batch=batch, new=_log_int(rng, 2, most // batch), past=rng.choice([0, 0, _log_int(rng, 1, 1500)]),
                    ragged=rng.random() < 0.5)
    if dtype == "float32":
        step["past"] = min(step["past"], 300)
    if kind == "attention":
        heads = 16 if small else 32
        return {**ATTENTION, **width, **step, "dtype": dtype, "heads": heads, "kv_heads": heads // rng.choice([2, 4, 8]),
                "head_dim": rng.choice([64, 128])}
    if kind == "latent":
        return {**LATENT, **width, **step, "dtype": dtype, "heads": 16 if small else 32, "vdim": 128,
                **rng.choice([dict(window=4096, sink=False, gate="head"), dict(window=1024, sink=True, gate="element")])}
    if kind == "delta":
        return {**DELTA, **width, **step, "dtype": dtype, "heads": 8 if small else 16, "qk_heads": 4 if small else 8,
                "dim": rng.choice([64, 128]), "vdim": rng.choice([64, 96, 128])}
    return {**GLA, **width, **step, "dtype": dtype, "heads": 16 if small else 32, "dim": rng.choice([48, 64, 128]),
            "vdim": rng.choice([64, 128])}


# ---- inputs, from the seed alone ------------------------------------------------------------------------------------
def _gen(seed, name):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 62))


def _normal(seed, name, shape, std=1.0, mean=0.0):
    return torch.randn(tuple(shape), generator=_gen(seed, name), device=DEV) * std + mean


def _uniform(seed, name, shape, lo, hi):
    return torch.rand(tuple(shape), generator=_gen(seed, name), device=DEV) * (hi - lo) + lo


def _dtype(case):
    return torch.bfloat16 if case.get("dtype", "bfloat16") == "bfloat16" else torch.float32


def _lengths(case, key):
    """What each sequence brings (or holds already): all the same, or from the given number down."""
    n, B = case[key], case["batch"]
    if not case["ragged"]:
        return [n] * B
    return [max(min(n, 1), n - i * n // (B + 1)) for i in range(B)]


def _spec(case):
    k, D = case["kind"], case["hidden"]
    if k == "attention":
        return AttentionSpec(hidden_size=D, num_heads=case["heads"], num_kv_heads=case["kv_heads"], head_dim=case["head_dim"],
                             position=RopeSpec(head_dim=case["head_dim"], theta=THETA),
                             qk_norm=RMSNormSpec(size=case["head_dim"], eps=EPS))
    if k == "latent":
        return LatentAttentionSpec(hidden_size=D, num_heads=case["heads"], dim=case["dim"], rot_dim=case["rot"], vdim=case["vdim"],
                                   kv_rank=case["rank"], scale=(case["dim"] + case["rot"]) ** -0.5, eps=EPS,
                                   position=RopePairsSpec(rotary_dim=case["rot"], theta=LATENT_THETA), window=case["window"],
                                   sink=case["sink"], gate=case["gate"])
    if k == "delta":
        return GatedDeltaSpec(hidden_size=D, num_heads=case["heads"], num_qk_heads=case["qk_heads"], dim=case["dim"],
                              vdim=case["vdim"], conv=case["conv"], decay_rank=case["decay_rank"], gate_rank=case["gate_rank"],
                              eps=EPS)
    if k == "gla":
        return GLASpec(hidden_size=D, num_heads=case["heads"], dim=case["dim"], vdim=case["vdim"], tau=GLA_TAU,
                       decay_rank=case["decay_rank"], eps=EPS)
    shared = None
    if case["shared"]:
        shared = GatedFFSpec(D, case["shared"], gate="clamped_swish", limit=MOE_LIMIT, alpha=MOE_ALPHA)
    return MoESpec(hidden_size=D, experts=case["experts"], top=case["top"], identity=case["identity"], shared=shared,
                   expert=GatedFFSpec(D, case["inter"], gate="clamped_swish", limit=MOE_LIMIT, alpha=MOE_ALPHA))


def _tensors(case, seed, infos):
    """The weights as a checkpoint holds them: matrices N(0, 0.02), gains around 1, and the rates of the recurrent mixers
    where trained ones lie (decays per token from about 0.8 to 0.999)."""
    out = {}
    for name, info in infos.items():
        shape = info.shape
        if name.endswith(".conv"):
            t = _uniform(seed, name, shape, -0.5, 0.5)
        elif name == "A_log":
            t = torch.log(_uniform(seed, name, shape, 1.0, 8.0))
        elif name == "dt_bias":
            t = torch.log(torch.expm1(torch.exp(_uniform(seed, name, shape, math.log(1e-3), math.log(1e-1)))))
        elif name == "a2.b":
            t = _uniform(seed, name, shape, 0.0, 4.0)
        elif name == "sink":
            t = _normal(seed, name, shape)
        elif info.role == "gain":
            t = _uniform(seed, name, shape, 0.9, 1.1)
        else:
            t = _normal(seed, name, shape, 0.02)
        out[name] = t.to(_dtype(case) if info.role == "matrix" else torch.float32)
    return out


def _family(case):
    return "ffn" if case["kind"] == "moe" else "mixer"


def _part_inputs(case, seed):
    """The part's tensors, the packed normed activations, and what the cache holds before the step."""
    spec = _spec(case)
    w = _tensors(case, seed, part_class(_family(case), spec).param_infos(spec))
    T = case["tokens"] if case["kind"] == "moe" else sum(_lengths(case, "new"))
    x = _normal(seed, "x", (T, case["hidden"])).to(_dtype(case))
    held = {}
    if case["kind"] == "attention" and case["past"]:
        shape = (case["batch"], case["past"], case["kv_heads"], case["head_dim"])
        held = {"k": _normal(seed, "held k", shape).to(_dtype(case)), "v": _normal(seed, "held v", shape).to(_dtype(case))}
    elif case["kind"] == "latent" and case["past"]:
        held = {"row": _normal(seed, "held row", (case["batch"], case["past"], case["rank"] + case["rot"])).to(_dtype(case))}
    elif case["kind"] in ("delta", "gla"):
        shape = (case["batch"], case["heads"], case["dim"], case["vdim"])
        held = {"state": _normal(seed, "held state", shape, 0.3 if case["past"] else 0.0)}
        if case["kind"] == "delta":
            C = 2 * case["qk_heads"] * case["dim"] + case["heads"] * case["vdim"]
            held["conv"] = _normal(seed, "held conv", (case["batch"], case["conv"] - 1, C), 1.0 if case["past"] else 0.0)
    return spec, w, x, held


# ---- what a program has before the call ---------------------------------------------------------------------------------
def _prepare_generate(case, seed):
    cfg = config_from_dict(_qwen3_config(case))
    model = Model(cfg.to_spec(), case["dtype"], DEV)
    model.config = cfg
    w = _tensors(case, seed, expected_tensors(model.spec))
    model.load_tensors(lambda name, info: w.pop(name, None))
    B, n = case["batch"], case["prompt"] + case["steps"]
    engine = Engine(model, max_tokens=B * (n + PAGE), max_seqs=B, max_seq_len=n + PAGE)
    return dict(kind="generate", engine=engine, ids=_ids(case, seed).tolist(), prompt=case["prompt"], steps=case["steps"])


def _ids(case, seed):
    return np.random.default_rng(int(seed)).integers(0, case["vocab"], size=(case["batch"], case["prompt"] + case["steps"]))


def _qwen3_config(case):
    return {"architectures": ["Qwen3ForCausalLM"], "vocab_size": case["vocab"], "hidden_size": case["hidden"],
            "intermediate_size": case["inter"], "num_hidden_layers": case["layers"], "num_attention_heads": case["heads"],
            "num_key_value_heads": case["kv_heads"], "head_dim": case["head_dim"], "rms_norm_eps": EPS, "rope_theta": THETA,
            "max_position_embeddings": 8192, "tie_word_embeddings": False}


def _i32(values):
    return torch.tensor(np.asarray(values, dtype=np.int32), device=DEV)


def _prepare_part(case, seed):
    spec, w, x, held = _part_inputs(case, seed)
    env = BuildEnv(_dtype(case), torch.device(DEV))
    part = build_part(_family(case), spec, env)
    part.load(w)
    state = dict(kind="part", part=part, x=x, graph=None, own=[], restore=[])
    if case["kind"] == "moe":
        T = case["tokens"]
        single = T <= 64                                                      # a decode step: a token per sequence
        state["ctx"] = _context(list(range(T)) if single else [0], [1] * T if single else [T], [0] * (T if single else 1))
        state["layer"] = None
    else:
        new, past = _lengths(case, "new"), _lengths(case, "past")
        if case["kind"] in ("delta", "gla"):
            past = [0] * case["batch"]                                        # the state is all that is held
        total = [a + b for a, b in zip(new, past)]
        cache = Cache([part.cache_request()], case["batch"], sum(-(-t // PAGE) for t in total), -(-max(total) // PAGE),
                      env.dtype, env.device, PAGE)
        part.prepare(max(total))
        slots = [cache.alloc_slot() for _ in new]
        cache.extend(list(zip(slots, total)))
        cache.upload()
        layer = cache.layer(0)
        for b, (slot, n) in enumerate(zip(slots, past)):
            if n and case["kind"] in ("attention", "latent"):
                at = torch.arange(n, device=DEV)
                page, off = layer.page_table[slot].long()[at // PAGE], at % PAGE
                if case["kind"] == "attention":
                    layer.k_pool[page, :, off] = held["k"][b, :n]
                    layer.v_pool[page, :, off] = held["v"][b, :n]
                else:
                    layer.k_pool[page, 0, off, :held["row"].shape[-1]] = held["row"][b, :n]
        if case["kind"] in ("delta", "gla"):
            rows = torch.tensor(slots, device=DEV)
            fresh = torch.zeros_like(layer.state)
            fresh[rows] = held["state"]
            state["restore"].append((layer.state, fresh))
            for i, t in enumerate(layer.more_state):
                fresh = torch.zeros_like(t)
                fresh[rows] = held["conv"]
                state["restore"].append((t, fresh))
            state["own"] = [layer.state]
        state.update(ctx=_context(slots, new, past), layer=layer, cache=cache)
    if state["ctx"].decode_only and part.graph_safe:
        _call(state)                                                          # libraries set themselves up
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _call(state)
        state.update(graph=graph, out=out)
    return state


def _context(slots, new, past):
    T, B = sum(new), len(new)
    seq = np.repeat(np.arange(B), new)
    start = np.concatenate([[0], np.cumsum(new)])
    pos = np.concatenate([np.arange(p, p + n) for n, p in zip(new, past)])
    length = [a + b for a, b in zip(new, past)]
    return StepContext(tok_seq=_i32(seq), tok_pos=_i32(pos), seq_slot=_i32(slots), seq_start=_i32(start), seq_len=_i32(length),
                       num_tokens=T, num_seqs=B, max_new=max(new), max_len=max(length), host_seq_slot=tuple(slots),
                       host_new=tuple(new), host_len=tuple(length))


def _call(state):
    for t, fresh in state["restore"]:              # a sequence takes up what a cache holds for it, the same on every pass
        t.copy_(fresh)
    if state["layer"] is None:
        return state["part"](state["x"], state["ctx"])
    return state["part"](state["x"], state["ctx"], state["layer"])


def prepare(case, seed):
    if case["kind"] == "generate":
        return _prepare_generate(case, seed)
    if case["kind"] == "sample":
        rows, vocab = case["rows"], case["vocab"]
        return dict(kind="sample", logits=_normal(seed, "logits", (rows, vocab), 2.5), u=_uniform(seed, "u", (rows,), 0.0, 1.0),
                    temperature=torch.full((rows,), 0.7, device=DEV), k=case["top_k"], p=case["top_p"],
                    top_k=torch.full((rows,), case["top_k"], dtype=torch.int32, device=DEV),
                    top_p=torch.full((rows,), case["top_p"], device=DEV))
    return _prepare_part(case, seed)


def run(state):
    if state["kind"] == "generate":
        engine, ids, n = state["engine"], state["ids"], state["prompt"]
        slots = [engine.new_sequence() for _ in ids]
        out = [engine.step([Entry(s, row[:n], "last") for s, row in zip(slots, ids)])]
        for i in range(n, n + state["steps"]):
            out.append(engine.step([Entry(s, row[i:i + 1], "last") for s, row in zip(slots, ids)]).clone())
        for s in slots:
            engine.release(s)
        return out
    if state["kind"] == "sample":
        return ops.sample(state["logits"], state["temperature"], state["u"], top_k=state["top_k"], top_p=state["top_p"],
                          uses_top_k=state["k"] > 0, uses_top_p=state["p"] < 1.0)
    if state["graph"] is not None:
        state["graph"].replay()
        return [state["out"]] + state["own"]
    return [_call(state)] + state["own"]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------
def _pairs(case):
    """(query, key) pairs of a step."""
    window = case.get("window", 0)
    total = 0
    for n, p in zip(_lengths(case, "new"), _lengths(case, "past")):
        seen = np.arange(p + 1, p + n + 1)
        total += int(np.minimum(seen, window).sum() if window else seen.sum())
    return total


def work(case):
    k = case["kind"]
    if k == "sample":
        return {"bytes": 4 * case["rows"] * case["vocab"], "flops": 0}
    D = case["hidden"]
    es = 2 if case["dtype"] == "bfloat16" else 4
    if k == "generate":
        H, KV, d, B, V = case["heads"], case["kv_heads"], case["head_dim"], case["batch"], case["vocab"]
        layer = D * d * (2 * H + 2 * KV) + 3 * D * case["inter"]
        body, head = case["layers"] * layer, V * D
        n, s = case["prompt"], case["steps"]
        cached = 2 * KV * d * case["layers"]
        seen = sum(range(n + 1, n + s + 1)) * B
        pairs = B * n * (n + 1) // 2 + seen
        return {"bytes": es * ((1 + s) * (body + head) + cached * (seen + B * (n + s))) + 4 * V * B * (1 + s),
                "flops": 2 * body * B * (n + s) + 2 * head * B * (1 + s) + 4 * H * d * pairs * case["layers"]}
    if k == "moe":
        T, E, top, I, S = case["tokens"], case["experts"], case["top"], case["inter"], case["shared"]
        real = top * E / (E + case["identity"])
        used = min(E, E * (1 - (1 - real / E) ** T))
        return {"bytes": es * (3 * D * (used * I + S) + 2 * T * D) + 4 * (E + case["identity"]) * D,
                "flops": 6 * T * D * (real * I + S)}
    T = sum(_lengths(case, "new"))
    H = case["heads"]
    if k == "attention":
        KV, d = case["kv_heads"], case["head_dim"]
        held = sum(_lengths(case, "past"))
        return {"bytes": es * (D * d * (2 * H + 2 * KV) + 2 * T * D + 2 * KV * d * (held + T)),
                "flops": 2 * T * D * d * (2 * H + 2 * KV) + 4 * H * d * _pairs(case)}
    if k == "latent":
        dim, rot, vd, r = case["dim"], case["rot"], case["vdim"], case["rank"]
        gate = H if case["gate"] == "head" else H * vd
        params = D * (H * (dim + rot) + r + rot + gate + H * vd) + H * r * (dim + vd)
        held = sum(min(p, case["window"]) for p in _lengths(case, "past"))
        # a prompt's scores over dim + rot and sums over vdim per pair; a single token's over the latent row
        pair = 2 * (dim + rot + vd) if case["new"] > 1 else 2 * (2 * r + rot)
        return {"bytes": es * (params + 2 * T * D + (r + rot) * (held + T)), "flops": 2 * T * params + pair * H * _pairs(case)}
    dim, vd = case["dim"], case["vdim"]
    state = 8 * case["batch"] * H * dim * vd
    if k == "delta":
        C = 2 * case["qk_heads"] * dim + H * vd
        params = D * (C + H + case["decay_rank"] + case["gate_rank"] + H * vd) + H * dim * case["decay_rank"] + H * vd * case["gate_rank"]
        return {"bytes": es * (params + 2 * T * D) + state, "flops": 2 * T * params + 7 * T * H * dim * vd}
    params = D * (2 * H * dim + 3 * H * vd + case["decay_rank"]) + H * dim * case["decay_rank"]
    return {"bytes": es * (params + 2 * T * D) + state, "flops": 2 * T * params + 5 * T * H * dim * vd}


# Four times what the path is off from its float64 restatement (`exact`), rounded up; bfloat16 weights and activations
# give some 0.3 to 0.5 % per layer, float32 sums 1e-7 to 1e-6.
def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.03 if case["kind"] == "generate" else 0.02}


# ---- the same arithmetic in float64 ---------------------------------------------------------------------------------------
def _rms(x, gain):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * gain


def _angles(pos, rot, theta, single=False):
    """float32 position times float32 frequency, as both position encodings define their angle."""
    i = np.arange(rot // 2)
    if single:                                     # the frequencies themselves in float32
        f = np.float32(1.0) / np.power(np.float32(theta), np.arange(0, rot, 2, dtype=np.float32) / np.float32(rot), dtype=np.float32)
    else:
        f = (float(theta) ** (-2.0 * i / rot)).astype(np.float32)
    a = (np.asarray(pos, dtype=np.float32)[:, None] * f[None, :].astype(np.float32)).astype(np.float32)
    a = torch.from_numpy(a.astype(np.float64)).to(DEV)
    return torch.cos(a), torch.sin(a)


def _rope_halves(x, pos, theta):
    cos, sin = (t[:, None] for t in _angles(pos, x.shape[-1], theta, single=True))
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _rope_pairs(x, pos, theta):
    cos, sin = (t[:, None] for t in _angles(pos, x.shape[-1], theta))
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * cos - b * sin, b * cos + a * sin], dim=-1).flatten(-2)


def _attend(q, k, v, past, scale, window=0, sink=None):
    """q [n, H, d] at positions past .., k [past + n, G, d], v [past + n, G, dv]; H a multiple of G."""
    n, H, _ = q.shape
    G = k.shape[1]
    i = torch.arange(past, past + n, device=DEV)[:, None]
    j = torch.arange(past + n, device=DEV)[None, :]
    hidden = (j > i) | ((i - j >= window) if window else torch.zeros_like(j > i))
    out = []
    for h in range(H):
        g = h * G // H
        s = (q[:, h] @ k[:, g].t() * scale).masked_fill(hidden, -math.inf)
        if sink is None:
            p = torch.softmax(s, dim=-1)
        else:
            p = torch.softmax(torch.cat([s, sink[h].expand(n, 1)], dim=1), dim=-1)[:, :-1]
        out.append(p @ v[:, g])
    return torch.stack(out, dim=1)


def _exact_attention(case, w, x, held, new, past):
    H, KV, d = case["heads"], case["kv_heads"], case["head_dim"]
    out, at = [], 0
    for b, (n, p) in enumerate(zip(new, past)):
        h = x[at:at + n]
        at += n
        pos = range(p, p + n)
        q = _rope_halves(_rms((h @ w["q_proj.weight"].t()).view(n, H, d), w["q_norm.weight"]), pos, THETA)
        k = _rope_halves(_rms((h @ w["k_proj.weight"].t()).view(n, KV, d), w["k_norm.weight"]), pos, THETA)
        v = (h @ w["v_proj.weight"].t()).view(n, KV, d)
        if p:
            k, v = torch.cat([held["k"][b, :p], k]), torch.cat([held["v"][b, :p], v])
        out.append(_attend(q, k, v, p, d ** -0.5).reshape(n, H * d) @ w["o_proj.weight"].t())
    return torch.cat(out)


def _exact_latent(case, w, x, held, new, past):
    H, dim, rot, vd, r = case["heads"], case["dim"], case["rot"], case["vdim"], case["rank"]
    out, at = [], 0
    for b, (n, p) in enumerate(zip(new, past)):
        h = x[at:at + n]
        at += n
        pos = range(p, p + n)
        q = (h @ w["q"].t()).view(n, H, dim + rot)
        q = torch.cat([q[..., :dim], _rope_pairs(q[..., dim:], pos, LATENT_THETA)], dim=-1)
        down = h @ w["dkv"].t()
        row = torch.cat([_rms(down[:, :r], w["dkv.norm"]), _rope_pairs(down[:, None, r:], pos, LATENT_THETA)[:, 0]], dim=-1)
        if p:
            row = torch.cat([held["row"][b, :p], row])
        k = torch.cat([(row[:, :r] @ w["uk"].t()).view(-1, H, dim), row[:, None, r:].expand(-1, H, rot)], dim=-1)
        v = (row[:, :r] @ w["uv"].t()).view(-1, H, vd)
        o = _attend(q, k, v, p, (dim + rot) ** -0.5, case["window"], w.get("sink"))
        g = torch.sigmoid(h @ w["g"].t())
        o = o * g[:, :, None] if case["gate"] == "head" else o * g.view(n, H, vd)
        out.append(o.reshape(n, H * vd) @ w["o"].t())
    return torch.cat(out)


def _recur(q, k, v, decay, S, beta=None):
    """Token by token: S <- decay S (the delta rule: what S predicts for k is taken off v), S <- S + k v^T, o = S^T q."""
    o = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * decay[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
        S = S + k[t][:, :, None] * u[:, None]
        o[t] = (S * q[t][:, :, None]).sum(1)
    return o, S


def _exact_gla(case, w, x, held, new):
    H, dim, vd = case["heads"], case["dim"], case["vdim"]
    out, states, at = [], [], 0
    for b, n in enumerate(new):
        h = x[at:at + n]
        at += n
        q, k = (h @ w["q"].t()).view(n, H, dim) * dim ** -0.5, (h @ w["k"].t()).view(n, H, dim)
        v = (h @ w["v"].t()).view(n, H, vd)
        z = ((h @ w["a1"].t()) @ w["a2"].t() + w["a2.b"]).view(n, H, dim)
        o, S = _recur(q, k, v, torch.sigmoid(z) ** (1.0 / GLA_TAU), held["state"][b])
        g = h @ w["g"].t()
        out.append((_rms(o, w["norm"]).reshape(n, H * vd) * g * torch.sigmoid(g)) @ w["o"].t())
        states.append(S)
    return torch.cat(out), torch.stack(states)


def _exact_delta(case, w, x, held, new):
    H, G, dim, vd, taps = case["heads"], case["qk_heads"], case["dim"], case["vdim"], case["conv"]
    conv = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]])
    out, states, at = [], [], 0
    for b, n in enumerate(new):
        h = x[at:at + n]
        at += n
        u = torch.cat([held["conv"][b], torch.cat([h @ w["q"].t(), h @ w["k"].t(), h @ w["v"].t()], dim=1)])
        u = torch.nn.functional.silu(sum(u[i:i + n] * conv[:, i] for i in range(taps)))
        q, k, v = u[:, :G * dim].view(n, G, dim), u[:, G * dim:2 * G * dim].view(n, G, dim), u[:, 2 * G * dim:].view(n, H, vd)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dim ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        q, k = (t.repeat_interleave(H // G, dim=1) for t in (q, k))
        z = ((h @ w["a1"].t()) @ w["a2"].t() + w["dt_bias"]).view(n, H, dim)
        decay = torch.exp(-torch.exp(w["A_log"])[None, :, None] * torch.nn.functional.softplus(z, threshold=40))
        o, S = _recur(q, k, v, decay, held["state"][b], torch.sigmoid(h @ w["b"].t()))
        gate = torch.sigmoid((h @ w["g1"].t()) @ w["g2"].t())
        out.append((_rms(o, w["norm"]).reshape(n, H * vd) * gate) @ w["o"].t())
        states.append(S)
    return torch.cat(out), torch.stack(states)


def _clamped_swish(x, gate, up, down):
    g, u = torch.clamp(x @ gate.t(), max=MOE_LIMIT), torch.clamp(x @ up.t(), -MOE_LIMIT, MOE_LIMIT)
    return (g * torch.sigmoid(MOE_ALPHA * g) * (u + 1.0)) @ down.t()


def _exact_moe(case, w, x):
    s = torch.softmax(x @ w["router"].t(), dim=-1)
    idx = torch.argsort(s + w["correction"], dim=-1, descending=True, stable=True)[:, :case["top"]]
    weight = torch.gather(s, 1, idx)
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    y = torch.zeros_like(x)
    for e in range(case["experts"] + case["identity"]):
        t, j = (idx == e).nonzero(as_tuple=True)
        if len(t):
            out = x[t] if e >= case["experts"] else _clamped_swish(x[t], w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"])
            y.index_add_(0, t, out * weight[t, j][:, None])
    if case["shared"]:
        y += _clamped_swish(x, w["shared.gate"], w["shared.up"], w["shared.down"])
    return y


def _exact_generate(case, seed):
    spec = config_from_dict(_qwen3_config(case)).to_spec()
    w = {n: t.double() for n, t in _tensors(case, seed, expected_tensors(spec)).items()}
    B, n, H, KV, d = case["batch"], case["prompt"], case["heads"], case["kv_heads"], case["head_dim"]
    ids = torch.from_numpy(_ids(case, seed)).to(DEV)
    L = n + case["steps"]
    h = w["model.embed_tokens.weight"][ids.reshape(-1)]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        local = {k[len(p) + len("self_attn."):]: t for k, t in w.items() if k.startswith(p + "self_attn.")}
        h = h + _exact_attention(case, local, _rms(h, w[p + "input_layernorm.weight"]), {}, [L] * B, [0] * B)
        m = _rms(h, w[p + "post_attention_layernorm.weight"])
        h = h + (torch.nn.functional.silu(m @ w[p + "mlp.gate_proj.weight"].t()) * (m @ w[p + "mlp.up_proj.weight"].t())) \
            @ w[p + "mlp.down_proj.weight"].t()
    h = _rms(h, w["model.norm.weight"]).view(B, L, -1)
    return [h[:, i] @ w["lm_head.weight"].t() for i in range(n - 1, L)]


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    with torch.no_grad():
        if case["kind"] == "generate":
            return _exact_generate(case, seed)
        _, w, x, held = _part_inputs(case, seed)
        w = {n: t.double() for n, t in w.items()}
        x, held = x.double(), {n: t.double() for n, t in held.items()}
        if case["kind"] == "moe":
            return [_exact_moe(case, w, x)]
        new, past = _lengths(case, "new"), _lengths(case, "past")
        if case["kind"] == "attention":
            return [_exact_attention(case, w, x, held, new, past)]
        if case["kind"] == "latent":
            return [_exact_latent(case, w, x, held, new, past)]
        y, S = (_exact_gla if case["kind"] == "gla" else _exact_delta)(case, w, x, held, new)
        return [y, S]
