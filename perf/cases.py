"""What a user of this engine has it do, as cases that can be timed and compared.

A case is one pass through the public entry points:

  step       ModelRunner.step_and_sample on an engine's runner: ``decoding`` requests with ``context``
             tokens in the cache (request i holds a few fewer, so that lengths are ragged) take their next
             token beside ``portion`` tokens of a prompt of which ``behind`` tokens are in the cache already.
             This is the engine's only forward pass; nothing is committed, so it can be run again.
             Outputs: the logits of every decoding request and of the portion's last token (in float32 the
             chosen tokens too; in bfloat16 random weights leave the two best of 152 thousand logits closer
             than one rounding, so the choice between them says nothing).
  generate   Engine.generate: ``requests`` prompts of ragged lengths, ``new`` greedy tokens each, scheduler and all.

``chunk`` is the engine's token budget a step (``Engine(chunk=...)``), which decides what steps it replays.
Layers with routed experts have no case: at random weights a rounding
changes which expert a token gets, and with it the whole row.  Weights are N(0, 0.02) (gains 1 + N(0, 0.1)) and the same for every seed; prompts come from the seed.
"""

import json
import math
import os
import random
import shutil
import struct
import tempfile
import weakref
import zlib

import numpy as np
import torch

from paged_llm_rs_b200 import Engine, StepEntry

QWEN3 = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_act="silu", attention_bias=False, head_dim=128,
             num_key_value_heads=8, rms_norm_eps=1e-6, vocab_size=151936, max_position_embeddings=40960, rope_theta=1000000.0,
             sliding_window=None, use_sliding_window=False)


def _pamarax(layers):
    att = dict(heads=16, kv_heads=8, dim=128, vdim=128, scale=128 ** -0.5, rot=dict(dims=64, base=10000.0))
    lstm = dict(heads=4, dim=128, vdim=256, gate_cap=15.0)
    left = dict(heads=16, kv_heads=8, dim=128, vdim=64, scale=128 ** -0.5, q_temp=dict(coef=0.5, every=256))
    right = dict(heads=8, kv_heads=4, dim=128, vdim=128, conv=4)
    cycle = [dict(type="attention", mixer=att), dict(type="mlstm", mixer=lstm),
             dict(type="parallel", mixer=dict(left=left, right=right, left_scale=1.0, right_scale=1.0)), dict(type="mlstm", mixer=lstm)]
    return dict(architecture="Pamarax", vocab=32768, width=1024, norm=dict(eps=1e-6), embedding=dict(scale=1.0),
                layers=[dict(cycle[i % 4], mlp=dict(kind="dense", ff=3072)) for i in range(layers)])


# The shapes of this repository's benchmark and its smallest test shape.  The 8B shape runs 6 of its 36 layers (all
# layers are alike) so that several states, and 64-bit results, fit the time and the card.
MODELS = {
    "tiny-a": dict(QWEN3, hidden_size=64, intermediate_size=128, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2,
                   head_dim=16, vocab_size=256, max_position_embeddings=128, rope_theta=10000.0, tie_word_embeddings=True),
    "qwen3-0.6b": dict(QWEN3, hidden_size=1024, intermediate_size=3072, num_hidden_layers=28, num_attention_heads=16,
                       tie_word_embeddings=True),
    "qwen3-8b": dict(QWEN3, hidden_size=4096, intermediate_size=12288, num_hidden_layers=6, num_attention_heads=32,
                     tie_word_embeddings=False),
    "pamarax": _pamarax(4),
}
DTYPES = {"bf16": "bfloat16", "f32": "float32"}
# tokens of cache an engine is given: room for five states of the largest case that runs on it
CACHE_TOKENS = {("tiny-a", "f32"): 4096, ("qwen3-0.6b", "bf16"): 180000, ("qwen3-0.6b", "f32"): 16000, ("qwen3-8b", "bf16"): 340000,
                ("pamarax", "bf16"): 80000}


def _step(name, model, dtype, chunk, decoding, context, portion, behind):
    return dict(name=name, task="step", model=model, dtype=dtype, chunk=chunk, decoding=decoding, context=context, portion=portion, behind=behind)


def listed():
    return [
        # three short prompts through the smallest model in float32: nothing but latency, launches and host work
        dict(name="tiny f32 generate", task="generate", model="tiny-a", dtype="f32", chunk=8, requests=3, longest=19, new=8),
        # one user in a chat, the engine's default budget: a token a step
        _step("0.6b decode 1", "qwen3-0.6b", "bf16", 128, 1, 700, 0, 0),
        # a short question from that user: the step before the first token
        _step("0.6b prompt 37", "qwen3-0.6b", "bf16", 128, 0, 0, 37, 0),
        # the benchmark's headline: eight requests at 4096 tokens
        _step("0.6b decode 8 at 4096", "qwen3-0.6b", "bf16", 128, 8, 4096, 0, 0),
        # a full server, right after its prompts
        _step("0.6b decode 64 at 512", "qwen3-0.6b", "bf16", 128, 64, 512, 0, 0),
        # a prompt arrives at a server with the default budget: portions of it ride beside decoded tokens
        _step("0.6b 8 beside 120", "qwen3-0.6b", "bf16", 128, 8, 800, 120, 480),
        # the benchmark's prompt
        _step("0.6b prompt 2048", "qwen3-0.6b", "bf16", 2048, 0, 0, 2048, 0),
        # float32, as used where results are checked: decoded tokens beside a portion
        _step("0.6b f32 4 beside 252", "qwen3-0.6b", "f32", 256, 4, 500, 252, 100),
        # the larger shape: a few users, a full server with a portion of a long prompt, and a prompt alone
        _step("8b decode 8 at 2048", "qwen3-8b", "bf16", 512, 8, 2048, 0, 0),
        _step("8b 64 beside 448", "qwen3-8b", "bf16", 512, 64, 900, 448, 1024),
        _step("8b prompt 2048", "qwen3-8b", "bf16", 2048, 0, 0, 2048, 0),
        # a model with recurrent layers (matrix LSTM, gated delta rule) beside attention
        _step("pamarax 8 beside 1016", "pamarax", "bf16", 1024, 8, 600, 1016, 0),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    """One more case: a model by how often it is listed, then what the step holds, sizes over their logarithm."""
    model = rng.choice(["qwen3-0.6b"] * 5 + ["qwen3-8b"] * 3 + ["0.6b f32", "pamarax", "tiny-a"])
    if model == "tiny-a":
        return dict(task="generate", model=model, dtype="f32", chunk=rng.choice([8, 16, 128]), requests=rng.randint(1, 6), longest=_log(rng, 2, 90),
                    new=rng.randint(2, 8))
    dtype, chunk, most = "bf16", rng.choice([128, 2048] if model == "qwen3-0.6b" else [512, 2048]), 32768
    if model == "0.6b f32":
        model, dtype, chunk, most = "qwen3-0.6b", "f32", 256, 2000
    elif model == "pamarax":
        chunk, most = 1024, 8000
    kind = rng.choice(["decode", "decode", "prompt", "beside"])
    decoding = 0 if kind == "prompt" else _log(rng, 1, {"f32": 4, "bf16": 64}[dtype] if model != "pamarax" else 16)
    context = _log(rng, 16, max(17, min(4096, most // decoding))) if decoding else 0
    # (a portion never reaches past the budget, which the decoded tokens share)
    portion = 0 if kind == "decode" else _log(rng, 2, chunk - decoding)
    reach = 700 if dtype == "f32" or model == "pamarax" else 4096 if portion <= 1024 else 256
    behind = 0 if kind == "decode" else rng.choice([0, _log(rng, 16, reach)])
    return dict(task="step", model=model, dtype=dtype, chunk=chunk, decoding=decoding, context=context, portion=portion, behind=behind)


# ---- weights: a function of the tensor's name, drawn on the GPU ---------------------------------------------------

def _tensors(model):
    """(name, shape, kind) of every tensor of the model's file; kind "matrix", "gain" (near one) or "offset" (near zero)."""
    c = MODELS[model]
    out = []

    def put(name, kind, *shape):
        out.append((name, shape, kind))
    if model == "pamarax":
        D = c["width"]
        put("embed", "matrix", c["vocab"], D)
        for i, L in enumerate(c["layers"]):
            p, m = f"l{i}", L["mixer"]
            if L["type"] == "attention":
                H, G = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
                for n, s in (("q", (H, D)), ("k", (G, D)), ("g", (H, D)), ("o", (D, H))):
                    put(f"{p}.mix.{n}", "matrix", *s)
                put(f"{p}.mix.q.norm", "gain", H)
                put(f"{p}.mix.k.norm", "gain", G)
            elif L["type"] == "mlstm":
                H, d, e = m["heads"], m["heads"] * m["dim"], m["heads"] * m["vdim"]
                for n, s in (("q", (d, D)), ("k", (d, D)), ("v", (e, D)), ("g", (e, D)), ("o", (D, e)), ("i", (H, D)), ("f", (H, D))):
                    put(f"{p}.mix.{n}", "matrix", *s)
                put(f"{p}.mix.norm", "gain", e)
                put(f"{p}.mix.i.b", "offset", H)
                put(f"{p}.mix.f.b", "offset", H)
            else:
                a, r = m["left"], m["right"]
                for n, s in (("q", (a["heads"] * a["dim"], D)), ("k", (a["kv_heads"] * a["dim"], D)), ("v", (a["kv_heads"] * a["vdim"], D)),
                             ("o", (D, a["heads"] * a["vdim"]))):
                    put(f"{p}.mix.left.{n}", "matrix", *s)
                put(f"{p}.mix.left.q.norm", "gain", a["dim"])
                put(f"{p}.mix.left.k.norm", "gain", a["dim"])
                d, e = r["kv_heads"] * r["dim"], r["heads"] * r["vdim"]
                for n, s in (("q", (d, D)), ("k", (d, D)), ("v", (e, D)), ("g", (e, D)), ("o", (D, e)), ("q.conv", (d, r["conv"])),
                             ("k.conv", (d, r["conv"])), ("v.conv", (e, r["conv"])), ("b", (r["heads"], D)), ("a", (r["heads"], D))):
                    put(f"{p}.mix.right.{n}", "matrix", *s)
                put(f"{p}.mix.right.A_log", "offset", r["heads"])
                put(f"{p}.mix.right.dt_bias", "offset", r["heads"])
                put(f"{p}.mix.right.norm", "gain", r["vdim"])
            F = L["mlp"]["ff"]
            for n, s in (("gate", (F, D)), ("up", (F, D)), ("down", (D, F))):
                put(f"{p}.mlp.{n}", "matrix", *s)
                put(f"{p}.mlp.{n}.b", "offset", s[0])
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                put(f"{p}.{n}", "gain", D)
        put("final.norm", "gain", D)
        put("head", "matrix", c["vocab"], D)
        return out
    D, F, d = c["hidden_size"], c["intermediate_size"], c["head_dim"]
    H, G = c["num_attention_heads"] * d, c["num_key_value_heads"] * d
    put("model.embed_tokens.weight", "matrix", c["vocab_size"], D)
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}"
        for n, s in (("self_attn.q_proj", (H, D)), ("self_attn.k_proj", (G, D)), ("self_attn.v_proj", (G, D)), ("self_attn.o_proj", (D, H)),
                     ("mlp.gate_proj", (F, D)), ("mlp.up_proj", (F, D)), ("mlp.down_proj", (D, F))):
            put(f"{p}.{n}.weight", "matrix", *s)
        for n, s in (("self_attn.q_norm", d), ("self_attn.k_norm", d), ("input_layernorm", D), ("post_attention_layernorm", D)):
            put(f"{p}.{n}.weight", "gain", s)
    put("model.norm.weight", "gain", D)
    if not c["tie_word_embeddings"]:
        put("lm_head.weight", "matrix", c["vocab_size"], D)
    return out


def _weights(model):
    """{name: bfloat16 tensor on the GPU}."""
    out = {}
    for name, shape, kind in _tensors(model):
        g = torch.Generator(device="cuda").manual_seed(zlib.crc32(f"{model}/{name}".encode()))
        t = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, 0.02 if kind == "matrix" else 0.1, generator=g)
        out[name] = (t + 1.0 if kind == "gain" else t).to(torch.bfloat16)
    return out


def _write_folder(folder, model):
    """A model folder as a user has it: config.json and model.safetensors."""
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(MODELS[model], f)
    w = _weights(model)
    head, at = {}, 0
    for name, t in w.items():
        head[name] = {"dtype": "BF16", "shape": list(t.shape), "data_offsets": [at, at + 2 * t.numel()]}
        at += 2 * t.numel()
    raw = json.dumps(head).encode()
    raw += b" " * (-len(raw) % 8)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(raw)) + raw)
        for t in w.values():
            t.reshape(-1).view(torch.int16).cpu().numpy().tofile(f)


_ENGINES = {}


def _engine(case):
    """The engine a user's program keeps: one for a model, dtype and budget."""
    key = (case["model"], case["dtype"], case["chunk"])
    if key not in _ENGINES:
        room = shutil.disk_usage("/dev/shm").free > (16 << 30) if os.path.isdir("/dev/shm") else False
        with tempfile.TemporaryDirectory(dir="/dev/shm" if room else None) as folder:
            _write_folder(folder, case["model"])
            _ENGINES[key] = Engine(folder, dtype=DTYPES[case["dtype"]], block_size=16, blocks=CACHE_TOKENS[key[:2]] // 16 + 64, max_batch=64,
                                   chunk=case["chunk"], prefix_cache=False, max_requests=512)
    return _ENGINES[key]


# ---- inputs -------------------------------------------------------------------------------------------------------

def _vocab(model):
    c = MODELS[model]
    return c["vocab"] if model == "pamarax" else c["vocab_size"]


def _lengths(case):
    """Tokens in the cache of each decoding request: the context, and up to a quarter less."""
    C = case["context"]
    return [C - (37 * i) % (C // 4 + 1) for i in range(case["decoding"])]


def _sequences(case, seed):
    """Token ids of every decoding request (the last one is the step's own), then the prompt's (behind + portion)."""
    rng, V = np.random.default_rng(seed), _vocab(case["model"])
    seqs = [rng.integers(0, V, n + 1).tolist() for n in _lengths(case)]
    return seqs, rng.integers(0, V, case["behind"] + case["portion"]).tolist() if case["portion"] else []


class _State:
    pass


_COUNT = [0]


def _close(cache, ids):
    for r in ids:
        if cache.has(r):
            cache.close(r)


FILL = 2048     # tokens a step while the cache is filled


def _fill(runner, ids, seqs):
    """Bring the requests' earlier tokens into the cache, as the engine does it: portions of prompts, steps of FILL tokens."""
    cache, none = runner.cache, np.zeros(0, dtype=np.float32)
    todo, step, room = [(r, s) for r, s in zip(ids, seqs) if s], [], FILL
    while todo or step:
        if todo and room:
            r, s = todo.pop(0)
            part, rest = s[:room], s[room:]
            step.append(StepEntry(r, part, []))
            room -= len(part)
            if rest:
                todo.insert(0, (r, rest))
            if room and todo:
                continue
        for e in step:
            if not cache.reserve(e.request_id, len(e.tokens)):
                raise RuntimeError("the cache is too small for the case")
        runner.step_and_sample(step, none, none)
        for e in step:
            cache.commit(e.request_id, len(e.tokens))
        step, room = [], FILL


def prepare(case, seed):
    eng = _engine(case)
    s = _State()
    s.task, s.engine, s.f32 = case["task"], eng, case["dtype"] == "f32"
    if s.task == "generate":
        rng = np.random.default_rng(seed)
        n = case["requests"]
        s.prompts = [rng.integers(0, _vocab(case["model"]), 1 + (case["longest"] - 1) * (i + 1) // n).tolist() for i in range(n)]
        s.new = case["new"]
        return s
    runner = eng.runner
    seqs, prompt = _sequences(case, seed)
    _COUNT[0] += 1
    ids = [(_COUNT[0], i) for i in range(len(seqs) + (1 if prompt else 0))]
    weakref.finalize(s, _close, runner.cache, ids)
    for r in ids:
        runner.cache.open(r)
    behind = case["behind"]
    _fill(runner, ids, [q[:-1] for q in seqs] + ([prompt[:behind]] if prompt else []))
    s.entries = [StepEntry(r, [q[-1]], [0]) for r, q in zip(ids, seqs)]
    if prompt:
        s.entries.append(StepEntry(ids[-1], prompt[behind:], [case["portion"] - 1]))
    for e in s.entries:
        if not runner.cache.reserve(e.request_id, len(e.tokens)):
            raise RuntimeError("the cache is too small for the case")
    s.temperature = np.zeros(len(ids), dtype=np.float32)
    s.uniform = np.zeros(len(ids), dtype=np.float32)
    return s


def run(state):
    if state.task == "generate":
        return [np.asarray(t, dtype=np.int32) for t in state.engine.generate(state.prompts, max_tokens=state.new)]
    logits, tokens = state.engine.runner.step_and_sample(state.entries, state.temperature, state.uniform)
    return {"logits": logits, "tokens": tokens} if state.f32 else {"logits": logits}


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def work(case):
    """Every matrix of the layers and the head once, the keys and values of the cached tokens once, the new ones' and the
    logits written; a multiply-add for every matrix entry and token, and for every query and key it may see."""
    model, esz = case["model"], 2 if case["dtype"] == "bf16" else 4
    c, V = MODELS[model], _vocab(case["model"])
    table = "embed" if model == "pamarax" else "model.embed_tokens.weight"
    layer = sum(math.prod(s) for n, s, kind in _tensors(model) if kind == "matrix" and n not in (table, "head", "lm_head.weight"))
    width = c["width"] if model == "pamarax" else c["hidden_size"]
    if model == "pamarax":
        every = len(c["layers"]) // 4
        row = every * (2 * 1024 + 1024 + 512)              # (the gated layer's values are its raw keys, kept beside the normed ones)
        pair = every * (16 * 256 + 16 * 192)
        state, token = every * (2 * 4 * 128 * 256 + 8 * 128 * 128), every * (2 * 4 * 128 * 256 + 8 * 128 * 128) * 4
    else:
        L, d = c["num_hidden_layers"], c["head_dim"]
        row, pair, state, token = 2 * L * c["num_key_value_heads"] * d, 2 * L * c["num_attention_heads"] * d, 0, 0
    if case["task"] == "generate":
        n = case["requests"]
        lens = [1 + (case["longest"] - 1) * (i + 1) // n for i in range(n)]
        T, new = sum(lens) + n * (case["new"] - 1), case["new"]
        passes = -(-T // case["chunk"])                    # (steps that the budget makes it take, at the least)
        seen = sum(sum(range(1, m + new)) for m in lens)
        return {"bytes": esz * (max(passes, new) * (layer + V * width) + seen * row) + 4 * n * new, "flops": 2 * T * layer + 2 * n * new * V * width + 2 * seen * pair}
    lens = _lengths(case)
    P, B = case["portion"], case["behind"]
    T, rows = len(lens) + P, len(lens) + (1 if P else 0)
    cached = sum(lens) + (B if P else 0)
    seen = sum(n + 1 for n in lens) + P * B + P * (P + 1) // 2
    return {"bytes": esz * (layer + V * width + T * width + (cached + T) * row) + 4 * rows * V + 8 * rows * state,
            "flops": 2 * T * layer + 2 * rows * V * width + 2 * seen * pair + T * token}


def tolerance(case):
    # float32 is 2e-6 from 64 bits; bfloat16 is 0.012 (0.6B shape), 0.020 (8B) and 0.024 (Pamarax) from them, and two orders of a
    # product's sum leave logits that differ by up to 0.015 (the largest by 0.07): the norms carry a rounding through every layer
    return {"rel": 1e-5, "max": 1e-4} if case["dtype"] == "f32" else {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------

F64 = torch.float64
_W64 = {}


def _exact_weights(model):
    if model not in _W64:
        _W64.clear()
        _W64[model] = _weights(model)
    w = _W64[model]
    return lambda name: w[name].to(F64)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, dims, base):
    """x [heads, T, dim]: the first ``dims`` entries turn by position * base^(-2i / dims), entry i with entry i + dims / 2."""
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / dims)
    a = torch.arange(x.shape[1], dtype=F64, device=x.device)[:, None] * f
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., dims:]], -1)


def _causal(q, k, v, scale, extra_one=False):
    """q [H, T, d], k [G, T, d], v [G, T, e] -> [T, H * e]; with ``extra_one`` the softmax's denominator holds one more."""
    H, T, _ = q.shape
    per = H // k.shape[0]
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=q.device)
    hidden = torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1)
    for h in range(H):
        s = (q[h] @ k[h // per].T * scale).masked_fill_(hidden, -math.inf)
        if extra_one:
            s = torch.cat([s, torch.zeros(T, 1, dtype=F64, device=q.device)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :T] @ v[h // per]
    return out.reshape(T, -1)


def _heads(x, n):
    return x.view(x.shape[0], n, -1).transpose(0, 1)


def _qwen3_layers(w, c, xs):
    eps, d = c["rms_norm_eps"], c["head_dim"]
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}"
        t = {n: w(f"{p}.{n}.weight") for n in ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj", "mlp.gate_proj",
                                               "mlp.up_proj", "mlp.down_proj", "self_attn.q_norm", "self_attn.k_norm", "input_layernorm",
                                               "post_attention_layernorm")}
        for j, x in enumerate(xs):
            h = _rms(x, eps) * t["input_layernorm"]
            q = _rms(_heads(h @ t["self_attn.q_proj"].T, c["num_attention_heads"]), eps) * t["self_attn.q_norm"]
            k = _rms(_heads(h @ t["self_attn.k_proj"].T, c["num_key_value_heads"]), eps) * t["self_attn.k_norm"]
            v = _heads(h @ t["self_attn.v_proj"].T, c["num_key_value_heads"])
            o = _causal(_rotate(q, d, c["rope_theta"]), _rotate(k, d, c["rope_theta"]), v, d ** -0.5)
            x = x + o @ t["self_attn.o_proj"].T
            h = _rms(x, eps) * t["post_attention_layernorm"]
            g = h @ t["mlp.gate_proj"].T
            xs[j] = x + (g * torch.sigmoid(g) * (h @ t["mlp.up_proj"].T)) @ t["mlp.down_proj"].T
    return [_rms(x, eps) * w("model.norm.weight") for x in xs]


def _gated_attention(w, p, m, h, eps):
    H, G, dims, base = m["heads"], m["kv_heads"], m["rot"]["dims"], m["rot"]["base"]
    q, k = h @ w(f"{p}.q").T, h @ w(f"{p}.k").T
    v = _heads(k, G)                                        # a token's value is its raw key
    q, k = _heads(_rms(q, eps) * w(f"{p}.q.norm"), H), _heads(_rms(k, eps) * w(f"{p}.k.norm"), G)
    o = _causal(_rotate(q, dims, base), _rotate(k, dims, base), v, m["scale"])
    return (o * torch.sigmoid(h @ w(f"{p}.g").T)) @ w(f"{p}.o").T


def _matrix_lstm(w, p, m, h, eps):
    """In closed form: with F the running sum of the log forget gates, token s weighs exp(F_t - F_s + i_s - m_t) for token t, and the
    start (a maximum of zero) exp(F_t - m_t)."""
    T, H, cap = h.shape[0], m["heads"], m["gate_cap"]
    q, k, v = _heads(h @ w(f"{p}.q").T, H) * m["dim"] ** -0.5, _heads(h @ w(f"{p}.k").T, H), _heads(h @ w(f"{p}.v").T, H)
    i = cap * torch.tanh((h @ w(f"{p}.i").T + w(f"{p}.i.b")) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w(f"{p}.f").T + w(f"{p}.f.b")) / cap)).cumsum(0)
    hidden = torch.ones(T, T, dtype=torch.bool, device=h.device).triu(1)
    out = torch.empty(T, H, m["vdim"], dtype=F64, device=h.device)
    for a in range(H):
        e = (f[:, a, None] - f[None, :, a] + i[None, :, a]).masked_fill_(hidden, -math.inf)
        top = torch.maximum(e.max(1).values, f[:, a])
        s = torch.exp(e - top[:, None]) * (q[a] @ k[a].T)
        out[:, a] = s @ v[a] / (torch.maximum(s.sum(1).abs(), torch.exp(-top)) + 1e-6)[:, None]
    o = _rms(out, eps).reshape(T, -1) * w(f"{p}.norm")
    return (o * torch.sigmoid(h @ w(f"{p}.g").T)) @ w(f"{p}.o").T


def _conv_silu(u, taps):
    """The last column of ``taps`` meets the current token; zeros before the start."""
    n = taps.shape[1]
    u = torch.cat([torch.zeros(n - 1, u.shape[1], dtype=F64, device=u.device), u], 0)
    return torch.nn.functional.silu(sum(u[j:u.shape[0] - n + 1 + j] * taps[:, j] for j in range(n)))


def _delta_rule(w, p, m, h, eps):
    T, H, G, d = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    q, k, v = (_conv_silu(h @ w(f"{p}.{n}").T, w(f"{p}.{n}.conv")).view(T, a, -1) for n, a in (("q", G), ("k", G), ("v", H)))
    q, k = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = (q * d ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    beta = torch.sigmoid(h @ w(f"{p}.b").T)
    g = torch.exp(-torch.exp(w(f"{p}.A_log")) * torch.nn.functional.softplus(h @ w(f"{p}.a").T + w(f"{p}.dt_bias"), threshold=50))
    S = torch.zeros(H, d, m["vdim"], dtype=F64, device=h.device)
    out = torch.empty(T, H, m["vdim"], dtype=F64, device=h.device)
    for t in range(T):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hde,hd->he", S, q[t])
    o = (_rms(out, eps) * w(f"{p}.norm")).reshape(T, -1) * torch.nn.functional.silu(h @ w(f"{p}.g").T)
    return o @ w(f"{p}.o").T


def _parallel(w, p, m, h, eps):
    a, T = m["left"], h.shape[0]
    q = _rms(_heads(h @ w(f"{p}.left.q").T, a["heads"]), eps) * w(f"{p}.left.q.norm")
    k = _rms(_heads(h @ w(f"{p}.left.k").T, a["kv_heads"]), eps) * w(f"{p}.left.k.norm")
    at = torch.arange(1, T + 1, device=h.device)
    q = q * (1.0 + a["q_temp"]["coef"] * torch.log(torch.div(at, a["q_temp"]["every"], rounding_mode="floor").to(F64) + 1))[None, :, None]
    o = _causal(q, k, _heads(h @ w(f"{p}.left.v").T, a["kv_heads"]), a["scale"], extra_one=True) @ w(f"{p}.left.o").T
    return m["left_scale"] * o + m["right_scale"] * _delta_rule(w, f"{p}.right", m["right"], h, eps)


def _pamarax_layers(w, c, xs):
    eps = c["norm"]["eps"]
    mix = {"attention": _gated_attention, "mlstm": _matrix_lstm, "parallel": _parallel}

    def norm(x, name):
        return _rms(x, eps) * (1.0 + w(name))
    for i, L in enumerate(c["layers"]):
        p = f"l{i}"
        for j, x in enumerate(xs):
            x = x + norm(mix[L["type"]](w, f"{p}.mix", L["mixer"], norm(x, f"{p}.norm1"), eps), f"{p}.norm1b")
            h = norm(x, f"{p}.norm2")
            g, u = (h @ w(f"{p}.mlp.{n}").T + w(f"{p}.mlp.{n}.b") for n in ("gate", "up"))
            f = (torch.nn.functional.silu(g) * u) @ w(f"{p}.mlp.down").T + w(f"{p}.mlp.down.b")
            xs[j] = x + norm(f, f"{p}.norm2b")
    return [norm(x, "final.norm") for x in xs]


@torch.no_grad()
def exact(case, seed):
    if case["task"] == "generate":
        return None                                         # (whole token ids: nothing that has a 64-bit value)
    model, c = case["model"], MODELS[case["model"]]
    w = _exact_weights(model)
    seqs, prompt = _sequences(case, seed)
    seqs = seqs + ([prompt] if prompt else [])
    table, head = ("embed", "head") if model == "pamarax" else ("model.embed_tokens.weight",
                                                                "model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight")
    rows = _W64[model][table]
    xs = [rows[torch.tensor(s, device="cuda")].to(F64) for s in seqs]
    xs = (_pamarax_layers if model == "pamarax" else _qwen3_layers)(w, c, xs)
    logits = torch.stack([x[-1] for x in xs]) @ w(head).T
    return {"logits": logits, "tokens": None} if case["dtype"] == "f32" else {"logits": logits}
