"""The work this engine is used for, as cases that can be timed and compared.

A pass goes through the package's public entry points as a user's program calls them.  Two kinds of use:

  replay  `Engine.step_tokens`: token ids in, 32-bit logits out (a caller with a sampler of its own, scoring, an
          evaluation).  Prompts are cut into steps of at most `portion` tokens, ragged prompts share steps; every prompt
          wants the logits of its last `want` rows; then every sequence takes `steps` single tokens, all of whose logits
          are wanted.  With `beside`, a longer prompt of that many tokens is computed in portions in the same steps as the
          single tokens.  Outputs: the logits of every step that wanted some.
  serve   `Engine.generate` (scheduling, sampling on the device, continuous batching) for ragged prompts, greedily, and then
          the score of what came out: the logits behind the last token of every answered prompt.  Outputs: tokens, logits.
          The model's matrices are small beside its tied table here (`matrix_std`), which gives greedy choices a margin far
          above rounding, as a trained model's have; the work does not depend on it.

Sizes are those of the repository's own workloads (bench.py): Qwen3 at 0.6B, 8B and 14B, Kazedra (attention beside a
recurrence) and Ribovik (attention, routed experts) with four layers at widths 1,024 and 4,096.  A program loads a model once
and sends it many requests, so the engine is kept between states of the same case; all that a request leaves in it is given back
at the end of a pass.
"""
import gc
import math

import numpy as np
import torch

from imp_b200 import Engine, EngineConfig, GenerateParams, StepEntry

# ------------------------------------------------------------------------------------------------ models
QWEN3 = {  # layers, width, query heads, kv heads, inner size, tied
    "qwen3-0.6b": (28, 1024, 16, 8, 3072, True), "qwen3-8b": (36, 4096, 32, 8, 12288, False), "qwen3-14b": (40, 5120, 40, 8, 17408, False)}
SHAPES = {"1b": (1024, 16, 8, 3072), "8b": (4096, 32, 8, 12288)}   # of the four-layer models: width, heads, kv heads, inner size
LONGEST = 8192
SEED = 3          # of the weights
HEAD = 128        # head size of all of them
EXPERTS, IDENTITIES, TOP = 32, 2, 8    # of the routed layer: experts of an eighth of the inner size, eight choices and a shared one


def model_config(model):
    if model in QWEN3:
        layers, width, heads, kv, inner, tied = QWEN3[model]
        return {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": layers, "hidden_size": width, "num_attention_heads": heads,
                "num_key_value_heads": kv, "head_dim": HEAD, "intermediate_size": inner, "vocab_size": 151936, "rope_theta": 1e6,
                "rms_norm_eps": 1e-6, "tie_word_embeddings": tied, "torch_dtype": "bfloat16", "max_position_embeddings": LONGEST}
    name, shape = model.split("-")
    width, heads, kv, inner = SHAPES[shape]
    if name == "kazedra":
        left = {"heads": heads, "kv_heads": kv, "dim": HEAD, "vdim": HEAD, "bias_max": 2048, "scale": HEAD ** -0.5,
                "q_temp": {"coef": 0.1, "every": 64}}
        right = {"heads": heads, "kv_heads": kv, "dim": HEAD, "vdim": HEAD, "conv": 4}
        layer = {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0},
                 "mlp": {"kind": "dense", "ff": inner}}
        return {"architecture": "Kazedra", "vocab": 32768, "width": width, "norm": {"eps": 1e-6}, "logit_scale": 1.0, "bias_buckets": 32,
                "layers": [layer] * 4, "max_positions": LONGEST}
    mixer = {"heads": heads, "kv_heads": kv, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5, "mask": {"size": 1024},
             "rot": {"base": 1e6, "dims": HEAD, "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}}
    dense = {"kind": "dense", "ff": inner}
    routed = {"kind": "moe", "expert": {"ff": inner // TOP, "limit": 7.0},
              "router": {"experts": EXPERTS, "identity": IDENTITIES, "top": TOP}, "shared": {"ff": inner // TOP, "limit": 7.0}}
    return {"architecture": "Ribovik", "vocab": 32768, "width": width, "norm": {"eps": 1e-5}, "max_positions": LONGEST,
            "layers": [{"type": "attention", "mixer": mixer, "mlp": routed if i % 3 == 1 else dense} for i in range(4)]}


def vocabulary(model):
    return 151936 if model in QWEN3 else 32768


def matrix_std(case):
    """Standard deviation of the random matrices: about 0.64 / sqrt(width), so that a sublayer adds as much at every width."""
    if case["use"] == "serve":
        return 0.002
    return {"qwen3-0.6b": 0.02, "qwen3-8b": 0.01, "qwen3-14b": 0.009}.get(case["model"], 0.02 if case["model"].endswith("1b") else 0.01)


# ------------------------------------------------------------------------------------------------- cases
def replay(name, model, batch, shortest, longest, steps, want=1, portion=2048, beside=0, dtype="bfloat16"):
    return {"name": name, "use": "replay", "model": model, "dtype": dtype, "batch": batch, "shortest": shortest, "longest": longest,
            "steps": steps, "want": want, "portion": portion, "beside": beside}


def listed():
    return [
        # a short question to the smallest model: the least work a call has, all launches and latency
        replay("one short chat", "qwen3-0.6b", 1, 24, 24, 16),
        # the throughput workload of the small model: 64 requests, prompts of 16 to 1,024 tokens, portions of 512
        {"name": "serve 64 requests", "use": "serve", "model": "qwen3-0.6b", "dtype": "bfloat16", "batch": 64, "shortest": 16, "longest": 1024,
         "steps": 48, "portion": 512},
        # the 32-bit path of the same model: scoring and checking, ragged prompts, then single tokens
        replay("float32 four prompts", "qwen3-0.6b", 4, 33, 257, 8, dtype="float32"),
        # one user of the 8B shape with a document of 2,048 tokens in context: every weight read for each token
        replay("8b one long chat", "qwen3-8b", 1, 2048, 2048, 32),
        # eight users of the 8B shape, prompts of a few hundred tokens
        replay("8b eight chats", "qwen3-8b", 8, 64, 512, 24),
        # a document of 2,048 tokens read at once (the prefill figure of the baseline)
        replay("8b prompt 2048", "qwen3-8b", 1, 2048, 2048, 0),
        # sixteen users keep getting tokens while a new one's document is read in portions
        replay("8b mixed steps", "qwen3-8b", 16, 20, 200, 5, portion=512, beside=2000),
        # the largest shape: a long document in portions beside the tokens of three users
        replay("14b long prompt", "qwen3-14b", 3, 100, 1000, 3, portion=2048, beside=6001),
        # a recurrence beside attention: a document, and eight users' tokens
        replay("kazedra prompt 2048", "kazedra-1b", 1, 2048, 2048, 0),
        replay("kazedra eight chats", "kazedra-8b", 8, 32, 128, 32),
        # routed experts: continuations of eight prompts scored, and sixty-four users' tokens
        replay("ribovik scoring", "ribovik-8b", 8, 150, 350, 0, want=8),
        replay("ribovik 64 chats", "ribovik-8b", 64, 9, 100, 12),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def draw(rng):
    """One more case: model, batch, prompt lengths and steps over the listed cases' ranges; its tokens stay within what the listed
    cases of that model compute."""
    model = rng.choice(["qwen3-0.6b", "qwen3-0.6b", "qwen3-8b", "qwen3-8b", "kazedra-1b", "kazedra-8b", "ribovik-1b", "ribovik-8b"])
    most = 8192 if model != "qwen3-8b" else 4096
    use = "serve" if model == "qwen3-0.6b" and rng.random() < 0.3 else "replay"
    dtype = "float32" if model == "qwen3-0.6b" and use == "replay" and rng.random() < 0.4 else "bfloat16"
    batch = log_int(rng, 1, 64 if use == "serve" else 16 if dtype == "bfloat16" else 4)
    longest = log_int(rng, 9, min(2048, most // batch) if dtype == "bfloat16" else 257)
    shortest = log_int(rng, max(8, longest // 16), longest)
    portion = rng.choice([512, 1024, 2048])
    steps = log_int(rng, 4, 32) if dtype == "bfloat16" else log_int(rng, 1, 8)
    if use == "serve":
        return {"use": "serve", "model": model, "dtype": dtype, "batch": batch, "shortest": shortest, "longest": longest, "steps": steps,
                "portion": portion}
    if model.startswith("ribovik"):   # 64 rows or so each: a choice between two nearly equal experts stays a small part of them
        if rng.random() < 0.5:
            case = replay("", model, rng.randrange(48, 65), 8, log_int(rng, 9, 128), log_int(rng, 4, 16), 1, portion)
        else:
            batch = min(batch, 8)
            case = replay("", model, batch, 64, max(64, longest), 0, 64 // batch, portion)
        case.pop("name")
        return case
    beside = rng.randrange(256, 2049) if dtype == "bfloat16" and rng.random() < 0.25 else 0
    steps = 0 if not beside and longest > 128 and rng.random() < 0.25 else min(steps, 8) if beside else steps
    case = replay("", model, batch, shortest, longest, steps, 1, portion, beside, dtype)
    case.pop("name")
    return case


# ------------------------------------------------------------------------------------------------ inputs
def inputs(case, seed):
    """Prompt token ids per sequence (the `beside` prompt last) and the single tokens [steps, batch] that follow them; the prompts'
    lengths are the case's, the tokens the seed's."""
    vocab, rng = vocabulary(case["model"]), np.random.default_rng([case["batch"], case["shortest"], case["longest"]])
    lengths = rng.integers(case["shortest"], case["longest"] + 1, case["batch"]).tolist()
    rng = np.random.default_rng(seed)
    if case.get("beside"):
        lengths.append(case["beside"])
    prompts = [rng.integers(0, vocab, n).tolist() for n in lengths]
    singles = rng.integers(0, vocab, (case["steps"], case["batch"])).tolist()
    return prompts, singles


def script(case, prompts, singles):
    """Steps of a replay: per step a list of (sequence, tokens, wanted indices)."""
    portion, batch, want = case["portion"], case["batch"], case.get("want", 1)
    out, step, room = [], [], portion

    def put(s, first, tokens, total, rows):
        wanted = [i for i in range(len(tokens)) if first + i >= total - rows]
        step.append((s, tokens, wanted))

    for s, p in enumerate(prompts[:batch]):
        at = 0
        while at < len(p):
            n = min(room, len(p) - at)
            put(s, at, p[at:at + n], len(p), want)
            at, room = at + n, room - n
            if room == 0:
                out.append(step)
                step, room = [], portion
    if step:
        out.append(step)
    at, long = 0, prompts[batch] if case.get("beside") else []
    k = 0
    while k < len(singles) or at < len(long):
        step = [(s, [t], [0]) for s, t in enumerate(singles[k])] if k < len(singles) else []
        n = min(portion - len(step), len(long) - at)
        if n > 0:
            put(batch, at, long[at:at + n], len(long), 1)
            at += n
        out.append(step)
        k += 1
    return out


_engine = {"key": None, "engine": None, "count": 0}


def engine_for(case):
    longest = max(case["longest"] + case["steps"], case.get("beside", 0)) + 8
    seqs = case["batch"] + (1 if case.get("beside") else 0)
    key = (case["model"], case["dtype"], case["use"], case["portion"], longest, seqs, case["longest"] + case["steps"], case.get("beside", 0))
    if _engine["key"] != key:
        old, _engine["engine"], _engine["key"] = _engine["engine"], None, None
        if old is not None:
            old.close()
        del old
        gc.collect()
        torch.cuda.empty_cache()   # what torch holds is not the engine's to use
        pages = 3 * (case["batch"] * -(-(case["longest"] + case["steps"] + 1) // 16) + -(-case.get("beside", 0) // 16) + seqs)
        config = EngineConfig(max_batch_size=max(seqs, 1), max_seq_len=longest, kv_cache_max_blocks=pages, kv_block_size=16,
                              max_batch_tokens=max(2048 if case["use"] == "serve" else case["portion"], seqs),
                              prefill_chunk_size=case["portion"] if case["use"] == "serve" else 0, compute_dtype=case["dtype"])
        _engine["engine"] = Engine.from_random(model_config(case["model"]), config, seed=SEED, std=matrix_std(case))
        _engine["key"] = key
    return _engine["engine"]


def prepare(case, seed):
    """What a program has in hand: the engine with its model, and the requests' token ids."""
    prompts, singles = inputs(case, seed)
    state = {"engine": engine_for(case), "prompts": prompts, "case": case}
    _engine["count"] += 1
    state["id"] = _engine["count"]
    if case["use"] == "replay":
        state["steps"] = [[StepEntry((state["id"], s), tokens, want) for s, tokens, want in step] for step in script(case, prompts, singles)]
    else:
        state["params"] = GenerateParams(max_tokens=case["steps"], temperature=0.0, ignore_eos=True)
    return state


def run_steps(engine, steps):
    """The logits of every step that wanted some; what the sequences held is given back."""
    seen, out = {}, []
    for step in steps:
        logits = engine.step_tokens(step)
        if len(logits):
            out.append(logits)
        for e in step:
            seen[e.rid] = True
    for rid in seen:
        engine.end(rid)
    return out


def run(state):
    engine, case = state["engine"], state["case"]
    if case["use"] == "replay":
        return run_steps(engine, state["steps"])
    tokens = engine.generate(state["prompts"], state["params"])
    whole = [p + t for p, t in zip(state["prompts"], tokens)]
    score = script(dict(case, portion=2048), whole, [])
    logits = run_steps(engine, [[StepEntry((state["id"], s), t, want) for s, t, want in step] for step in score])
    return {"tokens": np.array(tokens, dtype=np.int32), "logits": logits}


# -------------------------------------------------------------------------------------------------- work
def sizes(model):
    """Matrix elements that every token meets (without the head), elements read in a step of n tokens (a function), cached keys and
    values per token and layer, layers, head elements."""
    V = vocabulary(model)
    if model in QWEN3:
        L, d, H, G, F, _ = QWEN3[model]
        per = L * ((H + 2 * G) * HEAD * d + H * HEAD * d + 3 * F * d)
        return per, lambda n: per, 2 * G * HEAD, H * HEAD, L, V * d
    name, shape = model.split("-")
    d, H, G, F = SHAPES[shape]
    if name == "kazedra":
        per = 4 * ((H + G) * HEAD * d + H * HEAD * d + (2 * G + 2 * H) * HEAD * d + 2 * H * d + H * HEAD * d + 3 * F * d)
        return per, lambda n: per, 2 * G * HEAD, H * HEAD, 4, V * d
    outputs, expert = EXPERTS + IDENTITIES, 3 * (F // TOP) * d
    plain = 4 * ((H + 2 * G) * HEAD * d + H * HEAD * d) + 9 * F * d + outputs * d
    per = plain + int((1 + TOP * EXPERTS / outputs) * expert)
    read = lambda n: plain + int((1 + EXPERTS * (1 - (1 - TOP / outputs) ** n)) * expert)  # noqa: E731
    return per, read, 2 * G * HEAD, H * HEAD, 4, V * d


def work(case):
    """Per step: the weights once, the earlier keys and values once, new ones written once, the wanted logits written once;
    two operations a weight and token, four per visible key, query head and head entry; the recurrence's state once a step."""
    model, size = case["model"], 4 if case["dtype"] == "float32" else 2
    per, read, kv, heads, layers, head = sizes(model)
    prompts, singles = inputs(case, 1)
    steps = script(case, prompts, singles if case["use"] == "replay" else [])
    if case["use"] == "serve":
        steps = steps + [[(s, [0], [0]) for s in range(case["batch"])]] * (case["steps"] - 1)
        score = script(dict(case, portion=2048), [p + [0] * case["steps"] for p in prompts], [])
        runs = [steps, score]
    else:
        runs = [steps]
    nbytes = flops = 0.0
    state = 0
    if model.startswith("kazedra"):
        _, H, _, _ = SHAPES[model.split("-")[1]]
        state = layers * H * HEAD * HEAD
    window = 1024 if model.startswith("ribovik") else 1 << 30
    for steps in runs:
        length = {}
        for step in steps:
            tokens = sum(len(t) for _, t, _ in step)
            wanted = sum(len(w) for _, _, w in step)
            nbytes += size * read(tokens) + (size * head + 4.0 * wanted * vocabulary(model) if wanted else 0)
            flops += 2.0 * per * tokens + 2.0 * head * wanted
            for s, t, _ in step:
                a, n = length.get(s, 0), len(t)
                b = a + n
                length[s] = b
                start = a // window * window
                nbytes += layers * kv * size * (b - start) + 8.0 * state
                if window >= b:
                    keys = n * (a + b + 1) / 2
                else:
                    keys = sum(p % window + 1 for p in range(a, b))
                flops += 4.0 * layers * heads * keys + 8.0 * state * n
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Rounding of the element type over a whole model.  Ribovik: some token's eighth and ninth expert are nearly equal, and whoever
    adds in another order may choose the other one; its row then differs by some hundredths."""
    if case["dtype"] == "float32":
        return {"rel": 1e-4, "max": 1e-3}       # 3e-5 from 64 bits after 28 layers
    if case["model"].startswith("ribovik"):
        return {"rel": 0.03, "max": 0.6}        # sums in another order: 0.010, 0.15
    return {"rel": 0.03, "max": 0.2, "differ": 0.0}   # sums in another order: up to 0.011, 0.051; from 64 bits: 0.004 to 0.019


# ----------------------------------------------------------------------------- the same in 64 bits, in plain torch
def signed(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def normals(seed, name, count, first):
    """Elements first ... first + count - 1 of the random tensor `name`: two 24-bit uniforms from a hash of the tensor's seed and the
    index, one normal value from them (Box and Muller), in 32 bits."""
    m64 = (1 << 64) - 1
    h = 0xCBF29CE484222325 ^ (seed * 0x9E3779B97F4A7C15 & m64)
    for c in name.encode():
        h = (h ^ c) * 0x100000001B3 & m64
    h ^= h >> 29
    h = h * 0xBF58476D1CE4E5B9 & m64
    h ^= h >> 32

    def shifted(z, n):
        return z ^ ((z >> n) & ((1 << (64 - n)) - 1))

    z = torch.arange(first + 1, first + 1 + count, device="cuda") * signed(0x9E3779B97F4A7C15) + signed(h)
    z = shifted(z, 30) * signed(0xBF58476D1CE4E5B9)
    z = shifted(z, 27) * signed(0x94D049BB133111EB)
    z = shifted(z, 31)
    u1 = (((z >> 40) & 0xFFFFFF) + 1).float() * (1.0 / 16777216.0)
    u2 = (z & 0xFFFFFF).float() * (1.0 / 16777216.0)
    return torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(6.28318530717958647692 * u2)


class Weights:
    """Random tensors by name, stored in bfloat16 as a checkpoint holds them and widened to 64 bits when asked for."""

    def __init__(self, std):
        self.std, self.made = std, {}

    def __call__(self, name, *shape, norm=False):
        if name not in self.made:
            n, chunk = math.prod(shape), 1 << 27
            t = torch.empty(n, dtype=torch.bfloat16, device="cuda")
            for a in range(0, n, chunk):
                b = min(n, a + chunk)
                v = normals(SEED, name, b - a, a)
                t[a:b] = (1.0 + 0.01 * v if norm else self.std * v).bfloat16()
            self.made[name] = t.view(shape)
        return self.made[name].double()


def rms(x, eps, w=None):
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return x if w is None else x * w


def silu(x):
    return x * torch.sigmoid(x)


def turned_halves(x, first, theta):
    """Rotary positions: entry i of a head turns with entry i + half."""
    half = x.shape[-1] // 2
    f = theta ** (-torch.arange(half, device="cuda", dtype=torch.float64) / half)
    angle = torch.arange(first, first + x.shape[0], device="cuda", dtype=torch.float64)[:, None, None] * f
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos()], -1)


def attend(q, k, v, scale, first, bias=None, sink=None, chunk=0):
    """q [n, H, D] at positions first ..., k and v [first + n, G, D]; `sink`: per head, an extra term exp(sink) in the denominator."""
    n, H, D = q.shape
    L, G = k.shape[0], k.shape[1]
    i, j = torch.arange(first, first + n, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    hidden = j > i
    if chunk:
        hidden = hidden | (i // chunk != j // chunk)
    out = torch.empty(n, H, D, dtype=torch.float64, device="cuda")
    for g in range(G):
        r = slice(g * (H // G), (g + 1) * (H // G))
        s = torch.einsum("nhd,ld->hnl", q[:, r], k[:, g]) * scale
        if bias is not None:
            s = s + bias[r]
        s = s.masked_fill(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[r, None, None].expand(-1, n, 1)], -1)
        p = torch.softmax(s, -1)[..., :L]
        out[:, r] = torch.einsum("hnl,ld->nhd", p, v[:, g])
    return out.reshape(n, H * D)


class Qwen3Exact:
    def __init__(self, model, std):
        self.L, self.d, self.H, self.G, self.F, self.tied = QWEN3[model]
        self.W, self.V = Weights(std), vocabulary(model)

    def stream(self, tokens, caches):
        """The final stream of new tokens, a list per sequence; `caches`: per sequence a list per layer of keys and values, extended here."""
        W, d, H, G, F = self.W, self.d, self.H, self.G, self.F
        lens = [len(t) for t in tokens]
        x = W("model.embed_tokens.weight", self.V, d)[torch.tensor(sum(tokens, []), device="cuda")]
        for i in range(self.L):
            p = "model.layers.%d." % i
            h = rms(x, 1e-6, W(p + "input_layernorm.weight", d, norm=True))
            q = (h @ W(p + "self_attn.q_proj.weight", H * HEAD, d).T).view(-1, H, HEAD)
            k = (h @ W(p + "self_attn.k_proj.weight", G * HEAD, d).T).view(-1, G, HEAD)
            v = (h @ W(p + "self_attn.v_proj.weight", G * HEAD, d).T).view(-1, G, HEAD)
            q = rms(q, 1e-6, W(p + "self_attn.q_norm.weight", HEAD, norm=True)).split(lens)
            k = rms(k, 1e-6, W(p + "self_attn.k_norm.weight", HEAD, norm=True)).split(lens)
            v, got = v.split(lens), []
            for s, cache in enumerate(caches):
                if len(cache) <= i:
                    cache.append((k[s][:0], v[s][:0]))
                old_k, old_v = cache[i]
                first = old_k.shape[0]
                keys, values = torch.cat([old_k, turned_halves(k[s], first, 1e6)]), torch.cat([old_v, v[s]])
                cache[i] = (keys, values)
                got.append(attend(turned_halves(q[s], first, 1e6), keys, values, HEAD ** -0.5, first))
            x = x + torch.cat(got) @ W(p + "self_attn.o_proj.weight", d, H * HEAD).T
            h = rms(x, 1e-6, W(p + "post_attention_layernorm.weight", d, norm=True))
            h = silu(h @ W(p + "mlp.gate_proj.weight", F, d).T) * (h @ W(p + "mlp.up_proj.weight", F, d).T)
            x = x + h @ W(p + "mlp.down_proj.weight", d, F).T
        return x.split(lens)

    def logits(self, x):
        x = rms(x, 1e-6, self.W("model.norm.weight", self.d, norm=True))
        return x @ self.W("model.embed_tokens.weight" if self.tied else "lm_head.weight", self.V, self.d).T


class KazedraExact:
    def __init__(self, model, std):
        self.d, self.H, self.G, self.F = SHAPES[model.split("-")[1]]
        self.W, self.V, self.biases = Weights(std), vocabulary(model), {}

    def buckets(self, n):
        """Bucket of every distance below n: the first half of 32 as they are, then by the logarithm up to 2,048."""
        exact = [i if i < 16 else min(31, 16 + int(math.log(i / 16) / math.log(2048 / 16) * 16)) for i in range(n)]
        return torch.tensor(exact, device="cuda")

    def attention(self, h, p):
        W, d, H, G = self.W, self.d, self.H, self.G
        T = h.shape[0]
        q = h @ W(p + "q", H * HEAD, d).T + W(p + "q.b", H * HEAD)
        k = h @ W(p + "k", G * HEAD, d).T + W(p + "k.b", G * HEAD)
        v = k.view(T, G, HEAD)
        pos = torch.arange(T, device="cuda", dtype=torch.float64)
        warm = 1.0 + 0.1 * torch.log(torch.floor((pos + 1) / 64) + 1)
        q = rms(q, 1e-6, W(p + "q.norm", H * HEAD, norm=True)) * warm[:, None]
        k = rms(k, 1e-6, W(p + "k.norm", G * HEAD, norm=True))
        apart = (pos[:, None] - pos[None]).clamp(min=0).long()
        bias = W(p + "rel", 32, H)[self.buckets(T)[apart]].permute(2, 0, 1)
        out = attend(q.view(T, H, HEAD), k.view(T, G, HEAD), v, HEAD ** -0.5, 0, bias, W(p + "sink", H))
        return out @ W(p + "o", d, H * HEAD).T + W(p + "o.b", d)

    def delta(self, h, p):
        W, d, H, G = self.W, self.d, self.H, self.G
        T = h.shape[0]

        def mixed(name, n):
            y = torch.nn.functional.pad(h @ W(p + name, n * HEAD, d).T, (0, 0, 3, 0))
            taps = W(p + name + ".conv", n * HEAD, 4)
            return silu(sum(y[j:j + T] * taps[:, j] for j in range(4))).view(T, n, HEAD)

        def unit(x):
            return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)

        q, k, v = unit(mixed("q", G)) * HEAD ** -0.5, unit(mixed("k", G)), mixed("v", H)
        q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
        beta = torch.sigmoid(h @ W(p + "b", H, d).T)
        keep = torch.exp(-torch.exp(W(p + "A_log", H)) * torch.nn.functional.softplus(h @ W(p + "a", H, d).T + W(p + "dt_bias", H)))
        S = torch.zeros(H, HEAD, HEAD, dtype=torch.float64, device="cuda")
        out = torch.empty(T, H, HEAD, dtype=torch.float64, device="cuda")
        for t in range(T):
            S = S * keep[t, :, None, None]
            u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
            S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
            out[t] = torch.bmm(q[t, :, None], S)[:, 0]
        out = rms(out, 1e-6, W(p + "norm", HEAD, norm=True)) * silu(h @ W(p + "g", H * HEAD, d).T).view(T, H, HEAD)
        return out.reshape(T, H * HEAD) @ W(p + "o", d, H * HEAD).T

    def stream(self, tokens, caches):
        W, d, F = self.W, self.d, self.F
        out = []
        for t in tokens:
            x = W("embed", self.V, d)[torch.tensor(t, device="cuda")]
            for i in range(4):
                p = "l%d." % i
                h = rms(x, 1e-6, 1.0 + W(p + "norm1", d, norm=True))
                x = x + self.attention(h, p + "mix.left.") + self.delta(h, p + "mix.right.")
                h = rms(x, 1e-6, 1.0 + W(p + "norm2", d, norm=True))
                h = silu(h @ W(p + "mlp.gate", F, d).T) * (h @ W(p + "mlp.up", F, d).T)
                x = x + h @ W(p + "mlp.down", d, F).T
            out.append(x)
        return out

    def logits(self, x):
        return rms(x, 1e-6, 1.0 + self.W("final.norm", self.d, norm=True)) @ self.W("head", self.V, self.d).T


class RibovikExact:
    def __init__(self, model, std):
        self.d, self.H, self.G, self.F = SHAPES[model.split("-")[1]]
        self.W, self.V = Weights(std), vocabulary(model)
        base, half, factor, original = 1e6, HEAD // 2, 4.0, 2048.0

        def index(turns):   # the (real) index of the pair that turns that often over `original` positions
            return half * math.log(original / (2 * math.pi * turns)) / math.log(base)

        lo, hi = max(math.floor(index(32.0)), 0), min(math.ceil(index(1.0)), HEAD - 1)
        i = torch.arange(half, device="cuda", dtype=torch.float64)
        f, slow = base ** (-i / half), ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        self.f, self.stretch = f / factor * slow + f * (1 - slow), 0.1 * math.log(factor) + 1.0

    def turned(self, x):
        angle = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None, None] * self.f
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos()], -1).flatten(-2) * self.stretch

    def expert(self, h, p):
        W, d, F = self.W, self.d, self.F // TOP
        g, u = (h @ W(p + "gate", F, d).T).clamp(max=7.0), (h @ W(p + "up", F, d).T).clamp(-7.0, 7.0)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ W(p + "down", d, F).T

    def routed(self, h, p):
        W = self.W
        n = EXPERTS + IDENTITIES
        s = torch.softmax(h @ W(p + "router", n, self.d).T, -1)
        chosen = (s + W(p + "correction", n)).topk(TOP, -1).indices
        w = s.gather(1, chosen)
        w = w / (w.sum(-1, keepdim=True) + 1e-20)
        out = self.expert(h, p + "shared.")
        for e in range(n):
            row, at = (chosen == e).nonzero(as_tuple=True)
            if len(row):
                y = self.expert(h[row], p + "e%d." % e) if e < EXPERTS else h[row]
                out = out.index_add(0, row, w[row, at][:, None] * y)
        return out

    def stream(self, tokens, caches):
        W, d, H, G, F = self.W, self.d, self.H, self.G, self.F
        lens = [len(t) for t in tokens]
        x = rms(W("embed", self.V, d)[torch.tensor(sum(tokens, []), device="cuda")], 1e-5, W("embed.norm", d, norm=True))
        for i in range(4):
            p = "l%d.mix." % i
            q, k, v = (((x @ W(p + n, m * HEAD, d).T) + W(p + n + ".b", m * HEAD)).view(-1, m, HEAD).split(lens) for n, m in (("q", H), ("k", G), ("v", G)))
            got = [attend(rms(self.turned(q[s]), 1e-5), rms(self.turned(k[s]), 1e-5), v[s], HEAD ** -0.5, 0,
                          sink=torch.zeros(H, dtype=torch.float64, device="cuda"), chunk=1024) for s in range(len(lens))]
            x = x + rms(torch.cat(got) @ W(p + "o", d, H * HEAD).T, 1e-5, W("l%d.norm1" % i, d, norm=True))
            p = "l%d.mlp." % i
            if i % 3 == 1:
                y = self.routed(x, p)
            else:
                y = silu(x @ W(p + "gate", F, d).T + W(p + "gate.b", F)) * (x @ W(p + "up", F, d).T + W(p + "up.b", F))
                y = y @ W(p + "down", d, F).T + W(p + "down.b", d)
            x = x + rms(y, 1e-5, W("l%d.norm2" % i, d, norm=True))
        return x.split(lens)

    def logits(self, x):
        return rms(x, 1e-5, self.W("final.norm", self.d, norm=True)) @ self.W("embed", self.V, self.d).T


def exact(case, seed):
    if case["model"] == "qwen3-14b":
        return None   # takes longer than is useful
    with torch.no_grad():
        prompts, singles = inputs(case, seed)
        kind = Qwen3Exact if case["model"] in QWEN3 else KazedraExact if case["model"].startswith("kazedra") else RibovikExact
        m = kind(case["model"], matrix_std(case))
        if case["use"] == "serve":
            caches, new, answers = [[] for _ in prompts], prompts, [[] for _ in prompts]
            for _ in range(case["steps"] + 1):
                x = torch.stack([s[-1] for s in m.stream(new, caches)])
                rows = m.logits(x)
                new = [[t] for t in rows.argmax(-1).tolist()]
                for a, t in zip(answers, new):
                    a.append(t[0])
            tokens = [a[:case["steps"]] for a in answers]
            whole, last = [p + t for p, t in zip(prompts, tokens)], rows
            steps = script(dict(case, portion=2048), whole, [])
            logits = [last[[s for s, _, w in step if w]].cpu().numpy() for step in steps if any(w for _, _, w in step)]
            return {"tokens": None, "logits": logits}
        streams = m.stream([p + [row[s] for row in singles] if s < case["batch"] else p for s, p in enumerate(prompts)], [[] for _ in prompts])
        out, length = [], {}
        for step in script(case, prompts, singles):
            rows = []
            for s, t, want in step:
                a = length.get(s, 0)
                length[s] = a + len(t)
                rows += [streams[s][a + i] for i in want]
            if rows:
                out.append(m.logits(torch.stack(rows)).cpu().numpy())
        return out
