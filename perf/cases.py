"""What this engine's speed is measured on: passes that a user's program has it run, through its public entry points.

A pass is either

* a run of the step function (``make_runner`` / ``ModelRunner.step``, what ``bin/trace_run`` drives): the prompts of some
  requests in steps of at most 2,048 tokens, then decode steps in which every request brings its next, given token, and
  the requests are given back; its outputs are the logits; or
* ``LLMEngine.generate``: the scheduler, the steps and the sampler; its outputs are the tokens.

Models have random weights at sizes that ``bench.py`` measures: the GPT-2 style decoder at the 50M, GPT-2 small and GPT-2
XL sizes (XL with 4 of its 48 layers, so that the inputs are made quickly) and with heads of 128, Fakilorn (grouped heads,
routed experts) and Nogatar (attention over latents, mLSTM, routed experts) at a width of 1,024.

``exact`` repeats the model in 64 bits, whole sequences at a time, in plain torch.
"""

from __future__ import annotations

import math
import random

import torch

from mini_gpt_inference_b200 import EngineConfig, FakilornConfig, GPTConfig, LLMEngine, NogatarConfig, SamplingParams
from mini_gpt_inference_b200.config import lookup
from mini_gpt_inference_b200.engine import StepEntry, load_model, make_runner
from mini_gpt_inference_b200.kernels.ops import default_ops
from mini_gpt_inference_b200.parts import DecoderModel

STEP_TOKENS = 2048          # most tokens of one step, the engine's default
DEVICE = "cuda:0"


# ---- models ---------------------------------------------------------------------------------------
def _gpt(vocab, positions, layers, heads, width, inner, bias=True):
    return dict(vocab_size=vocab, n_positions=positions, n_layer=layers, n_head=heads, n_embd=width, n_inner=inner,
                bias=bias, layer_norm_epsilon=1e-5)


def _experts(ff):
    return {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": 8, "top": 2}, "shared": {"ff": ff}}


_FAKILORN_MIXER = {"heads": 16, "kv_heads": 4, "dim": 64, "vdim": 64, "scale": 0.125, "v_mix": True}
_LATENT = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "mask": {"size": 512},
           "rot": {"dims": 64, "base": 10000.0, "scaling": {"factor": 4.0, "original": 512, "fast": 32.0, "slow": 1.0}}}
_MLSTM = {"heads": 8, "dim": 64, "vdim": 128, "gate_cap": 10.0}

MODELS = {
    "50m": _gpt(50304, 2048, 8, 8, 512, 2048),
    "gpt2-small": _gpt(50257, 1024, 12, 12, 768, 3072),
    "gpt2-xl-4-layers": _gpt(50257, 1024, 4, 25, 1600, 6400),
    "heads-of-128": _gpt(32000, 2112, 2, 16, 2048, 8192, bias=False),
    "fakilorn": {"architecture": "Fakilorn", "vocab": 32000, "width": 1024, "embedding": {"scale": 1.0}, "logit_scale": 1.0,
                 "norm": {"eps": 1e-5},
                 "layers": [{"type": "attention", "mixer": _FAKILORN_MIXER,
                             "mlp": _experts(1024) if i % 2 else {"kind": "dense", "ff": 4096}} for i in range(4)]},
    "nogatar": {"architecture": "Nogatar", "vocab": 32000, "width": 1024, "norm": {"eps": 1e-6},
                "embedding": {"scale": 32.0}, "residual_mult": 0.2, "logit_softcap": 30.0,
                "layers": [{"type": kind, "mixer": _MLSTM if kind == "mlstm" else _LATENT, "mlp": _experts(1024)}
                           for kind in ("latent_attention", "mlstm", "latent_attention", "latent_attention")]},
}


def _config(name):
    raw = MODELS[name]
    kind = {"Fakilorn": FakilornConfig, "Nogatar": NogatarConfig}.get(raw.get("architecture"), GPTConfig)
    return kind.from_dict(raw)


def _weights(case, seed):
    """Random weights on the GPU, in the dtype in which a checkpoint holds them (by the scheme of ``random_tensors``)."""
    cfg = _config(case["model"])
    model = DecoderModel(lookup(cfg.architecture).describe(cfg))
    gen = torch.Generator(device=DEVICE).manual_seed(1000 + seed)
    n_layer, out = max(1, len(model.layers)), {}
    for name, spec in sorted(model.tensor_specs().items()):
        if spec.optional_alias_of is not None or spec.optional:
            continue
        noise = torch.randn(spec.init_shape, generator=gen, device=DEVICE)
        fan_in = spec.init_shape[-1] if spec.init_shape else 1
        t = {"residual_proj": lambda: noise * (0.02 / math.sqrt(2 * n_layer)), "norm_gain": lambda: 1.0 + 0.1 * noise,
             "norm_shift": lambda: 0.1 * noise, "unit_interval": lambda: torch.sigmoid(noise),
             "fan_in": lambda: noise / math.sqrt(fan_in), "fan_in_residual": lambda: noise / math.sqrt(fan_in * 2 * n_layer),
             "unit_normal": lambda: noise}.get(spec.init, lambda: 0.02 * noise)()
        if case["generate"] and name == "tok_emb.weight":
            # A model in use is sure of most of its tokens; five times the usual embedding makes this one sure of them
            # (the largest logit stands far off), so that no choice of a token hangs on the last bit of a logit.
            t = 5.0 * t
        if name.endswith("mlp.router"):
            # Router logits of this spread, as training leaves them: where two experts tie, the one that rounding chooses
            # has little weight.
            t = 5.0 * noise / math.sqrt(fan_in)
        out[name] = t.to(getattr(torch, case["dtype"]))
    return cfg, out


# ---- requests -------------------------------------------------------------------------------------
def _lengths(case):
    """Prompt lengths: all the same, or spread (by their logarithm) from an eighth of ``prompt`` to ``prompt``."""
    if not case["ragged"]:
        return [case["prompt"]] * case["requests"]
    rng = random.Random(case["prompt"] * 131 + case["requests"])
    return [max(1, round(case["prompt"] * 8.0 ** -rng.random())) for _ in range(case["requests"])]


def _sequences(case, seed):
    """Per request its prompt and the tokens that follow, which the decode steps bring."""
    gen = torch.Generator().manual_seed(seed)
    vocab = MODELS[case["model"]].get("vocab_size") or MODELS[case["model"]]["vocab"]
    return [torch.randint(0, vocab, (n + case["new"],), generator=gen).tolist() for n in _lengths(case)]


def _portions(case):
    """The prompts' steps: lists of (request, first token, tokens) of at most STEP_TOKENS tokens together."""
    steps, room = [], 0
    for r, n in enumerate(_lengths(case)):
        at = 0
        while at < n:
            if room == 0:
                steps.append([])
                room = STEP_TOKENS
            take = min(room, n - at)
            steps[-1].append((r, at, take))
            at, room = at + take, room - take
    return steps


# ---- what is measured --------------------------------------------------------------------------------
def _case(name, model, requests, prompt, new, dtype="bfloat16", ragged=False, want="last", page=64, generate=False):
    return dict(name=name, model=model, dtype=dtype, requests=requests, prompt=prompt, ragged=ragged, new=new, want=want,
                page=page, generate=generate)


def listed():
    return [
        # one user's short turn: every launch is a few tokens, the smallest work there is
        _case("chat_turn", "50m", 1, 23, 16, page=16),
        # the benchmark's headline: a batch of 8 whose contexts approach the end of the position table
        _case("decode_batch8_long", "50m", 8, 1999, 48),
        # a full server: 64 requests of different lengths decode together
        _case("decode_batch64", "50m", 64, 413, 8, ragged=True),
        # one prompt that fills a step
        _case("prompt_2048", "50m", 1, 2048, 0),
        # several odd prompts in one step, small pages
        _case("prompts_ragged", "50m", 11, 389, 0, ragged=True, page=16),
        # scoring a text: the logits of all its positions
        _case("score_text", "50m", 1, 511, 0, want="all"),
        # the 32-bit path: several prompts, then decoding
        _case("float32_batch8", "50m", 8, 509, 8, dtype="float32"),
        # the widest layers that are measured: prompts, then decoding at batch 4
        _case("wide_layers", "gpt2-xl-4-layers", 4, 511, 16),
        # heads of 128: one prompt that fills a step, then decoding alone
        _case("heads_of_128", "heads-of-128", 1, 2048, 8),
        # the whole engine: scheduler, mixed steps, overlapped decoding, greedy and drawn tokens
        _case("serve", "50m", 24, 301, 32, ragged=True, generate=True, page=16),
        # grouped heads and routed experts: prompts and decoding
        _case("fakilorn", "fakilorn", 3, 1279, 20),
        # attention over latents with a window, a matrix memory and experts in every layer
        _case("nogatar", "nogatar", 4, 1021, 16),
    ]


def _log(rng, low, high):
    return min(high, max(low, int(round(low * (high / low) ** rng.random()))))


def draw(rng: random.Random):
    """A case of the listed ones' ranges: a model and a dtype, 1 to 64 requests, prompts of 1 token to the end of the
    position table, and no more tokens, logits and decode steps than the largest listed case of that model has."""
    model, dtype, most, requests = rng.choice(
        [("50m", "bfloat16", 12000, 64)] * 4 + [("50m", "float32", 4000, 8), ("gpt2-small", "bfloat16", 6000, 48),
         ("gpt2-xl-4-layers", "bfloat16", 2000, 32), ("heads-of-128", "bfloat16", 2000, 32),
         ("fakilorn", "bfloat16", 4000, 32), ("fakilorn", "float32", 1000, 4), ("nogatar", "bfloat16", 4000, 8)])
    generate = model == "50m" and dtype == "bfloat16" and rng.random() < 0.2
    requests = _log(rng, 1, requests)
    new = rng.choice([0, _log(rng, 1, 40)]) if not generate else _log(rng, 2, 40)
    new = min(new, max(1, 400 // requests))
    table = MODELS[model].get("n_positions", 2048)
    prompt = _log(rng, 1, min(table - new, most // requests - new))
    want = "all" if not new and prompt * requests <= 700 and rng.random() < 0.5 else "last"
    return dict(model=model, dtype=dtype, requests=requests, prompt=prompt, ragged=requests > 1 and rng.random() < 0.6,
                new=new, want=want, page=rng.choice([16, 64]), generate=generate)


def prepare(case, seed):
    cfg, tensors = _weights(case, seed)
    loaded = load_model(config=cfg, tensors=tensors, dtype=case["dtype"], device=DEVICE)
    sequences, lengths, page = _sequences(case, seed), _lengths(case), case["page"]
    pages = sum(-(-(n + case["new"]) // page) for n in lengths) + 4
    if case["generate"]:
        engine = LLMEngine(loaded, EngineConfig(block_size=page, num_blocks=pages, max_batch_size=case["requests"],
                                                dtype=case["dtype"], device=DEVICE))
        engine.warm_up()
        # greedy and drawn in turn; a nucleus of this share holds the one token that the model is sure of
        params = [SamplingParams(max_tokens=case["new"], temperature=0.0) if r % 2 else
                  SamplingParams(max_tokens=case["new"], temperature=0.8, top_k=50, top_p=0.8, seed=seed + r)
                  for r in range(case["requests"])]
        return {"engine": engine, "prompts": [s[:n] for s, n in zip(sequences, lengths)], "params": params}
    runner = make_runner(loaded, default_ops(DEVICE), page, pages, case["requests"], max_step_tokens=STEP_TOKENS)
    names = [f"r{i}" for i in range(case["requests"])]
    prompts = []
    for step in _portions(case):
        entries = []
        for r, at, take in step:
            last = at + take == lengths[r]
            want = list(range(take)) if case["want"] == "all" else [take - 1] if last else []
            entries.append(StepEntry(names[r], sequences[r][at: at + take], want))
        prompts.append(entries)
    decode = [[StepEntry(names[r], [sequences[r][n + k]], [0]) for r, n in enumerate(lengths)] for k in range(case["new"])]
    return {"runner": runner, "names": names, "prompts": prompts, "decode": decode}


def run(state):
    if "engine" in state:
        results = state["engine"].generate(state["prompts"], state["params"])
        return torch.tensor([r["token_ids"] for r in results])
    runner = state["runner"]
    prompts = [logits for logits in (runner.step(entries) for entries in state["prompts"]) if logits is not None]
    decode = [runner.step(entries) for entries in state["decode"]]
    for name in state["names"]:
        runner.finish(name)
    out = {"prompts": torch.cat(prompts) if len(prompts) > 1 else prompts[0]}
    if decode:
        out["decode"] = torch.stack(decode)
    return out


# ---- what a pass cannot do without ------------------------------------------------------------------------
def _per_layer(raw):
    """Per layer: (weights that every token meets, experts, weights of one, experts a token chooses, multiply-adds per
    pair of query and key, cached values per token, window, multiply-adds of a token's state update and read-out)."""
    if "vocab" not in raw:
        c, f = raw["n_embd"], raw["n_inner"]
        return [(4 * c * c + 2 * c * f, 0, 0, 0, 2 * c, 2 * c, None, 0)] * raw["n_layer"]
    c, rows = raw["width"], []
    for layer in raw["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        window = (m.get("mask") or {}).get("size")
        h, d, dv = m["heads"], m["dim"], m["vdim"]
        if raw["architecture"] == "Fakilorn":
            own = c * (2 * h * dv + h * d + m["kv_heads"] * (d + dv))
            attention, cached, memory, matrices = h * (d + dv), m["kv_heads"] * (d + dv), 0, 3
        elif layer["type"] == "mlstm":
            own = c * (2 * h * d + 3 * h * dv + 2 * h)
            attention, cached, memory, matrices = 0, 0, 2 * h * (d + 1) * dv, 2
        else:
            rank, rot = m["kv_rank"], m["rot_dim"]
            own = c * (h * (d + rot) + rank + rot + h * dv) + rank * h * (d + dv)
            attention, cached, memory, matrices = h * (d + rot + dv), rank + rot, 0, 2
        if f["kind"] == "moe":
            one = matrices * c * f["expert"]["ff"]
            rows.append((own + one + c * (f["router"]["experts"] + 1), f["router"]["experts"], one, f["router"]["top"],
                         attention, cached, window, memory))
        else:
            rows.append((own + 2 * c * f["ff"], 0, 0, 0, attention, cached, window, memory))
    return rows


def work(case):
    """Every matrix once a step (of the experts as many as the step's tokens can choose), the cached keys and values of
    the contexts once a step, the wanted logits written; two operations a multiply-add."""
    raw, lengths, size = MODELS[case["model"]], _lengths(case), 2 if case["dtype"] == "bfloat16" else 4
    rows = _per_layer(raw)
    width, vocab = raw.get("n_embd") or raw["width"], raw.get("vocab_size") or raw["vocab"]
    steps = []                                                  # per step: (tokens before, tokens, wanted) of each request
    for step in _portions(case):
        steps.append([(at, n, n if case["want"] == "all" else int(at + n == lengths[r])) for r, at, n in step])
    # generate: the prompt's last position gives the first token
    for k in range(case["new"] - 1 if case["generate"] else case["new"]):
        steps.append([(n + k, 1, 1) for n in lengths])
    nbytes = flops = 0
    for step in steps:
        tokens, wanted = sum(n for _, n, _ in step), sum(w for _, _, w in step)
        if wanted:
            nbytes += vocab * width * size + 4 * wanted * vocab
            flops += 2 * wanted * vocab * width
        for own, experts, one, top, attention, cached, window, memory in rows:
            nbytes += size * (own + one * min(experts, tokens * top))
            flops += 2 * tokens * (own + one * top + memory)
            for before, n, _ in step:
                reach = before if window is None else min(before, window)
                nbytes += size * cached * (reach + 2 * n)
                for_window = [min(before + i + 1, window) for i in range(n)] if window else None
                pairs = sum(for_window) if window else n * before + n * (n + 1) // 2
                flops += 2 * attention * pairs
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["generate"]:
        return {"rel": 0.0, "max": 0.0, "differ": 0.005}          # tokens; no choice is close (see _weights)
    # about four times what these kernels are off from ``exact`` (in brackets)
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 6e-5}                         # 32-bit sums in another order (2.6e-6, 1.6e-5)
    if case["model"] in ("fakilorn", "nogatar"):
        # bfloat16 activations, and here and there a row for which rounding chose another expert (0.013, 0.38)
        return {"rel": 0.03, "max": 0.9}
    return {"rel": 0.015, "max": 0.08}                            # bfloat16 activations between the products (0.004, 0.02)


# ---- the same in 64 bits ------------------------------------------------------------------------------------
def _norm(x, w, b, eps):
    d = x - x.mean(-1, keepdim=True)
    y = d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w
    return y if b is None else y + b


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window=None, sink=None):
    """q ``[T, H, d]``, k ``[T, G, d]``, v ``[T, G, e]``: causal softmax attention, head by head; ``sink`` adds one term per
    head to the softmax's sum."""
    t, per = q.shape[0], q.shape[1] // k.shape[1]
    gap = torch.arange(t, device=q.device)[:, None] - torch.arange(t, device=q.device)[None, :]
    hidden = (gap < 0) | (gap >= (window or t))
    out = []
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // per].T * scale).masked_fill(hidden, -math.inf)
        top = s.amax(-1, keepdim=True) if sink is None else s.amax(-1, keepdim=True).clamp_min(float(sink[h]))
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[h] - top))
        out.append(e / total @ v[:, h // per])
    return torch.cat(out, dim=-1)


def _exact_gpt(raw, w, ids):
    c, heads, eps = raw["n_embd"], raw["n_head"], raw["layer_norm_epsilon"]
    d = c // heads

    def linear(x, name):
        y = x @ w[name + ".weight"].T
        return y + w[name + ".bias"] if raw["bias"] else y

    def norm(x, name):
        return _norm(x, w[name + ".weight"], w.get(name + ".bias"), eps)

    x = w["tok_emb.weight"][ids] + w["pos_emb.weight"][: len(ids)]
    for i in range(raw["n_layer"]):
        p = f"blocks.{i}."
        q, k, v = (t.view(-1, heads, d) for t in linear(norm(x, p + "ln1"), p + "attn.qkv").split(c, dim=-1))
        x = x + linear(_attend(q, k, v, d ** -0.5), p + "attn.proj")
        u = linear(norm(x, p + "ln2"), p + "mlp.fc")
        u = 0.5 * u * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (u + 0.044715 * u ** 3)))
        x = x + linear(u, p + "mlp.proj")
    return norm(x, "ln_f"), w["tok_emb.weight"]


def _exact_experts(h, weights, ids, n, expert):
    out = torch.zeros_like(h)
    for e in range(n):
        share = (weights * (ids == e)).sum(-1)
        rows = share.nonzero().flatten()
        out[rows] += share[rows, None] * expert(h[rows], f"e{e}.")
    return out


def _exact_fakilorn(raw, w, ids):
    eps, x, first = raw["norm"]["eps"], w["embed"][ids] * raw["embedding"]["scale"], None
    for i, layer in enumerate(raw["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        h = _norm(x, w[p + "norm1"], w[p + "norm1.b"], eps)
        q = _unit((h @ w[p + "mix.q"].T).view(-1, m["heads"], m["dim"]), eps)
        k = _unit((h @ w[p + "mix.k"].T).view(-1, m["kv_heads"], m["dim"]), eps)
        v = (h @ w[p + "mix.v"].T).view(-1, m["kv_heads"], m["vdim"])
        if first is None:
            first = v
        else:
            v = (1.0 - w[p + "mix.vmix"]) * v + w[p + "mix.vmix"] * first
        x = x + (_attend(q, k, v, m["scale"]) * torch.sigmoid(h @ w[p + "mix.g"].T)) @ w[p + "mix.o"].T
        h = _norm(x, w[p + "norm2"], w[p + "norm2.b"], eps)
        if f["kind"] == "dense":
            x = x + torch.relu(h @ w[p + "mlp.up"].T) ** 2 @ w[p + "mlp.down"].T
            continue

        def expert(h, e, p=p):
            a = h @ w[p + "mlp." + e + "gate"].T
            return (a * torch.sigmoid(a) * (h @ w[p + "mlp." + e + "up"].T)) @ w[p + "mlp." + e + "down"].T

        best, chosen = torch.topk(h @ w[p + "mlp.router"].T, f["router"]["top"], dim=-1)
        x = x + _exact_experts(h, torch.softmax(best, -1), chosen, f["router"]["experts"], expert)
        x = x + torch.sigmoid(h @ w[p + "mlp.shared.sg"].T) * expert(h, "shared.")
    return _norm(x, w["final.norm"], w["final.norm.b"], eps) * raw["logit_scale"], w["embed"]


def _rotary(m, t):
    """Cosines and sines ``[t, rot / 2]`` of the stretched frequencies (YaRN's ramp over the pairs)."""
    n, base, s = m["rot_dim"], m["rot"]["base"], m["rot"]["scaling"]

    def pair_of(turns):
        return n * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    low, high = max(math.floor(pair_of(s["fast"])), 0), min(math.ceil(pair_of(s["slow"])), n - 1)
    i = torch.arange(n // 2, dtype=torch.float64, device=DEVICE)
    ramp = ((i - low) / max(high - low, 0.001)).clamp(0, 1)
    freq = base ** (-2 * i / n) * (ramp / s["factor"] + 1 - ramp)
    angle = torch.arange(t, dtype=torch.float64, device=DEVICE)[:, None] * freq
    size = 0.1 * math.log(s["factor"]) + 1.0
    return size * torch.cos(angle)[:, None], size * torch.sin(angle)[:, None]


def _rotate(x, cos, sin):
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * cos - v * sin, v * cos + u * sin], dim=-1).flatten(-2)


def _exact_latent(h, w, p, m, eps):
    heads, d, rank, t = m["heads"], m["dim"], m["kv_rank"], h.shape[0]
    cos, sin = _rotary(m, t)
    q = (h @ w[p + "q"].T).view(t, heads, d + m["rot_dim"])
    low = h @ w[p + "dkv"].T
    c = _unit(low[:, :rank], eps) * w[p + "dkv.norm"]
    shared = _rotate(low[:, rank:].view(t, 1, -1), cos, sin).expand(t, heads, -1)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], cos, sin)], dim=-1)
    k = torch.cat([(c @ w[p + "uk"].T).view(t, heads, d), shared], dim=-1)
    v = (c @ w[p + "uv"].T).view(t, heads, m["vdim"])
    return _attend(q, k, v, m["scale"], m["mask"]["size"], w[p + "sink"]) @ w[p + "o"].T


def _exact_mlstm(h, w, p, m, eps):
    t, heads, d, e, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q = (h @ w[p + "q"].T).view(t, heads, d) * d ** -0.5
    k = (h @ w[p + "k"].T).view(t, heads, d)
    v = (h @ w[p + "v"].T).view(t, heads, e)
    gate_in = cap * torch.tanh((h @ w[p + "i"].T + w[p + "i.b"]) / cap)
    keep = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w[p + "f"].T + w[p + "f.b"]) / cap))
    # The recurrence S_t = e^(f + m' - m) S' + e^(i - m) k v^T with running maximum m, written as a sum over the tokens so
    # far: token j weighs e^(F_t - F_j + i_j - m_t) with F the running sum of f, and m_t the largest exponent or F_t.
    total = keep.cumsum(0)
    out = []
    for head in range(heads):
        a = total[:, head, None] - total[None, :, head] + gate_in[None, :, head]
        a = a.masked_fill(torch.ones(t, t, dtype=torch.bool, device=h.device).triu(1), -math.inf)
        top = torch.maximum(a.amax(-1), total[:, head])
        s = torch.exp(a - top[:, None]) * (q[:, head] @ k[:, head].T)
        out.append(s @ v[:, head] / (torch.maximum(s.sum(-1).abs(), torch.exp(-top)) + 1e-6)[:, None])
    o = _unit(torch.stack(out, dim=1), eps).reshape(t, heads * e) * w[p + "norm"]
    return (o * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T


def _exact_nogatar(raw, w, ids):
    eps, mult = raw["norm"]["eps"], raw["residual_mult"]
    x = w["embed"][ids] * raw["embedding"]["scale"]
    for i, layer in enumerate(raw["layers"]):
        p, router = f"l{i}.", layer["mlp"]["router"]
        mixer = _exact_mlstm if layer["type"] == "mlstm" else _exact_latent
        x = x + mult * _norm(mixer(x, w, p + "mix.", layer["mixer"], eps), w[p + "norm1"], None, eps)

        def expert(h, e, p=p):
            return torch.relu(h @ w[p + "mlp." + e + "up"].T) ** 2 @ w[p + "mlp." + e + "down"].T

        best, chosen = torch.topk(torch.softmax(x @ w[p + "mlp.router"].T, -1), router["top"], dim=-1)
        y = _exact_experts(x, best / (best.sum(-1, keepdim=True) + 1e-20), chosen, router["experts"], expert)
        y = y + torch.sigmoid(x @ w[p + "mlp.shared.sg"].T) * expert(x, "shared.")
        x = x + mult * _norm(y, w[p + "norm2"], None, eps)
    return _norm(x, w["final.norm"], None, eps), w["head"]


def exact(case, seed):
    if case["generate"]:
        return None                                             # tokens have no 64-bit value
    raw = MODELS[case["model"]]
    _, tensors = _weights(case, seed)
    w = {name: t.double() for name, t in tensors.items()}
    forward = {"Fakilorn": _exact_fakilorn, "Nogatar": _exact_nogatar}.get(raw.get("architecture"), _exact_gpt)
    rows, head = [], None                                       # per request: its final rows from the first wanted one on
    lengths = _lengths(case)
    for n, sequence in zip(lengths, _sequences(case, seed)):
        y, head = forward(raw, w, torch.tensor(sequence, device=DEVICE))
        rows.append(y if case["want"] == "all" else y[n - 1:])

    def logits(y):
        z = y @ head.T
        cap = raw.get("logit_softcap")
        return cap * torch.tanh(z / cap) if cap else z

    first = [n if case["want"] == "all" else 1 for n in lengths]
    out = {"prompts": logits(torch.cat([y[:n] for y, n in zip(rows, first)]))}
    if case["new"]:
        out["decode"] = logits(torch.stack([y[n:] for y, n in zip(rows, first)], dim=1))
    return out
