"""What the engine is measured on: steps and generations as its users run them.

A case is one step of a batch through `ModelRunner.step`, the step function that `Engine` and the replay
program run, or one whole generation through `Engine.generate`.  Weights are random, in the shapes of real
models (see `_weight`); all inputs are made from the seed.  Fields of a case:

  model, dtype     one of `MODELS`; float32, float16 or bfloat16
  kind             "step" or "generate"
  decodes          requests that bring one token each, with `context_lo` to `context_hi` positions cached
                   (spread evenly between the two, so that lengths are ragged)
  portions         requests that bring `tokens_lo` to `tokens_hi` tokens of a prompt (spread evenly), after
                   `past` cached positions; the last token of each wants logits
  prompts, new     generate: that many prompts of `tokens_lo` to `tokens_hi` ids, `new` greedy tokens each

Designs with routed experts are not here: two correct implementations choose another expert wherever a
router's logits nearly tie, so that their outputs cannot be held to a tolerance.
"""
import math
import zlib
from types import SimpleNamespace

import numpy as np
import torch

PAGE = 16
STD = 0.02
DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}


def _llama(width, layers, heads, kv_heads, dim, ff, vocab, theta, positions, tied, eps=1e-5, scaling=None):
    return {"architectures": ["LlamaForCausalLM"], "hidden_size": width, "num_hidden_layers": layers,
            "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": dim, "intermediate_size": ff,
            "vocab_size": vocab, "rope_theta": theta, "max_position_embeddings": positions, "rms_norm_eps": eps,
            "tie_word_embeddings": tied, "rope_scaling": scaling}


def _llama3(factor, original=8192):
    return {"rope_type": "llama3", "factor": factor, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
            "original_max_position_embeddings": original}


def _latent():
    """Ruperax, 2b layer sizes: latent attention with a window in parallel gated blocks."""
    mixer = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 768, "scale": 192 ** -0.5,
             "mask": {"size": 4096}, "rot": {"base": 10000.0, "dims": 64}}
    return {"architecture": "Ruperax", "vocab": 32000, "width": 2048, "max_positions": 4096, "embedding": {"scale": 1.0},
            "norm": {"eps": 1e-6, "groups": 8},
            "layers": [{"type": "latent_attention", "mixer": dict(mixer), "mlp": {"kind": "dense", "ff": 5632}} for _ in range(4)]}


def _hybrid():
    """Vikupel, 2b layer sizes: rotary attention, Mamba-2, windowed attention with a distance penalty, Mamba-2."""
    att = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    ssm = {"type": "mamba2", "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}}
    kinds = [{"type": "attention_2", "mixer": dict(att, rot={"base": 500000.0, "dims": 128, "scaling": {
                  "factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}})},
             ssm, {"type": "attention", "mixer": dict(att, mask={"size": 1024})}, ssm]
    return {"architecture": "Vikupel", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "residual_mult": 0.7,
            "token_side": {"dim": 256}, "layers": [dict(k, mlp={"kind": "dense", "ff": 5632}) for k in kinds]}


# name -> (config.json, positions that a server of it would keep room for)
MODELS = {
    "tiny-a": (_llama(64, 2, 4, 2, 16, 172, 256, 10000.0, 128, False), 128),
    "tiny-b": (_llama(96, 3, 3, 1, 32, 256, 512, 500000.0, 256, True, 1e-6, _llama3(8.0, 64)), 256),
    "llama31-8b": (_llama(4096, 32, 32, 8, 128, 14336, 128256, 500000.0, 131072, False, scaling=_llama3(8.0)), 8448),
    "llama32-3b": (_llama(3072, 28, 24, 8, 128, 8192, 128256, 500000.0, 131072, True, scaling=_llama3(32.0)), 8448),
    "llama2-7b": (_llama(4096, 32, 32, 32, 128, 11008, 32000, 10000.0, 4096, False), 4096),
    "latent-2b": (_latent(), 4096),
    "hybrid-2b": (_hybrid(), 4096),
}


def _step(name, model, dtype, decodes=0, context=(0, 0), portions=0, tokens=(0, 0), past=0):
    return {"name": name, "model": model, "dtype": dtype, "kind": "step", "decodes": decodes, "context_lo": context[0],
            "context_hi": context[1], "portions": portions, "tokens_lo": tokens[0], "tokens_hi": tokens[1], "past": past}


def _generate(name, model, dtype, prompts, tokens, new):
    return {"name": name, "model": model, "dtype": dtype, "kind": "generate", "prompts": prompts, "tokens_lo": tokens[0],
            "tokens_hi": tokens[1], "new": new}


def listed():
    return [
        # the smallest use: a toy model in true float32, a whole greedy generation through the Python API
        _generate("generate_tiny_fp32", "tiny-a", "float32", 1, (16, 16), 16),
        # prompts of very different lengths joining in one step of a small float16 model
        _step("mixed_tiny_fp16", "tiny-b", "float16", portions=3, tokens=(1, 33)),
        # one user chatting with an 8B model
        _step("decode_8b_batch1", "llama31-8b", "bfloat16", decodes=1, context=(1031, 1031)),
        # a few users with long contexts: the benchmark's headline point
        _step("decode_8b_batch8_long", "llama31-8b", "bfloat16", decodes=8, context=(8192, 8192)),
        # a full server between 1024-token prompts and 256 generated tokens
        _step("decode_8b_batch64", "llama31-8b", "bfloat16", decodes=64, context=(1024, 1280)),
        # the largest step a runner takes by default: a 2,048-token prompt
        _step("prompt_8b_2048", "llama31-8b", "bfloat16", portions=1, tokens=(2048, 2048)),
        # an everyday prompt of odd length on a 3B model
        _step("prompt_3b_391", "llama32-3b", "bfloat16", portions=1, tokens=(391, 391)),
        # continuous batching with chunked prefill: running requests beside a portion of a long prompt
        _step("serve_7b_fp16", "llama2-7b", "float16", decodes=20, context=(128, 1000), portions=1, tokens=(492, 492), past=512),
        # the true 32-bit path: decoding and a short prompt
        _step("decode_3b_fp32", "llama32-3b", "float32", decodes=8, context=(1500, 2048)),
        _step("prompt_3b_fp32", "llama32-3b", "float32", portions=1, tokens=(300, 300)),
        # other designs: latent attention over a prompt, recurrent and windowed mixers while decoding
        _step("prompt_latent", "latent-2b", "bfloat16", portions=1, tokens=(1500, 1500)),
        _step("decode_hybrid", "hybrid-2b", "bfloat16", decodes=8, context=(900, 1400)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["generate", "tiny", "decode", "decode", "decode", "prompt", "prompt", "prompt", "serve",
                       "decode32", "prompt32", "latent", "hybrid"])
    big = rng.choice(["llama31-8b", "llama32-3b", "llama2-7b"])
    dt = "float16" if big == "llama2-7b" else "bfloat16"
    if what == "generate":
        lo = _log(rng, 1, 40)
        c = _generate("", "tiny-a", "float32", rng.randint(1, 6), (lo, lo + rng.randint(0, 24)), rng.randint(4, 40))
    elif what == "tiny":
        lo = _log(rng, 1, 40)
        c = _step("", "tiny-b", "float16", decodes=rng.randint(0, 4), context=(rng.randint(1, 90), rng.randint(90, 180)),
                  portions=rng.randint(1, 4), tokens=(lo, lo + rng.randint(0, 40)))
    elif what == "decode":
        n = _log(rng, 1, 64)
        # as many cached positions as the largest listed batch holds
        hi = min(8192 if big != "llama2-7b" else 4000, int(9.6e9 / _kv_bytes(big, dt) / n))
        hi = _log(rng, 64, hi)
        c = _step("", big, dt, decodes=n, context=(int(hi * rng.uniform(0.5, 1.0)), hi))
    elif what == "prompt":
        n = rng.choice([1, 1, 1, 2, 3])
        past = rng.choice([0, 0, _log(rng, 16, 6000 if big != "llama2-7b" else 2000)])
        hi = _log(rng, 8, (1400 if past else 2040) // n)
        c = _step("", big, dt, portions=n, tokens=(int(hi * rng.uniform(0.3, 1.0)) + 1, hi + 1), past=past)
    elif what == "serve":
        room = 9.6e9 / _kv_bytes(big, dt)
        n = _log(rng, 2, 48)
        hi = _log(rng, 100, min(3000, int(room / n)))
        t = _log(rng, 16, 900)
        c = _step("", big, dt, decodes=n, context=(int(hi * rng.uniform(0.1, 1.0)) + 1, hi), portions=1, tokens=(t, t),
                  past=rng.choice([0, 512, _log(rng, 16, 900)]))
    elif what == "decode32":
        hi = _log(rng, 64, 2048)
        c = _step("", "llama32-3b", "float32", decodes=rng.randint(1, 16), context=(int(hi * rng.uniform(0.5, 1.0)), hi))
    elif what == "prompt32":
        t = _log(rng, 4, 300)
        c = _step("", "llama32-3b", "float32", portions=1, tokens=(t, t), past=rng.choice([0, 256]))
    else:
        model = what + "-2b"
        if rng.random() < 0.5:
            t = _log(rng, 8, 2048)
            c = _step("", model, "bfloat16", portions=1, tokens=(t, t))
        else:
            hi = _log(rng, 32, 1500)
            c = _step("", model, "bfloat16", decodes=rng.randint(1, 10), context=(int(hi * rng.uniform(0.5, 1.0)), hi))
    c.pop("name")
    return c


# ---------------------------------------------------------------------------------- what a case consists of
def _kv_bytes(model, dtype):
    """Bytes of keys and values per cached position of a Llama."""
    c = MODELS[model][0]
    return 2 * c["num_hidden_layers"] * c["num_key_value_heads"] * c["head_dim"] * (4 if dtype == "float32" else 2)


def _spread(n, lo, hi):
    """n whole numbers from lo to hi, evenly spread, in an order that mixes long and short."""
    v = [lo + (hi - lo) * i // max(1, n - 1) for i in range(n)]
    return v[::2] + v[1::2][::-1]


def _requests(case):
    """(cached positions, new tokens) of every request of a step."""
    return ([(p, 1) for p in _spread(case["decodes"], case["context_lo"], case["context_hi"])] +
            [(case["past"], n) for n in _spread(case["portions"], case["tokens_lo"], case["tokens_hi"])])


def _generator(seed, what):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + zlib.crc32(what.encode())) % (1 << 62))


def _tokens(seed, what, n, vocab):
    return torch.randint(0, vocab, (n,), generator=_generator(seed, "tokens " + what), device="cuda")


def _weight(seed, name, shape, kind, dtype, layers):
    """Matrices N(0, 0.02) in the compute dtype, vectors in float32 drawn as a fresh model of the design starts (norms
    about 1, shifts and slopes in [0, 1], a state's rates as usual).  As in a trained model a sublayer changes the
    residual rows a little: the embedding is N(0, 1) and the matrices that write into the rows are smaller by
    sqrt(2 layers).  (With 0.02 everywhere the rows are made of the sublayers' results alone, and what rounds to 16
    bits in one layer grows through the next ones to several percent of the logits.)"""
    g = _generator(seed, name)
    shape = tuple(shape)
    if kind == "matrix":
        std = 1.0 if name.startswith(("token_embd", "position")) else STD
        if name.endswith(("attn_output.weight", "mix.output.weight", "mix.o.weight", "down.weight")):
            std /= math.sqrt(2 * layers)
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)
    u = torch.rand(shape, generator=g, device="cuda")
    if name.endswith("A_log"):
        return torch.log(1.0 + 15.0 * u)
    if name.endswith("dt_bias"):
        dt = torch.exp(u * math.log(100.0) + math.log(0.001))
        return dt + torch.log(-torch.expm1(-dt))
    if name.endswith(("shift.weight", ".r1", ".r2")):
        return u
    r = STD * torch.randn(shape, generator=g, device="cuda")
    return 1.0 + r if name.endswith(("norm.weight", "norm1.weight", "norm2.weight", ".D")) else r


def _old_cache(seed, model, dtype, pages):
    """Keys and values that earlier steps of a Llama left: [layers, pages, 2, KV heads, PAGE, head size], spread as
    the products of normed rows with N(0, 0.02) matrices are."""
    c = MODELS[model][0]
    shape = (c["num_hidden_layers"], pages, 2, c["num_key_value_heads"], PAGE, c["head_dim"])
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, STD * math.sqrt(c["hidden_size"]), generator=_generator(seed, "cache"))


def _is_llama(model):
    return "architectures" in MODELS[model][0]


def _vocab(model):
    c = MODELS[model][0]
    return c["vocab_size"] if _is_llama(model) else c["vocab"]


def _layers(model):
    c = MODELS[model][0]
    return c["num_hidden_layers"] if _is_llama(model) else len(c["layers"])


def _pages(reqs):
    return sum(-(-(p + n) // PAGE) for p, n in reqs)


def prepare(case, seed):
    from ferrum_b200.cache import CacheStorage
    from ferrum_b200.config import registry
    from ferrum_b200.engine import ModelRunner, StepEntry
    from ferrum_b200.engine.api import Engine

    config, room = MODELS[case["model"]]
    dtype, vocab = DTYPES[case["dtype"]], _vocab(case["model"])
    arch = registry.lookup(registry.architecture_name(config))
    model = arch.build(arch.read_config(config), dtype, "cuda", max_positions=room)
    for name, (spec, part, local) in model.weight_specs().items():
        if not (spec.optional and config.get("tie_word_embeddings")):
            part.assign(local, _weight(seed, name, spec.shape, spec.kind, dtype, _layers(case["model"])))
    model.finalize()
    if case["kind"] == "generate":
        lengths = _spread(case["prompts"], case["tokens_lo"], case["tokens_hi"])
        engine = Engine(model=model, page_size=PAGE, num_pages=8 * room // PAGE, max_batch_seqs=8, max_model_len=room)
        return SimpleNamespace(engine=engine, new=case["new"],
                               prompts=[_tokens(seed, str(i), n, vocab).tolist() for i, n in enumerate(lengths)])
    reqs = _requests(case)
    llama = _is_llama(case["model"])
    pages = _pages(reqs) if llama else _pages([(p + PAGE, n + PAGE) for p, n in reqs])
    cache = CacheStorage(model, dtype, "cuda", page_size=PAGE, num_pages=pages, max_requests=max(8, len(reqs)), max_model_len=room)
    runner = ModelRunner(model, cache, max_batch_tokens=2048, max_batch_requests=max(8, len(reqs)))
    for pool in cache.pools:
        pool.zero_()
    if llama:
        cache.pools[0].copy_(_old_cache(seed, case["model"], dtype, pages))
    entries = []
    for i, (past, n) in enumerate(reqs):
        slot = cache.open()
        ids = _tokens(seed, str(i), past + n, vocab).tolist()
        if llama:
            cache.manager.grow(slot, past + n)
            cache.manager.commit(slot, past)
        elif past:           # caches that hold more than keys and values come from running what came before
            runner.step([StepEntry(slot, 0, ids[:past], [])])
        entries.append(StepEntry(slot, past, ids[past:], [n - 1]))
    return SimpleNamespace(engine=None, runner=runner, cache=cache, entries=entries)


def run(state):
    if state.engine is not None:
        return np.array(state.engine.generate(state.prompts, max_new_tokens=state.new), dtype=np.int64)
    # The lengths are not advanced, so that the same step can be run again.
    logits = state.runner.step(state.entries, commit=False, check=False)
    return {"logits": logits, "cache": state.cache.pools, "state": state.cache.states}


# ---------------------------------------------------------------------------------- bytes and operations
def _matrices(model):
    """Elements of the matrices that every token passes, and of the output matrix."""
    c = MODELS[model][0]
    if _is_llama(model):
        e, q, kv = c["hidden_size"], c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
        return c["num_hidden_layers"] * (2 * e * q + 2 * e * kv + 3 * e * c["intermediate_size"]), e * c["vocab_size"]
    e, total = c["width"], 0
    for layer in c["layers"]:
        m = layer["mixer"]
        total += 3 * e * layer["mlp"]["ff"]
        if layer["type"] == "latent_attention":
            h = m["heads"]
            total += (2 * e * e + e * m["q_rank"] + m["q_rank"] * h * (m["dim"] + m["rot_dim"]) + e * (m["kv_rank"] + m["rot_dim"]) +
                      m["kv_rank"] * h * (m["dim"] + m["vdim"]) + e * h + e * h * m["vdim"])
        elif layer["type"] == "mamba2":
            inner = m["heads"] * m["vdim"]
            total += e * (2 * inner + 2 * m["groups"] * m["state"] + m["heads"]) + e * inner
        else:
            total += e * (m["heads"] + m["kv_heads"]) * (m["dim"] + m["vdim"])
            total += e * m["heads"] * m["vdim"] if layer["type"] == "attention" else 0
        total += 2 * e * c["token_side"]["dim"] if "token_side" in c else 0
    return total, e * c["vocab"]


def _mixing(model, past, n):
    """(cached elements read, elements written to the cache, multiplications) of a request's new tokens beside the matrices."""
    c = MODELS[model][0]
    pairs = n * past + n * (n + 1) // 2              # (token, key) pairs of full causal attention
    if _is_llama(model):
        row = 2 * c["num_key_value_heads"] * c["head_dim"] * c["num_hidden_layers"]
        return row * past, row * n, 2 * c["num_attention_heads"] * c["head_dim"] * c["num_hidden_layers"] * pairs
    read = written = mults = 0
    for layer in c["layers"]:
        m = layer["mixer"]
        if layer["type"] == "mamba2":
            memory = m["heads"] * m["vdim"] * m["state"]
            read, written, mults = read + 2 * memory, written + 2 * memory, mults + 3 * memory * n     # (float32: twice two bytes)
            continue
        window = m["mask"]["size"] if "mask" in m else past + n
        seen = sum(min(window, past + i + 1) for i in range(n))
        row = m["kv_rank"] + m["rot_dim"] if "kv_rank" in m else m["kv_heads"] * (m["dim"] + m["vdim"])
        per = m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"])
        read, written, mults = read + row * min(past, window), written + row * n, mults + per * seen
    return read, written, mults


def work(case):
    body, head = _matrices(case["model"])
    size, vocab = (4 if case["dtype"] == "float32" else 2), _vocab(case["model"])
    e = head // vocab

    def step(reqs):
        parts = [_mixing(case["model"], p, n) for p, n in reqs]
        tokens, wanted = sum(n for _, n in reqs), len(reqs)
        nbytes = size * (body + head + tokens * e + sum(p[0] + p[1] for p in parts)) + 4 * wanted * vocab
        return nbytes, 2 * (body * tokens + head * wanted + sum(p[2] for p in parts))

    if case["kind"] == "step":
        nbytes, flops = step(_requests(case))
        return {"bytes": nbytes, "flops": flops}
    lengths = _spread(case["prompts"], case["tokens_lo"], case["tokens_hi"])
    steps = [step([(0, n) for n in lengths])] + [step([(n + i, 1) for n in lengths]) for i in range(case["new"] - 1)]
    return {"bytes": sum(s[0] for s in steps), "flops": sum(s[1] for s in steps)}


def tolerance(case):
    # Four times the largest error of logits against `exact`: 5.3e-3, 6.1e-4 and 2.2e-6.
    if case["kind"] == "generate":
        return "exact"           # greedy ids of float32 logits
    return {"bfloat16": {"rel": 0.02, "max": 0.15}, "float16": {"rel": 0.0025, "max": 0.02},
            "float32": {"rel": 1e-5, "max": 8e-5}}[case["dtype"]]


# ---------------------------------------------------------------------------------- the same in 64 bits
def _rms(v, eps):
    return v * torch.rsqrt((v * v).mean(-1, keepdim=True) + eps)


def _silu(v):
    return v * torch.sigmoid(v)


def _frequencies(base, dims, scaling=None):
    """Rotary frequencies; scaling: (factor, low, high, original) of the llama3 rule."""
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device="cuda") / dims)
    if scaling is None:
        return f
    factor, low, high, original = scaling
    wave = 2 * math.pi / f
    s = ((original / wave - low) / (high - low)).clamp(0, 1)
    return (1 - s) * f / factor + s * f


def _rotate(v, pos, f, sign=1.0):
    """v [T, heads, D]: elements i and i + len(f) turn by pos * f[i]; the rest stays."""
    half = f.numel()
    a = sign * pos.double()[:, None, None] * f
    x, y = v[..., :half], v[..., half:2 * half]
    return torch.cat([x * a.cos() - y * a.sin(), y * a.cos() + x * a.sin(), v[..., 2 * half:]], -1)


def _attend(q, k, v, pos, scale, window=0, bias=None):
    """q [T, H, D] at positions pos over k, v [S, G, D] at positions 0..S-1; bias(distance) [H, T, S] is subtracted."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64, device="cuda")
    far = pos[:, None] - torch.arange(k.shape[0], device="cuda")[None]
    hidden = (far < 0) | (far >= window) if window else far < 0
    for g in range(G):
        h = slice(g * H // G, (g + 1) * H // G)
        s = torch.einsum("thd,sd->hts", q[:, h], k[:, g]) * scale
        if bias is not None:
            s -= bias(far.clamp(min=0).double())[h]
        out[:, h] = torch.einsum("hts,sd->thd", s.masked_fill_(hidden, -math.inf).softmax(-1), v[:, g])
    return out


class _Weights:
    def __init__(self, case, seed):
        self.seed, self.dtype, self.layers = seed, DTYPES[case["dtype"]], _layers(case["model"])

    def matrix(self, name, *shape):
        return _weight(self.seed, name, shape, "matrix", self.dtype, self.layers).double()

    def vector(self, name, *shape):
        return _weight(self.seed, name, shape, "vector", torch.float32, self.layers).double()


def _exact_llama(c, w, reqs, ids, cache, last_only=True):
    """Logits of the wanted rows.  cache: float64 pages of the old positions, or None; receives the new keys and values."""
    e, H, G, D, L = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["num_hidden_layers"]
    eps, ff, sc = c["rms_norm_eps"], c["intermediate_size"], c["rope_scaling"]
    f = _frequencies(c["rope_theta"], D, sc and (sc["factor"], sc["low_freq_factor"], sc["high_freq_factor"],
                                                 sc["original_max_position_embeddings"]))
    pos = torch.cat([torch.arange(p, p + n, device="cuda") for p, n in reqs])
    table = w.matrix("token_embd.weight", c["vocab_size"], e)
    x = table[torch.cat(ids)]
    for i in range(L):
        b = f"blk.{i}."
        h = _rms(x, eps) * w.vector(b + "attn_norm.weight", e)
        q = _rotate((h @ w.matrix(b + "attn_q.weight", H * D, e).T).view(-1, H, D), pos, f)
        k = _rotate((h @ w.matrix(b + "attn_k.weight", G * D, e).T).view(-1, G, D), pos, f)
        v = (h @ w.matrix(b + "attn_v.weight", G * D, e).T).view(-1, G, D)
        parts, t, page = [], 0, 0
        for p, n in reqs:
            m = -(-(p + n) // PAGE)
            kk, vv = k[t:t + n], v[t:t + n]
            if p:
                old = cache(i, page, page + m).double().permute(1, 0, 3, 2, 4).reshape(2, m * PAGE, G, D)[:, :p]
                kk, vv = torch.cat([old[0], kk]), torch.cat([old[1], vv])
            parts.append(_attend(q[t:t + n], kk, vv, pos[t:t + n], D ** -0.5))
            t, page = t + n, page + m
        x = x + torch.cat(parts).view(-1, H * D) @ w.matrix(b + "attn_output.weight", e, H * D).T
        h = _rms(x, eps) * w.vector(b + "ffn_norm.weight", e)
        h = _silu(h @ w.matrix(b + "ffn_gate.weight", ff, e).T) * (h @ w.matrix(b + "ffn_up.weight", ff, e).T)
        x = x + h @ w.matrix(b + "ffn_down.weight", e, ff).T
    last = torch.tensor([n for _, n in reqs], device="cuda").cumsum(0) - 1
    x = _rms(x[last], eps) * w.vector("output_norm.weight", e)
    return x @ (table if c["tie_word_embeddings"] else w.matrix("output.weight", c["vocab_size"], e)).T


def _exact_latent(c, w, ids):
    """Logits of a whole sequence's last token."""
    e, eps, groups = c["width"], c["norm"]["eps"], c["norm"]["groups"]
    T = ids.numel()
    pos = torch.arange(T, device="cuda")

    def norm(x):
        return _rms(x.view(T, groups, -1), eps).reshape(T, e)

    def gate(x, name):
        return torch.sigmoid(x @ w.matrix(name + ".weight", e, e).T + w.vector(name + ".bias", e))

    x = w.matrix("token_embd.weight", c["vocab"], e)[ids] + w.matrix("position.weight", c["max_positions"], e)[pos]
    for i, layer in enumerate(c["layers"]):
        m, ff, b = layer["mixer"], layer["mlp"]["ff"], f"blk.{i}."
        H, Dn, Rr, Dv, R, Rq = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
        f = _frequencies(m["rot"]["base"], m["rot"]["dims"])
        n = norm(x)
        a = n * w.vector(b + "norm1.weight", e)
        before = torch.cat([torch.zeros_like(a[:1]), a[:-1]])
        h = a + (before - a) * w.vector(b + "shift.weight", e)
        d = h @ w.matrix(b + "mix.dkv.weight", R + Rr, e).T
        latent = _rms(d[:, :R], eps) * w.vector(b + "mix.dkv_norm.weight", R)
        kr = _rotate(d[:, None, R:], pos, f).expand(T, H, Rr)
        cq = _rms(h @ w.matrix(b + "mix.dq.weight", Rq, e).T, eps) * w.vector(b + "mix.dq_norm.weight", Rq)
        q = (cq @ w.matrix(b + "mix.uq.weight", H * (Dn + Rr), Rq).T).view(T, H, Dn + Rr)
        q = torch.cat([q[..., :Dn], _rotate(q[..., Dn:], pos, f)], -1)
        k = torch.cat([(latent @ w.matrix(b + "mix.uk.weight", H * Dn, R).T).view(T, H, Dn), kr], -1)
        v = (latent @ w.matrix(b + "mix.uv.weight", H * Dv, R).T).view(T, H, Dv)
        o = _attend(q, k, v, pos, m["scale"], m["mask"]["size"]) * torch.sigmoid(h @ w.matrix(b + "mix.g.weight", H, e).T)[..., None]
        y = (o.view(T, H * Dv) @ w.matrix(b + "mix.o.weight", e, H * Dv).T) * gate(a, b + "rg1")
        z = n * w.vector(b + "norm2.weight", e)
        u = (_silu(z @ w.matrix(b + "mlp.gate.weight", ff, e).T + w.vector(b + "mlp.gate.bias", ff)) *
             (z @ w.matrix(b + "mlp.up.weight", ff, e).T + w.vector(b + "mlp.up.bias", ff)))
        x = x + y + (u @ w.matrix(b + "mlp.down.weight", e, ff).T + w.vector(b + "mlp.down.bias", e)) * gate(z, b + "rg2")
    x = norm(x)[-1:] * w.vector("output_norm.weight", e)
    return x @ w.matrix("output.weight", c["vocab"], e).T


def _exact_mamba2(h, w, b, m, eps):
    T, e = h.shape
    H, P, N, taps = m["heads"], m["vdim"], m["state"], m["conv"]
    inner = H * P                                   # (one group shares B and C)
    proj = h @ w.matrix(b + "in.weight", 2 * inner + 2 * N + H, e).T
    z, u, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * N], proj[:, 2 * inner + 2 * N:]
    kernel, padded = w.vector(b + "conv.weight", inner + 2 * N, taps), torch.cat([torch.zeros_like(u[:taps - 1]), u])
    u = _silu(sum(padded[j:j + T] * kernel[:, j] for j in range(taps)) + w.vector(b + "conv.bias", inner + 2 * N))
    x, B, C = u[:, :inner].view(T, H, P), u[:, inner:inner + N], u[:, inner + N:]
    dt = torch.nn.functional.softplus(dt + w.vector(b + "dt_bias", H), threshold=1000)
    keep = torch.exp(-torch.exp(w.vector(b + "A_log", H)) * dt)[:, :, None, None]
    dx, S, y = dt[..., None] * x, torch.zeros(H, P, N, dtype=torch.float64, device="cuda"), torch.empty_like(x)
    for t in range(T):
        S = S * keep[t] + dx[t, :, :, None] * B[t]
        y[t] = S @ C[t]
    y = (y + w.vector(b + "D", H)[:, None] * x).reshape(T, inner) * _silu(z)
    y = _rms(y.view(T, m["norm_groups"], -1), eps).reshape(T, inner) * w.vector(b + "norm.weight", inner)
    return y @ w.matrix(b + "o.weight", e, inner).T


def _exact_hybrid(c, w, ids):
    """Logits of a whole sequence's last token."""
    e, eps, mult, side = c["width"], c["norm"]["eps"], c["residual_mult"], c["token_side"]["dim"]
    T, L = ids.numel(), len(c["layers"])
    pos = torch.arange(T, device="cuda")
    x = w.matrix("token_embd.weight", c["vocab"], e)[ids]
    extra = w.matrix("side_embd.weight", c["vocab"], L * side)[ids].view(T, L, side)
    for i, layer in enumerate(c["layers"]):
        m, ff, b = layer["mixer"], layer["mlp"]["ff"], f"blk.{i}."
        h = _rms(x, eps) * w.vector(b + "norm1.weight", e)
        if layer["type"] == "mamba2":
            y = _exact_mamba2(h, w, b + "mix.", m, eps)
        else:
            H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            q = (h @ w.matrix(b + "mix.q.weight", H * D, e).T).view(T, H, D)
            k = (h @ w.matrix(b + "mix.k.weight", G * D, e).T).view(T, G, D)
            v = (h @ w.matrix(b + "mix.v.weight", G * Dv, e).T).view(T, G, Dv)
            if layer["type"] == "attention_2":
                sc, base = m["rot"]["scaling"], m["rot"]["base"]
                f, fv = _frequencies(base, m["rot"]["dims"], (sc["factor"], sc["low"], sc["high"], sc["original"])), _frequencies(base, Dv)
                q, k, v = _rms(_rotate(q, pos, f), eps), _rms(_rotate(k, pos, f), eps), _rotate(v, pos, fv)
                o = _rotate(_attend(q, k, v, pos, m["scale"]), pos, fv, -1.0).reshape(T, H * Dv)
            else:
                r1, r2 = w.vector(b + "mix.r1", H)[:, None, None], w.vector(b + "mix.r2", H)[:, None, None]
                o = _attend(q, k, v, pos, m["scale"], m["mask"]["size"], lambda far: r1 * torch.log1p(r2 * far))
                o = o.reshape(T, H * Dv) * torch.sigmoid(h @ w.matrix(b + "mix.g.weight", H * Dv, e).T)
            y = o @ w.matrix(b + "mix.output.weight", e, H * Dv).T
        u = _silu(h @ w.matrix(b + "mlp.gate.weight", ff, e).T) * (h @ w.matrix(b + "mlp.up.weight", ff, e).T)
        x = x + mult * (y + u @ w.matrix(b + "mlp.down.weight", e, ff).T)
        g = torch.nn.functional.gelu(x @ w.matrix(b + "side.gate.weight", side, e).T, approximate="tanh") * extra[:, i]
        x = x + mult * _rms(g @ w.matrix(b + "side.proj.weight", e, side).T, eps) * w.vector(b + "side.norm.weight", e)
    x = _rms(x[-1:], eps) * w.vector("output_norm.weight", e)
    return x @ w.matrix("output.weight", c["vocab"], e).T


def exact(case, seed):
    """The logits (for a generation its ids).  Caches and states have no value here: their layout is the engine's own,
    and what a step writes there is read again by its own attention."""
    c, w, vocab = MODELS[case["model"]][0], _Weights(case, seed), _vocab(case["model"])
    if case["kind"] == "generate":
        out = []
        for i, n in enumerate(_spread(case["prompts"], case["tokens_lo"], case["tokens_hi"])):
            ids = _tokens(seed, str(i), n, vocab)
            for _ in range(case["new"]):
                ids = torch.cat([ids, _exact_llama(c, w, [(0, ids.numel())], [ids], None)[-1].argmax()[None]])
            out.append(ids[n:])
        return torch.stack(out)
    reqs = _requests(case)
    ids = [_tokens(seed, str(i), p + n, vocab) for i, (p, n) in enumerate(reqs)]
    if _is_llama(case["model"]):
        old = _old_cache(seed, case["model"], DTYPES[case["dtype"]], _pages(reqs))
        logits = _exact_llama(c, w, reqs, [t[p:] for t, (p, _) in zip(ids, reqs)], lambda i, a, b: old[i, a:b])
    else:
        logits = torch.cat([(_exact_latent if "Ruperax" in c["architecture"] else _exact_hybrid)(c, w, t) for t in ids])
    return {"logits": logits, "cache": None, "state": None}
