"""Latent attention with its keys and values written out (attention_rows) against the same in float64, over portions, windows,
sinks and batches, beside the path on the cached rows."""
import pytest
import torch

F64 = torch.float64


def test_rows_plan():
    """Every key a query of the step sees has a row, rows of a request begin on a border of 64 keys, items cover the tokens."""
    from ferrum_b200.parts import attention_plan
    from ferrum_b200.parts.latent_attention import rows_plan
    for q_len, pos0, window in (([300, 1, 700], [0, 900, 65], 0), ([300, 1, 700], [0, 900, 65], 100), ([1, 513], [63, 64], 64), ([256], [4000], 129)):
        start, first = rows_plan(q_len, pos0, window)
        assert start[0] == 0 and all(f % 64 == 0 for f in first)
        items = attention_plan.whole_items(q_len, pos0, window, 256)
        rows = {r: set() for r in range(len(q_len))}
        for r, row0, lo, hi, splits, slot, _, _ in items.tolist():
            assert splits == 1 and slot == -1 and row0 % 256 == 0
            last = min(row0 + 256, q_len[r])
            rows[r] |= set(range(row0, last))
            assert hi == pos0[r] + last and lo == (max(0, pos0[r] + row0 - window + 1) if window else 0)
            assert first[r] <= lo // 64 * 64 and start[r] + hi - first[r] <= start[r + 1]
        assert all(rows[r] == set(range(n)) for r, n in enumerate(q_len))
        assert [h - l for _, _, l, h, *_ in items.tolist()] == sorted((h - l for _, _, l, h, *_ in items.tolist()), reverse=True)


class Mixers:
    """A mixer that caches its rows and, if there is a second, a reader of them."""

    def __init__(self, mixers):
        from ferrum_b200.models import Run
        self.mixers, self.schedule = mixers, [Run(0)] + [Run(k, cache_of=0) for k in range(1, len(mixers))]

    def cache_needs(self):
        return [m.cache_need() for m in self.mixers]


def exact(w, writer, x, H, R, scale, window, rot, sink, eps):
    """float64, one sequence from position 0; the latent and the shared key part by the weights of `writer`."""
    T = x.shape[0]
    rms = lambda v: v * torch.rsqrt((v * v).mean(-1, keepdim=True) + eps)
    pos = torch.arange(T, device="cuda")

    def turn(v):          # [T, n, 64]: the table's leading dimensions turn, paired as it says
        if rot is None:
            return v
        n = rot.rope_dim
        a = rot.cos_sin[:T].double()
        c, s = a[:, None, :, 0], a[:, None, :, 1]
        head = v[..., :n]
        p, q = (head[..., :n // 2], head[..., n // 2:]) if rot.pairing else (head[..., ::2], head[..., 1::2])
        p, q = p * c - q * s, q * c + p * s
        head = torch.cat([p, q], -1) if rot.pairing else torch.stack([p, q], -1).flatten(-2)
        return torch.cat([head, v[..., n:]], -1)
    d = x @ writer["dkv.weight"].T
    c = rms(d[:, :R]) * writer["dkv_norm.weight"]
    kr = turn(d[:, None, R:]).expand(T, H, 64)
    q = ((rms(x @ w["dq.weight"].T) * w["dq_norm.weight"]) @ w["uq.weight"].T).view(T, H, 192)
    q = torch.cat([q[..., :128], turn(q[..., 128:])], -1)
    k = torch.cat([(c @ w["uk.weight"].T).view(T, H, 128), kr], -1)
    v = (c @ w["uv.weight"].T).view(T, H, 128)
    far = pos[:, None] - pos[None]
    s = torch.einsum("thd,shd->hts", q, k) * scale
    s = s.masked_fill((far < 0) | ((far >= window) if window else False), -torch.inf)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(H, T, 1)], -1)
    p = s.softmax(-1)[..., :T]
    o = torch.einsum("hts,shd->thd", p, v) * torch.sigmoid(x @ w["g.weight"].T)[..., None]
    return o.reshape(T, H * 128) @ w["o.weight"].T


# The plain case, sinks, windows and ranks; then scales that are not positive (which turn or level the scores), the other
# pairing, a table of half of the shared part, none, and a layer that reads the rows another one cached, which has a window of its own.
CASES = {"plain": dict(H=2, R=512), "sink-wide": dict(H=5, R=72, sink=True, wide=True), "window": dict(H=3, R=128, window=100),
         "window-sink": dict(H=1, R=64, window=300, sink=True),
         "negative": dict(H=2, R=512, scale=-0.07), "negative-window-sink-wide": dict(H=2, R=64, scale=-0.07, window=100, sink=True, wide=True),
         "zero": dict(H=2, R=64, scale=0.0, sink=True), "adjacent": dict(H=2, R=128, rot=(64, "adjacent")),
         "half-turned": dict(H=2, R=128, rot=(32, "half")), "half-turned-adjacent": dict(H=3, R=64, rot=(32, "adjacent")),
         "unturned": dict(H=2, R=128, rot=None), "reader": dict(H=2, R=128, reader=True), "reader-window": dict(H=3, R=64, reader=True, window=200)}


@pytest.mark.gpu
@pytest.mark.parametrize("td", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", list(CASES))
def test_latent_rows(td, case, monkeypatch):
    from ferrum_b200.cache import CacheStorage
    from ferrum_b200.engine.batch import StepContext, StepEntry
    from ferrum_b200.ops import lib as ops
    from ferrum_b200.parts import LatentAttention, RotaryEmbedding, latent_attention
    ops.require_cuda()
    spec = dict(window=0, sink=False, wide=False, scale=192 ** -0.5, rot=(64, "half"), reader=False)
    spec.update(CASES[case])
    H, R, window, sink, scale = (spec[k] for k in ("H", "R", "window", "sink", "scale"))
    E, Rq, eps = 256, 96, 1e-5
    rot = RotaryEmbedding(64, spec["rot"][0], 10000.0, None, spec["rot"][1], 1024, "cuda") if spec["rot"] else None
    g = torch.Generator(device="cuda").manual_seed(H + R)
    mixers, ws = [], []
    for k in range(1 + spec["reader"]):
        mixer = LatentAttention(E, H, 128, 64, 128, R, Rq, eps, scale, td, rotary=rot, own_latent=k == 0, sink=sink, wide_weights=spec["wide"],
                                window=window if k == spec["reader"] else 0)
        w = {}
        for name, p in mixer.param_specs().items():
            t = torch.randn(p.shape, device="cuda", generator=g)
            t = t * p.shape[-1] ** -0.5 if p.kind == "matrix" else (1.0 + 0.1 * t if "norm" in name else t)
            t = t.to(td) if p.kind == "matrix" else t
            mixer.assign(name, t.contiguous())
            w[name] = t.double()
        mixer.finalize()
        mixers.append(mixer)
        ws.append(w)
    cache = CacheStorage(Mixers(mixers), td, "cuda", page_size=16, max_tokens=4096, max_requests=4, max_model_len=1024)
    ctx = StepContext("cuda", 1024, 4, [cache.table_width])
    xs = [torch.randn(n, E, device="cuda", generator=g).to(td) for n in (700, 257, 300)]
    refs = [exact(ws[-1], ws[0], x.double(), H, R, scale, window, rot, ws[-1].get("sink"), eps) for x in xs]
    calls = []
    real = ops.attention_rows
    monkeypatch.setattr(ops, "attention_rows", lambda *a, **k: (calls.append(1), real(*a, **k))[1])
    # per step, the tokens of every request: whole prompts, portions on what was cached (odd borders), a batch with single tokens
    error = {}
    for limit in (8, 1 << 30):
        monkeypatch.setattr(latent_attention, "EXPAND_MIN_QUERIES", limit)
        before = len(calls)
        for steps in ([[700, 0, 0], [0, 257, 300]], [[129, 1, 0], [571, 256, 1], [0, 0, 299]]):
            slots, at, got = [cache.open() for _ in xs], [0, 0, 0], [[], [], []]
            for step in steps:
                rows = [(r, n) for r, n in enumerate(step) if n]
                for r, n in rows:
                    cache.manager.grow(slots[r], at[r] + n)
                ctx.fill([StepEntry(slots[r], at[r], [0] * n) for r, n in rows], cache.manager)
                x = torch.cat([xs[r][at[r]:at[r] + n] for r, n in rows])
                for k, mixer in enumerate(mixers):
                    y = torch.full((x.shape[0], E), float("nan"), device="cuda")
                    mixer.forward(x, ctx, cache.layer_cache(k), y, accumulate=False)
                assert ctx.err.item() == 0
                t = 0
                for r, n in rows:
                    got[r].append(y[t:t + n].double())
                    t += n
                    cache.manager.commit(slots[r], at[r] + n)
                    at[r] += n
            for s in slots:
                cache.close(s)
            for r, ref in enumerate(refs):
                out = torch.cat(got[r])
                # 16-bit roundings of the latent, the queries, keys, values, weights and heads: some six, of 2^-9 (2^-12) each
                assert (out - ref).abs().max() < (4e-2 if td == torch.bfloat16 else 5e-3) * ref.abs().max(), (limit, steps, r)
                error.setdefault(limit, []).append(((out - ref).norm() / ref.norm()).item())
        assert (len(calls) > before) == (limit == 8)
    assert sum(error[8]) <= 1.1 * sum(error[1 << 30])          # no less precise than on the cached rows


@pytest.mark.gpu
def test_portions_leave_captured_steps_alone(monkeypatch):
    """The keys that are written out grow with every portion of a prompt; no buffer that a captured step reads moves with them.
    And where the scratch of the keys would be too much, attention runs on the cached rows."""
    from ferrum_b200.cache import CacheStorage
    from ferrum_b200.engine.batch import StepContext, StepEntry
    from ferrum_b200.ops import lib as ops
    from ferrum_b200.parts import LatentAttention, latent_attention
    ops.require_cuda()
    td, E, H, R = torch.bfloat16, 256, 2, 64
    mixer = LatentAttention(E, H, 128, 64, 128, R, 96, 1e-5, 192 ** -0.5, td)
    g = torch.Generator(device="cuda").manual_seed(1)
    for name, p in mixer.param_specs().items():
        mixer.assign(name, torch.randn(p.shape, device="cuda", generator=g).mul_(p.shape[-1] ** -0.5).to(td if p.kind == "matrix" else torch.float32))
    mixer.finalize()
    cache = CacheStorage(Mixers([mixer]), td, "cuda", page_size=16, max_tokens=4096, max_requests=4, max_model_len=4096)
    calls = []
    real = ops.attention_rows
    monkeypatch.setattr(ops, "attention_rows", lambda *a, **k: (calls.append(a[4]), real(*a, **k))[1])

    def prompt(ctx):
        slot, seen = cache.open(), []
        x, y = torch.randn(256, E, device="cuda", generator=g).to(td), torch.empty(256, E, device="cuda")
        for at in range(0, 2048, 256):
            cache.manager.grow(slot, at + 256)
            ctx.fill([StepEntry(slot, at, [0] * 256)], cache.manager)
            mixer.forward(x, ctx, cache.layer_cache(0), y, accumulate=False)
            cache.manager.commit(slot, at + 256)
            seen.append(ctx.buffers_generation())
        assert ctx.err.item() == 0
        cache.close(slot)
        return seen
    monkeypatch.setattr(latent_attention, "EXPAND_MIN_QUERIES", 64)
    seen = prompt(StepContext("cuda", 256, 4, [cache.table_width]))
    assert calls == list(range(256, 2049, 256)) and len(set(seen)) == 1
    calls.clear()
    monkeypatch.setattr(latent_attention, "EXPAND_MAX_BYTES", 1100 * 2 * (R + 64 + H * 256))
    prompt(StepContext("cuda", 256, 4, [cache.table_width]))
    assert calls == [256, 512, 768, 1024]
