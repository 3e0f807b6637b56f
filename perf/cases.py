"""What a user of the engine has it do, as cases that can be timed and checked.

A pass of most cases is one step of a running engine: every request of the batch brings one token (decode), a
prompt or a piece of one (prefill), or both kinds ride together (continuous batching), on top of the keys and values that
are cached already.  The step is then taken back (`CacheManager.commit` by minus the tokens it brought), so that
the next pass does the same work at the same positions.  Models that keep a recurrent state per request cannot take a
step back: there a pass is a whole turn, from the prompts through some decoded tokens to the release of the requests.

Weights are the engine's random ones (N(0, 0.02), seeded), token ids are uniform, cached keys and values are normal with
the deviations that the random projections give.  Model shapes are those of `bench.py`, at twelve layers (its `--layers`):
what bfloat16 rounding does to random weights grows with the root of the depth, and at the full 36 layers two right
implementations differ by 0.026 to 0.032 of the logits, too much to tell a mistake from rounding; at twelve by 0.012 to 0.018
(a batch's rows through other kernels, a prompt in two pieces).  The logits are compared and not the sampled ids: with random
weights the two largest logits of a row often lie closer together than bfloat16 rounding moves them.
"""
import hashlib
import math
import random

import torch

from velox_b200 import Engine, EngineConfig
from velox_b200.config import BirelixConfig, KapuvikConfig, Qwen3Config
from velox_b200.engine import StepEntry

PAGE = 16
DEVICE = "cuda:0"

# ---- models -------------------------------------------------------------------------------------------

LAYERS = 12
QWEN3 = dict(vocab_size=151936, hidden_size=4096, intermediate_size=12288, num_hidden_layers=LAYERS, num_attention_heads=32, head_dim=128,
             attention_bias=False, num_key_value_heads=8, max_position_embeddings=40960, tie_word_embeddings=False,
             rope_theta=1000000.0, rms_norm_eps=1e-6, hidden_act="silu")
QWEN3_SHAPES = {
    "qwen3-0.6b": dict(hidden_size=1024, intermediate_size=3072, num_attention_heads=16, tie_word_embeddings=True),
    "qwen3-1.7b": dict(hidden_size=2048, intermediate_size=6144, num_attention_heads=16, tie_word_embeddings=True),
    "qwen3-4b": dict(hidden_size=2560, intermediate_size=9728, num_attention_heads=32, tie_word_embeddings=True),
    "qwen3-8b": dict(),
}
TURN_SIZES = {
    "1k": dict(width=1024, heads=8, kv_heads=2, lin_heads=8, expert_ff=512, shared_ff=512),
    "2k": dict(width=2048, heads=16, kv_heads=4, lin_heads=16, expert_ff=1024, shared_ff=1024),
}
VOCAB, EXPERTS, TOP = 32000, 8, 2
LATENT, ROT = dict(rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5), 64


def _kapuvik(sz):
    """Latent attention, two layers of linear attention with a decay per channel, softmax attention beside retention."""
    H, HL = sz["heads"], sz["lin_heads"]
    ff = dict(kind="dense", ff=TOP * sz["expert_ff"] + sz["shared_ff"], limit=7.0)
    latent = dict(LATENT, heads=H, dim=128, rot=dict(base=10000.0, dims=ROT))
    gla = dict(heads=HL, dim=128, vdim=128, tau=16.0, rank=16)
    left = dict(heads=H, kv_heads=sz["kv_heads"], dim=128, vdim=128, scale=128 ** -0.5, softcap=30.0, rot=dict(base=10000.0, dims=128))
    right = dict(heads=HL, dim=128, vdim=128, rot=dict(base=10000.0, dims=64),
                 decay=[1.0 - 2.0 ** (-5.0 - 5.0 * h / max(1, HL - 1)) for h in range(HL)])
    both = dict(left=left, right=right, left_scale=0.8, right_scale=0.9)
    kinds = [("latent_attention", latent), ("gla", gla), ("gla", gla), ("parallel", both)]
    return dict(architecture="Kapuvik", vocab=VOCAB, width=sz["width"], norm=dict(eps=1e-6), embedding=dict(scale=0.5), logit_softcap=15.0,
                layers=[dict(type=k, mixer=dict(m), mlp=dict(ff)) for k, m in kinds])


def _birelix(sz):
    """Latent attention with a gate per head, two layers of the gated delta rule, windowed attention; routed experts."""
    dense = dict(kind="dense", ff=TOP * sz["expert_ff"] + sz["shared_ff"])
    moe = dict(kind="moe", expert=dict(ff=sz["expert_ff"], limit=7.0), router=dict(experts=EXPERTS, top=TOP, groups=dict(count=4, keep=2)))
    latent = dict(LATENT, heads=sz["heads"], dim=128, q_rank=768, rot=dict(base=10000.0, dims=ROT))
    attention = dict(heads=sz["heads"], kv_heads=sz["kv_heads"], dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=1024))
    rule = dict(heads=sz["lin_heads"], kv_heads=sz["lin_heads"] // 2, dim=128, vdim=128, conv=4)
    kinds = [("latent_attention", latent, dense), ("delta", rule, moe), ("delta", rule, moe), ("attention", attention, moe)]
    return dict(architecture="Birelix", vocab=VOCAB, width=sz["width"], norm=dict(eps=1e-6), embedding=dict(scale=8.0),
                layers=[dict(type=k, mixer=dict(m), mlp=dict(f)) for k, m, f in kinds])


def _raw(model):
    if model in QWEN3_SHAPES:
        return dict(QWEN3, **QWEN3_SHAPES[model])
    family, size = model.split("-")
    return (_kapuvik if family == "kapuvik" else _birelix)(TURN_SIZES[size])


def _is_turn(case):
    return case["model"] not in QWEN3_SHAPES


# ---- cases --------------------------------------------------------------------------------------------
# decode: requests that bring one token, on up to `cached` positions each (ragged: spread from a quarter of that);
# portions: requests that bring `portion` tokens of a prompt, on `portion_cached` positions each.

def _step(model, decode=0, cached=0, ragged=False, portions=0, portion=0, portion_cached=0, dtype="bfloat16", temperature=0.0, top_p=1.0):
    return dict(model=model, dtype=dtype, decode=decode, cached=cached, ragged=ragged, portions=portions, portion=portion,
                portion_cached=portion_cached, temperature=temperature, top_p=top_p)


def _turn(model, portions, portion, steps):
    return dict(model=model, dtype="bfloat16", portions=portions, portion=portion, steps=steps)


def listed():
    return [
        # one user talking to the smallest model: the smallest call there is
        dict(_step("qwen3-0.6b", decode=1, cached=500), name="decode_1_small"),
        # one user with a long document behind them
        dict(_step("qwen3-4b", decode=1, cached=16000), name="decode_1_long"),
        # the benchmark's headline: eight users of the 8B shape at 4,096 cached tokens
        dict(_step("qwen3-8b", decode=8, cached=4095), name="decode_8"),
        # a served model under moderate load: users at different places, tokens drawn from the nucleus
        dict(_step("qwen3-4b", decode=20, cached=3001, ragged=True, temperature=0.8, top_p=0.95), name="decode_20_ragged"),
        # the 8B shape's server, full: the benchmark's largest batch at the headline's context
        dict(_step("qwen3-8b", decode=64, cached=4095), name="decode_64"),
        # the benchmark's prompt
        dict(_step("qwen3-8b", portions=1, portion=2048), name="prefill_2048"),
        # a prompt of an odd length on a smaller model
        dict(_step("qwen3-1.7b", portions=1, portion=777), name="prefill_777"),
        # the last piece of a long prompt that is brought in pieces
        dict(_step("qwen3-4b", portions=1, portion=512, portion_cached=7680), name="chunk_512"),
        # continuous batching: short prompts arrive while other users' tokens are decoded
        dict(_step("qwen3-4b", decode=12, cached=2000, ragged=True, portions=2, portion=150), name="mixed"),
        # the 32-bit path (traces, comparisons): a short prompt beside decoded tokens
        dict(_step("qwen3-0.6b", decode=3, cached=400, ragged=True, portions=1, portion=96, dtype="float32"), name="float32_mixed"),
        # a turn of eight users on a model with latent attention and recurrent states: prompts, then decoded tokens
        dict(_turn("kapuvik-2k", 8, 256, 24), name="kapuvik_turn"),
        # a prompt on a model with the delta rule, latent attention and routed experts
        dict(_turn("birelix-2k", 1, 2048, 0), name="birelix_prefill"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "chunk", "mixed", "float32", "turn"])
    if kind == "decode":
        model = rng.choice(["qwen3-0.6b", "qwen3-1.7b", "qwen3-4b", "qwen3-8b"])
        batch = _log_int(rng, 1, 64)
        cached = _log_int(rng, 100, min(16000, 260000 // batch))
        sampled = rng.random() < 0.3
        return _step(model, decode=batch, cached=cached, ragged=rng.random() < 0.5, temperature=0.8 if sampled else 0.0,
                     top_p=0.95 if sampled else 1.0)
    if kind == "prefill":
        model = rng.choice(["qwen3-0.6b", "qwen3-1.7b", "qwen3-4b", "qwen3-8b"])
        portions = rng.choice([1, 1, 2, 3])
        return _step(model, portions=portions, portion=_log_int(rng, 40, 2000 // portions))
    if kind == "chunk":
        model = rng.choice(["qwen3-1.7b", "qwen3-4b"])
        return _step(model, portions=1, portion=_log_int(rng, 64, 1024), portion_cached=_log_int(rng, 500, 15000))
    if kind == "mixed":
        return _step(rng.choice(["qwen3-1.7b", "qwen3-4b"]), decode=rng.randint(2, 24), cached=_log_int(rng, 200, 4000), ragged=True,
                     portions=rng.randint(1, 3), portion=_log_int(rng, 40, 600))
    if kind == "float32":
        return _step("qwen3-0.6b", decode=rng.randint(1, 8), cached=_log_int(rng, 50, 800), ragged=True, portions=rng.randint(0, 1),
                     portion=rng.randint(20, 150), dtype="float32")
    if rng.random() < 0.5:
        return _turn("kapuvik-" + rng.choice(["1k", "2k"]), rng.randint(1, 8), _log_int(rng, 40, 250), rng.randint(8, 24))
    return _turn("birelix-" + rng.choice(["1k", "2k"]), 1, _log_int(rng, 200, 2000), 0)


# ---- inputs -------------------------------------------------------------------------------------------

def _requests(case):
    """[(cached positions, new tokens)] of a step's requests, those that decode first."""
    out = []
    for i in range(case["decode"]):
        c = case["cached"]
        out.append((max(1, c // 4 + (3 * c // 4) * (i * 7919 % 1000) // 1000) if case["ragged"] else c, 1))
    return out + [(case["portion_cached"], case["portion"])] * case["portions"]


def _tables(requests):
    """Pages per request when all of them take their pages one by one in turn, as requests that grow side by side do."""
    tables, nxt = [[] for _ in requests], 0
    need = [-(-(c + n) // PAGE) for c, n in requests]
    for k in range(max(need)):
        for i, t in enumerate(tables):
            if k < need[i]:
                t.append(nxt)
                nxt += 1
    return tables, nxt


def _tokens(case, seed, vocab):
    rng = random.Random(seed * 1000003 + 7)
    if _is_turn(case):
        return [[rng.randrange(vocab) for _ in range(case["portion"] + case["steps"])] for _ in range(case["portions"])]
    return [[rng.randrange(vocab) for _ in range(n)] for _, n in _requests(case)]


def _fill_cache(storage, seed, layer, width):
    """Cached keys (normed and rotated: unit deviation) and values (what a random projection of unit rows gives) of one layer."""
    g = torch.Generator(device=storage.device)
    g.manual_seed((seed * 1000003 + layer) & 0x7FFFFFFF)
    storage.normal_(generator=g)
    storage[1].mul_(0.02 * math.sqrt(width))


def prepare(case, seed):
    raw = _raw(case["model"])
    engine_config = dict(dtype=case["dtype"], page_size=PAGE)
    if _is_turn(case):
        n, length = case["portions"], case["portion"] + case["steps"] + 1
        cfg = (KapuvikConfig if raw["architecture"] == "Kapuvik" else BirelixConfig).from_dict(raw)
        engine = Engine(model_config=cfg, random_seed=seed, config=EngineConfig(
            num_pages=n * (-(-length // PAGE) + 1), max_running_requests=n, max_model_len=length + PAGE, **engine_config))
        state = dict(engine=engine, tokens=_tokens(case, seed, VOCAB), portion=case["portion"], steps=case["steps"])
        run(state)   # (a server has served before: its graphs are there)
        return state
    requests = _requests(case)
    tables, pages = _tables(requests)
    engine = Engine(model_config=Qwen3Config.from_dict(raw), random_seed=seed, config=EngineConfig(
        num_pages=pages, max_running_requests=len(requests), max_model_len=max(len(t) for t in tables) * PAGE, **engine_config))
    for i in range(len(requests)):
        engine.cache.add_request(i)
    for k in range(max(len(t) for t in tables)):
        for i, t in enumerate(tables):
            if k < len(t):
                engine.cache.reserve(i, (k + 1) * PAGE)
    storage = engine.cache.groups[0].storage
    if any(c for c, _ in requests):
        for layer in range(storage.shape[0]):
            _fill_cache(storage[layer], seed, layer, raw["hidden_size"])
    tokens = _tokens(case, seed, raw["vocab_size"])
    for i, (c, _) in enumerate(requests):
        engine.cache.commit(i, c)
    entries = [StepEntry(i, t, [len(t) - 1]) for i, t in enumerate(tokens)]
    rng, n = random.Random(seed + 11), len(requests)
    state = dict(engine=engine, entries=entries, sampling=([case["temperature"]] * n, [case["top_p"]] * n, [rng.random() for _ in range(n)]))
    if not case["portions"]:
        run(state)   # (a server captures its decode steps before the first request)
    return state


# ---- the passes ---------------------------------------------------------------------------------------

def run(state):
    engine = state["engine"]
    if "entries" in state:
        logits, _ = engine.runner.step_and_sample(state["entries"], *state["sampling"])
        engine.runner.check_errors()
        for e in state["entries"]:
            engine.cache.commit(e.request_id, -len(e.tokens))
        return logits
    tokens, T = state["tokens"], state["portion"]
    for i in range(len(tokens)):
        engine.cache.add_request(i)
    out = [engine.run_step([StepEntry(i, t[:T], [T - 1]) for i, t in enumerate(tokens)])]
    for k in range(state["steps"]):
        logits = engine.run_step([StepEntry(i, [t[T + k]], [0]) for i, t in enumerate(tokens)])
        out.append(logits.clone())   # (a captured step's logits are its graph's buffer)
    for i in range(len(tokens)):
        engine.cache.release(i)
    return torch.stack(out)


# ---- what a pass cannot do without ----------------------------------------------------------------------

def _qwen3_counts(cfg):
    """(elements of the matrices of a layer, of the head)."""
    E, I, H, G, D = (cfg[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
    return (H + 2 * G) * D * E + H * D * E + 3 * I * E, cfg["vocab_size"] * E


def _turn_counts(cfg):
    """(elements of all matrices, of those that a token is multiplied with), the head's included."""
    E = cfg["width"]
    every = used = cfg["vocab"] * E
    for layer in cfg["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        if layer["type"] == "latent_attention":
            q, c = m["dim"] + m["rot_dim"], m["kv_rank"]
            n = (c + m["rot_dim"]) * E + m["heads"] * (m["dim"] + m["vdim"]) * c + m["heads"] * m["vdim"] * E
            n += m["q_rank"] * (E + m["heads"] * q) + m["heads"] * E if "q_rank" in m else m["heads"] * q * E
        elif layer["type"] == "gla":
            n = 5 * m["heads"] * m["dim"] * E + m["rank"] * (E + m["heads"] * m["dim"])
        elif layer["type"] == "parallel":
            a, b = m["left"], m["right"]
            n = (2 * a["heads"] + 2 * a["kv_heads"]) * a["dim"] * E + 5 * b["heads"] * b["dim"] * E
        elif layer["type"] == "delta":
            n = (2 * m["kv_heads"] + 3 * m["heads"]) * m["dim"] * E + 2 * m["heads"] * E
        else:
            n = (2 * m["heads"] + 2 * m["kv_heads"]) * m["dim"] * E
        every, used = every + n, used + n
        if f["kind"] == "dense":
            every, used = every + 3 * f["ff"] * E, used + 3 * f["ff"] * E
        else:
            one, r = 3 * f["expert"]["ff"] * E, f["router"]
            every, used = every + r["experts"] * (one + E), used + r["top"] * one + r["experts"] * E
    return every, used


def work(case):
    raw = _raw(case["model"])
    if _is_turn(case):
        every, used = _turn_counts(raw)
        head = raw["vocab"] * raw["width"]
        n, T, K = case["portions"], case["portion"], case["steps"]
        # (the steps follow one another: each reads the weights)
        return dict(bytes=2.0 * every * (1 + K) + 4.0 * n * (1 + K) * raw["vocab"],
                    flops=2.0 * (used - head) * n * (T + K) + 2.0 * head * n * (1 + K))
    elt = 4 if case["dtype"] == "float32" else 2
    layer, head = _qwen3_counts(raw)
    L, H, G, D = (raw[k] for k in ("num_hidden_layers", "num_attention_heads", "num_key_value_heads", "head_dim"))
    requests = _requests(case)
    tokens, keys = sum(n for _, n in requests), sum(c + n for c, n in requests)
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in requests)
    return dict(bytes=float(elt * (L * layer + head + 2 * L * G * D * keys) + 4 * raw["vocab_size"] * len(requests)),
                flops=float(2 * L * layer * tokens + 4 * L * H * D * pairs + 2 * head * len(requests)))


def tolerance(case):
    # bfloat16: 0.012 to 0.018 between two right orders of the sums (largest single difference 0.08); 32 bits: 1.2e-5
    # against 64 bits, most of it the rotation's angles
    return {"rel": 5e-5, "max": 5e-4} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits ----------------------------------------------------------------------------------

class _Weights:
    """The engine's random weights: every tensor from a generator of its own, keyed by the seed and the tensor's name;
    matrices rounded to the engine's element type, everything else 32-bit."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype = seed, getattr(torch, dtype)

    def __call__(self, name, shape, role="matrix"):
        digest = hashlib.sha256(("%d:%s" % (self.seed, name)).encode()).digest()
        g = torch.Generator(device=DEVICE)
        g.manual_seed(int.from_bytes(digest[:8], "little") & 0x7FFFFFFFFFFFFFFF)
        x = torch.randn(shape, generator=g, dtype=torch.float32, device=DEVICE)
        x = 1.0 + 0.05 * x if role == "norm" else (0.5 if role == "taps" else 0.02) * x
        return (x.to(self.dtype) if role == "matrix" else x).double()


def _unit(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _angles(positions, base, dims):
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEVICE)
    a = positions.double()[:, None] * base ** (-2.0 * i / dims)
    return a.cos()[:, None], a.sin()[:, None]     # [T, 1, dims / 2]


def _rotate(x, positions, base, dims, interleaved):
    """x [..., T, heads, D]: the first `dims` channels of every head turned."""
    c, s = _angles(positions, base, dims)
    out = x.clone()
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if interleaved else (x[..., :dims // 2], x[..., dims // 2:dims])
    u, v = a * c - b * s, b * c + a * s
    if interleaved:
        out[..., 0:dims:2], out[..., 1:dims:2] = u, v
    else:
        out[..., :dims // 2], out[..., dims // 2:dims] = u, v
    return out


def _attend(q, k, v, scale, offset=0, softcap=0.0, window=0, plus_one=False):
    """q [T, H, D] at positions offset + t, k [S, G, D], v [S, G, Dv]; causal, heads in groups."""
    T, H = q.shape[:2]
    S, G = k.shape[:2]
    out = torch.empty((T, H, v.shape[2]), dtype=torch.float64, device=q.device)
    apart = (offset + torch.arange(T, device=q.device))[:, None] - torch.arange(S, device=q.device)
    hidden = (apart < 0) | (apart >= window) if window else apart < 0
    for g in range(G):
        mine = slice(g * (H // G), (g + 1) * (H // G))
        s = torch.einsum("thd,sd->hts", q[:, mine], k[:, g]) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(hidden, -math.inf)
        if plus_one:   # (one more entry with score 0 and no value)
            s = torch.cat([s, torch.zeros_like(s[..., :1])], -1)
        p = s.softmax(-1)[..., :S]
        out[:, mine] = torch.einsum("hts,sd->thd", p, v[:, g])
    return out


def _silu(z):
    return z * torch.sigmoid(z)


def _qwen3_exact(case, seed):
    cfg = _raw(case["model"])
    W = _Weights(seed, case["dtype"])
    E, I, H, G, D, L, V = (cfg[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                             "num_hidden_layers", "vocab_size"))
    eps, base = cfg["rms_norm_eps"], cfg["rope_theta"]
    requests = _requests(case)
    tables, pages = _tables(requests)
    tokens = _tokens(case, seed, V)
    positions = torch.cat([torch.arange(c, c + n, device=DEVICE) for c, n in requests])
    embed = W("model.embed_tokens.weight", (V, E))
    x = embed[torch.tensor([t for ts in tokens for t in ts], device=DEVICE)]
    cached = any(c for c, _ in requests)
    pool = torch.empty((2, pages, G, PAGE, D), dtype=getattr(torch, case["dtype"]), device=DEVICE) if cached else None
    index = [torch.tensor(t, device=DEVICE) for t in tables]
    for i in range(L):
        p = "model.layers.%d." % i
        h = _unit(x, eps) * W(p + "input_layernorm.weight", (E,), "norm")
        q = (h @ W(p + "self_attn.q_proj.weight", (H * D, E)).T).view(-1, H, D)
        k = (h @ W(p + "self_attn.k_proj.weight", (G * D, E)).T).view(-1, G, D)
        v = (h @ W(p + "self_attn.v_proj.weight", (G * D, E)).T).view(-1, G, D)
        q = _rotate(_unit(q, eps) * W(p + "self_attn.q_norm.weight", (D,), "norm"), positions, base, D, False)
        k = _rotate(_unit(k, eps) * W(p + "self_attn.k_norm.weight", (D,), "norm"), positions, base, D, False)
        if cached:
            _fill_cache(pool, seed, i, E)
        parts, at = [], 0
        for (c, n), pages_of in zip(requests, index):
            ks, vs = k[at:at + n], v[at:at + n]
            if c:
                old = pool[:, pages_of].transpose(2, 3).reshape(2, -1, G, D)[:, :c].double()
                ks, vs = torch.cat([old[0], ks]), torch.cat([old[1], vs])
            parts.append(_attend(q[at:at + n], ks, vs, D ** -0.5, c))
            at += n
        x = x + torch.cat(parts).view(-1, H * D) @ W(p + "self_attn.o_proj.weight", (E, H * D)).T
        h = _unit(x, eps) * W(p + "post_attention_layernorm.weight", (E,), "norm")
        a = _silu(h @ W(p + "mlp.gate_proj.weight", (I, E)).T) * (h @ W(p + "mlp.up_proj.weight", (I, E)).T)
        x = x + a @ W(p + "mlp.down_proj.weight", (E, I)).T
    last = torch.tensor([n for _, n in requests], device=DEVICE).cumsum(0) - 1
    h = _unit(x[last], eps) * W("model.norm.weight", (E,), "norm")
    return h @ (embed if cfg["tie_word_embeddings"] else W("lm_head.weight", (V, E))).T


def _walk(q, k, v, decay):
    """S_t = decay_t S_(t-1) + k_t v_t^T, o_t = S_t^T q_t; q, k [B, T, H, D], v [B, T, H, Dv], decay [B, T, H, D] or [H, 1]."""
    B, T, H, D = q.shape
    S = torch.zeros((B, H, D, v.shape[3]), dtype=torch.float64, device=q.device)
    out = torch.empty_like(v)
    for t in range(T):
        d = decay if decay.dim() == 2 else decay[:, t]
        S = S * d[..., None] + k[:, t][..., None] * v[:, t][..., None, :]
        out[:, t] = (S * q[:, t][..., None]).sum(2)
    return out


def _latent(h, W, p, m, eps, pos, gated):
    B, T, E = h.shape
    H, D, R, C, Dv, base = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], m["vdim"], m["rot"]["base"]
    if gated:
        q = _unit(h @ W(p + "dq", (m["q_rank"], E)).T, eps) * W(p + "dq.norm", (m["q_rank"],), "norm")
        q = (q @ W(p + "uq", (H * (D + R), m["q_rank"])).T).view(B, T, H, D + R)
    else:
        q = (h @ W(p + "q", (H * (D + R), E)).T).view(B, T, H, D + R)
    down = h @ W(p + "dkv", (C + R, E)).T
    c = _unit(down[..., :C], eps) * W(p + "dkv.norm", (C,), "norm")
    turned = _rotate(down[..., None, C:], pos, base, R, True).expand(B, T, H, R)
    k = torch.cat([(c @ W(p + "uk", (H * D, C)).T).view(B, T, H, D), turned], -1)
    v = (c @ W(p + "uv", (H * Dv, C)).T).view(B, T, H, Dv)
    q = torch.cat([q[..., :D], _rotate(q[..., D:], pos, base, R, True)], -1)
    o = torch.stack([_attend(q[b], k[b], v[b], m["scale"]) for b in range(B)])
    if gated:
        o = o * torch.sigmoid(h @ W(p + "g", (H, E)).T)[..., None]
    return o.reshape(B, T, H * Dv) @ W(p + "o", (E, H * Dv)).T


def _heads(h, W, name, heads, dim):
    return (h @ W(name, (heads * dim, h.shape[-1])).T).view(*h.shape[:2], heads, dim)


def _kapuvik_layer(x, W, p, layer, eps, pos):
    B, T, E = x.shape
    h = _unit(x, eps) * (1.0 + W(p + "norm1", (E,), "bias"))
    m, f, kind, q_ = layer["mixer"], layer["mlp"], layer["type"], p + "mix."
    if kind == "latent_attention":
        y = _latent(h, W, q_, m, eps, pos, False)
    elif kind == "gla":
        H, D, Dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (_heads(h, W, q_ + n, H, D) for n in "qkv")
        z = h @ W(q_ + "a1", (m["rank"], E)).T @ W(q_ + "a2", (H * D, m["rank"])).T + W(q_ + "a2.b", (H * D,), "bias")
        alpha = torch.sigmoid(z).pow(1.0 / m["tau"]).view(B, T, H, D)
        o = _unit(_walk(q * D ** -0.5, k, v, alpha), eps) * W(q_ + "norm", (Dv,), "norm")
        y = (o.reshape(B, T, -1) * _silu(h @ W(q_ + "g", (H * Dv, E)).T)) @ W(q_ + "o", (E, H * Dv)).T
    else:
        a, b = m["left"], m["right"]
        H, G, D = a["heads"], a["kv_heads"], a["dim"]
        q, k, v = _heads(h, W, q_ + "left.q", H, D), _heads(h, W, q_ + "left.k", G, D), _heads(h, W, q_ + "left.v", G, D)
        q, k = (_rotate(t, pos, a["rot"]["base"], a["rot"]["dims"], True) for t in (q, k))
        o = torch.stack([_attend(q[i], k[i], v[i], a["scale"], softcap=a["softcap"]) for i in range(B)])
        y = m["left_scale"] * (o.reshape(B, T, -1) @ W(q_ + "left.o", (E, H * D)).T)
        H, D = b["heads"], b["dim"]
        q, k, v = (_heads(h, W, q_ + "right." + n, H, D) for n in "qkv")
        q, k = (_rotate(t, pos, b["rot"]["base"], b["rot"]["dims"], False) for t in (q, k))
        decay = torch.tensor(b["decay"], dtype=torch.float64, device=DEVICE)[:, None]
        o = _unit(_walk(q, k * D ** -0.5, v, decay), eps).reshape(B, T, -1) * _silu(h @ W(q_ + "right.g", (H * D, E)).T)
        y = y + m["right_scale"] * (o @ W(q_ + "right.o", (E, H * D)).T)
    p += "mlp."
    g = (h @ W(p + "gate", (f["ff"], E)).T + W(p + "gate.b", (f["ff"],), "bias")).clamp(max=f["limit"])
    u = (h @ W(p + "up", (f["ff"], E)).T + W(p + "up.b", (f["ff"],), "bias")).clamp(-f["limit"], f["limit"])
    a = g * torch.sigmoid(1.702 * g) * (u + 1.0)
    return x + y + a @ W(p + "down", (E, f["ff"])).T + W(p + "down.b", (E,), "bias")


def _convolved(x, w):
    taps, y = w.shape[1], torch.zeros_like(x)
    for j in range(min(taps, x.shape[1])):
        y[:, j:] += x[:, :x.shape[1] - j] * w[:, taps - 1 - j]
    return _silu(y)


def _delta(h, W, p, m, eps):
    B, T, E = h.shape
    H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_convolved(h @ W(p + n, (r, E)).T, W(p + n + ".conv", (r, m["conv"]), "taps")) for n, r in zip("qkv", (G * D, G * D, H * Dv)))
    q, k = (t.view(B, T, G, D) / (t.view(B, T, G, D).square().sum(-1, keepdim=True) + 1e-6).sqrt() for t in (q, k))
    q, k = ((t * s).repeat_interleave(H // G, 2) for t, s in ((q, D ** -0.5), (k, 1.0)))
    v = v.view(B, T, H, Dv)
    beta = torch.sigmoid(h @ W(p + "b", (H, E)).T)
    step = torch.nn.functional.softplus(h @ W(p + "a", (H, E)).T + W(p + "dt_bias", (H,), "bias"))
    g = torch.exp(-torch.exp(W(p + "A_log", (H,), "bias")) * step)
    S, o = torch.zeros((B, H, D, Dv), dtype=torch.float64, device=h.device), torch.empty_like(v)
    for t in range(T):
        S = S * g[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - (S * k[:, t][..., None]).sum(2))
        S = S + k[:, t][..., None] * u[..., None, :]
        o[:, t] = (S * q[:, t][..., None]).sum(2)
    y = _unit(o, eps) * W(p + "norm", (Dv,), "norm") * _silu(_heads(h, W, p + "g", H, Dv))
    return y.reshape(B, T, -1) @ W(p + "o", (E, H * Dv)).T


def _routed(h, W, p, f):
    E, r, F, limit = h.shape[-1], f["router"], f["expert"]["ff"], f["expert"]["limit"]
    x = h.reshape(-1, E)
    s = torch.sigmoid(x @ W(p + "router", (r["experts"], E), "matrix_f32").T)
    n, keep = r["groups"]["count"], r["groups"]["keep"]
    best = s.view(len(x), n, -1).topk(2, -1).values.sum(-1).topk(keep, -1).indices
    allowed = torch.zeros((len(x), n), dtype=torch.bool, device=h.device).scatter_(1, best, True).repeat_interleave(r["experts"] // n, 1)
    w, chosen = s.masked_fill(~allowed, -1.0).topk(r["top"], -1)
    w = w / (w.sum(-1, keepdim=True) + 1e-20)
    y = torch.zeros_like(x)
    for e in range(r["experts"]):
        rows, which = (chosen == e).nonzero(as_tuple=True)
        q = p + "e%d." % e
        g = (x[rows] @ W(q + "gate", (F, E)).T).clamp(max=limit)
        u = (x[rows] @ W(q + "up", (F, E)).T).clamp(-limit, limit)
        y.index_add_(0, rows, w[rows, which][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W(q + "down", (E, F)).T))
    return y.view_as(h)


def _birelix_layer(x, W, p, layer, eps, pos):
    B, T, E = x.shape
    m, f, kind, q_ = layer["mixer"], layer["mlp"], layer["type"], p + "mix."
    h = _unit(x, eps) * W(p + "norm1", (E,), "norm")
    if kind == "latent_attention":
        y = _latent(h, W, q_, m, eps, pos, True)
    elif kind == "delta":
        y = _delta(h, W, q_, m, eps)
    else:
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (_heads(h, W, q_ + n, c, D) + W(q_ + n + ".b", (c * D,), "bias").view(c, D) for n, c in zip("qkv", (H, G, G)))
        o = torch.stack([_attend(_unit(q[i], eps), _unit(k[i], eps), v[i], m["scale"], window=m["mask"]["size"], plus_one=True) for i in range(B)])
        y = o.reshape(B, T, -1) @ W(q_ + "o", (E, H * D)).T
    x = x + y
    h = _unit(x, eps) * W(p + "norm2", (E,), "norm")
    p += "mlp."
    if f["kind"] == "dense":
        a = torch.nn.functional.gelu(h @ W(p + "gate", (f["ff"], E)).T, approximate="tanh") * (h @ W(p + "up", (f["ff"], E)).T)
        return x + a @ W(p + "down", (E, f["ff"])).T
    return x + _routed(h, W, p, f)


def _turn_exact(case, seed):
    cfg = _raw(case["model"])
    W = _Weights(seed, case["dtype"])
    E, eps, T = cfg["width"], cfg["norm"]["eps"], case["portion"]
    embed = W("embed", (cfg["vocab"], E))
    tokens = torch.tensor(_tokens(case, seed, cfg["vocab"]), device=DEVICE)
    x = embed[tokens] * cfg["embedding"]["scale"]
    pos = torch.arange(tokens.shape[1], device=DEVICE)
    kapuvik = cfg["architecture"] == "Kapuvik"
    for i, layer in enumerate(cfg["layers"]):
        x = (_kapuvik_layer if kapuvik else _birelix_layer)(x, W, "l%d." % i, layer, eps, pos)
    h = _unit(x[:, T - 1:], eps) * (1.0 + W("final.norm", (E,), "bias") if kapuvik else W("final.norm", (E,), "norm"))
    logits = h @ (W("head", (cfg["vocab"], E)) if kapuvik else embed).T
    if kapuvik:
        logits = cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])
    return logits.transpose(0, 1).contiguous()


@torch.no_grad()
def exact(case, seed):
    return (_turn_exact if _is_turn(case) else _qwen3_exact)(case, seed)
