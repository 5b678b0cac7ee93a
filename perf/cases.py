"""The work whose speed is watched: steps of the engine as its users have it do them.

A case is one pass through the public entry points.  Three kinds:

  step       ``ModelRunner.step`` over a ragged batch: ``decoding`` requests that get one token each behind the tokens they
             hold, and ``prompts`` portions of together ``tokens`` tokens behind ``cached`` tokens each.  Prompts and portions
             end with the pass; a decoding request goes on for ``ROOM`` passes, then it ends and another of its first length
             takes its place.  Outputs are the logits of every request's last token and the cache's tensors.
  generate   ``Engine.generate``: prompts in, sampled tokens out, with everything between (sessions, scheduler, sampler).

Models (random weights): the Qwen3-8B shape of the benchmark in bfloat16, eight of its layers in float32, the Bubotar sizes of
the benchmark (latent attention, selective scan, chunked attention), and a tiny configuration of the tests.
"""
from __future__ import annotations

import math
import zlib

import torch

PAGE = 16
ROOM = 128                 # passes after which a decoding request ends and another takes its place
CHECKED_TOKENS = 8192      # exact() follows whole sequences of together at most this many tokens

QWEN_8B = dict(
    architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=151936, hidden_size=4096, intermediate_size=12288,
    num_hidden_layers=36, num_attention_heads=32, num_key_value_heads=8, head_dim=128, rope_theta=1000000.0, rms_norm_eps=1e-6,
    tie_word_embeddings=False, use_sliding_window=False, sliding_window=None, max_window_layers=36, hidden_act="silu",
    attention_bias=False, initializer_range=0.02, eos_token_id=151645)
QWEN_TINY = dict(
    QWEN_8B, vocab_size=336, hidden_size=192, intermediate_size=224, num_hidden_layers=2, num_attention_heads=16,
    num_key_value_heads=8, head_dim=64, rope_theta=200000.0, rms_norm_eps=5e-6, max_window_layers=2, initializer_range=0.03,
    eos_token_id=13)
BUBOTAR = {
    "2k": dict(width=2048, groups=2, heads=16, kv_heads=4, dim=128, rot=64, rank=512, inner=4096, state=16, dt_rank=128, conv=4,
               ff=8192, chunk=1024, vocab=32000),
    "4k": dict(width=4096, groups=2, heads=32, kv_heads=8, dim=128, rot=64, rank=512, inner=8192, state=16, dt_rank=256, conv=4,
               ff=12288, chunk=1024, vocab=32000),
}


def _step(name, model="qwen3-8b", decoding=0, context=0, ragged=False, prompts=0, tokens=0, cached=0):
    return dict(name=name, kind="step", model=model, decoding=decoding, context=context, ragged=ragged, prompts=prompts,
                tokens=tokens, cached=cached)


def listed():
    return [
        # one user who reads along: the latency of a token
        _step("decode_1", decoding=1, context=900),
        # the benchmark's headline: a few long conversations
        _step("decode_8", decoding=8, context=3900),
        # a busy server: many conversations of unlike length
        _step("decode_48_ragged", decoding=48, context=1900, ragged=True),
        # questions of a line or two that arrive together
        _step("prompts_short", prompts=4, tokens=111),
        # the benchmark's prompt
        _step("prompt_2048", prompts=1, tokens=2048),
        # documents: the largest step
        _step("prompts_long", prompts=2, tokens=6143),
        # what the scheduler makes of the default token budget of a step: a portion of a long prompt beside decoding requests
        _step("portion_beside_decoding", decoding=7, context=2900, ragged=True, prompts=1, tokens=505, cached=1536),
        # the float32 engine (reference outputs, replay of traces): a few requests decoding, and a prompt
        _step("float32_decode_4", model="qwen3-8b-float32", decoding=4, context=460),
        _step("float32_prompt", model="qwen3-8b-float32", prompts=1, tokens=387),
        # another design: its prompt and its decoding
        _step("bubotar_prompt", model="bubotar-2k", prompts=1, tokens=2048),
        _step("bubotar_decode_8", model="bubotar-2k", decoding=8, context=1900),
        # the smallest models, as tests and examples run them: latency of launches and of the host
        dict(name="generate_tiny", kind="generate", prompts=6, longest=40, new=24),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    what = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "float32_decode", "float32_prompt", "bubotar_decode",
                       "bubotar_prompt", "generate"])
    if what == "generate":
        case = dict(kind="generate", prompts=_log_uniform(rng, 1, 8), longest=_log_uniform(rng, 4, 64), new=_log_uniform(rng, 8, 32))
    elif what == "decode":
        n = _log_uniform(rng, 1, 64)
        case = _step("", decoding=n, context=_log_uniform(rng, 32, min(4096, 60000 // n)), ragged=rng.random() < 0.6)
    elif what == "prompt":
        tokens = _log_uniform(rng, 2, 6000)
        case = _step("", prompts=_log_uniform(rng, 1, min(8, tokens)), tokens=tokens,
                     cached=rng.choice([0, 0, 0, _log_uniform(rng, 16, 2048)]))
    elif what == "mixed":
        n = _log_uniform(rng, 1, 24)
        case = _step("", decoding=n, context=_log_uniform(rng, 32, 2000), ragged=True, prompts=rng.choice([1, 1, 2]),
                     tokens=_log_uniform(rng, 16, 2048), cached=rng.choice([0, _log_uniform(rng, 16, 2048)]))
    elif what == "float32_decode":
        case = _step("", model="qwen3-8b-float32", decoding=_log_uniform(rng, 1, 8), context=_log_uniform(rng, 32, 500), ragged=True)
    elif what == "float32_prompt":
        case = _step("", model="qwen3-8b-float32", prompts=rng.choice([1, 2]), tokens=_log_uniform(rng, 4, 600))
    else:
        model = rng.choice(["bubotar-2k", "bubotar-2k", "bubotar-4k"])
        if what == "bubotar_decode":
            case = _step("", model=model, decoding=_log_uniform(rng, 1, 16), context=_log_uniform(rng, 32, 3000), ragged=rng.random() < 0.5)
        else:
            case = _step("", model=model, prompts=rng.choice([1, 1, 2]), tokens=_log_uniform(rng, 20, 4096))
    case.pop("name", None)
    return case


# ------------------------------------------------------------------------------------------------------------ models
def _raw(model):
    """config.json of a case's model, as a dict."""
    if model.startswith("bubotar"):
        z = BUBOTAR[model.split("-")[1]]
        lat = dict(heads=z["heads"], dim=z["dim"], rot_dim=z["rot"], vdim=z["dim"], kv_rank=z["rank"],
                   scale=1.0 / math.sqrt(z["dim"] + z["rot"]), rot=dict(base=10000.0, dims=z["rot"]))
        mlp = dict(kind="dense", ff=z["ff"], limit=7.0)
        layers = []
        for g in range(z["groups"]):
            layers += [dict(type="latent_attention", mixer=dict(lat), mlp=dict(mlp)),
                       dict(type="mamba1", mixer=dict(inner=z["inner"], state=z["state"], dt_rank=z["dt_rank"], conv=z["conv"]), mlp=None),
                       dict(type="attention", mixer=dict(heads=z["heads"], kv_heads=z["kv_heads"], dim=z["dim"], vdim=z["dim"],
                                                         scale=1.0 / math.sqrt(z["dim"]), mask=dict(size=z["chunk"])), mlp=dict(mlp)),
                       dict(type="latent_attention", mixer=dict(lat, kv_from=4 * g), mlp=dict(mlp))]
        return dict(architecture="Bubotar", vocab=z["vocab"], width=z["width"], norm=dict(eps=1e-6), logit_scale=1.0, layers=layers)
    if model == "qwen3-tiny":
        return dict(QWEN_TINY)
    return dict(QWEN_8B, num_hidden_layers=8 if model.endswith("float32") else 36)


def _dtype(model):
    return torch.float32 if model.endswith("float32") or model == "qwen3-tiny" else torch.bfloat16


def _shapes(raw):
    """name -> (shape, how it is drawn); "v..." tensors are held in float32 by every engine."""
    out = {}
    if raw.get("architecture") == "Bubotar":
        d = raw["width"]
        out["embed"] = ((raw["vocab"], d), "m")
        for i, layer in enumerate(raw["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            mix = {}
            if layer["type"] == "latent_attention":
                mix["q"] = (m["heads"] * (m["dim"] + m["rot_dim"]), d), "m"
                if m.get("kv_from") is None:
                    mix["dkv"] = (m["kv_rank"] + m["rot_dim"], d), "m"
                    mix["dkv.norm"] = (m["kv_rank"],), "v one"
                mix["uk"], mix["uv"] = ((m["heads"] * m["dim"], m["kv_rank"]), "m"), ((m["heads"] * m["vdim"], m["kv_rank"]), "m")
                mix["g"], mix["o"] = ((m["heads"] * m["vdim"], d), "m"), ((d, m["heads"] * m["vdim"]), "m")
            elif layer["type"] == "mamba1":
                inner, n = m["inner"], m["state"]
                mix = {"in": ((2 * inner, d), "m"), "conv": ((inner, m["conv"]), "v taps"), "conv.b": ((inner,), "v small"),
                       "x": ((m["dt_rank"] + 2 * n, inner), "m"), "dt": ((inner, m["dt_rank"]), "m wide"), "dt.b": ((inner,), "v step"),
                       "A_log": ((inner, n), "v decay"), "D": ((inner,), "v one"), "o": ((d, inner), "m")}
            else:
                mix = {"q": ((m["heads"] * m["dim"], d), "m"), "k": ((m["kv_heads"] * m["dim"], d), "m"),
                       "v": ((m["kv_heads"] * m["vdim"], d), "m"), "o": ((d, m["heads"] * m["vdim"]), "m")}
            out.update({p + "mix." + n: s for n, s in mix.items()})
            out[p + "norm1"] = out[p + "norm1b"] = (d,), "v one"
            if layer["mlp"] is not None:
                ff = layer["mlp"]["ff"]
                out[p + "mlp.gate"] = out[p + "mlp.up"] = (ff, d), "m"
                out[p + "mlp.down"] = (d, ff), "m"
                out[p + "norm2"] = out[p + "norm2b"] = (d,), "v one"
        out["final.norm"], out["head"] = ((d,), "v one"), ((raw["vocab"], d), "m")
        return out
    d, hd, ff = raw["hidden_size"], raw["head_dim"], raw["intermediate_size"]
    hq, hkv = raw["num_attention_heads"] * hd, raw["num_key_value_heads"] * hd
    out["model.embed_tokens.weight"] = (raw["vocab_size"], d), "m embed"
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        out.update({p + "self_attn.q_proj.weight": ((hq, d), "m"), p + "self_attn.k_proj.weight": ((hkv, d), "m"),
                    p + "self_attn.v_proj.weight": ((hkv, d), "m"), p + "self_attn.o_proj.weight": ((d, hq), "m out"),
                    p + "self_attn.q_norm.weight": ((hd,), "v one"), p + "self_attn.k_norm.weight": ((hd,), "v one"),
                    p + "mlp.gate_proj.weight": ((ff, d), "m"), p + "mlp.up_proj.weight": ((ff, d), "m"),
                    p + "mlp.down_proj.weight": ((d, ff), "m out"), p + "input_layernorm.weight": ((d,), "v one"),
                    p + "post_attention_layernorm.weight": ((d,), "v one")})
    out["model.norm.weight"], out["lm_head.weight"] = ((d,), "v one"), ((raw["vocab_size"], d), "m")
    return out


class _Weights:
    """Random weights by name, each drawn on its own from the seed and its name, on the GPU."""

    def __init__(self, model, seed):
        self.raw, self.dtype, self.seed = _raw(model), _dtype(model), int(seed)
        self.shapes = _shapes(self.raw)

    def __getitem__(self, name):
        shape, how = self.shapes[name]
        gen = torch.Generator(device="cuda").manual_seed((self.seed << 32) ^ zlib.crc32(name.encode()))
        t = torch.empty(shape, dtype=torch.float32, device="cuda")
        t = t.uniform_(generator=gen) if how == "v decay" else t.normal_(generator=gen)
        if how == "m":
            t.mul_(0.02)
        elif how == "m out":                  # what a layer adds to the stream: smaller the deeper the model, as models begin
            t.mul_(0.02 * (2 * self.raw["num_hidden_layers"]) ** -0.5)
        elif how == "m wide":
            t.mul_(shape[-1] ** -0.5)
        elif how == "v one":
            t.mul_(0.1).add_(1.0)
        elif how == "v taps":
            t.mul_(0.5)
        elif how == "v small":
            t.mul_(0.1)
        elif how == "v step":                 # softplus of it is a step size around 0.1 to 0.7
            t.mul_(0.7).sub_(1.0)
        elif how == "v decay":                # exp of it is a decay rate between 0.5 and 8
            t.mul_(7.5).add_(0.5).log_()
        return t if how.startswith("v") else t.to(self.dtype)

    def exact(self, name):
        return self[name].double()


def _engine(model, seed, **options):
    from pulsar_b200.config import config_from_dict
    from pulsar_b200.engine.engine import Engine
    from pulsar_b200.models import build_model
    weights = _Weights(model, seed)
    cfg = config_from_dict(weights.raw)
    net = build_model(cfg, weights.dtype)
    net.load({name: weights[name] for name in weights.shapes})
    return Engine.from_model(cfg, net, dict(dtype="float32" if weights.dtype == torch.float32 else "bfloat16", device="cuda:0",
                                            page_size=PAGE, eos_id=-1, **options))


# ------------------------------------------------------------------------------------------------------------ requests
def _vocab(model):
    raw = _raw(model)
    return raw.get("vocab_size") or raw["vocab"]


def _held(case):
    """Tokens that each decoding request holds before the pass."""
    n, top = case["decoding"], case["context"]
    if not case["ragged"] or n == 1:
        return [top] * n
    return [max(1, int(top * (1.0 - 0.85 * i / (n - 1)))) for i in range(n)]


def _portions(case):
    """Tokens of each prompt or portion: together ``tokens``, of unlike length."""
    n, total = case["prompts"], case["tokens"]
    if n == 0:
        return []
    lens = [max(1, int(total * 2 * (i + 1) / (n * (n + 1)))) for i in range(n)]
    lens[-1] += total - sum(lens)
    return lens


def _sequences(case, seed):
    """(tokens held, tokens of the pass) of every request, decoding requests first."""
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 13)
    vocab = _vocab(case["model"])
    sizes = [(h, 1) for h in _held(case)] + [(case["cached"], p) for p in _portions(case)]
    rows = []
    for held, new in sizes:
        ids = torch.randint(0, vocab, (held + new,), generator=gen).tolist()
        rows.append((ids[:held], ids[held:]))
    return rows


def _checked(case):
    """How many of the last requests exact() follows."""
    lens = [h + 1 for h in _held(case)] + [case["cached"] + p for p in _portions(case)]
    n = total = 0
    while n < len(lens) and total + lens[-1 - n] <= CHECKED_TOKENS:
        total += lens[-1 - n]
        n += 1
    return n


def prepare(case, seed):
    if case["kind"] == "generate":
        gen = torch.Generator().manual_seed(int(seed) * 7919 + 13)
        n, longest = case["prompts"], case["longest"]
        prompts = [torch.randint(0, QWEN_TINY["vocab_size"], (max(1, longest * (i + 1) // n),), generator=gen).tolist() for i in range(n)]
        engine = _engine("qwen3-tiny", seed, num_pages=512, max_sessions=8, max_running=8, max_chunk_size=512)
        return dict(kind="generate", engine=engine, prompts=prompts, new=case["new"], seed=int(seed))
    from pulsar_b200.engine.runner import StepEntry
    rows = _sequences(case, seed)
    pages = sum(-(-(len(held) + max(len(new), ROOM) + 1) // PAGE) + 1 for held, new in rows)
    engine = _engine(case["model"], seed, num_pages=pages, max_sessions=len(rows), max_running=len(rows), max_chunk_size=8192)
    # What the requests hold is computed as the engine computes it: prompts, a few thousand tokens at a time.
    group, size = [], 0
    for i, (held, _) in enumerate(rows):
        if held:
            group.append(StepEntry(i, held, []))
            size += len(held)
        if group and (size >= 2048 or i + 1 == len(rows)):
            engine.runner.step(group)
            group, size = [], 0
    entries = [StepEntry(i, new, [len(new) - 1]) for i, (_, new) in enumerate(rows)]
    return dict(kind="step", engine=engine, entries=entries, held=[len(h) for h, _ in rows], decoding=case["decoding"], passes=0,
                checked=_checked(case))


def _again(state, i):
    """Request ``i`` ends; another that holds as many tokens takes its place (their keys and values are the pages' contents)."""
    engine = state["engine"]
    engine.runner.finish(i)
    if state["held"][i]:
        engine.cache.open(i)
        engine.cache.append(i, state["held"][i])


def run(state):
    engine = state["engine"]
    if state["kind"] == "generate":
        got = engine.generate(state["prompts"], state["new"], temperature=0.8, top_k=40, top_p=0.95, seed=state["seed"])
        return torch.tensor(got, dtype=torch.int64)
    logits = engine.runner.step(state["entries"])
    for i in range(state["decoding"], len(state["entries"])):
        _again(state, i)
    state["passes"] += 1
    if state["passes"] % ROOM == 0:
        for i in range(state["decoding"]):
            _again(state, i)
    split = logits.shape[0] - state["checked"]
    return {"checked": logits[split:], "others": logits[:split] if split else None,
            "cache": [g.pools for g in engine.cache.groups], "state": dict(engine.cache.state)}


# ------------------------------------------------------------------------------------------------------------ the work
def work(case):
    if case["kind"] == "generate":
        shapes = _shapes(_raw("qwen3-tiny"))
        weights = sum(math.prod(s) for n, (s, _) in shapes.items() if "embed" not in n)
        tokens = sum(max(1, case["longest"] * (i + 1) // case["prompts"]) for i in range(case["prompts"])) + case["prompts"] * case["new"]
        return {"bytes": 4.0 * weights * case["new"], "flops": 2.0 * weights * tokens}
    raw, model = _raw(case["model"]), case["model"]
    shapes = _shapes(raw)
    size = 4 if _dtype(model) == torch.float32 else 2
    seqs = [(h, 1) for h in _held(case)] + [(case["cached"], p) for p in _portions(case)]
    n_new, n_rows = sum(n for _, n in seqs), len(seqs)
    head = next(math.prod(s) for n, (s, _) in shapes.items() if n in ("head", "lm_head.weight"))
    matrices = sum(math.prod(s) for n, (s, how) in shapes.items() if "embed" not in n and how.startswith("m")) - head
    vectors = sum(math.prod(s) for _, (s, how) in shapes.items() if how.startswith("v"))
    width, vocab = raw.get("hidden_size") or raw["width"], _vocab(model)
    data = size * (matrices + head + n_new * width) + 4.0 * vectors + 4.0 * n_rows * vocab
    flops = 2.0 * (matrices * n_new + head * n_rows)
    pairs = lambda held, new, reach: sum(min(p + 1, reach) for p in range(held, held + new)) if reach < held + new \
        else new * held + new * (new + 1) / 2                                                        # noqa: E731
    if raw.get("architecture") == "Bubotar":
        for layer in raw["layers"]:
            m = layer["mixer"]
            if layer["type"] == "latent_attention":
                row = m["kv_rank"] + m["rot_dim"]
                own = 1 if m.get("kv_from") is None else 0
                data += size * sum(row * (held + own * new) for held, new in seqs)
                flops += sum(2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * pairs(held, new, 1 << 30) for held, new in seqs)
            elif layer["type"] == "mamba1":
                data += 2.0 * 4 * len(seqs) * m["inner"] * (m["state"] + m["conv"] - 1)
                flops += n_new * m["inner"] * (8.0 * m["state"] + 2.0 * m["conv"])
            else:
                chunk = m["mask"]["size"]
                seen = sum(sum(p % chunk + 1 for p in range(held, held + new)) for held, new in seqs)
                data += size * m["kv_heads"] * (m["dim"] + m["vdim"]) * sum(held % chunk + new for held, new in seqs)
                flops += 2.0 * m["heads"] * (m["dim"] + m["vdim"]) * seen
        return {"bytes": float(data), "flops": float(flops)}
    layers, hd = raw["num_hidden_layers"], raw["head_dim"]
    data += size * layers * 2 * raw["num_key_value_heads"] * hd * sum(held + new for held, new in seqs)
    flops += layers * 4.0 * raw["num_attention_heads"] * hd * sum(pairs(held, new, 1 << 30) for held, new in seqs)
    return {"bytes": float(data), "flops": float(flops)}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"                     # token ids
    if _dtype(case["model"]) == torch.float32:
        return {"rel": 2e-5}               # 4e-6 from 64 bits, eight layers and the head
    return {"rel": 0.03}                   # a whole model in bfloat16: 0.005 to 0.02 from 64 bits


# ------------------------------------------------------------------------------------------------------------ 64 bits
def _norm(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _attend(q, k, v, scale, slopes=None, chunk=None):
    """q [L, H, D], k [L, G, D], v [L, G, V] -> [L, H * V], causal; a distance slope per head and a chunk mask where given."""
    L, H = q.shape[:2]
    per = H // k.shape[1]
    i = torch.arange(L, device=q.device)
    hidden = i[None, :] > i[:, None]
    if chunk is not None:
        hidden |= (i[None, :] // chunk) != (i[:, None] // chunk)
    out = torch.empty(L, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h // per].T).mul_(scale)
        if slopes is not None:
            s -= slopes[h] * (i[:, None] - i[None, :])
        out[:, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1) @ v[:, h // per]
    return out.reshape(L, -1)


def _angles(L, dims, base):
    freq = torch.tensor([base ** (-2.0 * j / dims) for j in range(dims // 2)], dtype=torch.float64, device="cuda")
    a = torch.arange(L, dtype=torch.float64, device="cuda")[:, None] * freq
    return a.cos()[:, None, :], a.sin()[:, None, :]


def _rotate_halves(x, base):
    cos, sin = _angles(x.shape[0], x.shape[-1], base)
    u, v = x.chunk(2, dim=-1)
    return torch.cat([u * cos - v * sin, v * cos + u * sin], dim=-1)


def _rotate_pairs(x, base):
    cos, sin = _angles(x.shape[0], x.shape[-1], base)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * cos - v * sin, v * cos + u * sin], dim=-1).flatten(-2)


def _qwen_layer(x, w, i, raw):
    p, eps, hd = f"model.layers.{i}.", raw["rms_norm_eps"], raw["head_dim"]
    for t in range(len(x)):
        L = x[t].shape[0]
        h = _norm(x[t], w(p + "input_layernorm.weight"), eps)
        q, k, v = ((h @ w(p + f"self_attn.{r}_proj.weight").T).view(L, -1, hd) for r in "qkv")
        q = _rotate_halves(_norm(q, w(p + "self_attn.q_norm.weight"), eps), raw["rope_theta"])
        k = _rotate_halves(_norm(k, w(p + "self_attn.k_norm.weight"), eps), raw["rope_theta"])
        x[t] = x[t] + _attend(q, k, v, hd ** -0.5) @ w(p + "self_attn.o_proj.weight").T
        h = _norm(x[t], w(p + "post_attention_layernorm.weight"), eps)
        act = torch.nn.functional.silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)
        x[t] = x[t] + act @ w(p + "mlp.down_proj.weight").T


def _scan(h, w, m):
    L, inner, n, r = h.shape[0], m["inner"], m["state"], m["dt_rank"]
    x, z = (h @ w("in").T).split(inner, dim=-1)
    taps = w("conv")
    padded = torch.cat([x.new_zeros(taps.shape[1] - 1, inner), x])
    x = torch.nn.functional.silu(sum(padded[t:t + L] * taps[:, t] for t in range(taps.shape[1])) + w("conv.b"))
    dt, b, c = (x @ w("x").T).split([r, n, n], dim=-1)
    dt = torch.nn.functional.softplus(dt @ w("dt").T + w("dt.b"), threshold=1e9)
    rate, skip = -torch.exp(w("A_log")), w("D")
    state, y = x.new_zeros(inner, n), torch.empty_like(x)
    for t in range(L):
        state = torch.exp(dt[t][:, None] * rate) * state + (dt[t] * x[t])[:, None] * b[t]
        y[t] = state @ c[t]
    return ((y + skip * x) * torch.nn.functional.silu(z)) @ w("o").T


def _bubotar_layer(x, w, i, raw, lent):
    p, layer, eps = f"l{i}.", raw["layers"][i], raw["norm"]["eps"]
    m = layer["mixer"]
    mix = lambda name: w(p + "mix." + name)                                                          # noqa: E731
    for t in range(len(x)):
        L = x[t].shape[0]
        h = _norm(x[t], w(p + "norm1"), eps)
        if layer["type"] == "latent_attention":
            H, rank, base = m["heads"], m["kv_rank"], m["rot"]["base"]
            q = (h @ mix("q").T).view(L, H, -1)
            q = torch.cat([q[..., :m["dim"]], _rotate_pairs(q[..., m["dim"]:], base)], dim=-1)
            if m.get("kv_from") is None:
                down = h @ mix("dkv").T
                lent[t] = _norm(down[:, :rank], mix("dkv.norm"), eps), _rotate_pairs(down[:, None, rank:], base)
            latent, key_rot = lent[t]
            k = torch.cat([(latent @ mix("uk").T).view(L, H, -1), key_rot.expand(L, H, -1)], dim=-1)
            y = _attend(q, k, (latent @ mix("uv").T).view(L, H, -1), m["scale"])
            y = (y * torch.sigmoid(h @ mix("g").T)) @ mix("o").T
        elif layer["type"] == "mamba1":
            y = _scan(h, mix, m)
        else:
            H, G = m["heads"], m["kv_heads"]
            q, k, v = (h @ mix("q").T).view(L, H, -1), (h @ mix("k").T).view(L, G, -1), (h @ mix("v").T).view(L, G, -1)
            y = _attend(q, k, v, m["scale"], [2.0 ** (-8.0 * (j + 1) / H) for j in range(H)], m["mask"]["size"]) @ mix("o").T
        x[t] = x[t] + _norm(y, w(p + "norm1b"), eps)
        if layer["mlp"] is not None:
            limit = layer["mlp"]["limit"]
            h = _norm(x[t], w(p + "norm2"), eps)
            g, u = (h @ w(p + "mlp.gate").T).clamp(max=limit), (h @ w(p + "mlp.up").T).clamp(-limit, limit)
            x[t] = x[t] + _norm((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + "mlp.down").T, w(p + "norm2b"), eps)


def exact(case, seed):
    """The logits of the requests that ``_checked`` names, from their whole sequences in 64 bits.  The other requests' logits and
    the cache's tensors (whose pages are the cache manager's to choose) have none, nor have sampled tokens."""
    if case["kind"] == "generate":
        return None
    n = _checked(case)
    if n == 0:
        return None
    weights = _Weights(case["model"], seed)
    raw = weights.raw
    bubotar = raw.get("architecture") == "Bubotar"
    embed, head, final = ("embed", "head", "final.norm") if bubotar else ("model.embed_tokens.weight", "lm_head.weight", "model.norm.weight")
    table = weights[embed]
    x = [table[torch.tensor(held + new, device="cuda")].double() for held, new in _sequences(case, seed)[-n:]]
    del table
    lent = {}
    for i in range(len(raw["layers"]) if bubotar else raw["num_hidden_layers"]):
        kept = {}

        def w(name):
            if name not in kept:
                kept[name] = weights.exact(name)
            return kept[name]
        _bubotar_layer(x, w, i, raw, lent) if bubotar else _qwen_layer(x, w, i, raw)
    eps = raw["norm"]["eps"] if bubotar else raw["rms_norm_eps"]
    last = _norm(torch.stack([rows[-1] for rows in x]), weights.exact(final), eps)
    return {"checked": last @ weights.exact(head).T, "others": None, "cache": None, "state": None}
