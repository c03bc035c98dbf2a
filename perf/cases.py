"""The work this framework is timed on: steps of the served models through `Decoder` and `ModelRunner`.

A case is one step of a model with the layer shapes of one of the repository's configurations and fewer layers: a decode step (every sequence
gets one token, `ModelRunner.decode_step`, captured) or a prefill chunk (`ModelRunner.prefill`, prompts or the next portion of them). `prepare`
makes the weights, the paged cache with what earlier steps left in it, and the runner; `run` is one step and returns its logits and the cache.

Weights are random with the scales of a trained model where those matter for the numbers: the projections back into the stream are small (the
usual 1 / sqrt(2 x layers) of a 32-layer model), and a token's embedding leans towards two experts of every router, so that the choice of experts
is as decided as a trained router's and does not hang on the last bit of a 16-bit sum.
"""
import math

import torch

from skein_b200.models import config as mc
from skein_b200.models.decoder import Decoder, LayerWeights, ModelWeights, layered_weights, quantize_blocks
from skein_b200.models.layered import DenseFFSpec, unroll_loop
from skein_b200.models.parallel_layers import MixerPairSpec, RecurrentSpec, WindowAttnSpec
from skein_b200.runtime.runner import ModelRunner

DEV = "cuda"
PAGE = 16             # tokens per cache page of the uniform families
WINDOW_PAGE = 64      # of Sikalorn
BACK = 0.02 / 8       # standard deviation of the projections back into the stream: 0.02 / sqrt(2 x 32)

# layer shapes of configs/*.json
UNIFORM = {
    "mixtral": dict(arch="MixtralForCausalLM", hidden=4096, inter=14336, heads=32, kv_heads=8, vocab=32000, experts=8, theta=1e6, eps=1e-5),
    "mistral": dict(arch="MistralForCausalLM", hidden=4096, inter=14336, heads=32, kv_heads=8, vocab=32768, experts=0, theta=1e6, eps=1e-5),
    "qwen": dict(arch="Qwen2ForCausalLM", hidden=3584, inter=18944, heads=28, kv_heads=4, vocab=152064, experts=0, theta=1e6, eps=1e-6),
    "llama70b": dict(arch="LlamaForCausalLM", hidden=8192, inter=28672, heads=64, kv_heads=8, vocab=128256, experts=0, theta=5e5, eps=1e-5),
}
LAYERS = {"mixtral": 4, "mistral": 4, "qwen": 4, "llama70b": 4, "sikalorn": 6}
HEAD = 128
# Sikalorn: runs delta, pair, lightning, pair, lightning, pair (the middle two layers twice), sizes of the 7B configuration
SIK = dict(width=4096, heads=32, ff=14336, vocab=32000, window=1024, theta=5e5, factor=2.0, eps=1e-5, loop=(1, 3, 2))


def listed():
    return [
        # one user's chat on the headline model: nothing but latency
        {"name": "mixtral_decode_1", "model": "mixtral", "mode": "decode", "seqs": 1, "new": 1, "cached": 511, "ragged": False, "fp8": False},
        # the headline benchmark's step: 64 sequences, prompt 512 and half of the 256 tokens generated
        {"name": "mixtral_decode_64", "model": "mixtral", "mode": "decode", "seqs": 64, "new": 1, "cached": 639, "ragged": False, "fp8": False},
        # e4m3 experts, the sequences of one rank of the expert-parallel configuration, lengths as a server has them
        {"name": "mixtral_fp8_decode_32", "model": "mixtral", "mode": "decode", "seqs": 32, "new": 1, "cached": 1500, "ragged": True, "fp8": True},
        # long contexts and few sequences: a step that is mostly attention
        {"name": "mistral_decode_5_long", "model": "mistral", "mode": "decode", "seqs": 5, "new": 1, "cached": 8000, "ragged": True, "fp8": False},
        # Llama-3-70B with e4m3 blocks, 32 sequences behind prompts of 2048
        {"name": "llama70b_fp8_decode_32", "model": "llama70b", "mode": "decode", "seqs": 32, "new": 1, "cached": 2111, "ragged": False, "fp8": True},
        # a short question: time to first token
        {"name": "mixtral_prompt_37", "model": "mixtral", "mode": "prefill", "seqs": 1, "new": 37, "cached": 0, "ragged": False, "fp8": False},
        # the headline benchmark's prefill: a 4096-token chunk of 512-token prompts
        {"name": "mixtral_prompts_8x512", "model": "mixtral", "mode": "prefill", "seqs": 8, "new": 512, "cached": 0, "ragged": False, "fp8": False},
        # the last portion of an 8192-token prompt that is fed 2048 tokens at a time
        {"name": "mistral_portion_2048", "model": "mistral", "mode": "prefill", "seqs": 1, "new": 2048, "cached": 6144, "ragged": False, "fp8": False},
        # prompts of all lengths in one chunk, widths that are no powers of two, biases, a large vocabulary
        {"name": "qwen_prompts_ragged", "model": "qwen", "mode": "prefill", "seqs": 11, "new": 397, "cached": 0, "ragged": True, "fp8": False},
        # the longest prompt its configuration takes, as one chunk
        {"name": "llama70b_prompt_8191", "model": "llama70b", "mode": "prefill", "seqs": 1, "new": 8191, "cached": 0, "ragged": False, "fp8": False},
        # recurrences and window attention: prompts, and a decode step whose batch is no capture class
        {"name": "sikalorn_prompts_ragged", "model": "sikalorn", "mode": "prefill", "seqs": 6, "new": 1100, "cached": 0, "ragged": True, "fp8": False},
        {"name": "sikalorn_decode_48", "model": "sikalorn", "mode": "decode", "seqs": 48, "new": 1, "cached": 350, "ragged": True, "fp8": False},
    ]


def draw(rng):
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))      # noqa: E731
    model = rng.choice(("mixtral", "mixtral", "mistral", "llama70b", "qwen", "sikalorn"))
    fp8 = model in ("mixtral", "llama70b") and rng.random() < 0.35
    c = {"model": model, "mode": rng.choice(("decode", "prefill")), "ragged": rng.random() < 0.6, "fp8": fp8}
    if c["mode"] == "decode":
        seqs = spread(1, 64)
        cached = spread(16, min(8000, 131072 // seqs)) if model != "sikalorn" else spread(16, 500)
        return {**c, "seqs": seqs, "new": 1, "cached": cached}
    total = spread(16, 4096 if model == "llama70b" else 6000)
    seqs = spread(1, max(1, min(16, total // 16)))
    cached = spread(64, 6000 // seqs) if model != "sikalorn" and rng.random() < 0.3 else 0
    return {**c, "seqs": seqs, "new": max(1, total // seqs), "cached": cached}


def lengths(case):
    """(new tokens, cached tokens) of every sequence: all alike, or from a fifth of the given numbers up to them."""
    share = [0.2 + 0.8 * ((i + 1) * 0.6180339887 % 1.0) if case["ragged"] else 1.0 for i in range(case["seqs"])]
    return [max(1, round(case["new"] * f)) for f in share], [round(case["cached"] * f) for f in share]


# ---- inputs ---------------------------------------------------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _normal(g, *shape, std=0.02):
    return torch.empty(*shape, dtype=torch.bfloat16, device=DEV).normal_(0.0, std, generator=g)


def _batch(case, g, vocab, page):
    """Tokens of the step and, per sequence, its pages: scattered over the pool as a server leaves them."""
    new, cached = lengths(case)
    tokens = [torch.randint(vocab, (n,), device=DEV, generator=g).tolist() for n in new]
    blocks = [(n + c + page - 1) // page for n, c in zip(new, cached)]
    order = torch.randperm(sum(blocks) + 1, device=DEV, generator=g).tolist()
    tables, at = [], 0
    for b in blocks:
        tables.append(order[at:at + b])
        at += b
    return {"new": new, "cached": cached, "tokens": tokens, "tables": tables, "pages": sum(blocks) + 1}


def _uniform(case, seed):
    """Plain tensors of a uniform model's case: weights, cache pools, batch."""
    m, L, g = UNIFORM[case["model"]], LAYERS[case["model"]], _gen(seed)
    H, I, E, kv, q = m["hidden"], m["inter"], m["experts"], m["kv_heads"] * HEAD, m["heads"] * HEAD
    d = _batch(case, g, m["vocab"], PAGE)
    d["embed"] = _normal(g, m["vocab"], H, std=1.0)
    d["layers"], d["pools"] = [], []
    for _ in range(L):
        lead = (E,) if E else ()
        w = {"attn_norm": _normal(g, H, std=0.1) + 1, "ffn_norm": _normal(g, H, std=0.1) + 1, "wqkv": _normal(g, q + 2 * kv, H),
             "bqkv": _normal(g, q + 2 * kv) if m["arch"].startswith("Qwen2") else None, "wo": _normal(g, H, q, std=BACK),
             "router": _normal(g, E, H) if E else None, "w13": _normal(g, *lead, 2 * I, H), "w2": _normal(g, *lead, H, I, std=BACK)}
        if E:       # two experts per token and layer: 8 and 6 on the router's scale, where the others have a deviation of 1.3
            d["embed"] += _lean(g, w["router"], m["vocab"])
        d["layers"].append(w)
        d["pools"].append(_normal(g, d["pages"], 2, m["kv_heads"], PAGE, HEAD, std=1.2))
    d["final_norm"], d["head"] = _normal(g, H, std=0.1) + 1, _normal(g, m["vocab"], H)
    return d


def _lean(g, router, vocab):
    first = torch.randint(router.shape[0], (vocab,), device=DEV, generator=g)
    second = (first + torch.randint(1, router.shape[0], (vocab,), device=DEV, generator=g)) % router.shape[0]
    r = router.float()
    r = r / r.square().sum(-1, keepdim=True)
    return (8.0 * r[first] + 6.0 * r[second]).bfloat16()


def _sikalorn_specs():
    H, ff = SIK["heads"], DenseFFSpec(SIK["ff"])
    pair = MixerPairSpec(WindowAttnSpec(H, H // 4, HEAD, HEAD, HEAD ** -0.5, HEAD, SIK["theta"], SIK["factor"], SIK["window"]),
                         RecurrentSpec("ssd", 2 * H, 1, HEAD, 64, 4, 8), 0.7, 0.7)
    light = RecurrentSpec("lightning", H, H, HEAD, HEAD, decay=tuple(_light_decay()))
    return unroll_loop([(RecurrentSpec("delta", H, H // 2, HEAD, HEAD, 4), ff), (pair, ff), (light, ff), (pair, ff)], SIK["loop"])


def _light_decay():
    H = SIK["heads"]
    return [1 - 2.0 ** -(2 + 6 * i / (H - 1)) for i in range(H)]


def _sikalorn(case, seed):
    """Plain tensors of a Sikalorn case: checkpoint tensors by name, the whole sequences, batch."""
    g, C, H, ff, V = _gen(seed), SIK["width"], SIK["heads"], SIK["ff"], SIK["vocab"]
    d = _batch(case, g, V, WINDOW_PAGE)
    d["before"] = [torch.randint(V, (n,), device=DEV, generator=g).tolist() for n in d["cached"]]
    t = {"embed": _normal(g, V, C, std=1.0), "head": _normal(g, V, C)}
    around = lambda *s, mean, std: (torch.randn(s, device=DEV, generator=g) * std + mean).bfloat16()      # noqa: E731

    def norm(name):
        t[name], t[name + ".b"], t[name + ".alpha"] = around(C, mean=1, std=0.1), around(C, mean=0, std=0.1), around(mean=0.5, std=0.02)

    def decay(p, heads):        # step sizes from 0.001 to 0.1 and decay rates from 1 to 16, as these recurrences are initialised
        dt = torch.exp(torch.rand(heads, device=DEV, generator=g) * math.log(100.0) + math.log(1e-3))
        t[p + "dt_bias"] = (dt + torch.log(-torch.expm1(-dt))).bfloat16()
        t[p + "A_log"] = torch.log(1 + 15 * torch.rand(heads, device=DEV, generator=g)).bfloat16()

    def pair(p):
        G, ch = H // 4, 2 * H * 64 + 2 * HEAD
        for n, rows in (("q", H * HEAD), ("k", G * HEAD), ("v", G * HEAD)):
            t[p + "left." + n] = _normal(g, rows, C)
        t[p + "left.q.norm"], t[p + "left.k.norm"] = around(H * HEAD, mean=1, std=0.1), around(G * HEAD, mean=1, std=0.1)
        t[p + "left.o"] = _normal(g, C, H * HEAD, std=BACK)
        r = p + "right."
        t[r + "in"] = _normal(g, 2 * H * 64 + ch + 2 * H, C)        # z | x, B, C | dt
        t[r + "conv"], t[r + "conv.b"] = around(ch, 4, mean=0, std=0.5), around(ch, mean=0, std=0.1)
        decay(r, 2 * H)
        t[r + "D"], t[r + "norm"], t[r + "o"] = around(2 * H, mean=1, std=0.1), around(2 * H * 64, mean=1, std=0.1), _normal(g, C, 2 * H * 64, std=BACK)

    def delta(p):
        for n, rows in (("q", H // 2 * HEAD), ("k", H // 2 * HEAD), ("v", H * HEAD)):
            t[p + n], t[p + n + ".conv"] = _normal(g, rows, C), around(rows, 4, mean=0, std=0.5)
        t[p + "g"], t[p + "b"], t[p + "a"] = _normal(g, H * HEAD, C), _normal(g, H, C), _normal(g, H, C)
        decay(p, H)
        t[p + "norm"], t[p + "o"] = around(HEAD, mean=1, std=0.1), _normal(g, C, H * HEAD, std=BACK)

    def light(p):
        for n in ("q", "k", "v", "g"):
            t[p + n] = _normal(g, H * HEAD, C)
        t[p + "norm"], t[p + "o"] = around(H * HEAD, mean=1, std=0.1), _normal(g, C, H * HEAD, std=BACK)

    for i, mixer in enumerate((delta, pair, light, pair)):
        norm(f"l{i}.norm1")
        mixer(f"l{i}.mix.")
        t[f"l{i}.mlp.up"], t[f"l{i}.mlp.down"] = _normal(g, ff, C), _normal(g, C, ff, std=BACK)
    eye = 0.7 * torch.eye(C, device=DEV)
    t["loop.in"] = (torch.cat([eye, eye], dim=1) + _normal(g, C, 2 * C, std=0.002)).bfloat16()
    t["loop.step"] = around(SIK["loop"][2], C, mean=0, std=0.1)
    norm("final.norm")
    d["tensors"] = t
    return d


# ---- a step ---------------------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    if case["model"] == "sikalorn":
        d = _sikalorn(case, seed)
        cfg = mc.ModelConfig.layered("Sikalorn", _sikalorn_specs(), width=SIK["width"], vocab=SIK["vocab"], max_pos=8192, name="sikalorn",
                                     eps=SIK["eps"], loop=SIK["loop"])
        dec = Decoder(cfg, layered_weights(cfg, d["tensors"].__getitem__), num_pages=d["pages"], page_size=WINDOW_PAGE, state_slots=case["seqs"])
        page = WINDOW_PAGE
    else:
        d, m = _uniform(case, seed), UNIFORM[case["model"]]
        cfg = mc.ModelConfig(architecture=m["arch"], hidden_size=m["hidden"], intermediate_size=m["inter"], num_layers=LAYERS[case["model"]],
                             num_heads=m["heads"], num_kv_heads=m["kv_heads"], head_dim=HEAD, vocab_size=m["vocab"], rms_norm_eps=m["eps"],
                             rope_theta=m["theta"], num_experts=m["experts"], top_k=2 if m["experts"] else 0, max_position_embeddings=8192,
                             name=case["model"], qkv_bias=m["arch"].startswith("Qwen2"))
        w = ModelWeights(embed=d["embed"], layers=[LayerWeights(**lw) for lw in d["layers"]], final_norm=d["final_norm"], lm_head=d["head"])
        if case["fp8"]:
            quantize_blocks(w, range(len(w.layers)), names=("w13", "w2") if m["experts"] else ("wqkv", "wo", "w13", "w2"))
        dec = Decoder(cfg, w, num_pages=d["pages"], page_size=PAGE, kv_pools=d["pools"])
        page = PAGE
    total = max(n + c for n, c in zip(d["new"], d["cached"]))
    runner = ModelRunner(dec, max_blocks_per_seq=(total + page - 1) // page, ctx_hint=total)
    slots = list(range(case["seqs"]))
    bucket = runner.bucket(case["seqs"]) if case["mode"] == "decode" else None
    if bucket is not None:      # captured on padding rows, as a server does while it starts
        runner.load_decode_inputs(bucket, [], [], [], [])
        runner.decode_step(bucket)
    if case["model"] == "sikalorn" and case["cached"]:      # the prompts before this step leave cache pages and states; 16 of them a chunk
        for at in range(0, case["seqs"], 16):
            runner.prefill([(d["before"][i], d["tables"][i], 0, i) for i in slots[at:at + 16]])
    if bucket is not None:
        runner.load_decode_inputs(bucket, [ids[0] for ids in d["tokens"]], d["cached"], [c + 1 for c in d["cached"]], d["tables"], slots=slots)
    return {"runner": runner, "decoder": dec, "rows": case["seqs"], "bucket": bucket, "seqs": list(zip(d["tokens"], d["tables"], d["cached"], slots))}


def run(state):
    runner, dec, b = state["runner"], state["decoder"], state["bucket"]
    if b is not None:
        runner.decode_step(b)
        logits = b.graph_logits[(False, False)][:state["rows"]]
    else:
        _, logits = runner.prefill(state["seqs"], want_logits=True)
    states = [r.mat for r in getattr(dec, "rec_state", []) if r is not None]
    return {"logits": logits, "cache": [p for p in dec.kv if p is not None], "states": states}


# ---- what a step cannot do without ----------------------------------------------------------------------------------------------


def work(case):
    new, cached = lengths(case)
    rows, S = sum(new), case["seqs"]
    if case["model"] == "sikalorn":
        return _sikalorn_work(new, cached)
    m, L = UNIFORM[case["model"]], LAYERS[case["model"]]
    H, I, E, kv, q = m["hidden"], m["inter"], m["experts"], m["kv_heads"] * HEAD, m["heads"] * HEAD
    attn, ff = H * (2 * q + 2 * kv), 3 * H * I
    used = E * (1 - (1 - 2 / E) ** rows) if E else 1        # experts that some token chose
    attn_bytes = attn * (1 if case["fp8"] and not E else 2)
    ff_bytes = ff * used * (1 if case["fp8"] else 2)
    pairs = sum(n * c + n * (n + 1) / 2 for n, c in zip(new, cached))       # (query, key) pairs
    cache = 2 * kv * 2 * (sum(cached) + rows)
    return {"bytes": L * (attn_bytes + ff_bytes + cache) + 2 * m["vocab"] * (H + S) + 2 * H * rows,
            "flops": L * (2 * rows * (attn + ff * (2 if E else 1)) + 4 * q * pairs) + 2 * S * m["vocab"] * H}


def _sikalorn_work(new, cached):
    C, H, ff, S, rows = SIK["width"], SIK["heads"], SIK["ff"], len(new), sum(new)
    seen = lambda c, n: sum(min(SIK["window"], c + i + 1) for i in range(n))        # noqa: E731
    keys, pairs = sum(min(SIK["window"], c) + n for c, n in zip(cached, new)), sum(seen(c, n) for c, n in zip(cached, new))
    q, inner = H * HEAD, 2 * H * 64
    state = H * HEAD * HEAD         # elements of a sequence's state, alike for the three recurrences
    mixers = {"delta": C * (q // 2 * 2 + 3 * q + 2 * H), "light": C * 5 * q, "pair": C * (2 * q + q // 2 + 3 * inner + 2 * HEAD + 2 * H)}
    runs = ("delta", "pair", "light", "pair", "light", "pair")
    distinct = ("delta", "pair", "light", "pair")
    weights = sum(2 * (mixers[r] + 2 * C * ff) for r in distinct) + 2 * 2 * C * C + 2 * SIK["vocab"] * C
    carried = 2 if any(cached) else 1       # states read and written, or written
    moved = sum(4 * carried * state * S + (2 * q // 4 * 2 * keys if r == "pair" else 0) for r in runs)
    flops = sum(2 * rows * (mixers[r] + 2 * C * ff) + 6 * state * rows + (4 * q * pairs if r == "pair" else 0) for r in runs)
    return {"bytes": weights + moved + 2 * S * SIK["vocab"] + 2 * C * rows, "flops": flops + 2 * (2 * rows * 2 * C * C) + 2 * S * SIK["vocab"] * C}


def tolerance(case):
    return {"rel": 0.02, "max": 0.5}


# ---- the same step in 64 bits ---------------------------------------------------------------------------------------------------


def exact(case, seed):
    with torch.no_grad():
        return _sikalorn_exact(_sikalorn(case, seed)) if case["model"] == "sikalorn" else _uniform_exact(case, _uniform(case, seed))


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _mm(x, w):
    """x @ w^T, a part of the weight at a time in 64 bits."""
    return torch.cat([x @ p.double().T for p in w.split(8192)], dim=-1)


def _rotate(x, pos, theta, factor=1.0):
    """x [tokens, heads, HEAD]: coordinate i turns with coordinate i + HEAD / 2."""
    half = HEAD // 2
    a = pos.double()[:, None, None] * theta ** (-torch.arange(half, device=DEV, dtype=torch.float64) / half) / factor
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1)


def _attend(q, k, v, first, window=None):
    """q [n, heads, HEAD] at positions first.., k, v [keys, kv heads, HEAD]."""
    n, group, out = q.shape[0], q.shape[1] // k.shape[1], torch.empty_like(q)
    back = torch.arange(first, first + n, device=DEV)[:, None] - torch.arange(k.shape[0], device=DEV)
    hidden = (back < 0) if window is None else (back < 0) | (back >= window)
    per = max(1, 100_000_000 // (n * k.shape[0] * group))       # kv heads at a time
    for h in range(0, k.shape[1], per):
        kk, vv = k[:, h:h + per].permute(1, 2, 0), v[:, h:h + per].transpose(0, 1)
        qq = q[:, h * group:(h + per) * group].unflatten(1, (-1, group)).permute(1, 2, 0, 3)
        s = (qq @ kk[:, None]) * HEAD ** -0.5
        p = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1) @ vv[:, None]
        out[:, h * group:(h + per) * group] = p.permute(2, 0, 1, 3).flatten(1, 2)
    return out


def _e4m3(w):
    """The weight as a block-scaled e4m3 copy holds it: per 128 inputs the smallest power of two that brings the largest into range."""
    out = torch.empty_like(w)
    for o, i in zip(out.view(-1, w.shape[-1]).split(8192), w.reshape(-1, w.shape[-1]).split(8192)):
        b = i.float().unflatten(-1, (-1, 128))
        s = torch.exp2(torch.ceil(torch.log2(b.abs().amax(-1, keepdim=True) / 448)))
        o.copy_(((b / s).to(torch.float8_e4m3fn).float() * s).flatten(-2))
    return out


def _glu(x, w13, w2):
    gate, up = _mm(x, w13).chunk(2, dim=-1)
    return _mm(gate * torch.sigmoid(gate) * up, w2)


def _uniform_exact(case, d):
    m, E = UNIFORM[case["model"]], UNIFORM[case["model"]]["experts"]
    new, cached, kvh = d["new"], d["cached"], m["kv_heads"]
    q8 = (lambda w: _e4m3(w)) if case["fp8"] else (lambda w: w)
    dense8 = q8 if not E else (lambda w: w)
    x = d["embed"][torch.tensor(sum(d["tokens"], []), device=DEV)].double()
    pos = torch.cat([torch.arange(c, c + n, device=DEV) for n, c in zip(new, cached)])
    pools = []
    for w, pool in zip(d["layers"], d["pools"]):
        pool = pool.double()
        h = _mm(_rms(x, m["eps"]) * w["attn_norm"].double(), dense8(w["wqkv"]))
        h = h if w["bqkv"] is None else h + w["bqkv"].double()
        q, k, v = h.unflatten(-1, (-1, HEAD)).split([m["heads"], kvh, kvh], dim=1)
        q, k = _rotate(q, pos, m["theta"]), _rotate(k, pos, m["theta"])
        outs, at = [], 0
        for n, c, table in zip(new, cached, d["tables"]):
            pages = torch.tensor(table, device=DEV)
            ctx = pool[pages].permute(1, 0, 3, 2, 4).flatten(1, 2)          # [2, tokens, kv heads, HEAD]
            ctx[0, c:c + n], ctx[1, c:c + n] = k[at:at + n], v[at:at + n]
            pool[pages] = ctx.unflatten(1, (-1, PAGE)).permute(1, 0, 3, 2, 4)
            outs.append(_attend(q[at:at + n], ctx[0, :c + n], ctx[1, :c + n], c))
            at += n
        pools.append(pool)
        x = x + _mm(torch.cat(outs).flatten(1), dense8(w["wo"]))
        h = _rms(x, m["eps"]) * w["ffn_norm"].double()
        if not E:
            x = x + _glu(h, q8(w["w13"]), q8(w["w2"]))
            continue
        top = _mm(h, w["router"]).topk(2, dim=-1)
        share = torch.softmax(top.values, dim=-1)
        for e in range(E):
            rows, slot = (top.indices == e).nonzero(as_tuple=True)
            if rows.numel():
                x = x.index_add(0, rows, share[rows, slot][:, None] * _glu(h[rows], q8(w["w13"][e]), q8(w["w2"][e])))
    last = torch.tensor(new, device=DEV).cumsum(0) - 1
    return {"logits": _mm(_rms(x[last], m["eps"]) * d["final_norm"].double(), d["head"]), "cache": pools, "states": []}


def _sikalorn_exact(d):
    """Whole sequences from position 0, side by side and padded: x [S, tokens, width]."""
    t, C, H, eps = {n: v for n, v in d["tensors"].items()}, SIK["width"], SIK["heads"], SIK["eps"]
    seqs = [b + n for b, n in zip(d["before"], d["tokens"])]
    S, N = len(seqs), max(map(len, seqs))
    ids = torch.zeros(S, N, dtype=torch.int64)
    for i, s in enumerate(seqs):
        ids[i, :len(s)] = torch.tensor(s)
    live = torch.arange(N, device=DEV)[None] < torch.tensor([len(s) for s in seqs], device=DEV)[:, None]
    W = lambda n: t[n].double()         # noqa: E731
    silu = lambda z: z * torch.sigmoid(z)       # noqa: E731
    unit = lambda z: z * torch.rsqrt(z.square().sum(-1, keepdim=True) + 1e-6)       # noqa: E731
    heads = lambda z, n: z.unflatten(-1, (n, -1))       # noqa: E731
    caches, states = [], []

    def conv(h, w, b=0.0):
        taps = w.shape[1]
        h = torch.nn.functional.pad(h, (0, 0, taps - 1, 0))
        return sum(w[:, j] * h[:, j:j + N] for j in range(taps)) + b

    def recur(q, k, v, decay, beta=None):
        """S <- decay S + k v^T, or with beta the delta rule, up to every sequence's end; outputs S^T q. q, k [S, N, heads, D], v [.., V]."""
        st = torch.zeros(S, v.shape[2], k.shape[3], v.shape[3], dtype=torch.float64, device=DEV)
        out = torch.empty(S, N, v.shape[2], v.shape[3], dtype=torch.float64, device=DEV)
        wide = lambda z: z.repeat_interleave(v.shape[2] // z.shape[1], dim=1)       # noqa: E731
        for i in range(N):
            on, kk, u = live[:, i, None], wide(k[:, i]), v[:, i]
            st = st * torch.where(on, decay[:, i], 1.0)[..., None, None]
            if beta is not None:
                u = beta[:, i, :, None] * (u - (kk[:, :, None] @ st).squeeze(2))
            st = torch.addcmul(st, (kk * on[..., None])[..., None], u[:, :, None])
            out[:, i] = (wide(q[:, i])[:, :, None] @ st).squeeze(2)
        states.append(st)
        return out

    def gates(p, z):
        return torch.exp(-torch.exp(W(p + "A_log")) * torch.nn.functional.softplus(z + W(p + "dt_bias")))

    def delta(h, p):
        q, k, v = (silu(conv(_mm(h, t[p + n]), W(p + n + ".conv"))) for n in ("q", "k", "v"))
        q, k, v = unit(heads(q, H // 2)) * HEAD ** -0.5, unit(heads(k, H // 2)), heads(v, H)
        o = recur(q, k, v, gates(p, _mm(h, t[p + "a"])), torch.sigmoid(_mm(h, t[p + "b"])))
        o = _rms(o, eps) * W(p + "norm") * silu(heads(_mm(h, t[p + "g"]), H))
        return _mm(o.flatten(2), t[p + "o"])

    def light(h, p):
        q, k, v = (heads(silu(_mm(h, t[p + n])), H) for n in ("q", "k", "v"))
        o = recur(q, k, v, torch.tensor(_light_decay(), dtype=torch.float64, device=DEV).expand(S, N, H))
        return _mm(_rms(o.flatten(2), eps) * W(p + "norm") * torch.sigmoid(_mm(h, t[p + "g"])), t[p + "o"])

    def window(h, p):
        pos, G = torch.arange(N, device=DEV), H // 4
        q, k, v = (_mm(h, t[p + n]) for n in ("q", "k", "v"))
        q, k = heads(_rms(q, eps) * W(p + "q.norm"), H), heads(_rms(k, eps) * W(p + "k.norm"), G)
        q, k = (torch.stack([_rotate(z, pos, SIK["theta"], SIK["factor"]) for z in y]) for y in (q, k))
        v = heads(v, G)
        pool = torch.zeros(d["pages"], 2, G, WINDOW_PAGE, HEAD, dtype=torch.float64, device=DEV)
        for i, (s, table) in enumerate(zip(seqs, d["tables"])):
            kv = torch.zeros(2, len(table) * WINDOW_PAGE, G, HEAD, dtype=torch.float64, device=DEV)
            kv[0, :len(s)], kv[1, :len(s)] = k[i, :len(s)], v[i, :len(s)]
            pool[torch.tensor(table, device=DEV)] = kv.unflatten(1, (-1, WINDOW_PAGE)).permute(1, 0, 3, 2, 4)
        caches.append(pool.flatten(1))
        return _mm(torch.stack([_attend(q[i], k[i], v[i], 0, SIK["window"]).flatten(1) for i in range(S)]), t[p + "o"])

    def space(h, p):
        inner = 2 * H * 64
        z, xbc, dt = _mm(h, t[p + "in"]).split([inner, inner + 2 * HEAD, 2 * H], dim=-1)
        xs, b, c = silu(conv(xbc, W(p + "conv"), W(p + "conv.b"))).split([inner, HEAD, HEAD], dim=-1)
        xs, step = heads(xs, 2 * H), torch.nn.functional.softplus(dt + W(p + "dt_bias"))
        y = recur(c[:, :, None], b[:, :, None], step[..., None] * xs, gates(p, dt)) + W(p + "D")[:, None] * xs
        return _mm(_rms(heads(y.flatten(2) * silu(z), 8), eps).flatten(2) * W(p + "norm"), t[p + "o"])

    def pair(h, p):
        return 0.7 * window(h, p + "left.") + 0.7 * space(h, p + "right.")

    norm = lambda x, n: torch.tanh(W(n + ".alpha") * x) * W(n) + W(n + ".b")        # noqa: E731
    x0 = x = t["embed"][ids.to(DEV)].double()
    mixers, (a, b, times) = (delta, pair, light, pair), SIK["loop"]
    for i, turn in [(i, None) for i in range(a)] + [(i, n) for n in range(times) for i in range(a, b)] + [(i, None) for i in range(b, 4)]:
        if turn is not None and i == a:
            x = _mm(torch.cat([x, x0], dim=-1), t["loop.in"]) + W("loop.step")[turn]
        h = norm(x, f"l{i}.norm1")
        x = x + mixers[i](h, f"l{i}.mix.") + _mm(torch.relu(_mm(h, t[f"l{i}.mlp.up"])).square(), t[f"l{i}.mlp.down"])
    last = torch.tensor([len(s) - 1 for s in seqs], device=DEV)
    return {"logits": _mm(norm(x[torch.arange(S, device=DEV), last], "final.norm"), t["head"]), "cache": caches, "states": states}
