"""The work that a user of this engine has it do, as cases that can be timed and compared.

A case is one pass through ``ModelRunner.step`` (what ``Engine`` and ``bin/trace_run`` drive): requests that are in the cache
get one token each (``cached``, their lengths before the step), new requests bring their prompts in the same step
(``prompts``), and ``steps`` more steps of one given token per request follow; the logits of every step come back.  A pass
leaves the state as it found it: cached requests are cut back, new ones closed.

The layer sizes are those of the headline benchmark (Qwen2.5-7B, 0.5B) and of the design benchmark; weights are random, as
a checkpoint of that shape would be loaded once, and tokens, uniform over the vocabulary, come from the seed.
"""
from __future__ import annotations

import math
import zlib

import torch

QWEN2 = {
    "7b": dict(layers=28, width=3584, heads=28, kv=4, dim=128, ff=18944, vocab=152064, tied=False),
    "0.5b": dict(layers=24, width=896, heads=14, kv=2, dim=64, ff=4864, vocab=151936, tied=True),
}
GOSITAR = {
    "s": dict(width=1024, heads=8, dim=64, rot=32, vdim=64, rank=256, experts=16, top=4, groups=4, keep=2, ff=512, shared=1024, dense=4096, vocab=32000),
    "m": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, rank=512, experts=32, top=4, groups=4, keep=2, ff=768, shared=1536, dense=6144, vocab=32000),
}
MEMORY = {                          # both designs with matrix memories
    "s": dict(width=1024, heads=4, kv=2, dim=128, mem_heads=8, mem_dim=64, mem_vdim=128, delta_kv=4, lat_heads=8, lat_dim=64, lat_rot=32, rank=256, ff=4096, vocab=32000),
    "m": dict(width=2048, heads=8, kv=2, dim=128, mem_heads=16, mem_dim=128, mem_vdim=128, delta_kv=8, lat_heads=16, lat_dim=128, lat_rot=64, rank=512, ff=6144, vocab=32000),
}
WINDOW, TAPS, LAYERS = 1024, 4, 4   # LAYERS: of the designs; Dukolorn's period is four


def listed():
    q = {"family": "qwen2", "dtype": "bfloat16", "cached": "", "prompts": "", "steps": 0}
    d = {"dtype": "bfloat16", "size": "m", "cached": "", "prompts": "", "steps": 0}
    return [
        # one chat on the smallest model: a token at a time, all launches and latency
        dict(q, name="0.5b one token", size="0.5b", cached="300"),
        # a full server of the small model: 64 conversations of 16 to 2,048 tokens
        dict(q, name="0.5b 64 tokens", size="0.5b", cached=spread(64, 16, 2047)),
        # continuous batching in between: three prompts arrive while 40 requests decode
        dict(q, name="0.5b mixed step", size="0.5b", cached=spread(40, 16, 2047), prompts="700,37,255"),
        # the 32-bit path: a question of odd length and the first words of its answer
        dict(q, name="0.5b float32", size="0.5b", dtype="float32", prompts="301", steps=4),
        # the headline: decoding at 4,096 tokens of context, one request and eight
        dict(q, name="7b one token", size="7b", cached="4095"),
        dict(q, name="7b 8 tokens", size="7b", cached=",".join(["4095"] * 8)),
        # the headline's other half: a whole prompt
        dict(q, name="7b prompt", size="7b", prompts="2048"),
        # latent attention, residual streams, routed experts: a whole prompt, and eight requests decoding
        dict(d, name="gositar prompt", family="gositar", prompts="2048"),
        dict(d, name="gositar 8 tokens", family="gositar", cached=spread(8, 700, 2047)),
        # memories with decays per channel, latent attention over a window: prompts of several requests, and short answers
        dict(d, name="dukolorn prompts", family="dukolorn", prompts="1201,37,500"),
        dict(d, name="dukolorn answers", family="dukolorn", prompts=spread(8, 20, 150), steps=24),
        # delta rule and gated matrix memory: a whole prompt of odd length
        dict(d, name="nuvarax prompt", family="nuvarax", prompts="2047"),
    ]


def spread(n, lo, hi):
    """n lengths from lo to hi, evenly over their logarithm."""
    return ",".join(str(round(lo * (hi / lo) ** (i / max(1, n - 1)))) for i in range(n))


def draw(rng):
    def length(lo, hi):
        return round(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    family = rng.choice(["qwen2", "qwen2", "gositar", "dukolorn", "nuvarax"])
    case = {"family": family, "dtype": "bfloat16", "cached": "", "prompts": "", "steps": 0}
    case["size"] = rng.choice(["0.5b", "0.5b", "7b"]) if family == "qwen2" else rng.choice(["s", "m"])
    if case["size"] == "0.5b" and rng.random() < 0.2:
        return dict(case, dtype="float32", prompts=str(length(16, 300)), steps=rng.randrange(4))
    most = 8 if case["size"] == "7b" else 64
    kind = rng.choice(["prompts", "answers"] if family in ("dukolorn", "nuvarax") else ["prompts", "tokens", "mixed"])
    if kind == "answers":
        n = length(1, 32)
        return dict(case, prompts=",".join(str(length(8, max(8, min(400, 1500 // n)))) for _ in range(n)), steps=rng.randrange(8, 25))
    if kind in ("tokens", "mixed"):
        case["cached"] = ",".join(str(length(16, 2000)) for _ in range(length(1, most)))
    if kind in ("prompts", "mixed"):
        room, lens = length(24, 1900), []
        while room >= 8 and len(lens) < 4:
            lens.append(rng.randrange(8, room + 1))
            room -= lens[-1]
        case["prompts"] = ",".join(map(str, lens))
    return case


# ---- configurations ------------------------------------------------------------------------------------------------------
def config_of(case):
    if case["family"] == "qwen2":
        z = QWEN2[case["size"]]
        return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": z["layers"], "hidden_size": z["width"],
                "num_attention_heads": z["heads"], "num_key_value_heads": z["kv"], "head_dim": z["dim"], "intermediate_size": z["ff"],
                "vocab_size": z["vocab"], "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": z["tied"],
                "use_sliding_window": False, "max_position_embeddings": 32768, "hidden_act": "silu"}
    if case["family"] == "gositar":
        z = GOSITAR[case["size"]]
        mix = {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot"], "vdim": z["vdim"], "kv_rank": z["rank"], "scale": (z["dim"] + z["rot"]) ** -0.5,
               "rot": {"base": 10000.0, "dims": z["rot"], "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        moe = {"kind": "moe", "expert": {"ff": z["ff"], "limit": 7.0}, "shared": {"ff": z["shared"], "limit": 7.0},
               "router": {"experts": z["experts"], "top": z["top"], "groups": {"count": z["groups"], "keep": z["keep"]}}}
        return {"architecture": "Gositar", "vocab": z["vocab"], "width": z["width"], "norm": {"eps": 1e-5}, "streams": 4,
                "layers": [{"type": ("latent_attention", "latent_attention_2")[i % 2], "mixer": mix,
                            "mlp": moe if i % 2 else {"kind": "dense", "ff": z["dense"]}} for i in range(LAYERS)]}
    z = MEMORY[case["size"]]
    delta = {"heads": z["mem_heads"], "kv_heads": z["delta_kv"], "dim": z["mem_dim"], "vdim": z["mem_vdim"], "conv": TAPS}
    left = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"], "scale": z["dim"] ** -0.5, "bias_max": 512}
    right = {"heads": z["mem_heads"], "dim": z["mem_dim"], "vdim": z["mem_vdim"]}
    if case["family"] == "nuvarax":
        mlp = {"kind": "dense", "ff": z["ff"], "limit": 7.0}
        return {"architecture": "Nuvarax", "vocab": z["vocab"], "width": z["width"], "max_positions": 4096, "norm": {"eps": 1e-5},
                "embedding": {"scale": 1.0, "bigram": {"buckets": 2 * z["vocab"] + 1, "mul_prev": 31, "mul_cur": 17}}, "canon": {"taps": 4},
                "layers": [{"type": "parallel", "mixer": {"left": left, "right": dict(right, gate_cap=15.0)}, "mlp": mlp} if i % 2 else
                           {"type": "delta", "mixer": delta, "mlp": mlp} for i in range(LAYERS)]}
    par = {"left": dict(left, softcap=30.0, q_temp={"coef": 0.1, "every": 1024}), "right": dict(right, tau=16.0), "left_scale": 0.9, "right_scale": 1.1}
    lat = {"heads": z["lat_heads"], "dim": z["lat_dim"], "rot_dim": z["lat_rot"], "vdim": z["lat_dim"], "kv_rank": z["rank"],
           "scale": (z["lat_dim"] + z["lat_rot"]) ** -0.5, "rot": {"base": 10000.0, "dims": z["lat_rot"]}, "mask": {"size": WINDOW}}
    kinds = [("channel_delta", delta), ("parallel", par), ("latent_attention", lat), ("parallel", par)]
    return {"architecture": "Dukolorn", "vocab": z["vocab"], "width": z["width"], "norm": {"eps": 1e-5}, "logit_scale": 0.5,
            "layers": [{"type": k, "mixer": m, "mlp": {"kind": "dense", "ff": z["ff"]}} for k, m in (kinds[i % 4] for i in range(LAYERS))]}


def tensor_of(decl, dtype, device):
    """Random weights with the spreads that trained ones have: matrices of a gain below one (N(0, 0.02) at the smallest width),
    norms near one, memories that last from tens to thousands of tokens, forget gates that mostly keep, routers whose first
    choices carry most of the weight."""
    g = torch.Generator(device=device)
    g.manual_seed(zlib.crc32(decl.name.encode()))
    shape, name = tuple(decl.shape), decl.name

    def normal(std):
        return torch.randn(shape, generator=g, dtype=torch.float32, device=device) * std

    def uniform(lo, hi):
        return torch.rand(shape, generator=g, dtype=torch.float32, device=device) * (hi - lo) + lo

    if name.endswith("A_log"):
        t = uniform(1.0, 16.0).log()
    elif name.endswith("dt_bias"):
        t = uniform(math.log(1e-3), math.log(1e-1)).exp().expm1().log()
    elif name.endswith(".right.f.b"):
        t = uniform(3.0, 6.0)
    elif name.endswith(".router"):
        t = normal(2.4 * shape[-1] ** -0.5)
    elif decl.init in ("ones", "zeros"):
        t = normal(0.1) + (1.0 if decl.init == "ones" else 0.0)
    elif decl.init == "eye":
        t = normal(0.05) + torch.eye(shape[0], device=device)
    elif decl.init == "conv":
        t = normal(shape[-1] ** -0.5)
    else:
        t = normal(0.6 * shape[-1] ** -0.5 if len(shape) > 1 else 0.02)
    return t.to(dtype)


_model = {}


def model_of(case, device="cuda"):
    """(model, its tensors by name), kept until another one is asked for, as a server keeps its model."""
    from infero_b200.models.decoder import DecoderModel
    from infero_b200.registry import resolve_architecture
    key = (case["family"], case["size"], case["dtype"], device)
    if key not in _model:
        _model.clear()
        config = config_of(case)
        arch = resolve_architecture(config)
        model = DecoderModel(arch.to_spec(arch.read_config(config)))
        tensors = {d.name: tensor_of(d, getattr(torch, case["dtype"]), device) for d in model.declare()}
        model.bind(dict(tensors))
        _model[key] = (model, tensors)
    return _model[key]


# ---- a pass --------------------------------------------------------------------------------------------------------------
def lengths(text):
    return [int(n) for n in text.split(",")] if text else []


def tokens_of(case, seed):
    """Per request its tokens in full: what is cached, then what the pass brings."""
    vocab = config_of(case).get("vocab") or config_of(case)["vocab_size"]
    g = torch.Generator().manual_seed(int(seed))
    return [torch.randint(vocab, (n,), generator=g).tolist()
            for n in [c + 1 + case["steps"] for c in lengths(case["cached"])] + [p + case["steps"] for p in lengths(case["prompts"])]]


def prepare(case, seed):
    from infero_b200.config import EngineConfig
    from infero_b200.engine import ModelRunner, StepEntry
    model, _ = model_of(case)
    cached, prompts, steps = lengths(case["cached"]), lengths(case["prompts"]), case["steps"]
    tokens = tokens_of(case, seed)
    need = [len(t) for t in tokens]
    budget = max(2048, len(cached) + sum(prompts))
    runner = ModelRunner(model, EngineConfig(dtype=case["dtype"], num_pages=sum(-(-n // 16) for n in need) + 1, max_seqs=len(need),
                                             ctx=max(need), max_batch_tokens=budget, max_logit_rows=max(8, len(need))))
    for i, n in enumerate(cached):
        runner.open(i)
        for at in range(0, n, 2048):
            runner.step([StepEntry(i, tokens[i][at:min(n, at + 2048)], [])])
    first = [StepEntry(i, tokens[i][n:n + 1], [0]) for i, n in enumerate(cached)]
    first += [StepEntry(len(cached) + j, tokens[len(cached) + j][:n], [n - 1]) for j, n in enumerate(prompts)]
    start = [n + 1 for n in cached] + prompts
    more = [[StepEntry(i, tokens[i][n + s:n + s + 1], [0]) for i, n in enumerate(start)] for s in range(steps)]
    logits = torch.empty((1 + steps, len(need), model.spec.vocab_size), dtype=torch.float32, device="cuda") if steps else None
    return {"runner": runner, "cached": cached, "new": range(len(cached), len(need)), "first": first, "more": more, "logits": logits}


def run(state):
    runner = state["runner"]
    for i, n in enumerate(state["cached"]):
        if runner.length(i) > n:
            runner.truncate(i, n)
    for i in state["new"]:
        runner.open(i)
    logits = runner.step(state["first"])
    if state["more"]:
        state["logits"][0].copy_(logits)
        for s, entries in enumerate(state["more"]):
            state["logits"][s + 1].copy_(runner.step(entries))      # (a captured step's logits are its graph's own buffer)
        logits = state["logits"]
    for i in state["new"]:
        runner.close(i)
    return logits


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------
def work(case):
    esize = 4 if case["dtype"] == "float32" else 2
    cached, prompts, steps = lengths(case["cached"]), lengths(case["prompts"]), case["steps"]
    rows = len(cached) + len(prompts)
    passes = [([c for c in cached] + [0] * len(prompts), [1] * len(cached) + prompts)]
    passes += [([c + 1 + s for c in cached] + [p + s for p in prompts], [1] * rows) for s in range(steps)]
    nbytes = flops = 0.0
    for before, new in passes:
        b, f = step_work(case, before, new, esize)
        nbytes, flops = nbytes + b, flops + f
    return {"bytes": nbytes, "flops": flops}


def step_work(case, before, new, esize):
    """One step: every weight it uses read once, the cached rows of its requests read, its own written, states read and
    written, logits written; products, causal attention (scores and values) and memories (decay, update, read-out)."""
    T, rows = sum(new), len(new)
    keys = sum(before) + T                                                  # cache rows read or written

    def pairs(window):                                                      # (query, key) pairs of an attention layer
        total = 0.0
        for b, n in zip(before, new):
            last = b + n
            total += sum(min(i + 1, window) for i in range(b, last)) if last > window else n * b + n * (n + 1) / 2
        return total

    def seen(window):
        return sum(min(b + n, window + n) for b, n in zip(before, new))

    if case["family"] == "qwen2":
        z = QWEN2[case["size"]]
        qo, kv = z["heads"] * z["dim"], z["kv"] * z["dim"]
        params = z["layers"] * (z["width"] * (2 * qo + 2 * kv + 3 * z["ff"]))
        cache = z["layers"] * 2.0 * kv * keys
        flops = 2.0 * params * T + z["layers"] * 4.0 * qo * pairs(1 << 40)
        width, vocab = z["width"], z["vocab"]
    elif case["family"] == "gositar":
        z = GOSITAR[case["size"]]
        width, vocab = z["width"], z["vocab"]
        H, row = z["heads"], z["rank"] + z["rot"]
        attn = width * (H * (z["dim"] + z["rot"]) + row) + H * z["rank"] * (z["dim"] + z["vdim"]) + H * z["vdim"] * width
        expert, shared = 3 * width * z["ff"], 3 * width * z["shared"]
        touched = z["experts"] * (1 - (1 - z["top"] / z["experts"]) ** T)       # of uniformly chosen experts
        half = LAYERS / 2
        params = LAYERS * attn + half * (2 * width * z["dense"] + shared + touched * expert + z["experts"] * width)
        flops = 2.0 * T * (LAYERS * attn + half * (2 * width * z["dense"] + shared + z["top"] * expert + z["experts"] * width))
        # (scores and values per head in the plain sizes or, for few queries a key, the latent's: the smaller one)
        flops += LAYERS * 2.0 * H * (z["dim"] + z["rot"] + z["vdim"]) * pairs(1 << 40)
        cache = LAYERS * 1.0 * row * keys
    else:
        z = MEMORY[case["size"]]
        width, vocab, M = z["width"], z["vocab"], z["mem_heads"]
        K, V, dk = z["mem_dim"], z["mem_vdim"], z["delta_kv"] * z["mem_dim"]
        mem, att = width * (2 * M * K + 3 * M * V), width * (2 * z["heads"] + 2 * z["kv"]) * z["dim"]
        delta, ff = width * (2 * dk + 3 * M * V), 3 * width * z["ff"]
        nuv = case["family"] == "nuvarax"
        n_delta, n_par = (2, 2) if nuv else (1, 2)
        lat_row, H = z["rank"] + z["lat_rot"], z["lat_heads"]
        lat = 0 if nuv else width * (H * (z["lat_dim"] + z["lat_rot"]) + lat_row) + 2 * H * z["rank"] * z["lat_dim"] + H * z["lat_dim"] * width
        params = n_delta * delta + n_par * (mem + att) + lat + LAYERS * ff
        flops = 2.0 * T * params + T * M * K * V * (n_delta * 8.0 + n_par * 5.0)
        flops += n_par * 4.0 * z["heads"] * z["dim"] * pairs(1 << 40)
        cache = n_par * 2.0 * z["kv"] * z["dim"] * keys
        if not nuv:
            flops += 2.0 * H * (2 * z["lat_dim"] + z["lat_rot"]) * pairs(WINDOW)
            cache += lat_row * seen(WINDOW)
        cache += 2.0 * (n_delta + n_par) * M * K * V * rows * 4 / esize          # (states are 32-bit)
    nbytes = esize * (params + cache + vocab * width + T * width) + 4.0 * rows * vocab
    return nbytes, flops + 2.0 * rows * vocab * width


def tolerance(case):
    """Against 64 bits a pass is off by 1.3e-6 to 3e-6 in 32 bits and by 0.004 to 0.011 in bf16."""
    return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 0.03}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------
def exact(case, seed, device="cuda"):
    cost = sum(step_work(case, [0], [n], 2)[1] for n in map(len, tokens_of(case, seed)))
    if cost > 1.5e14:
        return None
    _, w = model_of(case, device)
    forward = {"qwen2": qwen2_rows, "gositar": gositar_rows, "dukolorn": dukolorn_rows, "nuvarax": nuvarax_rows}[case["family"]]
    n = 1 + case["steps"]
    rows = [forward(config_of(case), Wide(w), torch.tensor(t, device=device), n) for t in tokens_of(case, seed)]
    return torch.stack(rows, 1) if n > 1 else torch.cat(rows)


class Wide:
    """The tensors in 64 bits, one at a time."""

    def __init__(self, tensors):
        self.t = tensors

    def __getitem__(self, name):
        return self.t[name].double()

    def get(self, name):
        return self[name] if name in self.t else None


def rms(x, eps, weight=None):
    x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return x if weight is None else x * weight


def silu(z):
    return z * torch.sigmoid(z)


def softplus(z):
    return torch.log1p(torch.exp(-z.abs())) + z.clamp(min=0.0)


def conv(x, taps):
    K = taps.shape[1]
    x = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    return sum(x[j:j + x.shape[0] - K + 1] * taps[:, j] for j in range(K))


def rotate(x, freqs, amp=1.0, adjacent=False):
    """x [T, ..., D]: pairs (i, i + n) or (2i, 2i + 1) of the first 2n coordinates turn by position * freqs[i]."""
    n = len(freqs)
    at = torch.arange(x.shape[0], device=x.device, dtype=x.dtype).view(-1, *[1] * (x.dim() - 1))
    angle = at * torch.tensor(freqs, device=x.device, dtype=x.dtype)
    c, s = angle.cos() * amp, angle.sin() * amp
    a, b = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if adjacent else (x[..., :n], x[..., n:2 * n])
    u, v = a * c - b * s, b * c + a * s
    turned = torch.stack([u, v], -1).flatten(-2) if adjacent else torch.cat([u, v], -1)
    return torch.cat([turned, x[..., 2 * n:]], -1)


def weights(scores, window=None, sink=None):
    """Causal softmax of one head's scores [T, T]."""
    i = torch.arange(scores.shape[0], device=scores.device)
    hidden = i[None] > i[:, None]
    if window:
        hidden = hidden | (i[:, None] - i[None] >= window)
    scores = scores.masked_fill(hidden, float("-inf"))
    if sink is not None:
        return torch.softmax(torch.cat([scores, sink.expand(len(i), 1)], 1), 1)[:, :-1]
    return torch.softmax(scores, 1)


def qwen2_rows(cfg, w, tokens, n):
    H, G, D, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    T = len(tokens)
    freqs = [cfg["rope_theta"] ** (-2.0 * i / D) for i in range(D // 2)]
    x = w.t["model.embed_tokens.weight"][tokens].double()
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = rms(x, eps, w[p + "input_layernorm.weight"])
        q, k, v = (h @ w[f"{p}self_attn.{c}_proj.weight"].T + w[f"{p}self_attn.{c}_proj.bias"] for c in "qkv")
        q, k, v = rotate(q.view(T, H, D), freqs), rotate(k.view(T, G, D), freqs), v.view(T, G, D)
        o = torch.stack([weights(q[:, a] @ k[:, a * G // H].T * D ** -0.5) @ v[:, a * G // H] for a in range(H)], 1)
        x = x + o.reshape(T, H * D) @ w[p + "self_attn.o_proj.weight"].T
        h = rms(x, eps, w[p + "post_attention_layernorm.weight"])
        x = x + (silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    head = w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]
    return rms(x[-n:], eps, w["model.norm.weight"]) @ head.T


def latent(h, w, p, m, eps, freqs, amp, adjacent, window=None):
    T, H, D, C = len(h), m["heads"], m["dim"], m["kv_rank"]
    q, down = (h @ w[p + ".q"].T).view(T, H, -1), h @ w[p + ".dkv"].T
    c = rms(down[:, :C], eps, w[p + ".dkv.norm"])
    q = torch.cat([q[..., :D], rotate(q[..., D:], freqs, amp, adjacent)], -1)
    turned = rotate(down[:, C:], freqs, amp, adjacent)
    k, v, sink = (c @ w[p + ".uk"].T).view(T, H, D), (c @ w[p + ".uv"].T).view(T, H, -1), w.get(p + ".sink")
    return torch.stack([weights(q[:, a] @ torch.cat([k[:, a], turned], 1).T * m["scale"], window, None if sink is None else sink[a]) @ v[:, a]
                        for a in range(H)], 1)


def gositar_rows(cfg, w, tokens, n):
    eps, r = cfg["norm"]["eps"], cfg["layers"][0]["mixer"]["rot"]
    dims, sc = r["dims"], r["scaling"]

    def norm(x, name):
        x = x - x.mean(-1, keepdim=True)
        return rms(x, eps, w[name])

    def turns(t):
        return dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(r["base"]))

    lo, hi = max(math.floor(turns(sc["fast"])), 0), min(math.ceil(turns(sc["slow"])), dims - 1)
    freqs = []
    for i in range(dims // 2):
        f, ramp = r["base"] ** (-2.0 * i / dims), min(1.0, max(0.0, (i - lo) / max(hi - lo, 0.001)))
        freqs.append(f / sc["factor"] * ramp + f * (1 - ramp))
    amp = 0.1 * math.log(sc["factor"]) + 1.0

    def glu(h, p, limit):
        g, u = (h @ w[p + ".gate"].T).clamp(max=limit), (h @ w[p + ".up"].T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[p + ".down"].T

    def feed_forward(h, p, ml):
        if ml["kind"] == "dense":
            return torch.relu(h @ w[p + ".up"].T).square() @ w[p + ".down"].T
        E, top, groups = ml["router"]["experts"], ml["router"]["top"], ml["router"]["groups"]
        s = torch.softmax(h @ w[p + ".router"].T, -1)
        pick = s + w[p + ".correction"]
        best = pick.view(len(h), groups["count"], -1).amax(-1)
        kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(groups["keep"], 1).indices, True)
        at = pick.masked_fill(~kept.repeat_interleave(E // groups["count"], 1), float("-inf")).topk(top, 1).indices
        share = s.gather(1, at)
        share = share / share.sum(1, keepdim=True)
        y = glu(h, p + ".shared", ml["shared"]["limit"])
        for e in range(E):
            t, c = (at == e).nonzero(as_tuple=True)
            y.index_add_(0, t, share[t, c, None] * glu(h[t], f"{p}.e{e}", ml["expert"]["limit"]))
        return y

    def sublayer(xs, p, hc, name, fn):
        y = fn(norm(torch.einsum("s,std->td", w[f"{p}.{hc}.in"], xs), p + name))
        return torch.einsum("sr,std->rtd", w[f"{p}.{hc}.mix"], xs) + w[f"{p}.{hc}.out"].view(-1, 1, 1) * y

    xs = w.t["embed"][tokens].double().repeat(cfg["streams"], 1, 1)
    for i, L in enumerate(cfg["layers"]):
        p, first = f"l{i}", L["type"] == "latent_attention"

        def mixer(h):
            o = latent(h, w, p + ".mix", L["mixer"], eps, freqs, amp, first)
            if first:
                o = o * torch.sigmoid(h @ w[p + ".mix.g"].T).unsqueeze(-1)
            return o.reshape(len(h), -1) @ w[p + ".mix.o"].T

        xs = sublayer(xs, p, "hc1", ".norm1", mixer)
        xs = sublayer(xs, p, "hc2", ".norm2", lambda h: feed_forward(h, p + ".mlp", L["mlp"]))
    return norm(xs[:, -n:].sum(0), "final.norm") @ w["head"].T


def by_distance(rel, T, most):
    """A learned bias per distance, in buckets that widen with their logarithm, [T, heads]."""
    B = rel.shape[0]
    half = B // 2
    rows = [d if d < half else min(B - 1, half + math.floor(math.log(d / half) / math.log(most / half) * (B - half))) for d in range(T)]
    return rel[torch.tensor(rows, device=rel.device)]


def biased_scores(q, k, a, m, rel):
    """Head a's scores [T, T] without and the bias by distance of each."""
    i = torch.arange(len(q), device=q.device)
    return q[:, a] @ k[:, a * k.shape[1] // q.shape[1]].T * m["scale"], rel[:, a][(i[:, None] - i[None]).clamp(min=0)]


def delta_inputs(h, w, p, m):
    T, H, G, K = len(h), m["heads"], m["kv_heads"], m["dim"]
    q, k, v = (silu(conv(h @ w[f"{p}.{c}"].T, w[f"{p}.{c}.conv"])) for c in "qkv")
    q, k = (c.view(T, G, K) for c in (q, k))
    q, k = (c * torch.rsqrt(c.square().sum(-1, keepdim=True) + 1e-6) for c in (q, k))
    q, k = (q * K ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    return q, k, v.view(T, H, -1), torch.sigmoid(h @ w[p + ".b"].T)


def walk(q, k, v, g, beta=None, put=None):
    """Memories S [H, K, V] over time: rows decay by g [T, H, K or 1]; a delta rule with steps beta, else k v^T times put."""
    T, H, K = q.shape
    S, out = q.new_zeros(H, K, v.shape[2]), torch.empty_like(v)
    for t in range(T):
        S *= g[t].unsqueeze(2)
        if beta is not None:
            u = beta[t, :, None] * (v[t] - torch.bmm(k[t].unsqueeze(1), S)[:, 0])
        else:
            u = v[t] if put is None else v[t] * put[t, :, None]
        S.baddbmm_(k[t].unsqueeze(2), u.unsqueeze(1))
        out[t] = torch.bmm(q[t].unsqueeze(1), S)[:, 0]
    return out


def dukolorn_rows(cfg, w, tokens, n):
    eps, T = cfg["norm"]["eps"], len(tokens)

    def norm(x, name):
        return rms(x, eps, 1.0 + w[name])

    def narrow(h, p, a, b):
        return (h @ w[f"{p}.{a}"].T) @ w[f"{p}.{b}"].T

    def channel_delta(h, p, m):
        q, k, v, beta = delta_inputs(h, w, p, m)
        step = softplus(narrow(h, p, "a1", "a2") + w[p + ".dt_bias"]).view(T, m["heads"], -1)
        o = walk(q, k, v, torch.exp(-torch.exp(w[p + ".A_log"]).view(1, -1, 1) * step), beta)
        return ((rms(o, eps) * w[p + ".norm"]).reshape(T, -1) * torch.sigmoid(narrow(h, p, "g1", "g2"))) @ w[p + ".o"].T

    def left(h, p, m):
        q = rms(h @ w[p + ".q"].T, eps, w[p + ".q.norm"]).view(T, m["heads"], -1)
        k = rms(h @ w[p + ".k"].T, eps, w[p + ".k.norm"]).view(T, m["kv_heads"], -1)
        v, at, t = (h @ w[p + ".v"].T).view(T, m["kv_heads"], -1), torch.arange(T, device=h.device).double(), m["q_temp"]
        q = q * (1.0 + t["coef"] * torch.log(torch.floor((at + 1) / t["every"]) + 1)).view(T, 1, 1)
        rel, sink, o = by_distance(w[p + ".rel"], T, m["bias_max"]), w[p + ".sink"], []
        for a in range(m["heads"]):
            s, bias = biased_scores(q, k, a, m, rel)
            o.append(weights(m["softcap"] * torch.tanh(s / m["softcap"]) + bias, None, sink[a]) @ v[:, a * m["kv_heads"] // m["heads"]])
        return torch.stack(o, 1).reshape(T, -1) @ w[p + ".o"].T

    def right(h, p, m):
        q, k, v = ((h @ w[f"{p}.{c}"].T).view(T, m["heads"], -1) for c in "qkv")
        decay = (torch.sigmoid(narrow(h, p, "a1", "a2") + w[p + ".a2.b"]) ** (1.0 / m["tau"])).view(T, m["heads"], -1)
        o = rms(walk(q * m["dim"] ** -0.5, k, v, decay), eps) * w[p + ".norm"]
        return (o.reshape(T, -1) * silu(h @ w[p + ".g"].T)) @ w[p + ".o"].T

    def window(h, p, m):
        freqs = [m["rot"]["base"] ** (-2.0 * i / m["rot"]["dims"]) for i in range(m["rot"]["dims"] // 2)]
        return latent(h, w, p, m, eps, freqs, 1.0, True, m["mask"]["size"]).reshape(T, -1) @ w[p + ".o"].T

    x = rms(w.t["embed"][tokens].double(), eps, 1.0 + w["embed.norm"])
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}", L["mixer"]
        if L["type"] == "parallel":
            y = m["left_scale"] * left(x, p + ".mix.left", m["left"]) + m["right_scale"] * right(x, p + ".mix.right", m["right"])
        else:
            y = {"channel_delta": channel_delta, "latent_attention": window}[L["type"]](x, p + ".mix", m)
        x = x + norm(y, p + ".norm1")
        g, u = (x @ w[f"{p}.mlp.{c}"].T + w[f"{p}.mlp.{c}.b"] for c in ("gate", "up"))
        x = x + norm((silu(g) * u) @ w[p + ".mlp.down"].T + w[p + ".mlp.down.b"], p + ".norm2")
    return norm(x[-n:], "final.norm") @ w["head"].T * cfg["logit_scale"]


def nuvarax_rows(cfg, w, tokens, n):
    eps, T = cfg["norm"]["eps"], len(tokens)

    def norm(x, name):
        return rms(x, eps, 1.0 + w[name])

    def delta(h, p, m):
        q, k, v, beta = delta_inputs(h, w, p, m)
        g = torch.exp(-torch.exp(w[p + ".A_log"]) * softplus(h @ w[p + ".a"].T + w[p + ".dt_bias"]))
        o = rms(walk(q, k, v, g.unsqueeze(2), beta), eps) * w[p + ".norm"]
        return (o.reshape(T, -1) * silu(h @ w[p + ".g"].T)) @ w[p + ".o"].T

    def left(h, p, m):
        q, k, v = ((h @ w[f"{p}.{c}"].T + w[f"{p}.{c}.b"]).view(T, -1, m["dim"]) for c in "qkv")
        rel = by_distance(w[p + ".rel"], T, m["bias_max"])
        maps = torch.stack([weights(sum(biased_scores(q, k, a, m, rel))) for a in range(m["heads"])])
        talk = w[p + ".talk"]
        o = torch.stack([(talk[a].view(-1, 1, 1) * maps).sum(0) @ v[:, a * m["kv_heads"] // m["heads"]] for a in range(m["heads"])], 1)
        return (o.reshape(T, -1) * torch.sigmoid(h @ w[p + ".g"].T)) @ w[p + ".o"].T + w[p + ".o.b"]

    def right(h, p, m):
        H, cap = m["heads"], m["gate_cap"]
        q, k, v = ((h @ w[f"{p}.{c}"].T).view(T, H, -1) for c in "qkv")
        i = cap * torch.tanh((h @ w[p + ".i"].T + w[p + ".i.b"]) / cap)
        f = -softplus(-cap * torch.tanh((h @ w[p + ".f"].T + w[p + ".f.b"]) / cap))
        most, keep, put = [q.new_zeros(H)], [], []
        for t in range(T):
            most.append(torch.maximum(f[t] + most[-1], i[t]))
            keep.append(torch.exp(f[t] + most[-2] - most[-1]))
            put.append(torch.exp(i[t] - most[-1]))
        v = torch.cat([v, v.new_ones(T, H, 1)], 2)                        # (the last column: what divides)
        o = walk(q * m["dim"] ** -0.5, k, v, torch.stack(keep).unsqueeze(2), None, torch.stack(put))
        o = o[..., :-1] / (torch.maximum(o[..., -1].abs(), torch.exp(-torch.stack(most[1:]))) + 1e-6).unsqueeze(2)
        return (rms(o, eps).reshape(T, -1) * w[p + ".norm"] * torch.sigmoid(h @ w[p + ".g"].T)) @ w[p + ".o"].T

    b, t = cfg["embedding"]["bigram"], tokens
    pair = torch.cat([t.new_tensor([b["buckets"]]), (t[:-1] * b["mul_prev"] + t[1:] * b["mul_cur"]) % b["buckets"]])
    x = (w.t["embed"][t].double() * cfg["embedding"]["scale"] + w.t["bigram"][pair].double() + w.t["pos"][:T].double())
    for i, L in enumerate(cfg["layers"]):
        p, m, limit = f"l{i}", L["mixer"], L["mlp"]["limit"]
        h = norm(x, p + ".norm1")
        h = h + conv(h, w[p + ".canon1"])
        if L["type"] == "delta":
            y = delta(h, p + ".mix", m)
        else:
            y = 0.5 * (rms(left(h, p + ".mix.left", m["left"]), eps) * w[p + ".mix.left.out"]
                       + rms(right(h, p + ".mix.right", m["right"]), eps) * w[p + ".mix.right.out"])
        x = x + norm(y, p + ".norm1b")
        h = norm(x, p + ".norm2")
        g, u = (h @ w[p + ".mlp.gate"].T).clamp(max=limit), (h @ w[p + ".mlp.up"].T).clamp(-limit, limit)
        x = x + norm((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[p + ".mlp.down"].T, p + ".norm2b")
    return norm(x[-n:], "final.norm") @ w["embed"].T
