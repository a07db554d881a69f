"""What is timed of this engine, and how its results are checked: single passes through the entry points that serving
runs on, at the layer sizes `bench.py` measures, with random weights.

A case is one of
  decode   one step that brings one token for each of `batch` live requests (ModelRunner.step); every pass decodes one
           token more, and a request that has reached the model's last position starts over with its prompt
  prefill  one prompt of `tokens` tokens as one step, the logits of its last token wanted; the request ends afterwards
  mixed    one step of `batch` decoding requests beside a portion of `tokens` prompt tokens, which the scheduler makes
           whenever a prompt arrives while others decode
  sample   the choice of one token for each of `batch` rows of logits (Sampler.launch)
The live requests of a decode or mixed case have contexts of their own, up to a fifth shorter than `context`."""
import math

import torch

from tiny_llm_b200.config import config_from_dict
from tiny_llm_b200.engine import StepEntry, make_runner
from tiny_llm_b200.parts import DecoderModel
from tiny_llm_b200.sampling import Sampler, SamplingParams
from tiny_llm_b200.weights import load_state

DEVICE = "cuda:0"
PAGE = 16
MAX_STEP = 4096     # tokens in one step, the largest prompt of the cases included

_TINYLLAMA = dict(architectures=["LlamaForCausalLM"], model_type="llama", hidden_size=2048, num_attention_heads=32,
                  num_key_value_heads=4, intermediate_size=5632, vocab_size=32000, rope_theta=10000.0, rms_norm_eps=1e-5,
                  max_position_embeddings=2048, tie_word_embeddings=False, hidden_act="silu", initializer_range=0.02,
                  torch_dtype="bfloat16")
_LLAMA = {
    "tinyllama": _TINYLLAMA,
    "llama2_7b": dict(_TINYLLAMA, hidden_size=4096, num_key_value_heads=32, intermediate_size=11008,
                      max_position_embeddings=4096),
    "llama3_8b": dict(_TINYLLAMA, hidden_size=4096, num_key_value_heads=8, intermediate_size=14336, vocab_size=128256,
                      rope_theta=500000.0, max_position_embeddings=8192),
}


def _gevovik(layers):
    dense, rot = {"kind": "dense", "ff": 5632}, {"dims": 64, "base": 10000.0}
    latent = {"heads": 16, "dim": 64, "rot_dim": 64, "vdim": 128, "kv_rank": 192, "scale": 128 ** -0.5, "rot": rot}
    mamba = {"heads": 32, "vdim": 128, "state": 128, "groups": 4, "norm_groups": 4, "conv": 4}
    stretched = {"dims": 128, "base": 10000.0, "scaling": {"factor": 8.0, "original": 4096, "fast": 16.0, "slow": 2.0}}
    par = {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                    "rot": stretched},
           "right": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}, "left_scale": 0.5, "right_scale": 1.0}
    kinds = [lambda i: {"type": "latent_attention", "mixer": latent, "mlp": dense},
             lambda i: {"type": "mamba2", "mixer": mamba, "mlp": dense},
             lambda i: {"type": "parallel", "mixer": par, "mlp": dense},
             lambda i: {"type": "latent_attention", "mixer": dict(latent, kv_from=i - 3), "mlp": dense}]
    return {"architecture": "Gevovik", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "initializer_range": 0.02,
            "embedding": {"scale": 2048 ** 0.5, "bigram": {"buckets": 65521, "mul_prev": 1000003, "mul_cur": 40009}},
            "layers": [kinds[i % 4](i) for i in range(layers)]}


def _config(case):
    if case["model"] == "gevovik":
        return _gevovik(case["layers"])
    return dict(_LLAMA[case["model"]], num_hidden_layers=case["layers"])


# ---------------------------------------------------------------------------------------------- the cases

def listed():
    bf, f32 = "bfloat16", "float32"
    return [
        # the choice of the next tokens of a full batch with the default options of generation: once in every step
        {"name": "sample_b64", "kind": "sample", "batch": 64, "vocab": 32000, "temperature": 0.7, "top_k": 50, "top_p": 0.95},
        # one chat at a time: nothing but latency
        {"name": "tinyllama_decode_b1", "kind": "decode", "model": "tinyllama", "layers": 22, "dtype": bf, "batch": 1,
         "context": 300},
        # a small server, prompts of a page or two
        {"name": "tinyllama_decode_b8", "kind": "decode", "model": "tinyllama", "layers": 22, "dtype": bf, "batch": 8,
         "context": 1400},
        # a full server: as many requests as the runner takes by default
        {"name": "tinyllama_decode_b64", "kind": "decode", "model": "tinyllama", "layers": 22, "dtype": bf, "batch": 64,
         "context": 1300},
        # a larger model over long documents (8 of its 32 layers, so that the weights are quickly made)
        {"name": "llama3_8b_decode_b16", "kind": "decode", "model": "llama3_8b", "layers": 8, "dtype": bf, "batch": 16,
         "context": 5600},
        # a question of some lines
        {"name": "tinyllama_prefill_131", "kind": "prefill", "model": "tinyllama", "layers": 22, "dtype": bf, "tokens": 131},
        # a prompt as long as the model allows
        {"name": "tinyllama_prefill_2048", "kind": "prefill", "model": "tinyllama", "layers": 22, "dtype": bf,
         "tokens": 2048},
        # a long document into a model whose heads all have keys of their own (8 of its 32 layers)
        {"name": "llama2_7b_prefill_3001", "kind": "prefill", "model": "llama2_7b", "layers": 8, "dtype": bf,
         "tokens": 3001},
        # a prompt that arrives while others decode
        {"name": "tinyllama_mixed", "kind": "mixed", "model": "tinyllama", "layers": 22, "dtype": bf, "batch": 16,
         "context": 1400, "tokens": 487},
        # the 32-bit path, which results are checked against: decoding and a prompt
        {"name": "tinyllama_f32_decode_b8", "kind": "decode", "model": "tinyllama", "layers": 22, "dtype": f32, "batch": 8,
         "context": 700},
        {"name": "tinyllama_f32_prefill_509", "kind": "prefill", "model": "tinyllama", "layers": 22, "dtype": f32,
         "tokens": 509},
        # a prompt of a design that mixes recurrences with latent and windowed attention
        {"name": "gevovik_prefill_1777", "kind": "prefill", "model": "gevovik", "layers": 8, "dtype": bf, "tokens": 1777},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sample", "decode", "decode", "decode", "long", "prefill", "prefill", "mha", "mixed", "f32decode",
                       "f32prefill", "gevovik"])
    bf, f32 = "bfloat16", "float32"
    llama = {"model": "tinyllama", "layers": 22, "dtype": bf}
    if kind == "sample":
        return {"kind": "sample", "batch": _log(rng, 1, 64), "vocab": rng.choice([32000, _log(rng, 1000, 32000)]),
                "temperature": round(rng.uniform(0.3, 1.2), 2), "top_k": rng.choice([0, 1, 20, 50, 100]),
                "top_p": round(rng.uniform(0.7, 1.0), 2)}
    if kind == "decode":
        batch = _log(rng, 1, 64)
        return {"kind": "decode", **llama, "batch": batch, "context": _log(rng, 40, 1400 if batch < 60 else 1300)}
    if kind == "long":
        return {"kind": "decode", "model": "llama3_8b", "layers": 8, "dtype": bf, "batch": _log(rng, 1, 16),
                "context": _log(rng, 400, 5600)}
    if kind == "prefill":
        return {"kind": "prefill", **llama, "tokens": _log(rng, 17, 2048)}
    if kind == "mha":
        return {"kind": "prefill", "model": "llama2_7b", "layers": 8, "dtype": bf, "tokens": _log(rng, 60, 3001)}
    if kind == "mixed":
        return {"kind": "mixed", **llama, "batch": _log(rng, 2, 16), "context": _log(rng, 100, 1400), "tokens": _log(rng, 20, 487)}
    if kind == "f32decode":
        return {"kind": "decode", **dict(llama, dtype=f32), "batch": _log(rng, 1, 8), "context": _log(rng, 40, 700)}
    if kind == "f32prefill":
        return {"kind": "prefill", **dict(llama, dtype=f32), "tokens": _log(rng, 17, 509)}
    return {"kind": "prefill", "model": "gevovik", "layers": 8, "dtype": bf, "tokens": _log(rng, 60, 1777)}


# ---------------------------------------------------------------------------------------------- inputs from the seed

def _tensors(case):
    """Name -> (shape, how it is drawn) of every weight of the model."""
    cfg, out = _config(case), {}
    normal, unit = ("normal", 0.02), ("uniform", 0.5, 1.5)
    if case["model"] != "gevovik":
        h, ff, v = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
        hd = h // cfg["num_attention_heads"]
        kv = cfg["num_key_value_heads"] * hd
        out["model.embed_tokens.weight"] = ((v, h), normal)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out[p + "input_layernorm.weight"] = out[p + "post_attention_layernorm.weight"] = ((h,), unit)
            for n, shape in (("q", (h, h)), ("k", (kv, h)), ("v", (kv, h)), ("o", (h, h))):
                out[p + f"self_attn.{n}_proj.weight"] = (shape, normal)
            for n, shape in (("gate", (ff, h)), ("up", (ff, h)), ("down", (h, ff))):
                out[p + f"mlp.{n}_proj.weight"] = (shape, normal)
        out["model.norm.weight"] = ((h,), unit)
        out["lm_head.weight"] = ((v, h), normal)
        return out
    h, v = cfg["width"], cfg["vocab"]
    out.update({"embed": ((v, h), normal), "bigram": ((cfg["embedding"]["bigram"]["buckets"] + 1, h), normal),
                "head": ((v, h), normal), "final.norm": ((), unit)})
    rank = 12      # of the low-rank projections for decays and gate
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        ff = layer["mlp"]["ff"]
        out.update({f"l{i}.norm1": ((), unit), f"l{i}.norm2": ((), unit), f"l{i}.mlp.up": ((ff, h), normal),
                    f"l{i}.mlp.down": ((h, ff), normal)})
        if layer["type"] == "latent_attention":
            n, r = m["heads"], m["kv_rank"]
            out.update({p + "q": ((n * (m["dim"] + m["rot_dim"]), h), normal), p + "uk": ((n * m["dim"], r), normal),
                        p + "uv": ((n * m["vdim"], r), normal), p + "o": ((h, n * m["vdim"]), normal),
                        p + "sink": ((n,), ("normal", 1.0))})
            if "kv_from" not in m:
                out.update({p + "dkv": ((r + m["rot_dim"], h), normal), p + "dkv.norm": ((r,), unit)})
        elif layer["type"] == "mamba2":
            n, inner, bc = m["heads"], m["heads"] * m["vdim"], 2 * m["groups"] * m["state"]
            out.update({p + "in": ((2 * inner + bc + n, h), normal), p + "conv": ((inner + bc, m["conv"]), ("normal", 0.5)),
                        p + "conv.b": ((inner + bc,), ("normal", 0.2)), p + "dt_bias": ((n,), ("normal", 1.0)),
                        p + "A_log": ((n,), ("uniform", -3.0, 0.5)), p + "D": ((n,), ("normal", 1.0)),
                        p + "norm": ((inner,), unit), p + "o": ((h, inner), normal)})
        else:
            a, b = m["left"], m["right"]
            nq, nk = a["heads"] * a["dim"], a["kv_heads"] * a["dim"]
            out.update({p + "left.q": ((nq, h), normal), p + "left.k": ((nk, h), normal),
                        p + "left.v": ((a["kv_heads"] * a["vdim"], h), normal), p + "left.o": ((h, a["heads"] * a["vdim"]), normal),
                        p + "left.q.norm": ((a["dim"],), unit), p + "left.k.norm": ((a["dim"],), unit),
                        p + "left.g": ((a["heads"], h), normal), p + "left.temp": ((a["heads"],), ("uniform", 0.6, 1.6)),
                        p + "left.talk": ((a["heads"], a["heads"]), ("normal", 0.4))})
            qk, vd = b["kv_heads"] * b["dim"], b["heads"] * b["vdim"]
            for n, size in (("q", qk), ("k", qk), ("v", vd)):
                out[p + f"right.{n}"] = ((size, h), normal)
                out[p + f"right.{n}.conv"] = ((size, b["conv"]), ("normal", 0.5))
            out.update({p + "right.b": ((b["heads"], h), normal), p + "right.A_log": ((b["heads"],), ("uniform", -3.0, 0.5)),
                        p + "right.norm": ((b["vdim"],), unit), p + "right.o": ((h, vd), normal),
                        p + "right.a1": ((rank, h), normal), p + "right.a2": ((b["heads"] * b["dim"], rank), ("normal", 0.5)),
                        p + "right.dt_bias": ((b["heads"] * b["dim"],), ("normal", 1.0)),
                        p + "right.g1": ((rank, h), normal), p + "right.g2": ((vd, rank), ("normal", 0.5))})
    return out


def _weights(case, seed):
    """Every weight in the case's type, drawn on the GPU in the order of the names."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = getattr(torch, case["dtype"])
    out = {}
    for name, (shape, how) in sorted(_tensors(case).items()):
        t = torch.empty(shape, dtype=torch.float32, device=DEVICE)
        t = t.normal_(0.0, how[1], generator=g) if how[0] == "normal" else t.uniform_(how[1], how[2], generator=g)
        out[name] = t.to(dtype)
    return out


def _vocab(case):
    cfg = _config(case)
    return cfg["vocab"] if case["model"] == "gevovik" else cfg["vocab_size"]


def _contexts(case):
    """Tokens that each live request holds before the first pass."""
    if "context" not in case:
        return []
    return [max(1, case["context"] - (37 * i) % max(1, case["context"] // 5)) for i in range(case["batch"])]


def _token_lists(case, seed):
    """(the live requests' prompts, the tokens they are fed pass by pass, the prompt of this pass)."""
    g = torch.Generator().manual_seed(seed + 1)

    def ids(n):
        return torch.randint(0, _vocab(case), (n,), generator=g).tolist()
    held = [ids(n) for n in _contexts(case)]
    return held, [ids(64) for _ in held], ids(case.get("tokens", 0))


def _logits(case, seed):
    """Rows as a trained model gives them: most ids far below a handful of likely ones."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    return torch.randn(case["batch"], case["vocab"], generator=g, device=DEVICE) * 2.5


# ---------------------------------------------------------------------------------------------- one pass

def prepare(case, seed):
    if case["kind"] == "sample":
        n = case["batch"]
        params = [SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=seed + i)
                  for i in range(n)]
        return {"kind": "sample", "sampler": Sampler(DEVICE, case["vocab"], max_rows=max(2, n + n % 2)),
                "logits": _logits(case, seed), "params": params, "counters": [17 * i % 256 for i in range(n)]}
    config = config_from_dict(_config(case))
    model = DecoderModel(config.model_spec())
    dtype = getattr(torch, case["dtype"])
    model.load(load_state(model.weight_specs(), _weights(case, seed), dtype, DEVICE))
    held, feed, prompt = _token_lists(case, seed)
    limit = min(model.spec.max_positions, 8192)
    runner = make_runner(model, dtype, DEVICE, max_tokens=max(1, len(held)) * limit + (len(prompt) if held else 0),
                         page_size=PAGE, max_requests=len(held) + 1, max_tokens_per_step=MAX_STEP, max_positions=limit)
    state = {"kind": case["kind"], "runner": runner, "held": held, "feed": feed, "prompt": prompt, "limit": limit, "passes": 0}
    for rid in range(len(held)):
        _start(state, rid)
    return state


def _start(state, rid):
    """The request's prompt into the cache, in portions as large as a step takes."""
    runner, prompt = state["runner"], state["held"][rid]
    runner.cache.add_request(rid)
    for lo in range(0, len(prompt), MAX_STEP):
        runner.step([StepEntry(rid, prompt[lo: lo + MAX_STEP], [])])


def run(state):
    if state["kind"] == "sample":
        return state["sampler"].launch(state["logits"], state["params"], state["counters"]).device_out
    runner, prompt, entries = state["runner"], state["prompt"], []
    for rid, feed in enumerate(state["feed"]):
        if runner.cache.kv_len[rid] >= state["limit"]:
            runner.cache.free_request(rid)
            _start(state, rid)
        entries.append(StepEntry(rid, [feed[state["passes"] % len(feed)]], [0]))
    state["passes"] += 1
    if prompt:
        runner.cache.add_request("prompt")
        entries.append(StepEntry("prompt", prompt, [len(prompt) - 1]))
    logits = runner.step(entries)
    if prompt:
        runner.cache.free_request("prompt")
    return logits


# ---------------------------------------------------------------------------------------------- what a pass needs

def work(case):
    if case["kind"] == "sample":      # every logit read once; an exponential and a few comparisons each
        n = case["batch"] * case["vocab"]
        return {"bytes": 4.0 * n, "flops": 8.0 * n}
    cfg = _config(case)
    size = 4 if case["dtype"] == "float32" else 2
    gathered = ("model.embed_tokens.weight", "embed", "bigram")
    matrices = {n: s for n, (s, _) in _tensors(case).items() if n not in gathered}
    head = _vocab(case) * (cfg["width"] if case["model"] == "gevovik" else cfg["hidden_size"])
    params = float(sum(math.prod(s) for s in matrices.values()))
    contexts = _contexts(case)
    new, wanted = len(contexts) + case.get("tokens", 0), len(contexts) + (1 if case.get("tokens") else 0)
    t = case.get("tokens", 0)
    flops = 2.0 * new * (params - head) + 2.0 * wanted * head
    read = params * size + 4.0 * wanted * _vocab(case)
    if case["model"] == "gevovik":
        flops += case["layers"] // 4 * (
            2 * 2.0 * 16 * t * t / 2 * (64 + 64 + 128)                     # latent attention, keys and values per head
            + 2.0 * 16 * min(t, 1024) * max(t - min(t, 1024) / 2, 1) * 272  # windowed attention, scores mixed
            + 16 * 9.0 * t * 128 * 128 + 32 * 6.0 * t * 128 * 128)         # the two recurrences
        return {"bytes": read, "flops": flops}
    hd = cfg["hidden_size"] // cfg["num_attention_heads"]
    pairs = sum(c + 1 for c in contexts) + t * (t + 1) / 2.0
    flops += 4.0 * pairs * cfg["num_attention_heads"] * hd * cfg["num_hidden_layers"]
    row = 2.0 * cfg["num_key_value_heads"] * hd * size * cfg["num_hidden_layers"]
    return {"bytes": read + row * (sum(contexts) + new), "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":     # the logits were measured 7e-6 to 8e-6 away from 64 bits
        return {"rel": 3e-5, "max": 3e-4}
    return {"rel": 0.03, "max": 0.2}   # 0.011 to 0.029 away from 64 bits; two runs of one pass up to 0.009 apart


# ---------------------------------------------------------------------------------------------- the same in 64 bits

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, freq, mag, dims, pairs):
    """Rotation of the first `dims` values of x [T, heads, d] by position: value i with i + dims/2, or 2i with 2i + 1."""
    ang = torch.arange(x.shape[0], device=x.device, dtype=torch.float64)[:, None] * freq
    c, s = torch.cos(ang)[:, None] * mag, torch.sin(ang)[:, None] * mag
    out = x.clone()
    u, v = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., u], out[..., v] = x[..., u] * c - x[..., v] * s, x[..., v] * c + x[..., u] * s
    return out


def _attend(scores, v, window=None, sink=None):
    """scores [H, T, T], v [H, T, d] -> [T, H * d]: causal softmax, over a window, with a sink in the denominator."""
    t = scores.shape[1]
    i = torch.arange(t, device=v.device)
    seen = i[None, :] <= i[:, None]
    if window:
        seen &= i[:, None] - i[None, :] < window
    scores.masked_fill_(~seen, float("-inf"))
    top = scores.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink[:, None, None])
    p = scores.sub_(top).exp_()
    total = p.sum(-1, keepdim=True)
    if sink is not None:
        total = total + torch.exp(sink[:, None, None] - top)
    return ((p @ v) / total).transpose(0, 1).reshape(t, -1)


def _llama_row(cfg, w, tokens):
    """Logits of the last of `tokens`."""
    t, n, kv = len(tokens), cfg["num_attention_heads"], cfg["num_key_value_heads"]
    hd, eps = cfg["hidden_size"] // n, cfg["rms_norm_eps"]
    freq = cfg["rope_theta"] ** (-torch.arange(hd // 2, device=DEVICE, dtype=torch.float64) / (hd // 2))
    x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEVICE)]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w[p + "input_layernorm.weight"]
        q, k, v = ((h @ w[p + f"self_attn.{m}_proj.weight"].T).view(t, -1, hd) for m in "qkv")
        q, k = (_turn(y, freq, 1.0, hd, False).transpose(0, 1) for y in (q, k))
        v, out = v.transpose(0, 1), []
        for j in range(kv):
            mine = q[j * (n // kv): (j + 1) * (n // kv)]
            out.append(_attend((mine @ k[j].T) * hd ** -0.5, v[j].expand(n // kv, t, hd)))
        x = x + torch.cat(out, dim=1) @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, eps) * w[p + "post_attention_layernorm.weight"]
        gate = h @ w[p + "mlp.gate_proj.weight"].T
        x = x + (gate * torch.sigmoid(gate) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return (_rms(x[-1:], eps) * w["model.norm.weight"]) @ w["lm_head.weight"].T


def _conv(x, taps, bias=0.0):
    n = taps.shape[1]
    pad = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    y = sum(pad[j: j + x.shape[0]] * taps[:, j] for j in range(n)) + bias
    return y * torch.sigmoid(y)


def _frequencies(rot):
    dims, base = rot["dims"], rot["base"]
    i = torch.arange(dims // 2, device=DEVICE, dtype=torch.float64)
    f, s = base ** (-2.0 * i / dims), rot.get("scaling")
    if not s:
        return f, 1.0

    def at(turns):
        return dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _gevovik_row(cfg, w, tokens):
    """Logits of the last of `tokens`: the recurrences token by token, attention as whole score matrices."""
    t, eps, big = len(tokens), cfg["norm"]["eps"], cfg["embedding"]["bigram"]
    rows = [big["buckets"]] + [(a * big["mul_prev"] + b * big["mul_cur"]) % big["buckets"] for a, b in zip(tokens, tokens[1:])]
    x = w["embed"][torch.tensor(tokens, device=DEVICE)] * cfg["embedding"]["scale"] + w["bigram"][torch.tensor(rows, device=DEVICE)]
    kept = {}
    soft = torch.nn.functional.softplus
    for i, layer in enumerate(cfg["layers"]):
        m, p, h = layer["mixer"], f"l{i}.mix.", x
        if layer["type"] == "latent_attention":
            n, nd, rank = m["heads"], m["dim"], m["kv_rank"]
            freq, mag = _frequencies(m["rot"])
            if "kv_from" not in m:
                d = h @ w[p + "dkv"].T
                kept[i] = (_rms(d[:, :rank], eps) * w[p + "dkv.norm"], _turn(d[:, None, rank:], freq, mag, m["rot"]["dims"], True)[:, 0])
            c, kr = kept[m.get("kv_from", i)]
            q = (h @ w[p + "q"].T).view(t, n, -1)
            k, v = ((c @ w[p + name].T).view(t, n, -1).transpose(0, 1) for name in ("uk", "uv"))
            turned = _turn(q[..., nd:], freq, mag, m["rot"]["dims"], True).transpose(0, 1)
            scores = (q[..., :nd].transpose(0, 1) @ k.transpose(1, 2) + turned @ kr.T) * m["scale"]
            y = _attend(scores, v, sink=w[p + "sink"]) @ w[p + "o"].T
        elif layer["type"] == "mamba2":
            n, vd, st, groups = m["heads"], m["vdim"], m["state"], m["groups"]
            z, xbc, dt = (h @ w[p + "in"].T).split([n * vd, n * vd + 2 * groups * st, n], dim=1)
            u, b, c = _conv(xbc, w[p + "conv"], w[p + "conv.b"]).split([n * vd, groups * st, groups * st], dim=1)
            u = u.reshape(t, n, vd)
            b, c = (s.reshape(t, groups, st).repeat_interleave(n // groups, dim=1) for s in (b, c))
            dt = soft(dt + w[p + "dt_bias"])
            decay, b = torch.exp(-torch.exp(w[p + "A_log"]) * dt), b * dt[..., None]
            s, o = x.new_zeros(n, st, vd), []
            for j in range(t):
                s = torch.baddbmm(s * decay[j][:, None, None], b[j][:, :, None], u[j][:, None, :])
                o.append(torch.bmm(c[j][:, None, :], s)[:, 0])
            y = (torch.stack(o) + w[p + "D"][:, None] * u).reshape(t, -1) * (z * torch.sigmoid(z))
            y = (_rms(y.view(t, m["norm_groups"], -1), eps).reshape(t, -1) * w[p + "norm"]) @ w[p + "o"].T
        else:
            a, b, pl, pr = m["left"], m["right"], p + "left.", p + "right."
            n, kv, kd = a["heads"], a["kv_heads"], a["dim"]
            freq, mag = _frequencies(a["rot"])
            q = _rms((h @ w[pl + "q"].T).view(t, n, kd), eps) * w[pl + "q.norm"]
            k = _rms((h @ w[pl + "k"].T).view(t, kv, kd), eps) * w[pl + "k.norm"]
            q, k = (_turn(s, freq, mag, a["rot"]["dims"], False).transpose(0, 1) for s in (q, k))
            v = (h @ w[pl + "v"].T).view(t, kv, -1).transpose(0, 1).repeat_interleave(n // kv, dim=0)
            scores = q @ k.repeat_interleave(n // kv, dim=0).transpose(1, 2) * (a["scale"] * w[pl + "temp"][:, None, None])
            scores = (w[pl + "talk"] @ scores.view(n, -1)).view(n, t, t)
            o = _attend(scores, v, window=a["mask"]["size"]).view(t, n, -1) * torch.sigmoid(h @ w[pl + "g"].T)[:, :, None]
            left = o.reshape(t, -1) @ w[pl + "o"].T
            n, kv, kd = b["heads"], b["kv_heads"], b["dim"]
            q, k, v = (_conv(h @ w[pr + s].T, w[pr + s + ".conv"]).view(t, -1, kd) for s in "qkv")
            q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * kd ** -0.5
            k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            q, k = (s.repeat_interleave(n // kv, dim=1) for s in (q, k))
            beta = torch.sigmoid(h @ w[pr + "b"].T)
            low = (h @ w[pr + "a1"].T) @ w[pr + "a2"].T + w[pr + "dt_bias"]
            g = torch.exp(-torch.exp(w[pr + "A_log"])[:, None] * soft(low).view(t, n, kd))
            s, o = x.new_zeros(n, kd, b["vdim"]), []
            for j in range(t):
                s = s * g[j][:, :, None]
                u = beta[j][:, None, None] * (v[j][:, None, :] - torch.bmm(k[j][:, None, :], s))
                s = torch.baddbmm(s, k[j][:, :, None], u)
                o.append(torch.bmm(q[j][:, None, :], s)[:, 0])
            gate = torch.sigmoid((h @ w[pr + "g1"].T) @ w[pr + "g2"].T).view(t, n, -1)
            right = (_rms(torch.stack(o), eps) * w[pr + "norm"] * gate).reshape(t, -1) @ w[pr + "o"].T
            y = m["left_scale"] * left + m["right_scale"] * right
        x = x + _rms(y, eps) * w[f"l{i}.norm1"]
        f = torch.relu(x @ w[f"l{i}.mlp.up"].T)
        x = x + _rms((f * f) @ w[f"l{i}.mlp.down"].T, eps) * w[f"l{i}.norm2"]
    return (_rms(x[-1:], eps) * w["final.norm"]) @ w["head"].T


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "sample":
        return None
    w = {n: t.double() for n, t in _weights(case, seed).items()}
    held, feed, prompt = _token_lists(case, seed)
    row = _gevovik_row if case["model"] == "gevovik" else _llama_row
    sequences = [a + f[:1] for a, f in zip(held, feed)] + ([prompt] if prompt else [])
    return torch.cat([row(_config(case), w, s) for s in sequences])
