"""What the engine is asked to do in real use, as cases that can be timed and compared.

Every case is Hunyuan Dense, the architecture the engine's benchmark is quoted on, at the layer
sizes of that benchmark (1.8B, 4B, 7B; all 32 layers), random weights, through
``ModelForCausalLM.from_tensors`` and ``ModelRunner.step``, the one way tokens get through the
model.  A pass is

* ``decode``: one step with one token of each of ``batch`` requests whose ``context`` earlier
  positions are in the cache (``spread``: contexts of very different lengths up to ``context``,
  as continuous batching has them; the requests grow by a token per pass, as they do in use);
* ``prefill``: one new prompt of ``tokens`` tokens in portions of at most ``chunk``, whose last
  place's logits are wanted, after which the request ends;
* ``mixed``: one step with one token of each of ``batch`` requests beside a new prompt of
  ``tokens`` tokens, which ends with the pass.

The cache of the waiting requests is laid out with unit-variance keys and values: what the
per-head norms of keys produce, and values of the same scale.  Matrices have standard deviation
0.02, the two that add to the residual stream 0.02 / sqrt(2 layers), the embedding EMBED_STD: a
sublayer then adds a small part to the stream, as in a trained model.
"""
import math

import torch

from crane_b200.engine import StepEntry
from crane_b200.generation import ModelForCausalLM

PAGE = 64               # tokens per cache page, the engine's default
PORTION = 2048          # tokens per step, the engine's default budget
EMBED_STD = 0.5
DEVICE = "cuda:0"

_COMMON = {
    "architectures": ["HunYuanDenseV1ForCausalLM"], "model_type": "hunyuan_v1_dense",
    "num_hidden_layers": 32, "head_dim": 128, "hidden_act": "silu", "max_position_embeddings": 32768,
    "rms_norm_eps": 1e-5, "rope_theta": 10000.0, "rope_scaling": {"alpha": 1000.0, "type": "dynamic"},
    "use_qk_norm": True, "attention_bias": False,
}
SIZES = {
    "1.8b": {"hidden_size": 2048, "intermediate_size": 6144, "num_attention_heads": 16, "num_key_value_heads": 4,
             "vocab_size": 120818, "tie_word_embeddings": True},
    "4b": {"hidden_size": 3072, "intermediate_size": 8192, "num_attention_heads": 32, "num_key_value_heads": 8,
           "vocab_size": 120818, "tie_word_embeddings": True},
    "7b": {"hidden_size": 4096, "intermediate_size": 14336, "num_attention_heads": 32, "num_key_value_heads": 8,
           "vocab_size": 128167, "tie_word_embeddings": False},
}


def _decode(size, batch, context, spread=False):
    return {"kind": "decode", "size": size, "dtype": "bf16", "batch": batch, "context": context, "spread": spread}


def _prefill(size, tokens, dtype="bf16"):
    return {"kind": "prefill", "size": size, "dtype": dtype, "tokens": tokens}


def listed():
    return [
        # three short chats at once, a few dozen to a few hundred tokens in: launches and latency
        dict(_decode("1.8b", 3, 307, True), name="decode_1.8b_b3_short"),
        # one user far into a long conversation
        dict(_decode("1.8b", 1, 8192), name="decode_1.8b_b1_8k"),
        # the benchmark's headline: eight long conversations
        dict(_decode("1.8b", 8, 8192), name="decode_1.8b_b8_8k"),
        # a full server: the cache dominates
        dict(_decode("1.8b", 64, 8192), name="decode_1.8b_b64_8k"),
        # the middle of a serving mix: requests of very different lengths
        dict(_decode("4b", 21, 4096, True), name="decode_4b_b21_spread"),
        # the largest model for a few users: its weights dominate
        dict(_decode("7b", 4, 4096), name="decode_7b_b4_4k"),
        # a chat turn's prompt
        dict(_prefill("1.8b", 137), name="prefill_1.8b_137"),
        # the benchmark's prompt: one full step
        dict(_prefill("1.8b", 2048), name="prefill_1.8b_2048"),
        # a document in portions
        dict(_prefill("7b", 8192), name="prefill_7b_8192"),
        # continuous batching: running requests beside the prompt of a new one
        {"kind": "mixed", "size": "4b", "dtype": "bf16", "batch": 48, "context": 4096, "spread": True, "tokens": 600,
         "name": "mixed_4b_b48_600"},
        # the 32-bit path, which answers are checked with
        dict(_prefill("1.8b", 97, "fp32"), name="prefill_1.8b_97_fp32"),
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "mixed"])
    size = rng.choice(["1.8b", "1.8b", "4b", "7b"])
    if kind == "decode":
        batch = _log_uniform(rng, 1, 64)
        context = _log_uniform(rng, 16, 16384)
        # no more cached keys than the listed cases have
        return _decode(size, batch, min(context, (4096 if size != "1.8b" else 8192) * 48 // batch), rng.random() < 0.5)
    if kind == "mixed":
        return {"kind": "mixed", "size": rng.choice(["1.8b", "4b"]), "dtype": "bf16", "batch": _log_uniform(rng, 1, 48),
                "context": _log_uniform(rng, 64, 4096), "spread": True, "tokens": _log_uniform(rng, 16, 1900)}
    if rng.random() < 0.15:
        return _prefill("1.8b", _log_uniform(rng, 2, 160), "fp32")
    return _prefill(size, _log_uniform(rng, 2, 8192))


# ------------------------------------------------------------------ what a case consists of
def _config(case):
    return dict(_COMMON, **SIZES[case["size"]])


def _contexts(case):
    """How many positions every waiting request has in the cache."""
    if case["kind"] == "prefill":
        return []
    n, c = case["batch"], case["context"]
    if not case["spread"]:
        return [c] * n
    # from a thirty-second of the longest up to it, in no order
    return [max(1, int(round(c * 2.0 ** (-5.0 * ((i * 0.6180339887) % 1.0))))) for i in range(n)]


def _shapes(cfg):
    h, inner, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    nq, nkv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
    out = {"model.embed_tokens.weight": (cfg["vocab_size"], h), "model.norm.weight": (h,)}
    if not cfg["tie_word_embeddings"]:
        out["lm_head.weight"] = (cfg["vocab_size"], h)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        out.update({p + "input_layernorm.weight": (h,), p + "post_attention_layernorm.weight": (h,),
                    p + "self_attn.q_proj.weight": (nq, h), p + "self_attn.k_proj.weight": (nkv, h),
                    p + "self_attn.v_proj.weight": (nkv, h), p + "self_attn.o_proj.weight": (h, nq),
                    p + "self_attn.query_layernorm.weight": (d,), p + "self_attn.key_layernorm.weight": (d,),
                    p + "mlp.gate_proj.weight": (inner, h), p + "mlp.up_proj.weight": (inner, h),
                    p + "mlp.down_proj.weight": (h, inner)})
    return out


def _tensors(cfg, seed):
    """Weights by name, all from one stream of random numbers."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    out = {}
    for name, shape in _shapes(cfg).items():
        if len(shape) == 1:
            out[name] = 1.0 + 0.01 * torch.randn(shape, generator=g, device=DEVICE)
            continue
        std = 0.02
        if name.endswith(("o_proj.weight", "down_proj.weight")):
            std /= math.sqrt(2.0 * cfg["num_hidden_layers"])
        elif name == "model.embed_tokens.weight":
            std = EMBED_STD
        out[name] = torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(0.0, std, generator=g)
    return out


def _cached(case, cfg, seed):
    """Per layer the keys and the values of the waiting requests in whole pages,
    [pages of all requests, kv heads, page, head size]."""
    pages = sum(-(-c // PAGE) for c in _contexts(case))
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed + 1000003)
    shape = (pages, cfg["num_key_value_heads"], PAGE, cfg["head_dim"])
    for _ in range(cfg["num_hidden_layers"]):
        yield tuple(torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(0.0, 1.0, generator=g)
                    for _ in range(2))


def _tokens(seed, n, vocab):
    g = torch.Generator()
    g.manual_seed(seed + 2000003)
    return torch.randint(0, vocab, (n,), generator=g).tolist()


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    cfg = _config(case)
    contexts = _contexts(case)
    prompt = case.get("tokens", 0)
    room = max(1024, 8192 // max(1, len(contexts))) if contexts else 0    # tokens a request can grow by
    pages = sum(-(-(c + room) // PAGE) for c in contexts) + -(-prompt // PAGE) + 1
    model = ModelForCausalLM.from_tensors(
        cfg, _tensors(cfg, seed), case["dtype"], page_size=PAGE, num_pages=pages, max_concurrent=64,
        max_seq_len=max([c + room for c in contexts] + [prompt, PAGE]), max_batched_tokens=PORTION, chunk_size=PORTION)
    runner = model.runner
    ids = list(range(1, len(contexts) + 1))
    for rid, c in zip(ids, contexts):
        runner.table.admit(rid)
        runner.table.extend(rid, c)
    if ids:
        held = [runner.table.block_table(rid, 0, -(-c // PAGE)) for rid, c in zip(ids, contexts)]
        held = torch.cat([torch.from_numpy(h) for h in held]).to(DEVICE, torch.long)
        for layer, (k, v) in zip(runner.pools.layers, _cached(case, cfg, seed)):
            layer.k[held] = k
            layer.v[held] = v
    tokens = _tokens(seed, len(ids) + prompt, cfg["vocab_size"])
    torch.cuda.empty_cache()
    return {"model": model, "runner": runner, "ids": ids, "contexts": contexts, "next": tokens[:len(ids)],
            "prompt": tokens[len(ids):], "room": room, "left": room, "fresh": 1000}


def run(state):
    runner, prompt = state["runner"], state["prompt"]
    if state["ids"] and state["left"] == 0:
        # the requests have used up the positions they may have: they start again where they began
        for rid, c in zip(state["ids"], state["contexts"]):
            runner.end(rid)
            runner.table.admit(rid)
            runner.table.extend(rid, c)
        state["left"] = state["room"]
    state["left"] -= 1
    waiting = [StepEntry(rid, [t], [0]) for rid, t in zip(state["ids"], state["next"])]
    if not prompt:
        return runner.step(waiting)
    rid = state["fresh"]
    state["fresh"] += 1
    for a in range(0, len(prompt), PORTION):
        part = prompt[a:a + PORTION]
        want = [len(part) - 1] if a + len(part) == len(prompt) else []
        logits = runner.step(waiting + [StepEntry(rid, part, want)])
    runner.end(rid)
    if waiting:
        return logits
    # a prompt's result is its last place's logits and what it left in the cache; the last layer's
    # keys and values depend on every layer before it
    last = runner.pools.layers[-1]
    return {"logits": logits, "keys": last.k, "values": last.v}


def work(case):
    cfg = _config(case)
    h, inner, d, layers = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"], cfg["num_hidden_layers"]
    nq, nkv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
    matrices = h * (nq + 2 * nkv) + nq * h + 3 * h * inner
    head = cfg["vocab_size"] * h
    contexts, prompt = _contexts(case), case.get("tokens", 0)
    elem = 4 if case["dtype"] == "fp32" else 2
    rows = len(contexts) + (1 if prompt else 0)
    tokens = len(contexts) + prompt
    keys = sum(c + 1 for c in contexts) + prompt * (prompt + 1) / 2.0           # (query, key) pairs, causal
    return {"bytes": elem * (layers * (matrices + 2 * h) + head + tokens * h)
            + elem * layers * 2 * nkv * (sum(contexts) + tokens) + 4 * rows * cfg["vocab_size"],
            "flops": 2.0 * tokens * layers * matrices + 4.0 * layers * nq * keys + 2.0 * rows * head}


def tolerance(case):
    # 32-bit: sums of 2048 to 6144 terms in another order.  bfloat16: every layer's products round their
    # inputs and results to 8 bits; two such paths are up to 1.4 times as far apart as one is from the 64-bit result.
    return {"rel": 2e-5, "max": 2e-3} if case["dtype"] == "fp32" else {"rel": 2.5e-2, "max": 0.3}


# ------------------------------------------------------------------ the same in 64 bits
def _unit_rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, first, cfg):
    """x [tokens, heads, d] at positions first ..: element i turns with element i + d / 2."""
    d = cfg["head_dim"]
    base = cfg["rope_theta"] * cfg["rope_scaling"]["alpha"] ** (d / (d - 2.0))
    i = torch.arange(d // 2, dtype=torch.float64, device=DEVICE)
    # frequencies and angles are 32-bit numbers in the architecture's definition
    f = 1.0 / (base ** (2.0 * i / d)).float()
    pos = torch.arange(first, first + x.shape[0], dtype=torch.float32, device=DEVICE)
    a = (pos[:, None] * f[None, :]).double()[:, None, :]
    u, v = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1)


def _attend(q, k, v, first):
    """q [n, heads, d] at positions first .., k and v [positions, kv heads, d]: causal softmax attention."""
    n, heads, d = q.shape
    group = heads // k.shape[1]
    out = torch.empty_like(q)
    for h in range(heads):
        kh, vh = k[:, h // group], v[:, h // group]
        for a in range(0, n, 2048):
            b = min(n, a + 2048)
            seen = first + b
            s = q[a:b, h] @ kh[:seen].T / math.sqrt(d)
            later = torch.arange(seen, device=DEVICE)[None, :] > torch.arange(first + a, first + b, device=DEVICE)[:, None]
            out[a:b, h] = torch.softmax(s.masked_fill_(later, float("-inf")), dim=-1) @ vh[:seen]
    return out


def exact(case, seed):
    cfg = _config(case)
    eps, d = cfg["rms_norm_eps"], cfg["head_dim"]
    nq, nkv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    w = _tensors(cfg, seed)
    contexts, prompt = _contexts(case), case.get("tokens", 0)
    tokens = _tokens(seed, len(contexts) + prompt, cfg["vocab_size"])
    x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEVICE)].double()
    cached = _cached(case, cfg, seed) if contexts else None
    for layer in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        W = lambda name: w[p + name + ".weight"].double()          # noqa: E731
        y = _unit_rms(x, eps) * W("input_layernorm")
        q = (y @ W("self_attn.q_proj").T).view(-1, nq, d)
        k = (y @ W("self_attn.k_proj").T).view(-1, nkv, d)
        v = (y @ W("self_attn.v_proj").T).view(-1, nkv, d)
        att = torch.empty_like(q)

        def turned(first, a, b):
            return (_unit_rms(_rotate(q[a:b], first, cfg), eps) * W("self_attn.query_layernorm"),
                    _unit_rms(_rotate(k[a:b], first, cfg), eps) * W("self_attn.key_layernorm"))

        if contexts:
            old_k, old_v = next(cached)
            page = 0
            for i, c in enumerate(contexts):
                n = -(-c // PAGE)
                qi, ki = turned(c, i, i + 1)
                past = [t[page:page + n].double().transpose(1, 2).reshape(n * PAGE, nkv, d)[:c] for t in (old_k, old_v)]
                page += n
                keys, values = torch.cat([past[0], ki]), torch.cat([past[1], v[i:i + 1]])
                s = torch.einsum("ghd,ngd->ghn", qi.view(nkv, nq // nkv, d), keys) / math.sqrt(d)
                att[i] = torch.einsum("ghn,ngd->ghd", torch.softmax(s, dim=-1), values).reshape(nq, d)
        if prompt:
            n = len(contexts)
            qi, ki = turned(0, n, n + prompt)
            att[n:] = _attend(qi, ki, v[n:], 0)
        x = x + att.reshape(-1, nq * d) @ W("self_attn.o_proj").T
        y = _unit_rms(x, eps) * W("post_attention_layernorm")
        act = torch.nn.functional.silu(y @ W("mlp.gate_proj").T) * (y @ W("mlp.up_proj").T)
        x = x + act @ W("mlp.down_proj").T
    rows = list(range(len(contexts))) + ([len(tokens) - 1] if prompt else [])
    y = _unit_rms(x[rows], eps) * w["model.norm.weight"].double()
    head = w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]
    logits = torch.cat([y @ part.double().T for part in head.split(16384)], dim=1)
    if contexts:
        return logits
    # where a request's pages lie is the engine's own affair
    return {"logits": logits, "keys": None, "values": None}
