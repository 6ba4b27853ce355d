"""The engine's work in cases that can be timed: steps of prompts, portions and decode rows, and whole turns.

A case is a dict of plain values. Two kinds:

  step   one `Engine.step` over `decode` requests that bring one token each, at contexts spread evenly (on a logarithmic
         scale) over `context_low` .. `context_high`, beside `prompts` requests that bring `prompt_low` .. `prompt_high`
         tokens each, behind `prompt_context` tokens that are in the cache already. Returns the logits of every request's
         last token. A pass takes its tokens back afterwards (new requests are released, the others' length is set to what
         it was), so the next pass runs the same rows again.
  turn   what a short conversation turn is: `requests` requests are admitted, bring prompts of `prompt_low` .. `prompt_high`
         tokens in one step, decode `new` tokens step by step and are released. Returns the logits of every step.

Models have the layer sizes of `bench.py` with the first `layers` layers (every layer is as large as in the whole model; fewer
of them keep the preparation short). Weights are random, as in every benchmark here, and token ids uniform, but routers decide
as trained ones do (`decide`): rows of purely random routers lie at a near tie in every other layer or so, where two correct
implementations choose different experts and an output says nothing about the arithmetic.

`exact` is the same in 64-bit torch, written from the models' formulas: whole sequences, no cache, no kernel of the engine's.
"""

from __future__ import annotations

import math

import torch

from tandemllm_b200.config import Lfm2MoeConfig, PuripelConfig, SebilornConfig
from tandemllm_b200.engine import Engine, EngineArgs, StepEntry
from tandemllm_b200.kernels import tensorcore
from tandemllm_b200.parts.base import Runtime
from tandemllm_b200.parts.model import DecoderModel
from tandemllm_b200.weights.loader import DictWeights
from tandemllm_b200.weights.random_init import random_weights

DEVICE = "cuda:0"
DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
CODES, CODE_DIMS, CODE_SIZE = 64, 256, 4.0      # see `decide`
FEED_ROWS = 4096                        # rows a preparing step feeds (contexts)

LAYERS_8B = ["full_attention" if i in (2, 6, 10, 14, 18, 21) else "conv" for i in range(24)]
LAYERS_24B = ["full_attention" if i % 4 == 2 else "conv" for i in range(40)]
LFM2 = dict(
    model_type="lfm2_moe", architectures=["Lfm2MoeForCausalLM"], vocab_size=65536, hidden_size=2048, num_attention_heads=32,
    num_key_value_heads=8, head_dim=64, norm_eps=1e-5, max_position_embeddings=128000, conv_bias=False, conv_L_cache=3,
    num_dense_layers=2, num_experts_per_tok=4, use_expert_bias=True, routed_scaling_factor=1.0, norm_topk_prob=True,
    tie_word_embeddings=True, rope_parameters={"rope_type": "default", "rope_theta": 1000000.0}, eos_token_id=7, bos_token_id=1,
    pad_token_id=0)


# ---- models ----

def raw_config(case: dict) -> dict:
    """config.json of the case's model."""
    model, layers = case["model"], int(case["layers"])
    if model == "lfm2-8b":
        return dict(LFM2, intermediate_size=7168, moe_intermediate_size=1792, num_experts=32, num_hidden_layers=layers,
                    layer_types=LAYERS_8B[:layers])
    if model == "lfm2-24b":
        return dict(LFM2, intermediate_size=11776, moe_intermediate_size=1536, num_experts=64, num_hidden_layers=layers,
                    layer_types=LAYERS_24B[:layers])
    if model == "puripel-2k":
        mlp = {"kind": "moe", "router": {"experts": 64, "top": 6, "scale": 2.5, "groups": {"count": 8, "keep": 4}},
               "expert": {"ff": 768, "limit": 7.0}, "shared": {"ff": 1536, "limit": 7.0}}
        ssm = {"type": "mamba2", "mlp": mlp,
               "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}
        att = {"type": "latent_attention", "mlp": mlp,
               "mixer": {"heads": 32, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 1024, "scale": 192 ** -0.5,
                         "rot": {"base": 10000.0, "dims": 64}, "mask": {"size": 2048}}}
        return {"architecture": "Puripel", "vocab": 65536, "width": 2048, "norm": {"eps": 1e-5},
                "layers": [ssm if i % 2 == 0 else att for i in range(layers)]}
    if model == "sebilorn-2k":
        mlp = {"kind": "dense", "ff": 8192}
        rot = {"base": 500000.0, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
        att = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0, "rot": rot,
               "mask": {"size": 1024, "keep_first": 4}}
        left = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": {"base": 1e6, "dims": 128}}
        kinds = []
        for i in range(layers):
            kinds.append([{"type": "attention", "mixer": dict(att), "mlp": mlp},
                          {"type": "attention", "mixer": dict(att, kv_from=i - 1), "mlp": mlp},
                          {"type": "parallel", "mlp": mlp, "mixer": {"left": left, "right": {"heads": 16, "dim": 128},
                                                                     "left_scale": 0.8, "right_scale": 0.5}},
                          {"type": "lightning", "mlp": mlp,
                           "mixer": {"heads": 16, "dim": 128, "vdim": 128,
                                     "decay": [1.0 - 2.0 ** (-3 - 5 * h / 15) for h in range(16)]}}][i % 4])
        return {"architecture": "Sebilorn", "vocab": 65536, "width": 2048, "norm": {"eps": 1e-5},
                "embedding": {"scale": 2048 ** 0.5}, "logit_softcap": 30.0, "layers": kinds}
    raise ValueError(model)


def typed_config(case: dict):
    reader = {"lfm2": Lfm2MoeConfig, "puripel": PuripelConfig, "sebilorn": SebilornConfig}[case["model"].split("-")[0]]
    return reader.from_dict(raw_config(case))


def vocab_of(case: dict) -> int:
    raw = raw_config(case)
    return raw.get("vocab_size") or raw["vocab"]


def weights_of(case: dict, seed: int) -> dict:
    """The model's tensors by name, as `Engine.from_config` draws them, with routers that decide."""
    specs = DecoderModel(typed_config(case).to_spec()).weight_specs(None)
    tensors = random_weights(specs, seed, dtype=DTYPES[case["dtype"]], device=DEVICE)
    raw = raw_config(case)
    if case["model"].startswith("lfm2"):
        routers = {f"layers.{i}.feed_forward.": ("gate.weight", "expert_bias") for i in range(raw["num_dense_layers"], raw["num_hidden_layers"])}
        decide(tensors, routers, raw["num_experts"], raw["num_experts_per_tok"], None, "embed_tokens.weight", "embedding_norm.weight", seed)
    elif case["model"].startswith("puripel"):
        r = raw["layers"][0]["mlp"]["router"]
        decide(tensors, {f"l{i}.mlp.": ("router", "correction") for i in range(len(raw["layers"]))}, r["experts"], r["top"],
               r["groups"], "embed", "final.norm", seed)
    return tensors


def decide(tensors: dict, routers: dict, experts: int, top: int, groups: dict | None, embedding: str, last_norm: str, seed: int) -> None:
    """A token's embedding carries one of CODES codes in its first CODE_DIMS dimensions, which are large, as a few dimensions
    of trained models are (and which the last norm's weights take out again), and every router maps a code to `top` experts
    of its own, every expert as often as any other: the chosen scores are near 0.9 and the others near 0.5."""
    g = torch.Generator().manual_seed(104729 * int(seed) + 5)
    codes = (torch.randint(0, 2, (CODES, CODE_DIMS), generator=g) * 2.0 - 1.0)
    table = tensors[embedding]
    which = torch.randint(0, CODES, (table.shape[0],), generator=g)
    table[:, :CODE_DIMS] += (CODE_SIZE * codes)[which].to(table)
    tensors[last_norm][:CODE_DIMS] = 0.02
    for prefix, (router, bias) in routers.items():
        rows = torch.zeros(experts, CODE_DIMS)
        order: list[int] = []
        for c in range(CODES):
            if groups is None:
                if len(order) < top:
                    order = torch.randperm(experts, generator=g).tolist()
                chosen, order = order[:top], order[top:]
            else:
                per, chosen = experts // groups["count"], []
                for j, grp in enumerate(torch.randperm(groups["count"], generator=g)[:groups["keep"]].tolist()):
                    n = top // groups["keep"] + (j < top % groups["keep"])
                    chosen += (grp * per + torch.randperm(per, generator=g)[:n]).tolist()
            rows[chosen] += codes[c]
        t = tensors[prefix + router]
        t *= 0.25
        t[:, :CODE_DIMS] += (rows * (2.4 / (1.4 * CODE_DIMS))).to(t)
        tensors[prefix + bias] *= 0.2


# ---- sizes ----

def spread(low: int, high: int, count: int) -> list[int]:
    """`count` whole numbers from low to high, evenly on a logarithmic scale."""
    if count <= 0:
        return []
    if count == 1:
        return [high]
    return [int(round(low * (high / low) ** (i / (count - 1)))) for i in range(count)]


def lengths(case: dict) -> list[tuple[int, int]]:
    """(tokens in the cache, new tokens) of every request of the case's (first) step."""
    if case["kind"] == "turn":
        return [(0, n) for n in spread(case["prompt_low"], case["prompt_high"], case["requests"])]
    out = [(int(case["prompt_context"]), n) for n in spread(case["prompt_low"], case["prompt_high"], case["prompts"])]
    return out + [(c, 1) for c in spread(case["context_low"], case["context_high"], case["decode"])]


def draw_tokens(case: dict, seed: int) -> list[list[int]]:
    """The whole text of every request: its context, its new tokens and what it decodes afterwards."""
    g = torch.Generator().manual_seed(7919 * int(seed) + 17)
    more = int(case["new"]) if case["kind"] == "turn" else 0
    return [torch.randint(0, vocab_of(case), (c + n + more,), generator=g).tolist() for c, n in lengths(case)]


# ---- the cases ----

def step_case(name=None, model="lfm2-8b", layers=8, dtype="bfloat16", decode=0, context_low=1, context_high=1, prompts=0,
              prompt_low=1, prompt_high=1, prompt_context=0) -> dict:
    c = dict(kind="step", model=model, layers=layers, dtype=dtype, decode=decode, context_low=context_low, context_high=context_high,
             prompts=prompts, prompt_low=prompt_low, prompt_high=prompt_high, prompt_context=prompt_context)
    return dict(c, name=name) if name else c


def turn_case(name=None, model="puripel-2k", layers=4, dtype="bfloat16", requests=1, prompt_low=1, prompt_high=1, new=8) -> dict:
    c = dict(kind="turn", model=model, layers=layers, dtype=dtype, requests=requests, prompt_low=prompt_low, prompt_high=prompt_high,
             new=new)
    return dict(c, name=name) if name else c


def listed() -> list[dict]:
    return [
        # one user chats: a token of one request a step, the smallest call there is
        step_case("decode_1", decode=1, context_low=700, context_high=700),
        # eight long conversations decode together (the benchmark's headline batch and context)
        step_case("decode_8_long", decode=8, context_low=8192, context_high=8192),
        # a busy server between prompts: many requests, each as far as it has got
        step_case("decode_64_ragged", decode=64, context_low=130, context_high=2900),
        # the first words of a conversation
        step_case("prompt_37", prompts=1, prompt_low=37, prompt_high=37),
        # several questions that came at once
        step_case("prompts_5_ragged", prompts=5, prompt_low=61, prompt_high=402),
        # a page of text (the benchmark's prompt)
        step_case("prompt_2048", prompts=1, prompt_low=2048, prompt_high=2048),
        # a document read portion by portion
        step_case("portion_2048_at_14k", prompts=1, prompt_low=2048, prompt_high=2048, prompt_context=14300),
        # a portion of a newcomer's prompt beside the rows of those who decode
        step_case("portion_512_beside_decode_23", prompts=1, prompt_low=512, prompt_high=512, prompt_context=1531, decode=23,
                  context_low=201, context_high=4100),
        # the larger model of the family, a small server's batch
        step_case("24b_decode_16", model="lfm2-24b", layers=6, decode=16, context_low=512, context_high=4096),
        # the 32-bit path, as a check of answers runs it
        step_case("float32_prompt_150", layers=3, dtype="float32", prompts=1, prompt_low=150, prompt_high=150),
        # state spaces, latent attention and grouped experts with a shared one: a turn of two requests
        turn_case("puripel_turn", model="puripel-2k", layers=4, requests=2, prompt_low=300, prompt_high=700, new=16),
        # matrix states and capped, windowed attention over dense feed-forwards: a turn of four requests
        turn_case("sebilorn_turn", model="sebilorn-2k", layers=4, requests=4, prompt_low=120, prompt_high=1100, new=16),
    ]


def draw(rng) -> dict:
    def between(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    what = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "prompt", "mixed", "mixed", "24b", "float32", "puripel", "sebilorn"])
    if what == "decode":
        n, high = between(1, 64), between(64, 8192)
        return step_case(decode=n, context_low=max(1, int(high * rng.uniform(0.05, 1.0))), context_high=high)
    if what == "prompt":
        n = rng.choice([1, 1, 2, 5])
        high = between(5, 2048 // n)
        behind = 0 if n > 1 or rng.random() < 0.6 else between(16, 14300)
        return step_case(prompts=n, prompt_low=max(1, int(high * rng.uniform(0.2, 1.0))), prompt_high=high, prompt_context=behind)
    if what == "mixed":
        n, high = between(1, 40), between(100, 6000)
        portion = between(16, 1024)
        return step_case(prompts=1, prompt_low=portion, prompt_high=portion, prompt_context=rng.randrange(0, 3000), decode=n,
                         context_low=max(1, int(high * rng.uniform(0.05, 1.0))), context_high=high)
    if what == "24b":
        if rng.random() < 0.5:
            n, high = between(1, 40), between(64, 6000)
            return step_case(model="lfm2-24b", layers=6, decode=n, context_low=max(1, high // 3), context_high=high)
        n = between(9, 1400)
        return step_case(model="lfm2-24b", layers=6, prompts=1, prompt_low=n, prompt_high=n)
    if what == "float32":
        n = between(1, 300)
        return step_case(layers=3, dtype="float32", prompts=1, prompt_low=n, prompt_high=n)
    n = between(1, 8)
    high = between(20, 2000 // n)
    return turn_case(model=what + "-2k", layers=4, requests=n, prompt_low=max(1, int(high * rng.uniform(0.1, 1.0))), prompt_high=high,
                     new=rng.randrange(8, 25))


# ---- state and pass ----

def prepare(case: dict, seed: int):
    """The engine with its weights, and the requests that are already running with their contexts in the cache."""
    sizes = lengths(case)
    more = int(case["new"]) if case["kind"] == "turn" else 0
    texts = draw_tokens(case, seed)
    longest = max(c + n for c, n in sizes) + more
    rows = max(FEED_ROWS, sum(n for _, n in sizes))
    pages = sum(-(-(c + n + more) // 16) for c, n in sizes)
    runtime = Runtime(torch.device(DEVICE), DTYPES[case["dtype"]])
    if case["dtype"] == "bfloat16":
        tensorcore.enable(runtime)
    model = DecoderModel(typed_config(case).to_spec()).load(DictWeights(weights_of(case, seed)), runtime)
    engine = Engine(model, EngineArgs(dtype=case["dtype"], max_len=longest, parallel=len(sizes), kv_blocks=pages,
                                      max_batched_tokens=rows, chunk_size=rows))
    running = [(i, c) for i, (c, _) in enumerate(sizes) if c]
    for i, _ in running:
        engine.admit(i)
    at = {i: 0 for i, _ in running}
    while True:                             # the contexts, a batch of portions at a time
        room, entries = FEED_ROWS, []
        for i, c in running:
            n = min(room, c - at[i])
            if n > 0:
                entries.append(StepEntry(i, texts[i][at[i]:at[i] + n], []))
                at[i] += n
                room -= n
        if not entries:
            break
        engine.step(entries)
    if case["kind"] == "turn":
        first = [StepEntry(i, t[:n], [n - 1]) for i, (t, (_, n)) in enumerate(zip(texts, sizes))]
        then = [[StepEntry(i, [t[n + k]], [0]) for i, (t, (_, n)) in enumerate(zip(texts, sizes))] for k in range(more)]
        return {"engine": engine, "first": first, "then": then}
    entries = [StepEntry(i, t[c:c + n], [n - 1]) for i, (t, (c, n)) in enumerate(zip(texts, sizes))]
    return {"engine": engine, "entries": entries, "lengths": [c for c, _ in sizes]}


def run(state):
    engine = state["engine"]
    if "first" in state:
        for e in state["first"]:
            engine.admit(e.request)
        logits = [engine.step(state["first"])]
        for entries in state["then"]:
            logits.append(engine.step(entries).clone())     # the next step writes where this one's logits lie
        for e in state["first"]:
            engine.release(e.request)
        return logits
    for e, length in zip(state["entries"], state["lengths"]):
        if length == 0:
            engine.admit(e.request)
    logits = engine.step(state["entries"])
    for e, length in zip(state["entries"], state["lengths"]):
        if length == 0:
            engine.release(e.request)
        else:
            engine.cache.advance(e.request, length)         # the tokens are taken back
    return logits


# ---- what a pass cannot do without ----

def model_work(case: dict, sizes: list[tuple[int, int]]) -> tuple[float, float]:
    """(bytes, flops) of one step over requests of `sizes` = (tokens in the cache, new tokens): every weight a row uses once
    (of the experts those that uniform routing reaches), the cached rows that are read, the logits; multiply-adds times two."""
    raw, elem = raw_config(case), 4 if case["dtype"] == "float32" else 2
    rows, outs = sum(n for _, n in sizes), len(sizes)
    weights = flops = cache = 0.0

    def dense(numbers):
        nonlocal weights, flops
        weights += numbers
        flops += 2.0 * rows * numbers

    def experts(count, top, numbers):
        nonlocal weights, flops
        weights += numbers * count * (1.0 - (1.0 - top / count) ** rows)
        flops += 2.0 * rows * top * numbers

    def attention(heads, key_dim, value_dim, cached, window=None):
        """`cached`: numbers a cached row holds."""
        nonlocal flops, cache
        for c, n in sizes:
            reach = c + n if window is None else min(c + n, window + n)
            seen = sum(min(c + i + 1, window or c + n) for i in range(n))
            cache += cached * reach
            flops += 2.0 * seen * heads * (key_dim + value_dim)

    if case["model"].startswith("lfm2"):
        W, V = raw["hidden_size"], raw["vocab_size"]
        for i, kind in enumerate(raw["layer_types"]):
            if kind == "full_attention":
                dense(W * (32 + 8 + 8) * 64 + 32 * 64 * W)
                attention(32, 64, 64, 2 * 8 * 64)
            else:
                dense(4 * W * W)
            if i < raw["num_dense_layers"]:
                dense(3 * W * raw["intermediate_size"])
            else:
                dense(W * raw["num_experts"])
                experts(raw["num_experts"], raw["num_experts_per_tok"], 3 * W * raw["moe_intermediate_size"])
    else:
        W, V = raw["width"], raw["vocab"]
        for layer in raw["layers"]:
            m = layer["mixer"]
            if layer["type"] == "mamba2":
                inner, parts = m["heads"] * m["vdim"], 2 * m["groups"] * m["state"]
                dense(W * (2 * inner + parts + m["heads"]) + inner * W)
                flops += 4.0 * rows * inner * m["state"]
                cache += 2.0 * outs * inner * m["state"] * 4 / elem
            elif layer["type"] == "latent_attention":
                H, D, R, VD, L, Q = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
                dense(W * (Q + L + R) + Q * H * (D + R) + L * H * (D + VD) + H * VD * W)
                attention(H, D + R, VD, L + R, m["mask"]["size"])
            elif layer["type"] == "attention":
                H, G, D, VD = (m[k] for k in ("heads", "kv_heads", "dim", "vdim"))
                dense(W * H * D + (0 if "kv_from" in m else W * G * (D + VD)) + H * VD * W)
                attention(H, D, VD, G * (D + VD), m["mask"]["size"])
            elif layer["type"] == "parallel":
                a, d = m["left"], m["right"]
                H, G, D, VD = (a[k] for k in ("heads", "kv_heads", "dim", "vdim"))
                dense(W * (H * D + G * (D + VD) + H * VD) + H * VD * W)
                attention(H, D, VD, G * (D + VD))
                inner = d["heads"] * d["dim"]
                dense(W * 5 * inner + inner * W)
                flops += 10.0 * rows * inner * d["dim"]
                cache += 2.0 * outs * inner * d["dim"] * 4 / elem
            else:
                inner, vals = m["heads"] * m["dim"], m["heads"] * m["vdim"]
                dense(W * (2 * inner + 2 * vals) + vals * W)
                flops += 6.0 * rows * inner * m["vdim"]
                cache += 2.0 * outs * inner * m["vdim"] * 4 / elem
            mlp = layer["mlp"]
            if mlp["kind"] == "dense":
                dense(2 * W * mlp["ff"])
            else:
                dense(W * (mlp["router"]["experts"] + 1) + 3 * W * mlp["shared"]["ff"])
                experts(mlp["router"]["experts"], mlp["router"]["top"], 3 * W * mlp["expert"]["ff"])
    weights += W * V + rows * W                  # the head, the embedding's rows
    flops += 2.0 * outs * W * V
    return elem * (weights + cache) + 4.0 * outs * V, flops


def work(case: dict) -> dict:
    sizes = lengths(case)
    total_bytes, total_flops = model_work(case, sizes)
    if case["kind"] == "turn":
        for k in range(int(case["new"])):
            b, f = model_work(case, [(n + k, 1) for _, n in sizes])
            total_bytes, total_flops = total_bytes + b, total_flops + f
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case: dict) -> dict:
    """About four times what the outputs move by when the products' sums are put in another order (the CUDA-core products in
    place of the tensor cores': LFM2 1.3e-3, Puripel 2.0e-3, Sebilorn 7.3e-3; 32-bit: 4.4e-7 from the exact values)."""
    if case["dtype"] == "float32":
        return {"rel": 4e-6}
    return {"rel": {"lfm2": 5e-3, "puripel": 8e-3, "sebilorn": 0.029}[case["model"].split("-")[0]]}


# ---- the same in 64 bits ----

def unit_rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def turn_halves(x, positions, freqs, sign=1.0):
    """Entries i and i + d/2 of x's last axis (d = 2 len(freqs)) turn by sign * position * freqs[i]."""
    half = freqs.numel()
    a = sign * positions.double()[:, None] * freqs
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def turn_pairs(x, positions, freqs):
    """Entries 2i and 2i + 1 of x [T, heads, d] turn by position * freqs[i]."""
    a = positions.double()[:, None] * freqs
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def powers(base, dims):
    return base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=DEVICE) / dims)


def attend(q, k, v, scale, window=None, keep=0, cap=None):
    """Causal softmax attention [T, H, .] over [T, G, .], a block of query rows at a time."""
    T, H, _ = q.shape
    g = H // k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    block = max(16, (1 << 27) // (T * H))
    j = torch.arange(T, device=q.device)
    for lo in range(0, T, block):
        hi = min(T, lo + block)
        qb = q[lo:hi].reshape(hi - lo, -1, g, q.shape[2])
        s = torch.einsum("ikgd,jkd->kgij", qb, k[:hi]) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        i = torch.arange(lo, hi, device=q.device)[:, None]
        hidden = j[:hi] > i
        if window is not None:
            hidden |= (i - j[:hi] >= window) & (j[:hi] >= keep)
        s.masked_fill_(hidden, -math.inf)
        out[lo:hi] = torch.einsum("kgij,jkd->ikgd", torch.softmax(s, -1), v[:hi]).reshape(hi - lo, H, -1)
    return out


def conv_rows(x, taps, parts):
    """A causal depthwise convolution of every sequence's rows; the last tap multiplies the row itself."""
    out = torch.zeros_like(x)
    n = taps.shape[1]
    for a, b in parts:
        for k in range(n):
            back = n - 1 - k
            if b - a > back:
                out[a + back:b] += x[a:b - back] * taps[:, k]
    return out


def routed(n, ids, weights, expert):
    out = torch.zeros_like(n)
    for e in torch.unique(ids).tolist():
        rows, slot = torch.where(ids == e)
        out.index_add_(0, rows, expert(n[rows], e) * weights[rows, slot, None])
    return out


def exact_lfm2(raw, read, tokens, parts, wanted):
    eps, top = raw["norm_eps"], raw["num_experts_per_tok"]
    D, freqs = raw["head_dim"], powers(raw["rope_parameters"]["rope_theta"], raw["head_dim"])
    F = torch.nn.functional

    def mlp(x, p):
        return (F.silu(x @ read(p + "w1.weight").T) * (x @ read(p + "w3.weight").T)) @ read(p + "w2.weight").T

    x = read("embed_tokens.weight")[tokens]
    for i, kind in enumerate(raw["layer_types"]):
        p = f"layers.{i}."
        n = unit_rms(x, eps) * read(p + "operator_norm.weight")
        if kind == "full_attention":
            a = p + "self_attn."
            q, k, v = ((n @ read(a + f"{c}_proj.weight").T).view(len(n), -1, D) for c in "qkv")
            q = unit_rms(q, eps) * read(a + "q_layernorm.weight")
            k = unit_rms(k, eps) * read(a + "k_layernorm.weight")
            o = torch.empty_like(q)
            for lo, hi in parts:
                at = torch.arange(hi - lo, device=DEVICE)
                o[lo:hi] = attend(turn_halves(q[lo:hi], at, freqs), turn_halves(k[lo:hi], at, freqs), v[lo:hi], D ** -0.5)
            x = x + o.flatten(1) @ read(a + "out_proj.weight").T
            del q, k, v, o
        else:
            c = p + "conv."
            B, C, u = (n @ read(c + "in_proj.weight").T).chunk(3, -1)
            y = C * conv_rows(B * u, read(c + "conv.weight").reshape(x.shape[1], -1), parts)
            x = x + y @ read(c + "out_proj.weight").T
            del B, C, u, y
        n = unit_rms(x, eps) * read(p + "ffn_norm.weight")
        f = p + "feed_forward."
        if i < raw["num_dense_layers"]:
            x = x + torch.cat([mlp(part, f) for part in n.split(16384)])
        else:
            s = torch.sigmoid(n @ read(f + "gate.weight").T)
            ids = torch.sort(s + read(f + "expert_bias"), dim=-1, descending=True, stable=True).indices[:, :top]
            w = s.gather(1, ids)
            x = x + routed(n, ids, w / (w.sum(-1, keepdim=True) + 1e-6), lambda r, e: mlp(r, f"{f}experts.{e}."))
    return (unit_rms(x[wanted], eps) * read("embedding_norm.weight")) @ read("embed_tokens.weight").T


def exact_puripel(raw, read, tokens, parts, wanted):
    eps, F = raw["norm"]["eps"], torch.nn.functional

    def expert(x, p, limit):
        g = (x @ read(p + "gate").T).clamp(max=limit)
        return (g * torch.sigmoid(1.702 * g) * ((x @ read(p + "up").T).clamp(-limit, limit) + 1)) @ read(p + "down").T

    x = read("embed")[tokens]
    for i, layer in enumerate(raw["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        n, mix = unit_rms(x, eps) * read(p + "norm1"), p + "mix."
        if layer["type"] == "mamba2":
            H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            inner = H * P
            z, xbc, dt = (n @ read(mix + "in").T).split([inner, inner + 2 * G * N, H], -1)
            xbc = F.silu(conv_rows(xbc, read(mix + "conv"), parts) + read(mix + "conv.b"))
            u, B, C = xbc.split([inner, G * N, G * N], -1)
            u = u.reshape(-1, H, P)
            B, C = (t.reshape(-1, G, N).repeat_interleave(H // G, 1) for t in (B, C))
            dt = F.softplus(dt + read(mix + "dt_bias"))
            decay = torch.exp(-torch.exp(read(mix + "A_log")) * dt)
            y = torch.empty_like(u)
            for lo, hi in parts:
                S = torch.zeros(H, N, P, dtype=torch.float64, device=DEVICE)
                for t in range(lo, hi):
                    S = decay[t, :, None, None] * S + (dt[t, :, None] * B[t])[:, :, None] * u[t, :, None, :]
                    y[t] = (S * C[t, :, :, None]).sum(1)
            y = (y + read(mix + "D")[:, None] * u).flatten(1) * F.silu(z)
            parts_of = m["norm_groups"]
            d = (unit_rms(y.view(len(y), parts_of, -1), eps).flatten(1) * read(mix + "norm")) @ read(mix + "o").T
        else:
            H, D, R, VD, L = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
            freqs = powers(m["rot"]["base"], m["rot"]["dims"])
            q = ((unit_rms(n @ read(mix + "dq").T, eps) * read(mix + "dq.norm")) @ read(mix + "uq").T).view(-1, H, D + R)
            kv = n @ read(mix + "dkv").T
            c = unit_rms(kv[:, :L], eps) * read(mix + "dkv.norm")
            k, v = (c @ read(mix + "uk").T).view(-1, H, D), (c @ read(mix + "uv").T).view(-1, H, VD)
            o = torch.empty_like(v)
            for lo, hi in parts:
                at = torch.arange(hi - lo, device=DEVICE)
                kr = turn_pairs(kv[lo:hi, None, L:], at, freqs).expand(-1, H, -1)
                qq = torch.cat([q[lo:hi, :, :D], turn_pairs(q[lo:hi, :, D:], at, freqs)], -1)
                o[lo:hi] = attend(qq, torch.cat([k[lo:hi], kr], -1), v[lo:hi], m["scale"], m["mask"]["size"])
            d = o.flatten(1) @ read(mix + "o").T
        x = x + unit_rms(d, eps) * read(p + "norm1b")
        n, f, mlp = unit_rms(x, eps) * read(p + "norm2"), p + "mlp.", layer["mlp"]
        r = mlp["router"]
        s = torch.sigmoid(n @ read(f + "router").T)
        choice = s + read(f + "correction")
        count, keep = r["groups"]["count"], r["groups"]["keep"]
        by_group = choice.view(len(n), count, -1)
        best = by_group.topk(2, -1).values.sum(-1).topk(keep, -1).indices
        open_ = torch.zeros(len(n), count, dtype=torch.bool, device=DEVICE).scatter_(1, best, True)
        choice = by_group.masked_fill(~open_[:, :, None], -math.inf).flatten(1)
        ids = torch.sort(choice, dim=-1, descending=True, stable=True).indices[:, :r["top"]]
        w = s.gather(1, ids)
        d = routed(n, ids, w / (w.sum(-1, keepdim=True) + 1e-20) * r["scale"],
                   lambda rows, e: expert(rows, f"{f}e{e}.", mlp["expert"]["limit"]))
        d = d + torch.sigmoid(n @ read(f + "shared.sg").T) * expert(n, f + "shared.", mlp["shared"]["limit"])
        x = x + unit_rms(d, eps) * read(p + "norm2b")
    return (unit_rms(x[wanted], eps) * read("final.norm")) @ read("embed").T


def exact_sebilorn(raw, read, tokens, parts, wanted):
    eps, F = raw["norm"]["eps"], torch.nn.functional

    def layer_norm(x, name):
        return F.layer_norm(x, (x.shape[-1],), read(name), read(name + ".b"), eps)

    def frequencies(rot):
        f, sc = powers(rot["base"], rot["dims"]), rot.get("scaling")
        if not sc:
            return f
        wave = 2.0 * math.pi / f
        s = ((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)
        return (1.0 - s) * f / sc["factor"] + s * f

    def scan(q, k, v, decay, erase=None):
        """S <- decay S (- (a u)(u^T S)) + k v^T, o = S^T q, every sequence from zero."""
        o = torch.empty_like(v)
        for lo, hi in parts:
            S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=torch.float64, device=DEVICE)
            for t in range(lo, hi):
                new = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
                if erase is not None:
                    a, u = erase
                    new = new - (a[t] * u[t])[:, :, None] * (u[t][:, :, None] * S).sum(1)[:, None, :]
                S = new
                o[t] = (S * q[t][:, :, None]).sum(1)
        return o

    x = read("embed")[tokens] * raw["embedding"]["scale"]
    at = torch.cat([torch.arange(b - a, device=DEVICE) for a, b in parts])
    kept = {}
    for i, layer in enumerate(raw["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        n, mix = layer_norm(x, p + "norm1"), p + "mix."

        def heads(name, dim):
            return (n @ read(name).T).view(len(n), -1, dim)
        if layer["type"] == "attention":
            D, VD = m["dim"], m["vdim"]
            f, fv = frequencies(m["rot"]), powers(m["rot"]["base"], m["vdim"])
            src = m.get("kv_from")
            if src is None:
                kept[i] = turn_halves(heads(mix + "k", D), at, f), turn_halves(heads(mix + "v", VD), at, fv)
            k, v = kept[i if src is None else src]
            q = turn_halves(heads(mix + "q", D), at, f)
            o = torch.cat([attend(q[a:b], k[a:b], v[a:b], m["scale"], m["mask"]["size"], m["mask"]["keep_first"], m["softcap"])
                           for a, b in parts])
            x = x + turn_halves(o, at, fv, -1.0).flatten(1) @ read(mix + "o").T
        elif layer["type"] == "parallel":
            left, right, d = mix + "left.", mix + "right.", m["right"]["dim"]
            f = frequencies(m["left"]["rot"])
            q, k = (turn_halves(heads(left + c, m["left"]["dim"]), at, f) for c in "qk")
            v = heads(left + "v", m["left"]["vdim"])
            o = torch.cat([attend(q[a:b], k[a:b], v[a:b], m["left"]["scale"]) for a, b in parts]).flatten(1)
            a_out = (o * torch.sigmoid(n @ read(left + "g").T)) @ read(left + "o").T
            r, k, v = (heads(right + c, d) for c in "rkv")
            decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(n @ read(right + "w1").T) @ read(right + "w2").T
                                                              + read(right + "w0"))).view_as(k)
            a = torch.sigmoid(n @ read(right + "a").T + read(right + "a.b")).view_as(k)
            u = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            o = unit_rms(scan(r, k, v, decay, (a, u)), eps).flatten(1) * read(right + "norm")
            d_out = (o * torch.sigmoid(n @ read(right + "g").T)) @ read(right + "o").T
            x = x + m["left_scale"] * a_out + m["right_scale"] * d_out
        else:
            q, k, v = F.silu(heads(mix + "q", m["dim"])), F.silu(heads(mix + "k", m["dim"])), F.silu(heads(mix + "v", m["vdim"]))
            decay = torch.tensor(m["decay"], dtype=torch.float64, device=DEVICE)[None, :, None].expand_as(k)
            o = unit_rms(scan(q, k, v, decay).flatten(1), eps) * read(mix + "norm")
            x = x + (o * torch.sigmoid(n @ read(mix + "g").T)) @ read(mix + "o").T
        z = F.relu(layer_norm(x, p + "norm2") @ read(p + "mlp.up").T)
        x = x + (z * z) @ read(p + "mlp.down").T
    cap = raw["logit_softcap"]
    return cap * torch.tanh(layer_norm(x[wanted], "final.norm") @ read("head").T / cap)


def exact(case: dict, seed: int):
    raw, stored = raw_config(case), weights_of(case, seed)
    texts, sizes = draw_tokens(case, seed), lengths(case)
    parts, wanted, at = [], [], 0
    for text, (c, n) in zip(texts, sizes):
        parts.append((at, at + len(text)))
        wanted.append(at + c + n - 1)
        at += len(text)
    steps = 1 + (int(case["new"]) if case["kind"] == "turn" else 0)
    rows = torch.tensor([w + k for k in range(steps) for w in wanted], device=DEVICE)
    tokens = torch.tensor(sum(texts, []), device=DEVICE)
    model = {"lfm2": exact_lfm2, "puripel": exact_puripel, "sebilorn": exact_sebilorn}[case["model"].split("-")[0]]
    with torch.no_grad():
        logits = model(raw, lambda name: stored[name].double(), tokens, parts, rows)
    logits = logits.view(steps, len(sizes), -1)
    return logits[0] if case["kind"] == "step" else list(logits)
