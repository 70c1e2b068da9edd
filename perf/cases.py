"""Workloads of the engine, from a model folder to logits and sampled tokens.

A case is one batch of requests served by the step function: the prompts run in portions under a token
budget, beside single tokens of the requests that already decode, as the scheduler grants them; every
step's logits go through the sampler on the device.  The tokens a request continues with are given (the
text of a recorded conversation), so that a pass is the same work and has the same outputs every time.
The engine comes from a model folder with random weights and keeps serving, as a server does; the
requests of a pass begin and end within it.

Fields of a case: ``model`` and ``dtype``; ``requests`` prompts of ``shortest`` to ``longest`` tokens; ``new``
tokens per request (1: the pass ends with the first token); ``sampling``: "greedy", "default" (temperature
1, repetition penalty), "temperature" (0.8) or "top" (0.8 with top-k and top-p).

Outputs of a pass: ``tokens`` sampled at every place that wants one, in the order of the steps; ``first`` and
``last``: the logits after each request's prompt and after its last but one new token (``last`` is there when ``new`` > 1)."""
from __future__ import annotations

import functools
import json
import math
import os
import random
import shutil
import tempfile
import zlib

import numpy as np
import torch

_QWEN3 = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3")
_LARGE = dict(_QWEN3, vocab_size=151936, rms_norm_eps=1e-6, rope_theta=1e6, head_dim=128, num_key_value_heads=8,
              max_position_embeddings=40960)

# The five sets of shapes that the engine is configured, tested and benchmarked for; of the 64 layers of the
# largest four are kept (its weights would take minutes to write), every layer as wide as in the full model.
MODELS = {
    "tiny-a": dict(_QWEN3, hidden_size=64, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=4, head_dim=16,
                   intermediate_size=128, vocab_size=256, rms_norm_eps=1e-6, rope_theta=1e4, tie_word_embeddings=True,
                   max_position_embeddings=128),
    "tiny-b": dict(_QWEN3, hidden_size=96, num_hidden_layers=3, num_attention_heads=8, num_key_value_heads=2, head_dim=32,
                   intermediate_size=160, vocab_size=384, rms_norm_eps=1e-5, rope_theta=1e6, tie_word_embeddings=False,
                   max_position_embeddings=256),
    "0.6b": dict(_LARGE, hidden_size=1024, num_hidden_layers=28, num_attention_heads=16, intermediate_size=3072,
                 tie_word_embeddings=True),
    "8b": dict(_LARGE, hidden_size=4096, num_hidden_layers=36, num_attention_heads=32, intermediate_size=12288,
               tie_word_embeddings=False),
    "32b-4": dict(_LARGE, hidden_size=5120, num_hidden_layers=4, num_attention_heads=64, intermediate_size=25600,
                  tie_word_embeddings=False),
}

# How each model is served: context, page size (0: the engine's own choice), most requests, tokens per step.
ENGINES = {
    ("tiny-a", "float32"): dict(max_model_len=128, block_size=16, max_num_seqs=4, max_num_batched_tokens=128),
    ("tiny-b", "float32"): dict(max_model_len=256, block_size=8, max_num_seqs=8, max_num_batched_tokens=32),
    ("0.6b", "float32"): dict(max_model_len=2048, block_size=16, max_num_seqs=4, max_num_batched_tokens=1024, num_blocks=512),
    ("0.6b", "bfloat16"): dict(max_model_len=16384, block_size=0, max_num_seqs=128, max_num_batched_tokens=2048, num_blocks=3072),
    ("8b", "bfloat16"): dict(max_model_len=4096, block_size=0, max_num_seqs=64, max_num_batched_tokens=4096, num_blocks=640),
    ("32b-4", "bfloat16"): dict(max_model_len=8192, block_size=16, max_num_seqs=16, max_num_batched_tokens=4096, num_blocks=4096),
}


def _case(model, dtype, requests, shortest, longest, new, sampling="greedy"):
    return dict(model=model, dtype=dtype, requests=requests, shortest=shortest, longest=longest, new=new, sampling=sampling)


def listed():
    return [
        # the smallest calls: a handful of launches on a few kilobytes, in true 32-bit
        dict(_case("tiny-a", "float32", 3, 5, 31, 16), name="tiny a: 3 requests"),
        # prompts cut by a budget of 32 tokens, sampled with a repetition penalty
        dict(_case("tiny-b", "float32", 5, 1, 100, 24, "default"), name="tiny b: 5 requests sampled"),
        # a 32-bit run of a real model, what a bfloat16 deployment is checked against
        dict(_case("0.6b", "float32", 2, 77, 150, 12), name="0.6b float32: 2 requests"),
        # one user at a small model: latency of a step
        dict(_case("0.6b", "bfloat16", 1, 61, 61, 64), name="0.6b: 1 user"),
        # a burst of requests of all lengths: portions of prompts beside decoded tokens
        dict(_case("0.6b", "bfloat16", 96, 1, 1024, 24), name="0.6b: burst of 96"),
        # two long documents and a summary of each
        dict(_case("0.6b", "bfloat16", 2, 9001, 12000, 32), name="0.6b: 2 long documents"),
        # one user, a page of prompt
        dict(_case("8b", "bfloat16", 1, 512, 512, 48), name="8b: 1 user"),
        # the benchmark's batch
        dict(_case("8b", "bfloat16", 8, 512, 512, 48), name="8b: 8 requests"),
        # a busy server with short prompts
        dict(_case("8b", "bfloat16", 64, 33, 200, 32), name="8b: 64 requests"),
        # time to the first token of a long and of a short prompt
        dict(_case("8b", "bfloat16", 1, 2048, 2048, 1), name="8b: prompt of 2048"),
        dict(_case("8b", "bfloat16", 1, 203, 203, 1, "top"), name="8b: prompt of 203"),
        # wide layers, pages of 16
        dict(_case("32b-4", "bfloat16", 6, 1500, 2500, 16), name="32b 4 layers: 6 requests"),
    ]


def draw(rng):
    def log(low, high):
        return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))

    model, dtype = rng.choice(list(ENGINES) + [("8b", "bfloat16")] * 3 + [("0.6b", "bfloat16")] * 2)
    sampling = rng.choice(["greedy", "greedy", "greedy", "default", "temperature", "top"])
    if model.startswith("tiny"):
        requests, longest, new = rng.randint(1, 4 if model == "tiny-a" else 8), log(2, 100), log(2, 24)
    elif dtype == "float32":
        requests, longest, new = rng.randint(1, 4), log(8, 200), log(1, 12)
    elif model == "0.6b":
        requests = log(1, 128)
        longest, new = log(16, min(12000, 48000 // requests)), log(2, 48)
    elif model == "8b":
        requests = log(1, 64)
        longest, new = log(16, min(4000, 8192 // requests)), log(1, 32)
    else:
        requests = log(1, 12)
        longest, new = log(64, min(6000, 12000 // requests)), log(1, 16)
    return _case(model, dtype, requests, max(1, int(longest * rng.uniform(0.2, 1.0))), longest, new, sampling)


# ----------------------------------------------------------------------------- what a case asks for
def _lengths(case):
    """Prompt lengths, spread evenly over their range, in an order that has nothing to do with their size."""
    n, low, high = case["requests"], case["shortest"], case["longest"]
    lengths = [high if n == 1 else low + (high - low) * i // (n - 1) for i in range(n)]
    random.Random(n * 31 + high).shuffle(lengths)
    return lengths


def _plan(case):
    """Steps of (request, first token, tokens), as continuous batching grants them: the running requests in the
    order they came, then new ones, until the budget is used."""
    engine = ENGINES[(case["model"], case["dtype"])]
    lengths, new = _lengths(case), case["new"]
    done, steps, first = [0] * len(lengths), [], 0
    while first < len(lengths):
        left, step = engine["max_num_batched_tokens"], []
        for r in range(first, len(lengths)):
            if left == 0 or len(step) == engine["max_num_seqs"]:
                break
            if done[r] < lengths[r]:
                n = min(left, lengths[r] - done[r])
            elif done[r] < lengths[r] + new - 1:
                n = 1
            else:
                continue
            step.append((r, done[r], n))
            left -= n
        for r, _, n in step:
            done[r] += n
        steps.append(step)
        while first < len(lengths) and done[first] == lengths[first] + new - 1:
            first += 1
    return steps


def _tokens(case, seed):
    """Every request's prompt and the tokens it goes on with."""
    g = torch.Generator().manual_seed(int(seed))
    vocab = MODELS[case["model"]]["vocab_size"]
    return [torch.randint(0, vocab, (n + case["new"],), generator=g).tolist() for n in _lengths(case)]


def _wanted(case):
    """(request, place, is its first, is its last) of every sampled place, in the order of the steps."""
    lengths = _lengths(case)
    return [[(r, at + n - 1, at + n == lengths[r], case["new"] > 1 and at + n == lengths[r] + case["new"] - 1)
             for r, at, n in step if at + n >= lengths[r]] for step in _plan(case)]


# ----------------------------------------------------------------------------- weights
def _shapes(model):
    c = MODELS[model]
    h, d, ff = c["hidden_size"], c["head_dim"], c["intermediate_size"]
    q, kv = c["num_attention_heads"] * d, c["num_key_value_heads"] * d
    shapes = {"model.embed_tokens.weight": (c["vocab_size"], h)}
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        shapes.update({p + "input_layernorm.weight": (h,), p + "self_attn.q_proj.weight": (q, h),
                       p + "self_attn.k_proj.weight": (kv, h), p + "self_attn.v_proj.weight": (kv, h),
                       p + "self_attn.q_norm.weight": (d,), p + "self_attn.k_norm.weight": (d,),
                       p + "self_attn.o_proj.weight": (h, q), p + "post_attention_layernorm.weight": (h,),
                       p + "mlp.gate_proj.weight": (ff, h), p + "mlp.up_proj.weight": (ff, h),
                       p + "mlp.down_proj.weight": (h, ff)})
    shapes["model.norm.weight"] = (h,)
    if not c["tie_word_embeddings"]:
        shapes["lm_head.weight"] = (c["vocab_size"], h)
    return shapes


def _weight(model, name, dtype, device):
    """One tensor of the model: rows scaled by their length and the projections into the residual stream by the number of
    sub-layers too, as models are initialised; heads that attend to some keys more than to others; a head that
    has a favourite token, as trained models mostly do (so that a sampled token is no toss-up between near-equal ones)."""
    c, shape = MODELS[model], _shapes(model)[name]
    g = torch.Generator(device=device).manual_seed(zlib.crc32(name.encode()))
    w = torch.empty(shape, dtype=torch.float32, device=device)
    if len(shape) == 1:
        w = (1.4 if name.endswith(("q_norm.weight", "k_norm.weight")) else 1) * (1 + w.uniform_(-0.1, 0.1, generator=g))
    elif name == "model.embed_tokens.weight":
        w.normal_(0.0, 0.05, generator=g)
    elif name == "lm_head.weight":
        w = w.normal_(0.0, 0.02, generator=g) + 0.4 * _weight(model, "model.embed_tokens.weight", dtype, device).float()
    elif name.endswith(("o_proj.weight", "down_proj.weight")):
        w.normal_(0.0, 0.1 / math.sqrt(shape[1] * 2 * c["num_hidden_layers"]), generator=g)
    else:
        w.normal_(0.0, 1 / math.sqrt(shape[1]), generator=g)
    return w.to(getattr(torch, dtype))


def _write_folder(model, dtype, folder):
    """config.json and the weights in the safetensors format: the length of a header in JSON, the header, the bytes."""
    size = 4 if dtype == "float32" else 2
    header, at = {}, 0
    for name, shape in _shapes(model).items():
        n = size * math.prod(shape)
        header[name] = {"dtype": "F32" if size == 4 else "BF16", "shape": list(shape), "data_offsets": [at, at + n]}
        at += n
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(dict(MODELS[model], torch_dtype=dtype), f)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(np.array([len(text)], dtype="<u8").tobytes() + text)
        for name, shape in _shapes(model).items():
            w = _weight(model, name, dtype, "cuda").view(torch.uint8 if len(shape) == 1 else torch.int16)
            w.cpu().numpy().tofile(f)


@functools.cache
def _engine(model, dtype):
    """The serving engine: built once from a model folder, with its graphs captured, and kept."""
    from tinyserve_b200 import EngineConfig
    from tinyserve_b200.engine.runner import ModelRunner
    from tinyserve_b200.sampling import Sampler
    need = 4 * sum(math.prod(s) for s in _shapes(model).values())
    shm = "/dev/shm" if os.path.isdir("/dev/shm") and shutil.disk_usage("/dev/shm").free > 2 * need else None
    with tempfile.TemporaryDirectory(dir=shm) as folder:
        _write_folder(model, dtype, folder)
        runner = ModelRunner(EngineConfig(model=folder, dtype=dtype, **ENGINES[(model, dtype)]))
    runner.capture_decode_graphs()
    return runner, Sampler(0, runner.device, runner.cfg.max_num_seqs)


def _sampling(case):
    from tinyserve_b200 import SamplingParams
    return SamplingParams(max_tokens=case["new"], ignore_eos=True, **{
        "greedy": dict(temperature=0.0, repetition_penalty=1.0),
        "default": {},
        "temperature": dict(temperature=0.8, repetition_penalty=1.0),
        "top": dict(temperature=0.8, top_k=50, top_p=0.95, repetition_penalty=1.0)}[case["sampling"]])


# ----------------------------------------------------------------------------- a pass
def prepare(case, seed):
    runner, sampler = _engine(case["model"], case["dtype"])
    wanted = _wanted(case)

    def rows(step, which):
        """Rows of the step's logits to keep: None (no row), True (all of them) or their indices."""
        at = [i for i, w in enumerate(step) if w[which]]
        return None if not at else True if len(at) == len(step) else torch.tensor(at, device=runner.device)

    return {"runner": runner, "sampler": sampler, "tokens": _tokens(case, seed), "lengths": _lengths(case), "params": _sampling(case),
            "steps": _plan(case), "wanted": wanted, "keep": [(rows(s, 2), rows(s, 3)) for s in wanted]}


@torch.inference_mode()
def run(state):
    from tinyserve_b200.engine.batch import StepEntry
    from tinyserve_b200.engine.scheduler import Request
    runner, sampler, texts = state["runner"], state["sampler"], state["tokens"]
    manager = runner.manager
    requests = [Request(f"request {r}", text[:n], state["params"]) for r, (text, n) in enumerate(zip(texts, state["lengths"]))]
    sampled, kept = [], ([], [])
    for step, wanted, keep in zip(state["steps"], state["wanted"], state["keep"]):
        wants = {w[0] for w in wanted}
        entries = []
        for r, at, n in step:
            if at == 0:
                manager.begin(requests[r].request_id)
            entries.append(StepEntry(requests[r].request_id, texts[r][at:at + n], [n - 1] if r in wants else []))
        logits = runner.step(entries)
        if not wanted:
            continue
        for out, which in zip(kept, keep):
            if which is not None:
                out.append(logits.clone() if which is True else logits[which])
        sampled.append(sampler(logits, [requests[w[0]] for w in wanted]))
        for r, at, _, _ in wanted:
            requests[r].token_ids.append(texts[r][at + 1])
            if at + 2 == len(texts[r]):
                manager.free(requests[r].request_id)
    out = {"tokens": torch.cat(sampled), "first": torch.cat(kept[0])}
    if kept[1]:
        out["last"] = torch.cat(kept[1])
    return out


def work(case):
    """Per step: every weight read once (of the embedding the rows of the step's tokens), the keys and values of its requests
    read once and the new ones written, the logits written in 32-bit; the multiply-adds of the products and of causal attention."""
    c, size = MODELS[case["model"]], 4 if case["dtype"] == "float32" else 2
    h, d, ff, layers, vocab = c["hidden_size"], c["head_dim"], c["intermediate_size"], c["num_hidden_layers"], c["vocab_size"]
    heads, kv = c["num_attention_heads"], c["num_key_value_heads"]
    layer = (2 * heads + 2 * kv) * d * h + 3 * ff * h
    total_bytes = total_flops = 0
    for step, wanted in zip(_plan(case), _wanted(case)):
        tokens = sum(n for _, _, n in step)
        keys = sum(at + n for _, at, n in step)
        pairs = sum(n * at + n * (n + 1) // 2 for _, at, n in step)
        total_bytes += size * (layers * layer + tokens * h + layers * 2 * kv * d * (keys + tokens))
        total_flops += 2 * layers * layer * tokens + 4 * layers * heads * d * pairs
        if wanted:
            total_bytes += size * vocab * h + 4 * vocab * len(wanted)
            total_flops += 2 * vocab * h * len(wanted)
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "differ": 0.01}
    return {"rel": 2e-2, "differ": 0.01}


# ----------------------------------------------------------------------------- the same in 64 bits
def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, angles):
    a, b = x.chunk(2, -1)
    cos, sin = angles.cos()[:, None], angles.sin()[:, None]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, rows=1024):
    """Causal attention of one request: q [T, heads, d], k and v [T, kv heads, d]."""
    T, heads, d = q.shape
    q = q.view(T, k.shape[1], -1, d)
    out = torch.empty_like(q)
    for at in range(0, T, rows):
        to = min(T, at + rows)
        for g in range(k.shape[1]):
            s = torch.einsum("tnd,sd->nts", q[at:to, g], k[:to, g]) * d ** -0.5
            s.masked_fill_(torch.arange(to, device=q.device)[None] > torch.arange(at, to, device=q.device)[:, None], -math.inf)
            out[at:to, g] = torch.einsum("nts,sd->tnd", s.softmax(-1), v[:to, g])
    return out.reshape(T, heads * d)


@torch.inference_mode()
def exact(case, seed):
    c, dev = MODELS[case["model"]], "cuda"
    d, eps = c["head_dim"], c["rms_norm_eps"]

    def w(name):
        return _weight(case["model"], name, case["dtype"], dev).double()

    texts = [t[:-1] for t in _tokens(case, seed)]          # the last token is never run
    starts = np.cumsum([0] + [len(t) for t in texts]).tolist()
    ids = torch.tensor(sum(texts, []), device=dev)
    embedding = _weight(case["model"], "model.embed_tokens.weight", case["dtype"], dev)
    x = embedding[ids].double()
    positions = torch.cat([torch.arange(len(t), device=dev) for t in texts]).double()
    angles = positions[:, None] * c["rope_theta"] ** (-torch.arange(0, d, 2, device=dev).double() / d)
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        y = _norm(x, w(p + "input_layernorm.weight"), eps)
        q, k, v = (torch.mm(y, w(p + f"self_attn.{n}_proj.weight").T).view(len(ids), -1, d) for n in "qkv")
        q = _rotate(_norm(q, w(p + "self_attn.q_norm.weight"), eps), angles)
        k = _rotate(_norm(k, w(p + "self_attn.k_norm.weight"), eps), angles)
        o = torch.cat([_attend(q[a:b], k[a:b], v[a:b]) for a, b in zip(starts, starts[1:])])
        x += o @ w(p + "self_attn.o_proj.weight").T
        y = _norm(x, w(p + "post_attention_layernorm.weight"), eps)
        y = torch.nn.functional.silu(y @ w(p + "mlp.gate_proj.weight").T) * (y @ w(p + "mlp.up_proj.weight").T)
        x += y @ w(p + "mlp.down_proj.weight").T
    places = [(starts[r] + at, first, last) for step in _wanted(case) for r, at, first, last in step]
    x = _norm(x[torch.tensor([at for at, _, _ in places], device=dev)], w("model.norm.weight"), eps)
    head = (embedding if c["tie_word_embeddings"] else _weight(case["model"], "lm_head.weight", case["dtype"], dev)).double()
    tokens = torch.cat([(rows @ head.T).argmax(-1) for rows in x.split(256)])

    def logits(which):
        return x[torch.tensor([i for i, place in enumerate(places) if place[which]], device=dev)] @ head.T

    out = {"tokens": tokens if case["sampling"] == "greedy" else None, "first": logits(1)}
    if case["new"] > 1:
        out["last"] = logits(2)
    return out
