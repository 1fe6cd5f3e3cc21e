"""What a user of this library has it do, as cases that can be timed and compared.

Every case goes through ``espresso_b200.runtime.DecodeEngine``.  The models are the shapes of
``espresso_b200.model_config`` (the 8B shape also cut to fewer layers: its layers are all alike) with random weights,
arranged so that they decide like a trained model: the LM head row of token ``t + shift`` is the embedding of ``t``, the
residual stream keeps the embedding, and so the greedy choice leads the runner-up by far more than any rounding while
the other logits depend on every layer.  Projections back into the residual stream carry the usual 1/sqrt(2 layers).
"""
import dataclasses
import math

import numpy as np
import torch

from espresso_b200 import model_config as mc
from espresso_b200.runtime import DecodeEngine
from espresso_b200.synthetic_device import quantize_q4_0_torch, quantize_q8_0_torch
from espresso_b200.weight_blob import is_matrix, tensor_shapes

MODELS = {"6l": mc.llama_6l, "gpt2": mc.gpt2_117m, "1b": mc.llama_1b, "8b": mc.llama3_8b}
LAYERS = {"6l": 6, "gpt2": 12, "1b": 22, "8b": 32}
BYTES_PER_WEIGHT = {"f16": 2.0, "bf16": 2.0, "q8_0": 34 / 32, "q4_0": 18 / 32}
GPT2_STOP = 50256  # a GPT-2 engine stops on this token, so the streams below never reach it
DRAFT_MISSES = 0.3  # share of tokens after which the draft proposes something else than the target chooses


def _case(name, path, model, kind, seqs, prompt, new, layers=None):
    return {"name": name, "path": path, "model": model, "type": kind, "layers": layers or LAYERS[model], "seqs": seqs,
            "prompt": prompt, "new": new}


def listed():
    return [
        # a chat front end that shows every token as it comes: the smallest calls, one host round trip per token
        _case("stream 6l f16", "stream", "6l", "f16", 1, 16, 32),
        # greedy generation of one sequence on the small model, the default workload of the benchmark
        _case("generate 6l f16", "generate", "6l", "f16", 1, 16, 128),
        # the same with a one-layer draft and exact two-token verification
        _case("two-token 6l f16", "two_token", "6l", "f16", 1, 16, 128),
        # one GPT-2 sequence, an odd prompt
        _case("generate gpt2 f16", "generate", "gpt2", "f16", 1, 37, 64),
        # offline generation over many independent sequences
        _case("batch gpt2 f16", "batch", "gpt2", "f16", 256, 64, 32),
        # a GGUF model on one sequence, in both block types; the second with a longer, ragged context
        _case("generate 1b q8_0", "generate", "1b", "q8_0", 1, 128, 64),
        _case("generate 1b q4_0", "generate", "1b", "q4_0", 1, 401, 64),
        # a GGUF model serving a batch
        _case("batch 1b q8_0", "batch", "1b", "q8_0", 16, 128, 32),
        # a handful of users on a 16-bit model
        _case("few 1b f16", "batch", "1b", "f16", 5, 75, 32),
        # one user of a large bf16 model
        _case("generate 8b bf16", "generate", "8b", "bf16", 1, 60, 24, layers=8),
        # the largest: long prompts for 64 users of the large model, then decode
        _case("batch 8b bf16", "batch", "8b", "bf16", 64, 512, 16),
        # scoring: a long prompt and the logits that follow it
        _case("score 1b f16", "score", "1b", "f16", 1, 1531, 0),
    ]


_SINGLE = (("6l", "f16"), ("gpt2", "f16"), ("1b", "q8_0"), ("1b", "q4_0"), ("8b", "bf16"))
_BATCH = (("6l", "f16"), ("gpt2", "f16"), ("1b", "f16"), ("1b", "q8_0"), ("1b", "q4_0"), ("8b", "bf16"))
_PATHS = {"stream": _SINGLE, "generate": _SINGLE, "two_token": (("6l", "f16"),), "batch": _BATCH, "score": _BATCH}
_MOST_SEQS = {"6l": 256, "gpt2": 256, "1b": 64, "8b": 64}
_MOST_PROMPT = {"6l": 200, "gpt2": 600, "1b": 1600, "8b": 700}


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng):
    most = work(listed()[10])
    while True:
        path = rng.choice(("stream", "generate", "two_token", "batch", "batch", "batch", "score"))
        model, kind = rng.choice(_PATHS[path])
        seqs = _spread(rng, 2, _MOST_SEQS[model]) if path == "batch" else 1
        prompt = _spread(rng, 1, _MOST_PROMPT[model])
        longest = min(128, MODELS[model]().maxSeq - prompt - 1)
        new = 0 if path == "score" else _spread(rng, 4, max(4, min(longest, 32 if model == "8b" or path == "stream" else 128)))
        layers = _spread(rng, 2, 12) if model == "8b" else LAYERS[model]
        case = {"path": path, "model": model, "type": kind, "layers": layers, "seqs": seqs, "prompt": prompt, "new": new}
        w = work(case)
        # several hundred decode steps or a few hundred thousand prompt tokens are the largest case over again
        if w["bytes"] <= most["bytes"] and w["flops"] <= most["flops"] and seqs * prompt <= 40000:
            return case


def _config(case, layers=None):
    cfg = MODELS[case["model"]]()
    n = layers or case["layers"]
    return cfg if n == cfg.nLayer else dataclasses.replace(cfg, nLayer=n, name="%s-%dl" % (cfg.name, n))


def _build(cfg, kind, max_batch, gen, embedding, head_source):
    """An engine with random weights from `gen`; LM head row j points along the embedding of token head_source[j]."""
    dev = embedding.device
    dense_kind = "bf16" if kind == "bf16" else "f16"
    dense = torch.bfloat16 if kind == "bf16" else torch.float16
    eng = DecodeEngine.empty(cfg, max_batch=max_batch)
    back = 1.0 / math.sqrt(2 * cfg.nLayer)
    for name, shape in tensor_shapes(cfg).items():
        leaf = name.rsplit("/", 1)[-1]
        if name == "embeddings/token":
            t = embedding
        elif name == "lm_head":
            t = embedding[head_source] * 0.02
        elif leaf in ("rms_att", "rms_ffn", "rms_final", "ln_1_gamma", "ln_2_gamma", "final_norm_gamma"):
            t = torch.randn(shape, generator=gen, device=dev) * 0.05 + 1.0
        elif leaf == "position":
            t = torch.randn(shape, generator=gen, device=dev) * 0.1
        else:
            std = 0.02 * (back if leaf in ("wo", "w2") else 1.0)
            t = torch.randn(shape, generator=gen, device=dev, dtype=dense) * std
        if is_matrix(name) and kind in ("q8_0", "q4_0"):
            flat = t.float().reshape(-1)
            data, as_kind = (quantize_q8_0_torch if kind == "q8_0" else quantize_q4_0_torch)(flat), kind
        else:
            data, as_kind = t.to(dense).contiguous(), dense_kind
        torch.cuda.synchronize(dev)
        eng.load_tensor(name, as_kind, (data.data_ptr(), data.numel() * data.element_size()))
    eng.finalize()
    return eng


def prepare(case, seed):
    cfg = _config(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    host = np.random.default_rng(seed)
    embedding = torch.randn((cfg.vocab, cfg.dModel), generator=gen, device="cuda", dtype=torch.float16)
    usable = GPT2_STOP if cfg.architecture == "gpt2" else cfg.vocab  # tokens that the streams walk through
    source = torch.arange(cfg.vocab, device="cuda")
    source[:usable] = torch.roll(source[:usable], int(host.integers(1, usable)))
    state = {"case": case, "new": case["new"]}
    state["engine"] = _build(cfg, case["type"], case["seqs"], gen, embedding, source)
    if case["path"] == "two_token":
        other = source.clone()
        missed = torch.randperm(cfg.vocab, generator=gen, device="cuda")[:int(cfg.vocab * DRAFT_MISSES)]
        other[missed] = torch.roll(source[missed], 1)
        state["draft"] = _build(_config(case, layers=1), case["type"], 1, gen, embedding, other)
    prompts = host.integers(0, usable, (case["seqs"], case["prompt"]), dtype=np.uint32)
    state["prompts"] = prompts if case["path"] == "batch" else prompts[0]
    torch.cuda.empty_cache()
    return state


def run(state):
    eng, prompts, new, path = state["engine"], state["prompts"], state["new"], state["case"]["path"]
    if path == "score":
        eng.prefill(prompts)
        return {"logits": eng.logits()}
    if path == "stream":
        shown = []
        eng.generate(prompts, new, on_step=lambda token, index, ms: shown.append(token))
        return {"tokens": np.array(shown, np.int64), "logits": eng.logits()}
    if path == "generate":
        return {"tokens": eng.generate(prompts, new).tokens.astype(np.int64), "logits": eng.logits()}
    if path == "two_token":
        return {"tokens": eng.generate_two_token(state["draft"], prompts, new).tokens.astype(np.int64)}
    tokens, _ = eng.generate_batch(prompts, new)
    return {"tokens": np.stack(tokens).astype(np.int64), "logits": eng.logits(len(tokens) - 1)}


def work(case):
    """The weights once for the prompt and once for every further step, the visible keys and values once per step; two
    operations per weight and token, four per channel and visible position."""
    cfg = _config(case)
    seqs, prompt, new = case["seqs"], case["prompt"], case["new"]
    steps = max(new - 1, 0)
    bpw = BYTES_PER_WEIGHT[case["type"]]
    head = cfg.vocab * cfg.dModel
    layers = (cfg.weight_bytes_per_step(2.0) / 2.0) - head
    kv_token = cfg.kv_bytes_per_visible_token()
    visible = steps * prompt + steps * (steps + 1) / 2
    heads = max(new, 1)  # one pass over the LM head for every token (or for the scores)
    passes = 1 + steps
    extra = 0.0
    if case["path"] == "two_token":
        passes = 1 + steps / (2.0 - DRAFT_MISSES)
        heads = passes
        draft = _config(case, layers=1)
        extra = passes * bpw * draft.weight_bytes_per_step(2.0) / 2.0
    logits_out = 0 if case["path"] == "two_token" else 1
    nbytes = bpw * (passes * layers + (heads + logits_out * (new > 0)) * head) + extra
    nbytes += seqs * kv_token * (prompt + visible + steps) + 4 * cfg.vocab * logits_out + 4 * seqs * (prompt + new)
    tokens = seqs * (prompt + steps)
    att = 4 * cfg.nLayer * cfg.attentionDim * seqs * (prompt * (prompt + 1) / 2 + visible)
    return {"bytes": nbytes, "flops": 2 * layers * tokens + 2 * head * seqs * heads + att}


def tolerance(case):
    # tokens are exact; logits carry the rounding of activations (16 bits, in the weights' type) and of the fp16 cache
    return {"rel": 1.5e-2 if case["type"] == "bf16" else 4e-3, "differ": 0.0}
