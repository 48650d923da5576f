"""The work that speed is measured on: what a program that uses this engine has it do, at the sizes it does it at.

Kinds of cases:
  step      one call of the step function (`ModelRunner.step`): decoded tokens, whole prompts, a portion of a prompt, or any
            mix of them, at the layer sizes of the Llama 3.2 1B, 3.2 3B and 3.1 8B models, full depth, bfloat16
  serve     whole requests of another architecture through the same function: prompts of several lengths in one step, then
            decode steps over all of them, then the release
  experts   a mixture-of-experts feed-forward alone: router, grouping, the experts' products, the sum
  generate  `LLM.generate` in float32: scheduler, step function, sampler, stop rules, tokens to the host
  sample    the sampler alone on given logits

Weights are random, of the distributions that the random-weights mode draws; token ids are uniform.  `exact` holds plain
64-bit versions of the Llama, Karupel and Kutolix decoders and of the experts: whole sequences, no cache, no batch.
"""

from __future__ import annotations

import math
import tempfile
from pathlib import Path

import torch

from liteinfer_b200 import LLM, SamplingParams
from liteinfer_b200.config.registry import resolve
from liteinfer_b200.engine.loading import make_runner
from liteinfer_b200.engine.runner import StepEntry
from liteinfer_b200.parts.model import Model
from liteinfer_b200.parts.registry import build_part
from liteinfer_b200.parts.spec import PartSpec
from liteinfer_b200.sampling.sampler import Sampler
from liteinfer_b200.weights.random_init import write_random_model

DEVICE = "cuda:0"
PAGE = 16               # tokens of a cache page: the engine's default
PORTION = 8192          # most tokens of one step while a cache is filled

# ------------------------------------------------------------------ the models
_ROPE = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
         "original_max_position_embeddings": 8192}
_LLAMA = {"architectures": ["LlamaForCausalLM"], "vocab_size": 128256, "hidden_size": 2048, "intermediate_size": 8192,
          "num_hidden_layers": 16, "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 64, "rms_norm_eps": 1e-5,
          "rope_theta": 500000.0, "rope_scaling": _ROPE, "tie_word_embeddings": True, "max_position_embeddings": 131072,
          "hidden_act": "silu"}
LLAMA = {"1b": _LLAMA,
         "3b": dict(_LLAMA, hidden_size=3072, num_hidden_layers=28, num_attention_heads=24, head_dim=128),
         "8b": dict(_LLAMA, hidden_size=4096, intermediate_size=14336, num_hidden_layers=32, head_dim=128,
                    tie_word_embeddings=False, rope_scaling=dict(_ROPE, factor=8.0))}
# A model for the 32-bit path: small enough to be written to a folder and read back in a second.
SMALL = dict(_LLAMA, vocab_size=16000, hidden_size=768, intermediate_size=2048, num_hidden_layers=6, num_attention_heads=12,
             num_key_value_heads=4)


def _karupel(width: int, ff: int, layers: int, vocab: int) -> dict:
    """Three gated delta-rule layers with heads of 128, then an attention layer, over and over."""
    wide, heads = width // 128, width // 64
    mlp = {"kind": "dense", "ff": ff}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": wide, "kv_heads": wide, "dim": 128, "vdim": 128, "conv": 4}}
    attention = {"type": "attention", "mlp": mlp,
                 "mixer": {"heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 64, "scale": 64 ** -0.5, "v_mix": True,
                           "rot": {"dims": 32, "base": 10000.0, "scaling": {"factor": 2.0}}}}
    return {"architecture": "Karupel", "vocab": vocab, "width": width, "norm": {"eps": 1e-5},
            "layers": [(delta, delta, delta, attention)[i % 4] for i in range(layers)]}


def _kutolix(width: int, ff: int, layers: int, vocab: int) -> dict:
    """Gated attention and latent attention in turn, both within a window; dense feed-forwards (the experts, whose choice
    turns on a rounding, are a case of their own)."""
    heads, mlp = width // 128, {"kind": "dense", "ff": ff}
    attention = {"type": "attention", "mlp": mlp,
                 "mixer": {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                           "mask": {"size": 1024}, "rot": {"dims": 64, "base": 100000.0}}}
    latent = {"type": "latent_attention", "mlp": mlp,
              "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
                        "mask": {"size": 1024},
                        "rot": {"dims": 64, "base": 10000.0,
                                "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    return {"architecture": "Kutolix", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "embedding": {"scale": 2.0},
            "residual_mult": 0.7, "logit_softcap": 30.0, "layers": [(attention, latent)[i % 2] for i in range(layers)]}


def _config(case: dict) -> dict:
    if case["model"] in LLAMA:
        return LLAMA[case["model"]]
    return {"karupel": _karupel, "kutolix": _kutolix}[case["model"]](case["width"], 4 * case["width"], case["layers"], 32000)


# ------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    step = {"kind": "step", "model": "1b", "decodes": 0, "context": 0, "prompts": 0, "longest": 0, "held": 0, "spread": 0.0}
    return [
        # One user in a chat: one token after a short context, nothing to share the weights with.
        dict(step, name="decode_1b_b1", decodes=1, context=611),
        # A few users at long contexts: the setting that the decode rate is quoted at.
        dict(step, name="decode_1b_b8_4k", decodes=8, context=4090, spread=0.05),
        # A full batch of requests of every age, as continuous batching has it at a server.
        dict(step, name="decode_3b_b48", model="3b", decodes=48, context=1500, spread=0.95),
        # A large model, a handful of requests.
        dict(step, name="decode_8b_b3", model="8b", decodes=3, context=5003, spread=0.1),
        # Time to the first token of one prompt.
        dict(step, name="prompt_1b_2048", prompts=1, longest=2048),
        # Several prompts that arrive together, computed in one step of the usual token budget.
        dict(step, name="prompts_3b_ragged", model="3b", prompts=6, longest=1733, spread=0.9),
        # A long prompt that goes in by portions while others decode.
        dict(step, name="mixed_1b", decodes=23, context=700, spread=0.8, prompts=1, longest=509, held=1024),
        # Recurrent layers beside attention: prompts, then decode steps.
        {"kind": "serve", "name": "serve_karupel", "model": "karupel", "width": 2048, "layers": 8, "requests": 8, "longest": 450,
         "spread": 0.85, "steps": 8},
        # Windowed and latent attention: prompts beyond the window, then decode steps.
        {"kind": "serve", "name": "serve_kutolix", "model": "kutolix", "width": 2048, "layers": 8, "requests": 4, "longest": 1300,
         "spread": 0.9, "steps": 8},
        # The feed-forward of a mixture of experts over a prompt.
        {"kind": "experts", "name": "experts_2048", "tokens": 2048, "width": 2048, "ff": 2048, "experts": 32, "top": 4},
        # True 32-bit generation of a small batch, greedy and sampled requests together.
        {"kind": "generate", "name": "generate_f32", "requests": 12, "longest": 190, "new": 24},
        # The tokens of a full batch, every kind of sampling parameters among them.
        {"kind": "sample", "name": "sample_b48", "rows": 48, "vocab": 128256, "dtype": "bfloat16"},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.5))))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "mixed", "serve", "serve", "experts", "generate", "sample"])
    step = {"kind": "step", "model": rng.choice(["1b", "1b", "3b", "8b"]), "decodes": 0, "context": 0, "prompts": 0, "longest": 0,
            "held": 0, "spread": round(rng.uniform(0.0, 0.95), 2)}
    if kind == "decode":
        batch = _log_int(rng, 1, 64)
        most = min(8000, {"1b": 120000, "3b": 40000, "8b": 15000}[step["model"]] // batch)
        return dict(step, decodes=batch, context=_log_int(rng, min(16, most), most))
    if kind == "prompt":
        prompts = _log_int(rng, 1, 12)
        most = min(8000, {"1b": 16000, "3b": 6000, "8b": 2500}[step["model"]] // prompts)
        return dict(step, prompts=prompts, longest=_log_int(rng, 5, most))
    if kind == "mixed":
        step["model"] = rng.choice(["1b", "3b"])
        decodes = _log_int(rng, 1, 48)
        return dict(step, decodes=decodes, context=_log_int(rng, 16, 700), prompts=1, longest=_log_int(rng, 16, 1400),
                    held=rng.choice([0, rng.randrange(1, 1500)]))
    if kind == "serve":
        requests = _log_int(rng, 1, 16)
        return {"kind": "serve", "model": rng.choice(["karupel", "kutolix"]), "width": rng.choice([1024, 2048]),
                "layers": rng.choice([4, 8]), "requests": requests, "longest": _log_int(rng, 5, min(1500, 3000 // requests)),
                "spread": round(rng.uniform(0.0, 0.95), 2), "steps": rng.randint(2, 12)}
    if kind == "experts":
        return {"kind": "experts", "tokens": _log_int(rng, 1, 3000), "width": rng.choice([1024, 2048]), "ff": rng.choice([512, 2048]),
                "experts": rng.choice([8, 32]), "top": rng.choice([1, 2, 4])}
    if kind == "generate":
        return {"kind": "generate", "requests": _log_int(rng, 1, 16), "longest": _log_int(rng, 3, 200), "new": rng.randint(2, 24)}
    return {"kind": "sample", "rows": _log_int(rng, 1, 64), "vocab": rng.choice([32000, 50257, 128256]),
            "dtype": rng.choice(["bfloat16", "float32"])}


def _lengths(count: int, longest: int, spread: float) -> list[int]:
    """`count` lengths from `longest` down, the last one shorter by the share `spread`."""
    return [max(1, round(longest * (1.0 - spread * i / max(1, count - 1)))) for i in range(count)]


def _rows(case: dict) -> list[tuple[int, int]]:
    """(tokens held before the step, tokens that the step brings) of every request of a step."""
    rows = [(n, 1) for n in _lengths(case["decodes"], case["context"], case["spread"])] if case["decodes"] else []
    return rows + [(case["held"], n) for n in (_lengths(case["prompts"], case["longest"], case["spread"]) if case["prompts"] else [])]


# ------------------------------------------------------------------ inputs
def _generator(seed: int, where: str = "cpu"):
    return torch.Generator(device=where).manual_seed(seed)


def _spread(name: str, shape: tuple[int, ...], config: dict, layers: int) -> float:
    if name in ("model.embed_tokens.weight", "embed"):
        return 0.02 if config.get("architecture") == "Kutolix" else 1.0     # Kutolix normalises nothing on the way in
    if name.endswith(("o_proj.weight", "down_proj.weight")):
        return (2 * layers * shape[1]) ** -0.5
    return 0.02


def _drawn_weights(config: dict, seed: int, dtype: torch.dtype):
    """(the model, not yet bound; {tensor name: tensor}) with the distributions of the random-weights mode, but for two: a
    Llama (or Karupel) embedding is N(0, 1), as `torch.nn.Embedding` starts it, and the projections that end a Llama
    sublayer have unit gain over the root of their number, as GPT-2 scales them.  The residual stream is then led by the
    token, as in a trained model, and roundings do not grow from layer to layer."""
    arch, typed = resolve(config)
    spec = arch.build_spec(typed)
    model = Model(spec, dtype, torch.device(DEVICE))
    here, host = _generator(seed, DEVICE), _generator(seed)
    tensors = {}
    for name, want in model.tensor_specs().items():
        if name in spec.tied:
            continue
        shape, kind = want.drawn_shape(), torch.float32 if want.kind == "f32" else dtype
        if callable(want.init):
            tensors[name] = torch.as_tensor(want.init(shape, host), dtype=torch.float32).to(DEVICE, kind)
        elif want.init == "zeros":
            tensors[name] = torch.zeros(shape, device=DEVICE, dtype=kind)
        else:
            value = torch.randn(shape, generator=here, device=DEVICE, dtype=kind)
            tensors[name] = value.mul_(_spread(name, shape, config, len(spec.layers))) if want.init == "normal" else value.mul_(0.01).add_(1.0)
    for name, source in spec.tied.items():
        tensors[name] = tensors[source]
    return model, tensors


def _tokens(count: int, vocab: int, seed: int, request: int) -> list[int]:
    return torch.randint(0, vocab, (count,), generator=_generator(seed * 1009 + request)).tolist()


def _runner(case: dict, seed: int, totals: list[int]):
    model, tensors = _drawn_weights(_config(case), seed, torch.bfloat16)
    model.bind(tensors)
    return make_runner(model, torch.bfloat16, DEVICE, PAGE, sum(-(-n // PAGE) for n in totals), len(totals))


def _prepare_step(case: dict, seed: int) -> dict:
    rows = _rows(case)
    totals = [held + new for held, new in rows]
    runner = _runner(case, seed, totals)
    vocab = runner.model.spec.vocab_size
    tokens = [_tokens(n, vocab, seed, i) for i, n in enumerate(totals)]
    # The requests that are under way: what they hold is computed, as many at a time as a step's budget takes.
    batch, room = [], PORTION
    for i, (held, _) in enumerate(rows):
        for at in range(0, held, PORTION):
            part = tokens[i][at:min(held, at + PORTION)]
            if len(part) > room or any(e.request_id == f"r{i}" for e in batch):
                runner.step(batch)
                batch, room = [], PORTION
            batch.append(StepEntry(f"r{i}", part))
            room -= len(part)
    if batch:
        runner.step(batch)
    runner.enable_decode_graphs(max(32, len(rows)), 4096 if max(totals) <= 4096 else 8192)
    entries = [StepEntry(f"r{i}", tokens[i][held:], (new - 1,)) for i, (held, new) in enumerate(rows)]
    return {"runner": runner, "entries": entries, "held": [held for held, _ in rows]}


def _run_step(state: dict):
    runner = state["runner"]
    logits = runner.step(state["entries"])
    # The requests go back to where they stood, as for another candidate of the same position; whole prompts are done.
    for entry, held in zip(state["entries"], state["held"]):
        if held:
            runner.cache.commit(entry.request_id, held)
        else:
            runner.release(entry.request_id)
    if any(state["held"]):
        return {"logits": logits}
    return {"logits": logits, "cache": runner.cache.groups[0].pool}


def _prepare_serve(case: dict, seed: int) -> dict:
    lengths = _lengths(case["requests"], case["longest"], case["spread"])
    runner = _runner(case, seed, [n + case["steps"] for n in lengths])
    runner.enable_decode_graphs(max(32, len(lengths)), 4096)
    tokens = [_tokens(n + case["steps"], 32000, seed, i) for i, n in enumerate(lengths)]
    steps = [[StepEntry(f"r{i}", t[:n], (n - 1,)) for i, (t, n) in enumerate(zip(tokens, lengths))]]
    steps += [[StepEntry(f"r{i}", [t[n + k]], (0,)) for i, (t, n) in enumerate(zip(tokens, lengths))] for k in range(case["steps"])]
    return {"runner": runner, "steps": steps}


def _run_serve(state: dict):
    runner = state["runner"]
    logits = [runner.step(entries) for entries in state["steps"]]
    for entry in state["steps"][0]:
        runner.release(entry.request_id)
    return {"prompts": logits[0], "decoded": logits[1:]}


_EXPERTS = {"groups": 8, "groups_keep": 4, "activation": "capped_swiglu", "limit": 7.0, "alpha": 1.702}


def _expert_tensors(case: dict, seed: int):
    part = build_part("feed_forward", PartSpec("routed_experts", dict(
        _EXPERTS, hidden_size=case["width"], intermediate_size=case["ff"], experts=case["experts"], top=case["top"])),
        dtype=torch.bfloat16, device=torch.device(DEVICE))
    g = _generator(seed, DEVICE)
    tensors = {name: torch.randn(want.drawn_shape(), generator=g, device=DEVICE,
                                 dtype=torch.float32 if want.kind == "f32" else torch.bfloat16).mul_(0.02)
               for name, want in part.tensor_specs().items()}
    x = torch.randn(case["tokens"], case["width"], generator=g, device=DEVICE, dtype=torch.bfloat16)
    return part, tensors, x


def _prepare_experts(case: dict, seed: int) -> dict:
    part, tensors, x = _expert_tensors(case, seed)
    part.bind(tensors)
    return {"part": part, "x": x}


def _sampling(i: int, new: int) -> SamplingParams:
    kinds = ({"temperature": 0.0}, {"temperature": 0.8, "top_k": 50}, {"temperature": 1.0, "top_p": 0.9},
             {"temperature": 0.7, "top_k": 200, "top_p": 0.95})
    return SamplingParams(**kinds[i % 4], seed=i, max_tokens=new, ignore_eos=True)


def _prepare_generate(case: dict, seed: int) -> dict:
    with tempfile.TemporaryDirectory() as tmp:
        folder = write_random_model(SMALL, Path(tmp) / "small", seed, torch.float32)
        llm = LLM(str(folder), dtype="float32", device=DEVICE, max_num_seqs=16, max_model_len=512, max_num_batched_tokens=2048,
                  num_gpu_blocks=16 * 512 // PAGE)
    lengths = _lengths(case["requests"], case["longest"], 0.9)
    return {"llm": llm, "prompts": [_tokens(n, SMALL["vocab_size"], seed, i) for i, n in enumerate(lengths)],
            "params": [_sampling(i, case["new"]) for i in range(len(lengths))]}


def _prepare_sample(case: dict, seed: int) -> dict:
    logits = torch.randn(case["rows"], case["vocab"], generator=_generator(seed, DEVICE), device=DEVICE).mul_(2.5)
    return {"logits": logits.to(getattr(torch, case["dtype"])), "sampler": Sampler(0),
            "params": [_sampling(i, 1) for i in range(case["rows"])]}


def prepare(case: dict, seed: int) -> dict:
    makers = {"step": _prepare_step, "serve": _prepare_serve, "experts": _prepare_experts, "generate": _prepare_generate,
              "sample": _prepare_sample}
    return dict(makers[case["kind"]](case, seed), kind=case["kind"])


def run(state: dict):
    kind = state["kind"]
    if kind == "step":
        return _run_step(state)
    if kind == "serve":
        return _run_serve(state)
    if kind == "experts":
        return state["part"].forward(state["x"], None)
    if kind == "generate":
        return torch.tensor([out.token_ids for out in state["llm"].generate(state["prompts"], state["params"])])
    return state["sampler"](state["logits"], state["params"])


# ------------------------------------------------------------------ what a pass cannot do without
def _llama_counts(c: dict) -> tuple[int, int, int]:
    """(weights of the layers, weights of the head, numbers of keys and values of one token)."""
    q, kv = c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
    per = c["hidden_size"] * (2 * q + 2 * kv) + 3 * c["hidden_size"] * c["intermediate_size"]
    return c["num_hidden_layers"] * per, c["vocab_size"] * c["hidden_size"], c["num_hidden_layers"] * 2 * kv


def _llama_work(c: dict, rows: list[tuple[int, int]], element: int) -> dict:
    layers, head, kv = _llama_counts(c)
    new = sum(n for _, n in rows)
    read = layers + head + kv * sum(held for held, _ in rows)
    written = kv * new + c["vocab_size"] * len(rows)
    pairs = sum(n * held + n * (n + 1) / 2 for held, n in rows)
    attention = 4 * c["num_hidden_layers"] * c["num_attention_heads"] * c["head_dim"] * pairs
    return {"bytes": element * (read + written), "flops": 2 * layers * new + 2 * head * len(rows) + attention}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "step":
        return _llama_work(LLAMA[case["model"]], _rows(case), 2)
    if kind == "generate":      # every step reads the weights; the prompts go in with the first
        rows = [(0, n) for n in _lengths(case["requests"], case["longest"], 0.9)]
        every = [_llama_work(SMALL, [(n + k, 1) for _, n in rows] if k else rows, 4) for k in range(case["new"])]
        return {key: sum(w[key] for w in every) for key in ("bytes", "flops")}
    if kind == "experts":
        pairs, per = case["tokens"] * case["top"], 3 * case["width"] * case["ff"]
        return {"bytes": 2 * per * min(case["experts"], pairs) + 4 * case["tokens"] * case["width"] + 4 * case["experts"] * case["width"],
                "flops": 2 * pairs * per + 2 * case["tokens"] * case["experts"] * case["width"]}
    if kind == "sample":
        return {"bytes": case["rows"] * case["vocab"] * (2 if case["dtype"] == "bfloat16" else 4) + 4 * case["rows"], "flops": 0}
    width, requests = case["width"], case["requests"]
    weights, kept, state, pair_flops = width * 32000, 0, 0, 0       # kept: cache bytes of a token; state: bytes of a request
    for layer in _config(case)["layers"]:
        m, heads = layer["mixer"], layer["mixer"]["heads"]
        weights += 3 * width * layer["mlp"]["ff"]
        if layer["type"] == "delta":
            weights += 5 * width * heads * m["dim"]
            state += 4 * heads * m["dim"] * m["vdim"]
        elif layer["type"] == "latent_attention":
            kept += 2 * (m["kv_rank"] + m["rot_dim"])
            weights += width * (heads * (m["dim"] + m["rot_dim"] + m["vdim"]) + m["kv_rank"] + m["rot_dim"])
            weights += m["kv_rank"] * heads * (m["dim"] + m["vdim"])
            pair_flops += 2 * heads * (m["dim"] + m["rot_dim"] + m["vdim"])
        else:
            kept += 4 * m["kv_heads"] * m["dim"]
            weights += width * (2 * heads + 2 * m["kv_heads"]) * m["dim"] + (width * heads * m["dim"] if case["model"] == "kutolix" else 0)
            pair_flops += 4 * heads * m["dim"]
    lengths = _lengths(requests, case["longest"], case["spread"])
    window = 1024 if case["model"] == "kutolix" else 1 << 30
    total = {"bytes": 0.0, "flops": 0.0}
    for k in range(case["steps"] + 1):
        new = lengths if k == 0 else [1] * requests
        held = [0] * requests if k == 0 else [min(n + k - 1, window) for n in lengths]
        pairs = sum(sum(min(i + 1, window) for i in range(n)) for n in lengths) if k == 0 else sum(h + 1 for h in held)
        total["bytes"] += 2 * weights + kept * (sum(held) + sum(new)) + requests * (state * (1 if k == 0 else 2) + 2 * 32000)
        total["flops"] += 2 * (weights - width * 32000) * sum(new) + 2 * width * 32000 * requests + pair_flops * pairs + state * sum(new)
    return total


def tolerance(case: dict):
    """bfloat16 models: their logits differ by roundings that add up over the layers.  Tokens: the same."""
    if case["kind"] in ("generate", "sample"):
        return "exact"
    if case["kind"] == "experts":
        return {"rel": 0.01}
    return {"rel": 0.03}


# ------------------------------------------------------------------ the same in 64 bits
F = torch.float64


def _unit_rms(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _gated(x, gate, up, down):
    """down(silu(gate x) * (up x)), a few thousand rows at a time."""
    return torch.cat([(_silu(part @ gate.T) * (part @ up.T)) @ down.T for part in x.split(4096)])


def _turn(x, angles, stretch=1.0, interleaved=False):
    """x [T, heads, n]; angles [T, dims / 2]: rotates the first dims numbers of every head."""
    half = angles.shape[1]
    c, s = angles.cos()[:, None] * stretch, angles.sin()[:, None] * stretch
    out = x.clone()
    a, b = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if interleaved else (slice(0, half), slice(half, 2 * half))
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _attend(q, k, v, scale, window=None, sink=None):
    """One sequence: q [T, H, D], k [T, G, D], v [T, G, V] -> [T, H, V], a few hundred queries at a time."""
    T, H, _ = q.shape
    per = H // k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F, device=q.device)
    at = torch.arange(T, device=q.device)
    for t in range(0, T, 512):
        rows = slice(t, min(T, t + 512))
        low = 0 if window is None else max(0, t - window + 1)
        keys = slice(low, rows.stop)
        hidden = at[None, keys] > at[rows, None]
        if window is not None:
            hidden |= at[None, keys] <= at[rows, None] - window
        s = torch.einsum("tgpd,sgd->gpts", q[rows].unflatten(1, (-1, per)), k[keys]) * scale
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.view(-1, per, 1, 1).expand(*s.shape[:3], 1)], -1)
        p = torch.softmax(s, -1)
        p = p if sink is None else p[..., :-1]
        out[rows] = torch.einsum("gpts,sgv->tgpv", p, v[keys]).flatten(1, 2)
    return out


def _positions(spans):
    return torch.cat([torch.arange(n, dtype=F, device=DEVICE) for n in spans])


def _over_sequences(fn, spans, *tensors):
    return torch.cat([fn(*parts) for parts in zip(*(t.split(spans) for t in tensors))])


def _llama_exact(c, w, tokens):
    """The last hidden states [all tokens, hidden] after the final norm, and the head."""
    spans = [len(t) for t in tokens]
    d, eps, heads, groups = c["head_dim"], c["rms_norm_eps"], c["num_attention_heads"], c["num_key_value_heads"]
    r = c["rope_scaling"]
    freq = c["rope_theta"] ** (-torch.arange(0, d, 2, dtype=F, device=DEVICE) / d)
    wave = 2 * math.pi / freq
    share = ((r["original_max_position_embeddings"] / wave - r["low_freq_factor"])
             / (r["high_freq_factor"] - r["low_freq_factor"])).clamp(0, 1)
    freq = (1 - share) * freq / r["factor"] + share * freq
    angles = _positions(spans)[:, None] * freq
    get = lambda name: w[name].to(F)
    x = w["model.embed_tokens.weight"][torch.tensor(sum(tokens, []), device=DEVICE)].to(F)
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _unit_rms(x, eps) * get(p + "input_layernorm.weight")
        q, k, v = ((h @ get(p + f"self_attn.{n}_proj.weight").T).unflatten(1, (-1, d)) for n in "qkv")
        q, k = _turn(q, angles), _turn(k, angles)
        a = _over_sequences(lambda *qkv: _attend(*qkv, d ** -0.5), spans, q, k, v)
        x = x + a.flatten(1) @ get(p + "self_attn.o_proj.weight").T
        h = _unit_rms(x, eps) * get(p + "post_attention_layernorm.weight")
        x = x + _gated(h, *(get(p + f"mlp.{n}_proj.weight") for n in ("gate", "up", "down")))
    return _unit_rms(x, eps) * get("model.norm.weight"), w["lm_head.weight"]


def _conv(x, taps):
    """x [T, C], taps [C, K]: the last tap on the token itself, zeros before the first."""
    K = taps.shape[1]
    padded = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(K))


def _delta_memory(q, k, v, beta, decay):
    S, out = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(q.shape[0]):
        S = decay[t][:, None, None] * S
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return out


def _karupel_exact(c, w, tokens):
    spans, eps = [len(t) for t in tokens], c["norm"]["eps"]
    get = lambda name: w[name].to(F)
    norm = lambda x, name: _unit_rms(x, eps) * (1.0 + get(name))
    x = get("embed")[torch.tensor(sum(tokens, []), device=DEVICE)]
    first = None
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, D = m["heads"], m["dim"]
        product = lambda n: x @ get(p + n).T
        if layer["type"] == "delta":
            q, k, v = (_silu(_over_sequences(lambda s: _conv(s, get(p + n + ".conv")), spans, product(n))).unflatten(1, (H, D))
                       for n in "qkv")
            q, k = (z / torch.sqrt(z.pow(2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
            decay = torch.exp(-torch.exp(get(p + "A_log")) * torch.nn.functional.softplus(product("a") + get(p + "dt_bias")))
            o = _over_sequences(_delta_memory, spans, q * D ** -0.5, k, v, torch.sigmoid(product("b")), decay)
            y = (_unit_rms(o, eps) * get(p + "norm") * _silu(product("g")).unflatten(1, (H, D))).flatten(1) @ get(p + "o").T
        else:
            rot = m["rot"]
            freq = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=F, device=DEVICE) / rot["dims"]) / rot["scaling"]["factor"]
            angles = _positions(spans)[:, None] * freq
            q, k, v = ((product(n) + get(p + n + ".b")).unflatten(1, (-1, D)) for n in "qkv")
            q, k = (_turn(_unit_rms(z, eps) * get(p + n + ".norm"), angles) for z, n in ((q, "q"), (k, "k")))
            if first is None:
                first = v
            else:
                v = (1.0 - get(p + "vmix")) * v + get(p + "vmix") * first
            o = _over_sequences(lambda *qkv: _attend(*qkv, m["scale"]), spans, q, k, v) * torch.sigmoid(product("g"))[:, :, None]
            y = o.flatten(1) @ get(p + "o").T
        x = x + norm(y, f"l{i}.norm1")
        x = x + norm(_gated(x, *(get(f"l{i}.mlp.{n}") for n in ("gate", "up", "down"))), f"l{i}.norm2")
    return norm(x, "final.norm"), w["embed"]


def _yarn(rot):
    dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
    i = torch.arange(dims // 2, dtype=F, device=DEVICE)
    f = base ** (-2.0 * i / dims)
    if not s:
        return f, 1.0
    index = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    low, high = max(math.floor(index(s["fast"])), 0), min(math.ceil(index(s["slow"])), dims - 1)
    ramp = ((i - low) / max(high - low, 0.001)).clamp(0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _kutolix_exact(c, w, tokens):
    spans, eps, scale = [len(t) for t in tokens], c["norm"]["eps"], c["residual_mult"]
    get = lambda name: w[name].to(F)
    at = _positions(spans)[:, None]
    x = get("embed")[torch.tensor(sum(tokens, []), device=DEVICE)] * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, D, window = m["heads"], m["dim"], m["mask"]["size"]
        freq, stretch = _yarn(m["rot"])
        product = lambda n: x @ get(p + n).T
        if layer["type"] == "attention":
            q, k, v = (product(n).unflatten(1, (-1, D)) for n in "qkv")
            q, k = (_unit_rms(_turn(z, at * freq, stretch), eps) for z in (q, k))
            a = _over_sequences(lambda *qkv: _attend(*qkv, m["scale"], window, get(p + "sink")), spans, q, k, v)
            a = a.flatten(1) * torch.sigmoid(product("g"))
        else:
            q, down = product("q").unflatten(1, (H, -1)), product("dkv")
            latent = _unit_rms(down[:, :m["kv_rank"]], eps) * get(p + "dkv.norm")
            shared = _turn(down[:, None, m["kv_rank"]:], at * freq, stretch, True).expand(-1, H, -1)
            q = torch.cat([q[..., :D], _turn(q[..., D:], at * freq, stretch, True)], -1)
            k = torch.cat([(latent @ get(p + "uk").T).unflatten(1, (H, D)), shared], -1)
            v = (latent @ get(p + "uv").T).unflatten(1, (H, -1))
            a = _over_sequences(lambda *qkv: _attend(*qkv, m["scale"], window), spans, q, k, v).flatten(1)
        x = x + scale * _unit_rms(a @ get(p + "o").T, eps) * get(f"l{i}.norm1")
        y = _gated(x, *(get(f"l{i}.mlp.{n}") for n in ("gate", "up", "down")))
        x = x + scale * _unit_rms(y, eps) * get(f"l{i}.norm2")
    return _unit_rms(x, eps) * get("final.norm"), w["embed"]


def _expert_exact(case, seed):
    _, w, x = _expert_tensors(case, seed)
    x, out = x.to(F), torch.zeros(x.shape, dtype=F, device=DEVICE)
    scores = torch.softmax(x @ w["router.weight"].to(F).T, -1)
    grouped = scores.unflatten(1, (_EXPERTS["groups"], -1))
    best = grouped.amax(-1).topk(_EXPERTS["groups_keep"], -1).indices
    kept = torch.zeros(grouped.shape[:2], dtype=torch.bool, device=DEVICE).scatter_(1, best, True)
    chosen = torch.where(kept[:, :, None], grouped, -1.0).flatten(1).topk(case["top"], -1).indices
    limit = _EXPERTS["limit"]
    for e in range(case["experts"]):
        rows, slot = torch.nonzero(chosen == e, as_tuple=True)
        if len(rows):
            g, u = ((x[rows] @ w[f"experts.{e}.{n}_proj.weight"].to(F).T) for n in ("gate", "up"))
            g, u = g.clamp(max=limit), u.clamp(-limit, limit)
            y = (g * torch.sigmoid(_EXPERTS["alpha"] * g) * (u + 1.0)) @ w[f"experts.{e}.down_proj.weight"].to(F).T
            out[rows] += scores[rows, e][:, None] * y
    return out


@torch.no_grad()
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("generate", "sample"):
        return None             # tokens: they are compared as they are
    if kind == "experts":
        return _expert_exact(case, seed)
    config = _config(case)
    _, w = _drawn_weights(config, seed, torch.bfloat16)
    if kind == "step":
        totals = [held + new for held, new in _rows(case)]
        tokens = [_tokens(n, config["vocab_size"], seed, i) for i, n in enumerate(totals)]
        h, head = _llama_exact(config, w, tokens)
        last = torch.tensor(totals, device=DEVICE).cumsum(0) - 1
        logits = {"logits": h[last] @ head.to(F).T}
        return logits if any(held for held, _ in _rows(case)) else dict(logits, cache=None)
    lengths = _lengths(case["requests"], case["longest"], case["spread"])
    tokens = [_tokens(n + case["steps"], 32000, seed, i) for i, n in enumerate(lengths)]
    h, head = {"karupel": _karupel_exact, "kutolix": _kutolix_exact}[case["model"]](config, w, tokens)
    ends = torch.tensor([n + case["steps"] for n in lengths], device=DEVICE).cumsum(0) - 1 - case["steps"]
    cap = config.get("logit_softcap")
    steps = []
    for k in range(case["steps"] + 1):
        logits = h[ends + k] @ head.to(F).T
        steps.append(cap * torch.tanh(logits / cap) if cap else logits)
    return {"prompts": steps[0], "decoded": steps[1:]}
