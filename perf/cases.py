"""What the engine is measured on: steps of the models it serves, through `Model.open_request`, `Model.step` and
`Model.close_request`.

Two kinds of pass:

  decode    one step of a batch of open requests, one token each, over the context they hold (it grows by one a pass)
  complete  requests come in `arrive` at a time: a step runs their prompts beside one token of every request that is already
            in; when all are in, `new` more steps of one token each; then they are closed.  `all_logits` asks for the logits of
            every prompt position (scoring a text), otherwise for each prompt's last.

Tokens are given (uniform over the vocabulary), so a pass does the same work whatever the logits are.  A pass returns the
logits of every step, rows in the order of the steps and of the requests in them.

Models are the layer sizes of Qwen3-0.6B and Qwen3-8B, and one model of each other design at the widths the benchmark compares
them at (four layers: one of each kind the design has).  Weights are the engine's random ones, the same for every seed: they
stand for a model that is loaded once and serves many requests.
"""
import gc
import math
import random

import torch

from mini_llm_runtime_b200 import models as _models  # noqa: F401  (registers the architectures)
from mini_llm_runtime_b200.config.registry import config_from_dict, plan_for
from mini_llm_runtime_b200.engine.model import CacheConfig, Model, StepEntry
from mini_llm_runtime_b200.engine.runtime import Runtime
from mini_llm_runtime_b200.engine.structure import expected_weights
from mini_llm_runtime_b200.weights.random_init import random_tensors

DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
PAGE = 16                  # tokens to a cache page, the engine's default
WEIGHTS_SEED = 7


# ------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # One user's chat with a dense 8B model: what the answer's speed is.
        {"name": "qwen3-8b decode b1", "model": "qwen3-8b", "kind": "decode", "dtype": "bfloat16", "lengths": "2048"},
        # The headline: a small batch over a long context.
        {"name": "qwen3-8b decode b8", "model": "qwen3-8b", "kind": "decode", "dtype": "bfloat16", "lengths": " ".join(["8192"] * 8)},
        # A busy server: more requests than the few-row kernels take, contexts of all lengths.
        {"name": "qwen3-8b decode b40", "model": "qwen3-8b", "kind": "decode", "dtype": "bfloat16",
         "lengths": " ".join(str(257 + 61 * i) for i in range(40))},
        # Time to the first token of a long prompt.
        {"name": "qwen3-8b prompt 2048", "model": "qwen3-8b", "kind": "complete", "dtype": "bfloat16", "lengths": "2048", "arrive": 1, "new": 0,
         "all_logits": False},
        # A small model on short requests: launches and host work weigh most here.
        {"name": "qwen3-0.6b short", "model": "qwen3-0.6b", "kind": "complete", "dtype": "bfloat16", "lengths": "17 129 64 301", "arrive": 2, "new": 6,
         "all_logits": False},
        # Scoring texts in true 32-bit arithmetic: every position's logits.
        {"name": "qwen3-0.6b float32 score", "model": "qwen3-0.6b", "kind": "complete", "dtype": "float32", "lengths": "96 33", "arrive": 2, "new": 1,
         "all_logits": True},
        # Each other design: prompts and the tokens behind them, at the widths of a 1.7B and of an 8B dense model.
        {"name": "gopevik 2048", "model": "gopevik-2048", "kind": "complete", "dtype": "bfloat16", "lengths": "2048 1171", "arrive": 1, "new": 6,
         "all_logits": False},
        {"name": "niridra 2048", "model": "niridra-2048", "kind": "complete", "dtype": "bfloat16", "lengths": "2048 515 1300", "arrive": 3, "new": 6,
         "all_logits": False},
        {"name": "sopetar 4096", "model": "sopetar-4096", "kind": "complete", "dtype": "bfloat16", "lengths": "2048", "arrive": 1, "new": 6,
         "all_logits": False},
        {"name": "sokolorn 2048", "model": "sokolorn-2048", "kind": "complete", "dtype": "bfloat16", "lengths": "1024 999 77 2000 640 31 1500 256",
         "arrive": 4, "new": 6, "all_logits": False},
        {"name": "gelulix 2048", "model": "gelulix-2048", "kind": "complete", "dtype": "bfloat16", "lengths": "2048 900", "arrive": 2, "new": 6,
         "all_logits": False},
        {"name": "repolix 4096", "model": "repolix-4096", "kind": "complete", "dtype": "bfloat16", "lengths": "1999", "arrive": 1, "new": 6,
         "all_logits": False},
    ]


def draw(rng: random.Random):
    """A case of the same kinds: the dense model's decode steps and prompts at other batches and lengths, the other designs at
    other widths, numbers of requests and lengths.  No case has more than 8192 prompt tokens or 131072 tokens of context."""
    def length(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    roll = rng.random()
    if roll < 0.25:
        model = rng.choice(["qwen3-8b", "qwen3-0.6b"])
        batch = length(1, 64)
        longest = min(8192, 98304 // batch)
        top = length(128, longest)
        return {"model": model, "kind": "decode", "dtype": "bfloat16", "lengths": " ".join(str(rng.randint(max(1, top // 2), top)) for _ in range(batch))}
    if roll < 0.45:
        model = rng.choice(["qwen3-8b", "qwen3-0.6b"])
        requests = length(1, 6)
        small = model == "qwen3-0.6b" and rng.random() < 0.4
        top = 128 if small else 2048 // (2 if model == "qwen3-8b" and requests > 1 else 1)
        if model == "qwen3-8b":
            requests = min(requests, 2)
        return {"model": model, "kind": "complete", "dtype": "float32" if small else "bfloat16",
                "lengths": " ".join(str(length(9, top)) for _ in range(min(requests, 2) if small else requests)), "arrive": rng.randint(1, 2),
                "new": rng.randint(0, 2 if small else 4), "all_logits": small and rng.random() < 0.5}
    design = rng.choice(["gopevik", "niridra", "sopetar", "sokolorn", "gelulix", "repolix"])
    requests = length(1, 6)
    return {"model": f"{design}-{rng.choice([1024, 2048, 2048, 4096])}", "kind": "complete", "dtype": "bfloat16",
            "lengths": " ".join(str(length(16, 2048)) for _ in range(requests)), "arrive": rng.randint(1, requests), "new": rng.randint(1, 8),
            "all_logits": False}


# ----------------------------------------------------------------------------------------------------------- the models
def _qwen3(width, layers, heads, ff, tied):
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "hidden_size": width, "num_hidden_layers": layers,
            "num_attention_heads": heads, "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": ff, "vocab_size": 151936,
            "max_position_embeddings": 40960, "rms_norm_eps": 1e-6, "rope_theta": 1000000.0, "tie_word_embeddings": tied,
            "use_sliding_window": False, "hidden_act": "silu", "attention_bias": False, "torch_dtype": "bfloat16"}


def _moe(ff, **more):
    return {"kind": "moe", "expert": {"ff": ff // 6, **more}, "shared": {"ff": ff // 3, **more}}


def _gopevik(width, ff, heads, kv):
    side = {"type": "parallel", "mlp": {"kind": "dense", "ff": ff}, "mixer": {
        "left": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                 "rot": {"base": 1e6, "dims": 64, "scaling": {"factor": 4.0}}},
        "right": {"heads": heads // 2, "dim": 128, "vdim": 128, "decay": [1 - 2.0 ** (-5 - i % 4) for i in range(heads // 2)],
                  "rot": {"base": 1e4, "dims": 128}},
        "left_scale": 0.8, "right_scale": 0.9}}
    delta = {"type": "delta", "mlp": {"kind": "dense", "ff": ff}, "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}}
    return {"architecture": "Gopevik", "norm": {"eps": 1e-6, "groups": 4}, "layers": [side, side, delta, side]}


def _niridra(width, ff, heads, kv):
    mlp = {**_moe(ff), "router": {"experts": 16, "top": 4, "groups": {"count": 4, "keep": 2}}}
    latent = {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": 128, "scale": 128 ** -0.5}
    lightning = {"heads": heads, "dim": 128, "vdim": 128, "decay": [1 - 2.0 ** (-5 - i % 4) for i in range(heads)]}
    return {"architecture": "Niridra", "norm": {"eps": 1e-6}, "streams": 4,
            "embedding": {"scale": 50.0, "bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}},
            "layers": [{"type": "latent_attention", "mixer": latent, "mlp": mlp}, {"type": "lightning", "mixer": lightning, "mlp": mlp},
                       {"type": "latent_attention", "mixer": latent, "mlp": mlp}, {"type": "latent_attention", "mixer": {**latent, "kv_from": 2}, "mlp": mlp}]}


def _latent(heads, **more):
    return {"heads": heads, "dim": 128, "rot_dim": 32, "vdim": 128, "kv_rank": 96, "scale": 160 ** -0.5, **more}


def _sopetar(width, ff, heads, kv):
    latent = _latent(heads, rot={"base": 1e4, "dims": 32}, mask={"size": 1024})
    attention = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0, "v_mix": True,
                 "mask": {"size": 1024, "keep_first": 4}}
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    return {"architecture": "Sopetar", "norm": {"eps": 1e-5}, "embedding": {"scale": 50.0},
            "layers": [{"type": "attention", "mixer": attention, "mlp": mlp} if i % 2 else {"type": "latent_attention", "mixer": latent, "mlp": mlp}
                       for i in range(4)]}


def _sokolorn(width, ff, heads, kv):
    windowed = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024}}
    rotary = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
              "rot": {"base": 5e5, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    dense = {"kind": "dense", "ff": ff * 3 // 2}
    moe = {**_moe(ff, limit=7.0), "router": {"experts": 16, "top": 4}}
    return {"architecture": "Sokolorn", "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "layers": [{"type": "attention", "mixer": windowed, "mlp": dense}, {"type": "attention_2", "mixer": rotary, "mlp": moe},
                       {"type": "attention_2", "mixer": {**rotary, "kv_from": 1}, "mlp": dense}, {"type": "attention", "mixer": windowed, "mlp": moe}]}


_YARN = {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}


def _channel_delta(heads):
    return {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}


def _gelulix(width, ff, heads, kv):
    mlp, delta = {"kind": "dense", "ff": ff}, _channel_delta(heads)
    gla = {"heads": heads, "dim": 128, "vdim": 128, "tau": 16.0, "decay_rank": 64}
    latent = _latent(heads, rot={"base": 1e4, "dims": 32, "scaling": _YARN})
    return {"architecture": "Gelulix", "norm": {"eps": 1e-6}, "postln_alpha": 2.0,
            "layers": [{"type": kind, "mixer": m, "mlp": mlp}
                       for kind, m in (("channel_delta", delta), ("gla", gla), ("channel_delta", delta), ("latent_attention", latent))]}


def _repolix(width, ff, heads, kv):
    mlp = {**_moe(ff, limit=7.0), "router": {"experts": 16, "identity": 4, "top": 4, "groups": {"count": 4, "keep": 2}}}
    attention = {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 128, "scale": 64 ** -0.5, "diff": 0.5, "conv": 4, "mask": {"size": 1024},
                 "rot": {"base": 1e4, "dims": 64, "scaling": _YARN}}
    state = {"heads": width // 32, "groups": 8, "state": 128, "vdim": 64, "conv": 4, "norm_groups": 8}
    return {"architecture": "Repolix", "norm": {"eps": 1e-6}, "embedding": {"scale": 50.0},
            "layers": [{"type": kind, "mixer": m, "mlp": mlp}
                       for kind, m in (("attention", attention), ("mamba2", state), ("channel_delta", _channel_delta(heads)), ("mamba2", state))]}


_DESIGNS = {"gopevik": _gopevik, "niridra": _niridra, "sopetar": _sopetar, "sokolorn": _sokolorn, "gelulix": _gelulix, "repolix": _repolix}


def _config(name):
    """The config.json of a model of the cases."""
    if name == "qwen3-8b":
        return _qwen3(4096, 36, 32, 12288, False)
    if name == "qwen3-0.6b":
        return _qwen3(1024, 28, 16, 3072, True)
    design, width = name.split("-")
    width = int(width)
    heads = width // 128
    return {**_DESIGNS[design](width, 3 * width, heads, min(8, heads // 2)), "vocab": 32000, "width": width}


def _vocab(config):
    return config.get("vocab") or config["vocab_size"]


def _weights(config):
    """The engine's random weights, stored as bfloat16, with the proportions of a model that can be trained: the embedding of the size
    of a normed vector, what a sub-layer adds to the stream smaller by the root of their number, and routers that tell their experts
    apart (one of the size of the other matrices would leave a token's fourth and fifth choice to the last bit of its input)."""
    tensors = random_tensors(expected_weights(plan_for(config_from_dict(config))), WEIGHTS_SEED, torch.bfloat16, "cuda:0")
    layers = config.get("num_hidden_layers") or len(config["layers"])
    large = config.get("architecture") == "Gopevik" or config.get("tie_word_embeddings") is False
    for name, t in tensors.items():
        if name.endswith("mlp.router"):
            t.mul_(16.0)
        elif name.endswith((".o", ".down", "o_proj.weight", "down_proj.weight", "norm1b", "norm2b")):
            t.mul_((2 * layers) ** -0.5)
        elif large and name in ("embed", "model.embed_tokens.weight"):
            t.mul_(50.0)
    return tensors


def _lengths(case):
    return [int(n) for n in case["lengths"].split()]


# ------------------------------------------------------------------------------------------------------- prepare and run
_loaded = {}               # the one model that is loaded


def _model(case):
    """The case's model, loaded once for all the states of a case; a model for another case takes its place."""
    lengths, decode = _lengths(case), case["kind"] == "decode"
    states = 4 if decode else 1              # states whose requests are open at the same time
    growth = max(512, min(4096, 16384 // len(lengths))) if decode else 2 + case["new"] + len(lengths)
    rows, longest, room = states * len(lengths), max(lengths) + growth, states * (sum(lengths) + len(lengths) * growth)
    key = (case["model"], case["dtype"], rows, longest, room)
    if key not in _loaded:
        _loaded.clear()
        gc.collect()
        torch.cuda.empty_cache()
        config = _config(case["model"])
        model = Model(plan_for(config_from_dict(config)), Runtime(DTYPES[case["dtype"]], "cuda:0"))
        model.bind(_weights(config))
        pages = room // PAGE + 2 * rows + 1
        model.allocate_cache(CacheConfig(page_size=PAGE, num_pages=pages, max_requests=rows, max_model_len=longest + PAGE, fill_nan=False))
        _loaded[key] = model
    return _loaded[key]


class _Open:
    """Requests that stay open as long as the state that holds them."""

    def __init__(self, model, count):
        self.model, self.slots = model, [model.open_request() for _ in range(count)]

    def __del__(self):
        for slot in self.slots:
            self.model.close_request(slot)


def _tokens(case, seed):
    """Per request, the tokens of its prompt and all that follow it."""
    gen = torch.Generator().manual_seed(int(seed))
    vocab = _vocab(_config(case["model"]))
    tail = 1 if case["kind"] == "decode" else case["new"] + len(_lengths(case))
    return [torch.randint(0, vocab, (n + tail,), generator=gen).tolist() for n in _lengths(case)]


def _steps(case):
    """The steps of a `complete` pass: per step a list of (request, first token, tokens, places of the wanted logits)."""
    lengths, at, steps, arrived = _lengths(case), [0] * len(_lengths(case)), [], 0
    while arrived < len(lengths):
        step = [(i, at[i], 1, [0]) for i in range(arrived)]
        coming = range(arrived, min(len(lengths), arrived + case["arrive"]))
        step += [(i, 0, lengths[i], list(range(lengths[i])) if case["all_logits"] else [lengths[i] - 1]) for i in coming]
        arrived += len(coming)
        for i, _, count, _ in step:
            at[i] += count
        steps.append(step)
    for _ in range(case["new"]):
        steps.append([(i, at[i], 1, [0]) for i in range(arrived)])
        at = [a + 1 for a in at]
    return steps


def prepare(case, seed):
    model, tokens = _model(case), _tokens(case, seed)
    if case["kind"] == "decode":
        held = _Open(model, len(tokens))
        for slot, ids in zip(held.slots, tokens):
            for pos in range(0, len(ids) - 1, 2048):
                model.step([StepEntry(slot, ids[pos:min(pos + 2048, len(ids) - 1)], [])])
        return {"model": model, "held": held, "entries": [StepEntry(slot, [ids[-1]], [0]) for slot, ids in zip(held.slots, tokens)]}
    steps = [[(i, tokens[i][first:first + count], want) for i, first, count, want in step] for step in _steps(case)]
    rows = sum(len(want) for step in steps for _, _, want in step)
    return {"model": model, "requests": len(tokens), "steps": steps,
            "logits": torch.empty(rows, model.plan.vocab_size, dtype=torch.float32, device=model.rt.device)}


def run(state):
    model = state["model"]
    if "entries" in state:
        return model.step(state["entries"])
    slots = [model.open_request() for _ in range(state["requests"])]
    out, row = state["logits"], 0
    for step in state["steps"]:
        logits = model.step([StepEntry(slots[i], ids, want) for i, ids, want in step])
        out[row:row + logits.shape[0]].copy_(logits)         # the engine's own buffer is written again by the next step
        row += logits.shape[0]
    for slot in slots:
        model.close_request(slot)
    return out


# ------------------------------------------------------------------------------------------------- what a pass cannot avoid
def _mixers(config):
    """Per layer: what its mixer reads and computes: heads, key and value size of a score, bytes a token of the cache has (0: it
    reads another layer's), the keys a query may see (None: all), and the values of the state it keeps."""
    if "hidden_size" in config:
        return [dict(heads=config["num_attention_heads"], score=256, cache=2 * 8 * 128, span=None, state=0)] * config["num_hidden_layers"]
    made = []
    for layer in config["layers"]:
        m, kind = layer["mixer"], layer["type"]
        span = (m.get("mask") or {}).get("size")
        if kind == "parallel":
            left, right = m["left"], m["right"]
            made.append(dict(heads=left["heads"], score=256, cache=left["kv_heads"] * 256, span=left["mask"]["size"], state=right["heads"] * 128 * 128))
        elif kind == "latent_attention":
            # A latent and its rotated part are key and value of every head.
            per = m["kv_rank"] + m.get("rot_dim", 0)
            made.append(dict(heads=m["heads"], score=per + m["kv_rank"], cache=0 if m.get("kv_from") is not None else per, span=span, state=0))
        elif kind in ("attention", "attention_2"):
            maps = 2 if "diff" in m else 1
            made.append(dict(heads=m["heads"], score=maps * (m["dim"] + m["vdim"]), cache=0 if m.get("kv_from") is not None else m["kv_heads"] * (maps * m["dim"] + m["vdim"]),
                             span=span, state=0))
        else:
            made.append(dict(heads=0, score=0, cache=0, span=None, state=m["heads"] * m["vdim"] * m.get("state", m.get("dim"))))
    return made


def work(case):
    config = _config(case["model"])
    size = 4 if case["dtype"] == "float32" else 2
    matrices, experts, head = 0, 0, 0
    specs = expected_weights(plan_for(config_from_dict(config)))
    for name, spec in specs.items():
        count = math.prod(spec.shape)
        if name in ("head", "lm_head.weight") or (name in ("embed", "model.embed_tokens.weight") and "head" not in specs and "lm_head.weight" not in specs):
            head += count
        elif name in ("embed", "bigram", "model.embed_tokens.weight"):
            continue
        elif ".mlp.e" in name:
            experts += count
        else:
            matrices += count
    router = next((layer["mlp"]["router"] for layer in config.get("layers", []) if (layer.get("mlp") or {}).get("kind") == "moe"), None)
    outputs = router["experts"] + router.get("identity", 0) if router else 1
    share = router["top"] / outputs if router else 0.0
    if case["kind"] == "decode":
        steps = [[(i, n, 1, [0]) for i, n in enumerate(_lengths(case))]]
    else:
        steps = _steps(case)
    nbytes = flops = 0.0
    for step in steps:
        rows, wanted = sum(count for _, _, count, _ in step), sum(len(want) for *_, want in step)
        flops += 2.0 * rows * (matrices + share * experts) + 2.0 * wanted * head
        nbytes += size * (matrices + experts * (1.0 - (1.0 - share) ** rows) + (head if wanted else 0)) + 4.0 * wanted * _vocab(config) + rows * 4.0
        for m in _mixers(config):
            for _, first, count, _ in step:
                span = m["span"] or first + count
                pairs = sum(min(p + 1, span) for p in range(first, first + count))
                flops += 2.0 * m["heads"] * m["score"] * pairs + 4.0 * count * m["state"]
                nbytes += size * m["cache"] * (min(first, span) + count) + 8.0 * m["state"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the distance from `exact`: 2e-6 in float32; in bfloat16 0.002 to 0.007 by design, and 0.015 for Sokolorn, whose
    norms behind the sub-layers leave a router's close call its full size."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.03 if case["model"].startswith("sokolorn") else 0.025}


# ------------------------------------------------------------------------------------------------- the same in 64 bits, plainly
def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x, weight=None, eps=1e-6):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _grouped_rms(x, weight, groups, eps):
    return _rms(x.unflatten(-1, (groups, -1)), None, eps).flatten(-2) * weight


def _layer_norm(x, weight, bias, eps):
    c = x - x.mean(-1, keepdim=True)
    return c * torch.rsqrt((c * c).mean(-1, keepdim=True) + eps) * weight + bias


def _unit(x):
    return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _plain_freqs(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)


def _slowed_freqs(dims, base, scaling):
    f = _plain_freqs(dims, base)
    wave = 2 * math.pi / f
    s = ((scaling["original"] / wave - scaling["low"]) / (scaling["high"] - scaling["low"])).clamp(0, 1)
    return (1 - s) * f / scaling["factor"] + s * f


def _yarn_freqs(dims, base, scaling):
    f = _plain_freqs(dims, base)
    turns = lambda t: dims * math.log(scaling["original"] / (2 * math.pi * t)) / (2 * math.log(base))
    lo, hi = max(math.floor(turns(scaling["fast"])), 0), min(math.ceil(turns(scaling["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=torch.float64, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / scaling["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0


def _rotate(x, freqs, mult=1.0, pairs=False):
    """x [T, heads, n]: the first 2 len(freqs) values of a head turn by position * frequency, value i with its neighbour (`pairs`)
    or with value i + len(freqs)."""
    half = len(freqs)
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * freqs[None, :]
    c, s = (torch.cos(angle) * mult)[:, None], (torch.sin(angle) * mult)[:, None]
    head, rest = x[..., :2 * half], x[..., 2 * half:]
    u, v = (head[..., 0::2], head[..., 1::2]) if pairs else (head[..., :half], head[..., half:])
    a, b = u * c - v * s, v * c + u * s
    turned = torch.stack([a, b], -1).flatten(-2) if pairs else torch.cat([a, b], -1)
    return torch.cat([turned, rest], -1)


def _attend(q, k, v, scale, window=None, keep_first=0, chunk=None, cap=None, slopes=None, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, Dv]: causal attention, query rows in blocks."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = q.new_empty(T, H, v.shape[2])
    j = torch.arange(T, device=q.device)[None, :]
    for lo in range(0, T, 1024):
        i = torch.arange(lo, min(T, lo + 1024), device=q.device)[:, None]
        seen = j <= i
        if window is not None:
            seen = seen & ((i - j < window) | (j < keep_first))
        if chunk is not None:
            seen = seen & (torch.div(i, chunk, rounding_mode="floor") == torch.div(j, chunk, rounding_mode="floor"))
        for h in range(H):
            s = (q[lo:lo + 1024, h] @ k[:, h // (H // G)].T) * scale
            if cap is not None:
                s = cap * torch.tanh(s / cap)
            if slopes is not None:
                s = s - slopes[h] * (i - j)
            s = s.masked_fill(~seen, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                top = torch.maximum(top, sink[h])
            e = torch.exp(s - top)
            total = e.sum(-1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0.0)
            out[lo:lo + 1024, h] = (e / total) @ v[:, h // (H // G)]
    return out


def _recur(q, k, v, decay, beta=None):
    """q, k [T, H, D], v [T, H, Dv], decay broadcast over [T, H, D]; per token S <- decay S; S <- S + k u^T with u = v, or with `beta`
    [T, H] u = beta (v - S^T k); o = S^T q."""
    T, H, D = q.shape
    S = q.new_zeros(H, D, v.shape[2])
    out = torch.empty_like(v)
    decay, q4, k4 = decay.expand(T, H, D)[..., None], q[:, :, None, :], k[..., None]
    for t in range(T):
        S = S * decay[t]
        u = v[t][:, None, :]
        if beta is not None:
            u = beta[t][:, None, None] * (u - k[t][:, None, :] @ S)
        S = torch.baddbmm(S, k4[t], u)
        out[t] = (q4[t] @ S)[:, 0]
    return out


def _conv(x, taps, bias=None):
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    y = sum(padded[i:i + x.shape[0]] * taps[:, i] for i in range(n))
    return y if bias is None else y + bias


def _expert(x, W, p, limit):
    g, u = x @ W(p + "gate").T, x @ W(p + "up").T
    if limit is None:
        return (_silu(g) * u) @ W(p + "down").T
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W(p + "down").T


def _routed(x, W, p, mlp, chosen, weights):
    """Experts and identity experts by each token's choice, and the shared expert."""
    limit, out = mlp["expert"].get("limit"), torch.zeros_like(x)
    for e in range(mlp["router"]["experts"] + mlp["router"].get("identity", 0)):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            y = _expert(x[rows], W, f"{p}e{e}.", limit) if e < mlp["router"]["experts"] else x[rows]
            out.index_add_(0, rows, weights[rows, place, None] * y)
    return out


def _grouped_choice(choice, router, best_of):
    """The `top` experts of every token within its best groups; a group counts as the sum of its `best_of` largest choice scores."""
    count, keep = router["groups"]["count"], router["groups"]["keep"]
    T, E = choice.shape
    kept = choice.view(T, count, -1).topk(best_of, -1).values.sum(-1).topk(keep, -1).indices
    allowed = torch.zeros(T, count, dtype=torch.bool, device=choice.device).scatter_(1, kept, True)
    return choice.masked_fill(~allowed.repeat_interleave(E // count, 1), -math.inf).topk(router["top"], -1).indices


def _latent_attention(m, W, p, x, eps, kept, freqs=None, mult=1.0):
    """`kept`: another layer's latent and rotated key part, or None.  Returns the heads' results and this layer's own."""
    T, H, D, P, R = x.shape[0], m["heads"], m["dim"], m.get("rot_dim", 0), m["kv_rank"]
    q = (x @ W(p + "q").T).view(T, H, D + P)
    if kept is None:
        down = x @ W(p + "dkv").T
        kept = (_rms(down[:, :R], W(p + "dkv.norm"), eps), down[:, R:].reshape(T, 1, P))
    latent, part = kept
    if P:
        q = torch.cat([q[..., :D], _rotate(q[..., D:], freqs, mult, pairs=True)], -1)
        part = _rotate(part, freqs, mult, pairs=True)
    k = torch.cat([(latent @ W(p + "uk").T).view(T, H, D), part.expand(T, H, P)], -1)
    v = (latent @ W(p + "uv").T).view(T, H, m["vdim"])
    return _attend(q, k, v, m["scale"], window=(m.get("mask") or {}).get("size"), sink=W(p + "sink") if P else None), kept


def _delta_of(m, W, p, x, eps):
    """The gated delta rule with a decay per key channel, behind short convolutions."""
    T, H, G = x.shape[0], m["heads"], m["kv_heads"]
    q, k, v = (_silu(_conv(x @ W(p + r).T, W(p + r + ".conv"))) for r in "qkv")
    q = (_unit(q.view(T, G, -1)) * m["dim"] ** -0.5).repeat_interleave(H // G, 1)
    k = _unit(k.view(T, G, -1)).repeat_interleave(H // G, 1)
    z = torch.nn.functional.softplus((x @ W(p + "a1").T) @ W(p + "a2").T + W(p + "dt_bias"), threshold=1e9).view(T, H, -1)
    o = _recur(q, k, v.view(T, H, -1), torch.exp(-torch.exp(W(p + "A_log"))[None, :, None] * z), torch.sigmoid(x @ W(p + "b").T))
    return (_rms(o, W(p + "norm"), eps).flatten(1) * torch.sigmoid((x @ W(p + "g1").T) @ W(p + "g2").T)) @ W(p + "o").T


def _plain_qwen3(config, W, ids):
    eps, H, D = config["rms_norm_eps"], config["num_attention_heads"], config["head_dim"]
    x, T, freqs = W("model.embed_tokens.weight", ids), len(ids), _plain_freqs(D, config["rope_theta"])
    for i in range(config["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, W(p + "input_layernorm.weight"), eps)
        q, k, v = ((h @ W(f"{p}self_attn.{r}_proj.weight").T).view(T, -1, D) for r in "qkv")
        q, k = (_rotate(_rms(t, W(f"{p}self_attn.{r}_norm.weight"), eps), freqs) for t, r in ((q, "q"), (k, "k")))
        x = x + _attend(q, k, v, D ** -0.5).flatten(1) @ W(p + "self_attn.o_proj.weight").T
        h = _rms(x, W(p + "post_attention_layernorm.weight"), eps)
        x = x + (_silu(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)) @ W(p + "mlp.down_proj.weight").T
    return _rms(x, W("model.norm.weight"), eps), "model.embed_tokens.weight" if config["tie_word_embeddings"] else "lm_head.weight"


def _plain_gopevik(config, W, ids):
    eps, x, T = config["norm"]["eps"], W("embed", ids), len(ids)
    norm = lambda t, name: _grouped_rms(t, W(name), config["norm"]["groups"], eps)
    for i, layer in enumerate(config["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        h = norm(x, f"l{i}.norm1")
        if layer["type"] == "parallel":
            a, r = m["left"], m["right"]
            freqs = _plain_freqs(a["rot"]["dims"], a["rot"]["base"]) / a["rot"]["scaling"]["factor"]
            q, k, v = ((h @ W(f"{p}left.{n}").T).view(T, -1, 128) for n in "qkv")
            o = _attend(_rotate(q, freqs), _rotate(k, freqs), v, a["scale"], chunk=a["mask"]["size"], sink=torch.zeros(a["heads"], dtype=x.dtype, device=x.device))
            y = m["left_scale"] * (o.flatten(1) * torch.sigmoid(h @ W(p + "left.g").T)) @ W(p + "left.o").T
            freqs = _plain_freqs(r["rot"]["dims"], r["rot"]["base"])
            q, k, v = ((h @ W(f"{p}right.{n}").T).view(T, -1, 128) for n in "qkv")
            decay = torch.tensor(r["decay"], dtype=x.dtype, device=x.device)[None, :, None]
            o = _recur(_rotate(q, freqs), _rotate(k, freqs) * r["dim"] ** -0.5, v, decay)
            y = y + m["right_scale"] * (_rms(o, None, eps).flatten(1) * _silu(h @ W(p + "right.g").T)) @ W(p + "right.o").T
        else:
            H, G = m["heads"], m["kv_heads"]
            q, k, v = (_silu(_conv(h @ W(p + n).T, W(p + n + ".conv"))).view(T, -1, 128) for n in "qkv")
            q, k = ((_unit(q) * m["dim"] ** -0.5).repeat_interleave(H // G, 1), _unit(k).repeat_interleave(H // G, 1))
            g = torch.exp(-torch.exp(W(p + "A_log")) * torch.nn.functional.softplus(h @ W(p + "a").T + W(p + "dt_bias"), threshold=1e9))
            o = _rms(_recur(q, k, v, g[..., None], torch.sigmoid(h @ W(p + "b").T)), W(p + "norm"), eps)
            y = (o.flatten(1) * _silu(h @ W(p + "g").T)) @ W(p + "o").T
        x = x + norm(y, f"l{i}.norm1b")
        h, p = norm(x, f"l{i}.norm2"), f"l{i}.mlp."
        y = (_silu(h @ W(p + "gate").T + W(p + "gate.b")) * (h @ W(p + "up").T + W(p + "up.b"))) @ W(p + "down").T + W(p + "down.b")
        x = x + norm(y, f"l{i}.norm2b")
    return norm(x, "final.norm"), "head"


def _plain_niridra(config, W, ids):
    eps, T, kept = config["norm"]["eps"], len(ids), {}
    big = config["embedding"]["bigram"]
    rows = torch.cat([ids.new_tensor([big["buckets"]]), (ids[:-1] * big["mul_prev"] + ids[1:] * big["mul_cur"]) % big["buckets"]])
    x = W("embed", ids) * config["embedding"]["scale"] + W("bigram", rows)
    xs = x[:, None, :].repeat(1, config["streams"], 1)
    for i, layer in enumerate(config["layers"]):
        m = layer["mixer"]
        for at in (1, 2):
            p = f"l{i}.mix." if at == 1 else f"l{i}.mlp."
            h = _rms(torch.einsum("tsw,s->tw", xs, W(f"l{i}.hc{at}.in")), W(f"l{i}.norm{at}"), eps)
            if at == 2:
                scores = torch.sigmoid(h @ W(p + "router").T)
                chosen = _grouped_choice(scores + W(p + "correction"), layer["mlp"]["router"], 2)
                weights = scores.gather(1, chosen)
                y = _routed(h, W, p, layer["mlp"], chosen, weights / weights.sum(-1, keepdim=True))
                y = y + torch.sigmoid(h @ W(p + "shared.sg").T) * _expert(h, W, p + "shared.", None)
            elif layer["type"] == "lightning":
                q, k, v = (_silu(h @ W(p + n).T).view(T, m["heads"], -1) for n in "qkv")
                o = _recur(q, k, v, torch.tensor(m["decay"], dtype=x.dtype, device=x.device)[None, :, None]).flatten(1)
                y = (_rms(o, W(p + "norm"), eps) * torch.sigmoid(h @ W(p + "g").T)) @ W(p + "o").T
            else:
                o, kept[i] = _latent_attention(m, W, p, h, eps, kept.get(m.get("kv_from")))
                y = o.flatten(1) @ W(p + "o").T
            y = y * W(f"l{i}.ls{at}")
            xs = torch.einsum("tsw,sr->trw", xs, W(f"l{i}.hc{at}.mix")) + W(f"l{i}.hc{at}.out")[None, :, None] * y[:, None, :]
    return _rms(xs.sum(1), W("final.norm"), eps), "embed"


def _plain_sopetar(config, W, ids):
    eps, T, first = config["norm"]["eps"], len(ids), None
    x = W("embed", ids) * config["embedding"]["scale"]
    states = [x]
    for i, layer in enumerate(config["layers"]):
        p, m, ff = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        u = _layer_norm(x, W(f"l{i}.norm1"), W(f"l{i}.norm1.b"), eps)
        if layer["type"] == "latent_attention":
            o, _ = _latent_attention(m, W, p, u, eps, None, _plain_freqs(m["rot"]["dims"], m["rot"]["base"]))
            o = o * torch.sigmoid(u @ W(p + "g").T)[..., None]
        else:
            q, k, v = (_rms((u @ W(p + n).T + W(f"{p}{n}.b")).view(T, -1, 128), None, eps) for n in "qkv")
            if first is None:
                first = v
            else:
                v = (1.0 - W(p + "vmix")) * v + W(p + "vmix") * first
            slopes = [2.0 ** (-8.0 * (h + 1) / m["heads"]) for h in range(m["heads"])]
            o = _attend(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], cap=m["softcap"], slopes=slopes)
        y, p = o.flatten(1) @ W(p + "o").T, f"l{i}.mlp."
        g, up = (u @ W(p + "gate").T + W(p + "gate.b")).clamp(max=ff["limit"]), (u @ W(p + "up").T + W(p + "up.b")).clamp(-ff["limit"], ff["limit"])
        y = y + (g * torch.sigmoid(1.702 * g) * (up + 1.0)) @ W(p + "down").T + W(p + "down.b")
        states.append(x + y)
        x = sum(a * s for a, s in zip(W(f"l{i}.dwa"), states))
    return _layer_norm(x, W("final.norm"), W("final.norm.b"), eps), "head"


def _plain_sokolorn(config, W, ids):
    eps, x, T, kept = config["norm"]["eps"], W("embed", ids), len(ids), {}
    for i, layer in enumerate(config["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        if layer["type"] == "attention":
            q, k = (_rms(x @ W(p + n).T, W(f"{p}{n}.norm"), eps).view(T, -1, 128) for n in "qk")
            o = _attend(q, k, (x @ W(p + "v").T).view(T, -1, 128), m["scale"], m["mask"]["size"], sink=W(p + "sink"))
            o = o * torch.sigmoid(x @ W(p + "g").T)[..., None]
        else:
            freqs = _slowed_freqs(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
            made = lambda n: _rotate(_rms((x @ W(p + n).T + W(f"{p}{n}.b")).view(T, -1, 128), W(f"{p}{n}.norm"), eps), freqs)
            source = m.get("kv_from")
            kept[i] = kept[source] if source is not None else (made("k"), (x @ W(p + "v").T + W(p + "v.b")).view(T, -1, 128))
            o = _attend(made("q"), *kept[i], m["scale"])
        x = x + _rms(o.flatten(1) @ W(p + "o").T, 1.0 + W(f"l{i}.norm1"), eps)
        p, ff = f"l{i}.mlp.", layer["mlp"]
        if ff["kind"] == "dense":
            y = torch.relu(x @ W(p + "up").T) ** 2 @ W(p + "down").T
        else:
            values, chosen = (x @ W(p + "router").T + W(p + "router.b")).topk(ff["router"]["top"], -1)
            y = _routed(x, W, p, ff, chosen, torch.softmax(values, -1))
            y = y + torch.sigmoid(x @ W(p + "shared.sg").T) * _expert(x, W, p + "shared.", ff["shared"]["limit"])
        x = x + _rms(y, 1.0 + W(f"l{i}.norm2"), eps)
    return _rms(x, 1.0 + W("final.norm"), eps), "embed"


def _plain_gelulix(config, W, ids):
    eps, x, T, a = config["norm"]["eps"], W("embed", ids), len(ids), config["postln_alpha"]
    for i, layer in enumerate(config["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        if layer["type"] == "channel_delta":
            y = _delta_of(m, W, p, x, eps)
        elif layer["type"] == "gla":
            q, k, v = ((x @ W(p + n).T).view(T, m["heads"], -1) for n in "qkv")
            decay = torch.sigmoid((x @ W(p + "a1").T) @ W(p + "a2").T + W(p + "a2.b")) ** (1.0 / m["tau"])
            o = _rms(_recur(q * m["dim"] ** -0.5, k, v, decay.view(T, m["heads"], -1)), W(p + "norm"), eps)
            y = (o.flatten(1) * _silu(x @ W(p + "g").T)) @ W(p + "o").T
        else:
            o, _ = _latent_attention(m, W, p, x, eps, None, *_yarn_freqs(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"]))
            y = o.flatten(1) @ W(p + "o").T
        x, p = _rms(a * x + y, W(f"l{i}.norm1"), eps), f"l{i}.mlp."
        y = (_silu(x @ W(p + "gate").T + W(p + "gate.b")) * (x @ W(p + "up").T + W(p + "up.b"))) @ W(p + "down").T + W(p + "down.b")
        x = _rms(a * x + y, W(f"l{i}.norm2"), eps)
    return _rms(x, W("final.norm"), eps), "head"


def _differential(m, W, p, x, eps):
    T, H, D = x.shape[0], m["heads"], m["dim"]
    q, k, v = (_conv(x @ W(p + n).T, W(p + n + ".conv")) for n in "qkv")
    freqs, mult = _yarn_freqs(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
    q, k = q.view(T, -1, 2, D), k.view(T, -1, 2, D)
    maps = [_attend(_rotate(q[:, :, i], freqs, mult), _rotate(k[:, :, i], freqs, mult), v.view(T, -1, m["vdim"]), m["scale"], m["mask"]["size"]) for i in (0, 1)]
    factor = torch.exp((W(p + "lq1") * W(p + "lk1")).sum()) - torch.exp((W(p + "lq2") * W(p + "lk2")).sum()) + m["diff"]
    return (_rms(maps[0] - factor * maps[1], None, eps) * (1.0 - m["diff"])).flatten(1) @ W(p + "o").T


def _state_space(m, W, p, x, eps):
    T, H, N, G, inner = x.shape[0], m["heads"], m["state"], m["groups"], m["heads"] * m["vdim"]
    z, mixed, dt = (x @ W(p + "in").T).split([inner, inner + 2 * G * N, H], -1)
    v, k, q = _silu(_conv(mixed, W(p + "conv"), W(p + "conv.b"))).split([inner, G * N, G * N], -1)
    v = v.view(T, H, -1)
    k, q = (t.view(T, G, N).repeat_interleave(H // G, 1) for t in (k, q))
    step = torch.nn.functional.softplus(dt + W(p + "dt_bias"), threshold=1e9)
    y = _recur(q, k * step[..., None], v, torch.exp(-torch.exp(W(p + "A_log")) * step)[..., None]) + W(p + "D")[:, None] * v
    return _grouped_rms(y.flatten(1) * _silu(z), W(p + "norm"), m["norm_groups"], eps) @ W(p + "o").T


def _plain_repolix(config, W, ids):
    eps = config["norm"]["eps"]
    mixers = {"attention": _differential, "mamba2": _state_space, "channel_delta": _delta_of}
    x = W("embed", ids) * config["embedding"]["scale"]
    for i, layer in enumerate(config["layers"]):
        x = x + W(f"l{i}.ls1") * mixers[layer["type"]](layer["mixer"], W, f"l{i}.mix.", _rms(x, W(f"l{i}.norm1"), eps), eps)
        h, p, ff = _rms(x, W(f"l{i}.norm2"), eps), f"l{i}.mlp.", layer["mlp"]
        scores = torch.softmax(h @ W(p + "router").T, -1)
        chosen = _grouped_choice(scores + W(p + "correction"), ff["router"], 1)
        y = _routed(h, W, p, ff, chosen, scores.gather(1, chosen)) + _expert(h, W, p + "shared.", ff["shared"]["limit"])
        x = x + W(f"l{i}.ls2") * y
    return _rms(x, W("final.norm"), eps), "head"


_PLAIN = {"qwen3": _plain_qwen3, "gopevik": _plain_gopevik, "niridra": _plain_niridra, "sopetar": _plain_sopetar, "sokolorn": _plain_sokolorn,
          "gelulix": _plain_gelulix, "repolix": _plain_repolix}


def exact(case, seed):
    """The logits of the pass from whole sequences in float64; None where that takes too long (batches of the 8B model over long
    contexts)."""
    lengths, config = _lengths(case), _config(case["model"])
    if case["model"] == "qwen3-8b" and sum(lengths) > 4608:
        return None
    weights, tokens = _weights(config), _tokens(case, seed)

    def W(name, rows=None):
        t = weights[name]
        return (t if rows is None else t[rows]).double()

    steps = _steps(case) if case["kind"] == "complete" else [[(i, n, 1, [0]) for i, n in enumerate(lengths)]]
    if case["kind"] == "decode":           # a state's first pass
        ends = [n + 1 for n in lengths]
    else:
        ends = [max(first + count for step in steps for r, first, count, _ in step if r == i) for i in range(len(lengths))]
    hidden = []
    for ids, end in zip(tokens, ends):
        x, head = _PLAIN[case["model"].split("-")[0]](config, W, torch.tensor(ids[:end], device="cuda"))
        hidden.append(x)
    x = torch.stack([hidden[i][first + w] for step in steps for i, first, _, want in step for w in want])
    logits = x @ W(head).T
    cap = config.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits
