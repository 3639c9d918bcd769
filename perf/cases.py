"""The work that is measured on this framework: requests served from their prompts to their last decoded token.

A pass admits the case's requests, runs their prompts (packed into steps of at most 8,192 tokens), decodes `new` tokens of
each in captured steps whose sampled tokens are read back as a serving loop does, and releases the requests.  The tokens
that are fed back are given with the case instead of the sampled ones, as when a known continuation is scored, so that
the logits of every step are comparable whatever a near tie between two tokens does.  A case with `late` > 0 also has a
prompt of that many tokens that arrives while the others decode and enters in portions of `portion` tokens beside them.

A pass returns the logits of every prompt's last token, [requests, vocab], and of every decoded token, [new, requests,
vocab] (and of the late prompt's last token).  The sampled tokens are their arg max and are not returned.
"""

import math
import random

import torch

from libmir_b200 import CacheConfig, Library, RuntimeConfig, SchedulerConfig, StepEntry
from libmir_b200.config.generation import GenerationConfig
from libmir_b200.engine.api import Model
from libmir_b200.models.decoder import DecoderModel
from libmir_b200.parts.base import BuildEnv
from libmir_b200.registry import build_spec
from libmir_b200.sampling import RequestSampler
from libmir_b200.weights.random_init import parameter_specs

STEP_TOKENS = 8192
F64 = torch.float64


# ------------------------------------------------------------------------------ the models and their sizes
def _dense(hidden, inter, layers, heads, kv_heads, vocab, theta, tied, qwen=True, scaling=None, positions=40960):
    config = {"architectures": ["Qwen3ForCausalLM" if qwen else "LlamaForCausalLM"], "model_type": "qwen3" if qwen else "llama",
              "hidden_size": hidden, "intermediate_size": inter, "num_hidden_layers": layers, "num_attention_heads": heads,
              "num_key_value_heads": kv_heads, "head_dim": 128, "vocab_size": vocab, "max_position_embeddings": positions,
              "rms_norm_eps": 1e-6 if qwen else 1e-5, "rope_theta": theta, "tie_word_embeddings": tied, "hidden_act": "silu"}
    return dict(config, rope_scaling=scaling) if scaling else config


_LLAMA3 = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
           "original_max_position_embeddings": 8192}
_YARN = {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}
_DIM = 128                                     # of an attention head, in every configuration here


def _wide(size):
    """(width, feed-forward, heads, key heads) of the two sizes every design is measured at."""
    return (2048, 8192, 16, 4) if size == "w2048" else (4096, 14336, 32, 8)


def _doderax(size, layers):
    width, ff, heads, kv, = _wide(size)
    delta = {"heads": heads, "kv_heads": heads, "dim": _DIM, "vdim": _DIM, "conv": 4, "decay_rank": 64, "gate_rank": 64}
    left = {"heads": heads, "kv_heads": kv, "dim": _DIM, "vdim": _DIM, "scale": _DIM ** -0.5,
            "rot": {"dims": 64, "base": 1e6}, "mask": {"size": width // 2, "keep_first": 4}}
    right = {"heads": heads, "kv_heads": heads // 2, "dim": _DIM, "vdim": _DIM, "conv": 4}
    mlp = {"kind": "dense", "ff": ff}
    return {"architecture": "Doderax", "vocab": 65536, "width": width, "logit_scale": 1.0, "norm": {"eps": 1e-6},
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 8191, "mul_cur": 131}},
            "layers": [{"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": mlp} if i % 4 == 3 else
                       {"type": "channel_delta", "mixer": delta, "mlp": mlp} for i in range(layers)]}


def _moe(size, **router):
    return {"kind": "moe", "expert": {"ff": _wide(size)[0] // 2}, "router": dict(router, top=6)}


def _latent(size, **more):
    heads = _wide(size)[2]
    return dict(more, heads=heads, dim=_DIM, rot_dim=64, vdim=_DIM, kv_rank=512, scale=192 ** -0.5)


def _wkv(size):
    return {"type": "wkv", "mixer": {"heads": _wide(size)[0] // 64, "dim": 64, "decay_rank": 64}}


def _zufotar(size, layers):
    width, ff, _, _ = _wide(size)
    latent = {"type": "latent_attention", "mixer": _latent(size, q_rank=3 * width // 8, rot={"dims": 64, "base": 1e6, "scaling": _YARN})}
    moe = dict(_moe(size, experts=64, scale=2.5, groups={"count": 8, "keep": 4}), shared={"ff": width})
    return {"architecture": "Zufotar", "vocab": 65536, "width": width, "norm": {"eps": 1e-6}, "embedding": {"scale": width ** 0.5},
            "logit_softcap": 30.0, "loop": {"start": 2, "stop": 4, "times": 2},
            "layers": [dict(latent if i % 2 == 0 else _wkv(size), mlp={"kind": "dense", "ff": ff} if i == 0 else moe) for i in range(layers)]}


def _dalesun(size, layers):
    width, ff, heads, kv = _wide(size)
    decay = [1.0 - 2.0 ** (-4.0 - 8.0 * h / heads) for h in range(heads)]
    retention = {"heads": heads, "dim": _DIM, "vdim": _DIM, "rot": {"dims": _DIM, "base": 5e5}, "decay": decay}
    attention = {"heads": heads, "kv_heads": kv, "dim": _DIM, "vdim": _DIM, "scale": _DIM ** -0.5,
                 "rot": {"dims": 64, "base": 1e4}, "mask": {"size": width // 2}}
    kinds = lambda i: {"type": "retention", "mixer": retention} if i % 4 < 2 else \
        {"type": "attention", "mixer": attention if i % 4 == 2 else dict(attention, kv_from=i - 1)}
    return {"architecture": "Dalesun", "vocab": 65536, "width": width, "norm": {"eps": 1e-5}, "residual_mult": 0.5,
            "layers": [dict(kinds(i), mlp={"kind": "dense", "ff": ff}) for i in range(layers)]}


def _gumazen(size, layers):
    width, ff, heads, kv = _wide(size)
    base = {"heads": heads, "kv_heads": kv, "dim": _DIM, "vdim": _DIM, "scale": _DIM ** -0.5}
    kinds = ({"type": "attention_3", "mixer": dict(base, rot={"dims": 64, "base": 1e6, "scaling": {
                 "factor": 4.0, "low": 1.0, "high": 4.0, "original": 4096}})},
             {"type": "attention_2", "mixer": dict(base, softcap=50.0, bias_max=width / 4.0, bias_rows=32, mask={"size": width // 2})},
             {"type": "attention", "mixer": dict(base, rot={"dims": _DIM, "base": 1e4})})
    moe = dict(_moe(size, experts=56, identity=8, scale=2.0, groups={"count": 8, "keep": 4}), shared={"ff": width})
    return {"architecture": "Gumazen", "vocab": 65536, "width": width, "norm": {"eps": 1e-5}, "streams": 4,
            "loop": {"start": 2, "stop": layers - 2, "times": 2},
            "layers": [dict(kinds[i % 3], mlp={"kind": "dense", "ff": ff} if i == 0 else moe) for i in range(layers)]}


def _pedotar(size, layers):
    width, ff, heads, kv = _wide(size)
    mlp = {"kind": "dense", "ff": ff}
    scan = {"type": "mamba1", "mlp": None, "mixer": {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4}}
    latent = {"type": "latent_attention", "mlp": mlp, "mixer": _latent(size, rot={"dims": 64, "base": 1e6})}
    mixed = {"type": "attention", "mlp": mlp, "mixer": {"heads": heads, "kv_heads": kv, "dim": _DIM, "vdim": _DIM,
                                                       "scale": _DIM ** -0.5, "mask": {"size": 1536}}}
    return {"architecture": "Pedotar", "vocab": 65536, "width": width, "norm": {"eps": 1e-5},
            "loop": {"start": 2, "stop": layers - 2, "times": 2}, "layers": [(scan, latent, scan, mixed)[i % 4] for i in range(layers)]}


def _biravik(size, layers):
    width, ff, heads, kv = _wide(size)
    decay = [1.0 - 2.0 ** (-4.0 - 8.0 * h / heads) for h in range(heads)]
    left = {"heads": heads, "kv_heads": kv, "dim": _DIM, "vdim": 64, "scale": _DIM ** -0.5, "q_temp": {"coef": 0.1, "every": 4096}}
    right = {"heads": heads, "dim": _DIM, "vdim": _DIM, "decay": decay}
    both = {"type": "parallel", "mixer": {"left": left, "left_scale": 0.7, "right": right, "right_scale": 0.7}}
    attention = {"type": "attention", "mixer": {"heads": heads, "kv_heads": kv, "dim": _DIM, "vdim": _DIM, "scale": _DIM ** -0.5,
                 "mask": {"size": width // 2, "keep_first": 4}, "rot": {"dims": _DIM, "base": 1e6, "scaling": _YARN}}}
    return {"architecture": "Biravik", "vocab": 65536, "width": width, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0},
            "postln_alpha": 2.0, "layers": [dict((_wkv(size), both, both, attention)[i % 4],
                                                 mlp=_moe(size, experts=64) if i % 2 else {"kind": "dense", "ff": ff}) for i in range(layers)]}


_DESIGNS = {"doderax": _doderax, "zufotar": _zufotar, "dalesun": _dalesun, "gumazen": _gumazen, "pedotar": _pedotar, "biravik": _biravik}


def config_of(case):
    """config.json of the case's model."""
    model, layers = case["model"], case["layers"]
    if model == "qwen3-4b":
        return _dense(2560, 9728, layers, 32, 8, 151936, 1e6, True)
    if model == "qwen3-32b":
        return _dense(5120, 25600, layers, 64, 8, 151936, 1e6, False)
    if model == "llama-3.1-8b":
        return _dense(4096, 14336, layers, 32, 8, 128256, 5e5, False, qwen=False, scaling=_LLAMA3, positions=131072)
    name, size = model.split("-")
    if name == "dense":
        width, ff, heads, kv = _wide(size)
        return _dense(width, -(-(2 * ff // 3) // 128) * 128, layers, heads, kv, 65536, 1e6, False, positions=16384)
    return _DESIGNS[name](size, layers)


# ------------------------------------------------------------------------------ the cases
def _case(name, model, layers, requests, prompt, new, late=0, portion=0, dtype="bfloat16", page=16):
    return {"name": name, "model": model, "layers": layers, "dtype": dtype, "requests": requests, "prompt": prompt, "new": new,
            "late": late, "portion": portion, "page": page}


def listed():
    return [
        # a person's short question to a chat model, nobody else there: latency of single tokens
        _case("question_4b", "qwen3-4b", 36, 1, 37, 12),
        # the usual serving batch: 8 conversations of a few hundred tokens, most of the time spent decoding
        _case("chat_4b_8", "qwen3-4b", 36, 8, 320, 24),
        # a busy server: many short requests at once, not a power of two
        _case("busy_4b_53", "qwen3-4b", 36, 53, 72, 10),
        # decoding beside a long prompt that arrives and enters in portions
        _case("mixed_8b_13", "llama-3.1-8b", 16, 13, 190, 10, late=1999, portion=512),
        # long documents through the largest layers
        _case("documents_32b", "qwen3-32b", 8, 3, 2730, 8),
        # the 32-bit path, as a numerical check of a checkpoint runs it
        _case("check_float32", "dense-w2048", 4, 3, 130, 6, dtype="float32"),
        # one case for each further architecture: documents of one to two thousand tokens and a short answer (a summary,
        # a label), one or a few at a time
        _case("doderax_w2048", "doderax-w2048", 12, 2, 1400, 8),
        _case("zufotar_w2048", "zufotar-w2048", 8, 3, 1100, 8),
        _case("dalesun_w4096", "dalesun-w4096", 8, 1, 2048, 8),
        _case("gumazen_w2048", "gumazen-w2048", 8, 3, 1000, 8),
        _case("pedotar_w4096", "pedotar-w4096", 6, 2, 1500, 8),
        _case("biravik_w2048", "biravik-w2048", 12, 1, 2011, 8),
    ]


_LIMIT = None


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    global _LIMIT
    if _LIMIT is None:
        _LIMIT = max(_cost(case) for case in listed())
    spread = lambda low, high: int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    while True:
        kind = rng.choice(("dense", "dense", "dense", "float32") + tuple(_DESIGNS))
        late = portion = 0
        page, dtype = rng.choice((16, 16, 32, 64)), "bfloat16"
        if kind == "dense":
            model, layers = rng.choice((("qwen3-4b", 36), ("qwen3-4b", 18), ("llama-3.1-8b", 16), ("qwen3-32b", 8), ("dense-w2048", 12)))
            requests, prompt, new = spread(1, 64), spread(16, 4000), rng.randint(2, 24)
            if rng.random() < 0.3:
                late, portion = spread(200, 3000), rng.choice((256, 384, 512, 1024))
        elif kind == "float32":
            model, layers, dtype = "dense-w2048", rng.randint(2, 6), "float32"
            requests, prompt, new = rng.randint(1, 6), spread(16, 300), rng.randint(2, 8)
        else:
            size = rng.choice(("w2048", "w4096")) if kind in ("doderax", "dalesun", "pedotar") else "w2048"
            layers = {"doderax": 12, "dalesun": 12, "biravik": 12}.get(kind, 8) if size == "w2048" else {"pedotar": 6}.get(kind, 8)
            model = f"{kind}-{size}"
            requests, prompt, new = spread(1, 12), spread(32, 3000), rng.randint(2, 12)
        case = _case("", model, layers, requests, prompt, new, late, portion, dtype, page)
        del case["name"]
        # requests of more than 20,000 tokens in all, or dearer than the largest listed case, are left out
        if requests * prompt + late <= 20000 and _cost(case) <= _LIMIT:
            return case


def _lengths(case):
    """Prompt lengths of the requests, ragged between a quarter of `prompt` and all of it."""
    n, longest = case["requests"], case["prompt"]
    return [max(1, longest - (i * 3 * longest) // (4 * n) - (i % 3 if longest > 8 else 0)) for i in range(n)]


def _tokens(case, seed, vocab):
    """[(prompt, continuation)] of every request, and the late prompt."""
    rng = random.Random(f"tokens {seed}")
    ids = lambda count: [rng.randrange(vocab) for _ in range(count)]
    return [(ids(n), ids(case["new"])) for n in _lengths(case)], ids(case["late"])


# ------------------------------------------------------------------------------ weights
def _weight(name, spec, config, seed, dtype, device):
    """The values of one stored tensor, in the dtype the engine keeps it in: matrices N(0, 0.02^2), those that end a branch
    smaller by the root of the number of branches, embeddings on the residual's own scale, norms around their neutral
    weight, decays and steps over the ranges such models are initialised to."""
    generator = torch.Generator(device=device)
    generator.manual_seed(random.Random(f"{seed} {name}").getrandbits(62))
    last = name.rsplit(".", 1)[-1]
    if last in ("dt_bias", "w0", "A_log") or ".mu." in name or name.endswith("dt.b"):
        u = torch.rand(spec.shape, generator=generator, device=device, dtype=F64)
        if ".mu." in name:
            values = u
        elif last == "w0":
            values = -6.0 + 5.0 * u
        elif last == "A_log" and len(spec.shape) == 2:
            values = torch.log(torch.arange(1, spec.shape[1] + 1, device=device, dtype=F64) * (0.9 + 0.2 * u))
        elif last == "A_log":
            values = torch.log(1.0 + 15.0 * u)
        else:
            step = torch.exp(math.log(1e-3) + math.log(100.0) * u)
            values = torch.log(torch.expm1(step))
    else:
        values = torch.randn(spec.shape, generator=generator, device=device, dtype=torch.float32)
        if last == "talk":
            values = 0.1 * values + torch.eye(spec.shape[0], device=device)
        elif last == "mix" and len(spec.shape) == 2 and spec.shape[0] == spec.shape[1] <= 16:
            values = 0.05 * values + torch.eye(spec.shape[0], device=device)
        elif ".hc" in name and last == "in":
            values = (1.0 + 0.1 * values) / spec.shape[0]
        elif last in ("conv", "sink", "rel", "u"):
            values = 0.5 * values
        elif spec.init == "ones":
            values = 1.0 + 0.1 * values
        elif "norm" in name and spec.init == "zeros" and not name.endswith(".b"):
            values = 0.1 * values
        elif name in ("embed", "model.embed_tokens.weight"):
            values = {"Zufotar": 0.02, "Pedotar": 0.3, None: 0.3}.get(config.get("architecture"), 1.0) * values
        elif last in ("o", "down") or name.endswith(("o_proj.weight", "down_proj.weight")):
            values = 0.02 / math.sqrt(2 * len(_layer_runs(config))) * values
        else:
            values = 0.02 * values
    return values.to({"float32": torch.float32}.get(spec.store, dtype))


# ------------------------------------------------------------------------------ the measured path
def prepare(case, seed):
    """A loaded model, its cache, and the requests' tokens."""
    dtype, device = getattr(torch, case["dtype"]), torch.device("cuda", 0)
    config = config_of(case)
    longest = max(_lengths(case)) + case["new"]
    pages = case["requests"] * (-(-longest // case["page"]) + 1) + -(-(case["late"] + 1) // case["page"]) + 8
    library = Library(RuntimeConfig(
        kv_cache=CacheConfig(block_size=case["page"], block_count=pages),
        scheduler=SchedulerConfig(max_batch_requests=case["requests"] + 1, max_batch_tokens=STEP_TOKENS), dtype=case["dtype"]))
    decoder = DecoderModel(build_spec(config, None), BuildEnv(dtype, device))
    decoder.bind({name: _weight(name, spec, config, seed, dtype, device) for name, (_, _, spec) in decoder.parameter_table().items()})
    model = Model(library, decoder, GenerationConfig(), None, config)
    requests, late = _tokens(case, seed, config.get("vocab") or config["vocab_size"])
    return {"model": model, "requests": requests, "late": late, "portion": case["portion"], "new": case["new"]}


def run(state):
    model, requests, late = state["model"], state["requests"], state["late"]
    samplers = [RequestSampler() for _ in requests]
    for index in range(len(requests)):
        model.admit(index)
    first, batch, waiting = [], [], 0
    for index, (prompt, _) in enumerate(requests):                   # the prompts, as many as fit into each step
        if batch and waiting + len(prompt) > STEP_TOKENS:
            first.append(model.step(batch, samplers[:len(batch)]).logits.clone())
            batch, waiting = [], 0
        batch.append(StepEntry(index, prompt, [len(prompt) - 1]))
        waiting += len(prompt)
    result = model.step(batch, samplers[:len(batch)])
    first.append(result.logits.clone())
    result.tokens.tolist()
    if late:
        model.admit("late")
    entered, after, late_logits = 0, [], None
    for step in range(state["new"]):
        entries = [StepEntry(index, [continuation[step]], [0]) for index, (_, continuation) in enumerate(requests)]
        rows = len(entries)
        if entered < len(late):
            part = late[entered:entered + state["portion"]]
            entered += len(part)
            entries.append(StepEntry("late", part, [len(part) - 1] if entered == len(late) else []))
        with_late = len(entries) > rows and entered == len(late)
        result = model.step(entries, samplers + [RequestSampler()] if with_late else samplers)
        after.append(result.logits[:rows].clone())
        if with_late:
            late_logits = result.logits[rows:].clone()
        result.tokens.tolist()                                       # what a serving loop streams to its users
    for index in range(len(requests)):
        model.release(index)
    if late:
        model.release("late")
    outputs = {"prompt": torch.cat(first), "decode": torch.stack(after)}
    if late_logits is not None:
        outputs["late"] = late_logits
    return outputs


def tolerance(case):
    # Four times the distance of the logits from 64 bits.  32-bit: 2.7e-6.  bfloat16 activations through 8 to 36 layers:
    # 0.002 to 0.013; a row whose token's last two experts nearly tie may move by a few tenths of the logits' size.
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5}
    return {"rel": 0.03, "max": 0.5}


# ------------------------------------------------------------------------------ what a pass cannot do without
def _layer_runs(config):
    """Layer indices in the order they run."""
    count = config.get("num_hidden_layers") or len(config["layers"])
    loop = config.get("loop")
    if not loop:
        return list(range(count))
    return list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], count))


def _mixer_costs(config, index):
    """[(flops for each visible key, bytes of a cached key, window)] of the attentions of a layer, and (flops for each
    token, 32-bit numbers kept for each request) of its recurrences."""
    if "layers" not in config:
        d = config["head_dim"]
        return [(4 * d * config["num_attention_heads"], 2 * d * config["num_key_value_heads"], None)], 0, 0
    layer = config["layers"][index]
    attentions, flops, kept = [], 0, 0
    mixers = [layer["mixer"]] if layer["type"] != "parallel" else [layer["mixer"]["left"], layer["mixer"]["right"]]
    for place, m in enumerate(mixers):
        kind = layer["type"] if layer["type"] != "parallel" else ("attention", "recurrence")[place]
        if kind == "latent_attention":
            attentions.append((2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), m["kv_rank"] + m["rot_dim"], None))
        elif kind.startswith("attention"):
            attentions.append((2 * m["heads"] * (m["dim"] + m["vdim"]), (m["dim"] + m["vdim"]) * m["kv_heads"], (m.get("mask") or {}).get("size")))
        elif kind == "mamba1":
            flops, kept = flops + 6 * m["inner"] * m["state"], kept + m["inner"] * m["state"]
        else:
            cells = m["heads"] * m["dim"] * m.get("vdim", m["dim"])
            flops, kept = flops + (8 if kind == "channel_delta" or "conv" in m else 5) * cells, kept + cells
    return attentions, flops, kept


def work(case):
    config = config_of(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    runs = _layer_runs(config)
    times = {index: runs.count(index) for index in runs}
    dense = experts = 0                                              # weights read by every token; weights of all experts
    width = config.get("width") or config["hidden_size"]
    vocab = config.get("vocab") or config["vocab_size"]
    routed = 0
    for name, spec in parameter_specs(config).items():
        if len(spec.shape) != 2 or name.startswith(("embed", "model.embed", "bigram", "head", "lm_head")):
            continue
        parts = name.split(".")
        index = int(parts[2]) if "layers" in parts else int(parts[0][1:]) if parts[0][1:].isdigit() else None
        count = spec.shape[0] * spec.shape[1] * (times.get(index, 1) if index is not None else 1)
        if ".mlp.e" in name:
            experts += count
        else:
            dense += count
    router = next((l["mlp"]["router"] for l in config.get("layers", []) if (l.get("mlp") or {}).get("router")), None)
    share = 0.0
    if router:
        share = router["top"] / (router["experts"] + router.get("identity", 0))
        routed = experts
    lengths = _lengths(case)
    steps, waiting = [], []
    for n in lengths:
        if waiting and sum(t for t, _ in waiting) + n > STEP_TOKENS:
            steps.append(waiting)
            waiting = []
        waiting.append((n, 0))
    steps.append(waiting)
    entered = 0
    for step in range(case["new"]):
        rows = [(1, n + step) for n in lengths]
        if entered < case["late"]:
            part = min(case["portion"], case["late"] - entered)
            rows.append((part, entered))
            entered += part
        steps.append(rows)
    flops = moved = 0.0
    for rows in steps:
        tokens = sum(t for t, _ in rows)
        moved += size * (dense + routed * (1.0 - (1.0 - share) ** tokens) + vocab * width + tokens * width)
        moved += 4 * vocab * len(rows)
        flops += 2.0 * tokens * (dense + routed * share) + 2.0 * vocab * width * len(rows)
        for index in runs:
            attentions, scan_flops, kept = _mixer_costs(config, index)
            flops += scan_flops * tokens
            moved += 4 * kept * len(rows) * 2
            for each, key_bytes, window in attentions:
                for t, before in rows:
                    seen = sum(min(p + 1, window) for p in range(before, before + t)) if window else t * before + t * (t + 1) / 2
                    flops += each * seen
                    moved += size * key_bytes * (min(before, window) if window else before) + size * key_bytes * t
    return {"bytes": moved, "flops": flops}


# ------------------------------------------------------------------------------ the same in 64 bits, plainly
def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, weight, bias, eps):
    centred = x - x.mean(-1, keepdim=True)
    return centred * torch.rsqrt((centred * centred).mean(-1, keepdim=True) + eps) * weight + bias


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.where(x > 30, x, torch.log1p(torch.exp(x.clamp(max=30))))


def _frequencies(dims, base, scaling, device):
    """(frequency of every pair, factor on the rotated values); the three rules of stretching that the models use."""
    f = base ** (-torch.arange(0, dims, 2, dtype=F64) / dims)
    factor = 1.0
    if scaling and "fast" in scaling:                                # by the number of turns in the original context
        turn = lambda t: dims * math.log(scaling["original"] / (2 * math.pi * t)) / (2 * math.log(base))
        low, high = max(math.floor(turn(scaling["fast"])), 0), min(math.ceil(turn(scaling["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=F64) - low) / max(high - low, 0.001)).clamp(0, 1)
        f, factor = f / scaling["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0
    elif scaling:                                                    # by the wavelength
        low, high = scaling.get("low", scaling.get("low_freq_factor")), scaling.get("high", scaling.get("high_freq_factor"))
        original = scaling.get("original", scaling.get("original_max_position_embeddings"))
        smooth = ((original * f / (2 * math.pi) - low) / (high - low)).clamp(0, 1)
        f = f / scaling["factor"] * (1 - smooth) + f * smooth
    return f.to(torch.float32).to(device), factor


def _rotate(x, rot, interleaved=False):
    """x [n, heads, d] of one request from its first token; the angle is a 32-bit product."""
    dims = rot["dims"]
    f, factor = _frequencies(dims, rot["base"], rot.get("scaling"), x.device)
    angle = (torch.arange(x.shape[0], device=x.device, dtype=torch.float32)[:, None] * f).to(F64)
    cos, sin = (torch.cos(angle) * factor)[:, None], (torch.sin(angle) * factor)[:, None]
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., a] = x[..., a] * cos - x[..., b] * sin
    out[..., b] = x[..., b] * cos + x[..., a] * sin
    return out


def _attend(q, k, v, scale, window=None, keep=0, sink=None, cap=None, rel=None, farthest=None, slope=None, chunk=None, talk=None):
    """q [n, H, d], k [n, G, d], v [n, G, e] -> [n, H * e], causal."""
    n, heads = q.shape[:2]
    group = heads // k.shape[1]
    i, j = torch.arange(n, device=q.device)[:, None], torch.arange(n, device=q.device)[None, :]
    hidden = j > i
    if window:
        hidden = hidden | ((i - j >= window) & (j >= keep))
    if chunk:
        hidden = hidden | (i // chunk != j // chunk)
    buckets = None
    if rel is not None:
        rows, exact_rows = rel.shape[0], rel.shape[0] // 2
        distance = (i - j).clamp(min=0)
        far = exact_rows + torch.floor(torch.log(distance.clamp(min=1).to(F64) / exact_rows) / math.log(farthest / exact_rows)
                                       * (rows - exact_rows)).long()
        buckets = torch.where(distance < exact_rows, distance, far.clamp(max=rows - 1))
    out = torch.zeros(n, heads, v.shape[2], dtype=F64, device=q.device)
    for head in range(heads):
        s = (q[:, head] @ k[:, head // group].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if rel is not None:
            s = s + rel[:, head][buckets]
        if slope is not None:
            s = s - slope[head] * (i - j)
        s = s.masked_fill(hidden, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = top.clamp(min=float(sink[head]))
        s = torch.exp(s - top)
        total = s.sum(-1, keepdim=True)
        if sink is not None:
            total = total + torch.exp(sink[head] - top)
        s = s / total
        if talk is None:
            out[:, head] += s @ v[:, head // group]
        else:                                                        # every head takes a share of this head's weights
            for g in range(v.shape[1]):
                mixed = s @ v[:, g]
                out[:, g * group:(g + 1) * group] += talk[g * group:(g + 1) * group, head][None, :, None] * mixed[:, None]
    return out.reshape(n, -1)


def _padded(parts, value=0.0):
    """[n_i, ...] of every request -> [longest, requests, ...]: the recurrences walk all requests at once."""
    longest = max(p.shape[0] for p in parts)
    out = torch.full((longest, len(parts)) + tuple(parts[0].shape[1:]), value, dtype=F64, device=parts[0].device)
    for r, p in enumerate(parts):
        out[:p.shape[0], r] = p
    return out


def _unpadded(x, counts):
    return torch.cat([x[:n, r] for r, n in enumerate(counts)])


class _Plain:
    """Whole sequences through one model, in 64 bits; x holds the requests' tokens one behind the other."""

    def __init__(self, config, weight, counts, device):
        self.c, self.w, self.counts, self.device = config, weight, counts, device

    def each(self, function, *rows):
        """function on every request's rows."""
        cut = [r.split(self.counts) for r in rows]
        return torch.cat([function(*parts) for parts in zip(*cut)])

    def scan(self, step, *rows):
        """step(t, inputs of all requests) -> read-out, token after token."""
        padded = [_padded(r.split(self.counts)) for r in rows]
        return _unpadded(torch.stack([step(*(p[t] for p in padded)) for t in range(padded[0].shape[0])]), self.counts)

    # -- recurrences
    def conv(self, x, taps, bias=None):
        def one(part):
            wide = torch.cat([part.new_zeros(taps.shape[1] - 1, part.shape[1]), part])
            return sum(wide[j:j + part.shape[0]] * taps[:, j] for j in range(taps.shape[1]))
        y = self.each(one, x)
        return _silu(y if bias is None else y + bias)

    def linear_state(self, q, k, v, decay, silu=False, rot=None):
        """S <- decay S + k v^T, read as S^T q; [n, H, d]; decay [H]."""
        if rot:
            q, k = (self.each(lambda part: _rotate(part, rot), x) for x in (q, k))
        if silu:
            q, k, v = _silu(q), _silu(k), _silu(v)
        else:
            k = k * k.shape[2] ** -0.5
        g = torch.tensor(decay, dtype=F64, device=self.device)[:, None, None]
        box = [torch.zeros(len(self.counts), q.shape[1], k.shape[2], v.shape[2], dtype=F64, device=self.device)]

        def step(qt, kt, vt):
            box[0] = g * box[0] + kt[..., :, None] * vt[..., None, :]
            return (qt[..., None, :] @ box[0])[..., 0, :]
        return self.scan(step, q, k, v)

    def delta(self, h, p, m, channel):
        w, n = self.w, h.shape[0]
        heads, groups, d, e, eps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], self.c["norm"]["eps"]
        q, k, v = (self.conv(h @ w(p + x).T, w(p + x + ".conv")) for x in "qkv")
        unit = lambda x: x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)
        q, k, v = unit(q.view(n, groups, d)) * d ** -0.5, unit(k.view(n, groups, d)), v.view(n, heads, e)
        q, k = (x.repeat_interleave(heads // groups, 1) for x in (q, k))
        beta, rate = torch.sigmoid(h @ w(p + "b").T), torch.exp(w(p + "A_log"))[:, None]
        if channel:
            raw = (h @ w(p + "a1").T) @ w(p + "a2").T + w(p + "dt_bias")
            decay, gate = torch.exp(-rate * _softplus(raw.view(n, heads, d))), torch.sigmoid((h @ w(p + "g1").T) @ w(p + "g2").T)
        else:
            decay = torch.exp(-rate * _softplus(h @ w(p + "a").T + w(p + "dt_bias"))[:, :, None]).expand(n, heads, d)
            gate = _silu(h @ w(p + "g").T)
        box = [torch.zeros(len(self.counts), heads, d, e, dtype=F64, device=self.device)]

        def step(qt, kt, vt, bt, gt):
            s = gt[..., :, None] * box[0]
            u = bt[..., None] * (vt - (kt[..., None, :] @ s)[..., 0, :])
            box[0] = s + kt[..., :, None] * u[..., None, :]
            return (qt[..., None, :] @ box[0])[..., 0, :]
        read = self.scan(step, q, k, v, beta, decay)
        return ((_rms(read, eps) * w(p + "norm")).reshape(n, -1) * gate) @ w(p + "o").T

    def wkv(self, h, p, m):
        w, n, heads, d = self.w, h.shape[0], m["heads"], m["dim"]
        before = self.each(lambda part: torch.cat([part.new_zeros(1, part.shape[1]), part[:-1]]), h)
        mix = lambda x: h + (before - h) * w(p + "mu." + x)
        r, k, v = ((mix(x) @ w(p + x).T).view(n, heads, d) for x in "rkv")
        decay = torch.exp(-torch.exp(torch.tanh(mix("w") @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0"))).view(n, heads, d)
        bonus = w(p + "u").reshape(heads, d, 1)
        box = [torch.zeros(len(self.counts), heads, d, d, dtype=F64, device=self.device)]

        def step(rt, kt, vt, gt):
            outer = kt[..., :, None] * vt[..., None, :]
            out = (rt[..., None, :] @ (box[0] + bonus * outer))[..., 0, :]
            box[0] = gt[..., :, None] * box[0] + outer
            return out
        out = _rms(self.scan(step, r, k, v, decay), self.c["norm"]["eps"]).reshape(n, -1) * w(p + "norm")
        return (out * _silu(mix("g") @ w(p + "g").T)) @ w(p + "o").T

    def mamba(self, h, p, m):
        w, rank, n = self.w, m["dt_rank"], m["state"]
        x, z = (h @ w(p + "in").T).split(m["inner"], 1)
        x = self.conv(x, w(p + "conv"), w(p + "conv.b"))
        low = x @ w(p + "x").T
        step_size, a = _softplus(low[:, :rank] @ w(p + "dt").T + w(p + "dt.b")), -torch.exp(w(p + "A_log"))
        box = [torch.zeros(len(self.counts), m["inner"], n, dtype=F64, device=self.device)]

        def step(xt, dt, bt, ct):
            box[0] = torch.exp(dt[..., None] * a) * box[0] + (dt * xt)[..., None] * bt[:, None, :]
            return (box[0] @ ct[..., None])[..., 0]
        y = self.scan(step, x, step_size, low[:, rank:rank + n].contiguous(), low[:, rank + n:].contiguous()) + w(p + "D") * x
        return (y * _silu(z)) @ w(p + "o").T

    # -- attention
    def latent(self, h, p, m, interleaved):
        w, n, heads, d, rank, eps = self.w, h.shape[0], m["heads"], m["dim"], m["kv_rank"], self.c["norm"]["eps"]
        q = (_rms(h @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T if "q_rank" in m else h @ w(p + "q").T
        down = h @ w(p + "dkv").T
        latent = _rms(down[:, :rank], eps) * w(p + "dkv.norm")
        q, turned = q.view(n, heads, -1), down[:, rank:].reshape(n, 1, -1)
        keys, values = (latent @ w(p + "uk").T).view(n, heads, d), (latent @ w(p + "uv").T).view(n, heads, -1)

        def one(q, k, kr, v):
            q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"], interleaved)], -1)
            k = torch.cat([k, _rotate(kr, m["rot"], interleaved).expand(-1, heads, -1)], -1)
            return _attend(q, k, v, m["scale"])
        mixed = self.each(one, q, keys, turned, values)
        return (mixed * torch.sigmoid(h @ w(p + "g").T) if "q_rank" in m else mixed) @ w(p + "o").T

    def project(self, h, p, name, heads, biases):
        y = h @ self.w(p + name).T
        if biases:
            y = y + self.w(p + name + ".b")
        return y.view(h.shape[0], heads, -1)

    def attention(self, h, p, m, kind, lent):
        """The softmax attentions of the designs (`kind`: the design's name and the layer's type)."""
        w, eps, n = self.w, self.c["norm"]["eps"], h.shape[0]
        heads, kv = m["heads"], m["kv_heads"]
        rot, window = m.get("rot"), (m.get("mask") or {}).get("size")
        biases = kind in ("Dalesun", "Gumazen attention_3")
        norm = lambda x, name: _rms(x, eps) * w(p + name)
        whole = lambda x, name: (_rms(x.reshape(n, -1), eps) * w(p + name)).view(x.shape)
        q = self.project(h, p, "q", heads, biases)
        borrowed = kind == "Dalesun" and m.get("kv_from") is not None
        k = None if borrowed else self.project(h, p, "k", kv, biases)
        v = None if borrowed else k if kind == "Biravik attention" else self.project(h, p, "v", kv, biases)
        turn = lambda x: self.each(lambda part: _rotate(part, rot, kind in ("Dalesun", "Biravik attention")), x) if rot else x
        options = {"window": window}
        if kind in ("Dalesun", "Pedotar", "Biravik attention", "Biravik left"):
            q, k = turn(norm(q, "q.norm")), k if borrowed else turn(norm(k, "k.norm"))
        elif kind in ("Gumazen attention_2", "Gumazen attention_3"):
            q, k = turn(whole(q, "q.norm")), turn(whole(k, "k.norm"))
        elif kind == "Gumazen attention":
            q, k = _rms(turn(q), eps), _rms(turn(k), eps)
            options["sink"] = torch.zeros(heads, dtype=F64)
        else:
            q, k = turn(q), turn(k)
        if kind == "Dalesun":
            if borrowed:
                k, v = lent[m["kv_from"]]
            else:
                lent[int(p[1:].split(".")[0])] = (k, v)
        if kind in ("Dalesun", "Biravik attention", "Biravik left"):
            options["sink"] = w(p + "sink")
        if kind in ("Doderax", "Biravik attention"):
            options["keep"] = m["mask"]["keep_first"]
        if kind == "Gumazen attention_2":
            options.update(cap=m["softcap"], rel=w(p + "rel"), farthest=m["bias_max"])
        if kind == "Pedotar":
            options = {"chunk": window, "talk": w(p + "talk")}
        if kind == "Biravik left":
            options["slope"] = [2.0 ** (-8.0 * (head + 1) / heads) for head in range(heads)]
            warm = lambda x: x * (1 + m["q_temp"]["coef"] * torch.log(torch.floor(
                (torch.arange(x.shape[0], device=x.device, dtype=F64) + 1) / m["q_temp"]["every"]) + 1))[:, None, None]
            q = self.each(warm, q)
        mixed = self.each(lambda q, k, v: _attend(q, k, v, m["scale"], **options), q, k, v)
        if kind in ("Dalesun", "Biravik attention", "Biravik left"):
            mixed = mixed * torch.sigmoid(h @ w(p + "g").T)
        elif kind == "Gumazen attention_2":
            mixed = (mixed.view(n, heads, -1) * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).reshape(n, -1)
        out = mixed @ w(p + "o").T
        return out + w(p + "o.b") if kind == "Gumazen attention_3" else out

    # -- feed-forwards
    def gated(self, h, p):
        return (_silu(h @ self.w(p + "gate").T) * (h @ self.w(p + "up").T)) @ self.w(p + "down").T

    def experts(self, h, p, mlp, name):
        w, router = self.w, mlp["router"]
        logits = h @ w(p + "router").T
        if name == "Biravik":
            picked, chosen = logits.topk(router["top"], -1)
            share = torch.softmax(picked, -1)
        else:
            scores = torch.sigmoid(logits) if name == "Zufotar" else torch.softmax(logits, -1)
            choice = scores + w(p + "correction")
            grouped = choice.view(h.shape[0], router["groups"]["count"], -1)
            best = grouped.topk(2, -1).values.sum(-1) if name == "Zufotar" else grouped.amax(-1)
            allowed = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(router["groups"]["keep"], -1).indices, True)
            chosen = grouped.masked_fill(~allowed[..., None], -math.inf).view_as(choice).topk(router["top"], -1).indices
            share = scores.gather(1, chosen)
            share = share / (share.sum(-1, keepdim=True) + 1e-20) * router["scale"]
        out = torch.zeros_like(h)
        for e in range(router["experts"]):
            rows, place = (chosen == e).nonzero(as_tuple=True)
            if rows.numel():
                out[rows] += share[rows, place][:, None] * self.gated(h[rows], f"{p}e{e}.")
        out = out + (share * (chosen >= router["experts"])).sum(-1, keepdim=True) * h    # the experts that change nothing
        if mlp.get("shared"):
            fed = self.gated(h, p + "shared.")
            out = out + (fed * torch.sigmoid(h @ w(p + "shared.sg").T) if name == "Zufotar" else fed)
        return out

    def feed(self, h, p, mlp, name):
        if mlp["kind"] == "moe":
            return self.experts(h, p, mlp, name)
        if name == "Pedotar":
            return self.gated(h, p)
        up = h @ self.w(p + "up").T
        if name == "Doderax":
            up = 0.5 * up * (1 + torch.tanh(math.sqrt(2 / math.pi) * (up + 0.044715 * up ** 3)))
        elif name == "Zufotar":
            up = 0.5 * up * (1 + torch.erf(up / math.sqrt(2)))
        else:
            up = torch.relu(up) ** 2
        return up @ self.w(p + "down").T

    # -- the models
    def dense(self, ids):
        c, w, eps = self.c, self.w, self.c["rms_norm_eps"]
        heads, kv, d, n = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], len(ids)
        rot = {"dims": d, "base": c["rope_theta"], "scaling": c.get("rope_scaling")}
        x = w("model.embed_tokens.weight")[ids]
        for index in range(c["num_hidden_layers"]):
            p = f"model.layers.{index}."
            h = _rms(x, eps) * w(p + "input_layernorm.weight")
            q, k, v = ((h @ w(p + f"self_attn.{a}_proj.weight").T).view(n, -1, d) for a in "qkv")
            if c["model_type"] == "qwen3":
                q, k = (_rms(y, eps) * w(p + f"self_attn.{a}_norm.weight") for y, a in ((q, "q"), (k, "k")))
            one = lambda q, k, v: _attend(_rotate(q, rot), _rotate(k, rot), v, d ** -0.5)
            x = x + self.each(one, q, k, v) @ w(p + "self_attn.o_proj.weight").T
            h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
            x = x + (_silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
        return x, lambda rows: (_rms(rows, eps) * w("model.norm.weight")) @ w(
            "model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight").T

    def mixer(self, h, p, layer, name, lent):
        kind, m, eps = layer["type"], layer["mixer"], self.c["norm"]["eps"]
        w, n = self.w, h.shape[0]
        if kind == "wkv":
            return self.wkv(h, p, m)
        if kind == "mamba1":
            return self.mamba(h, p, m)
        if kind == "latent_attention":
            return self.latent(h, p, m, name == "Zufotar")
        if kind == "channel_delta":
            return self.delta(h, p, m, True)
        if kind == "retention":
            q, k, v = ((h @ w(p + a).T).view(n, m["heads"], -1) for a in "qkv")
            read = self.linear_state(q, k, v, m["decay"], rot=m["rot"])
            return (_rms(read, eps).reshape(n, -1) * _silu(h @ w(p + "g").T)) @ w(p + "o").T
        if kind == "parallel" and name == "Doderax":
            left = self.attention(h, p + "left.", m["left"], "Doderax", lent)
            right = self.delta(h, p + "right.", m["right"], False)
            return 0.5 * (_rms(left, eps) * w(p + "left.out") + _rms(right, eps) * w(p + "right.out"))
        if kind == "parallel":
            r, left = p + "right.", self.attention(h, p + "left.", m["left"], "Biravik left", lent)
            q, k, v = ((h @ w(r + a).T).view(n, m["right"]["heads"], -1) for a in "qkv")
            read = self.linear_state(q, k, v, m["right"]["decay"], silu=True).reshape(n, -1)
            right = (_rms(read, eps) * w(r + "norm") * torch.sigmoid(h @ w(r + "g").T)) @ w(r + "o").T
            return m["left_scale"] * left + m["right_scale"] * right
        return self.attention(h, p, m, name if name in ("Dalesun", "Pedotar") else f"{name} {kind}", lent)

    def design(self, ids):
        c, w, eps, name = self.c, self.w, self.c["norm"]["eps"], self.c["architecture"]
        x = w("embed")[ids] * (c.get("embedding") or {}).get("scale", 1.0)
        pairs = (c.get("embedding") or {}).get("bigram")
        if pairs:
            row = lambda part: torch.cat([part.new_full((1,), pairs["buckets"]),
                                          (part[:-1] * pairs["mul_prev"] + part[1:] * pairs["mul_cur"]) % pairs["buckets"]])
            x = x + w("bigram")[self.each(row, ids)]
        plus = lambda y, key: _rms(y, eps) * (1 + w(key))
        plain = lambda y, key: _rms(y, eps) * w(key)
        around = lambda y, key: _layer_norm(y, w(key), w(key + ".b"), eps)
        if name == "Dalesun":
            x = plus(x, "embed.norm")
        embedded, loop, lent, opened = x, c.get("loop"), {}, 0
        streams = x[None].repeat(c["streams"], 1, 1) if name == "Gumazen" else None
        for index in _layer_runs(c):
            layer, p = c["layers"][index], f"l{index}."
            if loop and index == loop["start"]:
                if opened and name in ("Zufotar", "Pedotar"):
                    x = x + embedded
                if name == "Zufotar":
                    x = x + w("loop.step")[opened]
                opened += 1
            mix = lambda h: self.mixer(h, p + "mix.", layer, name, lent)
            feed = lambda h: self.feed(h, p + "mlp.", layer["mlp"], name)
            if name == "Doderax":
                h = plus(x, p + "norm1")
                x = x + mix(h) + feed(h)
            elif name == "Zufotar":
                x = x + mix(plain(x, p + "norm1")) + feed(plain(x, p + "norm2"))
            elif name == "Dalesun":
                x = x + c["residual_mult"] * plus(mix(x), p + "norm1")
                x = x + c["residual_mult"] * plus(feed(x), p + "norm2")
            elif name == "Biravik":
                x = plus(c["postln_alpha"] * x + mix(x), p + "norm1")
                x = plus(c["postln_alpha"] * x + feed(x), p + "norm2")
            elif name == "Pedotar":
                x = x + around(mix(around(x, p + "norm1")), p + "norm1b")
                if layer.get("mlp"):
                    x = x + around(feed(around(x, p + "norm2")), p + "norm2b")
            else:
                for number, sublayer in ((1, mix), (2, feed)):
                    hc = f"{p}hc{number}."
                    y = sublayer(around((w(hc + "in")[:, None, None] * streams).sum(0), f"{p}norm{number}"))
                    streams = torch.einsum("st,sxw->txw", w(hc + "mix"), streams) + w(hc + "out")[:, None, None] * y
        if name == "Gumazen":
            x = streams.sum(0)

        def head(rows):
            rows = around(rows, "final.norm") if name in ("Gumazen", "Pedotar") else plain(rows, "final.norm") \
                if name == "Zufotar" else plus(rows, "final.norm")
            logits = rows @ w("embed" if name in ("Zufotar", "Pedotar") else "head").T * c.get("logit_scale", 1.0)
            cap = c.get("logit_softcap")
            return cap * torch.tanh(logits / cap) if cap else logits
        return x, head


def exact(case, seed, device="cuda"):
    """Every request as one whole sequence (prompt and continuation), without a cache, in 64 bits."""
    if work(case)["flops"] > 2.5e14:                                 # over about 20 seconds
        return None
    config, dtype = config_of(case), getattr(torch, case["dtype"])
    specs = parameter_specs(config)
    weight = lambda name: _weight(name, specs[name], config, seed, dtype, device).to(F64)
    requests, late = _tokens(case, seed, config.get("vocab") or config["vocab_size"])
    wholes = [prompt + continuation for prompt, continuation in requests] + ([late] if late else [])
    counts = [len(ids) for ids in wholes]
    plain = _Plain(config, weight, counts, device)
    ids = torch.tensor([i for whole in wholes for i in whole], device=device)
    x, head = plain.design(ids) if "architecture" in config else plain.dense(ids)
    starts = [sum(counts[:r]) for r in range(len(counts))]
    last = torch.tensor([starts[r] + len(prompt) - 1 for r, (prompt, _) in enumerate(requests)], device=device)
    outputs = {"prompt": head(x[last])}
    outputs["decode"] = torch.stack([head(x[last + 1 + step]) for step in range(case["new"])])
    if late and -(-len(late) // case["portion"]) <= case["new"]:
        outputs["late"] = head(x[-1:])
    return outputs
