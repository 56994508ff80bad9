"""What the engine is asked to do, as cases that can be timed and compared.

A case is one kind of work over one decoder at one of the layer sizes that ``bench.py`` measures:

* ``prompt``: whole prompts of unequal lengths in one step, the logits of their last positions wanted (what admission
  of new requests, scoring and trace replay do);
* ``decode``: requests with contexts of unequal lengths go on from them token by token, every step's logits read (what
  serving does nearly all of the time). Each pass continues forks of the same contexts, so that passes are equal;
* ``mixed``: steps of continuous batching: decoded tokens of many requests beside the next portion of a prompt.

All of it goes through ``Engine.step``, ``Engine.fork`` and ``Engine.release``, on random weights. Widths of matrices,
heads and experts are those of the 0.6B- and 8B-shaped layers; where depth only repeats the same layers there are fewer
of them. ``exact`` is the same decoders in 64 bits, whole sequences under a mask, in plain torch.
"""
import math
import random

import torch

QWEN3_SIZES = {"0.6b": (28, 1024, 16, 8, 3072, True), "8b": (8, 4096, 32, 8, 12288, False)}
WIDTHS = {"0.6b": (1024, 16, 8, 128, 3072), "8b": (4096, 32, 8, 128, 12288)}
VOCAB = 32768            # of the designs beside Qwen3
PAGE = 16
CLUSTERS = 32            # kinds of tokens that the routers tell apart
PROMPT_ROWS = 16         # logits wanted at the end of each prompt


# ------------------------------------------------------------------------------------------------- configurations
def _qwen3(size):
    layers, hidden, heads, kv_heads, inter, tied = QWEN3_SIZES[size]
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_act="silu", num_hidden_layers=layers,
                hidden_size=hidden, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=128,
                intermediate_size=inter, vocab_size=151936, rope_theta=1000000.0, rms_norm_eps=1e-6,
                tie_word_embeddings=tied, max_position_embeddings=40960)


def _mekazen(size):
    hidden, heads, kv_heads, dim, inter = WIDTHS[size]
    mixer = {"dim": dim, "heads": heads, "kv_heads": kv_heads, "mask": {"size": 1024}, "scale": dim ** -0.5, "vdim": dim,
             "rot": {"base": 5.0e5, "dims": dim // 2,
                     "scaling": {"factor": 32.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    layer = {"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": inter}}
    return {"architecture": "Mekazen", "vocab": VOCAB, "width": hidden, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "layers": [layer] * 4}


def _zitezen(size):
    hidden, heads, kv_heads, dim, inter = WIDTHS[size]
    memory, latent, beside = {"0.6b": ((8, 64, 128), (16, 64, 32, 64, 256, 384), (4, 64, 128)),
                              "8b": ((8, 128, 512), (32, 128, 64, 128, 512, 1536), (8, 64, 256))}[size]
    recurrence = lambda m: {"heads": m[0], "dim": m[1], "vdim": m[2], "gate_cap": 10.0}
    through_latent = {"heads": latent[0], "dim": latent[1], "rot_dim": latent[2], "vdim": latent[3], "kv_rank": latent[4],
                      "q_rank": latent[5], "scale": (latent[1] + latent[2]) ** -0.5, "rot": {"base": 1.0e4, "dims": latent[2]}}
    grouped = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 30.0,
               "rot": {"base": 1.0e4, "dims": dim // 2}}
    mlp = {"kind": "dense", "ff": inter}
    return {"architecture": "Zitezen", "vocab": VOCAB, "width": hidden, "streams": 2, "norm": {"eps": 1e-6},
            "layers": [{"type": "mlstm", "mixer": recurrence(memory), "mlp": None},
                       {"type": "latent_attention", "mixer": through_latent, "mlp": mlp},
                       {"type": "parallel", "mixer": {"left": grouped, "right": recurrence(beside), "left_scale": 0.5,
                                                      "right_scale": 0.5}, "mlp": mlp},
                       {"type": "mlstm", "mixer": recurrence(memory), "mlp": None}]}


def _sadosun(size):
    hidden, heads, kv_heads, dim, _ = WIDTHS[size]
    inner, rank, ff, side = {"0.6b": (2048, 64, 1536, 64), "8b": (8192, 256, 6144, 256)}[size]
    mlp = {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": 12, "identity": 1, "top": 3}}
    attention = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                 "mask": {"size": 1024}, "rot": {"base": 1.0e4, "dims": dim}}
    state_space = {"inner": inner, "state": 16, "dt_rank": rank, "conv": 4}
    return {"architecture": "Sadosun", "vocab": VOCAB, "width": hidden, "norm": {"eps": 1e-6},
            "embedding": {"scale": hidden ** 0.5}, "canon": {"taps": 4}, "token_side": {"dim": side},
            "layers": [{"type": "mamba1", "mixer": state_space, "mlp": mlp},
                       {"type": "attention", "mixer": attention, "mlp": mlp}] * 2}


def _dimorax(size):
    hidden, heads, kv_heads, dim, inter = WIDTHS[size]
    dh, rank, (lh, lrank), ff = {"0.6b": (16, 64, (16, 256), 1024), "8b": (32, 256, (32, 512), 4096)}[size]
    experts = {"kind": "moe", "expert": {"ff": ff}, "shared": {"ff": ff},
               "router": {"experts": 12, "top": 2, "scale": 2.0, "groups": {"count": 4, "keep": 2}}}
    dense = {"kind": "dense", "ff": inter}
    delta = {"heads": dh, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4, "ranks": {"decay": rank, "gate": rank}}
    attention = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 30.0,
                 "rot": {"base": 1.0e6, "dims": dim // 2,
                         "scaling": {"factor": 16.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    through_latent = {"heads": lh, "dim": 64, "rot_dim": 64, "vdim": 128, "kv_rank": lrank, "scale": 128 ** -0.5,
                      "rot": {"base": 1.0e4, "dims": 64}}
    return {"architecture": "Dimorax", "vocab": VOCAB, "width": hidden, "norm": {"eps": 1e-6}, "residual_mult": 0.5,
            "layers": [{"type": "channel_delta", "mixer": delta, "mlp": experts},
                       {"type": "attention", "mixer": attention, "mlp": dense},
                       {"type": "channel_delta", "mixer": delta, "mlp": dense},
                       {"type": "latent_attention", "mixer": through_latent, "mlp": experts}]}


def _kokolorn(size):
    hidden, heads, kv_heads, dim, inter = WIDTHS[size]
    dh, sh, ff = {"0.6b": (16, 32, 1536), "8b": (32, 128, 6144)}[size]
    experts = {"kind": "moe", "expert": {"ff": ff}, "shared": {"ff": ff}, "router": {"experts": 12, "top": 2}}
    attention = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                 "q_temp": {"coef": 0.1, "every": 4096}}
    delta = {"heads": dh, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}
    pair = {"left": dict(attention, bias_max=1024, bias_rows=32),
            "right": {"heads": sh, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}}
    return {"architecture": "Kokolorn", "vocab": VOCAB, "width": hidden, "norm": {"eps": 1e-6},
            "embedding": {"scale": hidden ** 0.5}, "loop": {"start": 0, "stop": 2, "times": 2},
            "layers": [{"type": "attention", "mixer": attention, "mlp": {"kind": "dense", "ff": inter, "limit": 7.0}},
                       {"type": "delta", "mixer": delta, "mlp": experts},
                       {"type": "parallel", "mixer": pair, "mlp": experts}]}


def _mekuvik(size):
    hidden, heads, kv_heads, dim, inter = WIDTHS[size]
    lh, q_rank, rank, ff = {"0.6b": (16, 512, 256, 1536), "8b": (32, 1536, 512, 6144)}[size]
    experts = {"kind": "moe", "expert": {"ff": ff}, "shared": {"ff": ff}, "router": {"experts": 12, "top": 2}}
    lightning = {"heads": lh, "dim": 128, "vdim": 128, "decay": [1.0 - 0.5 ** (1.0 + 9.0 * i / (lh - 1)) for i in range(lh)]}
    latent = {"heads": lh, "dim": 96, "rot_dim": 32, "vdim": 128, "q_rank": q_rank, "kv_rank": rank, "scale": 128 ** -0.5,
              "rot": {"base": 1.0e5, "dims": 32, "scaling": {"factor": 16.0, "original": 2048, "fast": 24.0, "slow": 1.0}}}
    attention = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                 "rot": {"base": 1.0e6, "dims": dim // 2}, "mask": {"size": 1024, "keep_first": 16}}
    return {"architecture": "Mekuvik", "vocab": VOCAB, "width": hidden, "norm": {"eps": 1e-6}, "logit_scale": 0.5,
            "loop": {"start": 0, "stop": 2, "times": 2},
            "layers": [{"type": "lightning", "mixer": lightning, "mlp": experts},
                       {"type": "latent_attention", "mixer": latent, "mlp": {"kind": "dense", "ff": inter}},
                       {"type": "attention", "mixer": attention, "mlp": experts}]}


DESIGNS = {"qwen3": _qwen3, "mekazen": _mekazen, "zitezen": _zitezen, "sadosun": _sadosun, "dimorax": _dimorax,
           "kokolorn": _kokolorn, "mekuvik": _mekuvik}


# ---------------------------------------------------------------------------------------------------------- cases
def _case(name, design, size, dtype, kind, requests, context, steps=1, portion=0):
    """``context``: the longest request's positions; the others have between half of them and all of them.
    ``steps``: decoded tokens (or mixed steps) a pass; ``portion``: prompt tokens beside the decoded ones in a step."""
    case = {"design": design, "size": size, "dtype": dtype, "kind": kind, "requests": requests, "context": context,
            "steps": steps, "portion": portion}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user and a short chat: launches and latency
        _case("qwen3 one request", "qwen3", "0.6b", "bfloat16", "decode", 1, 333, 4),
        # a small server's usual step
        _case("qwen3 eight requests", "qwen3", "0.6b", "bfloat16", "decode", 8, 2048, 8),
        # a full batch at wide layers: weights and cached keys both count
        _case("qwen3 full batch", "qwen3", "8b", "bfloat16", "decode", 64, 3001, 4),
        # a long prompt alone: time to the first token
        _case("qwen3 prompt", "qwen3", "0.6b", "bfloat16", "prompt", 1, 2048),
        # continuous batching: a prompt arrives in portions beside requests that decode
        _case("qwen3 mixed", "qwen3", "8b", "bfloat16", "mixed", 31, 1500, 3, 701),
        # the 32-bit path, which checkpoints and kernels are checked with
        _case("qwen3 float32 prompt", "qwen3", "0.6b", "float32", "prompt", 2, 517),
        # the other designs, prompts and decoding in turn
        _case("mekazen eight requests", "mekazen", "8b", "bfloat16", "decode", 8, 1900, 4),
        _case("zitezen prompt", "zitezen", "8b", "bfloat16", "prompt", 1, 2048),
        _case("sadosun prompts", "sadosun", "0.6b", "bfloat16", "prompt", 3, 1201),
        _case("dimorax prompt", "dimorax", "8b", "bfloat16", "prompt", 1, 1777),
        _case("kokolorn sixteen requests", "kokolorn", "8b", "bfloat16", "decode", 16, 700, 4),
        _case("mekuvik prompts", "mekuvik", "8b", "bfloat16", "prompt", 4, 1024),
    ]


def draw(rng):
    most = max(_cost(c) for c in listed())
    spread = lambda low, high: int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    while True:
        design = rng.choice(["qwen3", "qwen3", "qwen3", "mekazen", "zitezen", "sadosun", "dimorax", "kokolorn", "mekuvik"])
        size = rng.choice(["0.6b", "0.6b", "8b"])
        kind = rng.choice(["prompt", "decode", "decode", "mixed"])
        dtype = "float32" if design == "qwen3" and size == "0.6b" and rng.random() < 0.2 else "bfloat16"
        if kind == "prompt":
            case = _case(None, design, size, dtype, kind, spread(1, 8), spread(24, 2048 if dtype == "bfloat16" else 600))
            if case["requests"] * case["context"] > (6000 if dtype == "bfloat16" else 1200):
                continue
        else:
            portion = spread(16, 1024) if kind == "mixed" else 0
            case = _case(None, design, size, dtype, kind, spread(1, 64 if dtype == "bfloat16" else 8),
                         spread(24, 3000 if dtype == "bfloat16" else 600), rng.choice([2, 3, 4]), portion)
            if case["requests"] * case["context"] > (60000 if design == "qwen3" else 16000) or (portion and dtype == "float32"):
                continue
        if _cost(case) <= most:
            return case


def _lengths(case):
    """The requests' lengths: the first has the longest, the others odd ones down to half of it."""
    rng, longest = random.Random(case["context"] * 100 + case["requests"]), case["context"]
    return [longest] + [rng.randint((longest + 1) // 2, longest) for _ in range(case["requests"] - 1)]


# -------------------------------------------------------------------------------------------------------- weights
def _experts_of(config, name):
    """The router's settings of the layer that the tensor ``name`` is a router of."""
    return config["layers"][int(name.split(".")[0][1:])]["mlp"]["router"]


def _router(rng, gen, settings, shape, prototypes):
    """Rows that tell the tokens' kinds apart as a trained router does: each kind has its own few experts, well ahead."""
    rows, width = shape
    top, groups = settings["top"], settings.get("groups")
    score = torch.rand((CLUSTERS, rows), generator=gen, device="cuda") * 0.5 - 2.0
    for kind in range(CLUSTERS):
        if groups:   # one expert in each of the groups that are kept
            each = rows // groups["count"]
            chosen = [g * each + rng.randrange(each) for g in rng.sample(range(groups["count"]), top)]
        else:
            chosen = rng.sample(range(rows), top)
        score[kind, chosen] += 4.0
    return (score.t() @ prototypes) / (0.7 * width)


def _tensors(case, seed):
    """Random weights by name: matrices that keep the size of what they multiply, norms about one, decays and step sizes
    from the ranges that state-space models start from, tokens in ``CLUSTERS`` kinds."""
    from metallix_b200.config import parse_config
    raw = DESIGNS[case["design"]](case["size"])
    config = parse_config(raw)
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    rng = random.Random(seed)
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    normal = lambda shape: torch.randn(tuple(shape), generator=gen, device="cuda", dtype=dtype)
    uniform = lambda shape, low, high: torch.rand(tuple(shape), generator=gen, device="cuda") * (high - low) + low
    shapes = config.tensor_shapes()
    width = raw.get("width") or raw["hidden_size"]
    basis = torch.linalg.qr(torch.randn((width, CLUSTERS), generator=gen, device="cuda"))[0].t()
    prototypes = basis * math.sqrt(width)
    tensors = {}
    for name, shape in shapes.items():
        last = name.split(".")[-1]
        if name in ("embed", "model.embed_tokens.weight"):
            value = normal(shape).mul_(0.7)
            value += (prototypes * 0.7).to(dtype)[torch.arange(shape[0], device="cuda") % CLUSTERS]
            value /= (raw.get("embedding") or {}).get("scale", 1.0)
        elif name == "side.embed":
            value = normal(shape)
        elif last == "A_log":
            value = torch.log(uniform(shape, 1.0, 16.0) if len(shape) == 1 else
                              torch.arange(1, shape[1] + 1, device="cuda").float().expand(shape))
        elif last == "dt_bias" or name.endswith("dt.b"):
            step = torch.exp(uniform(shape, math.log(1e-3), math.log(1e-1)))
            value = step + torch.log(-torch.expm1(-step))       # softplus gives ``step`` back
        elif name.endswith(".f.b"):
            value = uniform(shape, 3.0, 6.0)
        elif last == "sink" or last == "rel":
            value = uniform(shape, -1.0, 1.0)
        elif last == "router":
            value = _router(rng, gen, _experts_of(raw, name), shape, prototypes)
        elif last in ("correction",) or name.endswith("router.b"):
            value = uniform(shape, -0.01, 0.01)
        elif last in ("conv", "canon1", "canon2"):
            value = uniform(shape, -0.5, 0.5)
        elif config.norm_tensor(name) or len(shape) < 2:
            kind = config.norm_tensor(name)
            value = uniform(shape, -0.1, 0.1) + (1.0 if kind in (True, "one") else 0.0)
            if kind == "identity":
                value = value + torch.eye(shape[0], shape[1], device="cuda")
        else:
            # what goes back into the residual stream is smaller than the stream, as in a trained decoder
            out = last in ("o", "down", "proj") or "o_proj" in name or "down_proj" in name
            value = normal(shape).mul_((0.4 if out else 1.0) / math.sqrt(shape[1]))
        matrix = len(shape) == 2 and not config.norm_tensor(name)
        tensors[name] = value.to(dtype if matrix else torch.float32).contiguous()
    return raw, config, tensors


def _tokens(case, seed):
    """Per request its context or prompt and the tokens that follow; the prompt that arrives beside them."""
    rng = random.Random(seed + 1)
    vocab = DESIGNS[case["design"]](case["size"]).get("vocab_size", VOCAB)
    some = lambda count: [rng.randrange(vocab) for _ in range(count)]
    contexts = [some(n) for n in _lengths(case)]
    following = [some(case["steps"]) for _ in contexts] if case["kind"] != "prompt" else []
    return contexts, following, some(case["portion"] * case["steps"])


# ------------------------------------------------------------------------------------------------------- the work
def prepare(case, seed):
    from metallix_b200.engine import Engine, StepEntry
    raw, config, tensors = _tensors(case, seed)
    contexts, following, arriving = _tokens(case, seed)
    kind, requests = case["kind"], case["requests"]
    tokens = sum(-(-len(c) // PAGE) * PAGE for c in contexts) + len(arriving) + (2 * requests + 2) * PAGE
    engine = Engine(config, tensors, dtype=case["dtype"], page_tokens=PAGE, max_tokens=tokens,
                    max_requests=2 * requests + 2, consume_tensors=True)
    vocab = engine.spec.vocab_size
    state = {"engine": engine, "entry": StepEntry, "case": case, "contexts": contexts, "following": following,
             "arriving": arriving}
    if kind == "prompt":
        state["wants"] = [tuple(range(max(0, len(c) - PROMPT_ROWS), len(c))) for c in contexts]
        return state
    # the contexts that the requests have when they start to decode, brought in as a server does
    batch, held = [], 0
    for index, context in enumerate(contexts):
        batch.append(StepEntry(request=("held", index), tokens=context))
        held += len(context)
        if held >= 4096 or index == requests - 1:
            engine.step(batch)
            batch, held = [], 0
    state["out"] = torch.empty((case["steps"], requests + (kind == "mixed"), vocab), dtype=torch.float32, device="cuda")
    if kind == "decode":
        run(state)   # a server that has been decoding: its steps are captured
    return state


def run(state):
    engine, StepEntry, case = state["engine"], state["entry"], state["case"]
    if case["kind"] == "prompt":
        logits = engine.step([StepEntry(request=index, tokens=tokens, want=want)
                              for index, (tokens, want) in enumerate(zip(state["contexts"], state["wants"]))])
        engine.release_all()
        return logits
    rows, portion, out = range(case["requests"]), case["portion"], state["out"]
    for row in rows:
        engine.fork(("held", row), row)
    for step in range(case["steps"]):
        entries = [StepEntry(request=row, tokens=state["following"][row][step:step + 1], want=(0,)) for row in rows]
        if portion:
            entries.append(StepEntry(request="new", tokens=state["arriving"][step * portion:(step + 1) * portion],
                                     want=(portion - 1,)))
        out[step].copy_(engine.step(entries))
    for row in rows:
        engine.release(row)
    if portion:
        engine.release("new")
    return out


# ----------------------------------------------------------------------------------------- what it cannot do without
def _runs(raw):
    """[(layer index, pass or None, first of its pass)] in the order in which the layers run."""
    count, loop = len(raw["layers"]), raw.get("loop")
    if not loop:
        return [(i, None, False) for i in range(count)]
    runs = [(i, None, False) for i in range(loop["start"])]
    for turn in range(loop["times"]):
        runs += [(i, turn, i == loop["start"]) for i in range(loop["start"], loop["stop"])]
    return runs + [(i, None, False) for i in range(loop["stop"], count)]


def _mixers(raw):
    """[(type, sizes)] of every mixer that runs, in order."""
    if "layers" not in raw:
        one = {"heads": raw["num_attention_heads"], "kv_heads": raw["num_key_value_heads"], "dim": raw["head_dim"]}
        return [("attention", one)] * raw["num_hidden_layers"]
    found = []
    for index, _, _ in _runs(raw):
        kind, mixer = raw["layers"][index]["type"], raw["layers"][index]["mixer"]
        if kind == "parallel":
            found += [("attention", mixer["left"]), ("dual" if "state" in mixer["right"] else "mlstm", mixer["right"])]
        else:
            found.append((kind, mixer))
    return found


def _step_work(case, raw, shapes, spans, wanted):
    """Bytes and operations of one step: ``spans`` = [(first position, tokens)] of its requests."""
    item = 2 if case["dtype"] == "bfloat16" else 4
    tokens = sum(count for _, count in spans)
    size = lambda name: math.prod(shapes[name])
    runs = [(None, None, None)] if "layers" not in raw else _runs(raw)
    vocab = raw.get("vocab_size", VOCAB)
    width = raw.get("width") or raw["hidden_size"]
    values = products = 0.0
    for index, _, first in runs:
        prefix = "" if index is None else f"l{index}."
        router = None if index is None or not raw["layers"][index].get("mlp") else raw["layers"][index]["mlp"].get("router")
        if first and "loop.in" in shapes:
            values, products = values + size("loop.in"), products + size("loop.in") * tokens
        for name in shapes:
            if not name.startswith(prefix) or "embed" in name or name in ("head", "lm_head.weight") or \
                    (index is None and len(shapes[name]) < 2) or name.startswith("loop."):
                continue
            if router and ".mlp.e" in name:
                share = router["top"] / (router["experts"] + (router.get("identity") or 0))
                values += size(name) * (1.0 - (1.0 - share) ** tokens)      # of the experts those that some token takes
                products += size(name) * tokens * share
            else:
                values, products = values + size(name), products + size(name) * tokens
    moved = item * (values + width * vocab + tokens * width) + 4.0 * wanted * vocab
    flops = 2.0 * (products + width * vocab * wanted)
    for kind, mixer in _mixers(raw):
        mask = mixer.get("mask") or {}
        if kind in ("attention", "latent_attention"):
            heads, groups = mixer["heads"], mixer.get("kv_heads") or mixer["heads"]
            key = mixer["dim"] + mixer.get("rot_dim", 0)
            value = mixer.get("vdim") or mixer["dim"]
            row = (mixer["kv_rank"] + mixer["rot_dim"]) if "kv_rank" in mixer else groups * (key + value)
            for start, count in spans:
                reach = min(mask["size"], start + count) if mask else start + count
                seen = sum(min(mask["size"], p + 1) if mask else p + 1 for p in (start, start + count - 1)) / 2.0
                moved += item * row * (reach if start else count)
                flops += 2.0 * heads * (key + value) * seen * count
        elif kind == "mamba1":
            moved += 8.0 * len(spans) * mixer["inner"] * mixer["state"]
            flops += 6.0 * tokens * mixer["inner"] * mixer["state"]
        else:
            state = mixer["heads"] * (mixer.get("state") or mixer["dim"]) * (mixer.get("vdim") or mixer["dim"])
            moved += 8.0 * len(spans) * state
            flops += (8.0 if "delta" in kind else 5.0) * tokens * state
    return moved, flops


def work(case):
    from metallix_b200.config import parse_config
    raw = DESIGNS[case["design"]](case["size"])
    shapes = parse_config(raw).tensor_shapes()
    lengths, total = _lengths(case), [0.0, 0.0]
    steps = [([(0, n) for n in lengths], sum(min(PROMPT_ROWS, n) for n in lengths))]
    if case["kind"] != "prompt":
        arriving = lambda t: [(t * case["portion"], case["portion"])] if case["portion"] else []
        steps = [([(n + t, 1) for n in lengths] + arriving(t), len(lengths) + len(arriving(t))) for t in range(case["steps"])]
    for spans, wanted in steps:
        total = [a + b for a, b in zip(total, _step_work(case, raw, shapes, spans, wanted))]
    return {"bytes": total[0], "flops": total[1]}


def _cost(case):
    found = work(case)
    return max(found["bytes"], found["flops"] / 50)


def tolerance(case):
    """Four times what the engine is off from ``exact`` (measured: 1e-6 in float32; in bfloat16 about 3e-3, 6e-3 where
    the logits are capped or a layer's output is normed again, 4e-4 where the embedding dominates the logits)."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": {"mekazen": 0.025, "sadosun": 0.02, "mekuvik": 0.004}.get(case["design"], 0.015), "max": 0.3}


# ------------------------------------------------------------------------------------- the decoders in 64 bits
class _Weights:
    """Tensors by name in float64, each made when it is asked for."""

    def __init__(self, tensors):
        self.tensors = tensors

    def __getitem__(self, name):
        return self.tensors[name].double()

    def __contains__(self, name):
        return name in self.tensors


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, taps):
    """Causal convolution over time, per channel; the last tap meets the current token."""
    count = taps.shape[1]
    padded = torch.cat([x.new_zeros((count - 1, x.shape[1])), x])
    return sum(taps[:, j] * padded[j:j + x.shape[0]] for j in range(count))


def _frequencies(rot):
    dims, base, stretch = rot["dims"], rot["base"], rot.get("scaling")
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    f, magnitude = base ** (-2.0 * i / dims), 1.0
    if stretch and "low" in stretch:
        wave = 2.0 * math.pi / f
        smooth = (stretch["original"] / wave - stretch["low"]) / (stretch["high"] - stretch["low"])
        mixed = (1.0 - smooth) * f / stretch["factor"] + smooth * f
        f = torch.where(wave > stretch["original"] / stretch["low"], f / stretch["factor"],
                        torch.where(wave < stretch["original"] / stretch["high"], f, mixed))
    elif stretch:
        where = lambda turns: dims * math.log(stretch["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        low, high = max(math.floor(where(stretch["fast"])), 0), min(math.ceil(where(stretch["slow"])), dims - 1)
        ramp = ((i - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        f, magnitude = f / stretch["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(stretch["factor"]) + 1.0
    return f, magnitude


def _turn(x, rot, pairs, sign=1.0):
    """x ``[tokens, heads, D]``: pairs among the first ``dims`` values turn with the position, neighbours or halves."""
    if not rot:
        return x
    f, magnitude = _frequencies(rot)
    angle = sign * torch.arange(x.shape[0], dtype=torch.float64, device="cuda")[:, None, None] * f
    c, s, half, out = torch.cos(angle) * magnitude, torch.sin(angle) * magnitude, rot["dims"] // 2, x.clone()
    a, b = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if pairs else (slice(0, half), slice(half, 2 * half))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _attend(q, k, v, scale, mask=None, chunk=0, cap=0.0, sink=None, bias=None):
    """q ``[T, H, D]``, k and v ``[T, G, ..]``: causal softmax attention, one key/value head at a time. ``sink``: a score
    per head that joins the denominator; ``bias``: ``[T, H]`` by distance."""
    count, heads, groups = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(count, device="cuda")
    distance = i[:, None] - i[None, :]
    seen = distance >= 0
    if mask:
        seen &= (distance < mask["size"]) | (i[None, :] < mask.get("keep_first", 0))
    if chunk:
        seen &= (i[:, None] // chunk) == (i[None, :] // chunk)
    out = q.new_empty((count, heads, v.shape[2]))
    for head in range(heads):
        g = head // (heads // groups)
        scores = (q[:, head] @ k[:, g].t()) * scale
        if cap:
            scores = cap * torch.tanh(scores / cap)
        if bias is not None:
            scores = scores + bias[:, head][distance.clamp(min=0)]
        scores = scores.masked_fill(~seen, -math.inf)
        if sink is not None:
            scores = torch.cat([scores, sink[head].expand(count, 1)], dim=1)
        out[:, head] = torch.softmax(scores, dim=1)[:, :count] @ v[:, g]
    return out.reshape(count, -1)


def _delta(q, k, v, beta, decay, w, base, eps):
    """The gated delta rule of all heads: q, k ``[T, G, D]``, v ``[T, H, V]``, decay ``[T, H, D or 1]``; normed per head."""
    per = v.shape[1] // q.shape[1]
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q, k = (unit(q) * q.shape[2] ** -0.5).repeat_interleave(per, 1), unit(k).repeat_interleave(per, 1)
    state, out = v.new_zeros((v.shape[1], q.shape[2], v.shape[2])), torch.empty_like(v)
    for t in range(v.shape[0]):
        state = state * decay[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", state, k[t]))
        state = state + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", state, q[t])
    return _rms(out, eps) * w[base + ".norm"]


def _mlstm(h, w, base, m, eps):
    heads, dim, vdim, cap, count = m["heads"], m["dim"], m["vdim"], m["gate_cap"], h.shape[0]
    q = (h @ w[base + ".q"].t()).view(count, heads, dim) * dim ** -0.5
    k, v = (h @ w[base + ".k"].t()).view(count, heads, dim), (h @ w[base + ".v"].t()).view(count, heads, vdim)
    take = cap * torch.tanh((h @ w[base + ".i"].t() + w[base + ".i.b"]) / cap)
    keep = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w[base + ".f"].t() + w[base + ".f.b"]) / cap))
    C, n, peak = q.new_zeros((heads, dim, vdim)), q.new_zeros((heads, dim)), q.new_zeros(heads)
    out = torch.empty_like(v)
    for t in range(count):
        higher = torch.maximum(keep[t] + peak, take[t])
        old, new, peak = torch.exp(keep[t] + peak - higher), torch.exp(take[t] - higher), higher
        C = C * old[:, None, None] + new[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
        n = n * old[:, None] + new[:, None] * k[t]
        below = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-peak)) + 1e-6
        out[t] = torch.einsum("hdv,hd->hv", C, q[t]) / below[:, None]
    normed = _rms(out, eps).reshape(count, -1) * w[base + ".norm"]
    return (normed * torch.sigmoid(h @ w[base + ".g"].t())) @ w[base + ".o"].t()


def _mamba1(h, w, base, m):
    inner, states, rank = m["inner"], m["state"], m["dt_rank"]
    both = h @ w[base + ".in"].t()
    x = _silu(_conv(both[:, :inner], w[base + ".conv"]) + w[base + ".conv.b"])
    low, b, c = (x @ w[base + ".x"].t()).split([rank, states, states], dim=1)
    dt = torch.nn.functional.softplus(low @ w[base + ".dt"].t() + w[base + ".dt.b"])
    a, state, y = -torch.exp(w[base + ".A_log"]), x.new_zeros((inner, states)), torch.empty_like(x)
    for t in range(x.shape[0]):
        state = torch.exp(dt[t][:, None] * a) * state + (dt[t] * x[t])[:, None] * b[t]
        y[t] = state @ c[t]
    return ((y + w[base + ".D"] * x) * _silu(both[:, inner:])) @ w[base + ".o"].t()


def _dual(h, w, base, m, eps):
    heads, vdim, states, groups, count = m["heads"], m["vdim"], m["state"], m["groups"], h.shape[0]
    inner = heads * vdim
    wide = h @ w[base + ".in"].t()
    z, mid, dt = wide.split([inner, inner + 2 * groups * states, heads], dim=1)
    mid = _silu(_conv(mid, w[base + ".conv"]) + w[base + ".conv.b"])
    x = mid[:, :inner].reshape(count, heads, vdim)
    spread = lambda part: part.reshape(count, groups, states).repeat_interleave(heads // groups, 1)
    b, c = spread(mid[:, inner:inner + groups * states]), spread(mid[:, inner + groups * states:])
    dt = torch.nn.functional.softplus(dt + w[base + ".dt_bias"])
    decay, state, y = torch.exp(-torch.exp(w[base + ".A_log"]) * dt), x.new_zeros((heads, states, vdim)), torch.empty_like(x)
    for t in range(count):
        state = state * decay[t][:, None, None] + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
        y[t] = torch.einsum("hnv,hn->hv", state, c[t])
    y = ((y + w[base + ".D"][:, None] * x).reshape(count, inner) * _silu(z)).view(count, m["norm_groups"], -1)
    return (_rms(y, eps).reshape(count, inner) * w[base + ".norm"]) @ w[base + ".o"].t()


def _lightning(h, w, base, m, eps):
    heads, count = m["heads"], h.shape[0]
    q, k, v = (_silu(h @ w[f"{base}.{n}"].t()).view(count, heads, -1) for n in "qkv")
    decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[:, None, None]
    state, out = q.new_zeros((heads, q.shape[2], v.shape[2])), torch.empty_like(v)
    for t in range(count):
        state = decay * state + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", state, q[t])
    return (_rms(out.reshape(count, -1), eps) * w[base + ".norm"] * torch.sigmoid(h @ w[base + ".g"].t())) @ w[base + ".o"].t()


def _latent(h, w, base, m, eps, pairs, sink=None):
    """Keys and values from one normed latent, beside one rotated key part for all heads; the heads side by side."""
    heads, dim, turned, rank, count = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], h.shape[0]
    if base + ".dq" in w:
        q = (_rms(h @ w[base + ".dq"].t(), eps) * w[base + ".dq.norm"]) @ w[base + ".uq"].t()
    else:
        q = h @ w[base + ".q"].t()
    q, down = q.view(count, heads, dim + turned), h @ w[base + ".dkv"].t()
    c = _rms(down[:, :rank], eps) * w[base + ".dkv.norm"]
    shared = _turn(down[:, None, rank:], m["rot"], pairs).expand(count, heads, turned)
    k = torch.cat([(c @ w[base + ".uk"].t()).view(count, heads, dim), shared], dim=2)
    q = torch.cat([q[..., :dim], _turn(q[..., dim:], m["rot"], pairs)], dim=2)
    return _attend(q, k, (c @ w[base + ".uv"].t()).view(count, heads, -1), m["scale"], m.get("mask"), sink=sink)


def _route(h, w, base, mlp, choose, expert):
    """Sum over the chosen experts; ``choose(logits)`` gives (chosen, weights), ``expert(e, rows, weights)`` its output."""
    chosen, weights = choose(h @ w[base + ".router"].t())
    out = torch.zeros_like(h)
    for e in range(mlp["router"]["experts"] + (mlp["router"].get("identity") or 0)):
        rows, place = torch.nonzero(chosen == e, as_tuple=True)
        if rows.numel():
            out[rows] += expert(e, h[rows], weights[rows, place][:, None])
    return out


def _qwen3_layers(x, ids, raw, w):
    heads, groups, dim, eps, count = (raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"],
                                      raw["rms_norm_eps"], x.shape[0])
    rot = {"base": raw["rope_theta"], "dims": dim}
    for index in range(raw["num_hidden_layers"]):
        at = f"model.layers.{index}."
        part = lambda name: w[f"{at}{name}.weight"]
        h = _rms(x, eps) * part("input_layernorm")
        q = (h @ part("self_attn.q_proj").t()).view(count, heads, dim)
        k = (h @ part("self_attn.k_proj").t()).view(count, groups, dim)
        v = (h @ part("self_attn.v_proj").t()).view(count, groups, dim)
        q = _turn(_rms(q, eps) * part("self_attn.q_norm"), rot, False)
        k = _turn(_rms(k, eps) * part("self_attn.k_norm"), rot, False)
        x = x + _attend(q, k, v, dim ** -0.5) @ part("self_attn.o_proj").t()
        h = _rms(x, eps) * part("post_attention_layernorm")
        x = x + (_silu(h @ part("mlp.gate_proj").t()) * (h @ part("mlp.up_proj").t())) @ part("mlp.down_proj").t()
    return _rms(x, eps) * w["model.norm.weight"]


def _mekazen_layers(x, ids, raw, w):
    eps, count = raw["norm"]["eps"], x.shape[0]
    for index, layer in enumerate(raw["layers"]):
        at, m = f"l{index}.", layer["mixer"]
        h = _rms(x, eps) * (1.0 + w[at + "norm1"])
        q, k = h @ w[at + "mix.q"].t(), h @ w[at + "mix.k"].t()
        v = k.view(count, m["kv_heads"], -1)
        q = _turn((_rms(q, eps) * w[at + "mix.q.norm"]).view(count, m["heads"], -1), m["rot"], True)
        k = _turn((_rms(k, eps) * w[at + "mix.k.norm"]).view(count, m["kv_heads"], -1), m["rot"], True)
        y = _attend(q, k, v, m["scale"], chunk=m["mask"]["size"]) * torch.sigmoid(h @ w[at + "mix.g"].t())
        x = x + _rms(y @ w[at + "mix.o"].t(), eps) * (1.0 + w[at + "norm1b"])
        h = _rms(x, eps) * (1.0 + w[at + "norm2"])
        y = (_silu(h @ w[at + "mlp.gate"].t()) * (h @ w[at + "mlp.up"].t())) @ w[at + "mlp.down"].t()
        x = x + _rms(y, eps) * (1.0 + w[at + "norm2b"])
    return _rms(x, eps) * (1.0 + w["final.norm"])


def _zitezen_layers(x, ids, raw, w):
    eps, count = raw["norm"]["eps"], x.shape[0]
    norm = lambda name, x: torch.tanh(w[name + ".alpha"] * x) * w[name] + w[name + ".b"]
    streams = x[None].repeat(raw["streams"], 1, 1)
    for index, layer in enumerate(raw["layers"]):
        at, m = f"l{index}.", layer["mixer"]
        for sub in (1, 2) if layer["mlp"] else (1,):
            hc = f"{at}hc{sub}"
            h = norm(f"{at}norm{sub}", torch.einsum("s,stw->tw", w[hc + ".in"], streams))
            if sub == 2:
                y = torch.relu(h @ w[at + "mlp.up"].t()).square() @ w[at + "mlp.down"].t()
            elif layer["type"] == "mlstm":
                y = _mlstm(h, w, at + "mix", m, eps)
            elif layer["type"] == "latent_attention":
                y = _latent(h, w, at + "mix", m, eps, True) @ w[at + "mix.o"].t()
            else:
                left, base = m["left"], at + "mix.left"
                head = lambda n, number: (h @ w[f"{base}.{n}"].t()).view(count, number, -1)
                q = _turn(_rms(head("q", left["heads"]), eps) * w[base + ".q.norm"], left["rot"], False)
                k = _turn(_rms(head("k", left["kv_heads"]), eps) * w[base + ".k.norm"], left["rot"], False)
                o = _attend(q, k, head("v", left["kv_heads"]), left["scale"], cap=left["softcap"]).view(count, left["heads"], -1)
                y = (o * torch.sigmoid(h @ w[base + ".g"].t())[:, :, None]).reshape(count, -1) @ w[base + ".o"].t()
                y = m["left_scale"] * y + m["right_scale"] * _mlstm(h, w, at + "mix.right", m["right"], eps)
            y = y * w[f"{at}ls{sub}"]
            streams = torch.einsum("st,sxw->txw", w[hc + ".mix"], streams) + w[hc + ".out"][:, None, None] * y
    return norm("final.norm", streams.sum(0))


def _sadosun_layers(x, ids, raw, w):
    eps, count, side = raw["norm"]["eps"], x.shape[0], raw["token_side"]["dim"]
    for index, layer in enumerate(raw["layers"]):
        at, m = f"l{index}.", layer["mixer"]
        h = _rms(x, eps) * w[at + "norm1"]
        h = h + _conv(h, w[at + "canon1"])
        if layer["type"] == "mamba1":
            x = x + _mamba1(h, w, at + "mix", m)
        else:
            head = lambda n, number: (h @ w[f"{at}mix.{n}"].t()).view(count, number, -1)
            q, k, v = (_turn(head(n, number), m["rot"], True)
                       for n, number in (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"])))
            o = _attend(_rms(q, eps), _rms(k, eps), v, m["scale"], m["mask"], sink=x.new_zeros(m["heads"]))
            o = _turn(o.view(count, m["heads"], -1), m["rot"], True, sign=-1.0)
            x = x + o.reshape(count, -1) @ w[at + "mix.o"].t()
        h = _rms(x, eps) * w[at + "norm2"]
        h = h + _conv(h, w[at + "canon2"])

        def choose(logits):
            scores = torch.softmax(logits, dim=-1)
            chosen = (scores + w[at + "mlp.correction"]).topk(layer["mlp"]["router"]["top"], dim=-1).indices
            picked = scores.gather(1, chosen)
            return chosen, picked / (picked.sum(-1, keepdim=True) + 1e-20)

        def expert(e, rows, weight):
            if e >= layer["mlp"]["router"]["experts"]:
                return weight * rows
            return weight * (torch.relu(rows @ w[f"{at}mlp.e{e}.up"].t()).square() @ w[f"{at}mlp.e{e}.down"].t())

        x = x + _route(h, w, at + "mlp", layer["mlp"], choose, expert)
        gate = torch.nn.functional.gelu(x @ w[at + "side.gate"].t(), approximate="tanh")
        own = w.tensors["side.embed"][ids][:, index * side:(index + 1) * side].double()
        x = x + _rms((gate * own) @ w[at + "side.proj"].t(), eps) * w[at + "side.norm"]
    return _rms(x, eps) * w["final.norm"]


def _dimorax_layers(x, ids, raw, w):
    eps, count = raw["norm"]["eps"], x.shape[0]
    for index, layer in enumerate(raw["layers"]):
        at, base, m = f"l{index}.", f"l{index}.mix", layer["mixer"]
        h = _rms(x, eps) * (1.0 + w[at + "norm1"])
        if layer["type"] == "channel_delta":
            q, k, v = (_silu(_conv(h @ w[f"{base}.{n}"].t(), w[f"{base}.{n}.conv"])).view(count, number, -1)
                       for n, number in (("q", m["kv_heads"]), ("k", m["kv_heads"]), ("v", m["heads"])))
            beta = torch.sigmoid(h @ w[base + ".b"].t())
            step = torch.nn.functional.softplus((h @ w[base + ".a1"].t()) @ w[base + ".a2"].t() + w[base + ".dt_bias"])
            decay = torch.exp(-torch.exp(w[base + ".A_log"])[:, None] * step.view(count, m["heads"], -1))
            gate = torch.sigmoid((h @ w[base + ".g1"].t()) @ w[base + ".g2"].t()).view(count, m["heads"], -1)
            y = (_delta(q, k, v, beta, decay, w, base, eps) * gate).reshape(count, -1)
        elif layer["type"] == "attention":
            head = lambda n, number: (h @ w[f"{base}.{n}"].t() + w[f"{base}.{n}.b"]).view(count, number, -1)
            q, k = _turn(head("q", m["heads"]), m["rot"], False), _turn(head("k", m["kv_heads"]), m["rot"], False)
            y = _attend(q, k, head("v", m["kv_heads"]), m["scale"], cap=m["softcap"], sink=w[base + ".sink"])
        else:
            y = _latent(h, w, base, m, eps, False, sink=w[base + ".sink"])
        y = y @ w[base + ".o"].t()
        h, ff, mlp = _rms(x, eps) * (1.0 + w[at + "norm2"]), at + "mlp", layer["mlp"]
        gated = lambda rows, name, act: (act(rows @ w[name + ".gate"].t()) * (rows @ w[name + ".up"].t())) @ w[name + ".down"].t()
        if mlp["kind"] == "dense":
            y = y + gated(h, ff, lambda z: torch.nn.functional.gelu(z, approximate="tanh"))
        else:
            router = mlp["router"]

            def choose(logits):
                scores = torch.sigmoid(logits)
                choice = scores + w[ff + ".correction"]
                parts = choice.view(count, router["groups"]["count"], -1)
                kept = parts.topk(2, dim=-1).values.sum(-1).topk(router["groups"]["keep"], dim=-1).indices
                allowed = torch.zeros(parts.shape[:2], dtype=torch.bool, device="cuda").scatter_(1, kept, True)
                choice = parts.masked_fill(~allowed[:, :, None], -math.inf).reshape(count, -1)
                chosen = choice.topk(router["top"], dim=-1).indices
                picked = scores.gather(1, chosen)
                return chosen, picked / (picked.sum(-1, keepdim=True) + 1e-20) * router["scale"]

            y = y + _route(h, w, ff, mlp, choose, lambda e, rows, weight: weight * gated(rows, f"{ff}.e{e}", _silu))
            y = y + torch.sigmoid(h @ w[ff + ".shared.sg"].t()) * gated(h, ff + ".shared", _silu)
        x = x + raw["residual_mult"] * y
    return _rms(x, eps) * (1.0 + w["final.norm"])


def _kokolorn_layers(x, ids, raw, w):
    eps, count, first = raw["norm"]["eps"], x.shape[0], x

    def attention(h, base, m, norms):
        q = (h @ w[base + ".q"].t() + w[base + ".q.b"]).view(count, m["heads"], -1)
        v = k = (h @ w[base + ".k"].t() + w[base + ".k.b"]).view(count, m["kv_heads"], -1)
        if norms:
            q, k = _rms(q, eps) * w[base + ".q.norm"], _rms(k, eps) * w[base + ".k.norm"]
        p = torch.arange(count, dtype=torch.float64, device="cuda")
        q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((p + 1) / m["q_temp"]["every"]) + 1.0))[:, None, None]
        bias = None
        if base + ".rel" in w:
            rows, far = m["bias_rows"], m["bias_max"]
            half = rows // 2
            step = lambda n: n if n < half else min(rows - 1, half + math.floor(
                math.log(n / half) / math.log(far / half) * (rows - half) + 1e-9))
            bias = w[base + ".rel"][torch.tensor([step(n) for n in range(count)], device="cuda")]
        return _attend(q, k, v, m["scale"], bias=bias) @ w[base + ".o"].t()

    for index, turn, opens in _runs(raw):
        if opens:
            x = torch.cat([x, first], dim=1) @ w["loop.in"].t() + w["loop.step"][turn]
        layer, at, base = raw["layers"][index], f"l{index}.", f"l{index}.mix"
        m, h = layer["mixer"], _rms(x, eps) * (1.0 + w[at + "norm1"])
        if layer["type"] == "attention":
            x = x + attention(h, base, m, True)
        elif layer["type"] == "delta":
            q, k, v = (_silu(_conv(h @ w[f"{base}.{n}"].t(), w[f"{base}.{n}.conv"])).view(count, number, -1)
                       for n, number in (("q", m["kv_heads"]), ("k", m["kv_heads"]), ("v", m["heads"])))
            step = torch.nn.functional.softplus(h @ w[base + ".a"].t() + w[base + ".dt_bias"])
            decay = torch.exp(-torch.exp(w[base + ".A_log"]) * step)[:, :, None]
            o = _delta(q, k, v, torch.sigmoid(h @ w[base + ".b"].t()), decay, w, base, eps).reshape(count, -1)
            x = x + (o * _silu(h @ w[base + ".g"].t())) @ w[base + ".o"].t()
        else:
            left = attention(h, base + ".left", m["left"], False) + w[base + ".left.o.b"]
            right = _dual(h, w, base + ".right", m["right"], eps)
            x = x + 0.5 * (_rms(left, eps) * w[base + ".left.out"] + _rms(right, eps) * w[base + ".right.out"])
        h, ff, mlp = _rms(x, eps) * (1.0 + w[at + "norm2"]), at + "mlp", layer["mlp"]
        if mlp["kind"] == "dense":
            g = (h @ w[ff + ".gate"].t()).clamp(max=mlp["limit"])
            u = (h @ w[ff + ".up"].t()).clamp(-mlp["limit"], mlp["limit"])
            x = x + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[ff + ".down"].t()
        else:
            squared = lambda rows, name: torch.relu(rows @ w[name + ".up"].t()).square() @ w[name + ".down"].t()

            def choose(logits):
                best = (logits + w[ff + ".router.b"]).topk(mlp["router"]["top"], dim=-1)
                return best.indices, torch.softmax(best.values, dim=-1)

            x = x + _route(h, w, ff, mlp, choose, lambda e, rows, weight: weight * squared(rows, f"{ff}.e{e}"))
            x = x + squared(h, ff + ".shared")
    return _rms(x, eps) * (1.0 + w["final.norm"])


def _mekuvik_layers(x, ids, raw, w):
    eps, count, first = raw["norm"]["eps"], x.shape[0], x
    for index, turn, opens in _runs(raw):
        if opens and turn:
            x = x + first
        layer, at, base = raw["layers"][index], f"l{index}.", f"l{index}.mix"
        m, h = layer["mixer"], _rms(x, eps) * w[at + "norm1"]
        if layer["type"] == "lightning":
            y = _lightning(h, w, base, m, eps)
        elif layer["type"] == "attention":
            q = (_rms(h @ w[base + ".q"].t(), eps) * w[base + ".q.norm"]).view(count, m["heads"], -1)
            k = (_rms(h @ w[base + ".k"].t(), eps) * w[base + ".k.norm"]).view(count, m["kv_heads"], -1)
            v = (h @ w[base + ".v"].t()).view(count, m["kv_heads"], -1)
            y = _attend(_turn(q, m["rot"], True), _turn(k, m["rot"], True), v, m["scale"], m["mask"]) @ w[base + ".o"].t()
        else:
            y = (_latent(h, w, base, m, eps, True) * torch.sigmoid(h @ w[base + ".g"].t())) @ w[base + ".o"].t()
        ff, mlp = at + "mlp", layer["mlp"]
        if mlp["kind"] == "dense":
            y = y + (_silu(h @ w[ff + ".gate"].t()) * (h @ w[ff + ".up"].t())) @ w[ff + ".down"].t()
        else:
            wide = lambda rows, name: torch.nn.functional.gelu(rows @ w[name + ".up"].t()) @ w[name + ".down"].t()

            def choose(logits):
                best = logits.topk(mlp["router"]["top"], dim=-1)
                return best.indices, torch.sigmoid(best.values)

            y = y + _route(h, w, ff, mlp, choose, lambda e, rows, weight: wide(weight * rows, f"{ff}.e{e}"))
            y = y + wide(h, ff + ".shared")
        x = x + y
    return _rms(x, eps) * w["final.norm"]


_LAYERS = {"qwen3": _qwen3_layers, "mekazen": _mekazen_layers, "zitezen": _zitezen_layers, "sadosun": _sadosun_layers,
           "dimorax": _dimorax_layers, "kokolorn": _kokolorn_layers, "mekuvik": _mekuvik_layers}


def _exact_logits(design, raw, w, ids, wanted):
    """Float64 logits ``[wanted, vocab]`` of one whole sequence."""
    table = "embed" if "embed" in w else "model.embed_tokens.weight"
    at = torch.tensor(ids, device="cuda")
    x = w.tensors[table][at].double() * (raw.get("embedding") or {}).get("scale", 1.0)
    x = _LAYERS[design](x, at, raw, w)[torch.tensor(wanted, device="cuda")]
    head = next((name for name in ("head", "lm_head.weight") if name in w), table)
    logits = torch.cat([x @ part.double().t() for part in w.tensors[head].split(16384)], dim=1) * raw.get("logit_scale", 1.0)
    cap = raw.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits


def exact(case, seed):
    lengths, kind = _lengths(case), case["kind"]
    tokens = sum(lengths) + case["portion"] * case["steps"]
    if tokens > (20000 if case["design"] in ("qwen3", "mekazen") else 9000):
        return None      # minutes of it
    raw, _, tensors = _tensors(case, seed)
    w = _Weights(tensors)
    contexts, following, arriving = _tokens(case, seed)
    with torch.no_grad():
        if kind == "prompt":
            return torch.cat([_exact_logits(case["design"], raw, w, c, range(max(0, len(c) - PROMPT_ROWS), len(c)))
                              for c in contexts])
        rows = [_exact_logits(case["design"], raw, w, c + f, range(len(c), len(c) + len(f)))
                for c, f in zip(contexts, following)]
        if arriving:
            portion = case["portion"]
            rows.append(_exact_logits(case["design"], raw, w, arriving, range(portion - 1, len(arriving), portion)))
        return torch.stack(rows, dim=1)
