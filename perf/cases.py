"""What this engine is used for, as measurable cases: prompts read and tokens decoded through ``Engine.step``.

A case is a model shape, a dtype and a load (how many requests, their prompt lengths, how many tokens each is then
given, how a prompt may be cut). ``plan`` turns the load into the steps a first-come-first-served scheduler makes of it:
each step carries one token of every request that is past its prompt beside prompt portions of the others, up to a
token budget. One pass runs all steps of the plan on the engine and ends its requests with the last of them, so it can
run again. The tokens after the prompt are given, as in a trace replay, so that every pass does the same work and all
logits can be compared; the logits of every wanted row (a prompt's last token, every token after it) are kept.

GPT-2 is the architecture the engine was made for: the XL, large and medium shapes with the loads of the benchmark, and
the two tiny shapes of the tests. Bonatar stands for the other architectures (separate projections, rotary positions,
grouped keys, gated heads, experts chosen by a table), at the sizes of the benchmark's design comparison.
"""
import math
import random

import torch

from damendaemon_b200.engine import Engine, StepEntry

PAGE = 16
SHAPES = {"tiny_a": (2, 64, 4, 256, 512, 128), "tiny_b": (3, 96, 2, 320, 1000, 256),
          "medium": (24, 1024, 16, 4096, 50257, 1024), "large": (36, 1280, 20, 5120, 50257, 1024),
          "xl": (48, 1600, 25, 6400, 50257, 1024)}


def gpt2(shape, dtype, **load):
    layers, width, heads, inner, vocab, positions = SHAPES[shape] if isinstance(shape, str) else shape
    case = {"model": "gpt2", "dtype": dtype, "layers": layers, "width": width, "heads": heads, "kv_heads": heads, "inner": inner,
            "vocab": vocab, "positions": positions, "activation": "gelu_new", "epsilon": 1e-5, "scale_by_layer": False}
    return {**case, **load_of(**load)}


def bonatar(layers, width, heads, kv_heads, experts, top, inner, vocab, dtype, **load):
    """experts = 0: dense feed-forwards of ``inner``; else ``inner`` is one expert's (and the shared expert's) size."""
    case = {"model": "bonatar", "dtype": dtype, "layers": layers, "width": width, "heads": heads, "kv_heads": kv_heads, "experts": experts,
            "top": top, "inner": inner, "vocab": vocab, "positions": 1024, "epsilon": 1e-6}
    return {**case, **load_of(**load)}


def load_of(requests, prompt, new=0, prompt_most=None, portion=0, budget=4096, lengths_seed=0):
    """Prompts of ``prompt`` tokens, or of a uniform length between ``prompt`` and ``prompt_most``; ``new`` tokens after
    each; portions of at most ``portion`` prompt tokens a step (0: no limit but the budget)."""
    return {"requests": requests, "prompt": prompt, "prompt_most": prompt_most or prompt, "new": new, "portion": portion, "budget": budget,
            "lengths_seed": lengths_seed}


def listed():
    return [
        # the smallest calls: a model and a load of the tests, where launches and host time are all there is
        dict(gpt2("tiny_a", "float32", requests=3, prompt=5, prompt_most=33, new=16), name="tiny_f32"),
        # erf gelu, heads of 48, scores scaled by layer, prompts cut into portions of 32 beside decoding requests
        dict(gpt2("tiny_b", "float32", requests=4, prompt=1, prompt_most=200, new=40, portion=32), name="tiny_cut_f32")
        | {"activation": "gelu", "epsilon": 1e-6, "scale_by_layer": True},
        # one user's answer: the latency of a token
        dict(gpt2("xl", "bfloat16", requests=1, prompt=512, new=64), name="xl_decode_1"),
        # the headline load: eight users
        dict(gpt2("xl", "bfloat16", requests=8, prompt=512, new=64), name="xl_decode_8"),
        # a full batch
        dict(gpt2("xl", "bfloat16", requests=64, prompt=256, new=48), name="xl_decode_64"),
        # prompts alone, their last logits wanted
        dict(gpt2("xl", "bfloat16", requests=2, prompt=1024), name="xl_prefill_2x1024"),
        # long prompts in a model with more positions
        dict(gpt2((48, 1600, 25, 6400, 50257, 4096), "bfloat16", requests=2, prompt=4096, budget=8192), name="xl_prefill_2x4096"),
        # requests of any length admitted together, then decoded as they come
        dict(gpt2("medium", "bfloat16", requests=32, prompt=16, prompt_most=768, new=32), name="medium_serve_32"),
        # prompts in portions of 256 beside requests that already decode
        dict(gpt2("large", "bfloat16", requests=64, prompt=1, prompt_most=1000, new=24, portion=256, budget=2048), name="large_mixed_64"),
        # true 32-bit: the parity path, and the reference's only GPT-2 mode
        dict(gpt2("xl", "float32", requests=8, prompt=64, new=16), name="xl_decode_8_f32"),
        dict(gpt2("large", "float32", requests=1, prompt=1000), name="large_prefill_f32"),
        # another architecture, prompts and decoding
        dict(bonatar(6, 1600, 25, 25, 16, 2, 1600, 50257, "bfloat16", requests=8, prompt=256, prompt_most=512, new=32), name="bonatar_serve_8"),
    ]


# seconds that a drawn pass may take by the estimate of `seconds`: below what the largest listed cases take
DRAW_SECONDS = 0.08


def draw(rng):
    def log_int(low, high):
        return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))

    kind = rng.choice(["tiny", "decode", "decode", "prefill", "prefill", "mixed", "decode_f32", "prefill_f32", "bonatar"])
    seed = rng.randrange(1 << 16)
    shape = rng.choice(["medium", "large", "xl"])
    if kind == "tiny":
        heads, size = rng.randint(1, 6), rng.choice([16, 32, 48, 64])
        sizes = (rng.randint(1, 4), heads * size, heads, 8 * rng.randint(8, 60), rng.randint(300, 2000), 256)
        low = rng.randint(1, 40)
        case = gpt2(sizes, rng.choice(["float32", "bfloat16"]), requests=rng.randint(1, 6), prompt=low, prompt_most=rng.randint(low, 200),
                    new=rng.randint(8, 40), portion=rng.choice([0, 32]), lengths_seed=seed)
        case.update(activation=rng.choice(["gelu_new", "gelu"]), scale_by_layer=rng.random() < 0.5)
    elif kind == "decode":
        low = log_int(16, 700)
        case = gpt2(shape, "bfloat16", requests=log_int(1, 64), prompt=low, prompt_most=rng.randint(low, 900), new=rng.randint(24, 64), lengths_seed=seed)
    elif kind == "prefill":
        low = log_int(17, 1024)
        case = gpt2(shape, "bfloat16", requests=log_int(1, 8), prompt=low, prompt_most=rng.randint(low, 1024), lengths_seed=seed)
    elif kind == "mixed":
        case = gpt2(shape, "bfloat16", requests=log_int(4, 64), prompt=1, prompt_most=log_int(100, 980), new=rng.randint(8, 32),
                    portion=rng.choice([128, 256, 300]), budget=rng.choice([1024, 2048]), lengths_seed=seed)
    elif kind == "decode_f32":
        low = log_int(4, 128)
        case = gpt2(shape, "float32", requests=log_int(1, 32), prompt=low, prompt_most=rng.randint(low, 160), new=rng.randint(8, 20), lengths_seed=seed)
    elif kind == "prefill_f32":
        low = log_int(17, 1000)
        case = gpt2(shape, "float32", requests=rng.randint(1, 2), prompt=low, prompt_most=rng.randint(low, 1000), lengths_seed=seed)
    else:
        experts = rng.choice([0, 16])
        heads = rng.choice([16, 25])
        low = log_int(16, 512)
        case = bonatar(rng.randint(4, 8), heads * 64, heads, heads if rng.random() < 0.5 else heads // (5 if heads == 25 else 4), experts, 2 if experts else 0,
                       heads * 64 if experts else heads * 256, 50257, "bfloat16", requests=log_int(1, 32), prompt=low,
                       prompt_most=rng.randint(low, 900), new=rng.randint(8, 32), lengths_seed=seed)
    while seconds(case) > DRAW_SECONDS:
        if case["requests"] > 1:
            case["requests"] = case["requests"] * 2 // 3
        else:
            case["prompt_most"] = max(1, case["prompt_most"] * 2 // 3)
            case["prompt"] = min(case["prompt"], case["prompt_most"])
    return case


# ------------------------------------------------------------------ the steps of a case
def prompt_lengths(case):
    rng = random.Random(case["lengths_seed"])
    return [rng.randint(case["prompt"], case["prompt_most"]) for _ in range(case["requests"])]


def plan(case):
    """A list of steps, each a list of (request, first position, tokens, whether the last one's logits are wanted)."""
    lengths, new = prompt_lengths(case), case["new"]
    done, steps = [0] * len(lengths), []
    while any(d < n + new for d, n in zip(done, lengths)):
        step = [(r, d, 1, True) for r, (d, n) in enumerate(zip(done, lengths)) if n <= d < n + new]
        left = case["budget"] - len(step)
        for r, n in enumerate(lengths):
            if done[r] < n and left > 0:
                count = min(n - done[r], left, case["portion"] or n)
                step.append((r, done[r], count, done[r] + count == n))
                left -= count
        for r, _, count, _ in step:
            done[r] += count
        steps.append(step)
    return steps


def work(case):
    element = 4 if case["dtype"] == "float32" else 2
    w, inner, layers, v = case["width"], case["inner"], case["layers"], case["vocab"]
    kv = case["kv_heads"] * (w // case["heads"])
    total_bytes = total_flops = 0
    for step in plan(case):
        tokens, rows = sum(n for _, _, n, _ in step), sum(wanted for *_, wanted in step)
        if case["model"] == "gpt2":
            matrix = held = 4 * w * w + 2 * w * inner
        else:
            mixer = 2 * w * w + 2 * w * kv + w * case["heads"]
            if case["experts"]:
                unit = 3 * w * inner
                reached = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** tokens)        # experts that some token of the step uses
                matrix, held = mixer + (case["top"] + 1) * unit, mixer + (reached + 1) * unit
            else:
                matrix = held = mixer + 2 * w * inner
        total_flops += 2 * layers * matrix * tokens + 2 * v * w * rows
        total_bytes += element * (layers * held + (v * w if rows else 0))
        for _, first, n, _ in step:
            pairs = n * first + n * (n + 1) // 2
            total_flops += 4 * layers * w * pairs
            total_bytes += 2 * element * layers * kv * (first + n)                # keys and values: earlier ones read, new ones written
        total_bytes += tokens * w * element + rows * v * 4
    return {"bytes": total_bytes, "flops": total_flops}


def seconds(case):
    w = work(case)
    return len(plan(case)) * 1e-4 + max(w["bytes"] / 4e12, w["flops"] / (3e13 if case["dtype"] == "float32" else 7e14))


# ------------------------------------------------------------------ weights
def gpt2_weights(case, seed, dtype):
    """Tables and matrices ~N(0, 0.02) as GPT-2 is initialised, both c_proj scaled down with the depth."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w, inner, out = case["width"], case["inner"], {}
    last = 0.02 / math.sqrt(2 * case["layers"])

    def matrix(name, rows, cols, std=0.02):
        out[name] = (torch.randn((rows, cols), generator=g, device="cuda") * std).to(dtype)

    def vector(name, n, mean=0.0):
        out[name] = torch.randn((n,), generator=g, device="cuda") * 0.02 + mean

    matrix("wte.weight", case["vocab"], w)
    matrix("wpe.weight", case["positions"], w)
    for i in range(case["layers"]):
        p = f"h.{i}."
        for norm in ("ln_1", "ln_2"):
            vector(p + norm + ".weight", w, 1.0)
            vector(p + norm + ".bias", w)
        for name, rows, cols, std in (("attn.c_attn", w, 3 * w, 0.02), ("attn.c_proj", w, w, last), ("mlp.c_fc", w, inner, 0.02),
                                      ("mlp.c_proj", inner, w, last)):
            matrix(p + name + ".weight", rows, cols, std)
            vector(p + name + ".bias", cols)
    vector("ln_f.weight", w, 1.0)
    vector("ln_f.bias", w)
    return out


def bonatar_weights(case, seed, dtype):
    """Matrices ~N(0, 1 / inputs), norm weights around zero, a table of distinct experts for every token id."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w, out = case["width"], {}
    size = w // case["heads"]

    def matrix(name, rows, cols):
        out[name] = (torch.randn((rows, cols), generator=g, device="cuda") / math.sqrt(cols)).to(dtype)

    def vector(name):
        out[name] = torch.randn((w,), generator=g, device="cuda") * 0.1

    matrix("embed", case["vocab"], w)
    for i in range(case["layers"]):
        p = f"l{i}."
        vector(p + "norm1")
        vector(p + "norm2")
        for name, rows in (("q", w), ("k", case["kv_heads"] * size), ("v", case["kv_heads"] * size), ("g", case["heads"]), ("o", w)):
            matrix(p + "mix." + name, rows, w)
        if not case["experts"]:
            matrix(p + "mlp.up", case["inner"], w)
            matrix(p + "mlp.down", w, case["inner"])
            continue
        for unit in [f"e{e}." for e in range(case["experts"])] + ["shared."]:
            matrix(p + "mlp." + unit + "gate", case["inner"], w)
            matrix(p + "mlp." + unit + "up", case["inner"], w)
            matrix(p + "mlp." + unit + "down", w, case["inner"])
        order = torch.rand((case["vocab"], case["experts"]), generator=g, device="cuda").argsort(dim=1)
        out[p + "mlp.table"] = order[:, :case["top"]].to(torch.int32).contiguous()
    vector("final.norm")
    matrix("head", case["vocab"], w)
    return out


def weights_of(case, seed):
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    return (gpt2_weights if case["model"] == "gpt2" else bonatar_weights)(case, seed, dtype)


def config_of(case):
    if case["model"] == "gpt2":
        return {"architectures": ["GPT2LMHeadModel"], "model_type": "gpt2", "n_layer": case["layers"], "n_embd": case["width"],
                "n_head": case["heads"], "n_inner": case["inner"], "vocab_size": case["vocab"], "n_positions": case["positions"],
                "layer_norm_epsilon": case["epsilon"], "activation_function": case["activation"],
                "scale_attn_by_inverse_layer_idx": case["scale_by_layer"]}
    size = case["width"] // case["heads"]
    mixer = {"heads": case["heads"], "kv_heads": case["kv_heads"], "dim": size, "vdim": size, "scale": size ** -0.5, "mask": {"size": 1024},
             "rot": {"dims": size, "base": 10000.0}}
    mlp = {"kind": "dense", "ff": case["inner"]}
    if case["experts"]:
        unit = {"ff": case["inner"], "limit": 7.0}
        mlp = {"kind": "moe", "router": {"experts": case["experts"], "top": case["top"]}, "expert": unit, "shared": unit}
    return {"architecture": "Bonatar", "vocab": case["vocab"], "width": case["width"], "embedding": {"scale": case["width"] ** 0.5},
            "norm": {"eps": case["epsilon"]}, "layers": [{"type": "attention", "mixer": mixer, "mlp": mlp} for _ in range(case["layers"])]}


def token_ids(case, seed):
    """Every request's tokens, uniform over the vocabulary: the prompt and what follows it."""
    rng = random.Random(seed)
    return [[rng.randrange(case["vocab"]) for _ in range(n + case["new"])] for n in prompt_lengths(case)]


# ------------------------------------------------------------------ a pass
def prepare(case, seed):
    """The engine with its weights and a cache for the load, and the steps' entries."""
    ids = token_ids(case, seed)
    held = sum(-(-len(t) // PAGE) * PAGE for t in ids)
    engine = Engine(None, config=config_of(case), tensors=weights_of(case, seed), dtype=case["dtype"], kv_tokens=held, page_size=PAGE,
                    max_requests=max(2, case["requests"]), max_context=case["positions"], use_graph=True, check_device_errors=False)
    steps, rows = [], 0
    for step in plan(case):
        entries = [StepEntry(r, ids[r][first:first + n], [n - 1] if wanted else []) for r, first, n, wanted in step]
        end = [r for r, first, n, _ in step if first + n == len(ids[r])]
        here = sum(wanted for *_, wanted in step)
        steps.append((entries, end, rows, here))
        rows += here
    return {"engine": engine, "steps": steps, "logits": torch.empty((rows, case["vocab"]), dtype=torch.float32, device="cuda")}


def run(state):
    """All steps of the load; the logits of the wanted rows, in the order in which they came."""
    engine, kept = state["engine"], state["logits"]
    for entries, end, row, n in state["steps"]:
        logits = engine.step(entries, end=end)
        if n:
            kept[row:row + n].copy_(logits)        # a replayed step's logits are overwritten by the next step of its shape
    return kept


def tolerance(case):
    """About four times what the logits were measured to be off the 64-bit ones: 0.0036 to 0.0054 with bfloat16 activations
    between the kernels, up to 2.3e-6 with 32-bit sums over 48 layers (five times that for the largest of them)."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 1.5e-2, "max": 0.15}


# ------------------------------------------------------------------ the same in 64 bits
def layer_norm(x, w, name, eps):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], w[name + ".weight"].double(), w[name + ".bias"].double(), eps)


def attend(q, k, v, scale):
    """Causal softmax attention over whole sequences; q [T, heads, d], k and v [T, groups, d]."""
    t, heads = q.shape[:2]
    hidden = torch.ones((t, t), dtype=torch.bool, device=q.device).triu(1)
    out = torch.empty_like(q)
    for h in range(heads):
        g = h // (heads // k.shape[1])
        scores = (q[:, h] @ k[:, g].t() * scale).masked_fill(hidden, -math.inf)
        out[:, h] = torch.softmax(scores, dim=-1) @ v[:, g]
    return out.reshape(t, -1)


def gpt2_layer(case, w, i, x, sequences):
    p, heads = f"h.{i}.", case["heads"]
    scale = (case["width"] // heads) ** -0.5 / ((i + 1) if case["scale_by_layer"] else 1)

    def linear(x, name):
        return x @ w[p + name + ".weight"].double() + w[p + name + ".bias"].double()

    qkv = linear(layer_norm(x, w, p + "ln_1", case["epsilon"]), "attn.c_attn")
    mixed = torch.cat([attend(*(t.reshape(len(s), heads, -1) for t in s.chunk(3, dim=-1)), scale) for s in qkv.split(sequences)])
    x = x + linear(mixed, "attn.c_proj")
    up = linear(layer_norm(x, w, p + "ln_2", case["epsilon"]), "mlp.c_fc")
    up = torch.nn.functional.gelu(up, approximate="tanh" if case["activation"] == "gelu_new" else "none")
    return x + linear(up, "mlp.c_proj")


def rms_norm(x, weight, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * (1.0 + weight.double())


def rotate(x):
    """Neighbouring dimensions of every head turned by position / 10000^(2 i / size)."""
    n = x.shape[-1]
    freqs = 10000.0 ** (-torch.arange(0, n, 2, dtype=torch.float64, device=x.device) / n)
    angle = (torch.arange(len(x), dtype=torch.float64, device=x.device)[:, None] * freqs)[:, None, :]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1).flatten(-2)


def bonatar_layer(case, w, i, x, ids, sequences):
    p, heads, groups = f"l{i}.", case["heads"], case["kv_heads"]

    def linear(x, name):
        return x @ w[p + name].double().t()

    h = rms_norm(x, w[p + "norm1"], case["epsilon"])
    q, k, v = (linear(h, "mix." + n).reshape(len(x), m, -1) for n, m in (("q", heads), ("k", groups), ("v", groups)))
    mixed = torch.cat([attend(rotate(a), rotate(b), c, (case["width"] // heads) ** -0.5)
                       for a, b, c in zip(q.split(sequences), k.split(sequences), v.split(sequences))])
    gate = torch.sigmoid(linear(h, "mix.g"))
    x = x + linear((mixed.reshape(len(x), heads, -1) * gate[:, :, None]).reshape(len(x), -1), "mix.o")
    h = rms_norm(x, w[p + "norm2"], case["epsilon"])
    if not case["experts"]:
        return x + linear(torch.relu(linear(h, "mlp.up")) ** 2, "mlp.down")

    def unit(rows, name):
        gate, up = linear(rows, f"mlp.{name}.gate").clamp(max=7.0), linear(rows, f"mlp.{name}.up").clamp(-7.0, 7.0)
        return linear(gate * torch.sigmoid(1.702 * gate) * (up + 1.0), f"mlp.{name}.down")

    out = unit(h, "shared")
    chosen = w[p + "mlp.table"][ids]
    for e in range(case["experts"]):
        here = (chosen == e).any(dim=1).nonzero()[:, 0]
        out[here] += unit(h[here], f"e{e}") / case["top"]
    return x + out


def exact(case, seed):
    w, all_ids = weights_of(case, seed), token_ids(case, seed)
    sequences = [len(t) for t in all_ids]
    starts = [sum(sequences[:r]) for r in range(len(sequences))]
    ids = torch.tensor([i for t in all_ids for i in t], device="cuda")
    rows = torch.tensor([starts[r] + first + n - 1 for step in plan(case) for r, first, n, wanted in step if wanted], device="cuda")
    if case["model"] == "gpt2":
        x = torch.cat([w["wte.weight"][t].double() + w["wpe.weight"][:len(t)].double() for t in ids.split(sequences)])
        for i in range(case["layers"]):
            x = gpt2_layer(case, w, i, x, sequences)
        return layer_norm(x[rows], w, "ln_f", case["epsilon"]) @ w["wte.weight"].double().t()
    x = w["embed"][ids].double() * case["width"] ** 0.5
    for i in range(case["layers"]):
        x = bonatar_layer(case, w, i, x, ids, sequences)
    return rms_norm(x[rows], w["final.norm"], case["epsilon"]) @ w["head"].double().t()
