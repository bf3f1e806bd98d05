"""What the framework is asked to do, as cases that can be timed and compared.

Ten of the twelve listed cases are single layers, each through the entry points that a program puts a model together
with (``build_part``, ``SequenceCache``, ``StepContext``, ``Part.forward``); two are whole calls, a small model and one
layer of MiniMax-M2's sizes between embedding and head, both through ``Engine.step``, which returns logits.

Every tensor is a function of a seed and a name alone (``tensor``), so the inputs of a case can be made again without
the framework: ``exact`` computes the same results from them with torch in float64.
"""
import math
import zlib

import numpy as np
import torch

from fieldrun_b200.api import build_model
from fieldrun_b200.cache import SequenceCache
from fieldrun_b200.config.plan import PartSpec
from fieldrun_b200.config.registry import architecture_for
from fieldrun_b200.engine.context import StepContext, Workspace
from fieldrun_b200.engine.engine import Engine
from fieldrun_b200.parts import build_part

DEVICE = "cuda"
PAGE = 64
DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
EPS = 1e-6

# hidden size, query heads, key heads, head size, rotated entries: MiniMax-M2's layer and the sizes of the comparison of designs
ATTENTION_SIZES = {"m2": (3072, 48, 8, 128, 64), "w2048": (2048, 16, 4, 128, 64), "w1024": (1024, 16, 4, 64, 32)}
# hidden size, experts, experts a token, width of an expert
EXPERT_SIZES = {"m2": (3072, 256, 8, 1536), "w2048": (2048, 16, 2, 2048), "w1024": (1024, 16, 2, 1024)}
# width of the model, heads, key size, value size
RECURRENT_SIZES = {"w2048": (2048, 16, 128, 128), "w4096": (4096, 32, 128, 128), "w1024": (1024, 16, 64, 64)}
DECAY_RANK, DECAY_TAU, TAPS = 32, 16.0, 4
STATE_SPACE_SIZE, STATE_SPACE_VALUES, STATE_SPACE_GROUPS = 128, 64, 8

MODELS = {
    # a small model end to end: every size differs from the large one's, a routing bias that decides, whole-head rotation
    "small": dict(architectures=["MiniMaxM2ForCausalLM"], model_type="minimax_m2", num_hidden_layers=3, hidden_size=96,
                  num_attention_heads=8, num_key_value_heads=2, head_dim=12, rotary_dim=12, rope_theta=1e6, use_qk_norm=False,
                  num_local_experts=8, num_experts_per_tok=3, intermediate_size=48, vocab_size=384, rms_norm_eps=1e-5,
                  tie_word_embeddings=False),
    # MiniMax-M2's layer sizes, one layer with embedding and head
    "m2": dict(architectures=["MiniMaxM2ForCausalLM"], model_type="minimax_m2", num_hidden_layers=1, hidden_size=3072,
               num_attention_heads=48, num_key_value_heads=8, head_dim=128, rotary_dim=64, rope_theta=5e6, use_qk_norm=True,
               num_local_experts=256, num_experts_per_tok=8, intermediate_size=1536, vocab_size=200064, rms_norm_eps=1e-6,
               tie_word_embeddings=False),
}
MODEL_STD = {"small": 0.03, "m2": 0.02}


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest call there is in earnest: a small model in float32, four prompts of 1 to 30 tokens and twelve more tokens
        # each, logits of every step (the replay of a trace); hundreds of launches of almost no work
        dict(name="model_small_float32", kind="model", model="small", dtype="float32", lengths="1,7,16,30", new=12),
        # serving: eight short prompts as one step and eight decode steps at MiniMax-M2's layer sizes, logits of every step
        dict(name="model_m2_bfloat16", kind="model", model="m2", dtype="bfloat16", lengths="40,61,64,77,90,111,128,200", new=8),
        # a prompt of 2,048 tokens through MiniMax-M2's attention layer
        dict(name="attention_prompt_bfloat16", kind="attention", size="m2", dtype="bfloat16", mode="prompt", lengths="2048"),
        # one more token for each of eight long conversations, 8,192 to 65,536 tokens held
        dict(name="attention_tokens_bfloat16", kind="attention", size="m2", dtype="bfloat16", mode="tokens",
             lengths="8192,16000,24576,30001,40960,48000,61635,65536"),
        # the same layer in float32, where results are checked: a ragged batch of prompts, and one token each over what they left
        dict(name="attention_prompts_float32", kind="attention", size="m2", dtype="float32", mode="prompt",
             lengths="17,130,333,700,1024,1500"),
        dict(name="attention_tokens_float32", kind="attention", size="m2", dtype="float32", mode="tokens",
             lengths="17,130,333,700,1024,1500"),
        # the experts of MiniMax-M2's layer: a prompt of 2,048 tokens, and in float32 the ragged batch and eight single tokens
        dict(name="experts_prompt_bfloat16", kind="experts", size="m2", dtype="bfloat16", mode="prompt", tokens=2048),
        dict(name="experts_prompts_float32", kind="experts", size="m2", dtype="float32", mode="prompt", tokens=3704),
        dict(name="experts_tokens_float32", kind="experts", size="m2", dtype="float32", mode="tokens", tokens=8),
        # the recurrent layers of the other designs at a width of 2,048, four prompts of 2,048 tokens
        dict(name="linear_attention_prompts", kind="linear_attention", size="w2048", dtype="bfloat16", lengths="2048,2048,2048,2048"),
        dict(name="delta_rule_prompts", kind="delta_rule", size="w2048", dtype="bfloat16", lengths="2048,2048,2048,2048"),
        dict(name="state_space_prompts", kind="state_space", size="w2048", dtype="bfloat16", lengths="2048,2048,2048,2048"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _lengths(rng, most_sequences, low, high, total):
    """Lengths of a batch, each drawn over its logarithm, cut so that they add up to at most ``total``."""
    out, left = [], total
    for _ in range(rng.randint(1, most_sequences)):
        n = min(_log_int(rng, low, high), left)
        if n < low:
            break
        out.append(n)
        left -= n
    return ",".join(str(n) for n in out)


def draw(rng):
    kind = rng.choice(["model", "attention", "attention", "attention", "experts", "experts", "experts", "linear_attention",
                       "delta_rule", "state_space"])
    if kind == "model":
        return dict(kind=kind, model="small", dtype="float32", lengths=_lengths(rng, 6, 1, 60, 200), new=rng.randint(1, 16))
    if kind == "attention":
        dtype, mode = rng.choice(["float32", "bfloat16"]), rng.choice(["prompt", "tokens"])
        case = dict(kind=kind, size=rng.choice(["m2", "m2", "w2048", "w1024"]), dtype=dtype, mode=mode)
        if mode == "prompt":
            return dict(case, lengths=_lengths(rng, 6, 2, 3000 if dtype == "float32" else 4096, 3704 if dtype == "float32" else 6000))
        return dict(case, lengths=_lengths(rng, 16, 16, 6000 if dtype == "float32" else 65536, 20000 if dtype == "float32" else 200000))
    if kind == "experts":
        mode = rng.choice(["prompt", "tokens"])
        return dict(kind=kind, size=rng.choice(["m2", "m2", "w2048", "w1024"]), dtype=rng.choice(["float32", "bfloat16"]), mode=mode,
                    tokens=_log_int(rng, 1, 64) if mode == "tokens" else _log_int(rng, 2, 3704))
    size = rng.choice(["w2048", "w2048", "w4096", "w1024"])
    total = 4096 if size == "w4096" else 8192
    return dict(kind=kind, size=size, dtype=rng.choice(["bfloat16", "bfloat16", "float32"]), lengths=_lengths(rng, 8, 2, 8192, total))


def _ints(text):
    return [int(n) for n in text.split(",")]


# ------------------------------------------------------------------------------------------------ inputs

def tensor(seed, name, shape, std=1.0, mean=0.0, dtype=torch.float32):
    """N(mean, std), a function of (seed, name) and the shape alone."""
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed((int(seed) << 32) ^ zlib.crc32(name.encode()))
    value = torch.randn(tuple(shape), generator=generator, device=DEVICE, dtype=torch.float32)
    return value.mul_(std).add_(mean).to(dtype)


def weight(seed, name, shape, role, dtype, std=0.02):
    """A tensor of a model by its name: matrices in the model's type, everything else float32."""
    if role == "matrix":
        return tensor(seed, name, shape, std, 0.0, dtype)
    local = name.rsplit("/", 1)[-1]
    if "norm" in local or local == "d":
        return tensor(seed, name, shape, 0.1, 1.0)
    if local.endswith("conv"):
        return tensor(seed, name, shape, 0.1, 0.5)
    if local == "decay_bias":
        return tensor(seed, name, shape, 1.0, 2.0)          # most decays close to one
    if local == "dt_bias":
        return tensor(seed, name, shape, 1.0, -3.0)         # step sizes of a few hundredths
    if local == "router" or local.endswith(".gate.weight"):
        return tensor(seed, name, shape, std)
    return tensor(seed, name, shape, 0.01)


class Source:
    """The tensors of a part or a model, by name."""

    def __init__(self, seed, dtype, std=0.02):
        self.seed, self.dtype, self.std = seed, dtype, std

    def fetch(self, need):
        return weight(self.seed, need.name, need.shape, need.role, self.dtype, self.std)


def _experts_spec(size):
    hidden, experts, top, width = EXPERT_SIZES[size]
    return PartSpec("routed_experts", {"hidden_size": hidden, "num_experts": experts, "top_k": top, "expert_width": width,
                                       "score": "sigmoid", "choice_bias": True, "renormalize": True},
                    {"router": "x/router", "choice_bias": "x/choice_bias", "w_gate": "x/{e}/gate", "w_up": "x/{e}/up", "w_down": "x/{e}/down"})


def _attention_spec(size):
    hidden, heads, kv_heads, dim, rot = ATTENTION_SIZES[size]
    names = ("q_proj", "k_proj", "v_proj", "o_proj", "q_norm", "k_norm")
    return PartSpec("gqa_attention", {"hidden_size": hidden, "num_heads": heads, "num_kv_heads": kv_heads, "head_dim": dim,
                                      "qk_norm": "full_width", "qk_norm_eps": EPS, "window": None,
                                      "position": {"kind": "rotary", "rotary_dim": rot, "theta": 5e6, "pairing": "half"}},
                    {n: "a/" + n for n in names})


def _recurrent_spec(kind, size):
    width, heads, dim, vdim = RECURRENT_SIZES[size]
    if kind == "linear_attention":
        args = {"hidden_size": width, "num_heads": heads, "head_dim": dim, "value_dim": vdim, "decay_rank": DECAY_RANK,
                "tau": DECAY_TAU, "norm_eps": EPS}
        names = ("q_proj", "k_proj", "v_proj", "gate_proj", "decay_in", "decay_out", "decay_bias", "out_norm", "o_proj")
        return PartSpec("gated_linear_attention", args, {n: "r/" + n for n in names})
    if kind == "delta_rule":
        args = {"hidden_size": width, "num_heads": heads, "num_kv_heads": heads // 4, "head_dim": dim, "value_dim": vdim, "conv": TAPS,
                "norm_eps": EPS}
        names = ("q_proj", "k_proj", "v_proj", "beta_proj", "decay_proj", "gate_proj", "q_conv", "k_conv", "v_conv", "a_log", "dt_bias",
                 "norm", "o_proj")
        return PartSpec("gated_delta_rule", args, {n: "r/" + n for n in names})
    args = {"hidden_size": width, "num_heads": 2 * width // STATE_SPACE_VALUES, "value_dim": STATE_SPACE_VALUES, "state": STATE_SPACE_SIZE,
            "groups": STATE_SPACE_GROUPS, "norm_groups": 1, "conv": TAPS, "norm_eps": EPS}
    names = ("in_proj", "conv", "conv_bias", "dt_bias", "a_log", "d", "norm", "o_proj")
    return PartSpec("scalar_decay_state_space", args, {n: "r/" + n for n in names})


def _state_shape(kind, size):
    width, heads, dim, vdim = RECURRENT_SIZES[size]
    return (2 * width // STATE_SPACE_VALUES, STATE_SPACE_SIZE, STATE_SPACE_VALUES) if kind == "state_space" else (heads, dim, vdim)


def _past(seed, index, tokens, kv_heads, dim, dtype):
    """Keys and values that a sequence already holds, [tokens, kv heads, head size] each."""
    return (tensor(seed, f"past/k{index}", (tokens, kv_heads, dim), 1.0, 0.0, dtype),
            tensor(seed, f"past/v{index}", (tokens, kv_heads, dim), 1.0, 0.0, dtype))


def _tokens(seed, vocab, count):
    return np.random.default_rng(seed + 7).integers(0, vocab, size=count)


# ------------------------------------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    dtype = DTYPES[case["dtype"]]
    kind = case["kind"]
    if kind == "model":
        config = dict(MODELS[case["model"]])
        arch = architecture_for(config, "config")
        model = build_model(arch, arch.config_from_dict(config, "config"), dtype)
        model.load(Source(seed, dtype, MODEL_STD[case["model"]]))
        lengths = _ints(case["lengths"])
        room = sum(-(-(n + case["new"]) // PAGE) * PAGE for n in lengths)
        engine = Engine(model, max_tokens=room, num_slots=len(lengths))
        ids = _tokens(seed, config["vocab_size"], sum(lengths) + case["new"] * len(lengths)).tolist()
        prompts, at = [], 0
        for n in lengths:
            prompts.append(ids[at:at + n])
            at += n
        steps = [[[t] for t in ids[at + i * len(lengths):at + (i + 1) * len(lengths)]] for i in range(case["new"])]
        return {"kind": kind, "engine": engine, "prompts": prompts, "steps": steps}
    if kind == "experts":
        spec = _experts_spec(case["size"])
        part = build_part("feed_forward", spec, dtype)
        part.load(Source(seed, dtype))
        tokens = case["tokens"]
        act32 = tensor(seed, "act", (tokens, part.hidden_size))
        lengths = [1] * tokens if case["mode"] == "tokens" else [tokens]
        starts = [100] * tokens if case["mode"] == "tokens" else [0]
        ctx = StepContext(Workspace(DEVICE), dtype, list(range(len(lengths))), starts, lengths)
        return {"kind": kind, "part": part, "ctx": ctx, "act": act32.to(dtype), "act32": act32}
    lengths = _ints(case["lengths"])
    tokens_mode = case.get("mode") == "tokens"
    spec = _attention_spec(case["size"]) if kind == "attention" else _recurrent_spec(kind, case["size"])
    part = build_part("mixer", spec, dtype)
    part.load(Source(seed, dtype))
    room = sum(-(-(n + 1) // PAGE) * PAGE for n in lengths)
    cache = SequenceCache([part.cache_need()], max_tokens=room, num_slots=len(lengths), dtype=dtype, device=DEVICE)
    part.prepare(cache.max_tokens, DEVICE)
    slots = [cache.alloc() for _ in lengths]
    line = cache.line(0)
    if tokens_mode:
        # each sequence holds its length less one token and brings one more
        held = [n - 1 for n in lengths]
        cache.begin_step(slots, held)
        cache.end_step(slots, held)
        kv_heads, dim = part.num_kv_heads, part.head_dim
        for i, n in enumerate(held):
            keys, values = _past(seed, i, n, kv_heads, dim, dtype)
            pages = -(-n // PAGE)
            padded = torch.zeros((2, pages * PAGE, kv_heads, dim), dtype=dtype, device=DEVICE)
            padded[0, :n], padded[1, :n] = keys, values
            at = line.page_table[slots[i], :pages].long()
            line.keys[at] = padded[0].view(pages, PAGE, kv_heads, dim).permute(0, 2, 1, 3)
            line.values[at] = padded[1].view(pages, PAGE, kv_heads, dim).permute(0, 2, 3, 1)
        starts, brought = held, [1] * len(lengths)
    else:
        starts, brought = [0] * len(lengths), lengths
    cache.begin_step(slots, brought)
    ctx = StepContext(Workspace(DEVICE), dtype, slots, starts, brought)
    act = tensor(seed, "act", (sum(brought), part.hidden_size), 1.0, 0.0, dtype)
    state = None
    if line.state is not None:
        shape = _state_shape(kind, case["size"])
        state = line.state.view(len(lengths), 2, -1)[:, :, :math.prod(shape)]
    return {"kind": kind, "part": part, "ctx": ctx, "act": act, "line": line, "cache": cache, "state": state}


def run(state):
    kind = state["kind"]
    if kind == "model":
        engine, logits = state["engine"], []
        slots = [engine.new_sequence() for _ in state["prompts"]]
        logits.append(engine.step(slots, state["prompts"]))
        for tokens in state["steps"]:
            logits.append(engine.step(slots, tokens))
        for slot in slots:
            engine.release(slot)
        return logits
    if kind == "experts":
        return {"update": state["part"].forward(state["ctx"], state["act"], state["act32"])}
    update = state["part"].forward(state["ctx"], state["act"], state["line"], True)
    if kind == "attention":
        return {"update": update, "keys": state["line"].keys, "values": state["line"].values}
    return {"update": update, "state": state["state"]}


# ------------------------------------------------------------------------------------------------ work and tolerance

def _experts_work(size, tokens, bytes_per):
    hidden, experts, top, width = EXPERT_SIZES[size]
    used = experts * (1.0 - (1.0 - top / experts) ** tokens)
    weights = used * 3 * hidden * width * bytes_per + experts * hidden * 4
    return weights + tokens * hidden * (bytes_per + 4 + 4), 2.0 * tokens * hidden * (3 * top * width + experts)


def _attention_work(size, pairs, held, tokens, bytes_per):
    hidden, heads, kv_heads, dim, _ = ATTENTION_SIZES[size]
    weights = (2 * heads + 2 * kv_heads) * dim * hidden
    moved = weights * bytes_per + tokens * hidden * (bytes_per + 4) + (held + tokens) * 2 * kv_heads * dim * bytes_per
    return moved, 2.0 * tokens * weights + 4.0 * heads * dim * pairs


def work(case):
    per = 4 if case["dtype"] == "float32" else 2
    kind = case["kind"]
    if kind == "model":
        c, lengths = MODELS[case["model"]], _ints(case["lengths"])
        hidden, layers, vocab = c["hidden_size"], c["num_hidden_layers"], c["vocab_size"]
        attention = 2 * (c["num_attention_heads"] + c["num_key_value_heads"]) * c["head_dim"] * hidden
        expert, experts, top = 3 * hidden * c["intermediate_size"], c["num_local_experts"], c["num_experts_per_tok"]
        moved = flops = 0.0
        for tokens, steps in ((sum(lengths), 1), (len(lengths), case["new"])):
            used = experts * (1.0 - (1.0 - top / experts) ** tokens)
            moved += steps * (per * (layers * (attention + used * expert) + vocab * hidden) + 4.0 * len(lengths) * vocab)
            flops += steps * 2.0 * (tokens * layers * (attention + top * expert) + len(lengths) * vocab * hidden)
        return {"bytes": moved, "flops": flops}
    if kind == "experts":
        moved, flops = _experts_work(case["size"], case["tokens"], per)
        return {"bytes": moved, "flops": flops}
    lengths = _ints(case["lengths"])
    if kind == "attention":
        if case["mode"] == "tokens":
            moved, flops = _attention_work(case["size"], sum(lengths), sum(lengths) - len(lengths), len(lengths), per)
        else:
            moved, flops = _attention_work(case["size"], sum(n * (n + 1) / 2 for n in lengths), 0, sum(lengths), per)
        return {"bytes": moved, "flops": flops}
    width = RECURRENT_SIZES[case["size"]][0]
    heads, dim, vdim = _state_shape(kind, case["size"])
    tokens, inner = sum(lengths), heads * vdim
    if kind == "linear_attention":
        columns, mults = 2 * heads * dim + 2 * inner + DECAY_RANK, 2
    elif kind == "delta_rule":
        columns, mults = 2 * (heads // 4) * dim + 2 * inner + 2 * heads, 4
    else:
        columns, mults = 2 * inner + 2 * STATE_SPACE_GROUPS * dim + heads, 2
    weights = (columns + inner) * width
    moved = weights * per + tokens * width * (per + 4) + 2 * 4 * len(lengths) * heads * dim * vdim
    return {"bytes": moved, "flops": 2.0 * tokens * weights + 2.0 * mults * tokens * heads * dim * vdim}


def tolerance(case):
    """About four times the distance that was measured between the results and ``exact``: 2e-6 in float32 (5.9e-6 for the
    states that a prompt of 2,048 tokens leaves), 1.7e-3 to 3.4e-3 for a layer in bfloat16, 5.8e-3 for a model's logits."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 4e-4}
    return {"rel": 2.3e-2, "max": 0.4} if case["kind"] == "model" else {"rel": 1e-2, "max": 0.2}


# ------------------------------------------------------------------------------------------------ the same in float64

def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(x, positions, rot, theta):
    """The first ``rot`` entries of every head turned by the position's angles, entry i with entry i + rot / 2."""
    half = rot // 2
    angles = positions.double()[:, None] * (theta ** (-torch.arange(half, device=DEVICE, dtype=torch.float64) * 2.0 / rot))[None]
    cos, sin = angles.cos()[:, None], angles.sin()[:, None]
    a, b = x[..., :half], x[..., half:rot]
    return torch.cat([a * cos - b * sin, b * cos + a * sin, x[..., rot:]], dim=-1)


def _attend(q, k, v, first):
    """q [n, heads, d] at positions first, first + 1, ...; k and v [m, kv heads, d] from position 0."""
    n, heads, dim = q.shape
    group = heads // k.shape[1]
    out = torch.empty_like(q)
    visible = torch.arange(k.shape[0], device=DEVICE)[None] <= (first + torch.arange(n, device=DEVICE))[:, None]
    for h in range(heads):
        scores = (q[:, h] @ k[:, h // group].T) * dim ** -0.5
        out[:, h] = scores.masked_fill_(~visible, -math.inf).softmax(-1) @ v[:, h // group]
    return out.reshape(n, heads * dim)


def _moe(x, x32, experts, top, fetch):
    """x: rows as the experts read them, x32: as the router reads them, both float64."""
    scores = torch.sigmoid(x32 @ fetch("router").T)
    picked = (scores + fetch("choice_bias")).topk(top, dim=-1).indices
    weights = scores.gather(1, picked)
    weights = weights / weights.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(experts):
        rows, rank = (picked == e).nonzero(as_tuple=True)
        if len(rows):
            z = x[rows]
            y = (torch.nn.functional.silu(z @ fetch("w_gate", e).T) * (z @ fetch("w_up", e).T)) @ fetch("w_down", e).T
            out.index_add_(0, rows, y * weights[rows, rank, None])
    return out


def _exact_attention(case, seed, dtype):
    hidden, heads, kv_heads, dim, rot = ATTENTION_SIZES[case["size"]]
    shapes = {"q_proj": (heads * dim, hidden), "k_proj": (kv_heads * dim, hidden), "v_proj": (kv_heads * dim, hidden),
              "o_proj": (hidden, heads * dim)}
    w = {n: weight(seed, "a/" + n, s, "matrix", dtype).double() for n, s in shapes.items()}
    q_norm, k_norm = (weight(seed, "a/" + n, (c * dim,), "vector", dtype).double() for n, c in (("q_norm", heads), ("k_norm", kv_heads)))
    lengths, tokens_mode = _ints(case["lengths"]), case["mode"] == "tokens"
    count = len(lengths) if tokens_mode else sum(lengths)
    act = tensor(seed, "act", (count, hidden), 1.0, 0.0, dtype).double()
    out, at = [], 0
    for i, n in enumerate(lengths):
        new, first = (1, n - 1) if tokens_mode else (n, 0)
        x = act[at:at + new]
        at += new
        positions = first + torch.arange(new, device=DEVICE)
        q = _rotate(_rms(x @ w["q_proj"].T, q_norm, EPS).view(new, heads, dim), positions, rot, 5e6)
        k = _rotate(_rms(x @ w["k_proj"].T, k_norm, EPS).view(new, kv_heads, dim), positions, rot, 5e6)
        v = (x @ w["v_proj"].T).view(new, kv_heads, dim)
        if tokens_mode:
            past = _past(seed, i, first, kv_heads, dim, dtype)
            k, v = torch.cat([past[0].double(), k]), torch.cat([past[1].double(), v])
        out.append(_attend(q, k, v, first) @ w["o_proj"].T)
    return {"update": torch.cat(out), "keys": None, "values": None}


def _exact_experts(case, seed, dtype):
    hidden, experts, top, width = EXPERT_SIZES[case["size"]]

    def fetch(local, e=None):
        if local == "router":
            return weight(seed, "x/router", (experts, hidden), "vector", dtype).double()
        if local == "choice_bias":
            return weight(seed, "x/choice_bias", (experts,), "vector", dtype).double()
        shape = (hidden, width) if local == "w_down" else (width, hidden)
        return weight(seed, f"x/{e}/{local[2:]}", shape, "matrix", dtype).double()
    act32 = tensor(seed, "act", (case["tokens"], hidden))
    return {"update": _moe(act32.to(dtype).double(), act32.double(), experts, top, fetch)}


def _exact_model(case, seed, dtype):
    c = MODELS[case["model"]]
    hidden, heads, kv_heads, dim, rot = (c[n] for n in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "rotary_dim"))
    experts, top, width, eps = c["num_local_experts"], c["num_experts_per_tok"], c["intermediate_size"], c["rms_norm_eps"]
    lengths, new = _ints(case["lengths"]), case["new"]

    def fetch(name, shape, role="matrix"):
        return weight(seed, name, shape, role, dtype, MODEL_STD[case["model"]])

    ids = torch.tensor(_tokens(seed, c["vocab_size"], sum(lengths) + new * len(lengths)), device=DEVICE)
    runs, at = [], 0
    for i, n in enumerate(lengths):
        runs.append(torch.cat([ids[at:at + n], ids[sum(lengths) + i::len(lengths)]]))
        at += n
    embedding = fetch("model.embed_tokens.weight", (c["vocab_size"], hidden))
    rows = [embedding[r].double() for r in runs]
    del embedding
    for layer in range(c["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        a = p + "self_attn."
        w = {n: fetch(a + n + ".weight", s).double() for n, s in
             (("q_proj", (heads * dim, hidden)), ("k_proj", (kv_heads * dim, hidden)), ("v_proj", (kv_heads * dim, hidden)),
              ("o_proj", (hidden, heads * dim)))}
        norm = fetch(p + "input_layernorm.weight", (hidden,), "vector").double()
        for i, x in enumerate(rows):
            y = _rms(x, norm, eps)
            n, positions = len(y), torch.arange(len(y), device=DEVICE)
            q, k, v = (y @ w[m].T for m in ("q_proj", "k_proj", "v_proj"))
            if c["use_qk_norm"]:
                q = _rms(q, fetch(a + "q_norm.weight", (heads * dim,), "vector").double(), eps)
                k = _rms(k, fetch(a + "k_norm.weight", (kv_heads * dim,), "vector").double(), eps)
            q, k = (_rotate(z.view(n, -1, dim), positions, rot, c["rope_theta"]) for z in (q, k))
            rows[i] = x + _attend(q, k, v.view(n, kv_heads, dim), 0) @ w["o_proj"].T
        flat = torch.cat(rows)
        y = _rms(flat, fetch(p + "post_attention_layernorm.weight", (hidden,), "vector").double(), eps)
        m = p + "block_sparse_moe."
        names = {"w_gate": ("w1", (width, hidden)), "w_up": ("w3", (width, hidden)), "w_down": ("w2", (hidden, width))}

        def expert(local, e=None):
            if local == "router":
                return fetch(m + "gate.weight", (experts, hidden), "vector").double()
            if local == "choice_bias":
                return fetch(m + "e_score_correction_bias", (experts,), "vector").double()
            return fetch(f"{m}experts.{e}.{names[local][0]}.weight", names[local][1]).double()
        flat = flat + _moe(y, y, experts, top, expert)
        rows = list(flat.split([n + new for n in lengths]))
    norm = fetch("model.norm.weight", (hidden,), "vector").double()
    head = fetch("lm_head.weight", (c["vocab_size"], hidden)).double()
    return [_rms(torch.stack([x[n - 1 + step] for x, n in zip(rows, lengths)]), norm, eps) @ head.T for step in range(new + 1)]


def _conv(x, taps):
    """A causal convolution along the tokens, taps [channels, T], the last tap on the token itself, from zeros."""
    padded = torch.cat([x.new_zeros(taps.shape[1] - 1, x.shape[1]), x])
    return sum(padded[i:i + len(x)] * taps[:, i] for i in range(taps.shape[1]))


def _exact_recurrent(case, seed, dtype):
    kind, silu = case["kind"], torch.nn.functional.silu
    width = RECURRENT_SIZES[case["size"]][0]
    heads, dim, vdim = _state_shape(kind, case["size"])
    inner, lengths = heads * vdim, _ints(case["lengths"])

    def matrix(local, rows, columns):
        return weight(seed, "r/" + local, (rows, columns), "matrix", dtype).double()

    def vector(local, *shape):
        return weight(seed, "r/" + local, shape, "vector", dtype).double()

    act = tensor(seed, "act", (sum(lengths), width), 1.0, 0.0, dtype).double()
    w_o = matrix("o_proj", width, inner)
    updates = []
    states = torch.zeros((len(lengths), 2, heads, dim, vdim), dtype=torch.float64, device=DEVICE)
    for index, x in enumerate(act.split(lengths)):
        n = len(x)
        state, outs = states.new_zeros(heads, dim, vdim), []
        if kind == "linear_attention":
            q, k = ((x @ matrix(m, heads * dim, width).T).view(n, heads, dim, 1) for m in ("q_proj", "k_proj"))
            v = (x @ matrix("v_proj", inner, width).T).view(n, heads, 1, vdim)
            inside = x @ matrix("decay_in", DECAY_RANK, width).T
            z = inside @ matrix("decay_out", heads * dim, DECAY_RANK).T + vector("decay_bias", heads * dim)
            alpha = torch.exp(torch.nn.functional.logsigmoid(z) / DECAY_TAU).view(n, heads, dim, 1)
            for t in range(n):
                state = alpha[t] * state + k[t] * v[t]
                outs.append((state * q[t]).sum(1))
            o = _rms(torch.stack(outs) * dim ** -0.5, vector("out_norm", vdim), EPS).view(n, inner)
            y = o * silu(x @ matrix("gate_proj", inner, width).T)
        elif kind == "delta_rule":
            kv = heads // 4
            q, k = (silu(_conv(x @ matrix(m + "_proj", kv * dim, width).T, vector(m + "_conv", kv * dim, TAPS))).view(n, kv, dim) for m in "qk")
            v = silu(_conv(x @ matrix("v_proj", inner, width).T, vector("v_conv", inner, TAPS))).view(n, heads, vdim)
            q, k = ((z * torch.rsqrt((z * z).sum(-1, keepdim=True) + EPS)).repeat_interleave(4, 1) for z in (q, k))
            q = q * dim ** -0.5
            beta = torch.sigmoid(x @ matrix("beta_proj", heads, width).T)
            step = torch.nn.functional.softplus(x @ matrix("decay_proj", heads, width).T + vector("dt_bias", heads))
            decay = torch.exp(-vector("a_log", heads).exp() * step)
            for t in range(n):
                state = state * decay[t][:, None, None]
                u = beta[t][:, None] * (v[t] - (state * k[t][:, :, None]).sum(1))
                state = state + k[t][:, :, None] * u[:, None]
                outs.append((state * q[t][:, :, None]).sum(1))
            o = _rms(torch.stack(outs), vector("norm", vdim), EPS).view(n, inner)
            y = o * silu(x @ matrix("gate_proj", inner, width).T)
        else:
            gn = STATE_SPACE_GROUPS * dim
            channels = inner + 2 * gn
            proj = x @ matrix("in_proj", inner + channels + heads, width).T
            xbc = silu(_conv(proj[:, inner:inner + channels], vector("conv", channels, TAPS)) + vector("conv_bias", channels))
            values = xbc[:, :inner].view(n, heads, vdim)
            b, c = (z.view(n, STATE_SPACE_GROUPS, dim).repeat_interleave(heads // STATE_SPACE_GROUPS, 1)
                    for z in (xbc[:, inner:inner + gn], xbc[:, inner + gn:]))
            step = torch.nn.functional.softplus(proj[:, inner + channels:] + vector("dt_bias", heads))
            decay = torch.exp(-vector("a_log", heads).exp() * step)
            for t in range(n):
                state = state * decay[t][:, None, None] + (step[t][:, None] * b[t])[:, :, None] * values[t][:, None]
                outs.append((state * c[t][:, :, None]).sum(1))
            y = torch.stack(outs) + vector("d", heads)[:, None] * values
            y = _rms(y.view(n, inner) * silu(proj[:, :inner]), vector("norm", inner), EPS)
        updates.append(y @ w_o.T)
        states[index, n & 1] = state
    return {"update": torch.cat(updates), "state": states.view(len(lengths), 2, -1)}


def exact(case, seed):
    dtype, kind = DTYPES[case["dtype"]], case["kind"]
    if kind == "model":
        return _exact_model(case, seed, dtype)
    if kind == "experts":
        return _exact_experts(case, seed, dtype)
    if kind == "attention":
        return _exact_attention(case, seed, dtype)
    return _exact_recurrent(case, seed, dtype)
