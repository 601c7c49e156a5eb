"""The engine's work as cases that can be timed and checked: steps of paged-cache decoding, prompts in one step or in
portions, and both in one batch, through ``EngineCore``'s step function as a serving loop or a replay drives it.

A case is a model (layer sizes of the benchmark's and the tests' configurations, seeded random weights), its compute
dtype, and what one pass does:

* ``batch`` live requests, of ``context`` cached tokens at most and ``spread`` of that apart, each take one token;
* a new request of ``prompt`` tokens arrives, runs in portions of ``portion`` tokens beside them and ends.

A pass returns the float32 logits of its last step: one row per decoding request and one for the prompt's last token.
The token ids are given (as in a replay), so two implementations are compared on the same tokens; the model stays
loaded from one state to the next, as it does in a server, and a state is a set of requests with their prompts cached.
Requests grow by a token a pass; when they have grown by ``room`` they end and are admitted anew, as in a server.

Feed-forwards are dense throughout: a routed layer's choice of experts is discontinuous, so in 16-bit two correct
implementations give logits that cannot be compared number by number.
"""

from __future__ import annotations

import gc
import math

import numpy as np
import torch

F64 = torch.float64
DEVICE = "cuda:0"
PAGE = 16
FILL = 2048              # tokens a step while a state's prompts are cached
SESSIONS = 4             # states that may be live at once


# ---------------------------------------------------------------------------------------------- models
def _starcoder2(layers, hidden, heads, kv_heads, ff, vocab, theta, tied):
    return {"model_type": "starcoder2", "architectures": ["Starcoder2ForCausalLM"], "num_hidden_layers": layers,
            "hidden_size": hidden, "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": 128,
            "intermediate_size": ff, "vocab_size": vocab, "rope_theta": theta, "sliding_window": 4096,
            "max_position_embeddings": 16384, "norm_epsilon": 1e-5, "use_bias": True, "tie_word_embeddings": tied,
            "hidden_act": "gelu_pytorch_tanh"}


def _busatar():
    """Two latent attentions, gated attention and a gated linear recurrence in turn, width 2,048."""
    mlp = {"kind": "dense", "ff": 8192, "limit": 7.0}
    rot = {"base": 10000.0, "dims": 64, "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    latent = {"type": "latent_attention", "mlp": mlp,
              "mixer": {"heads": 16, "dim": 128, "rot_dim": 64, "kv_rank": 512, "vdim": 128, "mask": {"size": 4096},
                        "scale": 192 ** -0.5, "rot": rot}}
    attention = {"type": "attention", "mlp": mlp, "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128,
                                                            "mask": {"size": 4096}, "scale": 128 ** -0.5}}
    recurrence = {"type": "rglru", "mlp": mlp, "mixer": {"width": 2048, "blocks": 16, "conv": 4}}
    return {"architecture": "Busatar", "vocab": 32768, "width": 2048, "postln_alpha": 2.0, "norm": {"eps": 1e-5},
            "layers": [latent, latent, attention, recurrence] * 2}


def _palelix():
    """Attention beside a delta rule, lightning attention and the gated delta rule in turn, the second and third layer
    run twice, width 2,048."""
    mlp = {"kind": "dense", "ff": 8192}
    parallel = {"type": "parallel", "mlp": mlp,
                "mixer": {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                   "rot": {"base": 1000000.0, "dims": 64}}, "left_scale": 1.0,
                          "right": {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4}, "right_scale": 1.0}}
    lightning = {"type": "lightning", "mlp": mlp, "mixer": {"heads": 16, "dim": 128, "vdim": 128,
                                                            "decay": [1.0 - 2.0 ** (-5 - 3.0 * i / 16) for i in range(16)]}}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}}
    return {"architecture": "Palelix", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-6},
            "loop": {"start": 1, "stop": 3, "times": 2},
            "layers": [parallel, lightning, delta, parallel, lightning, delta]}


# 3B: all thirty layers. 7B and 15B: their layer sizes, eight layers, so that a state of thousands of cached tokens a
# request is made in a fraction of a second; what a layer costs does not depend on how many there are.
MODELS = {
    "starcoder2-w1024": _starcoder2(8, 1024, 8, 4, 6144, 32768, 999999.4420358813, False),
    "starcoder2-3b": _starcoder2(30, 3072, 24, 2, 12288, 49152, 999999.4420358813, True),
    "starcoder2-3b-8": _starcoder2(8, 3072, 24, 2, 12288, 49152, 999999.4420358813, True),
    "starcoder2-7b": _starcoder2(8, 4608, 36, 4, 18432, 49152, 1000000.0, False),
    "starcoder2-15b": _starcoder2(8, 6144, 48, 4, 24576, 49152, 100000.0, False),
    "busatar-w2048": _busatar(),
    "palelix-w2048": _palelix(),
}


def _tensors(raw):
    """(name, shape, how it is drawn) of every tensor of a checkpoint of ``raw``, in a fixed order."""
    if raw.get("model_type") == "starcoder2":
        yield from _starcoder2_tensors(raw)
        return
    w = raw["width"]
    norm = "zero" if raw["architecture"] == "Busatar" else "one"      # Busatar stores a scale's distance from one
    yield "embed", (raw["vocab"], w), "matrix"
    yield "head", (raw["vocab"], w), "matrix"
    yield "final.norm", (w,), norm
    if raw.get("loop"):
        yield "loop.step", (raw["loop"]["times"], w), "bias"
    for i, layer in enumerate(raw["layers"]):
        p, ff = f"l{i}.", layer["mlp"]["ff"]
        yield p + "norm1", (w,), norm
        if raw["architecture"] == "Busatar":
            yield p + "norm2", (w,), norm
        yield p + "mlp.gate", (ff, w), "matrix"
        yield p + "mlp.up", (ff, w), "matrix"
        yield p + "mlp.down", (w, ff), "matrix"
        yield from _mixer_tensors(layer["type"], layer["mixer"], p + "mix.", w)


def _starcoder2_tensors(raw):
    h, ff, vocab = raw["hidden_size"], raw["intermediate_size"], raw["vocab_size"]
    q, kv = raw["num_attention_heads"] * raw["head_dim"], raw["num_key_value_heads"] * raw["head_dim"]
    yield "model.embed_tokens.weight", (vocab, h), "matrix"
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, rows, cols in (("self_attn.q_proj", q, h), ("self_attn.k_proj", kv, h), ("self_attn.v_proj", kv, h),
                                 ("self_attn.o_proj", h, q), ("mlp.c_fc", ff, h), ("mlp.c_proj", h, ff)):
            yield p + name + ".weight", (rows, cols), "matrix"
            yield p + name + ".bias", (rows,), "bias"
        for name in ("input_layernorm", "post_attention_layernorm"):
            yield p + name + ".weight", (h,), "one"
            yield p + name + ".bias", (h,), "zero"
    yield "model.norm.weight", (h,), "one"
    yield "model.norm.bias", (h,), "zero"
    if not raw["tie_word_embeddings"]:
        yield "lm_head.weight", (vocab, h), "matrix"


def _mixer_tensors(kind, m, p, w):
    if kind == "parallel":
        yield from _mixer_tensors("softmax", m["left"], p + "left.", w)
        yield from _mixer_tensors("channel_delta", m["right"], p + "right.", w)
        return
    if kind == "rglru":
        width, blocks = m["width"], m["blocks"]
        for name in ("x", "y"):
            yield p + name, (width, w), "matrix"
            yield p + name + ".b", (width,), "bias"
        yield p + "conv", (width, m["conv"]), "taps"
        yield p + "conv.b", (width,), "bias"
        for name in ("ra", "ri"):
            yield p + name, (blocks, width // blocks, width // blocks), "gate"
            yield p + name + ".b", (blocks, width // blocks), "bias"
        yield p + "lam", (width,), "lam"
        yield p + "o", (w, width), "matrix"
        return
    heads, dim, vdim = m["heads"], m["dim"], m["vdim"]
    yield p + "o", (w, heads * vdim), "matrix"
    if kind == "latent_attention":
        yield p + "q", (heads * (dim + m["rot_dim"]), w), "matrix"
        yield p + "dkv", (m["kv_rank"] + m["rot_dim"], w), "matrix"
        yield p + "dkv.norm", (m["kv_rank"],), "one"
        yield p + "uk", (heads * dim, m["kv_rank"]), "matrix"
        yield p + "uv", (heads * vdim, m["kv_rank"]), "matrix"
        return
    key_heads = m.get("kv_heads", heads)
    delta = kind in ("delta", "channel_delta")
    yield p + "q", ((key_heads if delta else heads) * dim, w), "matrix"
    yield p + "k", (key_heads * dim, w), "matrix"
    yield p + "v", ((heads if delta else key_heads) * vdim, w), "matrix"
    if kind == "attention":
        yield p + "q.norm", (dim,), "one"
        yield p + "k.norm", (dim,), "one"
    if kind == "lightning":
        yield p + "norm", (heads * vdim,), "one"
    if kind in ("attention", "lightning", "delta"):
        yield p + "g", (heads * vdim, w), "matrix"
    if delta:
        yield p + "q.conv", (key_heads * dim, m["conv"]), "taps"
        yield p + "k.conv", (key_heads * dim, m["conv"]), "taps"
        yield p + "v.conv", (heads * vdim, m["conv"]), "taps"
        yield p + "b", (heads, w), "matrix"
        yield p + "A_log", (heads,), "A_log"
        yield p + "norm", (vdim,), "one"
        if kind == "delta":
            yield p + "a", (heads, w), "matrix"
            yield p + "dt_bias", (heads,), "dt"
        else:
            rank = w // 128
            yield p + "a1", (rank, w), "matrix"
            yield p + "a2", (heads * dim, rank), "matrix"
            yield p + "dt_bias", (heads * dim,), "dt"
            yield p + "g1", (rank, w), "matrix"
            yield p + "g2", (heads * vdim, rank), "matrix"


class Weights:
    """Seeded random tensors by checkpoint name, each drawn on the GPU when it is read. Matrices and biases are
    N(0, 0.02), scales one; taps, decays and step sizes have the ranges in which such models are initialised."""

    def __init__(self, raw, store):
        self.table = {name: (k, shape, kind) for k, (name, shape, kind) in enumerate(_tensors(raw))}
        self.store = store

    def names(self):
        return list(self.table)

    def shape(self, name):
        return self.table[name][1]

    def dtype(self, name):
        return self.store

    def read(self, name):
        k, shape, kind = self.table[name]
        g = torch.Generator(device=DEVICE)
        g.manual_seed(7919 * k + 17)
        if kind in ("one", "zero"):
            return torch.full(shape, 1.0 if kind == "one" else 0.0, device=DEVICE).to(self.store)
        if kind in ("matrix", "bias", "gate", "taps"):
            std = {"gate": 0.1, "taps": 0.5}.get(kind, 0.02)
            return torch.randn(shape, generator=g, device=DEVICE).mul_(std).to(self.store)
        u = torch.rand(shape, generator=g, device=DEVICE)
        if kind == "lam":                                              # decays of about 0.8 to 0.99 at half a gate
            return (u * 3.0 - 6.0).to(self.store)
        if kind == "A_log":                                            # rates of 1 to 16
            return torch.log(1.0 + 15.0 * u).to(self.store)
        step = torch.exp(u * math.log(100.0) + math.log(1e-3))         # "dt": steps of 0.001 to 0.1 behind a softplus
        return torch.log(torch.expm1(step)).to(self.store)


# ---------------------------------------------------------------------------------------------- cases
def _case(name, model, dtype="bfloat16", batch=0, context=0, spread=0.0, prompt=0, portion=512):
    return {"name": name, "model": model, "dtype": dtype, "batch": batch, "context": context, "spread": spread,
            "prompt": prompt, "portion": portion}


def listed():
    return [
        # one user's completion on a small model, little context: a step is all latency and launches
        _case("small-decode-1", "starcoder2-w1024", batch=1, context=101),
        # the benchmark configuration of the 3B model: one user, eight, and sixty-four at contexts of their own
        _case("3b-decode-1", "starcoder2-3b", batch=1, context=3087),
        _case("3b-decode-8", "starcoder2-3b", batch=8, context=3087),
        _case("3b-decode-64", "starcoder2-3b", batch=64, context=2003, spread=0.5),
        # the benchmark's prompt in one step, and a prompt of odd length as the chat entry cuts it
        _case("3b-prompt-2048", "starcoder2-3b", prompt=2048, portion=2048),
        _case("3b-prompt-portions", "starcoder2-3b", prompt=1391, portion=512),
        # serving: thirty-one requests of a few to 6,000 tokens decode while another one's portion of 512 runs
        _case("7b-mixed-32", "starcoder2-7b", batch=31, context=6000, spread=0.97, prompt=512),
        # long requests behind a sliding window
        _case("15b-decode-long", "starcoder2-15b", batch=8, context=9001),
        # the 32-bit path of the same model: a prompt, and a few requests decoding
        _case("f32-prompt", "starcoder2-3b-8", dtype="float32", prompt=389, portion=512),
        _case("f32-decode-4", "starcoder2-3b-8", dtype="float32", batch=4, context=701, spread=0.3),
        # latent and gated attention and a gated recurrence, sixteen users
        _case("busatar-decode-16", "busatar-w2048", batch=16, context=1531, spread=0.4),
        # lightning attention and the delta rule over a long prompt
        _case("palelix-prompt-1777", "palelix-w2048", prompt=1777, portion=2048),
    ]


def _spread_over(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.5))))))


def draw(rng):
    """Any of the models and dtypes above; batches, contexts and prompts over their ranges on a logarithmic scale."""
    most = max(work(case)["flops"] for case in listed()), max(work(case)["bytes"] for case in listed())
    while True:
        model, dtype = rng.choice([("starcoder2-w1024", "bfloat16"), ("starcoder2-3b", "bfloat16"),
                                   ("starcoder2-3b", "bfloat16"), ("starcoder2-7b", "bfloat16"),
                                   ("starcoder2-15b", "bfloat16"), ("starcoder2-3b-8", "float32"),
                                   ("busatar-w2048", "bfloat16"), ("palelix-w2048", "bfloat16")])
        direction = rng.choice(["decode", "decode", "prompt", "prompt", "mixed"])
        wide = dtype == "float32"
        case = _case("", model, dtype)
        del case["name"]
        if direction != "prompt":
            case["batch"] = _spread_over(rng, 1, 8 if wide else 64 if direction == "decode" else 31)
            case["context"] = _spread_over(rng, 60, 900 if wide else 9000 if model == "starcoder2-15b" else 3500)
            case["spread"] = rng.choice([0.0, 0.3, 0.9])
        if direction != "decode":
            case["portion"] = rng.choice([256, 512, 2048]) if direction == "prompt" else 512
            case["prompt"] = _spread_over(rng, 17, 389 if wide else 512 if direction == "mixed" else 2048)
        need = work(case)
        cached = sum(_contexts(case))
        if need["flops"] <= most[0] and need["bytes"] <= most[1] and cached <= 100_000:
            if not wide or need["flops"] <= work(listed()[8])["flops"]:
                return case


def _contexts(case):
    """Tokens cached for each decoding request: from ``context`` down to ``1 - spread`` of it."""
    n = case["batch"]
    return [max(1, round(case["context"] * (1.0 - case["spread"] * ((i * 0.618) % 1.0)))) for i in range(n)]


def _portions(case):
    return [min(case["portion"], case["prompt"] - start) for start in range(0, case["prompt"], case["portion"])] or [0]


def _room(case):
    return max(256, case["context"] // 3)


def _ids(case, seed):
    """(token ids cached for each decoding request, the ids it takes pass by pass, the new request's prompt)."""
    raw = MODELS[case["model"]]
    vocab = raw.get("vocab_size") or raw["vocab"]
    rng = np.random.default_rng([int(seed), 5])
    steps = _room(case) + len(_portions(case))
    cached = [rng.integers(0, vocab, n).tolist() for n in _contexts(case)]
    taken = [rng.integers(0, vocab, steps).tolist() for _ in cached]
    return cached, taken, rng.integers(0, vocab, case["prompt"]).tolist()


# ---------------------------------------------------------------------------------------------- a pass
_loaded = {"key": None, "core": None, "count": 0}


def _core(case):
    """The engine of the case's model, with room in its cache for several states. One is loaded at a time."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _loaded["key"] == key:
        return _loaded["core"]
    from matricxon_b200.config.registry import config_from_dict
    from matricxon_b200.engine.core import EngineCore, build_model

    _loaded.update(key=None, core=None)
    gc.collect()
    torch.cuda.empty_cache()
    raw = MODELS[case["model"]]
    store = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    model = build_model(config_from_dict(raw), Weights(raw, store), case["dtype"], DEVICE, PAGE)
    longest = max([n + _room(case) + len(_portions(case)) for n in _contexts(case)] + [case["prompt"]])
    tokens = sum(n + _room(case) + FILL // 8 for n in _contexts(case)) + case["prompt"] + FILL + PAGE
    core = EngineCore(model, max_cache_tokens=SESSIONS * tokens, max_requests=SESSIONS * (case["batch"] + 1),
                      max_step_tokens=max(FILL, case["portion"] + case["batch"]), max_model_len=longest + PAGE)
    _loaded.update(key=key, core=core)
    return core


class Session:
    """The requests of one state: cached prompts, the ids they take next, and the prompt that arrives."""

    def __init__(self, core, case, seed):
        self.core, self.portions, self.room = core, _portions(case), _room(case)
        self.cached, self.taken, self.prompt = _ids(case, seed)
        _loaded["count"] += 1
        self.ids = [f"s{_loaded['count']}-{i}" for i in range(len(self.cached))]
        self.new = f"s{_loaded['count']}-new"
        self.used = 0
        self.admit()

    def admit(self):
        from matricxon_b200.engine.step import StepEntry

        self.used = 0
        for rid, tokens in zip(self.ids, self.cached):
            self.core.cache.add_request(rid)
            for start in range(0, len(tokens), FILL):
                self.core.runner.run([StepEntry(rid, tokens[start:start + FILL], [])])

    def close(self):
        for rid in (*self.ids, self.new):
            if self.core.cache.has_request(rid):
                self.core.cache.free_request(rid)

    def __del__(self):
        self.close()


def prepare(case, seed):
    return Session(_core(case), case, seed)


def run(state):
    from matricxon_b200.engine.step import StepEntry

    core = state.core
    if state.used >= state.room:
        state.close()
        state.admit()
    if state.prompt:
        core.cache.add_request(state.new)
    start, logits = 0, None
    for count in state.portions:
        entries = [StepEntry(rid, [ids[state.used]], [0]) for rid, ids in zip(state.ids, state.taken)]
        if count:
            last = start + count == len(state.prompt)
            entries.append(StepEntry(state.new, state.prompt[start:start + count], [count - 1] if last else []))
        logits = core.runner.run(entries)
        start += count
        state.used += 1
    if state.prompt:
        core.cache.free_request(state.new)
    return logits


# ---------------------------------------------------------------------------------------------- what a pass needs
def work(case):
    """Every matrix once a step, the live cache once, the new cache entries and the logits; two operations per
    multiply-add of every product and of attention's two."""
    raw = MODELS[case["model"]]
    size = 4 if case["dtype"] == "float32" else 2
    hidden, vocab = (raw.get("hidden_size") or raw["width"]), (raw.get("vocab_size") or raw["vocab"])
    matrices = {name: math.prod(shape) for name, shape, kind in _tensors(raw) if kind in ("matrix", "gate")}
    body = sum(n for name, n in matrices.items() if "embed" not in name and "head" not in name)
    runs = [i for i, _ in _layer_runs(raw)]
    again = 0 if "layers" not in raw else sum(n * (runs.count(int(name[1:].split(".")[0])) - 1)
                                              for name, n in matrices.items() if name.startswith("l"))
    contexts, portions = _contexts(case), _portions(case)
    rows, new = len(contexts), sum(portions)
    tokens = rows * len(portions) + new
    wanted = rows * len(portions) + (1 if new else 0)
    nbytes = (body + vocab * hidden) * size * len(portions) + tokens * hidden * size + wanted * vocab * 4
    flops = 2.0 * (body + again) * tokens + 2.0 * vocab * hidden * wanted
    for per_token, per_pair, window, state in _caches(raw):
        seen = lambda n: min(n, window or n)                                                        # noqa: E731
        live = sum(seen(n + 1) for n in contexts) * len(portions)
        before, pairs = 0, 0
        for count in portions:
            pairs += sum(seen(before + i + 1) for i in range(count))
            live += seen(before)
            before += count
        nbytes += (live + tokens) * per_token * size + 8 * state * (rows + (1 if new else 0)) * len(portions)
        pairs += sum(seen(n + 1) for n in contexts) * len(portions)
        flops += 2.0 * per_pair * pairs + 6.0 * state * tokens
    return {"bytes": float(nbytes), "flops": flops}


def _layer_runs(raw):
    """[(layer, number of the pass of the repeated run that it opens, or None)] in order of execution."""
    n = raw.get("num_hidden_layers") or len(raw["layers"])
    loop = raw.get("loop")
    if not loop:
        return [(i, None) for i in range(n)]
    again = range(loop["start"], loop["stop"])
    return ([(i, None) for i in range(loop["start"])]
            + [(i, t if i == loop["start"] else None) for t in range(loop["times"]) for i in again]
            + [(i, None) for i in range(loop["stop"], n)])


def _caches(raw):
    """Per layer run: (numbers cached a token, multiply-adds per query and key it sees, window, numbers of state)."""
    if raw.get("model_type") == "starcoder2":
        d = raw["head_dim"]
        one = (2 * raw["num_key_value_heads"] * d, 2 * raw["num_attention_heads"] * d, raw["sliding_window"], 0)
        return [one] * raw["num_hidden_layers"]
    found = []
    for i, _ in _layer_runs(raw):
        kind, m = raw["layers"][i]["type"], raw["layers"][i]["mixer"]
        if kind == "rglru":
            found.append((0, 0, None, m["width"]))
            continue
        left = m.get("left", m)
        window = left.get("mask", {}).get("size")
        state = 0
        if kind in ("lightning", "delta", "parallel"):
            right = m.get("right", m)
            state = right["heads"] * right["dim"] * right["vdim"]
        if kind == "latent_attention":
            found.append((m["kv_rank"] + m["rot_dim"], m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), window, 0))
        elif kind in ("attention", "parallel"):
            found.append((left["kv_heads"] * (left["dim"] + left["vdim"]), left["heads"] * (left["dim"] + left["vdim"]),
                          window, state))
        else:
            found.append((0, 0, None, state))
    return found


def tolerance(case):
    """Four times what is seen: against 64 bits the 32-bit path's logits are 4e-6 off; in 16-bit, sums in another order
    move roundings and two runs are 0.005 apart (0.026 at the worst single logit), 0.005 to 0.01 from 64 bits each."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4}
    return {"rel": 0.02, "max": 0.1}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """Logits of the first pass: every sequence as a whole, layer by layer, with plain torch in float64."""
    raw = MODELS[case["model"]]
    cached, taken, prompt = _ids(case, seed)
    last = len(_portions(case))
    sequences = [c + t[:last] for c, t in zip(cached, taken)] + ([prompt] if prompt else [])
    if 2.0 * sum(math.prod(s) for _, s, k in _tensors(raw) if k == "matrix") * sum(map(len, sequences)) > 3.5e14:
        return None
    weights = Weights(raw, torch.float32 if case["dtype"] == "float32" else torch.bfloat16)
    starcoder2 = raw.get("model_type") == "starcoder2"
    embed = weights.read("model.embed_tokens.weight" if starcoder2 else "embed")
    streams = [embed[torch.tensor(s, device=DEVICE)].to(F64) for s in sequences]
    del embed
    for i, opens in _layer_runs(raw):
        prefix = f"model.layers.{i}." if starcoder2 else f"l{i}."
        w = {name[len(prefix):]: weights.read(name).to(F64) for name in weights.names() if name.startswith(prefix)}
        if opens is not None:
            step = weights.read("loop.step")[opens].to(F64)
            streams = [x + step for x in streams]
        layer = {"Busatar": _busatar_layer, "Palelix": _palelix_layer}.get(raw.get("architecture"), _starcoder2_layer)
        for k in range(len(streams)):
            streams[k] = layer(streams[k], w, raw, i)
    rows = torch.stack([x[-1] for x in streams])
    if starcoder2:
        rows = _layer_norm(rows, weights.read("model.norm.weight").to(F64), weights.read("model.norm.bias").to(F64), 1e-5)
        head = weights.read("model.embed_tokens.weight" if raw["tie_word_embeddings"] else "lm_head.weight")
    else:
        scale = weights.read("final.norm").to(F64)
        rows = _rms(rows, raw["norm"]["eps"]) * (1.0 + scale if raw["architecture"] == "Busatar" else scale)
        head = weights.read("head")
    return rows @ head.to(F64).T


def _layer_norm(x, weight, bias, eps):
    mean = x.mean(dim=-1, keepdim=True)
    var = ((x - mean) ** 2).mean(dim=-1, keepdim=True)
    return (x - mean) / torch.sqrt(var + eps) * weight + bias


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _gelu_tanh(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _rotate(x, freq, factor=1.0):
    """Rotates the first entries of x [T, heads, D], entry i with entry i + len(freq); angles are formed in float32."""
    half = freq.numel()
    angle = torch.arange(x.shape[0], device=x.device, dtype=torch.float32)[:, None] * freq[None, :].to(x.device, torch.float32)
    cos, sin = (t.to(F64)[:, None, :] * factor for t in (torch.cos(angle.to(F64)), torch.sin(angle.to(F64))))
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., 2 * half:]], dim=-1)


def _attend(q, k, v, scale, window=None):
    """Causal softmax attention of q [T, H, D] over k [T, G, D] and v [T, G, V] -> [T, H * V], some rows at a time."""
    t, heads = q.shape[:2]
    group = heads // k.shape[1]
    out = torch.empty(t, heads, v.shape[2], dtype=F64, device=q.device)
    j = torch.arange(t, device=q.device)
    for first in range(0, t, 512):
        rows = j[first:first + 512]
        low = max(0, first - window + 1) if window else 0
        high = first + rows.numel()
        seen = j[None, low:high] <= rows[:, None]
        if window:
            seen &= rows[:, None] - j[None, low:high] < window
        for g in range(k.shape[1]):
            mine = slice(g * group, (g + 1) * group)
            scores = torch.einsum("ihd,jd->hij", q[first:high, mine], k[low:high, g]) * scale
            weights = torch.softmax(scores.masked_fill_(~seen, -math.inf), dim=-1)
            out[first:high, mine] = torch.einsum("hij,jv->ihv", weights, v[low:high, g])
    return out.reshape(t, -1)


def _starcoder2_layer(x, w, raw, _index):
    t, d = x.shape[0], raw["head_dim"]
    freq = 1.0 / (raw["rope_theta"] ** (torch.arange(0, d, 2, dtype=torch.float32) / d))

    def product(h, name):
        return h @ w[name + ".weight"].T + w[name + ".bias"]

    h = _layer_norm(x, w["input_layernorm.weight"], w["input_layernorm.bias"], raw["norm_epsilon"])
    q, k = (_rotate(product(h, f"self_attn.{n}_proj").view(t, -1, d), freq) for n in "qk")
    v = product(h, "self_attn.v_proj").view(t, -1, d)
    x = x + product(_attend(q, k, v, d ** -0.5, raw["sliding_window"]), "self_attn.o_proj")
    h = _layer_norm(x, w["post_attention_layernorm.weight"], w["post_attention_layernorm.bias"], raw["norm_epsilon"])
    return x + product(_gelu_tanh(product(h, "mlp.c_fc")), "mlp.c_proj")


def _frequencies(rot):
    """(frequency per pair, factor on cos and sin), interpolated between a fast and a slow wavelength under "scaling"."""
    dims, base = rot["dims"], rot["base"]
    freq = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64)
    scaling = rot.get("scaling")
    if not scaling:
        return freq, 1.0

    def at(turns):
        return dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    low, high = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64) - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
    return freq / scaling["factor"] * ramp + freq * (1.0 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0


def _convolve(u, taps):
    """y_t = sum_j taps[:, j] u_(t - n + 1 + j) for every channel of u [T, C]; zeros before the start."""
    n = taps.shape[1]
    padded = torch.cat([u.new_zeros(n - 1, u.shape[1]), u])
    return sum(taps[:, j] * padded[j:j + u.shape[0]] for j in range(n))


def _busatar_layer(x, w, raw, index):
    eps, alpha, layer = raw["norm"]["eps"], raw["postln_alpha"], raw["layers"][index]
    kind, m, t = layer["type"], layer["mixer"], x.shape[0]
    if kind == "latent_attention":
        heads, dim = m["heads"], m["dim"]
        freq, factor = _frequencies(m["rot"])
        down = x @ w["mix.dkv"].T
        latent = _rms(down[:, :m["kv_rank"]], eps) * w["mix.dkv.norm"]
        shared = _rotate(down[:, None, m["kv_rank"]:], freq, factor)
        q = (x @ w["mix.q"].T).view(t, heads, -1)
        q = torch.cat([q[..., :dim], _rotate(q[..., dim:], freq, factor)], dim=-1)
        k = torch.cat([(latent @ w["mix.uk"].T).view(t, heads, dim), shared.expand(t, heads, -1)], dim=-1)
        v = (latent @ w["mix.uv"].T).view(t, heads, -1)
        y = _attend(q, k, v, m["scale"], m["mask"]["size"])
    elif kind == "attention":
        q, k = (_rms((x @ w[f"mix.{n}"].T).view(t, -1, m["dim"]), eps) * w[f"mix.{n}.norm"] for n in "qk")
        v = (x @ w["mix.v"].T).view(t, -1, m["vdim"])
        y = _attend(q, k, v, m["scale"], m["mask"]["size"]) * torch.sigmoid(x @ w["mix.g"].T)
    else:
        u = _convolve(x @ w["mix.x"].T + w["mix.x.b"], w["mix.conv"]) + w["mix.conv.b"]
        parts = u.view(t, m["blocks"], -1)
        r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", parts, w[f"mix.{n}"]) + w[f"mix.{n}.b"]).reshape(t, -1)
                for n in ("ra", "ri"))
        a = torch.exp(-8.0 * r * torch.nn.functional.softplus(w["mix.lam"]))
        drive = torch.sqrt(1.0 - a * a) * i * u
        state, states = torch.zeros_like(u[0]), []
        for step in range(t):
            state = a[step] * state + drive[step]
            states.append(state)
        y = torch.stack(states) * _gelu_tanh(x @ w["mix.y"].T + w["mix.y.b"])
    x = _rms(alpha * x + y @ w["mix.o"].T, eps) * (1.0 + w["norm1"])
    limit = layer["mlp"]["limit"]
    g, u = (x @ w["mlp.gate"].T).clamp(max=limit), (x @ w["mlp.up"].T).clamp(-limit, limit)
    return _rms(alpha * x + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w["mlp.down"].T, eps) * (1.0 + w["norm2"])


def _silu(z):
    return z * torch.sigmoid(z)


def _delta(h, w, p, m, eps):
    t, heads, dim = h.shape[0], m["heads"], m["dim"]
    q, k, v = (_silu(_convolve(h @ w[p + n].T, w[p + n + ".conv"])) for n in "qkv")
    share = heads // m["kv_heads"]
    q, k = (z.view(t, -1, dim) / torch.sqrt((z.view(t, -1, dim) ** 2).sum(dim=-1, keepdim=True) + 1e-6) for z in (q, k))
    q, k, v = (q * dim ** -0.5).repeat_interleave(share, dim=1), k.repeat_interleave(share, dim=1), v.view(t, heads, -1)
    rate = torch.exp(w[p + "A_log"])
    if p + "a" in w:
        decay = torch.exp(-rate * torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))[:, :, None]
        gate = _silu(h @ w[p + "g"].T)
    else:
        z = ((h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "dt_bias"]).view(t, heads, dim)
        decay = torch.exp(-rate[:, None] * torch.nn.functional.softplus(z))
        gate = torch.sigmoid((h @ w[p + "g1"].T) @ w[p + "g2"].T)
    beta = torch.sigmoid(h @ w[p + "b"].T)[:, :, None]
    state, out = h.new_zeros(heads, dim, v.shape[2]), []
    for i in range(t):
        state = state * decay[i][:, :, None]
        write = beta[i] * (v[i] - torch.bmm(k[i][:, None, :], state)[:, 0])
        state = torch.baddbmm(state, k[i][:, :, None], write[:, None, :])
        out.append(torch.bmm(q[i][:, None, :], state)[:, 0])
    return (_rms(torch.stack(out), eps) * w[p + "norm"] * gate.view(t, heads, -1)).reshape(t, -1) @ w[p + "o"].T


def _palelix_layer(x, w, raw, index):
    eps, layer, t = raw["norm"]["eps"], raw["layers"][index], x.shape[0]
    kind, m = layer["type"], layer["mixer"]
    h = _rms(x, eps) * w["norm1"]
    if kind == "lightning":
        q, k, v = (_silu(h @ w[f"mix.{n}"].T).view(t, m["heads"], -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=F64, device=x.device)
        state, out = h.new_zeros(m["heads"], m["dim"], m["vdim"]), []
        for i in range(t):
            state = torch.baddbmm(state * decay[:, None, None], k[i][:, :, None], v[i][:, None, :])
            out.append(torch.bmm(q[i][:, None, :], state)[:, 0])
        o = _rms(torch.stack(out).reshape(t, -1), eps) * w["mix.norm"] * torch.sigmoid(h @ w["mix.g"].T)
        y = o @ w["mix.o"].T
    elif kind == "delta":
        y = _delta(h, w, "mix.", m, eps)
    else:
        left = m["left"]
        freq, factor = _frequencies(left["rot"])
        q, k = (_rotate((h @ w[f"mix.left.{n}"].T).view(t, -1, left["dim"]), freq, factor) for n in "qk")
        v = (h @ w["mix.left.v"].T).view(t, -1, left["vdim"])
        y = m["left_scale"] * (_attend(q, k, v, left["scale"]) @ w["mix.left.o"].T)
        y = y + m["right_scale"] * _delta(h, w, "mix.right.", m["right"], eps)
    return x + y + (_silu(h @ w["mlp.gate"].T) * (h @ w["mlp.up"].T)) @ w["mlp.down"].T
