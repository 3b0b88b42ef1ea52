"""What a user of this engine has it do, as cases that can be timed and compared.

A case is one of five kinds of work, each through the engine's own entry points
(``EngineCore.step`` on a ``DecoderModel``, ``Sampler.sample_device``):

* ``decode``   one token for every live request, whose contexts grow from pass to pass
* ``prefill``  whole prompts in one step, their pages given back afterwards
* ``portions`` one long prompt in portions, beside requests that decode a token a step
* ``serve``    prompts, then some tokens each, then the end of the requests
* ``sample``   the next token of every row of a batch of logits, options mixed

``run`` returns the logits (or the sampled ids).  Tokens are given, not sampled from the
model's own logits, so that two correct implementations run the same tokens.

Models: the layer sizes of Llama-3.1-8B and Qwen2.5-7B (eight of their layers: a layer costs
the same wherever it stands, and inputs are made many times here), Qwen2.5-0.5B sizes whole,
and the Zokelix and Gisodra designs with dense feed-forwards (delta rule and latent attention;
gated linear attention, window attention and latent attention).  Models with routed experts
are left out: the choice between two nearly equal router scores falls either way between
correct implementations, and what follows then differs by more than rounding.
"""
import math

import numpy as np
import torch

from helios_b200.config.registry import resolve_architecture
from helios_b200.engine.batch import StepEntry
from helios_b200.engine.core import EngineCore
from helios_b200.engine.model import DecoderModel, parse_dtype
from helios_b200.engine.types import SamplingParams
from helios_b200.sampling import Sampler
from helios_b200.weights import bind_tensors, expected_tensors

PAGE = 16
#: tokens a decoding request may grow by before it ends and begins again with its prompt
ROOM = 1024
#: tokens of prompts put into one step while contexts are filled
FILL = 2048
F64 = torch.float64


# ---------------------------------------------------------------------- models
def _llama(layers):
    return {
        "architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": 128256,
        "hidden_size": 4096, "intermediate_size": 14336, "num_hidden_layers": layers,
        "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 128,
        "max_position_embeddings": 131072, "rms_norm_eps": 1e-5, "rope_theta": 500000.0,
        "rope_scaling": {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0,
                         "high_freq_factor": 4.0, "original_max_position_embeddings": 8192},
        "attention_bias": False, "tie_word_embeddings": False, "hidden_act": "silu",
        "torch_dtype": "bfloat16",
    }


def _qwen(hidden, inter, layers, heads, kv_heads, head_dim, vocab, tied):
    return {
        "architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": vocab,
        "hidden_size": hidden, "intermediate_size": inter, "num_hidden_layers": layers,
        "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": head_dim,
        "max_position_embeddings": 32768, "rms_norm_eps": 1e-6, "rope_theta": 1000000.0,
        "attention_bias": True, "tie_word_embeddings": tied, "hidden_act": "silu",
        "use_sliding_window": False, "torch_dtype": "bfloat16",
    }


def _design_sizes(size):
    """width, heads, KV heads, head size, latent rank, feed-forward, vocabulary"""
    return (2048, 16, 4, 128, 512, 8192, 32000) if size == "large" else (1024, 8, 2, 64, 256, 4096, 32000)


def _zokelix(size):
    width, heads, _kv, hd, rank, ff, vocab = _design_sizes(size)
    mlp = {"kind": "dense", "ff": ff}
    rot = {"base": 10000.0, "dims": hd // 2, "scaling": {"factor": 4.0, "fast": 32.0, "slow": 1.0, "original": 4096}}
    latent = {"type": "latent_attention", "mlp": mlp,
              "mixer": {"heads": heads, "dim": hd, "rot_dim": hd // 2, "vdim": hd, "kv_rank": rank,
                        "scale": (hd + hd // 2) ** -0.5, "rot": rot}}
    delta = {"type": "channel_delta", "mlp": mlp,
             "mixer": {"heads": heads, "kv_heads": heads, "dim": hd, "vdim": hd, "conv": 4, "low_rank": 64}}
    return {"architecture": "Zokelix", "vocab": vocab, "width": width, "norm": {"eps": 1e-5},
            "layers": [delta, delta, latent, delta, delta, latent]}


def _gisodra(size):
    width, heads, kv, hd, rank, ff, vocab = _design_sizes(size)
    mlp, mask = {"kind": "dense", "ff": ff}, {"size": 1024}
    lat = {"type": "latent_attention", "mlp": mlp,
           "mixer": {"heads": heads, "dim": hd, "rot_dim": hd // 2, "vdim": hd, "kv_rank": rank, "q_rank": 3 * rank // 2,
                     "scale": (hd + hd // 2) ** -0.5, "rot": {"dims": hd // 2, "base": 10000.0}, "mask": mask}}
    att = {"heads": heads, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": mask}
    gla = {"type": "gla", "mlp": mlp, "mixer": {"heads": heads, "dim": hd, "vdim": hd, "tau": 16.0, "decay_rank": 16}}
    return {"architecture": "Gisodra", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "logit_softcap": 30.0,
            "layers": [lat, {"type": "attention", "mixer": att, "mlp": mlp}, gla,
                       {"type": "attention", "mixer": dict(att, kv_from=1), "mlp": mlp}, gla, lat]}


MODELS = {
    "llama8b": lambda: _llama(8),
    "qwen7b": lambda: _qwen(3584, 18944, 8, 28, 4, 128, 152064, False),
    "qwen0.5b": lambda: _qwen(896, 4864, 24, 14, 2, 64, 151936, True),
    "zokelix_small": lambda: _zokelix("small"),
    "zokelix_large": lambda: _zokelix("large"),
    "gisodra_small": lambda: _gisodra("small"),
    "gisodra_large": lambda: _gisodra("large"),
}


# ---------------------------------------------------------------------- the cases
def listed():
    return [
        # one user's chat with a small model: the smallest step there is, bound by its launches
        {"name": "decode_0.5b_1", "kind": "decode", "model": "qwen0.5b", "dtype": "bfloat16", "requests": 1, "context": 512},
        # a small model under load, a number of requests that fills no tile evenly
        {"name": "decode_0.5b_200", "kind": "decode", "model": "qwen0.5b", "dtype": "bfloat16", "requests": 200, "context": 512},
        # the headline: eight requests at 4,096 tokens
        {"name": "decode_8b_8", "kind": "decode", "model": "llama8b", "dtype": "bfloat16", "requests": 8, "context": 4096},
        # a loaded server of the larger model
        {"name": "decode_8b_64", "kind": "decode", "model": "llama8b", "dtype": "bfloat16", "requests": 64, "context": 2048},
        # the headline's prompt
        {"name": "prefill_8b_2048", "kind": "prefill", "model": "llama8b", "dtype": "bfloat16", "lengths": "2048"},
        # a long document in full portions and a ragged rest, nobody beside it
        {"name": "portions_8b_12001", "kind": "portions", "model": "llama8b", "dtype": "bfloat16", "requests": 0,
         "context": 0, "prompt": 12001, "budget": 2048},
        # continuous batching: a prompt in portions beside 24 requests that decode
        {"name": "portions_7b_24", "kind": "portions", "model": "qwen7b", "dtype": "bfloat16", "requests": 24,
         "context": 1000, "prompt": 3333, "budget": 2048},
        # the 32-bit path, a few users from prompt to answer
        {"name": "serve_0.5b_float32", "kind": "serve", "model": "qwen0.5b", "dtype": "float32", "lengths": "37,128,301",
         "tokens": 12},
        # a prompt and a loaded server of the design with the delta rule and latent attention
        {"name": "prefill_zokelix_2048", "kind": "prefill", "model": "zokelix_large", "dtype": "bfloat16", "lengths": "2048"},
        {"name": "decode_zokelix_64", "kind": "decode", "model": "zokelix_large", "dtype": "bfloat16", "requests": 64,
         "context": 1000},
        # prompts of several lengths in one step of the design with gated linear and window attention
        {"name": "prefill_gisodra_ragged", "kind": "prefill", "model": "gisodra_large", "dtype": "bfloat16",
         "lengths": "700,1500,333"},
        # the step's last launch for a batch of users with options of their own
        {"name": "sample_64", "kind": "sample", "rows": 64, "vocab": 128256},
    ]


def _log_uniform(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "portions", "serve", "sample"])
    if kind == "sample":
        return {"kind": kind, "rows": _log_uniform(rng, 1, 256), "vocab": rng.choice([32000, 128256, 151936, 152064])}
    model = rng.choice(["llama8b", "qwen7b", "qwen0.5b", "qwen0.5b", "zokelix_small", "zokelix_large", "gisodra_small",
                        "gisodra_large"])
    case = {"kind": kind, "model": model, "dtype": "bfloat16"}
    if kind == "decode":
        case["requests"] = _log_uniform(rng, 1, 160)
        # at most the 131,072 tokens of context that the largest listed batch holds
        case["context"] = _log_uniform(rng, 64, max(64, min(4096, 131072 // case["requests"])))
    elif kind == "prefill":
        case["lengths"] = ",".join(str(_log_uniform(rng, 5, 2048)) for _ in range(rng.randint(1, 4)))
    elif kind == "portions":
        case.update(requests=rng.randint(0, 24), context=_log_uniform(rng, 64, 1024), prompt=_log_uniform(rng, 600, 6000),
                    budget=rng.choice([512, 1024, 2048]))
    else:
        case["model"] = rng.choice(["qwen0.5b", "zokelix_small", "gisodra_small"])
        case["dtype"] = rng.choice(["float32", "float32", "bfloat16"])
        case["lengths"] = ",".join(str(_log_uniform(rng, 3, 300)) for _ in range(rng.randint(1, 5)))
        case["tokens"] = rng.randint(2, 12)
    return case


# ---------------------------------------------------------------------- inputs
def _lengths(case):
    return [int(n) for n in case["lengths"].split(",")]


def _config(case):
    return MODELS[case["model"]]()


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _bound_plan(case, seed):
    """The model's plan with random weights bound, and those weights by name."""
    cfg = _config(case)
    arch = resolve_architecture(cfg)
    plan = arch.build_plan(arch.parse_config(cfg))
    tensors = _draw_weights(plan, case, seed)
    return plan, tensors


def _draw_weights(plan, case, seed):
    """Matrices N(0, 0.02) in the compute dtype, vectors in 32 bits.  As in trained models, and
    unlike in freshly drawn ones, a sublayer adds a fraction to the stream that the embedding
    began (the last matrix of a sublayer, or the norm on its output, is small beside the
    embedding): otherwise the logits are the rounding of the last layers' sums."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + 17)
    dtype = parse_dtype(case["dtype"])
    stream = 0.1 if plan.tied else 1.0           # a table that is the head as well has smaller rows
    output_norms = {"zokelix": (".norm1", ".norm2"), "gisodra": (".norm1b", ".norm2b")}.get(
        case["model"].split("_")[0], ())
    tensors = {}
    for name, (_part, _local, spec) in expected_tensors(plan).items():
        if name in plan.tied:
            continue
        t = torch.randn(spec.shape, generator=gen, device="cuda") * spec.std
        if spec.init == "ones_jitter":
            t += 1.0
        if name in ("embed", "model.embed_tokens.weight"):
            t *= stream / 0.02
        elif name.endswith((".o_proj.weight", ".down_proj.weight")):
            t *= 0.2 * stream
        elif name.endswith(output_norms):
            t *= 0.3 * stream
        tensors[name] = t if spec.kind == "vector" else t.to(dtype)
    return tensors


def _tokens(case, seed):
    """Token ids of every request: decoding ones first (context + ROOM + a step each), prompts after."""
    gen = torch.Generator().manual_seed(seed * 7919 + 5)
    vocab = _vocab(_config(case))

    def ids(n):
        return torch.randint(0, vocab, (n,), generator=gen).tolist()

    live = [ids(case["context"] + ROOM + 64) for _ in range(case.get("requests", 0))]
    if case["kind"] == "portions":
        prompts = [ids(case["prompt"])]
    elif case["kind"] == "serve":
        prompts = [ids(n + case["tokens"]) for n in _lengths(case)]
    elif case["kind"] == "prefill":
        prompts = [ids(n) for n in _lengths(case)]
    else:
        prompts = []
    return live, prompts


class _Live:
    """Requests that decode: their ids (new ones every time they begin again), given tokens and
    how far they are."""

    def __init__(self, core, tokens, context):
        self.core, self.tokens, self.context = core, tokens, context
        self.at, self.life = None, 0

    def fill(self):
        """Prompts of ``context`` tokens each, as many in a step as FILL tokens hold."""
        for i in range(len(self.tokens)):
            if self.at is not None:
                self.core.end((self.life, i))
        self.life += 1
        parts = []
        for i, toks in enumerate(self.tokens):
            for lo in range(0, self.context, FILL):
                parts.append((i, toks[lo:min(self.context, lo + FILL)]))
        step, used, names = [], 0, set()
        for i, part in parts + [(None, [0] * (FILL + 1))]:
            if step and (used + len(part) > FILL or i in names):
                self.core.step([StepEntry((self.life, j), p, (len(p) - 1,)) for j, p in step])
                step, used, names = [], 0, set()
            if i is not None:
                step.append((i, part))
                names.add(i)
                used += len(part)
        self.at = self.context

    def entries(self):
        """The next token of every request."""
        if not self.tokens:
            return []
        if self.at + 1 > self.context + ROOM:
            self.fill()
        out = [StepEntry((self.life, i), (toks[self.at],), (0,)) for i, toks in enumerate(self.tokens)]
        self.at += 1
        return out


def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    plan, tensors = _bound_plan(case, seed)
    bind_tensors(plan, tensors)
    del tensors
    model = DecoderModel(plan, parse_dtype(case["dtype"]), torch.device("cuda:0"))
    live, prompts = _tokens(case, seed)
    context = case.get("context", 0)
    longest = max([context + ROOM + 64 if live else 0] + [len(p) for p in prompts])
    pages = len(live) * ((context + ROOM + 64) // PAGE + 1) + sum(len(p) // PAGE + 2 for p in prompts) + 8
    core = EngineCore(model, page_size=PAGE, num_pages=pages, max_slots=len(live) + len(prompts) + 1,
                      max_model_len=longest)
    state = {"case": case, "core": core, "prompts": prompts, "live": _Live(core, live, context), "served": 0}
    # a running server: contexts there, the shapes that come again and again captured
    if live:
        state["live"].fill()
    for _ in range({"decode": 4, "prefill": 10, "portions": 10 if not live else 9, "serve": 4}[case["kind"]]):
        run(state)
    if live:
        state["live"].fill()
    return state


def _prepare_sample(case, seed):
    """Logits as a trained model has them: a normal bulk (a few hundred tokens hold most of the mass),
    and users with the usual mixture of options."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 31 + 3)
    rows = case["rows"]
    logits = torch.randn(rows, case["vocab"], generator=gen, device="cuda") * 4.0
    kinds = [SamplingParams(max_tokens=1, temperature=0.0),
             SamplingParams(max_tokens=1, temperature=0.8, top_k=50, top_p=0.9),
             SamplingParams(max_tokens=1, temperature=1.0),
             SamplingParams(max_tokens=1, temperature=0.7, top_p=0.95),
             SamplingParams(max_tokens=1, temperature=1.1, top_k=20)]
    pick = np.random.RandomState(seed % (1 << 31)).permutation(max(rows, len(kinds)))[:rows] % len(kinds)
    pick[0] = 1                      # the batch has somebody with a top-k and a top-p
    return {"case": case, "logits": logits, "params": [kinds[int(i)] for i in pick],
            "seeds": [seed * 1009 + i for i in range(rows)], "offsets": [3 * i % 101 for i in range(rows)],
            "sampler": Sampler()}


# ---------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sample":
        return state["sampler"].sample_device(state["logits"], state["params"], state["seeds"], state["offsets"])
    core, live, prompts = state["core"], state["live"], state["prompts"]
    state["served"] += 1
    ids = [("prompt", state["served"], i) for i in range(len(prompts))]
    if kind == "decode":
        return core.step(live.entries())
    if kind == "prefill":
        logits = core.step([StepEntry(i, p, (len(p) - 1,)) for i, p in zip(ids, prompts)])
        for i in ids:
            core.end(i)
        return logits
    out = []
    if kind == "portions":
        prompt, done = prompts[0], 0
        while done < len(prompt):
            entries = live.entries()
            part = prompt[done:done + case["budget"] - len(entries)]
            done += len(part)
            # only the prompt's end has a next token to choose
            last = done == len(prompt)
            logits = core.step(entries + [StepEntry(ids[0], part, (len(part) - 1,) if last else ())])
            if logits is not None:
                out.append(logits.clone())       # a step's logits hold until the next step
        core.end(ids[0])
        return out
    n = _lengths(case)                           # serve
    out.append(core.step([StepEntry(i, p[:k], (k - 1,)) for i, p, k in zip(ids, prompts, n)]).clone())
    for t in range(case["tokens"]):
        out.append(core.step([StepEntry(i, (p[k + t],), (0,)) for i, p, k in zip(ids, prompts, n)]).clone())
    for i in ids:
        core.end(i)
    return out


# ---------------------------------------------------------------------- what a pass cannot do without
def _layer_sizes(cfg):
    """Per layer: (parameters, kind of mixer, numbers for attention or state)."""
    if "layers" not in cfg:
        H, I = cfg["hidden_size"], cfg["intermediate_size"]
        nh, nkv, hd = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        return [(H * hd * (2 * nh + 2 * nkv) + 3 * H * I, "attention",
                 {"qk": nh * hd, "pv": nh * hd, "row": 2 * nkv * hd, "window": None})] * cfg["num_hidden_layers"]
    out, H = [], cfg["width"]
    for layer in cfg["layers"]:
        m = layer["mixer"]
        ff = 3 * H * layer["mlp"]["ff"]
        nh, d, dv = m["heads"], m["dim"], m["vdim"]
        window = m.get("mask", {}).get("size")
        if layer["type"] == "latent_attention":
            r, dr, rq = m["kv_rank"], m["rot_dim"], m.get("q_rank")
            p = H * (r + dr) + nh * (d + dv) * r + nh * dv * H + ((H * rq + rq * nh * (d + dr) + nh * H) if rq else H * nh * (d + dr))
            out.append((p + ff, "attention", {"qk": nh * (d + dr), "pv": nh * dv, "row": r + dr, "window": window}))
        elif layer["type"] == "attention":
            own = m.get("kv_from") is None
            kv = m["kv_heads"] * (d + dv)
            out.append((H * nh * (d + dv) + (H * kv if own else 0) + ff, "attention",
                        {"qk": nh * d, "pv": nh * dv, "row": kv, "window": window}))
        else:
            low = (2 * m["low_rank"] * H + m["low_rank"] * nh * (d + dv) + nh * H) if layer["type"] == "channel_delta" \
                else m["decay_rank"] * (H + nh * d) + H * nh * dv
            out.append((H * nh * (2 * d + dv) + nh * dv * H + low + ff, "state",
                        {"state": nh * d * dv, "ops": (8 if layer["type"] == "channel_delta" else 6) * nh * d * dv}))
    return out


def _step_work(cfg, size, pieces, wanted):
    """Bytes and flops of one step; pieces: (tokens before, new tokens) per request."""
    tokens = sum(n for _s, n in pieces)
    H, V = cfg.get("hidden_size") or cfg["width"], _vocab(cfg)
    nbytes, flops = V * H * size * bool(wanted) + tokens * H * size + 4 * wanted * V, 2 * V * H * wanted
    for params, kind, m in _layer_sizes(cfg):
        nbytes += params * size
        flops += 2 * params * tokens
        for start, n in pieces:
            if kind == "state":
                nbytes += 4 * m["state"] * (1 if start == 0 else 2)
                flops += m["ops"] * n
                continue
            w = m["window"] or (1 << 60)
            nbytes += size * m["row"] * (min(start, w - 1) + n)
            # keys a query at position i sees: min(i + 1, window)
            keys = sum(min(i + 1, w) for i in range(start, start + n))
            flops += 2 * (m["qk"] + m["pv"]) * keys
    return nbytes, flops


def work(case):
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n, "flops": 2 * n}
    cfg, size = _config(case), 4 if case["dtype"] == "float32" else 2
    live = [(case.get("context", 0), 1)] * case.get("requests", 0)
    steps = []
    if case["kind"] == "decode":
        steps.append((live, len(live)))
    elif case["kind"] == "prefill":
        steps.append(([(0, n) for n in _lengths(case)], len(_lengths(case))))
    elif case["kind"] == "portions":
        done = 0
        while done < case["prompt"]:
            n = min(case["budget"] - len(live), case["prompt"] - done)
            steps.append((live + [(done, n)], len(live) + (done + n == case["prompt"])))
            done += n
    else:
        n = _lengths(case)
        steps.append(([(0, k) for k in n], len(n)))
        steps += [([(k + t, 1) for k in n], len(n)) for t in range(case["tokens"])]
    total = [_step_work(cfg, size, *s) for s in steps]
    return {"bytes": sum(b for b, _f in total), "flops": sum(f for _b, f in total)}


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.005}     # a draw that falls on a rounding of the mass
    # Measured against 64 bits: 7e-7 in float32, 0.002 to 0.006 in bfloat16 (matrices, the
    # products' inputs and the cache have 8 bits); about four times that between two
    # correct implementations.
    return {"rel": 5e-6, "max": 1e-4} if case["dtype"] == "float32" else {"rel": 0.02, "max": 0.25}


# ---------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _angles(dims, base, scaling, positions):
    """cos and sin [T, dims / 2] of position * frequency, with the scaling of the configuration."""
    i = torch.arange(dims // 2, dtype=F64, device="cuda")
    f, factor = base ** (-2.0 * i / dims), 1.0
    if scaling and "low_freq_factor" in scaling:
        wave, orig = 2.0 * math.pi / f, scaling["original_max_position_embeddings"]
        lo, hi = scaling["low_freq_factor"], scaling["high_freq_factor"]
        s = ((orig / wave - lo) / (hi - lo)).clamp(0.0, 1.0)
        f = (1.0 - s) * f / scaling["factor"] + s * f
    elif scaling:
        def at(t):
            return dims * math.log(scaling["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, factor = f / scaling["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0
    a = positions.to(F64)[:, None] * f[None, :]
    return torch.cos(a) * factor, torch.sin(a) * factor


def _rotate(x, cs, pairs):
    """x [T, heads, d]: halves of the first 2 * len values, or neighbouring pairs, are turned."""
    c, s = cs[0][:, None, :], cs[1][:, None, :]
    n = c.shape[-1]
    out = x.clone()
    if pairs:
        u, v = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
        out[..., 0:2 * n:2], out[..., 1:2 * n:2] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., :n], x[..., n:2 * n]
        out[..., :n], out[..., n:2 * n] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, window, sink):
    """Causal (and windowed) softmax attention of one request; sink [heads] or None."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device="cuda")
    dist = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None, :]
    hidden = (dist < 0) if window is None else (dist < 0) | (dist >= window)
    # (heads one at a time where T is long: the scores are T x T in 64 bits)
    per = max(1, (1 << 28) // (T * T))
    for h0 in range(0, H, per):
        hs = list(range(h0, min(H, h0 + per)))
        g = torch.tensor([h // (H // G) for h in hs], device="cuda")
        s = torch.matmul(q[:, hs].transpose(0, 1), k[:, g].permute(1, 2, 0)) * scale
        s.masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[hs][:, None, None].expand(-1, T, 1)], dim=-1)
        p = torch.softmax(s, -1)[..., :T]
        del s
        out[:, hs] = torch.matmul(p, v[:, g].transpose(0, 1)).transpose(0, 1)
    return out


def _per_request(fn, bounds, *rows):
    """``fn`` on every request's rows, results one after the other."""
    return torch.cat([fn(*(r[a:b] for r in rows)) for a, b in bounds], 0)


def _recurrence(step, bounds, rows, shape):
    """Walks every request's rows (tensors [T, heads, ...]) token by token: ``step(S, rows of a
    token [requests, heads, ...]) -> (S, out)``; requests side by side, shorter ones padded."""
    n = max(b - a for a, b in bounds)
    idx = torch.tensor([[min(a + t, b - 1) for a, b in bounds] for t in range(n)], device="cuda")
    S = torch.zeros(len(bounds), *shape, dtype=F64, device="cuda")
    outs = []
    for t in range(n):
        S, o = step(S, *(r[idx[t]] for r in rows))
        outs.append(o)
    o = torch.stack(outs)                                # [n, requests, ...]
    return torch.cat([o[:b - a, i] for i, (a, b) in enumerate(bounds)], 0)


def _conv_silu(x, w, bounds):
    taps = w.shape[1]

    def one(r):
        rp = torch.cat([torch.zeros(taps - 1, r.shape[1], dtype=F64, device="cuda"), r], 0)
        y = sum(rp[j:j + r.shape[0]] * w[:, j] for j in range(taps))
        return y * torch.sigmoid(y)
    return _per_request(one, bounds, x)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _exact_logits(case, seed, sequences, wanted):
    """Logits [len(wanted), vocab] of whole sequences; wanted: (sequence, place)."""
    cfg = _config(case)
    plan = resolve_architecture(cfg)
    plan = plan.build_plan(plan.parse_config(cfg))
    W = _draw_weights(plan, case, seed)

    def w(name):
        return W[name].to(F64)
    bounds, at = [], 0
    for s in sequences:
        bounds.append((at, at + len(s)))
        at += len(s)
    ids = torch.tensor([t for s in sequences for t in s], device="cuda")
    positions = torch.cat([torch.arange(len(s), device="cuda") for s in sequences])
    rows = torch.tensor([bounds[i][0] + place for i, place in wanted], device="cuda")
    dense = "layers" not in cfg
    x = W["model.embed_tokens.weight" if dense else "embed"][ids].to(F64)
    if dense:
        x = _exact_dense(cfg, w, x, positions, bounds)
        head = "lm_head.weight" if "lm_head.weight" in W else "model.embed_tokens.weight"
        return _rms(x[rows], w("model.norm.weight"), cfg["rms_norm_eps"]) @ w(head).T
    x = (_exact_zokelix if cfg["architecture"] == "Zokelix" else _exact_gisodra)(cfg, w, x, positions, bounds)
    logits = _rms(x[rows], w("final.norm"), cfg["norm"]["eps"]) @ w("head" if "head" in W else "embed").T
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits


def _exact_dense(cfg, w, x, positions, bounds):
    nh, nkv, hd, eps = (cfg[k] for k in ("num_attention_heads", "num_key_value_heads", "head_dim", "rms_norm_eps"))
    cs = _angles(hd, cfg["rope_theta"], cfg.get("rope_scaling"), positions)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w(p + "input_layernorm.weight"), eps)
        qkv = []
        for name, heads in (("q", nh), ("k", nkv), ("v", nkv)):
            y = h @ w(f"{p}self_attn.{name}_proj.weight").T
            if cfg["attention_bias"]:
                y += w(f"{p}self_attn.{name}_proj.bias")
            qkv.append(y.view(-1, heads, hd))
        q, k = _rotate(qkv[0], cs, False), _rotate(qkv[1], cs, False)
        o = _per_request(lambda a, b, c: _attend(a, b, c, hd ** -0.5, None, None), bounds, q, k, qkv[2])
        x = x + o.reshape(-1, nh * hd) @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, w(p + "post_attention_layernorm.weight"), eps)
        g = h @ w(p + "mlp.gate_proj.weight").T
        g *= torch.sigmoid(g)
        g *= h @ w(p + "mlp.up_proj.weight").T
        x = x + g @ w(p + "mlp.down_proj.weight").T
    return x


def _exact_latent(h, w, p, m, eps, positions, bounds, q, pairs, sink):
    """Latent attention from its queries [T, heads, dim + rot_dim]; returns [T, heads, vdim]."""
    H, d, dv, r, rot = m["heads"], m["dim"], m["vdim"], m["kv_rank"], m["rot"]
    cs = _angles(rot["dims"], rot["base"], rot.get("scaling"), positions)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], cs, pairs)], -1)
    both = h @ w(p + "dkv").T
    c = _rms(both[:, :r], w(p + "dkv.norm"), eps)
    kr = _rotate(both[:, None, r:], cs, pairs)
    k = torch.cat([(c @ w(p + "uk").T).view(-1, H, d), kr.expand(-1, H, -1)], -1)
    v = (c @ w(p + "uv").T).view(-1, H, dv)
    window = m.get("mask", {}).get("size")
    return _per_request(lambda a, b, e: _attend(a, b, e, m["scale"], window, sink), bounds, q, k, v)


def _exact_zokelix(cfg, w, x, positions, bounds):
    eps = cfg["norm"]["eps"]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "latent_attention":
            q = (x @ w(p + "q").T).view(-1, H, d + m["rot_dim"])
            o = _exact_latent(x, w, p, m, eps, positions, bounds, q, True, None)
        else:
            KH = m["kv_heads"]
            q, k, v = (_conv_silu(x @ w(p + n).T, w(p + n + ".conv"), bounds) for n in "qkv")
            q, k, v = q.view(-1, KH, d), k.view(-1, KH, d), v.view(-1, H, dv)
            q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(H // KH, 1)
            k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // KH, 1)
            beta = torch.sigmoid(x @ w(p + "b").T)
            a = ((x @ w(p + "a1").T) @ w(p + "a2").T + w(p + "dt_bias")).view(-1, H, d)
            g = torch.exp(-torch.exp(w(p + "A_log"))[None, :, None] * torch.nn.functional.softplus(a))

            def step(S, q, k, v, b, g):
                S = g[..., None] * S
                u = b[..., None] * (v - torch.einsum("rhdm,rhd->rhm", S, k))
                S = S + k[..., None] * u[..., None, :]
                return S, torch.einsum("rhdm,rhd->rhm", S, q)
            o = _recurrence(step, bounds, (q, k, v, beta, g), (H, d, dv))
            o = _rms(o, w(p + "norm"), eps) * torch.sigmoid((x @ w(p + "g1").T) @ w(p + "g2").T).view(-1, H, dv)
        x = x + _rms(o.reshape(-1, H * dv) @ w(p + "o").T, w(f"l{i}.norm1"), eps)
        f = f"l{i}.mlp."
        y = _gelu(x @ w(f + "gate").T + w(f + "gate.b")) * (x @ w(f + "up").T + w(f + "up.b"))
        x = x + _rms(y @ w(f + "down").T + w(f + "down.b"), w(f"l{i}.norm2"), eps)
    return x


def _exact_gisodra(cfg, w, x, positions, bounds):
    eps, kept = cfg["norm"]["eps"], {}
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        h = _rms(x, w(f"l{i}.norm1"), eps)
        if layer["type"] == "latent_attention":
            q = (_rms(h @ w(p + "dq").T, w(p + "dq.norm"), eps) @ w(p + "uq").T).view(-1, H, d + m["rot_dim"])
            o = _exact_latent(h, w, p, m, eps, positions, bounds, q, False, w(p + "sink"))
            o = o * torch.sigmoid(h @ w(p + "g").T)[:, :, None]
        elif layer["type"] == "attention":
            q = _rms((h @ w(p + "q").T + w(p + "q.b")).view(-1, H, d), w(p + "q.norm"), eps)
            if m.get("kv_from") is None:
                k = _rms((h @ w(p + "k").T + w(p + "k.b")).view(-1, m["kv_heads"], d), w(p + "k.norm"), eps)
                kept[i] = k, (h @ w(p + "v").T + w(p + "v.b")).view(-1, m["kv_heads"], dv)
            k, v = kept[i if m.get("kv_from") is None else m["kv_from"]]
            sink = w(p + "sink")
            o = _per_request(lambda a, b, c: _attend(a, b, c, m["scale"], m["mask"]["size"], sink), bounds, q, k, v)
        else:
            q = (h @ w(p + "q").T).view(-1, H, d) * d ** -0.5
            k, v = (h @ w(p + "k").T).view(-1, H, d), (h @ w(p + "v").T).view(-1, H, dv)
            z = (h @ w(p + "a1").T) @ w(p + "a2").T + w(p + "a2.b")
            g = torch.sigmoid(z).view(-1, H, d) ** (1.0 / m["tau"])

            def step(S, q, k, v, g):
                S = g[..., None] * S + k[..., None] * v[..., None, :]
                return S, torch.einsum("rhdm,rhd->rhm", S, q)
            o = _rms(_recurrence(step, bounds, (q, k, v, g), (H, d, dv)), w(p + "norm"), eps).reshape(-1, H * dv)
            g = h @ w(p + "g").T
            o = o * g * torch.sigmoid(g)
        x = x + _rms(o.reshape(-1, H * dv) @ w(p + "o").T, w(f"l{i}.norm1b"), eps)
        f, h = f"l{i}.mlp.", _rms(x, w(f"l{i}.norm2"), eps)
        x = x + _rms((_gelu(h @ w(f + "gate").T) * (h @ w(f + "up").T)) @ w(f + "down").T, w(f"l{i}.norm2b"), eps)
    return x


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    # (a pass of 1.3e14 multiply-adds in 64 bits takes about ten seconds)
    cfg = _config(case)
    per_token = sum(p for p, _k, _m in _layer_sizes(cfg))
    contexts = case.get("requests", 0) * case.get("context", 0)
    prompts = case.get("prompt", 0) + sum(_lengths(case) if "lengths" in case else [])
    if (contexts + prompts) * per_token > 1.3e14:
        return None
    live, given = _tokens(case, seed)
    C, R = case.get("context", 0), len(live)
    if case["kind"] == "decode":
        return _exact_logits(case, seed, [t[:C + 1] for t in live], [(i, C) for i in range(R)])
    if case["kind"] == "prefill":
        return _exact_logits(case, seed, given, [(i, len(t) - 1) for i, t in enumerate(given)])
    if case["kind"] == "serve":
        n = _lengths(case)
        steps = [[(i, k - 1 + t) for i, k in enumerate(n)] for t in range(case["tokens"] + 1)]
        flat = _exact_logits(case, seed, given, [pl for s in steps for pl in s])
        return [flat[len(n) * t:len(n) * (t + 1)] for t in range(len(steps))]
    steps = -(-case["prompt"] // (case["budget"] - R))
    wanted = [[(i, C + t) for i in range(R)] + ([(R, case["prompt"] - 1)] if t == steps - 1 else []) for t in range(steps)]
    wanted = [s for s in wanted if s]
    flat = _exact_logits(case, seed, [t[:C + steps] for t in live] + given, [pl for s in wanted for pl in s])
    out, at = [], 0
    for s in wanted:
        out.append(flat[at:at + len(s)])
        at += len(s)
    return out
