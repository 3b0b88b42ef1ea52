"""The Zokelix design in the engine against the plain implementation (tests/plain_zokelix.py):
each mechanism alone, whole prompts, token-by-token decoding, portions down to one and two
tokens, mixed batches with pages and slots used again, ``bin/trace_run``, greedy generation
through the scheduler; plus kernel-level cases whose inputs make one far key, a page border
or the first token stand out.  Small configurations that differ in every size."""
from __future__ import annotations

import copy
import json
import math

import pytest
import torch

from conftest import random_tokens, read_folder
import plain_zokelix as pz
import trace_util as tu

DTYPES = ["float32", "bfloat16"]
YARN = {"factor": 4.0, "fast": 16.0, "slow": 2.0, "original": 64}


def _latent(heads, dim, rot_dim, vdim, rank, scale, base=10000.0, scaling=None):
    rot = {"base": base, "dims": rot_dim}
    if scaling:
        rot["scaling"] = scaling
    return {"type": "latent_attention",
            "mixer": {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": vdim, "kv_rank": rank,
                      "scale": scale, "rot": rot}}


def _delta(heads, kv_heads, dim, vdim, conv, low_rank):
    return {"type": "channel_delta",
            "mixer": {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "conv": conv,
                      "low_rank": low_rank}}


def _dense(ff):
    return {"kind": "dense", "ff": ff}


def _moe(ff, experts, top, limit):
    return {"kind": "moe", "expert": {"ff": ff, "limit": limit}, "router": {"experts": experts, "top": top}}


def _model(vocab, width, eps, layers):
    return {"architecture": "Zokelix", "vocab": vocab, "width": width, "norm": {"eps": eps},
            "layers": [dict(layer, mlp=mlp) for layer, mlp in layers]}


# Four layers, every kind of part, grouped q/k heads in the recurrent mixer, sizes that are
# no multiple of 32, two experts a token, a layer without a feed-forward.
ZK_A = _model(211, 96, 1e-5, [
    (_latent(3, 16, 8, 24, 40, 0.2, 10000.0, YARN), _dense(136)),
    (_delta(4, 2, 24, 40, 3, 16), _moe(48, 5, 2, 2.5)),
    (_delta(2, 2, 32, 16, 2, 8), None),
    (_latent(5, 24, 16, 8, 24, 0.11, 500000.0), _moe(48, 5, 2, 2.5)),
])
# Recurrent layer first, five taps, one and three experts a token, heads of 1, a latent wider
# than a head, a dense feed-forward behind a recurrent mixer, another eps.
ZK_B = _model(150, 80, 3e-6, [
    (_delta(1, 1, 40, 72, 5, 24), _dense(88)),
    (_latent(1, 8, 24, 40, 72, 0.3, 1000.0, {"factor": 16.0, "fast": 8.0, "slow": 1.0, "original": 32}), _moe(24, 3, 1, 0.7)),
    (_latent(4, 32, 8, 16, 16, 0.05, 10000.0), None),
    (_delta(6, 3, 16, 8, 4, 8), _moe(16, 7, 3, 1.0)),
])
ZK_CONFIGS = {"zk_a": ZK_A, "zk_b": ZK_B}
ZK_SEEDS = {"zk_a": 5, "zk_b": 6}
# one layer each: a mechanism alone
ZK_ALONE = {
    "latent_only": _model(97, 64, 1e-5, [(_latent(2, 16, 16, 24, 32, 0.17, 10000.0, YARN), None)]),
    "delta_only": _model(97, 64, 1e-5, [(_delta(2, 1, 16, 24, 4, 8), None)]),
    "dense_ff": _model(97, 64, 1e-5, [(_latent(2, 8, 8, 8, 16, 0.25), _dense(72))]),
    "routed_ff": _model(97, 64, 1e-5, [(_delta(2, 2, 8, 8, 2, 8), _moe(24, 6, 2, 1.5))]),
}


def _matrix_names(weights):
    return [k for k, v in weights.items() if v.dim() >= 2 and not k.endswith(".conv")]


def _bf16(weights):
    """What the bfloat16 path keeps: matrices rounded; vectors and convolution taps as stored."""
    names = set(_matrix_names(weights))
    return {k: (v.to(torch.bfloat16).float() if k in names else v) for k, v in weights.items()}


def _wide_router_margins(cfg, weights):
    """Make every routed layer's choice a matter of the token id with margins far beyond
    rounding, so that bfloat16 and float64 choose alike: channels 0..E-1 of the embedding
    hold a code (the token's j-th expert gets 4 - j), the norms leave those channels alone
    (weight 0 there, so the residual keeps the code exactly), and router row e reads the channels
    c with c % experts == e."""
    w = {k: v.clone() for k, v in weights.items()}
    E = max((l["mlp"]["router"]["experts"] for l in cfg["layers"] if l.get("mlp") and l["mlp"]["kind"] == "moe"),
            default=0)
    if not E:
        return w
    vocab = cfg["vocab"]
    w["embed"][:, :E] = 0.0
    for i, layer in enumerate(cfg["layers"]):
        for n in ("norm1", "norm2"):
            if f"l{i}.{n}" in w:
                w[f"l{i}.{n}"][:E] = 0.0
        ml = layer.get("mlp")
        if ml and ml["kind"] == "moe":
            e_here, top = ml["router"]["experts"], ml["router"]["top"]
            r = w[f"l{i}.mlp.router"]
            r[:, :E] = 0.0
            for c in range(E):
                r[c % e_here, c] = 2.0
    top_most = max(l["mlp"]["router"]["top"] for l in cfg["layers"] if l.get("mlp") and l["mlp"]["kind"] == "moe")
    for tok in range(vocab):
        for j in range(top_most):
            w["embed"][tok, (tok + j) % E] = 4.0 - j
    return w


@pytest.fixture(scope="module")
def zk_folders(tmp_path_factory):
    """name -> folder; the router margins are made wide, and ``low_rank`` is taken out of
    config.json again, so that the loader has to read it off the tensor shapes."""
    from safetensors.torch import save_file
    from helios_b200.weights import write_model_folder

    out = {}
    base = tmp_path_factory.mktemp("zokelix")
    for name, cfg in {**ZK_CONFIGS, **ZK_ALONE}.items():
        folder = write_model_folder(base / name, cfg, ZK_SEEDS.get(name, 9))
        _cfg, weights = read_folder(folder)
        save_file(_wide_router_margins(cfg, weights), str(folder / "model.safetensors"))
        stripped = copy.deepcopy(cfg)
        for layer in stripped["layers"]:
            layer["mixer"].pop("low_rank", None)
        with open(folder / "config.json", "w") as f:
            json.dump(stripped, f)
        out[name] = folder
    return out


def _plain(cfg, weights, dtype, requests):
    w = _bf16(weights) if dtype == "bfloat16" else weights
    return {rid: pz.forward_logits(cfg, w, toks) for rid, toks in requests.items()}


def _core(folder, dtype, max_tokens, page_size=16, max_slots=4, graphs=True):
    from helios_b200.engine.core import EngineCore
    from helios_b200.engine.model import DecoderModel

    model = DecoderModel.from_folder(folder, dtype=dtype)
    return EngineCore(model, page_size=page_size, num_pages=-(-max_tokens // page_size),
                      max_slots=max_slots, poison_cache=float("nan"), use_cuda_graphs=graphs)


# bfloat16 against the plain model on the rounded weights, row by row: the root mean square
# of the error (its mean taken off) over that of the logits.  Every sublayer's output is
# normalised before it is added, so its relative rounding error enters the residual stream
# undamped: under one per cent for the median row after four layers, but 6 % for a row where
# a sublayer's output nearly cancels before it is normalised, while a fault (a lost state, a
# stale page, a wrong slot) gives tens of per cent.  float32 keeps the 2e-5 of the other
# models' tests and is the sharp comparison.
ZK_BF16_RMS = 1e-1


def _check(tb, got, plain, dtype, what):
    if dtype == "float32":
        return tu.check(tb, got, plain, dtype, what)
    assert set(got) == set(tb.rows)
    for step, rows in tb.rows.items():
        want = torch.stack([plain[rid][pos] for rid, pos in rows])
        g = torch.from_numpy(got[step]).double()
        assert torch.isfinite(g).all(), f"{what} step {step}: non-finite logits"
        d = g - want
        d = d - d.mean(-1, keepdim=True)
        w = want - want.mean(-1, keepdim=True)
        rel = (d.pow(2).mean(-1) / w.pow(2).mean(-1)).sqrt()
        worst = int(rel.argmax())
        assert rel.max() <= ZK_BF16_RMS, (f"{what} step {step}: relative error {float(rel.max()):.3e} at "
                                          f"(request, position) {rows[worst]}; the step was {tb.steps[step]}")


def _requests(cfg, lengths, seed):
    return {f"q{i}": random_tokens(cfg["vocab"], n, seed + i) for i, n in enumerate(lengths)}


# ====================================================================== without a GPU
def test_configuration_is_read_layer_by_layer_and_faults_name_the_key():
    from helios_b200.config import ConfigError
    from helios_b200.config.registry import resolve_architecture
    from helios_b200.config.zokelix_config import ChannelDeltaConfig, LatentAttentionConfig, MoeMlpConfig

    arch = resolve_architecture(ZK_A)
    assert arch.name == "Zokelix"
    cfg = arch.parse_config(ZK_A)
    assert cfg.vocab_size == 211 and cfg.width == 96 and len(cfg.layers) == 4
    assert isinstance(cfg.layers[0].mixer, LatentAttentionConfig) and cfg.layers[0].mixer.rot.scaling.factor == 4.0
    assert isinstance(cfg.layers[1].mixer, ChannelDeltaConfig) and cfg.layers[1].mixer.kv_heads == 2
    assert isinstance(cfg.layers[1].mlp, MoeMlpConfig) and cfg.layers[1].mlp.top == 2 and cfg.layers[2].mlp is None
    assert cfg.layers[3].mixer.rot.scaling is None
    for path, value, word in ((("layers", 0, "type"), "conv_mixer", "type"),
                              (("layers", 1, "mixer", "kv_heads"), 3, "kv_heads"),
                              (("layers", 1, "mlp", "router", "top"), 9, "top"),
                              (("layers", 0, "mixer", "rot", "dims"), 7, "dims"),
                              (("norm",), {}, "eps")):
        bad = copy.deepcopy(ZK_A)
        node = bad
        for key in path[:-1]:
            node = node[key]
        node[path[-1]] = value
        with pytest.raises(ConfigError, match=word):
            arch.parse_config(bad)


def test_plan_names_every_tensor_and_sizes_its_cache_and_state():
    from helios_b200.cache.manager import cache_groups_of
    from helios_b200.config.registry import resolve_architecture
    from helios_b200.weights.loader import expected_tensors

    arch = resolve_architecture(ZK_A)
    plan = arch.build_plan(arch.parse_config(ZK_A))
    names = expected_tensors(plan)
    assert names["embed"][2].shape == (211, 96) and names["head"][2].shape == (211, 96)
    assert names["final.norm"][2].shape == (96,) and names["l0.norm1"][2].shape == (96,)
    assert names["l0.mix.q"][2].shape == (3 * 24, 96) and names["l0.mix.dkv"][2].shape == (48, 96)
    assert names["l0.mix.uk"][2].shape == (48, 40) and names["l0.mix.uv"][2].shape == (72, 40)
    assert names["l0.mlp.gate.b"][2].shape == (136,) and names["l0.mlp.down.b"][2].shape == (96,)
    assert names["l1.mix.q"][2].shape == (48, 96) and names["l1.mix.v"][2].shape == (160, 96)
    assert names["l1.mix.k.conv"][2].shape == (48, 3) and names["l1.mix.a2"][2].shape == (96, 16)
    assert names["l1.mix.dt_bias"][2].shape == (96,) and names["l1.mix.A_log"][2].shape == (4,)
    assert names["l1.mlp.e4.down"][2].shape == (96, 48) and names["l1.mlp.router"][2].shape == (5, 96)
    assert "l2.norm2" not in names and "l2.mlp.router" not in names
    specs, where = cache_groups_of(plan)
    # one row a token: the latent and the shared rotated key part; two sizes, two groups
    assert [(s.num_kv_heads, s.head_dim, s.planes) for s in specs] == [(1, 48, 1), (1, 40, 1)]
    assert sorted(where) == [0, 3]
    d = plan.layers[1].mixer
    assert d.state_spec().shape == (4 * 24 * 40 + (2 * 48 + 160) * 2,)


def test_sizes_the_file_leaves_out_come_from_the_tensor_shapes(tmp_path):
    from helios_b200.config.registry import load_config
    from helios_b200.weights import write_model_folder

    folder = write_model_folder(tmp_path / "m", ZK_B, 3)
    stripped = copy.deepcopy(ZK_B)
    for layer in stripped["layers"]:
        layer["mixer"].pop("low_rank", None)
    with open(folder / "config.json", "w") as f:
        json.dump(stripped, f)
    cfg = load_config(folder)
    assert (cfg.layers[0].mixer.decay_rank, cfg.layers[0].mixer.gate_rank) == (24, 24)
    assert cfg.layers[3].mixer.decay_rank == 8


def test_yarn_frequencies_and_factor():
    from helios_b200.parts.rotary import yarn_attention_factor, yarn_frequencies

    for rot in ({"base": 10000.0, "dims": 8, "scaling": YARN},
                {"base": 250000.0, "dims": 48, "scaling": {"factor": 6.0, "fast": 24.0, "slow": 2.0, "original": 1024}},
                {"base": 1000.0, "dims": 24, "scaling": {"factor": 16.0, "fast": 8.0, "slow": 1.0, "original": 32}}):
        s = rot["scaling"]
        want, factor = pz.rotary_frequencies(rot)
        got = yarn_frequencies(rot["dims"], rot["base"], s["factor"], s["original"], s["fast"], s["slow"])
        assert torch.allclose(got, want, rtol=1e-14, atol=0)
        assert yarn_attention_factor(s["factor"]) == pytest.approx(factor, rel=1e-15)
        plain = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=torch.float64) / rot["dims"])
        assert torch.all(got <= plain * (1 + 1e-12)) and torch.all(got >= plain / s["factor"] * (1 - 1e-12))
    # some pair keeps its frequency and some pair is fully stretched in the first case
    got = yarn_frequencies(64, 10000.0, 4.0, 512, 32.0, 1.0)
    plain = 10000.0 ** (-2.0 * torch.arange(32, dtype=torch.float64) / 64)
    assert got[0] == plain[0] and got[-1] == pytest.approx(float(plain[-1]) / 4.0)


def test_toy_model_of_the_design_from_the_command_line(tmp_path):
    from helios_b200.cli import main

    out = tmp_path / "toy"
    assert main(["make-toy-model", "--arch", "zokelix", "--out", str(out), "--layers", "3", "--hidden-size", "48",
                 "--heads", "2", "--kv-heads", "1", "--vocab-size", "120"]) == 0
    cfg, weights = read_folder(out)
    assert cfg["architecture"] == "Zokelix" and [l["type"] for l in cfg["layers"]] == \
        ["latent_attention", "channel_delta", "latent_attention"]
    assert "l1.mix.A_log" in weights and "l2.mlp.router" in weights
    assert main(["info", "--model", str(out)]) == 0
    logits = pz.forward_logits(cfg, weights, [1, 2, 3])
    assert logits.shape == (3, 120) and torch.isfinite(logits).all()


# ====================================================================== kernels, inputs made to show faults
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
def test_latent_attention_kernel_far_key_page_borders_and_first_tokens(dtype):
    """One request of 300 tokens in pages of 16 handed out in a scrambled order.  A query's
    latent part is aligned with the row of ONE chosen key and scaled so that this key takes
    nearly all the weight: a far key among hundreds, the last key of a page, the first of the
    next, position 0, and the query's own position.  The kernel must return that key's latent."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    dev = "cuda"
    g = torch.Generator().manual_seed(3)
    n, page, rank, rot, heads = 300, 16, (40 if dtype == "float32" else 64), (8 if dtype == "float32" else 16), 3
    rows = torch.randn(n, rank + rot, generator=g)
    rows = (rows / rows.norm(dim=-1, keepdim=True)).to(dt).float()
    n_pages = -(-n // page)
    order = torch.randperm(n_pages + 3, generator=g)[:n_pages]
    pages = torch.full((n_pages + 4, 1, page, rank + rot), float("nan"), dtype=dt)
    for j in range(n):
        pages[order[j // page], 0, j % page] = rows[j].to(dt)
    cases = [(299, 2), (299, 15), (299, 16), (299, 0), (299, 299), (299, 287), (160, 159), (17, 16),
             (16, 16), (15, 0), (0, 0), (1, 0), (1, 1), (255, 31), (256, 32)]
    q_pos = torch.tensor([c[0] for c in cases], dtype=torch.int32)
    q = torch.zeros(len(cases), heads, rank + rot)
    for i, (_p, key) in enumerate(cases):
        for h in range(heads):
            q[i, h] = rows[key] * (40.0 + 10 * h)         # score 40..60 at the chosen key, |.| < that elsewhere
    q = q.to(dt)
    from helios_b200.engine.batch import SeqSlice
    # every query is a request of its own with one token, all reading the same pages
    ctx = SimpleNamespace(seq_of_token=torch.arange(len(cases), dtype=torch.int32, device=dev),
                          positions=q_pos.to(dev), start_pos=q_pos.to(dev), extras={}, max_context_len=n,
                          cu_tokens=torch.arange(len(cases) + 1, dtype=torch.int32, device=dev),
                          seqs=[SeqSlice(None, 0, p, 1, i) for i, (p, _k) in enumerate(cases)], num_seqs=len(cases))
    table = order.to(torch.int32).view(1, -1).repeat(len(cases), 1).contiguous().to(dev)
    qd = q.to(dev)
    out = ops.latent_attention(ctx, qd[:, :, :rank], qd[:, :, rank:], pages.to(dev), table, rank, rot, page, 1.0)
    out = out.float().cpu()
    for i, (pos, key) in enumerate(cases):
        s = torch.einsum("hd,jd->hj", q[i].double(), rows[:pos + 1].double())
        want = torch.softmax(s, -1) @ rows[:pos + 1, :rank].double()
        tol = 2e-5 if dtype == "float32" else 2e-2
        assert torch.isfinite(out[i]).all(), f"case {cases[i]}: read beyond position {pos}"
        assert (out[i].double() - want).abs().max() < tol, f"query at {pos}, key {key}"
        if pos != key or pos == 0:
            assert (out[i, -1].double() - rows[key, :rank].double()).abs().max() < 0.05


@pytest.mark.gpu
@pytest.mark.parametrize("heads,rank,rot", [(5, 160, 48), (40, 64, 16), (16, 256, 64), (3, 32, 0)])
def test_latent_attention_tensor_core_kernel_against_plain_softmax(heads, rank, rot):
    """bfloat16 sizes the tensor-core kernel takes: a decode batch of requests of unequal
    lengths (1, 2, 31, 32, 33, 300, 1000 keys; the key range cut into several blocks) and a
    portion of 77 tokens behind 200 cached ones, pages scattered, unwritten rows poisoned."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops
    from helios_b200.engine.batch import SeqSlice

    dev, page = "cuda", 16
    g = torch.Generator().manual_seed(heads)
    lens = [1, 2, 31, 32, 33, 300, 1000]
    n_pages = sum(-(-n // page) for n in lens) + 20
    pages = torch.full((n_pages + 2, 1, page, rank + rot), float("nan"), dtype=torch.bfloat16)
    order = torch.randperm(n_pages, generator=g).tolist()
    width = max(-(-n // page) for n in lens)
    rows_of, table = [], torch.full((len(lens) + 1, width), -1, dtype=torch.int32)
    for i, n in enumerate(lens + [277]):
        rows = (torch.randn(n, rank + rot, generator=g) * 0.5).to(torch.bfloat16)
        rows_of.append(rows)
        if i == len(lens):
            table = torch.cat([table[:len(lens)], torch.full((1, width), -1, dtype=torch.int32)])
        for j in range(-(-n // page)):
            pg = order.pop()
            table[i, j] = pg
            chunk = rows[j * page:(j + 1) * page]
            pages[pg, 0, :len(chunk)] = chunk
    pages, table_d = pages.to(dev), table.contiguous().to(dev)

    def run(seq_ids, starts, counts, max_ctx):
        T = sum(counts)
        q = (torch.randn(T, heads, rank + rot, generator=g) * 0.7).to(torch.bfloat16)
        seq_of_token = torch.tensor([i for i, c in enumerate(counts) for _ in range(c)], dtype=torch.int32)
        positions = torch.tensor([s + k for s, c in zip(starts, counts) for k in range(c)], dtype=torch.int32)
        cu = torch.tensor([sum(counts[:i]) for i in range(len(counts) + 1)], dtype=torch.int32)
        ctx = SimpleNamespace(seq_of_token=seq_of_token.to(dev), positions=positions.to(dev), cu_tokens=cu.to(dev),
                              start_pos=torch.tensor(starts, dtype=torch.int32, device=dev), extras={},
                              seqs=[SeqSlice(None, 0, s, c, int(cu[i])) for i, (s, c) in enumerate(zip(starts, counts))],
                              max_context_len=max_ctx, num_seqs=len(counts))
        qd = q.to(dev)
        tab = table_d[seq_ids].contiguous()
        got = ops.latent_attention(ctx, qd[:, :, :rank], qd[:, :, rank:], pages, tab, rank, rot, page, 0.3)
        ops.LATENT_ATTENTION_TENSOR_CORES = False
        try:
            plain_kernel = ops.latent_attention(ctx, qd[:, :, :rank], qd[:, :, rank:], pages, tab, rank, rot, page, 0.3)
        finally:
            ops.LATENT_ATTENTION_TENSOR_CORES = True
        got, plain_kernel = got.float().cpu().double(), plain_kernel.float().cpu().double()
        assert torch.isfinite(got).all()
        t = 0
        for i, (sid, s0, c) in enumerate(zip(seq_ids, starts, counts)):
            rows = rows_of[sid].double()
            for k in range(c):
                sc = torch.einsum("hd,jd->hj", q[t].double(), rows[:s0 + k + 1]) * 0.3
                want = torch.softmax(sc, -1) @ rows[:s0 + k + 1, :rank]
                assert (got[t] - want).abs().max() < 2e-2, f"request {sid}, position {s0 + k}"
                assert (plain_kernel[t] - want).abs().max() < 2e-2
                t += 1

    run(list(range(len(lens))), [n - 1 for n in lens], [1] * len(lens), 1000)      # decode, ranges split
    run([len(lens)], [200], [77], 277)                                             # a portion behind a cached prefix
    run([5, 2, 6], [290, 0, 990], [10, 31, 10], 1000)                              # mixed


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
def test_delta_rule_kernel_against_the_scan_in_portions(dtype):
    """The recurrence kernel on two requests in slots 2 and 0, fed in portions of 1, 2, 17 and
    45 tokens, against the plain scan of the whole sequences; strong writes (beta near 1) and
    slow decays so that a token written long ago still shows at the end."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    dev = "cuda"
    g = torch.Generator().manual_seed(8)
    heads, kv_heads, dk, dv, n = 4, 2, 24, 40, 65
    lens = {"a": n, "b": n - 20}
    qk, C = kv_heads * dk, 2 * kv_heads * dk + heads * dv
    data = {r: dict(qkv=torch.randn(m, C, generator=g).to(dt), beta=(torch.randn(m, heads, generator=g) + 3).to(dt),
                    a=(torch.randn(m, heads * dk, generator=g) - 4).to(dt)) for r, m in lens.items()}
    a_log = torch.randn(heads, generator=g) * 0.3
    dt_bias = torch.randn(heads * dk, generator=g) * 0.3
    state = torch.full((4, heads * dk * dv + 5), float("nan"), device=dev)
    state[0].zero_()
    state[2].zero_()
    slots = {"a": 2, "b": 0}
    got = {r: [] for r in lens}
    fed = {r: 0 for r in lens}
    for sizes in ([1, 2], [2, 1], [17, 17], [45, 1], [0, 1], [0, 1], [0, 1], [0, 1]):
        parts = [(r, s) for r, s in zip(lens, sizes) if s and fed[r] < lens[r]]
        parts = [(r, min(s, lens[r] - fed[r])) for r, s in parts]
        cat = lambda k: torch.cat([data[r][k][fed[r]:fed[r] + s] for r, s in parts]).contiguous().to(dev)
        cu = torch.tensor([sum(s for _r, s in parts[:i]) for i in range(len(parts) + 1)], dtype=torch.int32, device=dev)
        ctx = SimpleNamespace(cu_tokens=cu, slots=torch.tensor([slots[r] for r, _s in parts], dtype=torch.int32, device=dev),
                              num_seqs=len(parts))
        o = ops.delta_rule(ctx, cat("qkv"), (0, qk, 2 * qk), cat("beta"), cat("a"), a_log.to(dev), dt_bias.to(dev),
                           state[:, :heads * dk * dv], heads, kv_heads, dk, dv).cpu()
        off = 0
        for r, s in parts:
            got[r].append(o[off:off + s])
            off += s
            fed[r] += s
    for r, m in lens.items():
        d = {k: v.double() for k, v in data[r].items()}
        q = d["qkv"][:, :qk].view(m, kv_heads, dk)
        k = d["qkv"][:, qk:2 * qk].view(m, kv_heads, dk)
        v = d["qkv"][:, 2 * qk:].view(m, heads, dv)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        beta = torch.sigmoid(d["beta"])
        gdec = torch.exp(-torch.exp(a_log.double())[None, :, None]
                         * torch.nn.functional.softplus(d["a"] + dt_bias.double()).view(m, heads, dk))
        have = torch.cat(got[r])[:fed[r]].double().view(-1, heads, dv)
        for h in range(heads):
            want = pz.delta_scan(q[:, h // 2], k[:, h // 2], v[:, h], beta[:, h], gdec[:, h])[:fed[r]]
            assert (have[:, h] - want).abs().max() < 2e-5, f"request {r}, head {h}"
    # nothing beyond the two slots' matrices was touched
    assert torch.isnan(state[1]).all() and torch.isnan(state[3]).all() and float(state[[0, 2], -5:].abs().max()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
def test_short_convolution_carries_its_inputs_across_portions_shorter_than_its_taps(dtype):
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    dev = "cuda"
    g = torch.Generator().manual_seed(2)
    C, taps, n = 37, 5, 40
    x = torch.randn(n, C + 3, generator=g).to(dt)
    w = torch.randn(C, taps, generator=g)
    want = pz.short_conv_silu(x[:, :C].double(), w.double())
    state = torch.zeros(3, 7 + C * (taps - 1), device=dev)
    got, pos = [], 0
    for size in (1, 1, 2, 1, 3, 9, 2, 1, 1, 1, 4, 14):
        xs = x[pos:pos + size].contiguous().to(dev)
        ctx = SimpleNamespace(seq_of_token=torch.zeros(size, dtype=torch.int32, device=dev),
                              cu_tokens=torch.tensor([0, size], dtype=torch.int32, device=dev),
                              slots=torch.tensor([1], dtype=torch.int32, device=dev), num_seqs=1)
        got.append(ops.causal_conv_silu(ctx, xs, C, w.to(dev), state[:, 7:]).float().cpu())
        pos += size
    assert pos == n
    err = (torch.cat(got).double() - want).abs()
    assert (err.max() < 1e-5) if dtype == "float32" else bool((err <= 1e-2 * want.abs() + 1e-3).all())
    assert float(state[0].abs().max()) == 0 and float(state[2].abs().max()) == 0 and float(state[1, :7].abs().max()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("ff", [40, 20])
@pytest.mark.parametrize("dtype", DTYPES)
def test_router_and_experts_against_the_plain_functions(dtype, ff):
    """Same input for both sides, three of seven experts a token, a limit that clips.  An inner
    size of 20 is one the grouped product of the bfloat16 path does not take: every pair then
    streams its expert's rows, as in float32."""
    from helios_b200.csrc import ops

    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    dev = "cuda"
    g = torch.Generator().manual_seed(4)
    T, width, E, top, limit = 19, 72, 7, 3, 0.6
    h = torch.randn(T, width, generator=g).to(dt)
    W = {"router": (torch.randn(E, width, generator=g) * 0.2).to(dt).float()}
    for e in range(E):
        W[f"e{e}.gate"] = (torch.randn(ff, width, generator=g) * 0.2).to(dt).float()
        W[f"e{e}.up"] = (torch.randn(ff, width, generator=g) * 0.2).to(dt).float()
        W[f"e{e}.down"] = (torch.randn(width, ff, generator=g) * 0.2).to(dt).float()
    Wd = {k: v.double() for k, v in W.items()}
    ml = {"router": {"experts": E, "top": top}, "expert": {"ff": ff, "limit": limit}}
    want_ids, want_w = pz.router_choice(h.double(), Wd, "", top)
    logits = ops.linear_logits(h.to(dev), W["router"].to(dt).to(dev))
    ids, weights = ops.moe_topk(logits, top)
    assert torch.equal(ids.cpu().long(), want_ids)
    assert (weights.cpu().double() - want_w).abs().max() < 1e-5
    w_gu = torch.stack([torch.cat([W[f"e{e}.gate"], W[f"e{e}.up"]]) for e in range(E)]).to(dt).to(dev)
    w_d = torch.stack([W[f"e{e}.down"] for e in range(E)]).to(dt).to(dev)
    got = ops.moe_experts(h.to(dev), ids, weights, w_gu, w_d, limit).float().cpu().double()
    want = pz.routed_ff(h.double(), Wd, "", ml)
    tol = 2e-5 if dtype == "float32" else 3e-2 * float(want.abs().max())
    assert (got - want).abs().max() < tol


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
def test_gated_activations_and_the_norm_on_a_sublayer_output(dtype):
    from helios_b200.csrc import ops

    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    g = torch.Generator().manual_seed(6)
    gu = (torch.randn(11, 2 * 52, generator=g) * 2).to(dt)
    gate, up = gu[:, :52].double(), gu[:, 52:].double()
    tol = 1e-5 if dtype == "float32" else 3e-2
    got = ops.glu_act(gu.cuda(), "gelu_tanh").float().cpu().double()
    assert (got - pz.gelu_tanh(gate) * up).abs().max() < tol
    got = ops.glu_act(gu.cuda(), "clamped_swish", 1.25).float().cpu().double()
    gc, uc = gate.clamp(max=1.25), up.clamp(-1.25, 1.25)
    assert (got - gc * torch.sigmoid(1.702 * gc) * (uc + 1)).abs().max() < tol
    res = torch.randn(11, 52, generator=g)
    y = torch.randn(11, 52, generator=g).to(dt)
    w = torch.randn(52, generator=g)
    want = res.double() + pz.rms_norm(y.double(), w.double(), 1e-3)
    r = res.cuda()
    copy_ = ops.rmsnorm_add(r, y.cuda(), w.cuda(), 1e-3, dt)
    assert (r.cpu().double() - want).abs().max() < 1e-5          # the residual is float32 in both modes
    assert (copy_.float().cpu().double() - want).abs().max() < (1e-5 if dtype == "float32" else 3e-2)


# ====================================================================== the engine
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", list(ZK_ALONE) + list(ZK_CONFIGS))
def test_whole_prompts_and_every_layer(zk_folders, name, dtype):
    """Logits at every position of whole prompts (the first tokens of a sequence among them),
    and the residual stream after every layer."""
    cfg, weights = read_folder(zk_folders[name])
    reqs = _requests(cfg, [1, 2, 3, 41, 90], 100)
    plain = _plain(cfg, weights, dtype, reqs)
    tb = tu.TraceBuilder()
    for rid, toks in reqs.items():
        tu.whole(tb, rid, toks)
    core = _core(zk_folders[name], dtype, tb.live_tokens_peak)
    _check(tb, tu.run_in_process(core, tb), plain, dtype, f"{name} whole")
    # layer by layer
    from helios_b200.engine.batch import StepEntry
    w = _bf16(weights) if dtype == "bfloat16" else weights
    want_layers, _ = pz.forward_layers(cfg, w, reqs["q3"])
    seen = []

    def recording(inner):
        def forward(*args):
            residual, delta = inner(*args)
            seen.append(residual.detach().double().cpu().clone())
            return residual, delta
        return forward

    for blk in core.model.plan.layers:
        blk.forward = recording(blk.forward)
    core.step([StepEntry("layers", reqs["q3"], [0])])
    for i, (got, want) in enumerate(zip(seen, want_layers)):
        tol = 2e-5 if dtype == "float32" else 3e-2 * float(want.abs().max())
        assert (got - want).abs().max() < tol, f"{name}: residual after layer {i}"


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", list(ZK_CONFIGS))
def test_prefill_then_long_decoding_token_by_token(zk_folders, name, dtype):
    """Most of the prompt in one step, then 70 single tokens (captured decode steps): the
    state of the recurrent layers and the latent cache carry on from token to token."""
    cfg, weights = read_folder(zk_folders[name])
    reqs = _requests(cfg, [75, 131], 200)
    plain = _plain(cfg, weights, dtype, reqs)
    tb = tu.TraceBuilder()
    for rid, toks in reqs.items():
        tu.prefill_then_decode(tb, rid, toks, n_decode=70)
    core = _core(zk_folders[name], dtype, tb.live_tokens_peak)
    _check(tb, tu.run_in_process(core, tb), plain, dtype, f"{name} decode")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", list(ZK_CONFIGS))
def test_portions_of_changing_size_down_to_one_token(zk_folders, name, dtype):
    cfg, weights = read_folder(zk_folders[name])
    reqs = _requests(cfg, [64, 97, 50, 33], 300)
    plain = _plain(cfg, weights, dtype, reqs)
    tb = tu.TraceBuilder()
    sizes = [[7], [2, 31, 3, 16, 2, 17], [1, 2, 1, 1, 3, 13, 2, 1, 5], [16, 1, 15, 1]]
    for (rid, toks), sz in zip(reqs.items(), sizes):
        tu.portions(tb, rid, toks, sz)
    core = _core(zk_folders[name], dtype, tb.live_tokens_peak)
    _check(tb, tu.run_in_process(core, tb), plain, dtype, f"{name} portions")


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", list(ZK_CONFIGS))
def test_mixed_batches_with_pages_and_slots_used_again(zk_folders, name, dtype, graphs):
    """Nine unequal requests through three slots: portions of some beside single tokens of
    others; every finished request's pages and slot go to the next one."""
    cfg, weights = read_folder(zk_folders[name])
    reqs = _requests(cfg, [40, 23, 77, 18, 52, 31, 66, 20, 45], 400)
    plain = _plain(cfg, weights, dtype, reqs)
    tb = tu.TraceBuilder()
    tu.mixed(tb, reqs, seed=7, max_live=3, decode_tail=10)
    core = _core(zk_folders[name], dtype, tb.live_tokens_peak, max_slots=3, graphs=graphs)
    _check(tb, tu.run_in_process(core, tb), plain, dtype, f"{name} mixed")
    assert core.cache.num_free_slots == 3 and all(p.num_used == 0 for p in core.cache.pools)


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("name", ["latent_only", "zk_a", "zk_b"])
def test_models_whose_portions_expand_their_latent_rows(zk_folders, name, graphs, monkeypatch):
    """Portions of 16 tokens and more by way of keys and values per head (no window, no sink, no
    gate; the queries are columns of wider rows), beside decoded tokens that attend the rows."""
    from helios_b200.csrc import ops

    made = []
    monkeypatch.setattr(ops, "LATENT_EXPAND", True)
    inner = ops.latent_attention_expanded
    monkeypatch.setattr(ops, "latent_attention_expanded", lambda *a, **kw: made.append(1) or inner(*a, **kw))
    cfg, weights = read_folder(zk_folders[name])
    reqs = _requests(cfg, [140, 23, 177, 18, 52, 131], 700)
    plain = _plain(cfg, weights, "bfloat16", reqs)
    tb = tu.TraceBuilder()
    tu.mixed(tb, reqs, seed=5, max_live=3, decode_tail=10, portion_choices=(2, 16, 40, 70))
    core = _core(zk_folders[name], "bfloat16", tb.live_tokens_peak, max_slots=3, graphs=graphs)
    _check(tb, tu.run_in_process(core, tb), plain, "bfloat16", f"{name} expanded")
    assert made


@pytest.mark.gpu
def test_a_batch_gives_each_request_what_it_gets_alone(zk_folders):
    """float32: the same rows bit for bit, alone or beside others, whatever the slots and pages."""
    from helios_b200.engine.batch import StepEntry

    cfg, _w = read_folder(zk_folders["zk_a"])
    reqs = _requests(cfg, [37, 5, 60], 500)
    core = _core(zk_folders["zk_a"], "float32", 512, max_slots=4)
    alone = {}
    for rid, toks in reqs.items():
        alone[rid] = core.step([StepEntry(rid, toks, range(len(toks)))]).clone()
        core.end(rid)
    core.step([StepEntry("other", random_tokens(cfg["vocab"], 21, 1), [0])])      # shifts slots and pages
    got = core.step([StepEntry(rid, toks, range(len(toks))) for rid, toks in reqs.items()])
    off = 0
    for rid, toks in reqs.items():
        assert torch.equal(got[off:off + len(toks)], alone[rid]), rid
        off += len(toks)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
def test_through_trace_run(zk_folders, dtype, tmp_path):
    cfg, weights = read_folder(zk_folders["zk_b"])
    reqs = _requests(cfg, [30, 47, 22, 39, 28], 600)
    plain = _plain(cfg, weights, dtype, reqs)
    tb = tu.TraceBuilder()
    tu.mixed(tb, reqs, seed=3, max_live=4, decode_tail=8)
    got = tu.run_trace_run(zk_folders["zk_b"], dtype, tb, tmp_path / "out", tb.live_tokens_peak, cfg["vocab"])
    _check(tb, got, plain, dtype, "zk_b trace_run")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", list(ZK_CONFIGS))
def test_greedy_generation_through_the_scheduler(zk_folders, name, dtype):
    from helios_b200 import LLM, SamplingParams

    cfg, weights = read_folder(zk_folders[name])
    w = _bf16(weights) if dtype == "bfloat16" else weights
    prompts = [random_tokens(cfg["vocab"], n, 40 + n) for n in (1, 5, 17, 33, 9, 26)]
    llm = LLM(str(zk_folders[name]), dtype=dtype, kv_cache_bytes=1 << 22, max_num_batched_tokens=24,
              max_num_seqs=4, max_model_len=256)
    outs = llm.generate(prompt_token_ids=prompts, sampling_params=SamplingParams(max_tokens=12))
    for prompt, out in zip(prompts, outs):
        assert out.completion_tokens == 12
        toks = list(prompt)
        for t in out.token_ids:
            logits = pz.forward_logits(cfg, w, toks)[-1]
            best = int(torch.argmax(logits))
            if t != best:
                assert dtype == "bfloat16", f"token {t} instead of {best} after {len(toks)} tokens"
                assert float(logits[best] - logits[t]) <= 0.03 * float(logits.abs().max())
            toks.append(t)


@pytest.mark.gpu
@pytest.mark.parametrize("dk,dv", [(4, 4), (24, 30), (32, 128), (36, 40), (64, 132), (100, 17), (128, 128), (130, 20), (256, 8)])
def test_delta_rule_a_token_a_step_is_the_walk_over_all_tokens_bit_for_bit(dk, dv):
    """float32: the kernel for steps of single tokens (values in whole 16-byte pieces; the walk
    otherwise) and the walk at both column widths leave the same outputs and states, and both are
    the plain scan's."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    dev, heads, n, S = "cuda", 2, 21, 3
    g = torch.Generator().manual_seed(dk + dv)
    C = heads * (2 * dk + dv)
    qkv, beta = torch.randn(S, n, C, generator=g), torch.randn(S, n, heads, generator=g) + 2
    a = torch.randn(S, n, heads * dk, generator=g) - 2
    a_log, dt_bias = torch.randn(heads, generator=g) * 0.3, torch.randn(heads * dk, generator=g) * 0.3
    stride = -(-heads * dk * dv // 4) * 4

    def run(rows, lens, state, slots):
        cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int().to(dev)
        ctx = SimpleNamespace(cu_tokens=cu, slots=torch.tensor(slots, dtype=torch.int32, device=dev), num_seqs=len(lens))
        return ops.delta_rule(ctx, rows(qkv), (0, heads * dk, 2 * heads * dk), rows(beta), rows(a), a_log.to(dev),
                              dt_bias.to(dev), state[:, :heads * dk * dv], heads, heads, dk, dv)

    whole = torch.zeros(S, stride, device=dev)
    want = run(lambda t: t.reshape(S * n, -1).to(dev), [n] * S, whole, [0, 1, 2]).view(S, n, -1)
    # many requests: the wide blocks (the same three again and again)
    many = torch.zeros(240, stride, device=dev)
    got = run(lambda t: t.repeat(80, 1, 1).reshape(240 * n, -1).to(dev), [n] * 240, many, list(range(240)))
    assert torch.equal(got.view(80, S, n, -1), want.expand(80, S, n, -1)) and torch.equal(many.view(80, S, -1), whole.expand(80, S, -1))
    # a token a step, other slots
    state = torch.zeros(4, stride, device=dev)
    for t in range(n):
        got = run(lambda x: x[:, t].contiguous().to(dev), [1] * S, state, [3, 0, 2])
        assert torch.equal(got, want[:, t])
    assert torch.equal(state[[3, 0, 2]], whole) and not state[1].any()
    for s in range(S):
        x = qkv[s].double()
        for h in range(heads):
            q, k = x[:, h * dk:(h + 1) * dk], x[:, (heads + h) * dk:(heads + h + 1) * dk]
            q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
            k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            v = x[:, 2 * heads * dk + h * dv:2 * heads * dk + (h + 1) * dv]
            gd = torch.exp(-torch.exp(a_log[h].double()) * torch.nn.functional.softplus(
                a[s, :, h * dk:(h + 1) * dk].double() + dt_bias[h * dk:(h + 1) * dk].double()))
            o = pz.delta_scan(q, k, v, torch.sigmoid(beta[s, :, h].double()), gd)
            assert (want[s, :, h * dv:(h + 1) * dv].cpu().double() - o).abs().max() < 2e-5


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[1], [16], [17], [15, 40, 1, 33], [20] * 60], ids=lambda x: f"{len(x)}x{x[0]}")
@pytest.mark.parametrize("dk,dv", [(4, 4), (64, 16), (65, 17), (100, 36), (128, 128)])
def test_delta_rule_by_chunks_of_tokens_is_the_plain_scan(dk, dv, lens, monkeypatch):
    """bfloat16: whole, short and ragged last chunks, blocks of one and of two column groups, slots in any
    order, a slot that nobody owns; a token that holds NaN reaches neither the tokens before it nor
    other requests."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    monkeypatch.setattr(ops, "DELTA_CHUNK_TOKENS", (0, 0, 0))
    monkeypatch.setattr(ops, "DELTA_CHUNK_MEAN", 0)
    dev, heads, kv_heads, S, T = "cuda", 4, 2, len(lens), sum(lens)
    g = torch.Generator().manual_seed(dk + dv + T)
    qkv = torch.randn(T, 2 * kv_heads * dk + heads * dv, generator=g).bfloat16()
    beta = (torch.randn(T, heads, generator=g) + 1).bfloat16()
    a = (torch.randn(T, heads * dk, generator=g) - 2).bfloat16()
    a_log, dt_bias = torch.randn(heads, generator=g) * 0.3, torch.randn(heads * dk, generator=g) * 0.3
    before = torch.randn(S + 1, heads * dk * dv, generator=g) * 0.3
    slots = list(range(S, 0, -1))
    ctx = SimpleNamespace(cu_tokens=torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int().to(dev),
                          slots=torch.tensor(slots, dtype=torch.int32, device=dev), num_seqs=S)

    def run(rows):
        state = before.to(dev)
        o = ops.delta_rule(ctx, rows.to(dev), (0, kv_heads * dk, 2 * kv_heads * dk), beta.to(dev), a.to(dev),
                           a_log.to(dev), dt_bias.to(dev), state, heads, kv_heads, dk, dv)
        return o.cpu(), state.cpu()

    got, state = run(qkv)
    assert torch.equal(state[0], before[0])
    x, at = qkv.double(), 0
    for s in range(S if S <= 4 else 2):
        r = slice(at, at + lens[s])
        for h in range(heads):
            kh = h // (heads // kv_heads)
            q, k = x[r, kh * dk:(kh + 1) * dk], x[r, (kv_heads + kh) * dk:(kv_heads + kh + 1) * dk]
            q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
            k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            v = x[r, 2 * kv_heads * dk + h * dv:2 * kv_heads * dk + (h + 1) * dv]
            gd = torch.exp(-torch.exp(a_log[h].double()) * torch.nn.functional.softplus(
                a[r, h * dk:(h + 1) * dk].double() + dt_bias[h * dk:(h + 1) * dk].double()))
            b = torch.sigmoid(beta[r, h].double())
            want = before[slots[s]].double().view(heads, dk, dv)[h].clone()
            for t in range(lens[s]):
                want = gd[t][:, None] * want
                want = want + k[t][:, None] * (b[t] * (v[t] - want.T @ k[t]))[None, :]
                o = want.T @ q[t]
                # 32-bit sums of dk values of about one: some dk / 2 roundings of 6e-8, most averaged out
                assert (got[at + t, h * dv:(h + 1) * dv].double() - o).abs().max() < 1e-5
            assert (state[slots[s]].double().view(heads, dk, dv)[h] - want).abs().max() < 1e-5
        at += lens[s]
    if lens[0] < 2:
        return
    bad = qkv.clone()
    bad[lens[0] - 1] = float("nan")
    o2, state2 = run(bad)
    assert torch.equal(o2[:lens[0] - 1], got[:lens[0] - 1]) and torch.equal(o2[lens[0]:], got[lens[0]:])
    assert o2[lens[0] - 1].isnan().all() and torch.equal(state2[:S], state[:S])


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[300, 0, 130, 17], [17, 64, 0, 65, 130, 300]], ids=["one_group", "two_groups"])
@pytest.mark.parametrize("dk,dv", [(64, 128), (40, 116), (128, 128), (100, 116)])
def test_delta_rule_by_chunks_walks_its_ring_of_chunks_around(dk, dv, lens, monkeypatch):
    """More chunks than stages, with blocks of one and of two column groups; requests without tokens; q, k, v, beta, a
    and the states as columns of wider rows, as a model passes them; the same bits twice."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    monkeypatch.setattr(ops, "DELTA_CHUNK_TOKENS", (0, 0, 0))
    monkeypatch.setattr(ops, "DELTA_CHUNK_MEAN", 0)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    dev, heads, S, T = "cuda", 4, len(lens), sum(lens)
    assert (S * heads * -(-dv // 16) <= 148) == (S == 4)
    g = torch.Generator(device=dev).manual_seed(dk + dv + S)
    r = lambda *s: torch.randn(*s, generator=g, device=dev)
    qkv = torch.nn.functional.silu(r(T, 24 + heads * (2 * dk + dv))).bfloat16()
    wide = (r(T, heads * dk + 40) - 1).bfloat16()
    beta, a = wide[:, 3:3 + heads], wide[:, 17:17 + heads * dk]
    a_log, dt_bias, rows = r(heads) * 0.3, r(heads * dk) * 0.3, r(S + 2, heads * dk * dv + 12) * 0.3
    slots = list(range(S, 0, -1))
    ctx = SimpleNamespace(cu_tokens=torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int().to(dev),
                          slots=torch.tensor(slots, dtype=torch.int32, device=dev), num_seqs=S)
    at = (8, 8 + heads * dk, 24 + 2 * heads * dk)

    def run():
        kept = rows.clone()
        return ops.delta_rule(ctx, qkv, at, beta, a, a_log, dt_bias, kept[:, :heads * dk * dv], heads, heads, dk, dv), kept

    (got, kept), again = run(), run()
    assert torch.equal(got, again[0]) and torch.equal(kept, again[1])
    idle = [0, S + 1] + [slots[i] for i in range(S) if lens[i] == 0]
    assert torch.equal(kept[idle], rows[idle]) and torch.equal(kept[:, heads * dk * dv:], rows[:, heads * dk * dv:])
    q, k, v = (qkv.double()[:, c:c + heads * n].view(T, heads, n) for c, n in zip(at, (dk, dk, dv)))
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    gd = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus(
        (a.double() + dt_bias.double()).view(T, heads, dk)))
    b, first = torch.sigmoid(beta.double()), 0
    for n, slot in zip(lens, slots):
        state, outs = rows[slot, :heads * dk * dv].double().view(heads, dk, dv), []
        for t in range(first, first + n):
            state = gd[t][:, :, None] * state
            u = b[t][:, None] * (v[t] - torch.einsum("hdc,hd->hc", state, k[t]))
            state = state + k[t][:, :, None] * u[:, None, :]
            outs.append(torch.einsum("hdc,hd->hc", state, q[t]).flatten())
        # relative 2-norms: some roundings of 2^-24 a token, which decays of 0.8 forget
        bound = 3e-7
        if n:
            o = torch.stack(outs)
            assert (got[first:first + n].double() - o).norm() < bound * o.norm()
        assert (kept[slot, :heads * dk * dv].double() - state.flatten()).norm() < bound * state.norm()
        first += n


@pytest.mark.parametrize("heads,dk,portions,takes", [
    (16, 128, [64], True), (16, 128, [63], False), (16, 128, [64, 40], True), (16, 128, [47] * 8, False),
    (16, 128, [64] + [24] * 7, False), (16, 128, [64] * 32, True), (16, 128, [1000] + [1] * 24, True),
    (16, 128, [300] + [1] * 24, False), (16, 129, [2048], False), (8, 64, [64] * 8, True), (8, 64, [64] * 32, False),
    (8, 64, [128] * 32, True), (8, 64, [1476] + [1] * 60, True), (16, 24, [64], False), (16, 24, [128] * 4, True),
    (16, 24, [2048] * 20, False), (16, 24, [1000] + [1] * 24, True)])
def test_which_portions_the_delta_rule_takes_by_chunks(heads, dk, portions, takes, monkeypatch):
    """Eagerly, and in a captured step, which knows only whether there is one long portion beside short ones."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops
    from helios_b200.engine.batch import long_class, one_long_portion

    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    T, S = sum(portions), len(portions)
    for dtype in (torch.bfloat16, torch.float32):
        ctx = SimpleNamespace(num_seqs=S, longest_portion=max(portions), one_long=one_long_portion(max(portions), T, S))
        assert ops.delta_rule_by_chunks(ctx, dtype, T, heads, dk, dk) == (takes and dtype == torch.bfloat16)
    known = long_class(max(portions), T, S)
    ctx = SimpleNamespace(num_seqs=S, longest_portion=known or -(-T // S), one_long=known > 0)
    assert ops.delta_rule_by_chunks(ctx, torch.bfloat16, T, heads, dk, dk) == (takes and portions != [64, 40])


def test_a_captured_step_of_one_long_portion_goes_by_chunks_whatever_its_padding(monkeypatch):
    """1,014 tokens beside ten of one, padded to 12 requests and 1,280 tokens."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops
    from helios_b200.engine.batch import long_class

    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    known = long_class(1014, 1024, 12)
    assert (known, long_class(1014, 1280, 12), long_class(64, 70, 3), long_class(40, 42, 3)) == (128, 0, 64, 0)
    ctx = SimpleNamespace(num_seqs=12, longest_portion=known, one_long=True)
    assert ops.delta_rule_by_chunks(ctx, torch.bfloat16, 1280, 8, 64, 64)


@pytest.mark.gpu
@pytest.mark.parametrize("portions", [[70, 1, 1, 1], [130, 1, 1, 1, 1], [24, 24, 24, 24]])
def test_captured_steps_take_the_delta_rule_as_the_same_steps_run_kernel_by_kernel(zk_folders, portions, monkeypatch):
    from helios_b200.csrc import ops
    from helios_b200.engine.batch import StepEntry

    rule, routes = ops.delta_rule_by_chunks, []
    monkeypatch.setattr(ops, "DELTA_CHUNK_TOKENS", (50, 50, 50))
    monkeypatch.setattr(ops, "DELTA_CHUNK_MEAN", 16)

    def noted(*args):
        routes.append(rule(*args))
        return routes[-1]

    monkeypatch.setattr(ops, "delta_rule_by_chunks", noted)
    core = _core(zk_folders["zk_a"], "bfloat16", 900, max_slots=6)
    for i in range(4):
        core.step([StepEntry((i, j), tuple(k % 20 for k in range(n)), (n - 1,)) for j, n in enumerate(portions)])
        for j in range(len(portions)):
            core.end((i, j))
    assert any(g.graph is not None for g in core._graphs.values())
    assert set(routes) == {portions[0] >= 70}


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [4.0, 0.0, -2.0, -10.0])
@pytest.mark.parametrize("dk,dv", [(64, 64), (128, 128)])
def test_delta_rule_by_chunks_is_as_near_to_64_bits_as_the_walk_by_tokens(dk, dv, shift, monkeypatch):
    """Decays from 0.02 to 0.9999 on average: outputs and states of a prompt, both ways, against the scan in 64
    bits."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    dev, heads, T = "cuda", 6, 300
    g = torch.Generator(device=dev).manual_seed(dk)
    r = lambda *s: torch.randn(*s, generator=g, device=dev)
    qkv = torch.nn.functional.silu(r(T, heads * (2 * dk + dv))).bfloat16()
    beta, a = (r(T, heads) + 1).bfloat16(), (r(T, heads * dk) + shift).bfloat16()
    a_log, dt_bias, before = r(heads) * 0.3, r(heads * dk) * 0.3, r(1, heads * dk * dv) * 0.3
    ctx = SimpleNamespace(cu_tokens=torch.tensor([0, T], dtype=torch.int32, device=dev),
                          slots=torch.zeros(1, dtype=torch.int32, device=dev), num_seqs=1)
    q, k, v = (x.view(T, heads, -1) for x in qkv.double().split([heads * dk, heads * dk, heads * dv], 1))
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    gd = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus(
        (a.double() + dt_bias.double()).view(T, heads, dk)))
    b, S, outs = torch.sigmoid(beta.double()), before.double().view(heads, dk, dv), []
    for t in range(T):
        S = gd[t][:, :, None] * S
        S = S + k[t][:, :, None] * (b[t][:, None] * (v[t] - torch.einsum("hdc,hd->hc", S, k[t])))[:, None, :]
        outs.append(torch.einsum("hdc,hd->hc", S, q[t]))
    want = torch.stack(outs).flatten(1), S.flatten()[None]

    def errors(limit):
        monkeypatch.setattr(ops, "DELTA_CHUNK_TOKENS", (limit,) * 3)
        state = before.clone()
        o = ops.delta_rule(ctx, qkv, (0, heads * dk, 2 * heads * dk), beta, a, a_log, dt_bias, state, heads, heads, dk, dv)
        return [float((x.double() - w).norm() / w.norm()) for x, w in zip((o, state), want)]

    for walk, chunks in zip(errors(T + 1), errors(0)):
        assert chunks <= walk
        # (a product that is left out shows at once: roundings of 2^-24, as many as a decay lets pile up)
        assert chunks < (2.5e-7 if shift > -3 else 3e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("y_dtype", DTYPES)
@pytest.mark.parametrize("H", [4, 37, 1020, 1024, 1028, 2052, 4100, 8192, 8196])
def test_norm_on_an_output_at_the_widths_its_rows_are_kept_at(H, y_dtype):
    """One to eight groups of four values a thread, and the widths that go value by value; with and
    without the copy, and the copy alone."""
    from helios_b200.csrc import ops

    g = torch.Generator().manual_seed(H)
    dt = torch.float32 if y_dtype == "float32" else torch.bfloat16
    res, w = torch.randn(5, H, generator=g), torch.rand(H, generator=g) + 0.5
    y = (torch.randn(5, H, generator=g) * 3).to(dt)
    yd = y.double()
    want = res.double() + yd / torch.sqrt((yd * yd).mean(-1, keepdim=True) + 1e-5) * w.double()
    r = res.cuda()
    copy = ops.rmsnorm_add(r, y.cuda(), w.cuda(), 1e-5, torch.bfloat16)
    # a sum of H squares, a root and two products: some H / 256 + 12 roundings, most of them averaged out
    torch.testing.assert_close(r.cpu().double(), want, atol=4e-6, rtol=4e-6)
    assert torch.equal(copy, r.to(torch.bfloat16))
    assert torch.equal(ops.rmsnorm_add(r, None, None, 0.0, torch.bfloat16), copy)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,rank,rot,count", [(16, 512, 64, 60), (11, 512, 64, 75), (1, 512, 96, 149), (16, 480, 112, 300)])
@pytest.mark.parametrize("window", [None, 40, 700])
def test_latent_attention_of_many_single_tokens_takes_sixteen_rows_a_block(heads, rank, rot, count, window):
    """Rows wide enough that 32 query rows fill an SM, more ranges than SMs: contexts at the edges of
    key tiles, one and more ranges a request, a window, a sink; against the kernel with a warp a row."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops
    from helios_b200.engine.batch import SeqSlice

    dev, page = "cuda", 16
    g = torch.Generator().manual_seed(heads + count)
    lens = [(1, 2, 31, 32, 33, 300, 1000)[i % 7] for i in range(count)]
    width, n_pages = 63, 200
    table = torch.stack([torch.randperm(n_pages, generator=g)[:width] for _ in lens]).int()
    pages = (torch.randn(n_pages, 1, page, rank + rot, generator=g) * 0.5).to(torch.bfloat16).to(dev)
    q = (torch.randn(count, heads, rank + rot, generator=g) * 0.7).to(torch.bfloat16).to(dev)
    sink = (torch.randn(heads, generator=g) * 2).to(dev) if window == 700 else None
    start = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=dev)
    ctx = SimpleNamespace(seq_of_token=torch.arange(count, dtype=torch.int32, device=dev), positions=start, start_pos=start,
                          cu_tokens=torch.arange(count + 1, dtype=torch.int32, device=dev), extras={}, num_seqs=count,
                          seqs=[SeqSlice(None, 0, n - 1, 1, i) for i, n in enumerate(lens)], max_context_len=1000)
    call = lambda: ops.latent_attention(ctx, q[:, :, :rank], q[:, :, rank:], pages, table.to(dev), rank, rot, page, 0.3,
                                        window, sink).float()
    got = call()
    ops.LATENT_ATTENTION_TENSOR_CORES = False
    try:
        want = call()
    finally:
        ops.LATENT_ATTENTION_TENSOR_CORES = True
    assert torch.isfinite(got).all()
    # weights and results have 8 bits: two results of at most about 1.5 in size, each within 2^-8 of it
    torch.testing.assert_close(got, want, atol=1.6e-2, rtol=1.6e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("dv,pad", [(4, 0), (30, 0), (128, 0), (128, 3), (128, 8), (132, 4), (260, 0)])
def test_gated_norm_in_pieces_and_value_by_value(dtype, dv, pad):
    """Value sizes and gate strides that are, and are not, whole pieces of four."""
    from helios_b200.csrc import ops

    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    g = torch.Generator().manual_seed(dv + pad)
    T, heads = 7, 3
    o, w = torch.randn(T, heads * dv, generator=g) * 2, torch.rand(dv, generator=g) + 0.5
    gate = torch.randn(T, heads * dv + pad, generator=g).to(dt)
    got = ops.gated_rmsnorm(o.cuda(), gate.cuda()[:, :heads * dv], w.cuda(), heads, dv, 1e-5)
    x = o.double().view(T, heads, dv)
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()
    want = (want.reshape(T, -1) * torch.sigmoid(gate.double()[:, :heads * dv]))
    tol = 2e-6 if dtype == "float32" else 2.0 ** -8      # some ten roundings of 24 bits; one of 8
    torch.testing.assert_close(got.double().cpu(), want, atol=tol * 0.5, rtol=tol)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("C,pad", [(4, 0), (36, 4), (36, 1), (37, 3), (1028, 0)])
def test_short_convolution_a_token_a_step_is_the_whole_sequence_bit_for_bit(dtype, taps, C, pad):
    """Single tokens of several requests in scattered slots (one launch where channels, rows and the
    slots' inputs are whole pieces, and 2 to 4 taps), with and without a bias, against the
    kernels for portions, and the inputs they leave."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    g = torch.Generator().manual_seed(C + taps)
    S, n = 3, 9
    x = torch.randn(S, n, C + pad, generator=g).to(dt)
    w, bias = torch.randn(C, taps, generator=g).cuda(), (torch.randn(C, generator=g).cuda() if pad else None)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")

    def run(rows, counts, state, slots):
        cu = [sum(counts[:i]) for i in range(len(counts) + 1)]
        ctx = SimpleNamespace(seq_of_token=ints([i for i, c in enumerate(counts) for _ in range(c)]), cu_tokens=ints(cu),
                              slots=ints(slots), num_seqs=len(counts))
        return ops.causal_conv_silu(ctx, rows.contiguous().cuda(), C, w, state, bias)

    first = torch.randn(5, C * (taps - 1), generator=g).cuda()
    whole, state = first.clone(), first.clone()
    want = run(x.reshape(S * n, -1), [n] * S, whole, [3, 0, 2]).view(S, n, C)
    for t in range(n):
        assert torch.equal(run(x[:, t], [1] * S, state, [3, 0, 2]), want[:, t])
    assert torch.equal(state, whole) and torch.equal(state[[1, 4]], first[[1, 4]])
    # as many tokens as requests, but not one each
    a, b = first.clone(), first.clone()
    got = run(x[0, :3], [0, 2, 1], a, [1, 4, 0])
    assert torch.equal(got[:2], run(x[0, :2], [2], b, [4])) and torch.equal(got[2:], run(x[0, 2:3], [1], b, [0]))
    assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,rank,rot,count", [(16, 512, 64, 200), (1, 512, 96, 170), (16, 480, 112, 333)])
@pytest.mark.parametrize("window", [None, 40, 700])
def test_latent_attention_with_sixteen_rows_a_block_at_every_window(heads, rank, rot, count, window):
    """As above, where the rule chooses the kernel for each window and with the sink."""
    from helios_b200.csrc import ops

    assert ops.latent_block_rows(count, True, heads, rank + rot, min(1000, window or 1000)) == 16
    test_latent_attention_of_many_single_tokens_takes_sixteen_rows_a_block(heads, rank, rot, count, window)


@pytest.mark.parametrize("tokens,single,heads,width,keys,rows", [
    (1, True, 16, 576, 131072, 32), (4, True, 16, 576, 20480, 32), (8, True, 16, 576, 5120, 32), (8, True, 16, 576, 6144, 16),
    (8, True, 16, 576, 32768, 16), (10, True, 16, 576, 4096, 16), (9, True, 16, 576, 4096, 32), (16, True, 16, 576, 2560, 16),
    (16, True, 16, 576, 2303, 32), (64, True, 16, 576, 1000, 16), (64, False, 16, 576, 1000, 32), (64, True, 17, 576, 1000, 32),
    (64, True, 16, 288, 1000, 32), (64, True, 16, 704, 1000, 32), (149, True, 1, 576, 1, 16), (148, True, 1, 576, 511, 32)])
def test_query_rows_a_block_of_latent_attention(tokens, single, heads, width, keys, rows, monkeypatch):
    """On 148 SMs: the edges of the ranges, of a quarter more for up to eight requests, and of what fits an SM."""
    from helios_b200.csrc import ops

    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    assert ops.latent_block_rows(tokens, single, heads, width, keys) == rows


@pytest.mark.gpu
@pytest.mark.parametrize("dk,dv", [(96, 32), (40, 36), (24, 64), (128, 68), (200, 64)])
def test_delta_rule_a_token_a_step_at_the_widths_of_its_blocks(dk, dv):
    """As above: values of exactly 32 and 64 columns a head, and of four more."""
    test_delta_rule_a_token_a_step_is_the_walk_over_all_tokens_bit_for_bit(dk, dv)


@pytest.mark.gpu
@pytest.mark.parametrize("dk,dv", [(24, 24), (64, 64), (128, 128), (200, 36)])
def test_delta_rule_of_as_many_tokens_as_requests_but_not_one_each(dk, dv):
    """The kernel for single tokens walks what a request has, and leaves a request without tokens alone."""
    from types import SimpleNamespace
    from helios_b200.csrc import ops

    dev, heads = "cuda", 2
    g = torch.Generator().manual_seed(dk)
    new = lambda *shape: torch.randn(*shape, generator=g).to(dev)
    qkv, beta, a = new(4, heads * (2 * dk + dv)), new(4, heads) + 2, new(4, heads * dk) - 2
    a_log, dt_bias, first = new(heads) * 0.3, new(heads * dk) * 0.3, new(5, heads * dk * dv)

    def run(t0, lens, state, slots):
        cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int().to(dev)
        ctx = SimpleNamespace(cu_tokens=cu, slots=torch.tensor(slots, dtype=torch.int32, device=dev), num_seqs=len(lens))
        part = slice(t0, t0 + sum(lens))
        return ops.delta_rule(ctx, qkv[part], (0, heads * dk, 2 * heads * dk), beta[part], a[part], a_log, dt_bias, state, heads,
                              heads, dk, dv)

    state, alone = first.clone(), first.clone()
    got = run(0, [0, 3, 0, 1], state, [1, 4, 2, 0])
    assert torch.equal(got[:3], run(0, [3], alone, [4])) and torch.equal(got[3:], run(3, [1], alone, [0]))
    assert torch.equal(state, alone)


@pytest.mark.gpu
@pytest.mark.parametrize("dk,dv", [(160, 36), (161, 4), (192, 30), (193, 16)])
def test_delta_rule_at_the_sizes_its_keys_are_padded_to(dk, dv):
    """As above, for keys of more than 128 values."""
    test_delta_rule_a_token_a_step_is_the_walk_over_all_tokens_bit_for_bit(dk, dv)
