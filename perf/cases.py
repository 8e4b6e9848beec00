"""Workloads of this package as its users call it, with what each has to move and compute and what its results are in 64 bits.

Kinds of cases (a case is a dict of plain values, see `listed`):

  attn_decode   one decode step of the full-attention layers of a model: 8 query heads on 2 key/value heads of 256, 16-token
                pages, rotation of the first 64 dimensions, appended token, sigmoid gate.  form "fused": the engine's call with
                the head norms inside; "operators": the drop-in operators in the order a runner calls them.  The layers of a
                step are one CUDA graph over caches of their own, as a decode loop replays them.
  attn_prefill  the same layer over packed prompts of ragged lengths ("fused" with the cache written, or the bare operator).
  gdn_decode    one decode step of the Gated-DeltaNet layers (16 heads of 128 x 128 states in 32 bits), one CUDA graph;
                form "mixer": convolution, norms, gates, state and gated norm; "operator": the state update alone.
  gdn_prefill   the Gated-DeltaNet recurrence over packed prompts, or over one long prompt (form "single").
  model         a whole model with random weights: packed prefill of prompts, then greedy decode steps from a captured graph.

Lengths belong to the case, values to the seed.  Sizes are those of the configurations, tests and benchmark of this repository;
serving runs in bf16 (states and gates in 32 bits), so every case does.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "qwen3_5-triton-inference-engine_b200"))

DEV, BF, F32, F64 = "cuda", torch.bfloat16, torch.float32, torch.float64
HQ, HKV, D, ROT, THETA, PAGE, EPS = 8, 2, 256, 64, 1e7, 16, 1e-6
GH, GD = 16, 128                                     # Gated-DeltaNet heads and their size
QD, KVD, KD = HQ * D, HKV * D, GH * GD
VOCAB = {"Qwen3.5": 248320, "Tofilorn": 65536, "Dugilorn": 65536}


def listed() -> list[dict]:
    return [
        # one user, a short conversation: launches and latency are everything
        dict(name="attn_decode_1", kind="attn_decode", form="fused", layers=6, batch=1, low=512, high=4096),
        # the ordinary serving batch
        dict(name="attn_decode_32", kind="attn_decode", form="fused", layers=6, batch=32, low=512, high=4096),
        # a full box: one layer, the cache by far larger than any on-chip memory
        dict(name="attn_decode_256", kind="attn_decode", form="fused", layers=1, batch=256, low=512, high=4096),
        # newcomers of a batch: short ragged prompts
        dict(name="attn_prefill_ragged", kind="attn_prefill", form="fused", batch=32, low=16, high=512),
        # documents
        dict(name="attn_prefill_long", kind="attn_prefill", form="fused", batch=8, low=4096, high=4096),
        # the recurrent layers of the ordinary serving batch
        dict(name="gdn_decode_32", kind="gdn_decode", form="mixer", layers=18, batch=32),
        # recurrent layers over newcomers, and over one document
        dict(name="gdn_prefill_32", kind="gdn_prefill", form="packed", batch=32, low=128, high=128),
        dict(name="gdn_prefill_1", kind="gdn_prefill", form="packed", batch=1, low=2048, high=2048),
        # whole models: a batch of short prompts with short answers; one long prompt and the start of its answer
        dict(name="qwen_batch", kind="model", family="Qwen3.5", width=1024, batch=32, low=128, high=128, new=8),
        dict(name="qwen_long", kind="model", family="Qwen3.5", width=1024, batch=1, low=2048, high=2048, new=4),
        # the hybrid stacks: a few users with ragged prompts
        dict(name="tofilorn_ragged", kind="model", family="Tofilorn", width=1024, batch=8, low=256, high=1024, new=4),
        dict(name="dugilorn_ragged", kind="model", family="Dugilorn", width=1024, batch=8, low=256, high=1024, new=4),
    ]


def _spread(rng, low: int, high: int) -> int:
    """A whole number between low and high, evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng) -> dict:
    kind = rng.choice(["attn_decode", "attn_decode", "attn_prefill", "gdn_decode", "gdn_prefill", "gdn_prefill", "model", "model"])
    if kind == "attn_decode":
        batch = _spread(rng, 1, 256)
        low = _spread(rng, 16, max(32, min(32768, 600_000 // batch)))
        high = low if rng.random() < 0.3 else min(2 * low + rng.randrange(64), 32768)
        layers = 6 if batch * high <= 160_000 else 1
        return dict(kind=kind, form=rng.choice(["fused", "fused", "operators"]), layers=layers, batch=batch, low=low, high=high)
    if kind == "gdn_decode":
        batch = _spread(rng, 1, 256)
        return dict(kind=kind, form=rng.choice(["mixer", "mixer", "operator"]), layers=18 if batch <= 48 else 3, batch=batch)
    if kind == "model":
        batch = _spread(rng, 1, 32)
        high = _spread(rng, 8, max(16, min(4096, 4096 // batch)))
        low = high if rng.random() < 0.3 else max(1, high // rng.randint(2, 8))
        return dict(kind=kind, family=rng.choice(sorted(VOCAB)), width=rng.choice([1024, 1024, 2048]), batch=batch, low=low, high=high,
                    new=rng.randint(1, 4))
    batch = _spread(rng, 1, 64)
    high = _spread(rng, 16, min(8192, 32768 // batch))
    low = high if rng.random() < 0.3 else max(1, high // rng.randint(2, 8))
    if kind == "attn_prefill":
        return dict(kind=kind, form=rng.choice(["fused", "fused", "operators"]), batch=batch, low=low, high=high)
    if batch == 1 and rng.random() < 0.5:
        return dict(kind=kind, form="single", batch=1, low=high, high=high)
    return dict(kind=kind, form="packed", batch=batch, low=low, high=high)


# ------------------------------------------------------------------------------------------------------------- shared
def _lengths(case) -> list[int]:
    rs = np.random.RandomState((case["batch"] * 8191 + case["low"] * 131 + case["high"]) % 2**31)
    return rs.randint(case["low"], case["high"] + 1, case["batch"]).tolist()


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(gen, *shape, dtype=BF):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=dtype if dtype == F32 else BF).to(dtype)


def _inv_freq() -> torch.Tensor:
    return (1.0 / (THETA ** (torch.arange(0, ROT, 2, dtype=F32) / ROT))).to(DEV)


def _table(gen, lengths: list[int]) -> tuple[torch.Tensor, int]:
    """Page table [batch, most pages] over randomly placed pages, and the pages of the pool."""
    pages = [-(-n // PAGE) for n in lengths]
    perm = torch.randperm(sum(pages) + 8, generator=gen, device=DEV).to(torch.int32)
    table, at = torch.zeros(len(lengths), max(pages), dtype=torch.int32, device=DEV), 0
    for i, n in enumerate(pages):
        table[i, :n] = perm[at: at + n]
        at += n
    return table, perm.numel()


def _cumulative(lengths: list[int]) -> torch.Tensor:
    return torch.tensor([0, *np.cumsum(lengths).tolist()], dtype=torch.int32, device=DEV)


def _captured(calls):
    """A CUDA graph of `calls` and what they return (the kernels have run before: first calls set things up)."""
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = calls()
    return graph, out


# -------------------------------------------------------------------------------------------------------------- inputs
def _attn_decode_inputs(case, seed):
    gen, lengths = _generator(seed), _lengths(case)
    batch = case["batch"]
    layers = []
    for _ in range(case["layers"]):
        table, pages = _table(gen, [n + 1 for n in lengths])
        layers.append(dict(x=_randn(gen, batch, 2 * QD + 2 * KVD), table=table, k=_randn(gen, pages, HKV, PAGE, D),
                           v=_randn(gen, pages, HKV, PAGE, D), qn=_randn(gen, D) * 0.1, kn=_randn(gen, D) * 0.1))
    return lengths, layers


def _attn_prefill_inputs(case, seed):
    gen, lengths = _generator(seed), _lengths(case)
    table, pages = _table(gen, lengths)
    return lengths, table, pages, _randn(gen, sum(lengths), 2 * QD + 2 * KVD)


def _heads(x):
    """(q, gate, k, v) of rows [q | gate | k | v], as views."""
    n = x.shape[0]
    return (x[:, :QD].view(n, HQ, D), x[:, QD: 2 * QD], x[:, 2 * QD: 2 * QD + KVD].view(n, HKV, D), x[:, 2 * QD + KVD:].view(n, HKV, D))


def _gdn_decode_inputs(case, seed):
    gen, batch = _generator(seed), case["batch"]
    layers = []
    for _ in range(case["layers"]):
        x = _randn(gen, batch, 4 * KD + 2 * GH)
        layers.append(dict(x=x, conv=_randn(gen, batch, 4, 3 * KD), w4=_randn(gen, 4, 3 * KD), a_log=torch.rand(GH, generator=gen, device=DEV) * 2.7,
                           dt=_randn(gen, GH) * 0.02, norm=1.0 + 0.02 * _randn(gen, GD, dtype=F32),
                           state=_randn(gen, batch, GH, GD, GD, dtype=F32) * 0.1,
                           q=F.normalize(_randn(gen, batch, GH, GD, dtype=F32), dim=-1).mul(GD ** -0.5).to(BF),
                           k=F.normalize(_randn(gen, batch, GH, GD, dtype=F32), dim=-1).to(BF),
                           beta=torch.rand(batch, GH, generator=gen, device=DEV), g=-F.softplus(_randn(gen, batch, GH, dtype=F32))))
    return layers


def _gdn_prefill_inputs(case, seed):
    """What the convolution, the norms and the gates in front of the recurrence give: unit keys and queries, v a column range of
    the convolution's output, decays -softplus(N(0, 1)) exp(A) with A in [0, 2.7)."""
    gen, lengths = _generator(seed), _lengths(case)
    total = sum(lengths)
    q = F.normalize(_randn(gen, total, GH, GD, dtype=F32), dim=-1).mul_(GD ** -0.5).to(BF)
    k = F.normalize(_randn(gen, total, GH, GD, dtype=F32), dim=-1).to(BF)
    v = _randn(gen, total, 3 * KD)[:, 2 * KD:].view(total, GH, GD)
    beta = torch.sigmoid(_randn(gen, total, GH, dtype=F32))
    g = -F.softplus(_randn(gen, total, GH, dtype=F32)) * torch.exp(torch.rand(GH, generator=gen, device=DEV) * 2.7)
    return lengths, q, k, v, beta, g


def _config(case) -> dict:
    """Layer sizes of the stacks that the benchmark steps, at the two widths it uses."""
    width, family = case["width"], case["family"]
    count, heads, vocab = (24, 16, VOCAB[family]) if width == 1024 else (12, 32, 65536)
    ff = {"kind": "dense", "ff": 7 * width // 2}
    if family == "Qwen3.5":
        return dict(architecture=family, hidden=width, num_layers=count, num_q_heads=heads // 2, num_kv_heads=heads // 8, gdn_heads=heads,
                    intermediate=7 * width // 2, vocab=vocab)
    if family == "Tofilorn":
        latent = dict(type="latent_attention",
                      mixer=dict(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=512, q_rank=3 * width // 4, mask={"size": 4096}, scale=192 ** -0.5,
                                 rot=dict(base=1e6, dims=64, scaling=dict(factor=4.0, original=4096, fast=32.0, slow=1.0))))
        hgrn2 = dict(type="hgrn2", mixer=dict(heads=heads, dim=128, vdim=128))
        order = [hgrn2, dict(type="mingru", mixer=dict(width=2 * width)), hgrn2, latent]
        return dict(architecture=family, vocab=vocab, width=width, streams=2, norm={"eps": EPS}, layers=[{**order[i % 4], "mlp": ff} for i in range(count)])
    left = dict(heads=width // 128, kv_heads=width // 512, dim=128, vdim=128, mask={"size": 4096}, rot=dict(base=1e6, dims=128), scale=128 ** -0.5)
    right = dict(heads=width // 32, vdim=64, state=128, groups=1, conv=4, norm_groups=1)
    parallel = dict(type="parallel", mixer=dict(left=left, right=right, left_scale=0.7, right_scale=0.7))
    gla = dict(type="gla", mixer=dict(heads=width // 64, dim=128, vdim=128, tau=16.0))
    return dict(architecture=family, vocab=vocab, width=width, norm={"eps": EPS}, logit_softcap=30.0,
                layers=[{**(gla if i % 4 == 3 else parallel), "mlp": ff} for i in range(count)])


def _model_inputs(case, seed):
    """(prompts, configuration, weights).  Random weights; embedding rows as large against what the layers add as a
    trained model's residual, and a head that points the same way, so that greedy choices are decided and not left to rounding."""
    lengths, config = _lengths(case), _config(case)
    flat = torch.randint(0, config["vocab"], (sum(lengths),), generator=_generator(seed), device=DEV).tolist()
    at = np.cumsum([0, *lengths]).tolist()
    prompts = [flat[a:b] for a, b in zip(at, at[1:])]
    if case["family"] == "Qwen3.5":
        from b200attn import engine, models
        weights = engine.random_weights(models.family(config).config(config), seed, DEV)
        weights["embed"].mul_(200.0)
    else:
        from b200attn import hybrid
        weights = hybrid.random_tensors(hybrid.HybridWeights(hybrid.HybridConfig.from_config(config)), seed, DEV)
        weights["embed"], weights["head"] = weights["embed"] * 100.0, weights["embed"] * 20.0
    return prompts, config, weights


# ------------------------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    with torch.no_grad():
        return {"attn_decode": _prepare_attn_decode, "attn_prefill": _prepare_attn_prefill, "gdn_decode": _prepare_gdn_decode,
                "gdn_prefill": _prepare_gdn_prefill, "model": _prepare_model}[case["kind"]](case, seed)


def _prepare_attn_decode(case, seed):
    from b200attn import ops
    lengths, layers = _attn_decode_inputs(case, seed)
    batch, inv = case["batch"], _inv_freq()
    pos = torch.tensor(lengths, dtype=torch.int64, device=DEV)
    if case["form"] == "fused":
        ws = ops.fused_decode_workspace(DEV)

        def one(c):
            q, gate, k, v = _heads(c["x"])
            return ops.fused_decode_attention(q, k, v, gate, c["k"], c["v"], c["table"], pos, inv, ROT, ws, q_norm_weight=c["qn"],
                                              k_norm_weight=c["kn"], eps=EPS)
    else:
        scratch, ids = ops.allocate_split_scratch(HQ, D, batch=batch, device=DEV), pos.view(batch, 1)

        def one(c):
            q, gate, k, v = _heads(c["x"])
            q, k = (ops.partial_rope(t.unsqueeze(2), ids, inv, ROT)[:, :, 0] for t in (q, k))
            ctx = ops.call_paged_gqa_attention_decode_triton(q, k, v, c["k"], c["v"], c["table"], pos, scratch)
            return ops.attention_gate_pack(ctx.permute(1, 0, 2).unsqueeze(0), gate.view(batch, HQ, D).permute(1, 0, 2).unsqueeze(0))
    for c in layers:
        one(c)
    graph, out = _captured(lambda: [one(c) for c in layers])
    return dict(case=case, graph=graph, keep=(layers, pos, inv, one), out=dict(out=out, k=[c["k"] for c in layers], v=[c["v"] for c in layers]))


def _prepare_attn_prefill(case, seed):
    lengths, table, pages, x = _attn_prefill_inputs(case, seed)
    ids = torch.cat([torch.arange(n, dtype=torch.int32, device=DEV) for n in lengths])
    caches = [torch.zeros(pages, HKV, PAGE, D, dtype=BF, device=DEV) for _ in range(2)]
    return dict(case=case, x=x, table=table, ids=ids, cu=_cumulative(lengths), longest=max(lengths), caches=caches, inv=_inv_freq())


def _prepare_gdn_decode(case, seed):
    from b200attn import ops
    layers = _gdn_decode_inputs(case, seed)

    def one(c, conv, state):
        if case["form"] == "mixer":
            return ops.gdn_decode_fused(c["x"], conv, c["w4"], c["a_log"], c["dt"], c["norm"], state, GH)
        return ops.gdn_recurrent_decode(c["q"], c["k"], c["x"][:, :KD].view(-1, GH, GD), c["beta"], c["g"], state)
    one(layers[0], layers[0]["conv"].clone(), layers[0]["state"].clone())
    graph, out = _captured(lambda: [one(c, c["conv"], c["state"]) for c in layers])
    return dict(case=case, graph=graph, keep=(layers, one), out=dict(out=out, state=[c["state"] for c in layers], conv=[c["conv"] for c in layers]))


def _prepare_gdn_prefill(case, seed):
    lengths, q, k, v, beta, g = _gdn_prefill_inputs(case, seed)
    return dict(case=case, args=(q, k, v, beta, g), cu=_cumulative(lengths))


def _prepare_model(case, seed):
    from b200attn import models
    prompts, config, weights = _model_inputs(case, seed)
    room = max(map(len, prompts)) + case["new"] + 2
    family = models.family(config)
    cfg = family.config(config)
    if case["family"] == "Qwen3.5":
        engine = family.engine(cfg, weights, case["batch"], room, DEV)
    else:
        engine = family.engine(cfg, family.load(cfg, weights, BF, DEV), case["batch"], room, DEV, on_demand_pages=True)
    engine.prefill(prompts)
    if engine.pages is not None:
        for slot in range(case["batch"]):
            engine.pages.ensure(slot, room)
    engine.step()
    engine.capture()
    return dict(case=case, engine=engine, prompts=prompts)


# ----------------------------------------------------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    from b200attn import ops
    if case["kind"] == "gdn_prefill":
        if case["form"] == "single":
            return ops.call_gdn_recurrent_prefill_chunked_triton(*state["args"])
        return ops.gdn_chunked_prefill_packed(*state["args"], state["cu"])
    if case["kind"] == "attn_prefill":
        q, gate, k, v = _heads(state["x"])
        if case["form"] == "operators":
            return ops.gqa_attention_varlen_causal(q.contiguous(), k.contiguous(), v.contiguous(), state["cu"], state["longest"])
        out = ops.fused_prefill_attention(q, k, v, gate, *state["caches"], state["table"], state["cu"], state["ids"], state["inv"], ROT,
                                          state["longest"])
        return dict(out=out, k=state["caches"][0], v=state["caches"][1])
    engine, slots = state["engine"], list(range(case["batch"]))
    if case["family"] == "Qwen3.5":
        ids = [engine.prefill(state["prompts"])]
    else:       # portions into slots give the logits; the first choice is the caller's
        logits = engine.extend(slots, [0] * len(slots), state["prompts"])
        ids = [logits.argmax(-1)]
        engine.tok.copy_(ids[0])
    for _ in range(case["new"]):
        ids.append(engine.step().clone())
    out = dict(ids=torch.stack(ids))
    if case["family"] == "Qwen3.5":
        out |= dict(state=list(engine.rec_state.values()), conv=list(engine.conv_state.values()))
    else:
        out |= dict(logits=logits, state=[s["state"] for s in engine.states.values() if "state" in s])
    return out


# ---------------------------------------------------------------------------------------------------- work and tolerance
def work(case) -> dict:
    lengths, kind, b = ([0] * case["batch"] if case["kind"] == "gdn_decode" else _lengths(case)), case["kind"], case["batch"]
    total = sum(lengths)
    if kind == "attn_decode":
        nbytes = sum(2 * HKV * D * 2 * (n + 1) + 4 * -(-(n + 1) // PAGE) for n in lengths) + b * (3 * QD * 2 + 4 * KVD * 2 + 8)
        return dict(bytes=case["layers"] * nbytes, flops=case["layers"] * 4 * QD * sum(n + 1 for n in lengths))
    if kind == "attn_prefill":
        fused = case["form"] == "fused"
        return dict(bytes=total * (2 * QD * 2 + 2 * KVD * 2 + (QD * 2 + 2 * KVD * 2 if fused else 0)), flops=2 * QD * sum(n * (n + 1) for n in lengths))
    if kind == "gdn_decode":
        state, rows = 2 * GH * GD * GD * 4, 4 * KD * 2 + GH * 8
        if case["form"] == "mixer":
            rows = (4 * KD + 2 * GH + KD) * 2 + 2 * 4 * 3 * KD * 2
        return dict(bytes=case["layers"] * b * (state + rows), flops=case["layers"] * b * GH * 7 * GD * GD)
    if kind == "gdn_prefill":
        return dict(bytes=total * GH * (4 * GD * 2 + 8) + b * GH * GD * GD * 4, flops=total * GH * 6 * GD * GD)
    c = _config(case)
    width, vocab, count = case["width"], c["vocab"], 24 if case["width"] == 1024 else 12
    heads, ff = (16 if width == 1024 else 32), 3 * width * (7 * width // 2)
    if case["family"] == "Qwen3.5":       # three Gated-DeltaNet layers and one attention layer in turn
        mix = (3 * (5 * heads * 128 * width) + width * (3 * heads * 128 + heads // 4 * 256)) / 4
    elif case["family"] == "Tofilorn":    # two HGRN2, one minGRU, one latent
        latent = width * (3 * width // 4 + 576) + 3 * width // 4 * heads * 192 + 512 * heads * 256 + heads * 128 * width
        mix = (2 * 4 * heads * 128 * width + 8 * width * width + latent) / 4
    else:                                 # three of attention beside state space, one of gated linear attention
        mix = (3 * (width * (3 * width + width // 2) + width * (6 * width + 256 + width // 32)) + 5 * 2 * width * width) / 4
    per_token = count * (mix + ff)
    states = count * 3 / 4 * b * heads * GD * GD * 4 * 2
    steps = case["new"]
    pairs = sum(n * (n + 1) / 2 for n in lengths) * count / 4 * (1 if case["family"] != "Dugilorn" else 3)
    return dict(bytes=(1 + steps) * (per_token + vocab * width) * 2 + (0.5 + steps) * states,
                flops=2 * per_token * (total + b * steps) + 2 * vocab * width * b * (steps + 1) + pairs * 4 * heads * 128)


def tolerance(case):
    """About four times what a pass is off from `exact` (kernels: the rounding of bf16 outputs; models: roundings that add up
    over the layers)."""
    if case["kind"] == "model":
        return {"rel": 0.03, "max": 0.99, "differ": 0.0}
    if case["kind"] in ("attn_decode", "attn_prefill"):
        return {"rel": 1e-2, "max": 0.3}
    return {"rel": 7e-3, "max": 0.2}


# --------------------------------------------------------------------------------------------------- results in 64 bits
def exact(case, seed):
    with torch.no_grad():
        return {"attn_decode": _exact_attn_decode, "attn_prefill": _exact_attn_prefill, "gdn_decode": _exact_gdn_decode,
                "gdn_prefill": _exact_gdn_prefill, "model": _exact_model}[case["kind"]](case, seed)


def _rms(x, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, pos, freqs, interleaved=False, amplitude=1.0):
    """x [..., heads, size], pos over its leading dimensions: the first 2 len(freqs) entries rotated, as halves or as neighbours."""
    n = freqs.numel()
    angle = pos.double().unsqueeze(-1) * freqs.double()
    cos, sin = (angle.cos() * amplitude).unsqueeze(-2), (angle.sin() * amplitude).unsqueeze(-2)
    u, v = (x[..., 0: 2 * n: 2], x[..., 1: 2 * n: 2]) if interleaved else (x[..., :n], x[..., n: 2 * n])
    a, b = u * cos - v * sin, v * cos + u * sin
    turned = torch.stack((a, b), -1).flatten(-2) if interleaved else torch.cat((a, b), -1)
    return torch.cat((turned, x[..., 2 * n:]), -1)


def _attend(q, k, v, scale):
    """Causal attention of one sequence, q [T, heads, size], k and v [T, kv heads, size]: one group of heads at a time."""
    T, group = q.shape[0], q.shape[1] // k.shape[1]
    hidden = torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1)
    out = []
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // group].T).mul_(scale).masked_fill_(hidden, float("-inf"))
        out.append(torch.softmax(s, -1) @ v[:, h // group])
    return torch.stack(out, 1)


def _delta_rule(q, k, v, beta, g, state):
    """S <- e^g S, S <- S + k (beta (v - k^T S))^T, o = S^T q, token by token; [batch, T, heads, ...], state changed in place."""
    out, keep = torch.empty_like(v), g.exp()
    for t in range(q.shape[1]):
        state *= keep[:, t, :, None, None]
        kt = k[:, t].unsqueeze(-2)
        delta = (v[:, t].unsqueeze(-2) - kt @ state) * beta[:, t, :, None, None]
        state += kt.transpose(-1, -2) @ delta
        out[:, t] = (q[:, t].unsqueeze(-2) @ state).squeeze(-2)
    return out


def _padded(x, lengths):
    """Packed rows -> [batch, longest, ...] with zeros behind every sequence."""
    return torch.nn.utils.rnn.pad_sequence(list(x.split(lengths)), batch_first=True)


def _unpadded(x, lengths):
    return torch.cat([x[i, :n] for i, n in enumerate(lengths)])


def _exact_attn_decode(case, seed):
    lengths, layers = _attn_decode_inputs(case, seed)
    pos, freqs, outs, ks, vs = torch.tensor(lengths, device=DEV), _inv_freq(), [], [], []
    row, place, at = torch.arange(case["batch"], device=DEV), pos % PAGE, pos // PAGE
    for c in layers:
        q, gate, k, v = (t.double() for t in _heads(c["x"]))
        if case["form"] == "fused":
            q, k = _rms(q) * (1 + c["qn"].double()), _rms(k) * (1 + c["kn"].double())
        q, k = _rotate(q, pos, freqs), _rotate(k, pos, freqs)
        kc, vc = c["k"].double(), c["v"].double()
        kc[c["table"][row, at].long(), :, place], vc[c["table"][row, at].long(), :, place] = k, v
        out = []
        for i, n in enumerate(lengths):
            pages = c["table"][i, : n // PAGE + 1].long()
            kk, vv = (t[pages].transpose(0, 1).flatten(1, 2)[:, : n + 1] for t in (kc, vc))
            s = torch.softmax(q[i].view(HKV, HQ // HKV, D) @ kk.transpose(1, 2) / 16, -1)
            out.append((s @ vv).flatten())
        outs.append(torch.stack(out) * gate.sigmoid())
        ks.append(kc)
        vs.append(vc)
    return dict(out=outs, k=ks, v=vs)


def _exact_attn_prefill(case, seed):
    lengths, table, pages, x = _attn_prefill_inputs(case, seed)
    q, gate, k, v = (t.double() for t in _heads(x))
    if case["form"] == "operators":
        return torch.cat([_attend(a, b, c, D ** -0.5) for a, b, c in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
    ids = torch.cat([torch.arange(n, device=DEV) for n in lengths])
    q, k = _rotate(q, ids, _inv_freq()), _rotate(k, ids, _inv_freq())
    out = torch.cat([_attend(a, b, c, D ** -0.5) for a, b, c in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
    owner = torch.repeat_interleave(torch.arange(len(lengths), device=DEV), torch.tensor(lengths, device=DEV))
    page = table[owner, ids // PAGE].long()
    caches = [torch.zeros(pages, HKV, PAGE, D, dtype=F64, device=DEV) for _ in range(2)]
    caches[0][page, :, ids % PAGE], caches[1][page, :, ids % PAGE] = k, v
    return dict(out=out.flatten(1) * gate.sigmoid(), k=caches[0], v=caches[1])


def _gates(qkv, a, b, a_log, dt):
    """Convolved rows [..., q | k | v] and gate inputs -> what the delta rule takes."""
    q, k, v = (t.unflatten(-1, (-1, GD)) for t in qkv.chunk(3, -1))
    q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * GD ** -0.5
    k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    return q, k, v, b.sigmoid(), -a_log.exp() * F.softplus(a + dt)


def _exact_gdn_decode(case, seed):
    outs, states, convs = [], [], []
    for c in _gdn_decode_inputs(case, seed):
        x, state, conv = c["x"].double(), c["state"].double(), c["conv"].double()
        if case["form"] == "mixer":
            qkv, z, a, b = x.split([3 * KD, KD, GH, GH], -1)
            conv = torch.cat((conv[:, 1:], qkv.unsqueeze(1)), 1)
            args = _gates(F.silu((conv * c["w4"].double()).sum(1)), a, b, c["a_log"].double(), c["dt"].double())
        else:
            args = c["q"].double(), c["k"].double(), x[:, :KD].view(-1, GH, GD), c["beta"].double(), c["g"].double()
        out = _delta_rule(*(t.unsqueeze(1) for t in args), state)[:, 0]
        if case["form"] == "mixer":
            out = (_rms(out) * c["norm"].double()).flatten(1) * F.silu(z)
        outs.append(out)
        states.append(state)
        convs.append(conv)
    return dict(out=outs, state=states, conv=convs)


def _exact_gdn_prefill(case, seed):
    lengths, *args = _gdn_prefill_inputs(case, seed)
    state = torch.zeros(case["batch"], GH, GD, GD, dtype=F64, device=DEV)
    out = _unpadded(_delta_rule(*(_padded(t.double(), lengths) for t in args), state), lengths)
    return out, state[0] if case["form"] == "single" else state


def _exact_model(case, seed):
    """The prompts with a continuation in one causal pass: the continuation is right when it is what the pass itself chooses."""
    prompts, config, weights = _model_inputs(case, seed)
    lengths, new = [len(p) for p in prompts], case["new"]
    forward = {"Qwen3.5": _qwen, "Tofilorn": _tofilorn, "Dugilorn": _dugilorn}[case["family"]]
    guess = [p[-1:] * new for p in prompts]
    full = [n + new for n in lengths]
    rows = torch.tensor([[n - 1 + j for j in range(new + 1)] for n in lengths], device=DEV)
    for _ in range(new + 1):
        tokens = _padded(torch.tensor(sum((p + t for p, t in zip(prompts, guess)), []), device=DEV), full)
        h, more = forward(config, weights, tokens, full)
        h = h.gather(1, rows[..., None].expand(-1, -1, h.shape[-1]))
        head = weights.get("head", weights["embed"]).double()
        logits = h @ head.T
        ids = logits.argmax(-1)
        if ids[:, :new].tolist() == guess:
            break
        guess = ids[:, :new].tolist()
    if case["family"] == "Qwen3.5":
        return dict(ids=ids.T.contiguous(), **more)
    cap = config.get("logit_softcap")
    return dict(ids=ids.T.contiguous(), logits=cap * torch.tanh(logits[:, 0] / cap) if cap else logits[:, 0], **more)


def _conv(x, taps):
    """Causal depthwise convolution, x [batch, T, channels], taps [channels, K] with the newest token's last."""
    return sum(F.pad(x, (0, 0, j, 0))[:, : x.shape[1]] * taps[:, -1 - j] for j in range(taps.shape[1]))


def _live(tokens, lengths):
    """Which rows of padded sequences are tokens."""
    return torch.arange(tokens.shape[1], device=DEV) < torch.tensor(lengths, device=DEV)[:, None]


def _attend_all(q, k, v, scale):
    return torch.stack([_attend(a, b, c, scale) for a, b, c in zip(q, k, v)])


def _qwen(config, w, tokens, lengths):
    width, T = config["hidden"], tokens.shape[1]
    heads, nq, nkv = config["gdn_heads"], config["num_q_heads"], config["num_kv_heads"]
    live, x, at = _live(tokens, lengths), w["embed"].double()[tokens], torch.arange(T, device=DEV)
    freqs, states, convs = _inv_freq(), [], []
    last = torch.tensor([[n - 4 + j for j in range(4)] for n in lengths], device=DEV)
    for layer in w["layers"]:
        p = {n: t.double() for n, t in layer.items() if isinstance(t, torch.Tensor)}
        h = _rms(x) * (1 + p["ln1"])
        if layer["kind"] == "gdn":
            kd = heads * GD
            qkv, z, a, b = (h @ p["in_proj"].T).split([3 * kd, kd, heads, heads], -1)
            q, k, v, beta, g = _gates(F.silu(_conv(qkv, p["conv"])), a, b, p["a_log"], p["dt_bias"])
            state = torch.zeros(len(lengths), heads, GD, GD, dtype=F64, device=DEV)
            core = _delta_rule(q, k, v, beta * live[..., None], g * live[..., None], state)
            mixed = ((_rms(core) * p["norm"]).flatten(2) * F.silu(z)) @ p["out_proj"].T
            states.append(state)
            convs.append(torch.where((last >= 0)[..., None], qkv.gather(1, last.clamp(min=0)[..., None].expand(-1, -1, 3 * kd)), 0.0))
        else:
            q, gate, k, v = (h @ p["qkvg"].T).split([nq * D, nq * D, nkv * D, nkv * D], -1)
            q, k, v = (t.unflatten(-1, (-1, D)) for t in (q, k, v))
            q, k = (_rotate(_rms(t) * (1 + n), at, freqs) for t, n in ((q, p["q_norm"]), (k, p["k_norm"])))
            mixed = (_attend_all(q, k, v, D ** -0.5).flatten(2) * gate.sigmoid()) @ p["o_proj"].T
        x = x + mixed
        gate, up = ((_rms(x) * (1 + p["ln2"])) @ p["gate_up"].T).chunk(2, -1)
        x = x + (F.silu(gate) * up) @ p["down"].T
    return _rms(x) * (1 + w["norm"].double()), dict(state=states, conv=convs)


def _outer_recurrence(q, keep, k, v, live, states):
    """S <- keep S + k v^T, o = S^T q; q, k [batch, T, heads, size], keep the same or with one entry per head.  Rows that are no
    tokens leave S as it is; the last S goes to `states`."""
    state, out, live = torch.zeros(*k[:, 0].shape, v.shape[-1], dtype=F64, device=DEV), torch.empty_like(v), live[..., None, None]
    keep, k = torch.where(live, keep, 1.0), k * live
    for t in range(q.shape[1]):
        state = keep[:, t].unsqueeze(-1) * state + k[:, t].unsqueeze(-1) * v[:, t].unsqueeze(-2)
        out[:, t] = (q[:, t].unsqueeze(-2) @ state).squeeze(-2)
    states.append(state)
    return out


def _yarn(rot):
    """Frequencies and amplitude of a scaled rotation."""
    i = torch.arange(rot["dims"] // 2, dtype=F64, device=DEV)
    f, s = float(rot["base"]) ** (-2 * i / rot["dims"]), rot.get("scaling")
    if s is None:
        return f, 1.0

    def turns(t):
        return rot["dims"] * math.log(s["original"] / (2 * math.pi * t)) / (2 * math.log(rot["base"]))
    low, high = max(math.floor(turns(s["fast"])), 0), min(math.ceil(turns(s["slow"])), rot["dims"] - 1)
    ramp = ((i - low) / max(high - low, 0.001)).clamp(0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1


def _tofilorn(config, w, tokens, lengths):
    x = w["embed"].double()[tokens]
    streams, at = x.unsqueeze(0).repeat(config["streams"], 1, 1, 1), torch.arange(tokens.shape[1], device=DEV)
    live, states = _live(tokens, lengths), []

    def joined(streams, pre, part, sublayer):
        hc = {n: w[f"{pre}hc{part}.{n}"].double() for n in ("in", "out", "mix")}
        h = _rms(torch.einsum("s,sbtw->btw", hc["in"], streams)) * w[f"{pre}norm{part}"].double()
        return torch.einsum("st,sbnw->tbnw", hc["mix"], streams) + hc["out"][:, None, None, None] * sublayer(h)

    for i, layer in enumerate(config["layers"]):
        pre, m = f"l{i}.", layer["mixer"]
        p = {n[len(pre) + 4:]: t.double() for n, t in w.items() if n.startswith(pre + "mix.")}

        def mixer(h):
            if layer["type"] == "mingru":
                z, u = (h @ p["z"].T + p["z.b"]).sigmoid(), h @ p["x"].T + p["x.b"]
                candidate, s, out = torch.where(u >= 0, u + 0.5, u.sigmoid()), torch.zeros_like(u[:, 0]), torch.empty_like(u)
                kept = z * live[..., None]
                for t in range(u.shape[1]):
                    s = (1 - kept[:, t]) * s + kept[:, t] * candidate[:, t]
                    out[:, t] = s
                states.append(s)
                return (out * F.silu(h @ p["g"].T)) @ p["o"].T
            if layer["type"] == "hgrn2":
                q, v = (t.unflatten(-1, (m["heads"], -1)) for t in (F.silu(h @ p["q"].T), h @ p["v"].T))
                f = (p["lower"] + (1 - p["lower"]) * (h @ p["f"].T + p["f.b"]).sigmoid()).unflatten(-1, (m["heads"], -1))
                return (_rms(_outer_recurrence(q, f, 1 - f, v, live, states)) * p["norm"]).flatten(2) @ p["o"].T
            freqs, amplitude = _yarn(m["rot"])
            q = ((_rms(h @ p["dq"].T) * p["dq.norm"]) @ p["uq"].T).unflatten(-1, (m["heads"], -1))
            q = torch.cat((q[..., : m["dim"]], _rotate(q[..., m["dim"]:], at, freqs, True, amplitude)), -1)
            c, turned = (h @ p["dkv"].T).split([m["kv_rank"], m["rot_dim"]], -1)
            c, turned = _rms(c) * p["dkv.norm"], _rotate(turned.unsqueeze(2), at, freqs, True, amplitude)
            k = torch.cat(((c @ p["uk"].T).unflatten(-1, (m["heads"], -1)), turned.expand(-1, -1, m["heads"], -1)), -1)
            return _attend_all(q, k, (c @ p["uv"].T).unflatten(-1, (m["heads"], -1)), m["scale"]).flatten(2) @ p["o"].T
        streams = joined(streams, pre, 1, mixer)
        g = {n: w[f"{pre}mlp.{n}"].double() for n in ("gate", "up", "down")}
        streams = joined(streams, pre, 2, lambda h: (F.silu(h @ g["gate"].T) * (h @ g["up"].T)) @ g["down"].T)
    return _rms(streams.sum(0)) * w["final.norm"].double(), dict(state=states)


def _dugilorn(config, w, tokens, lengths):
    x, at = w["embed"].double()[tokens], torch.arange(tokens.shape[1], device=DEV)
    live, states = _live(tokens, lengths), []
    for i, layer in enumerate(config["layers"]):
        pre = f"l{i}."
        p = {n[len(pre):]: t.double() for n, t in w.items() if n.startswith(pre)}
        h, m = _rms(x) * p["norm1"], layer["mixer"]
        if layer["type"] == "gla":
            q, k, v = ((h @ p["mix." + n].T).unflatten(-1, (m["heads"], -1)) for n in "qkv")
            keep = torch.exp(-F.softplus(-((h @ p["mix.a1"].T) @ p["mix.a2"].T + p["mix.a2.b"])) / m["tau"]).unflatten(-1, (m["heads"], -1))
            o = _rms(_outer_recurrence(q * m["dim"] ** -0.5, keep, k, v, live, states)) * p["mix.norm"]
            y = (o.flatten(2) * F.silu(h @ p["mix.g"].T)) @ p["mix.o"].T
        else:
            a, s, left, right = m["left"], m["right"], "mix.left.", "mix.right."
            q, k, v = ((h @ p[left + n].T + p[left + n + ".b"]).unflatten(-1, (-1, 128)) for n in "qkv")
            freqs, _ = _yarn(a["rot"])
            o = _attend_all(_rotate(q, at, freqs), _rotate(k, at, freqs), v, a["scale"]).flatten(2)
            y = m["left_scale"] * ((o * (h @ p[left + "g"].T).sigmoid()) @ p[left + "o"].T)
            inner, bc = s["heads"] * s["vdim"], s["groups"] * s["state"]
            z, xbc, dt = (h @ p[right + "in"].T).split([inner, inner + 2 * bc, s["heads"]], -1)
            xs, B, C = F.silu(_conv(xbc, p[right + "conv"]) + p[right + "conv.b"]).split([inner, bc, bc], -1)
            xs, B, C = (t.unflatten(-1, (n, -1)) for t, n in ((xs, s["heads"]), (B, s["groups"]), (C, s["groups"])))
            B, C = (t.repeat_interleave(s["heads"] // s["groups"], 2) for t in (B, C))
            dt = F.softplus(dt + p[right + "dt_bias"])[..., None]
            o = _outer_recurrence(C, torch.exp(-p[right + "A_log"].exp()[:, None] * dt), B * dt, xs, live, states) + p[right + "D"][:, None] * xs
            o = _rms((o.flatten(2) * F.silu(z)).unflatten(-1, (s["norm_groups"], -1))).flatten(2) * p[right + "norm"]
            y = y + m["right_scale"] * (o @ p[right + "o"].T)
        x = x + y + (F.gelu(h @ p["mlp.gate"].T, approximate="tanh") * (h @ p["mlp.up"].T)) @ p["mlp.down"].T
    return _rms(x) * w["final.norm"].double(), dict(state=states)
