"""The calls a host makes of this library, as timed cases: decode steps (one row to a few dozen, layer by layer
on the device or a whole stack from host buffers), prefill chunks, one layer from host buffers, and the
expert-parallel layer on one rank -- at the three model shapes the benchmark and the tests use.

A case names its entry point, its shape, its rows and layers, and the options of the configuration that
are used in earnest: activation and output types, fp16 or bf16 scales, fp32 or packed int8 router rows, a
skewed router. All experts are resident; every layer has weights, router and inputs of its own.
"""
from __future__ import annotations

import math
import random

import torch

from shrike_b200 import capi
from shrike_b200.ep import ExpertParallelLayer
from shrike_b200.moe import DecodeStack, ExpertCellArena, MoE, MoEConfig, RouterOperands, expert_offsets, round_up

# The layers of the benchmark's workloads: Qwen3.5-35B-A3B, gpt-oss-20B and Kimi-Linear-48B expert shapes.
SHAPES = {
    "qwen": dict(d=2048, f=512, num_experts=256, top_k=8, weight_bits=4, group_size=64, activation=capi.ACT_SILU,
                 has_shared=True, shared_gated=True, shared_f=512),
    "gptoss": dict(d=2880, f=2880, num_experts=32, top_k=4, weight_bits=4, group_size=32,
                   activation=capi.ACT_CLAMPED_SWIGLU, expert_bias=True),
    "kimi": dict(d=2304, f=1024, num_experts=256, top_k=8, weight_bits=8, group_size=64, activation=capi.ACT_SILU,
                 router_kind=capi.ROUTER_SIGMOID, routed_scaling=2.446, has_shared=True, shared_f=1024),
}
DTYPES = {"bf16": capi.DTYPE_BF16, "fp16": capi.DTYPE_FP16, "fp32": capi.DTYPE_FP32}
# the longest prefill chunk of each shape, and the most layers of a decode case
MOST_ROWS = {"qwen": 4096, "gptoss": 1024, "kimi": 2064}
MOST_LAYERS = {"qwen": 8, "gptoss": 4, "kimi": 2}


def case(name, entry, shape, rows, layers=1, act="bf16", out="fp32", meta="bf16", router_bits=0, skew=False):
    c = dict(entry=entry, shape=shape, rows=rows, layers=layers, act=act, out=out, meta=meta,
             router_bits=router_bits, skew=skew)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a decode step of a whole model for one sequence: host rows in, 40 layers, host rows out
        case("token through 40 layers", "stack", "qwen", 1, layers=40),
        # the smallest call: one MoE layer of one decode row, between the host's attention layers
        case("one layer, 1 row", "layer", "qwen", 1),
        # decode steps of a few concurrent sequences (or a speculative draft), device rows, layer after layer
        case("decode 4 rows", "layer", "qwen", 4, layers=8),
        case("decode 16 rows", "layer", "qwen", 16, layers=8),
        # a larger batch, an odd number of rows, on handles that serve prefill as well
        case("decode 37 rows", "layer", "qwen", 37, layers=4),
        # few large experts with biases: one row, and a full decode batch
        case("gpt-oss decode 1 row", "layer", "gptoss", 1, layers=4),
        case("gpt-oss decode 64 rows", "layer", "gptoss", 64, layers=4),
        # int8 experts, sigmoid router, fp16 host
        case("kimi decode 13 rows", "layer", "kimi", 13, layers=2, act="fp16", out="fp16", router_bits=8),
        # the prefill chunk of a long prompt with the skew that real routing has
        case("prefill 4096 rows", "prefill", "qwen", 4096, skew=True),
        # a prompt's ragged last chunk
        case("prefill 333 rows", "prefill", "qwen", 333, act="fp16", out="bf16", meta="fp16"),
        # a mixed batch (16 decode rows + a 2048-row chunk) through the expert-parallel layer of one rank
        case("expert-parallel 2064 rows", "ep", "kimi", 2064),
        # a prompt from host memory through one layer and back
        case("host prefill 777 rows", "host", "gptoss", 777, out="bf16"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng: random.Random):
    entry = rng.choice(["stack", "layer", "layer", "layer", "prefill", "prefill", "host", "ep"])
    shape = rng.choice(["qwen", "qwen", "gptoss", "kimi"])
    layers = 1
    if entry == "stack":
        rows, layers = _log_int(rng, 1, 16), _log_int(rng, 2, 2 * MOST_LAYERS[shape])
    elif entry == "layer":
        rows, layers = _log_int(rng, 1, 64), rng.randint(1, MOST_LAYERS[shape])
    elif entry == "prefill":
        rows = _log_int(rng, 65, MOST_ROWS[shape])
    else:
        rows = _log_int(rng, 1, min(2064, MOST_ROWS[shape]))
    act = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    # the host-buffer call hands y back in the activations' type
    out = act if entry == "host" else rng.choice(["fp32", "fp32", act])
    return case(None, entry, shape, rows, layers, act, out, rng.choice(["bf16", "fp16"]), rng.choice([0, 0, 8]),
                rng.random() < 0.5)


def _config(c) -> MoEConfig:
    rows = c["rows"]
    # decode handles of small batches are made for 16 rows, those of larger ones serve short prefills as well
    most = rows if c["entry"] in ("prefill", "ep") else 16 if rows <= 16 else max(128, rows)
    return MoEConfig(**SHAPES[c["shape"]], meta_dtype=DTYPES[c["meta"]], act_dtype=DTYPES[c["act"]],
                     y_dtype=DTYPES[c["out"]], router_weight_bits=c["router_bits"],
                     max_tokens=max(65, most) if c["entry"] in ("prefill", "ep") else most)


def _pack_int8(w: torch.Tensor):
    """Affine int8 rows with a bf16 scale and bias per 64 columns."""
    g = w.view(w.shape[0], -1, 64)
    lo, hi = g.amin(2), g.amax(2)
    scale, bias = ((hi - lo) / 255).bfloat16(), lo.bfloat16()
    q = ((g - bias.float()[..., None]) / scale.float()[..., None]).round().clamp(0, 255)
    return q.to(torch.uint8).view(w.shape).contiguous(), scale.contiguous(), bias.contiguous()


def _router(cfg: MoEConfig, c, gen) -> RouterOperands:
    ne, d = cfg.num_experts, cfg.d
    w = torch.randn((ne, d), generator=gen, device="cuda") * 0.02
    bias = None
    if c["skew"] and cfg.router_kind == capi.ROUTER_SOFTMAX:   # a Zipf(1.1) prior over the experts
        p = torch.arange(1, ne + 1, device="cuda", dtype=torch.float64) ** -1.1
        bias = (p / p.sum()).log()[torch.randperm(ne, generator=gen, device="cuda")].bfloat16()
    elif cfg.router_kind == capi.ROUTER_SIGMOID:               # the selection-only correction bias
        bias = ((torch.rand(ne, generator=gen, device="cuda") - 0.5) * (0.6 if c["skew"] else 0.2)).bfloat16()
    gate = torch.randn(d, generator=gen, device="cuda") * 0.02 if cfg.shared_gated else None
    scales = biases = None
    if cfg.router_weight_bits:
        w, scales, biases = _pack_int8(w)
    return RouterOperands(weights=w, scales=scales, biases=biases, logit_bias=bias, shared_gate=gate)


class State:
    """What the host keeps: handles, the pool with every layer's experts, routers, activation buffers."""

    def __init__(self):
        self.closers = []

    def __del__(self):
        torch.cuda.synchronize()
        for close in reversed(self.closers):
            close()


def _prepare_ep(s: State, c, cfg: MoEConfig, seed: int, gen) -> None:
    s.layer = ExpertParallelLayer(cfg, 0, 1, 0, c["rows"])
    s.closers.append(s.layer.close)
    s.layer.pool.fill_synthetic(0, s.layer.epr, seed, 0, first_expert=s.layer.lo)
    s.router = _router(cfg, c, gen)
    if cfg.has_shared:   # the shared expert's block sits in a pool cell of its own
        soff, sbytes = expert_offsets(cfg, shared=True)
        s.shared_pool = ExpertCellArena(s.layer.home, 1, round_up(sbytes, 256))
        s.closers.append(s.shared_pool.close)
        s.shared_pool.fill_synthetic(0, 1, seed, 0, first_expert=100000, shared=True)
        s.layer.set_shared(capi.SharedExpert(s.shared_pool.cell_address(0), soff))


def prepare(c, seed):
    cfg = _config(c)
    rows, n, entry = c["rows"], c["layers"], c["entry"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = State()
    s.entry = entry

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda").to(cfg.torch_act_dtype)

    if entry == "ep":
        _prepare_ep(s, c, cfg, seed, gen)
    else:
        ne = cfg.num_experts
        s.moes = [MoE(cfg) for _ in range(n)]
        s.closers += [m.close for m in s.moes]
        s.off, block = expert_offsets(cfg)
        soff, sblock = expert_offsets(cfg, shared=True) if cfg.has_shared else (None, 0)
        s.pool = ExpertCellArena(s.moes[0], n * (ne + 1), round_up(max(block, sblock), 256), chunks=min(n, 8))
        s.closers.append(s.pool.close)
        s.routers, s.shared = [], []
        for l, moe in enumerate(s.moes):
            s.pool.fill_synthetic(l * ne, ne, seed, l)
            moe.create_residency(1)
            moe.residency_set_layer_identity(0, l * ne)
            s.routers.append(_router(cfg, c, gen))
            s.shared.append(None)
            if cfg.has_shared:
                s.pool.fill_synthetic(n * ne + l, 1, seed, l, first_expert=100000, shared=True)
                s.shared[l] = capi.SharedExpert(s.pool.cell_address(n * ne + l), soff)
    k = cfg.top_k
    if entry == "stack":
        s.rows_in = rand(n + 1, rows, cfg.d).cpu().pin_memory()
        s.rows_out = torch.empty((rows, cfg.d), dtype=cfg.torch_act_dtype).pin_memory()
        s.stack = DecodeStack([(s.moes[l], s.pool, s.off, 0, s.routers[l], s.shared[l]) for l in range(n)], rows)
        s.closers.append(s.stack.close)
        return s
    if entry == "host":
        s.x = rand(rows, cfg.d).cpu().pin_memory()
        s.y = torch.empty((rows, cfg.d), dtype=cfg.torch_y_dtype).pin_memory()
        s.ids = torch.empty((rows, k), dtype=torch.int32).pin_memory()
        s.w = torch.empty((rows, k)).pin_memory()
        return s
    # a layer's input stands for what attention and normalisation made of the residual stream
    s.x = rand(n, rows, cfg.d)
    s.y = torch.empty((n, rows, cfg.d), dtype=cfg.torch_y_dtype, device="cuda")
    s.ids = torch.empty((n, rows, k), dtype=torch.int32, device="cuda")
    s.w = torch.empty((n, rows, k), device="cuda")
    s.slots = torch.empty((rows, k), dtype=torch.int32, device="cuda")
    s.gate = torch.empty(rows, device="cuda") if cfg.shared_gated else None
    s.step = list(zip(getattr(s, "moes", [None]), getattr(s, "routers", [None]), s.x, s.y,
                      getattr(s, "shared", [None]), s.ids, s.w))
    # the residual stream that every layer of a decode step adds to; a lone layer's host adds y itself
    s.rows = rand(rows, cfg.d) if n > 1 else None
    s.hidden = torch.empty_like(s.rows) if n > 1 else None
    return s


def run(s):
    if s.entry == "stack":
        s.stack.forward_host(s.rows_in, s.rows_out)
        return s.rows_out
    if s.entry == "host":
        s.moes[0].layer_forward_host(s.pool, s.off, 0, s.routers[0], s.x, s.y, s.shared[0], s.ids, s.w)
        return {"y": s.y, "ids": s.ids, "weights": s.w}
    if s.entry == "ep":
        s.layer.forward(s.router, s.x[0], s.y[0])
        return s.y
    if s.entry == "prefill":
        moe, router, x, y, shared, ids, w = s.step[0]
        moe.encode_router(router, x, ids, w, s.gate)
        moe.encode_residency_classification(ids, 0, s.slots)
        moe.encode_prefill(s.pool, s.off, ids, s.slots, w, x, y, None, shared, s.gate)
        return {"y": s.y, "ids": s.ids, "weights": s.w}
    if s.hidden is not None:   # the step's rows enter the residual stream
        s.hidden.copy_(s.rows)
    for moe, router, x, y, shared, ids, w in s.step:
        moe.encode_decode_layer(s.pool, s.off, 0, router, x, y, s.hidden, shared, ids, w)
    return {"y": s.y, "ids": s.ids, "weights": s.w, "hidden": s.hidden}


def work(c):
    cfg = _config(c)
    rows, ne, k, d = c["rows"], cfg.num_experts, cfg.top_k, cfg.d
    if c["skew"]:   # the share of rows that pick expert e, from the Zipf(1.1) prior
        p = [(e + 1) ** -1.1 for e in range(ne)]
        p = [min(1.0, k * v / sum(p)) for v in p]
    else:
        p = [k / ne] * ne
    experts = max(k, sum(1 - (1 - v) ** rows for v in p))
    blocks = experts * expert_offsets(cfg)[1] + (expert_offsets(cfg, shared=True)[1] if cfg.has_shared else 0)
    router = ne * d * (4 if not cfg.router_weight_bits else 1)
    esz = {"bf16": 2, "fp16": 2, "fp32": 4}
    io = rows * (d * (esz[c["act"]] + esz[c["out"]]) + k * 8)
    flops = rows * (6 * d * (k * cfg.f + cfg.shared_f) + 2 * ne * d)
    return {"bytes": c["layers"] * (blocks + router + io), "flops": c["layers"] * flops}


def tolerance(c):
    # a stack's layers feed each other through rows of the activations' type: one unit of those, and a near-tie
    # that turns
    if c["entry"] == "stack":
        return {"rel": 2e-3 if c["act"] == "fp32" else 1e-2, "max": 0.5}
    # operands and the activations between the projections are fp16 with fp32 sums; 16-bit outputs (the residual
    # stream among them) round once more. Picks and their weights are exact.
    half = c["out"] != "fp32" or (c["layers"] > 1 and c["act"] != "fp32")
    return {"rel": 4e-3 if half else 1e-3, "max": 0.05, "differ": 0.0}
