"""The streaming expert kernel at the edges of its tiling, against the oracle: rows of weights that end inside a
128-byte piece, group counts that leave a quad of groups open, shared and routed experts of different widths, one to
eight rows per instance, and the shapes it leaves to the per-tile kernels (an odd number of groups)."""
import numpy as np
import pytest
import torch

from shrike_b200 import capi
from gpu_harness import Layer, inputs, rel_l2, small_config, to_act_tensor
from test_gpu_parity import TOL, check_layer, test_fused_decode_layer_equals_the_separate_calls as equals_the_separate_calls

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [9, 17, 64])
@pytest.mark.parametrize("kw", [
    dict(d=256, f=128, shared_f=384),                                    # whole pieces
    dict(d=384, f=640, shared_f=128),                                    # a piece of two groups at the end
    dict(d=320, f=192, shared_f=192),                                    # odd numbers of groups: the per-tile kernels
    dict(d=128, f=128, has_shared=0, shared_gated=0, num_experts=4, top_k=2),   # many instances of the same experts
    dict(d=1216, f=1344, shared_f=2880, group_size=32),                  # two and four warps to a row, some from the middle of a piece
    dict(d=384, f=192, shared_f=320, group_size=32, weight_bits=4, meta_dtype=capi.DTYPE_FP16),
    dict(d=128, f=384, shared_f=128, group_size=64, weight_bits=8),
    dict(d=192, f=320, shared_f=64, group_size=32, weight_bits=8, expert_bias=1, activation=capi.ACT_GELU_TANH),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_stream_edges(cuda_device, kw, T):
    """The layer call, and the projections as calls of their own behind the plan and behind the route kernel."""
    layer = Layer(small_config(**kw))
    x = inputs(T, kw["d"], seed=T)
    check_layer(layer, x, fused=True)
    check_layer(layer, x)
    y, ids, w, hidden = by_separate_calls(layer, x)
    ids_ref, w_ref, _ = layer.oracle_route(x)
    assert (ids == ids_ref).all() and (w == w_ref).all()
    assert rel_l2(y, layer.oracle_forward(x, ids_ref, w_ref)) <= TOL
    assert np.abs(hidden - (x + y)).max() <= 1e-5 * np.abs(x).max()
    layer.close()


def by_separate_calls(layer: Layer, x: np.ndarray):
    cfg, T = layer.cfg, len(x)
    x_dev = to_act_tensor(x, cfg.act_dtype, layer.device)
    y, hidden = torch.empty_like(x_dev), x_dev.clone()
    ids = torch.empty((T, cfg.top_k), dtype=torch.int32, device=layer.device)
    w = torch.empty((T, cfg.top_k), dtype=torch.float32, device=layer.device)
    gate = torch.empty(T, device=layer.device) if cfg.shared_gated else None
    layer.moe.encode_route_decode(layer.router_ops, layer.layer, layer.pool, x_dev, ids, w, gate)
    layer.moe.encode_phase1(layer.pool, layer.offsets, T, layer.shared)
    layer.moe.encode_phase2_reduce(layer.pool, layer.offsets, w, y, T, hidden, layer.shared, gate)
    layer.moe.status()
    return y.cpu().numpy(), ids.cpu().numpy().astype(np.uint32), w.cpu().numpy(), hidden.cpu().numpy()


def weights_last(cfg, off: capi.ExpertOffsets, block: np.ndarray, f: int):
    """The block with every matrix's weights behind its scales and biases, and its offsets."""
    out, moved, at = np.empty_like(block), capi.ExpertOffsets(), 0
    for name, rows, cols in (("gate", f, cfg.d), ("up", f, cfg.d), ("down", cfg.d, f)):
        meta = rows * (cols // cfg.group_size) * 2
        for part, size in (("s", meta), ("b", meta), ("w", rows * cols * cfg.weight_bits // 8)):
            old = getattr(off, f"{name}_{part}")
            out[at:at + size] = block[old:old + size]
            setattr(moved, f"{name}_{part}", at)
            at += size
    assert at == block.nbytes
    return out, moved


def test_blocks_that_end_with_weights(cuda_device):
    """Rows of 192 bytes are one and a half pieces: a copy of the last row's second piece would leave the block (248,832
    bytes, a whole cell). The streaming kernel leaves such blocks to the per-tile kernels; the one-row kernel reads whole groups
    and keeps them, with the same sums as ever."""
    cfg = small_config(d=384, f=384, shared_f=384)
    layer = Layer(cfg)
    assert layer.block_bytes == layer.pool.cell_stride
    x = inputs(1, cfg.d, seed=2)
    usual = layer.forward(x, fused=True)[0]
    for e in range(cfg.num_experts):
        block, moved = weights_last(cfg, layer.offsets, layer.block(e), cfg.f)
        layer.pool.upload(layer.first_cell + e, block)
    shared, moved_shared = weights_last(cfg, layer.shared.offsets, layer.shared_block_host, cfg.shared_f)
    layer.offsets, layer._shared_dev = moved, torch.from_numpy(shared).to(layer.device)
    layer.shared = capi.SharedExpert(layer._shared_dev.data_ptr(), moved_shared)
    assert (layer.forward(x, fused=True)[0] == usual).all()
    for T in (3, 17):
        check_layer(layer, inputs(T, cfg.d, seed=T), fused=True)
    layer.close()


@pytest.mark.parametrize("k", [3, 8])
@pytest.mark.parametrize("alike,left", [(9, 64), (32, 64), (33, 64), (64, 64), (9, 5), (1, 8), (40, 36)])
def test_picks_among_equal_scores(cuda_device, alike, left, k):
    """Experts whose router rows are the same score the same: of up to 32 candidates the lower ids win by comparison, of more by
    rounds. `left` experts have a score at all (the others' bias is minus infinity): fewer than the picks leave id 0."""
    bias = np.where(np.arange(64) < left, 0.0, -np.inf).astype(np.float32)
    layer = Layer(small_config(num_experts=64, top_k=k), logit_bias=bias, router_sigma=0.2)
    at = np.random.default_rng(alike).permutation(64)[:alike]
    layer.router_w[at] = 3 * layer.router_w[at[0]]
    layer._rw.copy_(torch.from_numpy(layer.router_w))
    x = inputs(24, layer.cfg.d, seed=alike)
    _, ids, w, _ = layer.forward(x, fused=True)
    ids_ref, w_ref, _ = layer.oracle_route(x)
    assert (ids == ids_ref).all()
    assert np.array_equal(w, w_ref, equal_nan=True)
    layer.close()


@pytest.mark.parametrize("kw", [
    dict(d=256, f=128, shared_f=384),
    dict(d=384, f=192, shared_f=320, group_size=32, weight_bits=4, meta_dtype=capi.DTYPE_FP16),
    dict(d=192, f=320, shared_f=64, group_size=32, weight_bits=8, expert_bias=1, activation=capi.ACT_GELU_TANH),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
@pytest.mark.parametrize("T", [2, 3, 5, 8])
def test_few_rows(cuda_device, kw, T):
    """The rows' groups in the router: one, two, four of them, with unequal numbers of rows."""
    test_stream_edges(cuda_device, kw, T)


@pytest.mark.parametrize("kw", [
    dict(),
    dict(weight_bits=8, router_weight_bits=8, router_kind=capi.ROUTER_SIGMOID, routed_scaling=2.446, shared_gated=False),
], ids=["int4", "int8"])
def test_two_rows_are_the_separate_calls_rows(cuda_device, kw):
    """The smallest number of rows that layer calls and projections of their own both give to this kernel: bit for bit the same."""
    equals_the_separate_calls(cuda_device, 2, kw)
