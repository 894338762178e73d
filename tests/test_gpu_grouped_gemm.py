"""The expert-grouped GEMM with more tiles than SMs, against the oracle: instances on both sides of every stage layout
(1, 16, 64, 65, 128, 129 and 256 rows and one more than 256) follow one another on an SM, shared and routed experts have
different numbers of row tiles, and the last ones are partial. Wide tiles of two K blocks, which use two of the three activation stages,
before narrow ones; narrow tiles alone, more of them on an SM than it has places for tiles."""
import numpy as np
import pytest
import torch

from shrike_b200 import capi
from shrike_b200.moe import MoE, ShrikeError
import fixtures as fx
from gpu_harness import Layer, inputs, rel_l2, small_config, to_act_tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(d=1088, f=192, shared_f=448),
    dict(d=1024, f=320, shared_f=64, weight_bits=8, group_size=32, meta_dtype=capi.DTYPE_FP16),
    dict(d=960, f=448, shared_f=192, weight_bits=4, group_size=32, expert_bias=1, activation=capi.ACT_CLAMPED_SWIGLU),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_tiles_of_every_layout(cuda_device, kw):
    run_sizes([257, 256, 129, 128, 65, 64, 17, 16] + [1] * 40, kw)


@pytest.mark.parametrize("kw", [
    dict(d=2048, f=128, shared_f=384),
    dict(d=2048, f=128, shared_f=192, weight_bits=8, group_size=32),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_a_short_tile_before_another_layout(cuda_device, kw):
    """The routed experts' wide tiles have two K blocks in the down projection, the shared expert's three or six: the tiles of one and
    of 24 rows that follow on the same SMs have the other layout, while the accumulators of the last wide tile are still read."""
    run_sizes([257] * 24, kw, sample=24)


@pytest.mark.parametrize("kw", [
    dict(d=576, f=64, shared_f=192),                                                # odd numbers of K blocks, one K block
    dict(d=2112, f=576, shared_f=64, weight_bits=8),                                # odd numbers of groups
    dict(d=1088, f=320, shared_f=512, weight_bits=4, group_size=32),                # scale rows of 34 and 10 groups
    dict(d=1024, f=512, shared_f=512, weight_bits=8, group_size=32, meta_dtype=capi.DTYPE_FP16, expert_bias=1),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_narrow_tiles(cuda_device, kw):
    """The routed experts' tiles have up to 128 rows (the shared expert's full ones come before them): on both sides of every number
    of K blocks in an activation stage (32 and 64 rows) and of the second pair of accumulators (64), with K lengths that end in the middle of a packed slot, a pair of K blocks and a scale block."""
    run_sizes([128, 113, 112, 65, 64, 49, 33, 32, 31, 17, 16, 15] + [3] * 40, kw)


@pytest.mark.parametrize("kw", [
    dict(d=640, f=640),
    dict(d=704, f=576, group_size=32, expert_bias=1),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_narrow_tiles_alone(cuda_device, kw):
    """No wide tile and no shared expert: 768 tiles and more in both projections, five and more on an SM of 148, so that the four
    places for tiles, the accumulators' barriers and both kinds of narrow tile come round again."""
    sizes = [128, 97, 96, 80, 72, 66, 65, 64, 63, 48, 33, 32, 17, 16] + [1 + 7 * e % 24 for e in range(242)]
    run_sizes(sizes, dict(kw, num_experts=256, has_shared=False, shared_f=0), sample=100)


def test_a_handle_whose_pool_offsets_or_shared_block_change(cuda_device):
    """A handle keeps the maps of its last call's operands: another pool (of other chunks), another shared block, other offsets in
    the same structure, and the first ones again give what a handle of their own gives. (A row's two sums are added to zero: in
    either order the same.)"""
    cfg = small_config(d=256, f=192, shared_f=128, num_experts=24, top_k=1, max_tokens=300, shared_gated=False)
    layers = [Layer(cfg, seed=s, chunks=n) for s, n in ((1, 1), (2, 8))]
    first, second = layers
    ids = torch.from_numpy(np.random.default_rng(3).integers(0, 24, (300, 1)).astype(np.int32)).cuda()
    w = torch.rand((300, 1), generator=torch.Generator().manual_seed(4)).cuda()
    x = to_act_tensor(inputs(300, cfg.d, seed=5), cfg.act_dtype, first.device)
    slots, _ = first.classify(ids)

    def run(moe, pool, offsets, shared):
        y = torch.empty(x.shape, dtype=cfg.torch_y_dtype, device=x.device)
        moe.encode_prefill(pool, offsets, ids, slots, w, x, y, None, shared)
        moe.status()
        return y

    def alone(*operands):
        moe = MoE(cfg)
        y = run(moe, *operands)
        moe.close()
        return y

    seen = []
    for pool, shared in ((first.pool, first.shared), (second.pool, second.shared), (second.pool, first.shared),
                         (first.pool, first.shared)):
        got = run(first.moe, pool, first.offsets, shared)
        assert torch.equal(got, alone(pool, first.offsets, shared))
        seen.append(got)
    assert torch.equal(seen[0], seen[3]) and not any(torch.equal(a, b) for a, b in zip(seen, seen[1:]))
    o = first.offsets
    for part in ("w", "s", "b"):
        gate, up = getattr(o, f"gate_{part}"), getattr(o, f"up_{part}")
        setattr(o, f"gate_{part}", up)
        setattr(o, f"up_{part}", gate)
    got = run(first.moe, first.pool, o, first.shared)
    assert torch.equal(got, alone(first.pool, o, first.shared)) and not torch.equal(got, seen[0])
    for L in layers:
        L.close()


@pytest.mark.parametrize("T", [1, 100])
def test_rows_in_place(cuda_device, T):
    """y is x: the down projection may not add into rows that are still read, so the call takes the rows of its own."""
    cfg = small_config(d=256, f=192, shared_f=128, num_experts=24, top_k=1, max_tokens=100, shared_gated=False)
    layer = Layer(cfg)
    ids = torch.from_numpy(np.random.default_rng(3).integers(0, 24, (T, 1)).astype(np.int32)).cuda()
    w = torch.rand((T, 1), generator=torch.Generator().manual_seed(4)).cuda()
    x = to_act_tensor(inputs(T, cfg.d, seed=5), cfg.act_dtype, layer.device)
    slots, _ = layer.classify(ids)
    y, same = torch.empty_like(x), x.clone()
    for rows, out in ((x, y), (same, same)):
        layer.moe.encode_prefill(layer.pool, layer.offsets, ids, slots, w, rows, out, None, layer.shared)
        layer.moe.status()
    assert torch.equal(y, same) and not torch.equal(y, x)
    layer.close()


@pytest.mark.parametrize("path", ["umma", "mma"])
@pytest.mark.parametrize("T", [65, 300])
def test_experts_with_pairs_that_miss(cuda_device, monkeypatch, path, T):
    """Pairs at SLOT_MISS, and outside the pool, of experts whose other pairs have a cell, after a larger call on the same handle:
    they contribute nothing, what the larger call left in the order of the pairs is not followed, and nothing is added behind y."""
    if path == "mma":
        monkeypatch.setenv("SHRIKE_PREFILL_PATH", "mma")
    cfg = small_config(d=256, f=192, shared_f=128, num_experts=12, top_k=4, max_tokens=700, shared_gated=False)
    layer = Layer(cfg, router_sigma=0.05)
    layer.forward(inputs(700, cfg.d, seed=1))
    x = inputs(T, cfg.d, seed=2)
    x_dev = to_act_tensor(x, cfg.act_dtype, layer.device)
    ids, w, _ = layer.route(x_dev)
    slots, _ = layer.classify(ids)
    ids_np, w_np = ids.cpu().numpy().astype(np.uint32), w.cpu().numpy()
    missing = np.random.default_rng(3).random((T, 4)) < 0.4
    missing[ids_np == 3] = True     # no pair with a cell
    missing[ids_np == 7] = False    # every pair
    for e, at in ((0, -1), (1, 0)):   # only the last, only the first pair misses
        rows = np.flatnonzero((ids_np == e).any(axis=1))
        missing[ids_np == e] = False
        missing[rows[at], ids_np[rows[at]] == e] = True
    y_ref = layer.oracle_forward(x, ids_np, np.where(missing, np.float32(0), w_np))
    for cell in (-1, cfg.num_experts + 5):
        slots_in = torch.where(torch.from_numpy(missing).cuda(), torch.full_like(slots, cell), slots)
        out = torch.full((700, cfg.d), 7.0, device=layer.device)
        layer.moe.encode_prefill(layer.pool, layer.offsets, ids, slots_in, w, x_dev, out[:T], None, layer.shared)
        if cell < 0:
            layer.moe.status()
        else:
            with pytest.raises(ShrikeError) as err:
                layer.moe.status()
            assert err.value.code == capi.ERANGE
        assert rel_l2(out[:T].cpu().numpy(), y_ref) <= 1e-3
        assert (out[T:] == 7.0).all()
    ids[5, 1] = ids[5, 0]   # a row that names an expert twice is reported, whatever its slots are
    for cells in ((-1, -1), (-1, 2), (2, -1), (2, 2)):
        slots[5, 0], slots[5, 1] = cells
        layer.moe.encode_prefill(layer.pool, layer.offsets, ids, slots, w, x_dev, out[:T], None, layer.shared)
        with pytest.raises(ShrikeError) as err:
            layer.moe.status()
        assert err.value.code == capi.ERANGE
    layer.close()


class LayerOfLargeScales(Layer):
    """Expert blocks whose groups' scales and biases are up to 2^6 (gate, up) and 2^20 (down) times the fixture's: from 0.0013,
    or 2^-14 for bytes, to where a converted weight still is an fp16 number. Most rows keep some groups as they are."""

    def block(self, e):
        if e not in self._blocks:
            b = fx.synth_block(self.cfg, self.seed, self.layer, e)
            o, cfg, rng = self.offsets, self.cfg, np.random.default_rng(e)
            for name, rows, cols, most in (("gate", cfg.f, cfg.d, 6), ("up", cfg.f, cfg.d, 6), ("down", cfg.d, cfg.f, 20)):
                n = rows * cols // cfg.group_size
                by = 2.0 ** (rng.integers(0, most + 1, n) * rng.integers(0, 2, n))
                for part in "sb":
                    at = getattr(o, f"{name}_{part}")
                    v = b[at:at + 2 * n].view(np.uint16)
                    v[:] = fx.meta_bits(fx.meta_to_f32(v, cfg.meta_dtype) * by, cfg.meta_dtype)
            self._blocks[e] = b
        return self._blocks[e]


@pytest.mark.parametrize("kw", [
    dict(d=640, f=192),
    dict(d=704, f=192, group_size=32),
    dict(d=512, f=256, weight_bits=8, meta_dtype=capi.DTYPE_FP16),
    dict(d=576, f=192, weight_bits=8, group_size=32),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_large_scales(cuda_device, kw):
    """Scales that leave fp16's range when they are multiplied up for integers below its normal range, beside ones that do not."""
    run_sizes([257, 129, 65, 17] + [3] * 10, dict(kw, num_experts=16, has_shared=False, shared_f=0), layer_of=LayerOfLargeScales)


def run_sizes(sizes, kw, sample=None, layer_of=Layer):
    cfg = small_config(**dict(dict(num_experts=64, top_k=1, max_tokens=max(1024, sum(sizes)), shared_gated=False), **kw))
    layer = layer_of(cfg)
    ids = np.concatenate([np.full(n, e, np.uint32) for e, n in enumerate(sizes)])
    ids = np.random.default_rng(3).permutation(ids)[:, None]
    x = inputs(len(ids), kw["d"], seed=5)
    w = np.random.default_rng(4).uniform(0.2, 1.0, ids.shape).astype(np.float32)
    x_dev = to_act_tensor(x, cfg.act_dtype, layer.device)
    ids_dev = torch.from_numpy(ids.view(np.int32)).to(layer.device)
    slots, _ = layer.classify(ids_dev)
    y = torch.empty(x_dev.shape, dtype=cfg.torch_y_dtype, device=layer.device)
    layer.moe.encode_prefill(layer.pool, layer.offsets, ids_dev, slots, torch.from_numpy(w).to(layer.device), x_dev, y, None,
                             layer.shared, None)
    layer.moe.status()
    # all rows, or every expert's last one (the remainders) and a few others
    rows = np.arange(len(ids)) if sample is None else np.unique(np.concatenate(
        [[np.flatnonzero(ids[:, 0] == e)[-1] for e in range(len(sizes))], np.random.default_rng(6).choice(len(ids), sample)]))
    want = layer.oracle_forward(x, ids, w, rows=rows)
    got = y.cpu().numpy()[rows]
    assert rel_l2(got, want) <= 1e-3
    # a single row: scale, offset and value of a weight and the activation are rounded to fp16, 2^-11 each
    assert max(rel_l2(g, v) for g, v in zip(got, want)) <= 4 * 2.0 ** -11
    layer.close()
