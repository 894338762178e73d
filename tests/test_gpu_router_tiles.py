"""The router's register tiles: calls of more than eight rows, every weight format and activation type, against the oracle bit for
bit, and against the kernel with a warp per expert row, which takes smaller calls and rows that are not 16-byte aligned."""
import numpy as np
import pytest
import torch

from gpu_harness import Layer, bf16_tensor, inputs, small_config, to_act_tensor
from shrike_b200 import capi

pytestmark = pytest.mark.gpu

ACTS = [capi.DTYPE_FP32, capi.DTYPE_BF16, capi.DTYPE_FP16]


def make(bits, act, d, ne, T, **kw):
    cfg = small_config(d=d, num_experts=ne, top_k=min(8, ne), act_dtype=act, router_weight_bits=bits, max_tokens=T, **kw)
    layer = Layer(cfg, router_sigma=0.05, device_fill=True)
    x = inputs(T, d, seed=T)
    return layer, x.astype(np.float16).astype(np.float32) if act == capi.DTYPE_FP16 else x


# tiles of 4 x 8 up to 96 Ki logits (9, 77, 383 rows), of 8 x 8 (fp32 activations) or 8 x 16 beyond; 1,100 rows: above 256 Ki
@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("bits", [0, 8, 4])
@pytest.mark.parametrize("d,ne,T", [(320, 250, 9), (2880, 31, 77), (64, 256, 383), (192, 256, 401), (320, 250, 1100)])
def test_ids_and_weights_are_the_oracles(cuda_device, bits, act, d, ne, T):
    layer, x = make(bits, act, d, ne, T)
    ids, w, gate = layer.route(to_act_tensor(x, act, layer.device))
    ids_ref, w_ref, _ = layer.oracle_route(x)
    assert (ids.cpu().numpy().astype(np.uint32) == ids_ref).all()
    assert (w.cpu().numpy() == w_ref).all()
    for t0 in (0, T - 8):
        few = layer.route(to_act_tensor(x[t0:t0 + 8], act, layer.device))
        for a, b in zip(few, (ids, w, gate)):
            assert (a == b[t0:t0 + 8]).all()
    layer.close()


@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("bits", [0, 8])
def test_strides_column_scales_and_values_that_are_no_numbers(cuda_device, bits, act):
    """Rows a stride apart with a scale per column, NaN, infinities and zeros among them: the tiles (a stride of whole 16 bytes)
    and the kernel of a warp per expert row (any other) give the same."""
    d, ne, T = 192, 40, 70
    layer, x = make(bits, act, d, ne, T)
    x[3, 17] = np.nan
    x[11, 100] = np.inf
    x[12, 5] = -np.inf
    x[40] = 0.0
    layer.router_ops.effective_scale = bf16_tensor(np.random.default_rng(5).uniform(0.5, 1.5, d).astype(np.float32), layer.device)
    got = []
    for pad in (64, 4):
        wide = np.full((T, d + pad), 3.0, dtype=np.float32)
        wide[:, :d] = x
        got.append(layer.route(to_act_tensor(wide, act, layer.device), stride=d + pad))
    assert act == capi.DTYPE_FP32 or (d + 4) * 2 % 16 != 0
    for a, b in zip(*got):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    few = layer.route(to_act_tensor(x[8:16], act, layer.device))
    for a, b in zip(few, got[0]):
        assert torch.equal(a.view(torch.int32), b[8:16].view(torch.int32))
    layer.close()


@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("bits", [0, 8, 4])
@pytest.mark.parametrize("d,ne,T", [(2048, 5, 64), (2048, 16, 33), (2304, 7, 12)])
def test_rows_of_few_experts(cuda_device, bits, act, d, ne, T):
    """fp32 rows of 2048 or 2304 columns: a warp each up to 64 rows where the tiles would be a few."""
    test_ids_and_weights_are_the_oracles(cuda_device, bits, act, d, ne, T)


@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("bits", [0, 8, 4])
def test_every_group_of_eight_rows(cuda_device, bits, act):
    """Rows a stride apart with a scale per column, NaN, infinities and zeros among them: the tiles against the kernel of a warp per
    expert row, eight rows at a time."""
    d, ne, T, pad = 192, 40, 70, 8
    layer, x = make(bits, act, d, ne, T)
    x[3, 17] = np.nan
    x[11, 100], x[12, 5] = np.inf, -np.inf
    x[40] = 0.0
    layer.router_ops.effective_scale = bf16_tensor(np.random.default_rng(5).uniform(0.5, 1.5, d).astype(np.float32), layer.device)
    wide = np.full((T, d + pad), 3.0, dtype=np.float32)
    wide[:, :d] = x
    got = layer.route(to_act_tensor(wide, act, layer.device), stride=d + pad)
    for t0 in [*range(0, T - 8, 8), T - 8]:
        few = layer.route(to_act_tensor(x[t0:t0 + 8], act, layer.device))
        for a, b in zip(few, got):
            assert torch.equal(a.view(torch.int32), b[t0:t0 + 8].view(torch.int32))
    layer.close()
