"""The streaming expert kernel at the edges of its tiling, against the oracle: rows of weights that end inside a
128-byte piece, group counts that leave a quad of groups open, shared and routed experts of different widths, one to
eight rows per instance, and the shapes it leaves to the per-tile kernels (an odd number of groups)."""
import pytest

from shrike_b200 import capi
from gpu_harness import Layer, inputs, small_config
from test_gpu_parity import check_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [9, 17, 64])
@pytest.mark.parametrize("kw", [
    dict(d=256, f=128, shared_f=384),                                    # whole pieces
    dict(d=384, f=640, shared_f=128),                                    # a piece of two groups at the end
    dict(d=320, f=192, shared_f=192),                                    # odd numbers of groups: the per-tile kernels
    dict(d=128, f=128, has_shared=0, shared_gated=0, num_experts=4, top_k=2),   # many instances of the same experts
    dict(d=384, f=192, shared_f=320, group_size=32, weight_bits=4, meta_dtype=capi.DTYPE_FP16),
    dict(d=128, f=384, shared_f=128, group_size=64, weight_bits=8),
    dict(d=192, f=320, shared_f=64, group_size=32, weight_bits=8, expert_bias=1, activation=capi.ACT_GELU_TANH),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_stream_edges(cuda_device, kw, T):
    layer = Layer(small_config(**kw))
    check_layer(layer, inputs(T, kw["d"], seed=T), fused=True)
    layer.close()
