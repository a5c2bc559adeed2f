"""The codes-on-the-tensor-core linear (5 - 16 rows) at the edges of its tiles and runs, against float64 (GPU).

Activations are exact after their power-of-two scaling, codes are exact, sums are fp32 over at most K terms: an output differs
from float64 on the same inputs by its own rounding (2^-11 / 2^-8 of its value) and K * 2^-23 of the magnitudes added (which
include the codes' zero-point: sum |x| * scale * 15)."""

import pytest
import torch

from pare_b200.decode import synthetic_linear
from pare_b200.kernels import _lib
from pare_b200.kernels.matmul_int4 import prepare, w4a16_forward

pytestmark = pytest.mark.gpu


def _layer_reference(layer, x):
    n, k = layer.out_features, layer.in_features
    q = torch.stack([layer.packed_weight & 15, layer.packed_weight >> 4], -1).reshape(n, k).double()
    rep = k // layer.scale.reshape(n, -1).shape[1]
    s = layer.scale.double().reshape(n, -1).repeat_interleave(rep, 1)
    z = layer.zero.double().reshape(n, -1).repeat_interleave(rep, 1)
    return x.double() @ ((q - z) * s).T, x.double().abs() @ (15.0 * s).T


def _check(n, k, m, dtype, group=128, scale=1.0):
    layer = synthetic_linear(n, k, seed=n + k + m, device="cuda", group_size=group)
    x = (torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(m)) * scale).to(dtype)
    x[:, :128] = 0          # a step without a largest magnitude
    y = layer(x)
    ref, mag = _layer_reference(layer, x)
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert bool(((y.double() - ref).abs() <= ulp * ref.abs() + k * 2.0 ** -23 * mag + 1e-7 * scale).all())
    for _ in range(5):
        assert torch.equal(y, layer(x))
    assert torch.equal(y, layer.forward_prepared(prepare(x)))
    assert _lib.workspace_status(x.device) == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [9, 10, 15, 16])
@pytest.mark.parametrize("n,k", [(1, 256), (127, 512), (129, 768), (1000, 4096), (18944, 1024), (640, 16384)])
def test_edges(n, k, m, dtype, cuda_lib):
    _check(n, k, m, dtype)


@pytest.mark.parametrize("m", [5, 6, 7, 8])
@pytest.mark.parametrize("n,k", [(6144, 4096), (6272, 4096), (1792, 14336), (3000, 8448)])
def test_both_sides_of_the_row_rule(n, k, m, cuda_lib):
    _check(n, k, m, torch.bfloat16)


@pytest.mark.parametrize("group", [256, 512, 2048])
def test_wide_groups(group, cuda_lib):
    _check(300, 2048, 11, torch.float16, group=group)


@pytest.mark.parametrize("scale", [1e-4, 1e4])
def test_magnitudes(scale, cuda_lib):
    """Activations far from 1: the per-step factors keep fp16 operands in range."""
    _check(256, 1024, 16, torch.bfloat16, scale=scale)


def test_cold_weights_many_units(cuda_lib):
    """A layer larger than L2, read cold, over and over: the same bits every time (a ring slot refilled too early shows here)."""
    layer = synthetic_linear(57344, 8192, seed=1, device="cuda")
    x = torch.randn(16, 8192, device="cuda", generator=torch.Generator("cuda").manual_seed(3)).bfloat16()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    first = layer(x)
    for _ in range(8):
        flush.zero_()
        assert torch.equal(layer(x), first)
    xl = torch.randn(64, 8192, device="cuda", generator=torch.Generator("cuda").manual_seed(4)).bfloat16()
    first = layer(xl)
    for _ in range(4):
        flush.zero_()
        assert torch.equal(layer(xl), first)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("act_order", [False, True])
@pytest.mark.parametrize("n,k,m", [(129, 768, 9), (640, 4096, 16), (2048, 14336, 6), (6144, 4096, 8)])
def test_bias_input_scale_and_act_order(n, k, m, act_order, dtype, cuda_lib):
    """What the preparation launch does (quotient by a run-time scale rounded to the dtype, gather) and what the fold adds."""
    g = torch.Generator("cuda").manual_seed(n + m)
    layer = synthetic_linear(n, k, seed=n, device="cuda")
    scale_in = torch.exp(0.5 * torch.randn(k, device="cuda", generator=g))
    bias = torch.randn(n, device="cuda", generator=g).to(dtype)
    perm = torch.randperm(k, device="cuda", generator=g).to(torch.int32) if act_order else None
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    y = w4a16_forward(x, layer.packed_weight, layer.scale.squeeze(-1).contiguous(), layer.zero.squeeze(-1).contiguous(), 128, bias=bias,
                      col_perm=perm, input_scale=scale_in)
    xs = (x.float() / scale_in).to(dtype)
    ref, mag = _layer_reference(layer, xs[:, perm.long()] if act_order else xs)
    ref = ref + bias.double()
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert bool(((y.double() - ref).abs() <= ulp * ref.abs() + k * 2.0 ** -23 * mag + 1e-7).all())
