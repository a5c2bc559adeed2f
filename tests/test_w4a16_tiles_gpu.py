"""Tensor-core linear at the edges of its tiles, runs and rings, against float64 (GPU).

The operand is the 16-bit weight the reference's eager path casts, exactly (tests/test_w4a16_gpu.py), products are exact in
fp32 and at most K of them are added, so against float64 on the SAME rounded weights an output differs by the fp32 sum
(<= K * 2^-24 of the sum of magnitudes, far below the next term) and its own rounding: 2^-11 (fp16) / 2^-8 (bf16) of its value.
"""

import pytest
import torch

from pare_b200.decode import synthetic_linear
from pare_b200.kernels import _lib

pytestmark = pytest.mark.gpu


def _reference(layer, x):
    w = layer.dequantize().to(x.dtype).double()
    return x.double() @ w.T, x.double().abs() @ w.abs().T


def _check(layer, x):
    y = layer(x)
    ref, mag = _reference(layer, x)
    ulp = 2.0 ** -11 if x.dtype == torch.float16 else 2.0 ** -8
    bound = ulp * ref.abs() + layer.in_features * 2.0 ** -24 * mag + 1e-7
    assert bool(((y.double() - ref).abs() <= bound).all())
    assert torch.equal(y, layer(x))
    assert _lib.workspace_status(x.device) == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [17, 33, 48, 65, 127, 129, 255, 257, 272, 513])
def test_row_edges(m, dtype, cuda_lib):
    """Tile heights between 32 and 256 rows, last tiles of one row and of all but one; runs that end inside a tile."""
    layer = synthetic_linear(640, 1536, seed=m, device="cuda")
    _check(layer, torch.randn(m, 1536, device="cuda", generator=torch.Generator("cuda").manual_seed(m)).to(dtype))


@pytest.mark.parametrize("n,k,m", [(1, 512, 17), (127, 512, 40), (129, 1024, 200), (128, 28672, 64), (4096, 14336, 130),
                                   (19072, 2048, 70), (18944, 512, 300), (3001, 2560, 256)])
def test_column_and_depth_edges(n, k, m, cuda_lib):
    """One column, ragged last weight tiles (odd heights take the two-byte stores), tiles cut into many parts, more tiles than
    SMs, the deepest and the shallowest rings."""
    layer = synthetic_linear(n, k, seed=n + m, device="cuda")
    _check(layer, torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).half())


@pytest.mark.parametrize("group", [256, 512, 1536])
def test_wide_groups(group, cuda_lib):
    """A scale that serves several 128-column stages."""
    layer = synthetic_linear(256, 1536, seed=group, device="cuda", group_size=group)
    _check(layer, torch.randn(80, 1536, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).half())


def test_odd_output_pitch(cuda_lib):
    """An output whose rows are not 4-byte aligned, and a bias."""
    from pare_b200.kernels.matmul_int4 import w4a16_forward
    layer = synthetic_linear(384, 1024, seed=3, device="cuda")
    x = torch.randn(50, 1024, device="cuda", generator=torch.Generator("cuda").manual_seed(2)).half()
    bias = torch.randn(384, device="cuda", generator=torch.Generator("cuda").manual_seed(4)).half()
    sc, ze = layer.scale.squeeze(-1).contiguous(), layer.zero.squeeze(-1).contiguous()
    want = w4a16_forward(x, layer.packed_weight, sc, ze, 128, bias=bias)
    out = torch.zeros(50, 385, device="cuda", dtype=torch.float16)
    w4a16_forward(x, layer.packed_weight, sc, ze, 128, bias=bias, out=out[:, :384])
    assert torch.equal(out[:, :384], want) and bool((out[:, 384] == 0).all())


def test_weight_tiles_inner(cuda_lib):
    """Activations larger than L2 whose runs cut tiles: weight tiles are the inner direction of the order."""
    layer = synthetic_linear(1000, 28672, seed=7, device="cuda")
    x = torch.randn(2300, 28672, device="cuda", generator=torch.Generator("cuda").manual_seed(5)).half()
    _check(layer, x)
