"""Linears of one to four rows: activations brought into operand order inside the kernel or by a launch before it (GPU)."""

import pytest
import torch

from pare_b200.decode import synthetic_linear
from pare_b200.kernels.matmul_int4 import prepare, w4a16_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k", [(16, 256), (1000, 768), (4096, 4096), (6144, 4096), (28672, 4096), (2048, 14336), (57344, 8192)])
def test_same_bits_as_prepared_activations(n, k, m, dtype, cuda_lib):
    """Both sides of the rule, one-slice and many-slice layers; a row pitch larger than K, and rows off the 16-byte alignment
    (which always take the launch)."""
    layer = synthetic_linear(n, k, seed=n + k, device="cuda")
    wide = torch.randn(m, k + 8, device="cuda", generator=torch.Generator("cuda").manual_seed(m)).to(dtype)
    x = wide[:, :k]
    want = layer.forward_prepared(prepare(x.contiguous()))
    assert torch.equal(layer(x.contiguous()), want)
    assert torch.equal(layer(x), want)
    odd = torch.empty(m * k + 1, device="cuda", dtype=dtype)[1:].view(m, k)
    odd.copy_(x)
    assert torch.equal(layer(odd), want)
    sc, ze = layer.scale.squeeze(-1).contiguous(), layer.zero.squeeze(-1).contiguous()
    perm = torch.arange(k, device="cuda", dtype=torch.int32)
    assert torch.equal(w4a16_forward(x.contiguous(), layer.packed_weight, sc, ze, 128, col_perm=perm), want)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 8, 16])
@pytest.mark.parametrize("n", [256, 2048, 4096, 8192])
def test_output_over_the_activations(n, m, cuda_lib):
    """``out`` may be the activations themselves, or overlap them: they are read before anything is written."""
    layer = synthetic_linear(n, n, seed=n, device="cuda")
    sc, ze = layer.scale.squeeze(-1).contiguous(), layer.zero.squeeze(-1).contiguous()
    x = torch.randn(m, n, device="cuda", generator=torch.Generator("cuda").manual_seed(m)).half()
    want = layer(x)
    for shift in (0, 8, n // 2):                 # out starts `shift` elements into the activations
        for _ in range(5):
            buf = torch.zeros(m * n + shift, device="cuda", dtype=torch.float16)
            a, out = buf[: m * n].view(m, n), buf[shift:].view(m, n)
            a.copy_(x)
            w4a16_forward(a, layer.packed_weight, sc, ze, 128, out=out)
            assert torch.equal(out, want)
