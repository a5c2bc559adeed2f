"""The one-launch ``update()`` result and the vectorised quantizer at their edges (GPU), bit for bit."""

import numpy as np
import pytest
import torch

from oracle import kivi as ok
from pare_b200.kv_cache import (KVCacheConfig, QuantizedKVCache, _dequantize_keys, _dequantize_values, _quantize_keys,
                                _quantize_values)

pytestmark = pytest.mark.gpu
D = 128


def _want(cache):
    """Dense K / V from the logical views: fp32 code * scale + zero, rounded to the dtype, then the window."""
    c, st = cache._compressed[0], cache._stores[0]
    k, v = [cache._residual_k[0]], [cache._residual_v[0]]
    if c is not None:
        k.insert(0, _dequantize_keys(c.k_quant, c.k_scale, c.k_zero, st.cfg.group_size).to(st.dtype))
        v.insert(0, _dequantize_values(c.v_quant, c.v_scale, c.v_zero).to(st.dtype))
    return torch.cat(k, 2), torch.cat(v, 2)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,group,v_group", [(4, 32, None), (2, 16, 32), (4, 64, 32), (2, 128, None), (8, 32, None)])
def test_update_returns_reconstruction_and_window(bits, group, v_group, dtype, cuda_lib):
    """Prompts shorter and longer than the window, single tokens that stay in it, fill it, and push a group out."""
    g = torch.Generator("cuda").manual_seed(bits + group)
    cache = QuantizedKVCache(1, KVCacheConfig(bits=bits, group_size=group, residual_length=64, v_group_size=v_group))
    given = [[], []]
    for n in (300, 1, 1, group - 2, 2, 1, 40, 200, 1):
        k = (torch.randn(2, 3, n, D, device="cuda", generator=g) * 2).to(dtype)
        v = torch.randn(2, 3, n, D, device="cuda", generator=g).to(dtype)
        given[0].append(k)
        given[1].append(v)
        fk, fv = cache.update(0, k, v)
        wk, wv = _want(cache)
        assert torch.equal(fk, wk) and torch.equal(fv, wv)
        assert torch.equal(cache._residual_k[0], torch.cat(given[0], 2)[:, :, -cache._residual_k[0].shape[2]:])
        assert torch.equal(cache._residual_v[0], torch.cat(given[1], 2)[:, :, -cache._residual_v[0].shape[2]:])


@pytest.mark.parametrize("n", [7, 500])
def test_forms_of_new_tokens(n, cuda_lib):
    """Views of a fused projection, broadcast heads, a channel stride, rows off the 16-byte alignment, float32 values beside
    float16 keys, tokens that require a gradient: the same bits as dense float16 tokens."""
    g = torch.Generator("cuda").manual_seed(n)
    fused = torch.randn(2, n, 9 * D, device="cuda", generator=g).half()
    k = fused[..., : 2 * D].unflatten(2, (2, D)).transpose(1, 2)
    v = fused[..., 3 * D: 5 * D].unflatten(2, (2, D)).transpose(1, 2)
    odd = torch.empty(k.numel() + 1, device="cuda", dtype=torch.float16)[1:].view(k.shape)
    odd.copy_(k)
    one = k[:, :1]
    forms = [(k, v), (odd, v), (k.transpose(2, 3).contiguous().transpose(2, 3), v),
             (k.contiguous().requires_grad_(True), v), (k.contiguous(), v.contiguous().requires_grad_(True))]
    if n < 64:
        forms.append((k, v.float()))
    base = QuantizedKVCache(1, KVCacheConfig(residual_length=64))
    want = base.update(0, k.contiguous(), v.contiguous())
    for a, b in forms:
        cache = QuantizedKVCache(1, KVCacheConfig(residual_length=64))
        got = cache.update(0, a, b)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    cache = QuantizedKVCache(1, KVCacheConfig(residual_length=64))
    got = cache.update(0, one.expand(2, 2, n, D), v)
    dense = QuantizedKVCache(1, KVCacheConfig(residual_length=64)).update(0, one.expand(2, 2, n, D).contiguous(), v.contiguous())
    assert torch.equal(got[0], dense[0]) and torch.equal(got[1], dense[1])


def test_gradients_through_the_window(cuda_lib):
    k = torch.randn(1, 2, 5, D, device="cuda").half().requires_grad_(True)
    v = torch.randn(1, 2, 5, D, device="cuda").half()
    fk, _ = QuantizedKVCache(1, KVCacheConfig()).update(0, k, v)
    fk.float().sum().backward()
    assert torch.equal(k.grad, torch.ones_like(k))


@pytest.mark.parametrize("bits", [2, 4])
@pytest.mark.parametrize("group", [16, 32, 64])
def test_quotients_on_rounding_boundaries(bits, group, cuda_lib):
    """Values at lo + scale * (n + 1/2) and next to it, constants, infinities and NaNs: codes, scales and zeros as the oracle's
    divisions give them; with infinities and NaNs the scales and zeros are those of the element-wise kernel (reached through
    float32 input)."""
    q = (1 << bits) - 1
    g = torch.Generator().manual_seed(group)
    n = 4 * group
    base = torch.randint(0, 2 * q + 1, (1, 2, n, D), generator=g).float() * 0.5      # multiples of half a step, 0 .. q
    base[:, :, 0::group] = 0.0
    base[:, :, 1::group] = float(q)
    base[..., 0] = 0.0
    base[..., 1] = float(q)
    x = (base * 0.25).half()
    x[:, :, 2::group, 5] += 2.0 ** -10
    x[:, :, 3::group] = 1.5
    x = x.cuda()
    for got, ref in zip((*_quantize_keys(x, bits, group), *_quantize_values(x, bits, group)),
                        ok.quantize_keys(x.float().cpu().numpy(), bits, group) + ok.quantize_values(x.float().cpu().numpy(), bits, group)):
        assert np.array_equal(got.cpu().numpy(), ref)
    x[0, 0, 4, 9], x[0, 1, 5, 10], x[0, 1, 6, 11] = float("inf"), float("-inf"), float("nan")
    for a, b in zip((*_quantize_keys(x, bits, group)[1:], *_quantize_values(x, bits, group)[1:]),
                    (*_quantize_keys(x.float(), bits, group)[1:], *_quantize_values(x.float(), bits, group)[1:])):
        assert np.array_equal(a.cpu().numpy(), b.cpu().numpy(), equal_nan=True)
