"""Prompt attention at the edges of its 128-query / 128-key tiles, against float64 (GPU).

Probabilities enter as two 16-bit terms (error 2^-16 of a probability or less), sums are fp32, so an output differs from the
float64 softmax by its own rounding (2^-11 / 2^-8 of its value) and about 2^-15 of the largest value that it averages.
"""

import pytest
import torch

from pare_b200.kv_cache import prefill_attention

pytestmark = pytest.mark.gpu


def _reference(q, k, v, causal, scale):
    rep, tq, tk = q.shape[1] // k.shape[1], q.shape[2], k.shape[2]
    s = q.double() @ k.double().repeat_interleave(rep, 1).transpose(-1, -2) * scale
    if causal:
        hidden = torch.arange(tk, device="cuda")[None] > torch.arange(tq, device="cuda")[:, None] + tk - tq
        s = s.masked_fill(hidden, float("-inf"))
    return torch.softmax(s, -1) @ v.double().repeat_interleave(rep, 1)


def _check(b, hq, h, tq, tk, dtype, causal=True, spread=1.0, scale=128 ** -0.5):
    g = torch.Generator("cuda").manual_seed(tq * 31 + tk)
    q = (torch.randn(b, hq, tq, 128, device="cuda", generator=g) * spread).to(dtype)
    k = torch.randn(b, h, tk, 128, device="cuda", generator=g).to(dtype)
    v = torch.randn(b, h, tk, 128, device="cuda", generator=g).to(dtype)
    out = prefill_attention(q, k, v, scale=scale, causal=causal)
    ref = _reference(q, k, v, causal, scale)
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    # 2^-21 of a logit's magnitude (fp32 product and sum) goes into the exponent
    bound = ulp * ref.abs() + (2.0 ** -15 + 2.0 ** -21 * float((q.double().norm(dim=-1).max() * 12 * scale))) * float(v.abs().max())
    assert bool(((out.double() - ref).abs() <= bound).all())
    assert torch.equal(out, prefill_attention(q, k, v, scale=scale, causal=causal))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tq,tk", [(1, 1), (1, 129), (127, 127), (128, 128), (129, 129), (255, 511), (257, 257), (300, 1000), (640, 641)])
def test_length_edges(tq, tk, dtype, cuda_lib):
    _check(1, 4, 2, tq, tk, dtype)
    _check(1, 2, 2, tq, tk, dtype, causal=False)


@pytest.mark.parametrize("hq,h", [(1, 1), (3, 1), (7, 1), (14, 2), (5, 5), (16, 2)])
@pytest.mark.parametrize("t", [100, 260, 400])
def test_heads_that_share_a_kv_head(hq, h, t, cuda_lib):
    """Even and odd numbers of query heads per KV head, odd and even numbers of query tiles: every (head, tile) exactly once."""
    _check(2, hq, h, t, t, torch.float16)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_maximum_that_keeps_growing(dtype, cuda_lib):
    """Logits with a standard deviation of 12, later keys larger than earlier ones: the running maximum is raised again and again."""
    g = torch.Generator("cuda").manual_seed(1)
    t = 700
    k = torch.randn(1, 1, t, 128, device="cuda", generator=g) * torch.linspace(0.2, 4.0, t, device="cuda")[None, None, :, None]
    q = torch.randn(1, 2, t, 128, device="cuda", generator=g) * 3.0
    v = torch.randn(1, 1, t, 128, device="cuda", generator=g)
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    out = prefill_attention(q, k, v)
    ref = _reference(q, k, v, True, 128 ** -0.5)
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert bool(((out.double() - ref).abs() <= ulp * ref.abs() + 2.0 ** -12 * float(v.abs().max())).all())


def test_broadcast_and_negative_scale_take_the_general_path(cuda_lib):
    """What a tensor map cannot describe (a broadcast batch) and a negative scale: the same results."""
    g = torch.Generator("cuda").manual_seed(2)
    q = torch.randn(2, 4, 200, 128, device="cuda", generator=g).half()
    k = torch.randn(1, 2, 200, 128, device="cuda", generator=g).half().expand(2, 2, 200, 128)
    v = torch.randn(1, 2, 200, 128, device="cuda", generator=g).half().expand(2, 2, 200, 128)
    for scale in (128 ** -0.5, -0.1):
        out = prefill_attention(q, k, v, scale=scale)
        ref = _reference(q, k, v, True, scale)
        assert bool(((out.double() - ref).abs() <= 2.0 ** -11 * ref.abs() + 2.0 ** -13 * float(v.abs().max())).all())


def test_infinite_logit_gives_nan_and_hidden_keys_do_not_matter(cuda_lib):
    q = torch.ones(1, 2, 130, 128, device="cuda").half()
    k = torch.ones(1, 1, 130, 128, device="cuda").half()
    v = torch.randn(1, 1, 130, 128, device="cuda").half()
    k[0, 0, 64] = float("inf")
    out = prefill_attention(q, k, v)
    assert bool(torch.isfinite(out[:, :, :64]).all()) and bool(torch.isnan(out[:, :, 64:]).all())


@pytest.mark.parametrize("loads", [0, 1, 2, 3, 7])
@pytest.mark.parametrize("hq,h,t", [(2, 1, 600), (3, 1, 600), (1, 1, 100)])
def test_a_wait_that_runs_out_gives_nan(hq, h, t, loads, cuda_lib):
    """Key and value tiles that never arrive: whichever warp gives up first, no row that depends on them passes for a result, and the
    next call is served as ever.  (Query tiles that had all they need before that are as they should be.)"""
    g = torch.Generator("cuda").manual_seed(loads)
    q = torch.randn(1, hq, t, 128, device="cuda", generator=g).half()
    k = torch.randn(1, h, t, 128, device="cuda", generator=g).half()
    v = torch.randn(1, h, t, 128, device="cuda", generator=g).half()
    want, out = prefill_attention(q, k, v), torch.zeros_like(q)
    assert cuda_lib.pare_selftest_prefill_wait(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), 1, hq, h, t, loads, 300,
                                               torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    whole = loads // 2 * 128                       # keys whose K and V tiles both arrive
    assert bool(torch.isnan(out[:, :, whole:]).all())
    assert bool((torch.isnan(out[:, :, :whole]) | (out[:, :, :whole] == want[:, :, :whole])).all())
    assert torch.equal(prefill_attention(q, k, v), want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hq,h", [(1, 1), (2, 1), (3, 1)])
@pytest.mark.parametrize("tq,tk", [(300, 300), (129, 256), (200, 520), (640, 641)])
def test_values_of_hidden_keys_do_not_matter(hq, h, tq, tk, dtype, cuda_lib):
    """An infinity or a NaN among the values reaches the queries that see its key, in its channel, and nothing else: the channel of the
    queries before it is what it is with a zero in that place (to the bound of the length tests: it is summed again), every other
    output keeps its bits."""
    g = torch.Generator("cuda").manual_seed(tk)
    q = torch.randn(2, hq, tq, 128, device="cuda", generator=g).to(dtype)
    k = torch.randn(2, h, tk, 128, device="cuda", generator=g).to(dtype)
    v = torch.randn(2, h, tk, 128, device="cuda", generator=g).to(dtype)
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    off = tk - tq
    for key, channel, bad in ((off + 1, 3, "nan"), (off + 63, 64, "inf"), (off + 64, 127, "-inf"), (off + 100, 0, "nan"), (off + 127, 70, "inf"),
                              (min(off + 128, tk - 1), 9, "inf"), (tk - 1, 33, "nan"), (tk - 1, 96, "-inf"), (0, 5, "inf")):
        w = v.clone()
        w[0, 0, key, channel] = 0.0
        want = prefill_attention(q, k, w)
        w[0, 0, key, channel] = float(bad)
        out = prefill_attention(q, k, w)
        share = slice(0, hq // h)                         # the query heads of that KV head, in the first sequence only
        first = max(0, key - off)                         # the first query that sees the key
        assert bool((~torch.isfinite(out[0, share, first:, channel])).all()), key
        before, ref = out[0, share, :first, channel].double(), want[0, share, :first, channel].double()
        assert bool(((before - ref).abs() <= 2 * ulp * ref.abs() + 2.0 ** -13).all()), key
        out[0, share, :, channel] = want[0, share, :, channel]
        assert torch.equal(out, want), key
