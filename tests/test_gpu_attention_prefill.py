"""`jq_attention_prefill_dev` (16-bit terms on the tensor cores) against float64 attention: query and key counts around the
tiles of 128 queries and 64 keys, both head sizes, grouped heads, earlier positions in the cache, rows behind the last key
that hold NaN, values and keys decades apart, infinities."""
import math

import pytest

pytestmark = pytest.mark.gpu

# (new tokens, earlier positions, q heads, kv heads, head size)
SHAPES = [(1, 0, 4, 1, 128), (1, 63, 2, 2, 64), (17, 0, 4, 2, 128), (64, 0, 2, 1, 64), (63, 65, 8, 1, 128), (127, 1, 2, 2, 128),
          (128, 0, 4, 2, 64), (129, 0, 2, 1, 128), (130, 62, 4, 4, 64), (300, 37, 8, 2, 128), (257, 511, 2, 1, 64)]


def reference(q, k, v, p0):
    import torch

    S, nq, hd = q.shape
    n, grp = p0 + S, nq // k.shape[0]
    kk, vv = (t[:, :n].double().repeat_interleave(grp, 0) for t in (k, v))
    s = torch.einsum("shd,htd->hst", q.double(), kk) / math.sqrt(hd)
    hidden = torch.arange(n, device=q.device)[None] > (p0 + torch.arange(S, device=q.device))[:, None]
    s = s.masked_fill(hidden, -math.inf)
    return torch.einsum("hst,htd->shd", s.softmax(-1), vv), float(s[~hidden.expand_as(s)].abs().max())


def run(q, k, v, p0, max_ctx):
    import torch

    from joshua_b200 import _lib

    S, nq, hd = q.shape
    pos = torch.tensor([p0], dtype=torch.int32, device=q.device)
    bad = torch.zeros(1, dtype=torch.int32, device=q.device)
    out = torch.full_like(q, 3.0)
    _lib.check(_lib.lib().jq_attention_prefill_dev(q.data_ptr(), k.data_ptr(), v.data_ptr(), pos.data_ptr(), S, nq, k.shape[0], hd,
                                                   max_ctx, out.data_ptr(), bad.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out, int(bad.item())


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("spread", [False, True])
def test_prefill_attention_matches_float64(shape, spread):
    import torch

    S, p0, nq, nkv, hd = shape
    dev, max_ctx = torch.device("cuda", 0), p0 + S + 5
    gen = torch.Generator(device=dev).manual_seed(S * 7 + p0)
    q = torch.randn(S, nq, hd, device=dev, generator=gen)
    k = torch.randn(nkv, max_ctx, hd, device=dev, generator=gen)
    v = torch.randn(nkv, max_ctx, hd, device=dev, generator=gen)
    if spread:  # a value dimension 1e4 times the others, a key row 1e-3 and one query row 1e-2 of them
        v[:, :, 7] *= 1e4
        k[:, p0 + S // 2] *= 1e-3
        q[S // 2] *= 1e-2
    k[:, p0 + S:] = math.nan  # the cache behind the newest key: never written
    v[:, p0 + S:] = math.nan
    got, bad = run(q, k, v, p0, max_ctx)
    want, s_max = reference(q, k, v, p0)
    assert bad == 0
    # Terms hold 2^-22 of a row's or column's largest values and a chain of 12 products adds a few 2^-24; a score's error
    # is that of its size and makes a relative error of its probability, above and below the fraction line.
    tol = 2.0 ** -20 * (1.0 + s_max) * v[:, :p0 + S].abs().amax((0, 1)).double()
    assert bool(((got.double() - want).abs() <= tol).all()), float(((got.double() - want).abs() / tol).max())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("S, p0", [(16, 0), (130, 0), (200, 37)])
def test_later_tokens_do_not_reach_earlier_ones(S, p0, hd):
    """Bit for bit, whatever the keys and values of tokens behind a query hold."""
    import torch

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(S + hd)
    q = torch.randn(S, 4, hd, device=dev, generator=gen)
    k = torch.randn(2, p0 + S, hd, device=dev, generator=gen)
    v = torch.randn(2, p0 + S, hd, device=dev, generator=gen)
    first, _ = run(q, k, v, p0, p0 + S)
    for cut in (1, S // 2, S - 1):  # tokens cut .. S - 1 change
        for later in (0.0, 1e6, 3e38, 1e-30, math.inf, -math.inf, math.nan):
            k2, v2 = k.clone(), v.clone()
            k2[:, p0 + cut:, ::3] = later
            v2[:, p0 + cut:, ::2] = later
            got, bad = run(q, k2, v2, p0, p0 + S)
            assert bad == 0 and bool((got[:cut] == first[:cut]).all()), (cut, later)


@pytest.mark.parametrize("hd", [64, 128])
def test_infinities_reach_the_queries_that_see_them(hd):
    import torch

    S, at, dev = 150, 70, torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(hd)
    q = torch.randn(S, 2, hd, device=dev, generator=gen)
    k = torch.randn(1, S, hd, device=dev, generator=gen)
    v = torch.randn(1, S, hd, device=dev, generator=gen)
    first, _ = run(q, k, v, 0, S)
    v[0, at, 3], v[0, at, hd - 1], v[0, at + 1, 5] = math.inf, -math.inf, math.nan
    got, _ = run(q, k, v, 0, S)
    assert bool((got[at:, :, 3] == math.inf).all()) and bool((got[at:, :, hd - 1] == -math.inf).all())
    assert bool(got[at + 1:, :, 5].isnan().all())
    for t in (got, first):
        t[at:, :, [3, 5, hd - 1]] = 0
    assert bool((got == first).all())
    # a key of minus infinity in a dimension where the query is positive has no weight, one of plus infinity no result
    v[0, at:at + 2] = 1.0
    q[:, :, 7] = q[:, :, 7].abs() + 0.1
    k[0, at, 7] = -math.inf
    got, _ = run(q, k, v, 0, S)
    want, _ = reference(q, k, v, 0)
    assert float((got.double() - want).norm() / want.norm()) <= 1e-6
    k[0, at, 7] = math.inf
    got, _ = run(q, k, v, 0, S)
    assert bool(got[at:].isnan().all()) and bool(got[:at].isfinite().all())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("S", [16, 64, 200])
def test_values_decades_apart_keep_their_bits(S, hd):
    """One value of 1e6 and a dimension of 1e-6 beside N(0, 1): each output to the size of what it adds up."""
    import torch

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(S + hd)
    q = torch.randn(S, 4, hd, device=dev, generator=gen)
    k = torch.randn(1, S, hd, device=dev, generator=gen)
    v = torch.randn(1, S, hd, device=dev, generator=gen)
    v[0, S // 2, 3], v[0, :, 9] = 1e6, v[0, :, 9] * 1e-6
    got, _ = run(q, k, v, 0, S)
    want, s_max = reference(q, k, v, 0)
    size, _ = reference(q, k, v.abs(), 0)
    # a score's error is 2^-22 of its size and makes a relative error of its probability, above and below the fraction line;
    # the terms of probabilities and values hold 2^-24, their chain of 24 products adds a few 2^-24 of the sum of magnitudes
    tol = 2.0 ** -20 * (1.0 + s_max) * size
    assert bool(((got.double() - want).abs() <= tol).all()), float(((got.double() - want).abs() / tol).max())


def test_positions_outside_the_cache_are_reported():
    import torch

    dev = torch.device("cuda", 0)
    q, k = torch.randn(9, 2, 64, device=dev), torch.randn(1, 16, 64, device=dev)
    out, bad = run(q, k, k.clone(), 8, 16)
    assert bad == 1 and bool((out == 3.0).all())
