"""`jq_attention_prefill_dev` (f16 terms on the tensor cores) against float64 attention: query and key counts around the
tiles of 128 queries and 64 keys, both head sizes, grouped heads, earlier positions in the cache, rows behind the last key
that hold NaN, values and keys decades apart."""
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


def test_positions_outside_the_cache_are_reported():
    import torch

    dev = torch.device("cuda", 0)
    q, k = torch.randn(9, 2, 64, device=dev), torch.randn(1, 16, 64, device=dev)
    out, bad = run(q, k, k.clone(), 8, 16)
    assert bad == 1 and bool((out == 3.0).all())
