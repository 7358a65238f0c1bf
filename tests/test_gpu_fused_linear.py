"""The quantized linear with the RMS norm in its prologue and the residual add in its epilogue against the
separate kernels (norm kernel, plain matmul, add), and the gate/up SwiGLU pair with the norm folded in."""
import numpy as np
import pytest

from joshua_b200 import synth

pytestmark = pytest.mark.gpu

TYPES = [synth.Q8_0, synth.Q2_K, synth.Q4_K, synth.IQ2_XXS, synth.MXFP4]


def _close(got, want, tol=1e-5):
    assert float((got - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("type_id", TYPES)
@pytest.mark.parametrize("m,k,n", [(1, 1024, 272), (3, 2048, 130), (8, 4096, 64), (2, 512, 40)])
@pytest.mark.parametrize("use_norm,use_res", [(True, False), (False, True), (True, True)])
def test_linear_with_norm_and_residual(type_id, m, k, n, use_norm, use_res):
    import torch

    from joshua_b200 import _lib
    from joshua_b200.qtensor import QTensor

    L = _lib.lib()
    w = QTensor.from_bytes(type_id, synth.random_weight(type_id, n, k, 3))
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + n)
    x = torch.randn(m, k, device="cuda", generator=g)
    nw = 1.0 + 0.1 * torch.randn(k, device="cuda", generator=g)
    res = torch.randn(m, n, device="cuda", generator=g)
    s = torch.cuda.current_stream().cuda_stream
    xn = torch.empty_like(x)
    if use_norm:
        _lib.check(L.jq_rmsnorm_dev(x.data_ptr(), None, nw.data_ptr(), 1e-5, m, k, None, xn.data_ptr(), s))
    else:
        xn.copy_(x)
    want = torch.empty(m, n, device="cuda")
    _lib.check(L.jq_matmul_t_dev(w._h, m, k, n, xn.data_ptr(), want.data_ptr(), s))
    if use_res:
        want += res
    got = res.clone() if use_res else torch.empty(m, n, device="cuda")   # residual in place
    _lib.check(L.jq_matmul_norm_dev(w._h, m, k, n, x.data_ptr(), nw.data_ptr() if use_norm else None, 1e-5,
                                    got.data_ptr() if use_res else None, got.data_ptr(), s))
    torch.cuda.synchronize()
    _close(got, want)


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.Q8_0])
@pytest.mark.parametrize("m", [1, 4])
def test_swiglu_pair_with_norm(type_id, m):
    import torch

    from joshua_b200 import _lib
    from joshua_b200.qtensor import QTensor

    L = _lib.lib()
    k, n = 1024, 304
    gate = QTensor.from_bytes(type_id, synth.random_weight(type_id, n, k, 1))
    up = QTensor.from_bytes(type_id, synth.random_weight(type_id, n, k, 2))
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=g) * 0.05
    nw = 1.0 + 0.1 * torch.randn(k, device="cuda", generator=g)
    s = torch.cuda.current_stream().cuda_stream
    xn = torch.empty_like(x)
    _lib.check(L.jq_rmsnorm_dev(x.data_ptr(), None, nw.data_ptr(), 1e-6, m, k, None, xn.data_ptr(), s))
    want = torch.empty(m, n, device="cuda")
    _lib.check(L.jq_matmul_swiglu_dev(gate._h, up._h, m, k, n, xn.data_ptr(), want.data_ptr(), 0.0, s))
    got = torch.empty(m, n, device="cuda")
    _lib.check(L.jq_matmul_swiglu_norm_dev(gate._h, up._h, m, k, n, x.data_ptr(), nw.data_ptr(), 1e-6, got.data_ptr(),
                                           0.0, s))
    torch.cuda.synchronize()
    _close(got, want, 1e-4)


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.Q6_K, synth.Q8_0, synth.Q5_0])
@pytest.mark.parametrize("m", [1, 7, 40])
def test_bad_buffers_are_refused_before_a_launch(type_id, m):
    """Rows and norm weights are read as 16-byte vectors: other addresses, NULL and wrong sizes are errors of the host, with
    and without norm and residual, whatever kernel the batch would take."""
    import torch

    from joshua_b200 import _lib
    from joshua_b200.qtensor import QTensor

    L, k, n = _lib.lib(), 512, 96
    w = QTensor.from_bytes(type_id, np.zeros(synth.tensor_bytes(type_id, n, k), np.uint8))
    x, nw, res, out = (torch.zeros(size, device="cuda") for size in (m * k + 4, k + 4, m * n, m * n))
    s = torch.cuda.current_stream().cuda_stream

    def norm(lhs, norm_w, residual, kk=k):
        return L.jq_matmul_norm_dev(w._h, m, kk, n, lhs, norm_w, 1e-5, residual, out.data_ptr(), s)

    def pair(lhs, norm_w, kk=k):
        return L.jq_matmul_swiglu_norm_dev(w._h, w._h, m, kk, n, lhs, norm_w, 1e-5, out.data_ptr(), 0.0, s)

    X, N, R = x.data_ptr(), nw.data_ptr(), res.data_ptr()
    for lhs, norm_w, residual, kk in [(X + 4, None, R, k), (X + 8, N, None, k), (X, N + 4, R, k), (X + 4, N, R, k),
                                      (None, N, R, k), (None, None, R, k), (X, N, R, 2 * k)]:
        assert norm(lhs, norm_w, residual, kk) == _lib.E_INVALID
    for lhs, norm_w, kk in [(X + 4, None, k), (X + 8, N, k), (X, N + 4, k), (None, N, k), (None, None, k), (X, N, 2 * k)]:
        assert pair(lhs, norm_w, kk) == _lib.E_INVALID
    assert norm(X, N, R) == 0 and pair(X, N) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, torch.zeros_like(out))


@pytest.mark.parametrize("m", [16, 700])
def test_pair_on_tiles_with_its_output_over_its_input(m):
    """From five rows on the gate product goes to dst and the up product to scratch: dst may be lhs (k = n), and the scratch
    that stays with the context holds m * n values beside the split activations, not twice that."""
    import torch

    from joshua_b200 import _lib
    from joshua_b200.qtensor import Context, QTensor

    L, n, ctx = _lib.lib(), 4096, Context(0)
    gate, up = (QTensor.from_bytes(synth.Q4_K, synth.random_weight(synth.Q4_K, n, n, seed), ctx) for seed in (1, 2))
    x = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m))
    s = torch.cuda.current_stream().cuda_stream
    g, u, want = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    _lib.check(L.jq_matmul_t_dev(gate._h, m, n, n, x.data_ptr(), g.data_ptr(), s))
    _lib.check(L.jq_matmul_t_dev(up._h, m, n, n, x.data_ptr(), u.data_ptr(), s))
    _lib.check(L.jq_swiglu_dev(g.data_ptr(), u.data_ptr(), m * n, 0.0, want.data_ptr(), s))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _lib.check(L.jq_matmul_swiglu_dev(gate._h, up._h, m, n, n, x.data_ptr(), x.data_ptr(), 0.0, s))
    torch.cuda.synchronize()
    # one launch for both tensors may cut k into other pieces: products differ by 3e-6 of their 2-norm, six times that at
    # most for one value; silu's slope is below 1.1
    dg, du = 2e-5 * g.square().mean().sqrt(), 2e-5 * u.square().mean().sqrt()
    assert bool(((x - want).abs() <= 1.1 * dg * u.abs() + torch.nn.functional.silu(g).abs() * du + 1.1 * dg * du).all())
    # the split is there already; allocations come in pieces of at most 32 MB
    assert free - torch.cuda.mem_get_info()[0] <= m * n * 4 + (32 << 20)
