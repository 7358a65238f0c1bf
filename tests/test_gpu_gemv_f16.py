"""The half-precision decode kernel (batches of 3 to 8 rows of Q4_K and MXFP4) against float64 products of the decoded
weights: row counts around its tiles of 16, columns that give four to 112 units a row (teams of two to eight warps, idle
warps, several stages a tile, k split over clusters of up to eight CTAs), the gate / up pair, norm and residual, activations
decades apart."""
import numpy as np
import pytest

from joshua_b200 import synth
from joshua_b200.qtensor import QMatMul, QTensor

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1024), (17, 1024), (100, 1280), (48, 1536), (4097, 2048), (33, 4096), (5000, 4096), (333, 7168), (40, 14336),
          (700, 14336), (20, 16384), (31, 28672)]


def setup(type_id, n, k, m, seed, spread=False):
    import torch

    raw = synth.random_weight(type_id, n, k, seed)
    q = QTensor.from_bytes(type_id, raw)
    w = torch.empty(n * k, device="cuda")
    q.dequantize_dev(w, two_step=False)
    x = torch.from_numpy(np.random.default_rng(seed + 1).standard_normal((m, k), dtype=np.float32)).cuda()
    if spread:  # a unit 1e4 times the others, one 1e-6 of them, a row of zeros
        x[:, :256] *= 1e4
        x[m - 1] *= 1e-6
        x[1] = 0
    return q, w.reshape(n, k).double(), x


def bound(w, x, units):
    """Terms hold 2^-22 of a unit's largest value; a group's four instructions add with truncation (2^-23 of the largest
    partial sum each), sums go on in f32: a few 2^-23 of sum |w| max|x| over each unit, and of the magnitudes added."""
    import torch

    m, k = x.shape
    ax = x.double().abs().reshape(m, units, 256)
    aw = w.abs().reshape(w.shape[0], units, 256)
    peak = torch.einsum("mu,nu->mn", ax.amax(-1), aw.sum(-1))
    return 2.0 ** -21 * peak + 1e-30


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.MXFP4])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("m", [3, 4, 5, 8])
def test_products_match_float64(type_id, shape, m):
    n, k = shape
    q, w, x = setup(type_id, n, k, m, n + k + m, spread=m == 4)
    got = QMatMul(q, n, k).forward(x)
    err = (got.double() - x.double() @ w.T).abs()
    assert bool((err <= bound(w, x, k // 256)).all()), float((err / bound(w, x, k // 256)).max())
    assert bool((QMatMul(q, n, k).forward(x) == got).all())  # the order of the sums does not depend on timing


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.MXFP4])
@pytest.mark.parametrize("shape", [(40, 1024), (1000, 2048), (333, 4096), (70, 14336)])
@pytest.mark.parametrize("m", [3, 8])
def test_norm_residual_and_pair(type_id, shape, m):
    import torch

    from joshua_b200 import _lib

    n, k = shape
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    q, w, x = setup(type_id, n, k, m, 3 * n + m)
    up, wu, _ = setup(type_id, n, k, m, 3 * n + m + 50)
    norm = torch.rand(k, device="cuda") + 0.5
    xn = x.double() * torch.rsqrt(x.double().pow(2).mean(1, keepdim=True) + 1e-6) * norm.double()
    scale = 2.0  # the f32 norm rounds its values as much again
    tol = scale * bound(w, xn.float(), k // 256)
    out = torch.randn(m, n, device="cuda")
    want = out.double() + xn @ w.T
    tol_r = tol + 2.0 ** -23 * want.abs()
    _lib.check(L.jq_matmul_norm_dev(q._h, m, k, n, x.data_ptr(), norm.data_ptr(), 1e-6, out.data_ptr(), out.data_ptr(), st))
    assert bool(((out.double() - want).abs() <= tol_r).all())
    for clamp in (0.0, 0.7):
        g, u = xn @ w.T, xn @ wu.T
        tol_u = scale * bound(wu, xn.float(), k // 256)
        if clamp:
            g, u = g.clamp(max=clamp), u.clamp(-clamp, clamp)
        s = g * torch.sigmoid(g)
        # silu changes by at most 1.1 of its argument's change
        tol_p = 1.1 * tol * u.abs() + (s.abs() + 1.1 * tol) * tol_u + 2.0 ** -20 * (s * u).abs() + 1e-30
        dst = torch.empty(m, n, device="cuda")
        _lib.check(L.jq_matmul_swiglu_norm_dev(q._h, up._h, m, k, n, x.data_ptr(), norm.data_ptr(), 1e-6, dst.data_ptr(),
                                               clamp, st))
        assert bool(((dst.double() - s * u).abs() <= tol_p).all()), float(((dst.double() - s * u).abs() / tol_p).max())


@pytest.mark.parametrize("m", [5, 8])
def test_a_result_over_its_input_splits_the_input_first(m):
    """k = n and dst = lhs, as the tile GEMM takes it: the kernel that reads lhs while it stores is passed by."""
    import torch

    from joshua_b200 import _lib

    n = 4096
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    q, w, x = setup(synth.Q4_K, n, n, m, m)
    up, wu, _ = setup(synth.Q4_K, n, n, m, m + 50)
    want = x.double() @ w.T
    pair = want * torch.sigmoid(want) * (x.double() @ wu.T)
    for call, ref in ((lambda d: L.jq_matmul_t_dev(q._h, m, n, n, d, d, st), want),
                      (lambda d: L.jq_matmul_swiglu_dev(q._h, up._h, m, n, n, d, d, 0.0, st), pair)):
        y = x.clone()
        _lib.check(call(y.data_ptr()))
        # 2-norm of the tile GEMM's error below 1e-6, three times that for a product of two and silu
        assert float((y.double() - ref).norm() / ref.norm()) <= 3e-6


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.MXFP4, synth.Q8_0, synth.Q4_0])
@pytest.mark.parametrize("m", [1, 3, 4, 6, 20])
def test_a_result_over_its_input_at_every_batch(type_id, m):
    """dst = lhs, or one row behind it, on the routes whose CTAs would read lhs while others store: the rows go through scratch.
    Plain, with norm and residual, and as a gate / up pair."""
    import torch

    from joshua_b200 import _lib

    n = 2048
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    q, w, x = setup(type_id, n, n, m, m)
    up, wu, _ = setup(type_id, n, n, m, m + 50)
    norm, res = torch.rand(n, device="cuda") + 0.5, torch.randn(m, n, device="cuda")
    xn = x.double() * torch.rsqrt(x.double().pow(2).mean(1, keepdim=True) + 1e-6) * norm.double()

    def pair(v):
        g = v @ w.T
        return g * torch.sigmoid(g) * (v @ wu.T)

    for call, ref in (
            (lambda a, d: L.jq_matmul_t_dev(q._h, m, n, n, a, d, st), x.double() @ w.T),
            (lambda a, d: L.jq_matmul_norm_dev(q._h, m, n, n, a, norm.data_ptr(), 1e-6, res.data_ptr(), d, st), xn @ w.T + res.double()),
            (lambda a, d: L.jq_matmul_norm_dev(q._h, m, n, n, a, None, 0.0, res.data_ptr(), d, st), x.double() @ w.T + res.double()),
            (lambda a, d: L.jq_matmul_swiglu_dev(q._h, up._h, m, n, n, a, d, 0.0, st), pair(x.double())),
            (lambda a, d: L.jq_matmul_swiglu_norm_dev(q._h, up._h, m, n, n, a, norm.data_ptr(), 1e-6, d, 0.0, st), pair(xn))):
        for behind in (0, 1):
            buf = torch.zeros(m + 1, n, device="cuda")
            buf[:m] = x
            _lib.check(call(buf.data_ptr(), buf[behind:].data_ptr()))
            got = buf[behind:behind + m]
            # as above: 1e-6 for one product, three times that for two of them and silu
            assert float((got.double() - ref).norm() / ref.norm()) <= 3e-6


@pytest.mark.parametrize("k", [1280, 4096, 14336])
@pytest.mark.parametrize("m", [3, 4])
def test_rows_of_one_sign_are_as_exact_in_four_columns_as_in_eight(k, m):
    """Q4_K weights of mean zero are a difference of two large sums for positive rows.  Up to four rows first and second terms
    have columns of their own, so fewer bits are cut off than where they share one: the error of the same rows among eight is
    the bound, a tenth more for the sample.  (Second terms of the minima beside the first ones gave 1.7 to 4 times as much.)"""
    import torch

    n, rng = 512, np.random.default_rng(k)
    raw = rng.integers(0, 256, (n * k // 256, 144), dtype=np.uint8)
    raw[:, 8:12] = raw[:, 4:8]                 # minima = the scales, times 7.5: the middle of the codes
    raw[:, 12:16] = (raw[:, 12:16] & 15) * 17
    d = rng.uniform(0.5, 1.5, raw.shape[0]).astype(np.float16).astype(np.float32) * np.float32(2.0 ** -13)
    raw[:, 0:2] = d.astype(np.float16).view(np.uint8).reshape(-1, 2)
    raw[:, 2:4] = (d * 7.5).astype(np.float16).view(np.uint8).reshape(-1, 2)
    q = QTensor.from_bytes(synth.Q4_K, raw.reshape(-1))
    w = torch.empty(n * k, device="cuda")
    q.dequantize_dev(w, two_step=False)
    lin, total = QMatMul(q, n, k), {m: 0.0, 8: 0.0}
    for seed in range(8):
        x = torch.from_numpy(np.abs(np.random.default_rng(seed).standard_normal((8, k), dtype=np.float32)) + 1).cuda()
        ref = x[:m].double() @ w.reshape(n, k).double().T
        for rows in total:
            total[rows] += float((lin.forward(x[:rows])[:m].double() - ref).square().sum())
    assert total[m] <= 1.1 ** 2 * total[8]


def kernels_of(call):
    """Names of the kernels that a call launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return [e.key for e in p.key_averages() if "_kernel" in e.key]


@pytest.mark.parametrize("type_id,n,k,m,mine", [
    (synth.Q4_K, 100, 1280, 3, True), (synth.Q4_K, 100, 1280, 8, True), (synth.Q4_K, 700, 14336, 8, True),
    (synth.Q4_K, 100, 1024, 5, True), (synth.Q4_K, 100, 768, 5, False), (synth.Q4_K, 100, 1280, 2, False),
    (synth.Q4_K, 100, 1280, 9, False), (synth.MXFP4, 48, 1536, 3, True), (synth.MXFP4, 48, 1536, 8, True),
    (synth.MXFP4, 100, 1280, 3, False), (synth.MXFP4, 40, 14336, 4, True), (synth.MXFP4, 40, 14336, 5, False),
    (synth.Q8_0, 100, 1280, 4, False)])
def test_the_route_by_type_columns_and_rows(type_id, n, k, m, mine):
    q, _, x = setup(type_id, n, k, m, 1)
    names = kernels_of(lambda: QMatMul(q, n, k).forward(x))
    assert any("gemv_f16_kernel" in v for v in names) == mine, names
    assert names


@pytest.mark.parametrize("type_id,k", [(synth.Q4_K, 1280), (synth.Q4_K, 4096), (synth.Q4_K, 14336), (synth.MXFP4, 1536),
                                       (synth.MXFP4, 4096)])
@pytest.mark.parametrize("m", [3, 4, 5, 6, 7, 8])
def test_units_and_rows_decades_apart(type_id, k, m):
    """Both layouts of the terms: a unit 1e4 times the others, one 1e-6 of them, a row 1e-6 of the others, a row of zeros."""
    n = 100
    q, w, x = setup(type_id, n, k, m, k + m)
    x[:, :256] *= 1e4
    x[:, 512:768] *= 1e-6
    x[m - 1] *= 1e-6
    x[1] = 0
    got = QMatMul(q, n, k).forward(x)
    err = (got.double() - x.double() @ w.T).abs()
    assert bool((err <= bound(w, x, k // 256)).all()), float((err / bound(w, x, k // 256)).max())
    assert bool((got[1] == 0).all())


def test_a_result_over_its_input_under_capture():
    """The copy's scratch is the stream's, and a capture cannot allocate it: refused with nothing launched on a stream that has
    none, captured and replayed on one that has run the call before."""
    import torch

    from joshua_b200 import _lib
    from joshua_b200.qtensor import Context

    L, n, m = _lib.lib(), 1024, 3
    raw, ctx = synth.random_weight(synth.Q4_K, n, n, 9), Context(0)
    q = QTensor.from_bytes(synth.Q4_K, raw, ctx)
    w = torch.empty(n * n, device="cuda")
    q.dequantize_dev(w, two_step=False)
    x = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    y, st = x.clone(), torch.cuda.Stream()
    torch.cuda.synchronize()
    refused, graph = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    call = lambda: L.jq_matmul_t_dev(q._h, m, n, n, y.data_ptr(), y.data_ptr(), st.cuda_stream)
    with torch.cuda.stream(st):
        with torch.cuda.graph(refused, stream=st):
            assert call() == _lib.E_INVALID
            y.mul_(2.0)  # the capture goes on
        _lib.check(call())
        with torch.cuda.graph(graph, stream=st):
            _lib.check(call())
        y.copy_(x)
        refused.replay()
        graph.replay()
        st.synchronize()
    want = 2.0 * x.double() @ w.reshape(n, n).double().T
    assert float((y.double() - want).norm() / want.norm()) <= 1e-6
    del refused, graph
