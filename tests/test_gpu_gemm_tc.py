"""The tensor-core tile GEMMs (prefill and batched decode, from five rows on) against the oracle."""
import numpy as np
import pytest

import oracle
from joshua_b200 import synth
from joshua_b200.qtensor import QTensor
from tests.gpu_util import assert_close, bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tc_ctx():
    """A context without slices of the decode kernel: what the f16 tiles do not take runs on the TF32 tile GEMM (by default
    batches of up to 64 of those go in slices of eight rows)."""
    import os

    from joshua_b200.qtensor import Context

    old = os.environ.get("JQ_SLICED_MAX_M")
    os.environ["JQ_SLICED_MAX_M"] = "0"
    try:
        ctx = Context(0)
    finally:
        if old is None:
            del os.environ["JQ_SLICED_MAX_M"]
        else:
            os.environ["JQ_SLICED_MAX_M"] = old
    return ctx

CASES = [
    (synth.Q4_K, (9, 256, 16)), (synth.Q4_K, (16, 512, 128)), (synth.Q4_K, (33, 768, 130)),
    (synth.Q4_K, (64, 4096, 256)), (synth.Q4_K, (100, 2048, 768)), (synth.Q4_K, (512, 4096, 384)),
    (synth.Q4_K, (300, 1024, 77)), (synth.Q8_0, (32, 4096, 512)), (synth.Q8_0, (129, 512, 200)),
    (synth.Q2_K, (40, 1024, 129)), (synth.Q2_K, (256, 7680, 128)), (synth.IQ2_XXS, (17, 1024, 23)),
    (synth.IQ2_XXS, (128, 7168, 256)), (synth.MXFP4, (16, 2048, 300)), (synth.MXFP4, (257, 7168, 128)),
    (synth.MXFP4, (12, 96, 40)),
]


@pytest.mark.parametrize("type_id,mkn", CASES)
def test_matches_oracle(type_id, mkn, tc_ctx):
    m, k, n = mkn
    raw = synth.random_weight(type_id, n, k, seed=n + k)
    lhs = synth.random_activations(m, k, seed=m)
    q = QTensor.from_bytes(type_id, raw, tc_ctx)
    got = q.matmul_t(mkn, lhs)
    want = oracle.matmul_t(type_id, mkn, lhs, raw)
    assert_close(got, want, what=f"{synth.NAMES[type_id]} {mkn}")
    assert np.array_equal(bits(got), bits(q.matmul_t(mkn, lhs)))  # run-to-run identical


def test_assigns_and_leaves_neighbours_alone(tc_ctx):
    m, k, n = 20, 512, 70
    raw = synth.random_weight(synth.Q4_K, n, k, seed=1)
    lhs = synth.random_activations(m, k, seed=2)
    q = QTensor.from_bytes(synth.Q4_K, raw, tc_ctx)
    dirty = np.full((m, n), 123.75, dtype=np.float32)
    q.matmul_t((m, k, n), lhs, dst=dirty)
    assert_close(dirty, oracle.matmul_t(synth.Q4_K, (m, k, n), lhs, raw))


@pytest.mark.parametrize("type_id,mkn", [(synth.Q4_K, (9, 256, 16)), (synth.Q4_K, (20, 4096, 130)), (synth.Q8_0, (64, 2048, 96)),
                                         (synth.MXFP4, (33, 1024, 40)), (synth.IQ2_XXS, (17, 1024, 23)), (synth.Q2_K, (40, 1024, 129))])
def test_sliced_batches_match_oracle(type_id, mkn):
    """Batches 9..64 through the default context: f16 tiles of 16 and 32 rows (what still goes in slices: OLDER below)."""
    m, k, n = mkn
    raw = synth.random_weight(type_id, n, k, seed=n + k)
    lhs = synth.random_activations(m, k, seed=m)
    q = QTensor.from_bytes(type_id, raw)
    got = q.matmul_t(mkn, lhs)
    assert_close(got, oracle.matmul_t(type_id, mkn, lhs, raw), what=f"{synth.NAMES[type_id]} {mkn} sliced")
    assert np.array_equal(bits(got), bits(q.matmul_t(mkn, lhs)))


def _edge_blocks(type_id, n, k, kind):
    """Random blocks whose scales sit at an edge of the tile GEMM's per-window factors."""
    raw = synth.random_weight(type_id, n, k, seed=n + k).reshape(-1, synth.BLOCK[type_id][1]).copy()
    rng = np.random.default_rng(5)

    def put(offset, values):
        raw[:, offset:offset + 2] = np.asarray(values, np.float16).view(np.uint8).reshape(-1, 2)

    blocks = raw.shape[0]
    if type_id in (synth.Q4_K, synth.Q2_K):
        at = 0 if type_id == synth.Q4_K else 80
        if kind == "minima":   # dmin from nothing to far above d, and d = 0
            put(at, np.where(rng.random(blocks) < 0.2, 0.0, 10.0 ** rng.uniform(-6, -1, blocks)))
            put(at + 2, np.where(rng.random(blocks) < 0.2, 0.0, 10.0 ** rng.uniform(-6, 2, blocks)))
        else:                  # negative and zero scales
            put(at, rng.choice([-0.01, 0.0, 0.02, 6e-8], blocks))
            put(at + 2, rng.choice([-0.01, 0.0, 0.05], blocks))
    elif type_id == synth.MXFP4:
        raw[:, 0] = rng.integers(90, 150, blocks) if kind == "minima" else rng.choice([0, 1, 100, 127, 255], blocks)
    else:
        put(0, np.where(rng.random(blocks) < 0.2, 0.0, 10.0 ** rng.uniform(-7, 1, blocks)))
    return raw.reshape(-1)


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.Q2_K, synth.Q8_0, synth.IQ2_XXS, synth.MXFP4])
@pytest.mark.parametrize("mkn,kind", [((9, 512, 16), "minima"), ((33, 2560, 130), "minima"), ((129, 1536, 257), "signs"),
                                      ((65, 7168, 128), "minima"), ((64, 512, 600), "signs")])
def test_scales_and_rows_at_the_edges(type_id, mkn, kind, tc_ctx):
    """The f16 terms of the tile GEMM against float64: block scales and minima decades apart inside a window, rows of lhs
    from 1e-30 to 1e30 and rows of zeros, one to four CTAs along k.  Bound: at most 48 truncating additions of 2^-23 per
    window and terms good to 2^-22, so 48 * 2^-23 + 2^-21 < 7e-6 of the sum of the terms' absolute values; a term below
    2^-35 of its window's largest may go missing, inside the same bound."""
    m, k, n = mkn
    raw = _edge_blocks(type_id, n, k, kind)
    lhs = synth.random_activations(m, k, seed=m).reshape(m, k).astype(np.float64)
    lhs *= 10.0 ** np.random.default_rng(1).integers(-30, 31, m)[:, None]
    lhs[m // 2] = 0.0
    lhs = lhs.astype(np.float32)
    got = QTensor.from_bytes(type_id, raw, tc_ctx).matmul_t(mkn, lhs).astype(np.float64)
    w = oracle.dequantize(type_id, raw).reshape(n, k).astype(np.float64)
    x = lhs.astype(np.float64)
    parts = [w]
    if type_id in (synth.Q4_K, synth.Q2_K):   # the codes' and the minima's terms are summed apart
        at, parts = (0 if type_id == synth.Q4_K else 80), []
        for gone in (at, at + 2):
            blk = raw.reshape(-1, synth.BLOCK[type_id][1]).copy()
            blk[:, gone:gone + 2] = 0
            parts.append(oracle.dequantize(type_id, blk.reshape(-1)).reshape(n, k).astype(np.float64))
    want, size = x @ w.T, np.abs(x) @ sum(np.abs(p) for p in parts).T
    inside = size < 1e38   # f32 results
    assert np.all(np.abs(got - want)[inside] <= 7e-6 * size[inside] + 1e-42)


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.Q2_K, synth.Q8_0, synth.IQ2_XXS, synth.MXFP4, synth.Q6_K])
@pytest.mark.parametrize("m,n", [(9, 130), (20, 70), (33, 300), (70, 129)])
@pytest.mark.parametrize("outlier", [1e3, 1e6])
def test_one_large_value_costs_the_others_no_bits(type_id, m, n, outlier):
    """Rows of N(0, 1) with one value far above the rest, whose weights are zeros: nothing of it is in the result, all of it
    is in the activations' scale.  The split keeps 2^-39 of the largest value of the same 256 columns, 2e-6 here, for
    those columns alone; a window's sum is at most 48 additions that truncate in the last of 24 places, half of it on
    average: 48 * 2^-24 = 3e-6 of the result's 2-norm.  Types with blocks of 32 columns have other weights beside the zeros."""
    k = 4096
    if type_id == synth.Q8_0:
        m = max(m, 17)   # below, the type runs on the decode kernel
    elems, nbytes = synth.BLOCK[type_id]
    raw = synth.random_weight(type_id, n, k, seed=n).reshape(n, k // elems, nbytes).copy()
    raw[:, 1024 // elems] = 0
    raw = raw.reshape(-1)
    lhs = np.random.default_rng(m).standard_normal((m, k)).astype(np.float32)
    lhs[:, 1030] = outlier
    got = QTensor.from_bytes(type_id, raw).matmul_t((m, k, n), lhs).astype(np.float64)
    want = lhs.astype(np.float64) @ oracle.dequantize(type_id, raw).reshape(n, k).astype(np.float64).T
    assert np.linalg.norm(got - want) <= 3e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("type_id,kind", [(synth.MXFP4, "blocks"), (synth.Q8_0, "blocks"), (synth.Q4_K, "codes"), (synth.Q2_K, "codes"),
                                          (synth.Q4_K, "minima"), (synth.Q2_K, "minima")])
@pytest.mark.parametrize("m,n,k", [(9, 130, 1024), (20, 70, 4096), (40, 300, 1024), (70, 129, 4096), (130, 19000, 512)])
def test_small_weights_beside_large_ones_keep_their_bits(type_id, kind, m, n, k):
    """Scales further apart than f16 reaches inside one factor, and activations that are zero where the large ones are: the
    result is the small ones' alone.  Blocks: the first of every window is 2^50 (MXFP4) or 2^33 (Q8_0) above the rest.
    Codes: dmin = 2^32 d, only columns with a minimum of 0 count.  Minima: dmin = 2^-12 d, only columns with a code of 0
    count.  Exact tiles, 128-row tiles, one and several CTAs along k.  The bound is that of the test above."""
    elems, nbytes = synth.BLOCK[type_id]
    if type_id == synth.Q8_0:
        m = max(m, 17)
    raw = synth.random_weight(type_id, n, k, seed=n).reshape(n, k // elems, nbytes).copy()
    lhs = np.random.default_rng(m).standard_normal((m, k)).astype(np.float32)
    cols = np.arange(k) % 256

    def f16(v):
        return np.float16(v).view(np.uint16).reshape(1).view(np.uint8)

    if kind == "blocks":
        lhs[:, cols < 32] = 0
        if type_id == synth.MXFP4:
            raw[:, :, 0] = 100 + raw[:, :, 0] % 8
            raw[:, ::8, 0] = 158
        else:
            raw[:, :, :2] = f16(2.0 ** -20)
            raw[:, ::8, :2] = f16(2.0 ** 13)
    else:
        lhs[:, cols >= 32] = 0
        at = 0 if type_id == synth.Q4_K else 80
        raw[:, :, at:at + 2] = f16(2.0 ** -20 if kind == "codes" else 2.0 ** 4)
        raw[:, :, at + 2:at + 4] = f16(2.0 ** 12 if kind == "codes" else 2.0 ** -8)
        if kind == "codes" and type_id == synth.Q4_K:
            raw[:, :, 8] &= 0xC0
        elif kind == "codes":
            raw[:, :, 0:2] &= 0x0F
        elif type_id == synth.Q4_K:
            raw[:, :, 16:48] &= 0xF0
        else:
            raw[:, :, 16:48] &= 0xFC
    got = QTensor.from_bytes(type_id, raw.reshape(-1)).matmul_t((m, k, n), lhs).astype(np.float64)
    want = lhs.astype(np.float64) @ oracle.dequantize(type_id, raw.reshape(-1)).reshape(n, k).astype(np.float64).T
    assert np.linalg.norm(got - want) <= 3e-6 * np.linalg.norm(want)


# Shapes the f16 tiles leave to the older routes: rows that are no whole number of windows (Q8_0, MXFP4: 256 columns,
# IQ2_XXS: 512) on the TF32 kernel, all its tile widths and ragged edges; Q8_0 of 9 to 16 rows and IQ2_XXS batches in slices.
OLDER = [(t, (m, 4128, n)) for t in (synth.Q8_0, synth.MXFP4) for m, n in ((20, 130), (40, 257), (65, 130), (130, 257))] + \
        [(synth.IQ2_XXS, (m, k, n)) for k in (768, 2304) for m, n in ((20, 130), (65, 257), (130, 130))] + \
        [(synth.Q8_0, (m, 2048, 257)) for m in (9, 12, 16)]


@pytest.mark.parametrize("type_id,mkn", OLDER)
@pytest.mark.parametrize("sliced", [True, False])
def test_routes_the_f16_tiles_leave_to_others(type_id, mkn, sliced, tc_ctx):
    """The default context and the one without slices, against the oracle, run to run identical."""
    m, k, n = mkn
    raw = synth.random_weight(type_id, n, k, seed=n + k)
    lhs = synth.random_activations(m, k, seed=m)
    q = QTensor.from_bytes(type_id, raw) if sliced else QTensor.from_bytes(type_id, raw, tc_ctx)
    got = q.matmul_t(mkn, lhs)
    assert_close(got, oracle.matmul_t(type_id, mkn, lhs, raw), what=f"{synth.NAMES[type_id]} {mkn}")
    assert np.array_equal(bits(got), bits(q.matmul_t(mkn, lhs)))


@pytest.mark.parametrize("mkn,kind", [((17, 512, 16), "minima"), ((40, 512, 600), "signs")])
def test_scales_at_the_edges_of_q8_0_tiles(mkn, kind, tc_ctx):
    """As test_scales_and_rows_at_the_edges, with the row counts from which Q8_0 takes the f16 tiles."""
    test_scales_and_rows_at_the_edges(synth.Q8_0, mkn, kind, tc_ctx)


@pytest.mark.parametrize("type_id", [synth.Q8_0, synth.MXFP4, synth.IQ2_XXS, synth.Q6_K, synth.Q2_K])
@pytest.mark.parametrize("m,n", [(20, 70), (70, 130), (200, 96)])
def test_slices_that_start_on_a_word_boundary(type_id, m, n):
    """A slice of blocks may start anywhere in its tensor: four bytes past an eight-byte boundary here, two past a word for
    the second one (which takes the older routes).  The same blocks in a tensor of their own give the reference."""
    k, (elems, nbytes) = 1024, synth.BLOCK[type_id]
    count = n * (k // elems)
    lhs = synth.random_activations(m, k, seed=m)
    whole = synth.random_weight(type_id, n + 8, k, seed=n)
    parent = QTensor.from_bytes(type_id, whole)
    for want_mod in (4, 2):
        skip = next((s for s in range(1, 33) if s * nbytes % 8 == want_mod), None)
        if skip is None:
            continue
        raw = whole[skip * nbytes:(skip + count) * nbytes]
        got = parent.slice_blocks(skip, count).matmul_t((m, k, n), lhs).astype(np.float64).reshape(m, n)
        want = lhs.reshape(m, k).astype(np.float64) @ oracle.dequantize(type_id, raw).reshape(n, k).astype(np.float64).T
        assert np.linalg.norm(got - want) <= 3e-6 * np.linalg.norm(want)   # the sums' bound of the tests above


@pytest.mark.parametrize("m", [5, 8, 9, 40, 100])
def test_a_stream_under_capture_without_scratch_takes_the_older_route(m):
    """The tile GEMM needs scratch; a capture on a stream that has none yet must not allocate, so the decode kernel runs
    there (its planes fit shared memory at this k) as it did before the tiles took these batches."""
    import torch

    from joshua_b200.qtensor import Context

    n, k = 384, 1024
    raw = synth.random_weight(synth.Q4_K, n, k, seed=6)
    lhs = synth.random_activations(m, k, seed=7).reshape(m, k)
    want = oracle.matmul_t(synth.Q4_K, (m, k, n), lhs, raw)
    x, out = torch.from_numpy(lhs).cuda(), torch.zeros(m, n, device="cuda")
    QTensor.from_bytes(synth.Q4_K, raw).matmul_t((m, k, n), lhs)   # kernels of this process are loaded
    warm = torch.cuda.Stream()
    with torch.cuda.stream(warm):
        for rows in range(1, 9):                                    # every row-count variant of the decode kernel
            QTensor.from_bytes(synth.Q4_K, raw, Context(0)).matmul_t_dev((min(rows, m), k, n), x, out)
    torch.cuda.synchronize()
    q = QTensor.from_bytes(synth.Q4_K, raw, Context(0))
    s = torch.cuda.Stream()
    out.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        q.matmul_t_dev((m, k, n), x, out)
    g.replay()
    torch.cuda.synchronize()
    assert_close(out.cpu().numpy(), want)


@pytest.mark.parametrize("type_id,m", [(synth.Q4_K, 8), (synth.Q4_K, 16), (synth.Q8_0, 20), (synth.Q8_0, 12), (synth.MXFP4, 40)])
def test_a_graph_survives_larger_calls_on_its_stream(type_id, m):
    """A captured product and a captured gate / up pair hold addresses of the stream's scratch.  Larger eager calls on
    the stream outgrow every role of it; replays then still give the captured batch's values, bit for bit."""
    import torch

    from joshua_b200 import _lib
    from joshua_b200.qtensor import Context

    n, k, big = 384, 4096, 700
    L, ctx = _lib.lib(), Context(0)
    raw = [synth.random_weight(type_id, n, k, seed=s) for s in (1, 2)]
    q = [QTensor.from_bytes(type_id, r, ctx) for r in raw]
    lhs = synth.random_activations(big, k, seed=3).reshape(big, k)
    x, nw = torch.from_numpy(lhs).cuda(), torch.ones(k, device="cuda")
    s = torch.cuda.Stream()

    def calls(rows, out):
        q[0].matmul_t_dev((rows, k, n), x, out[0], stream=s.cuda_stream)
        _lib.check(L.jq_matmul_swiglu_norm_dev(q[0]._h, q[1]._h, rows, k, n, x.data_ptr(), nw.data_ptr(), 1e-5,
                                               out[1].data_ptr(), 0.0, s.cuda_stream))
        _lib.check(L.jq_matmul_norm_dev(q[0]._h, rows, k, n, x.data_ptr(), nw.data_ptr(), 1e-5, out[1].data_ptr(),
                                        out[2].data_ptr(), s.cuda_stream))

    small, large = torch.zeros(3, m, n, device="cuda"), torch.zeros(3, big, n, device="cuda")
    torch.cuda.synchronize()
    calls(m, small)
    s.synchronize()
    want = small.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        calls(m, small)
    for rows in (200, big):
        calls(rows, large)
    s.synchronize()
    junk = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(64)]   # what was freed gets new owners
    for _ in range(2):
        small.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            g.replay()
        torch.cuda.synchronize()
        assert torch.equal(small, want)
        calls(big, large)
    assert all(bool(torch.isnan(j).all()) for j in junk)
    assert_close(small[0].cpu().numpy(), oracle.matmul_t(type_id, (m, k, n), lhs[:m], raw[0]))


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.Q8_0, synth.Q2_K, synth.Q6_K])
@pytest.mark.parametrize("m", [5, 7, 16, 17, 33, 64, 65, 128, 130])
def test_norm_and_residual_inside_the_tile_gemm(type_id, m):
    """dst = residual + rmsnorm(x) . W^T with dst = residual, over the tile widths and both sides of their edges, k split
    over a cluster (n = 96 is one tile), against float64.  Bound as in the test above, plus the norm's own rounding."""
    import torch

    from joshua_b200 import _lib

    n, k = 96, 4608 if type_id != synth.Q6_K else 4096
    raw = synth.random_weight(type_id, n, k, seed=11)
    w = oracle.dequantize(type_id, raw).reshape(n, k).astype(np.float64)
    rng = np.random.default_rng(m)
    x, nw, res = rng.standard_normal((m, k)), rng.uniform(0.5, 1.5, k), rng.standard_normal((m, n))
    x, nw, res = (v.astype(np.float32) for v in (x, nw, res))
    q = QTensor.from_bytes(type_id, raw)
    xd, nd, rd = (torch.from_numpy(v).cuda() for v in (x, nw, res))
    _lib.check(_lib.lib().jq_matmul_norm_dev(q._h, m, k, n, xd.data_ptr(), nd.data_ptr(), 1e-5, rd.data_ptr(), rd.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    x64 = x.astype(np.float64)
    xn = x64 / np.sqrt((x64 ** 2).mean(1, keepdims=True) + 1e-5) * nw.astype(np.float64)
    want = res + xn @ w.T
    size = np.abs(res) + np.abs(xn) @ np.abs(w.T) * (3 if type_id in (synth.Q4_K, synth.Q2_K) else 1)
    assert np.all(np.abs(rd.cpu().numpy() - want) <= 8e-6 * size)
