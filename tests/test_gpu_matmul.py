"""matmul_t through the C ABI against the oracle: the reference's own shapes and error cases."""
import numpy as np
import pytest

import oracle
from joshua_b200 import synth
from joshua_b200.qtensor import QTensor, QMatMul
from joshua_b200._lib import JoshuaB200Error
from tests.gpu_util import assert_close, bits
from tests.test_oracle_iq2xxs import fixture_rhs, lhs_pattern
from tests.test_oracle_mxfp4 import spread_rhs

pytestmark = pytest.mark.gpu

# (m, k, n) of the reference's unit tests (src/kquant_dot.rs:893-929, src/quant_matmul.rs:498-533,
# src/iq2xxs.rs:761-873, src/mxfp4.rs:354-423): odd n, m off the 4-row tile.
SMALL = {
    synth.Q8_0: [(1, 256, 40), (3, 512, 17), (1, 256, 64), (5, 128, 9), (3, 256, 24), (2, 256, 8)],
    synth.Q2_K: [(1, 256, 40), (3, 512, 11), (5, 768, 9), (3, 256, 24), (2, 256, 8)],
    synth.Q4_K: [(1, 256, 40), (3, 512, 13), (4, 768, 25), (3, 256, 24), (2, 256, 8)],
    synth.IQ2_XXS: [(3, 512, 7), (3, 1024, 11), (4, 1024, 23)],
    synth.MXFP4: [(2, 64, 3), (1, 32, 2), (4, 1024, 23), (2, 64, 6)],
}
# decode shapes of the benchmark configurations, and batches up to and past the 8-row tile
MODEL = [
    (synth.Q4_K, (1, 4096, 4096)), (synth.Q8_0, (1, 4096, 4096)), (synth.Q2_K, (1, 4096, 4096)),
    (synth.Q2_K, (1, 7680, 2048)), (synth.Q4_K, (1, 2048, 7680)), (synth.Q8_0, (32, 4096, 4096)),
    (synth.Q4_K, (8, 4096, 1024)), (synth.Q4_K, (1, 14336, 512)), (synth.Q4_K, (7, 2048, 768)),
    (synth.Q4_K, (13, 768, 2048)), (synth.IQ2_XXS, (1, 7168, 2048)), (synth.IQ2_XXS, (5, 2048, 7168)),
    (synth.MXFP4, (1, 7168, 2048)), (synth.MXFP4, (16, 2048, 7168)), (synth.Q8_0, (2, 7168, 1536)),
]


@pytest.mark.parametrize("type_id,mkn", [(t, c) for t, cs in SMALL.items() for c in cs] + MODEL)
def test_matmul_matches_oracle(type_id, mkn):
    m, k, n = mkn
    raw = synth.random_weight(type_id, n, k, seed=n + k)
    lhs = synth.random_activations(m, k, seed=m)
    got = QTensor.from_bytes(type_id, raw).matmul_t(mkn, lhs)
    want = oracle.matmul_t(type_id, mkn, lhs, raw)
    assert_close(got, want, what=f"{synth.NAMES[type_id]} {mkn}")


@pytest.mark.parametrize("type_id", synth.GENERIC_TYPES)
@pytest.mark.parametrize("mkn", [(1, 256, 40), (3, 512, 13), (8, 1024, 64), (40, 512, 24), (1, 4096, 256)])
def test_generic_path_types_match_oracle(type_id, mkn):
    """The block types the reference serves by decoding a row and dotting it (src/quant_matmul.rs:228-249): here
    the exact-decode float kernel, any batch."""
    m, k, n = mkn
    raw = synth.random_weight(type_id, n, k, seed=n + k)
    lhs = synth.random_activations(m, k, seed=m)
    q = QTensor.from_bytes(type_id, raw)
    got = q.matmul_t(mkn, lhs)
    assert_close(got, oracle.matmul_t(type_id, mkn, lhs, raw), what=f"{synth.NAMES[type_id]} {mkn}")
    assert np.array_equal(bits(got), bits(q.matmul_t(mkn, lhs)))      # run-to-run bit equality


@pytest.mark.parametrize("mkn", [(1, 256, 1), (2, 512, 17), (4, 4096, 33), (8, 4352, 16), (3, 14336, 31), (5, 8192, 130), (9, 512, 40),
                                 (70, 768, 47)])
@pytest.mark.parametrize("skip", [0, 1])
def test_q6_k_decode_kernel(mkn, skip):
    """Q6_K on the decode kernel: one unit to several ring chunks per row, every row-count variant, batches in slices,
    and tensors that start on an odd multiple of two bytes (a slice of `skip` blocks; blocks are 210 bytes).  The bound
    is the activation split's 6.1e-8 of a unit's largest value per term and f32 sums of k / 256 units: 1e-5 of the
    terms' 2-norm leaves a factor of ten."""
    m, k, n = mkn
    raw = synth.random_weight(synth.Q6_K, n + 1, k, seed=n + k)
    lhs = synth.random_activations(m, k, seed=m)
    rows = raw[skip * 210:skip * 210 + n * (k // 256) * 210]
    got = QTensor.from_bytes(synth.Q6_K, raw).slice_blocks(skip, n * (k // 256)).matmul_t(mkn, lhs)
    w = oracle.dequantize(synth.Q6_K, rows).reshape(n, k).astype(np.float64)
    want = lhs.astype(np.float64).reshape(m, k) @ w.T
    scale = np.sqrt((lhs.astype(np.float64).reshape(m, k) ** 2) @ (w.T ** 2))
    assert np.all(np.abs(got - want) <= 1e-5 * scale + 1e-30)


def test_iq2xxs_golden_block_fixture():
    for mkn, mult in [((3, 512, 7), 7919), ((3, 1024, 11), 7919), ((4, 1024, 23), 104729)]:
        m, k, n = mkn
        rhs, lhs = fixture_rhs(k, n), lhs_pattern(m, k, mult)
        got = QTensor.from_bytes(synth.IQ2_XXS, rhs).matmul_t(mkn, lhs)
        assert_close(got, oracle.matmul_t(synth.IQ2_XXS, mkn, lhs, rhs), tol=1e-4)


def test_mxfp4_reference_fixtures():
    m, k, n = 2, 64, 3
    rhs = spread_rhs(n, k // 32)
    lhs = (np.arange(m * k, dtype=np.float32) % 7.0 - 3.0).reshape(m, k)
    got = QTensor.from_bytes(synth.MXFP4, rhs).matmul_t((m, k, n), lhs)
    assert np.all(np.abs(got - oracle.matmul_t(synth.MXFP4, (m, k, n), lhs, rhs)) < 1e-3)
    # a per-expert slice of a borrowed tensor (src/mmap_tensor.rs:923-954): rows 3..6 of a 6-row tensor
    full = spread_rhs(6, 2)
    q = QTensor.from_bytes(synth.MXFP4, full)
    part = q.slice_blocks(3 * 2, 3 * 2)
    got = part.matmul_t((m, k, 3), lhs)
    want = oracle.matmul_t(synth.MXFP4, (m, k, 3), lhs, full[3 * 2 * 17:])
    assert np.all(np.abs(got - want) < 1e-3)


@pytest.mark.parametrize("type_id", list(SMALL))
def test_assigns_into_dirty_destination_and_is_deterministic(type_id):
    elems, _ = synth.BLOCK[type_id]
    m, k, n = 3, 4 * elems if elems == 256 else 256, 19
    raw = synth.random_weight(type_id, n, k, seed=2)
    lhs = synth.random_activations(m, k, seed=3)
    q = QTensor.from_bytes(type_id, raw)
    fresh = q.matmul_t((m, k, n), lhs)
    dirty = np.full((m, n), 123.75, dtype=np.float32)
    q.matmul_t((m, k, n), lhs, dst=dirty)
    assert np.array_equal(bits(fresh), bits(dirty))
    assert np.array_equal(bits(fresh), bits(q.matmul_t((m, k, n), lhs)))


@pytest.mark.parametrize("type_id", list(SMALL))
def test_shape_errors_and_noops(type_id):
    elems, nbytes = synth.BLOCK[type_id]
    k = 256
    raw = synth.random_weight(type_id, 8, k, seed=0)
    q = QTensor.from_bytes(type_id, raw)
    with pytest.raises(JoshuaB200Error, match="not a multiple"):
        q.matmul_t((1, 100, 8), np.zeros(100, np.float32))
    with pytest.raises(JoshuaB200Error, match="blocks, expected"):
        q.matmul_t((1, k, 7), np.zeros(k, np.float32))
    with pytest.raises(JoshuaB200Error, match="lhs/dst sized"):
        q.matmul_t((2, k, 8), np.zeros(k, np.float32), dst_len=16)
    with pytest.raises(JoshuaB200Error, match="lhs/dst sized"):
        q.matmul_t((1, k, 8), np.zeros(k, np.float32), dst_len=7)
    assert q.matmul_t((0, k, 8), np.zeros(0, np.float32)).size == 0
    empty = QTensor.from_bytes(type_id, raw[:0])
    assert empty.matmul_t((2, k, 0), np.zeros(2 * k, np.float32)).size == 0


@pytest.mark.parametrize("type_id", [synth.IQ2_XXS, synth.MXFP4, synth.Q4_K])
def test_f16_entry(type_id):
    m, k, n = 3, 512, 21
    raw = synth.random_weight(type_id, n, k, seed=7)
    lhs16 = synth.random_activations(m, k, seed=8).astype(np.float16)
    got = QTensor.from_bytes(type_id, raw).matmul_t_f16((m, k, n), lhs16)
    want = oracle.matmul_t(type_id, (m, k, n), lhs16.astype(np.float32), raw).astype(np.float16)
    assert_close(got.astype(np.float32), want.astype(np.float32), tol=2e-3)


def test_qmatmul_forward_on_device_tensors():
    import torch

    n, k = 96, 512
    raw = synth.random_weight(synth.Q4_K, n, k, seed=4)
    mm = QMatMul.from_qtensor(QTensor.from_bytes(synth.Q4_K, raw), (n, k))
    x = torch.randn(2, 3, k, device="cuda")
    y = mm.forward(x)
    assert y.shape == (2, 3, n)
    want = oracle.matmul_t(synth.Q4_K, (6, k, n), x.reshape(6, k).cpu().numpy(), raw)
    assert_close(y.reshape(6, n).cpu().numpy(), want)
    # views and other layouts: the same values through a copy; one row; no rows; a side stream
    want = mm.forward(x)
    xt = x.transpose(0, 1)
    assert torch.equal(mm.forward(xt), want.transpose(0, 1)) and torch.equal(mm.forward(x[0, 0]), mm.forward(x[:1, :1])[0, 0])
    assert mm.forward(x[:0]).shape == (0, 3, n) and mm.forward(x.reshape(-1, k)[:, :]).shape == (6, n)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y2 = mm.forward(x)
    side.synchronize()
    assert torch.equal(y2, want)
    with pytest.raises(JoshuaB200Error):
        mm.forward(x.half())
    with pytest.raises(JoshuaB200Error):
        QMatMul.from_qtensor(QTensor.from_bytes(synth.Q4_K, raw), (n + 1, k))


def test_q6_k_takes_more_rows_than_a_grid_of_tiles():
    """A tile launch covers 65535 tiles of 32 rows of lhs; larger batches of Q6_K go through the decode kernel in slices."""
    import torch

    n, k, m = 2, 256, 65535 * 32 + 9
    raw = synth.random_weight(synth.Q6_K, n, k, seed=4)
    w = torch.from_numpy(oracle.dequantize(synth.Q6_K, raw).reshape(n, k)).cuda().double()
    x = torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    out = torch.empty(m, n, device="cuda")
    QTensor.from_bytes(synth.Q6_K, raw).matmul_t_dev((m, k, n), x, out)
    torch.cuda.synchronize()
    for a in (0, m // 2, m - 64):
        rows = x[a:a + 64].double()
        # one unit a row: 6.1e-8 of its largest value per term, f32 sums of the pieces (the bound above, per 2-norm)
        scale = ((rows ** 2) @ (w.T ** 2)).sqrt()
        assert bool(((out[a:a + 64].double() - rows @ w.T).abs() <= 1e-5 * scale).all())


@pytest.mark.parametrize("m,k", [(1, 28160), (1, 28672), (2, 13824), (2, 14336), (3, 8960), (3, 9472), (4, 7168), (5, 5632), (7, 4096),
                                 (8, 3328), (8, 3584), (8, 4096)])
def test_q8_0_planes_around_the_shared_memory_limit(m, k):
    """Q8_0 keeps up to 100 KB of activation planes in shared memory from three rows on and 96 KB below: both sides of either
    line, with a residual (fused where the planes are in shared memory).  The bound is that of the split and of f32 sums, as
    for Q6_K above."""
    import torch

    from joshua_b200 import _lib

    n = 70
    raw = synth.random_weight(synth.Q8_0, n, k, seed=m)
    x = synth.random_activations(m, k, seed=k).reshape(m, k)
    res = np.random.default_rng(m).standard_normal((m, n)).astype(np.float32)
    q = QTensor.from_bytes(synth.Q8_0, raw)
    xd, out = torch.from_numpy(x).cuda(), torch.from_numpy(res).cuda()
    _lib.check(_lib.lib().jq_matmul_norm_dev(q._h, m, k, n, xd.data_ptr(), None, 0.0, out.data_ptr(), out.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    w, x64 = oracle.dequantize(synth.Q8_0, raw).reshape(n, k).astype(np.float64), x.astype(np.float64)
    scale = np.sqrt((x64 ** 2) @ (w.T ** 2)) + np.abs(res)
    assert np.all(np.abs(out.cpu().numpy() - (res + x64 @ w.T)) <= 1e-5 * scale)
