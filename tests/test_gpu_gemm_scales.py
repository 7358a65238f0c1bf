"""The tile GEMM's windows (256 columns) with scales of their own: the split kernel says so by the sign of a row's scale,
which the product's kernel may not read before that one is through."""
import numpy as np
import pytest

from joshua_b200 import synth
from joshua_b200.qtensor import QMatMul, QTensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("type_id", [synth.Q4_K, synth.Q2_K, synth.MXFP4, synth.IQ2_XXS, synth.Q8_0, synth.Q6_K])
@pytest.mark.parametrize("m", [20, 200])
def test_scales_of_windows_hold_from_the_first_call(type_id, m):
    """Calls on one scratch in turn: no window far below its row's largest value, then one in every row."""
    import torch

    n, k = 512, 14336
    q = QTensor.from_bytes(type_id, synth.random_weight(type_id, n, k, 1))
    w = torch.empty(n * k, device="cuda")
    q.dequantize_dev(w, two_step=False)
    w, lin = w.reshape(n, k).double(), QMatMul(q, n, k)
    g = torch.Generator(device="cuda").manual_seed(m)
    x = [torch.randn(m, k, device="cuda", generator=g) for _ in range(40)]
    for i in range(1, len(x), 2):
        at = torch.randint(0, k // 256, (m,), device="cuda", generator=g)
        x[i].reshape(m, k // 256, 256)[torch.arange(m, device="cuda"), at] *= 2.0 ** -12
    got = [lin.forward(v) for v in x]
    for v, y in zip(x, got):
        ref = v.double() @ w.T
        # two f16 terms of both operands, truncated sums of 256 columns: below 1e-6 of a row's norm for N(0, 1) rows, times
        # four for weights of one sign; one window counted 2^12 times is some hundreds
        assert float(((y.double() - ref).norm(dim=1) / ref.norm(dim=1)).max()) <= 4e-6 * float(w.abs().mean() / w.std() + 1)
