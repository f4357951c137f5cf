"""The activation preparation of the tcgen05 path where a row is longer than one CTA keeps in registers: spread over a cluster of two to
eight CTAs at few rows, read twice at many rows, beyond eight CTAs or below 8,192 activations."""
import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [5120, 5376, 10496, 17408, 41216])
@pytest.mark.parametrize("m", [33, 100, 400, 1500])
def test_a_rows_scale_covers_all_of_it(m, k):
    """The largest magnitude of a row sits in its first, a middle or its last chunk; the others are about 2^-12 of it (2^-6 beside
    64), which a scale taken from a part of the row would carry out of fp16's range or, unscaled, below its precision.  Also a row of zeros, rows at both ends of bf16's range and a NaN.
    Weights are rounded to fp16 (2^-11 each), activations exact: 3e-3 of the norm is five times what K of them leave."""
    n, t = 70, F.Q4_0
    raw = synth.random_blocks(n, k, t, seed=k)
    packed = ops.repack_tiles(raw.cuda(), n, t).reshape(-1)
    d = torch.from_numpy(ops.build_descs([t], [n], k, 1)).cuda()
    x = synth.activations(m, k, device="cuda")
    x[:, :] *= 2.0 ** -6
    for r, c in ((0, 0), (1, k // 2), (2, k - 1), (3, 5119), (4, min(5120, k - 1))):
        x[r, c] = 64.0
    x[5] = 0
    x[6] *= 2.0 ** 90
    x[7] *= 2.0 ** -60
    x[8, k - 1] = float("nan")
    y = ops.prefill_gemm(x, packed, d, n, wtypes=[t]).double().cpu()
    assert bool(torch.isnan(y[8]).all()) and not bool(torch.isnan(torch.cat([y[:8], y[9:]])).any())
    w = torch.from_numpy(oracle.dequantize(raw.numpy(), t)).double()
    xd = x.double().cpu()
    exact, norm = xd @ w.T, ((xd ** 2) @ (w ** 2).T).sqrt()
    for rows in (slice(0, 8), slice(9, m)):
        err = (y[rows] - exact[rows]).abs() - exact[rows].abs() * 2.0 ** -8
        assert float((err / norm[rows].clamp_min(1e-300)).max()) < 3e-3
    assert ops.device_status() == 0


@pytest.mark.parametrize("m, k", [(64, 7680), (80, 7680), (33, 8192), (148, 8192), (300, 10496), (480, 8704), (592, 8704), (600, 8704), (480, 17408), (600, 17408), (672, 17408)])
def test_where_the_ctas_of_a_row_change(m, k):
    """Row counts on both sides of each step of the rule that picks them."""
    test_a_rows_scale_covers_all_of_it(m, k)
