"""The grouped kernel's fp16 form (17 to 64 rows) where its shapes end: three, four and eight column tiles, an odd number of tiles, runs of
two types, a ragged last tile, fewer k-blocks than ring stages, every way a split is reduced; and what its tables and run_info may say."""
import numpy as np
import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


def _beyond_rounding(y, exact, norm):
    """What an output is off by beyond half a bf16 ulp of the exact value, over the 2-norm of its products."""
    ulp = 2.0 ** (np.floor(np.log2(np.maximum(np.abs(exact), 1e-30))) - 7)
    return float(np.max((np.abs(y - exact) - 0.5 * ulp) / norm))


@pytest.mark.parametrize("t", sorted(F.SUPPORTED_TYPES))
@pytest.mark.parametrize("m, k, splits", [(17, 256, [1]), (24, 1280, [1, 2, 5]), (25, 2048, [3, 8]), (32, 2560, [4, 9]), (33, 512, [1, 2]), (64, 768, [3])])
def test_every_type_beside_another(t, m, k, splits):
    """A run of five tiles, three of type t (the last one of 6 rows) and two of another: their codebook tables differ.  Weights and activations enter exactly, so beyond the output rounding there are the fp32 sums: at most
    K / 256 + 17 roundings of 2^-23 (the tensor core truncates) of partial sums of a few norms, below 2^-15 of the norm here."""
    other = F.IQ2_S if t != F.IQ2_S else F.Q8_0
    types, n_outs = [t, other], [134, 100]
    raws = [synth.random_blocks(n, k, w, seed=11 * w + n) for n, w in zip(n_outs, types)]
    packed = torch.cat([ops.repack_tiles(r.cuda(), n, w).reshape(-1) for r, n, w in zip(raws, n_outs, types)])
    x = synth.activations(m, k, device="cuda")
    xd = x.double().cpu().numpy()
    w = np.concatenate([oracle.dequantize(r.numpy(), wt) for r, wt in zip(raws, types)]).astype(np.float64)
    exact, norm = xd @ w.T, np.sqrt((xd ** 2) @ (w ** 2).T)
    first = None
    for s in splits:
        d = torch.from_numpy(ops.build_descs(types, n_outs, k, s)).cuda()
        y = ops.grouped_gemm(x, packed, d, s, types, sum(n_outs))
        assert _beyond_rounding(y.double().cpu().numpy(), exact, norm) < 2.0 ** -15, (F.TYPE_NAMES[t], m, k, s)
        assert torch.equal(y, ops.grouped_gemm(x, packed, d, s, types, sum(n_outs)))          # a fixed order of the additions
    assert ops.device_status() == 0


@pytest.mark.parametrize("m", [17, 40])
def test_scales_zeros_and_non_finite_rows(m):
    """Per-block activation scales: rows of very different magnitude, a block of zeros, and a row with an infinity, which must not reach
    the other rows."""
    n, k, t = 192, 1024, F.Q5_K
    raw = synth.random_blocks(n, k, t, seed=3)
    packed = ops.repack_tiles(raw.cuda(), n, t).reshape(-1)
    d = torch.from_numpy(ops.build_descs([t], [n], k, 2)).cuda()
    x = synth.activations(m, k, device="cuda")
    x[1] *= 2.0 ** 60
    x[2] *= 2.0 ** -60
    x[3, 256:512] = 0
    x[4, :256] *= 2.0 ** 20
    x[m - 1, 700] = float("inf")
    y = ops.grouped_gemm(x, packed, d, 2, [t], n).double().cpu().numpy()
    assert not np.isfinite(y[m - 1]).any()
    xd, w = x.double().cpu().numpy()[:m - 1], oracle.dequantize(raw.numpy(), t).astype(np.float64)
    assert _beyond_rounding(y[:m - 1], xd @ w.T, np.sqrt((xd ** 2) @ (w ** 2).T)) < 2.0 ** -15


@pytest.mark.parametrize("m, split", [(17, 1), (24, 2), (32, 1), (33, 1), (64, 2), (40, 9)])
@pytest.mark.parametrize("named, tiles", [((F.IQ3_S,), (F.IQ3_S, F.IQ3_XXS)), ((F.IQ3_S,), (F.Q2_K, F.IQ3_S)), ((F.IQ3_S,), (F.IQ3_XXS, F.IQ3_XXS)),
                                          ((F.Q4_K,), (F.Q4_K, F.Q2_K)), ((F.Q8_0,), (F.IQ2_S, F.Q8_0)), ((F.Q2_K, F.IQ2_S), (F.Q2_K, F.IQ3_S)),
                                          ((F.IQ2_XXS, F.Q4_K), (F.IQ2_XS, F.Q4_K))])
def test_tiles_that_run_info_does_not_name(named, tiles, m, split):
    """A tile of a type that run_info leaves out is reported (status 2) or multiplied as what its table row says it is; never anything else
    under status 0.  (No tile that fits its stage reads or writes out of bounds, one that does not is not copied.)"""
    n, k = 64, 2560
    raws = [synth.random_blocks(n, k, t, seed=5 + t) for t in tiles]
    packed = torch.cat([ops.repack_tiles(r.cuda(), n, t).reshape(-1) for r, t in zip(raws, tiles)])
    d = torch.from_numpy(ops.build_descs(list(tiles), [n, n], k, split)).cuda()
    x = synth.activations(m, k, device="cuda")
    assert ops.device_status() == 0
    y = ops.grouped_gemm(x, packed, d, split, list(named), 2 * n)
    status = ops.device_status()
    want = ops.grouped_gemm(x, packed, d, split, list(tiles), 2 * n)
    assert ops.device_status() == 0 and status in (0, 2)
    assert status == 2 or torch.equal(y, want)


@pytest.mark.parametrize("m", [8, 16, 17, 24, 32, 40])
def test_a_table_stands_for_itself(m):
    """Each row of a descriptor table names its tile, its k-blocks and its part, so the rows of a split that does not reduce in a cluster may
    stand in any order, and a table without its last row leaves out that row's product only."""
    types, n_outs, k, split = [F.Q4_K, F.IQ3_S], [134, 100], 2560, 10
    raws = [synth.random_blocks(n, k, t, seed=t + n, device="cuda") for n, t in zip(n_outs, types)]
    packed = torch.cat([ops.repack_tiles(r, n, t).reshape(-1) for r, n, t in zip(raws, n_outs, types)])
    x, n = synth.activations(m, k, device="cuda"), sum(n_outs)
    table = torch.from_numpy(ops.build_descs(types, n_outs, k, split)).cuda()
    want = ops.grouped_gemm(x, packed, table, split, types, n)
    for order in (torch.arange(len(table) - 1, -1, -1), torch.randperm(len(table), generator=torch.Generator().manual_seed(m))):
        assert torch.equal(ops.grouped_gemm(x, packed, table[order.cuda()].contiguous(), split, types, n), want)
    last = int(table[-1, 2])
    for s in (2, split):
        full = torch.from_numpy(ops.build_descs(types, n_outs, k, s)).cuda()
        ws = torch.zeros(1 << 22, dtype=torch.uint8, device="cuda")
        y = ops.grouped_gemm(x, packed, full[:-1], s, types, n, workspace=ws)
        cut = x.clone()
        cut[:, int(full[-1, 4]) * 256:] = 0
        for cols, xx in ((slice(0, last), x), (slice(last, n), cut)):
            ref = ops.grouped_gemm(xx, packed, table, split, types, n)[:, cols].double()
            assert float((y[:, cols].double() - ref).norm() / ref.norm()) < 4e-3       # bf16 of the same sums in another order
    assert ops.device_status() == 0


@pytest.mark.parametrize("t", [F.IQ3_S, F.IQ3_XXS, F.IQ2_XXS, F.IQ2_XS, F.IQ2_S, F.IQ1_M])
@pytest.mark.parametrize("m", [17, 32, 64])
def test_fp32_sums_of_the_codebook_types(t, m):
    """The sums of one k-block before any rounding to bf16 (a split of one k-block a part, not summed up): eight pair sums are added in fp32 and
    scaled, eight roundings of at most 2^-24 of a value no larger than about the 2-norm of the products, evenly spread: rms 2^-24 (8 / 3)^0.5."""
    n, k = 256, 2560
    raw = synth.random_blocks(n, k, t, seed=t, device="cuda")
    tiles = ops.repack_tiles(raw, n, t)
    w = ops.dequantize_tiles(tiles, n, k, t).double()
    x = synth.activations(m, k, device="cuda")
    s = k // 256
    d = torch.from_numpy(ops.build_descs([t], [n], k, s)).cuda()
    ws = torch.zeros(ops.lib().gq_workspace_bytes(m, k, n, s), dtype=torch.uint8, device="cuda")
    ops.grouped_gemm(x, tiles.reshape(-1), d, s, [t], n, workspace=ws, phases=3)
    parts = ws[-(s * m * n * 4):].view(torch.float32).view(s, m, n).double()         # a multiple of 256 bytes at the end
    xs, wk = x.double().view(m, s, 256).transpose(0, 1), w.view(n, s, 256).permute(1, 2, 0)
    err = (parts - xs @ wk) / ((xs ** 2) @ (wk ** 2)).sqrt()
    assert float(err.square().mean().sqrt()) < 2.0 ** -24 * (8 / 3) ** 0.5
    assert ops.device_status() == 0
