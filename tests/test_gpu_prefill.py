"""The tcgen05 path where its cuts end, in each of its shapes (named by the plan that the library states): batch tiles in
16-row steps up to 128 (two CTAs per SM), up to 256 and up to 384 (CTA pairs), several balanced tiles, K split over a cluster,
last pairs with one, two or three of their four tiles, and outputs whose rows are not four-byte aligned."""
import numpy as np
import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from oracle import oracle

pytestmark = pytest.mark.gpu
TOL = 6e-3      # bf16 output rounding (2^-8 of the value) plus the fp16 rounding of the weights


def test_a_run_of_more_columns_than_a_grid_has_units():
    """131,080 tiles, 65,540 pairs of them: more than one launch takes.  Every row of the table names the same tile."""
    k, n, m, t = 256, 131080, 33, F.Q4_K
    raw = synth.random_blocks(64, k, t, seed=8)
    tiles = ops.repack_tiles(raw.cuda(), 64, t)
    table = np.repeat(ops.build_descs([t], [64], k, 1), n, axis=0)
    table[:, 2] = 64 * np.arange(n)
    x = synth.activations(m, k, device="cuda")
    y = ops.prefill_gemm(x, tiles.reshape(-1), torch.from_numpy(table).cuda(), 64 * n, wtypes=[t]).view(m, n, 64)
    assert oracle.rel_err(y[:, 0].float().cpu().numpy(), oracle.matmul_f64(x.float().cpu().numpy(), raw.numpy(), t)) < TOL
    assert bool((y == y[:, :1]).all())
    assert ops.device_status() == 0


@pytest.mark.parametrize("m", [33, 48, 49, 127, 128, 129, 144, 255, 256, 257, 513, 520])
@pytest.mark.parametrize("parts,k", [([(64, F.Q4_K), (64, F.Q8_0), (70, F.IQ3_S)], 512), ([(129, F.IQ1_M), (33, F.Q2_K)], 2048), ([(200, F.Q6_K)], 4352)])
def test_tiles_splits_and_ragged_outputs(m, parts, k):
    n_outs, types = [n for n, _ in parts], [t for _, t in parts]
    raws = [synth.random_blocks(n, k, t, seed=300 + i) for i, (n, t) in enumerate(parts)]
    tiles = [ops.repack_tiles(r.cuda(), n, t) for r, (n, t) in zip(raws, parts)]
    packed, _, descs, splits, _, _ = ops.prepare_grouped_layer(tiles, n_outs, types)
    d1, n = descs[splits.index(1)], sum(n_outs)
    x = synth.activations(m, k, device="cuda")
    ref = np.concatenate([oracle.matmul_f64(x.float().cpu().numpy(), r.numpy(), t) for r, t in zip(raws, types)], axis=1)
    y = ops.prefill_gemm(x, packed, d1, n, wtypes=types)
    assert oracle.rel_err(y.float().cpu().numpy(), ref) < TOL
    for pad in (0, 1):      # a view at an odd column, in rows of even and odd stride
        wide = torch.full((m, n + 6 + pad), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.prefill_gemm(x, packed, d1, n, out=wide[:, 3:3 + n], wtypes=types)
        assert torch.equal(wide[:, 3:3 + n], y) and bool(torch.isnan(wide[:, :3]).all()) and bool(torch.isnan(wide[:, 3 + n:]).all())
    assert ops.device_status() == 0


# (tiles of 64 rows, k-blocks, batch rows) -> (batch rows of a tile, batch tiles, parts of K, sets, wide) on 148 SMs
PLANS = [((33, 16, 257), (288, 1, 4, 2, 1)), ((34, 16, 300), (320, 1, 4, 2, 1)), ((35, 16, 300), (320, 1, 4, 2, 1)), ((37, 16, 257), (288, 1, 4, 2, 1)),
         ((45, 16, 384), (384, 1, 4, 2, 1)), ((74, 16, 383), (384, 1, 3, 2, 1)), ((97, 17, 350), (352, 1, 2, 2, 1)), ((33, 16, 520), (288, 2, 3, 2, 1)),
         ((149, 4, 300), (320, 1, 1, 2, 1)), ((147, 5, 641), (352, 2, 1, 2, 1)),
         ((35, 16, 256), (256, 1, 4, 2, 0)), ((33, 16, 385), (208, 2, 3, 2, 0)), ((75, 9, 385), (208, 2, 1, 2, 0)),
         ((35, 16, 128), (128, 1, 4, 1, 0)), ((35, 34, 40), (48, 1, 7, 1, 0)), ((149, 5, 100), (112, 1, 1, 1, 0))]


@pytest.mark.parametrize("size,plan", PLANS)
def test_every_shape_with_ragged_pairs_and_mixed_types(size, plan):
    """A run of four types, three with a codebook table beside the rings, whose tiles share CTAs and pairs: the plan is the
    one named, and the outputs agree with the oracle in a sample of columns from every tile."""
    tiles, nb, m = size
    if ops.sm_count() == 148:
        assert tuple(ops.prefill_plan(m, 256 * nb, tiles).values()) == plan
    k, types = 256 * nb, [F.Q8_0, F.IQ1_M, F.IQ3_S, F.IQ2_S]
    n_outs = [64 * 5, 64 * 7 - 3, 64 * 9 - 61, 64 * (tiles - 21) - 1]
    raws = [synth.random_blocks(n, k, t, seed=500 + tiles + i, device="cuda") for i, (n, t) in enumerate(zip(n_outs, types))]
    packed, _, descs, splits, _, _ = ops.prepare_grouped_layer([ops.repack_tiles(r, n, t) for r, n, t in zip(raws, n_outs, types)], n_outs, types)
    d1, n = descs[splits.index(1)], sum(n_outs)
    x = synth.activations(m, k, device="cuda")
    y = ops.prefill_gemm(x, packed, d1, n, wtypes=types)
    xf, at = x.float().cpu().numpy(), 0
    for raw, rows, t in zip(raws, n_outs, types):
        pick = np.unique(np.concatenate([np.arange(0, rows, 61), np.arange(63, rows, 64), [rows - 1]]))
        ref = oracle.matmul_f64(xf, raw[torch.from_numpy(pick).cuda()].cpu().numpy(), t)
        assert oracle.rel_err(y[:, torch.from_numpy(at + pick).cuda()].float().cpu().numpy(), ref) < TOL, F.TYPE_NAMES[t]
        at += rows
    wide = torch.full((m, n + 7), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.prefill_gemm(x, packed, d1, n, out=wide[:, 3:3 + n], wtypes=types)
    assert torch.equal(wide[:, 3:3 + n], y) and bool(torch.isnan(wide[:, :3]).all()) and bool(torch.isnan(wide[:, 3 + n:]).all())
    assert ops.device_status() == 0


@pytest.mark.parametrize("types", [[F.Q8_0], [F.Q6_K], [F.Q4_0], [F.Q4_0, F.Q2_K], [F.Q8_0, F.IQ2_S], [F.IQ1_M, F.Q8_0]])
@pytest.mark.parametrize("m", [64, 65, 80, 96, 112, 113, 128])
def test_slices_handed_over_singly_and_in_pairs(types, m):
    """Up to 128 rows two k-slices share a barrier where the activation ring holds a k-block or a codebook type decodes slowly; else each has
    its own: rings of two, three and four slices, both ways.  A row's result does not depend on the batch around it, so calls of 16 rows,
    which cut the rings otherwise, agree to the bit."""
    k, n_outs = 2304, [134, 100][:len(types)]
    raws = [synth.random_blocks(n, k, t, seed=n + t) for n, t in zip(n_outs, types)]
    packed = torch.cat([ops.repack_tiles(r.cuda(), n, t).reshape(-1) for r, n, t in zip(raws, n_outs, types)])
    d1, n = torch.from_numpy(ops.build_descs(types, n_outs, k, 1)).cuda(), sum(n_outs)
    x = synth.activations(m, k, device="cuda")
    y = ops.prefill_gemm(x, packed, d1, n, wtypes=types)
    ref = np.concatenate([oracle.matmul_f64(x.float().cpu().numpy(), r.numpy(), t) for r, t in zip(raws, types)], axis=1)
    assert oracle.rel_err(y.float().cpu().numpy(), ref) < TOL
    if ops.prefill_plan(m, k, 3 + len(types) * 2 - 2)["split"] == ops.prefill_plan(16, k, 3 + len(types) * 2 - 2)["split"]:
        assert torch.equal(torch.cat([ops.prefill_gemm(x[i:i + 16], packed, d1, n, wtypes=types) for i in range(0, m, 16)]), y)
    assert ops.device_status() == 0
