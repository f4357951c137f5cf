"""The tcgen05 path's last batch tile: only its own rows enter the MMAs, so the second of a wide tile's two MMAs may be shorter or left out."""
import numpy as np
import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from oracle import oracle

TOL = 6e-3      # bf16 output rounding (2^-8 of the value) plus the fp16 rounding of the weights
SHAPES = [(70, 2304), (19200 - 3, 512)]      # few units, which take narrow tiles; many, which take wide ones


def _last(m, n_tiles, nb):
    p = ops.prefill_plan(m, 256 * nb, n_tiles, 148)
    return p["wide"], p["rows"], p["tiles"], m - (p["tiles"] - 1) * p["rows"]


def _sizes(n_out, k):
    """For each kind of last tile the smallest batch that has one."""
    kinds = {}
    for m in range(129, 2400):
        wide, rows, tiles, last = _last(m, -(-n_out // 64), k // 256)
        if tiles > 1 or wide:
            first = rows // 2 if wide else rows
            kind = (wide, "one short" if last <= 16 else "first part" if last < first - 16 else "first" if last <= first else "second one" if last <= first + 16
                    else "second part" if last <= rows - 16 else "full", m % 16 == 0)
            kinds.setdefault(kind, m)
    return sorted(set(kinds.values()))


def test_every_tile_has_a_row_of_the_batch():
    for n_tiles, nb in ((2, 9), (80, 20), (136, 20), (544, 20)):
        for m in list(range(1, 1200)) + list(range(1200, 9000, 37)):
            wide, rows, tiles, last = _last(m, n_tiles, nb)
            assert 1 <= last <= rows and rows % (32 if wide else 16) == 0 and rows <= 384


@pytest.mark.gpu
@pytest.mark.parametrize("n_out, k, m", [(n, k, m) for n, k in SHAPES for m in _sizes(n, k)])
def test_last_tiles_of_every_size(n_out, k, m):
    raw = synth.random_blocks(n_out, k, F.Q4_K, seed=m, device="cuda")
    packed = ops.repack_tiles(raw, n_out, F.Q4_K).reshape(-1)
    d = torch.from_numpy(ops.build_descs([F.Q4_K], [n_out], k, 1)).cuda()
    x = synth.activations(m, k, device="cuda")
    wide = torch.full((m + 1, n_out), float("nan"), dtype=torch.bfloat16, device="cuda")
    y = ops.prefill_gemm(x, packed, d, n_out, out=wide[:m], wtypes=[F.Q4_K])
    assert bool(torch.isnan(wide[m]).all()) and not bool(torch.isnan(y).any())
    rows = np.unique(np.concatenate([np.arange(max(0, m - 400), m, 7), np.arange(0, m, 131), [m - 1]]))
    cols = np.unique(np.concatenate([np.arange(0, n_out, 211), [n_out - 1]]))
    r, c = torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda()
    assert oracle.rel_err(y[r][:, c].float().cpu().numpy(), oracle.matmul_f64(x[r].float().cpu().numpy(), raw[c].cpu().numpy(), F.Q4_K)) < TOL
    assert ops.device_status() == 0
