"""How many CTAs of a grouped launch an SM is held to: launches of one, two, three and four to an SM and of more than a wave, with and without
a split, in each of the kernel's forms."""
import numpy as np
import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from hyperqwen_rtx4080s32_b200.linear import GGUFLinear
from oracle import oracle

TOL = 6e-3      # bf16 output rounding (2^-8 of the value) plus fp32 accumulation


@pytest.mark.gpu
@pytest.mark.parametrize("t", [F.Q4_K, F.IQ2_S, F.Q8_0])
@pytest.mark.parametrize("tiles, nb", [(2, 3), (13, 16), (14, 16), (21, 8), (68, 5), (80, 4), (113, 4), (136, 6), (150, 3), (280, 2), (560, 2), (640, 1)])
def test_launches_of_every_density(t, tiles, nb):
    n, k = 64 * tiles - 5, 256 * nb
    raw = synth.random_blocks(n, k, t, seed=tiles, device="cuda")
    lin = GGUFLinear(k, [n])
    lin.load_shard(raw, t)
    lin.finalize()
    cols = np.unique(np.concatenate([np.arange(0, n, 977), np.arange(63, n, 64 * 41), [n - 1]]))
    pick = torch.from_numpy(cols).cuda()
    rows = raw[pick].cpu().numpy()
    for m in (1, 4, 8, 16, 20, 32):
        x = synth.activations(m, k, device="cuda")
        y = lin(x)
        assert oracle.rel_err(y[:, pick].float().cpu().numpy(), oracle.matmul_f64(x.float().cpu().numpy(), rows, t)) < TOL, m
        assert torch.equal(y, lin(x))
    assert ops.device_status() == 0


@pytest.mark.parametrize("m", [1, 8, 9, 16])
def test_the_split_leaves_no_part_empty_and_follows_the_tile_width(m):
    for nb in (1, 2, 5, 8, 17, 20, 68):
        for tiles in (1, 4, 15, 16, 56, 80, 112, 136, 148, 272, 544, 593, 3880):
            splits = [ops.grouped_split_for(tiles, nb, m=m, block_bytes=b, sms=148) for b in (84, 144, 210, 272)]
            assert all(1 <= s <= min(nb, 8) for s in splits) and splits[0] == splits[1] and splits[2] == splits[3]
            assert m > 8 or nb < 8 or splits[2] <= max(1, nb // 3) or tiles * splits[2] <= 3 * 148


@pytest.mark.parametrize("tiles, nb, split", [(112, 20, 3), (80, 20, 4), (80, 68, 4), (544, 20, 1), (80, 17, 3), (136, 20, 2), (272, 20, 1)])
def test_9_to_16_rows_keep_the_split_of_one_wave_unless_another_saves_an_eighth(tiles, nb, split):
    """The first four: q + k + v, o, down and gate + up of 5,120 x 17,408; the others: shards of them."""
    assert [ops.grouped_split_for(tiles, nb, m=m, block_bytes=b, sms=148) for m in (9, 13, 16) for b in (84, 144, 272)] == [split] * 9


def test_a_run_prepared_with_other_splits_uses_the_nearest_below():
    assert [ops._table_split(s, [1, 3, 6]) for s in (1, 2, 3, 5, 6, 8)] == [1, 1, 3, 3, 6, 6]
    assert ops._table_split(2, [6]) == 1


@pytest.mark.parametrize("types, n_outs, flags", [([F.Q4_K], [640], 0), ([F.Q4_K, F.IQ3_S], [17408, 17408], 3), ([F.IQ3_S, F.Q4_K], [17408, 17408], 0),
                                                  ([F.IQ3_S, F.IQ4_XS], [640, 640], 1), ([F.IQ4_XS, F.IQ3_S], [640, 640], 2), ([F.Q2_K, F.Q2_K], [64, 640], 0),
                                                  ([F.Q4_K, F.IQ2_XS], [0, 64], 0), ([F.Q4_K, F.IQ2_XS], [17408, 64], 0)])
def test_which_end_of_a_run_is_begun_with(types, n_outs, flags):
    assert ops.run_order(types, n_outs) == flags << 28


@pytest.mark.parametrize("types, n_outs", [([], []), ([F.Q4_K, F.IQ2_XS], [64]), ([F.Q4_K], [64, 64]), ([F.Q4_K, 999], [0, 0])])
def test_no_order_for_lists_that_name_no_run(types, n_outs):
    """Calls of no rows, and lists of unequal length, were taken before there was an order: it is 0 there, and nothing is read past a list's end."""
    assert ops.run_order(types, n_outs) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n_outs, k", [([64 * 280, 64 * 270 - 7], 256), ([64 * 130 + 3, 64 * 140], 2560), ([70, 200, 130], 5120), ([64, 64 * 13], 256 * 17)])
def test_a_run_begun_at_its_end_gives_the_same_bits(n_outs, k):
    types = [F.Q4_K, F.IQ3_S, F.IQ2_XS][:len(n_outs)]
    raws = [synth.random_blocks(n, k, t, seed=n, device="cuda") for n, t in zip(n_outs, types)]
    packed, _, descs, splits, _, _ = ops.prepare_grouped_layer([ops.repack_tiles(r, n, t) for r, n, t in zip(raws, n_outs, types)], n_outs, types)
    assert ops.run_order(types, n_outs) == 3 << 28
    for m in (1, 4, 8, 16, 33, 64, 128, 200):
        x = synth.activations(m, k, device="cuda")
        for s, d in zip(splits, descs):
            if m <= 64:
                got = [ops.grouped_gemm(x, packed, d, s, types, sum(n_outs), order=o) for o in (0, 3 << 28)]
                assert torch.equal(*got), (m, s)
        got = [ops.prefill_gemm(x, packed, descs[splits.index(1)], sum(n_outs), wtypes=types, order=o) for o in (0, 3 << 28)]
        assert torch.equal(*got), m
    assert ops.device_status() == 0
