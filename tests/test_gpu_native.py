"""The native call path of GGUFLinearMethod.apply against the custom op, which runs the same kernels: the same bits for
every row count at the edges of the dispatch and every input layout, and the general path where the native one steps aside."""
import copy

import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import _lib, ops, synth
from hyperqwen_rtx4080s32_b200.linear import GGUFLinear
from oracle import oracle

pytestmark = pytest.mark.gpu


def _layer(parts, k):
    lin = GGUFLinear(k, [n for n, _ in parts])
    for sid, (n, t) in zip(["q", "k", "v"], parts):
        lin.load_shard(synth.random_blocks(n, k, t, seed=n + t, device="cuda"), t, sid)
    return lin.finalize()


@pytest.mark.parametrize("m", [1, 4, 5, 8, 9, 16, 17, 24, 25, 32, 33, 64, 65, 300])
def test_native_path_equals_the_custom_op(m):
    k, parts = 1024, [(192, F.Q4_K), (70, F.IQ3_S), (64, F.Q6_K)]
    lin = _layer(parts, k)
    packed, descs, splits, run, nb, bb = lin.gguf_groups["q"]
    args = (packed, descs, splits, [lin.gguf_tiles[i] for i in run], [n for n, _ in parts], [t for _, t in parts], nb, bb)
    x = synth.activations(m, k, device="cuda")
    want = ops.fused_mul_mat_gguf_tiles_grouped(x, *args)
    assert lin.gguf_native(lin.gguf_groups, x, None) is not None
    assert torch.equal(lin(x), want)
    wide = torch.zeros((m, k + 64), dtype=torch.bfloat16, device="cuda")
    wide[:, 8:8 + k] = x
    assert torch.equal(lin(wide[:, 8:8 + k]), want)                          # a strided view
    assert torch.equal(lin(x.reshape(1, m, k)), want.reshape(1, m, -1))      # leading dimensions
    col = x.t().contiguous().t()                                             # unit row stride: the general path
    assert m == 1 or lin.gguf_native(lin.gguf_groups, col, None) is None
    assert torch.equal(lin(col), want)
    assert copy.deepcopy(lin.gguf_native)(lin.gguf_groups, x, None) is None  # a copy starts without the native run
    assert tuple(lin(x[:0]).shape) == (0, want.shape[1])


@pytest.mark.parametrize("t", sorted(F.SUPPORTED_TYPES))
def test_load_and_lookup_kernels_at_the_edges(t):
    """Repack, dequantise and row lookup against the oracle where their splits end: one k-block, fewer and more k-blocks than a
    CTA's warps or a repack CTA take, rows that end inside a slab and inside a tile, sources at odd alignments, an output
    with a row stride that allows no wide stores, ids repeated, out of range (reported, not read) and in both index types."""
    bb = F.BYTES_PER_256[t]
    for n, nb, pad in [(1, 1, 0), (17, 7, 3), (63, 9, 1), (130, 17, 0)]:
        k = 256 * nb
        raw = synth.random_blocks(n, k, t, seed=900 + n + t)
        want = torch.from_numpy(oracle.dequantize(raw.numpy(), t))
        base = torch.zeros(n * (nb * bb + pad) + 5, dtype=torch.uint8, device="cuda")
        src = base[5:].view(n, nb * bb + pad)[:, :nb * bb]           # rows at odd addresses
        src.copy_(raw)
        tiles = ops.repack_tiles(src, n, t)
        assert torch.equal(tiles, ops.repack_tiles(raw.cuda(), n, t))
        assert torch.equal(ops.unrepack_tiles(tiles, n, t).cpu(), raw)
        assert torch.equal(ops.dequantize_tiles(tiles, n, k, t).cpu(), want)
        assert torch.equal(ops.dequantize_tiles(tiles, n, k, t, torch.bfloat16).cpu(), want.to(torch.bfloat16))
        for bits, dt in ((0, torch.float32), (1, torch.bfloat16)):
            wide = torch.full((n, k + 3), 7.0, dtype=dt, device="cuda")
            assert _lib.lib().gq_dequant(t, tiles.data_ptr(), n, k, wide.data_ptr(), bits, k + 3, torch.cuda.current_stream().cuda_stream) == 0
            assert torch.equal(wide[:, :k].cpu(), want.to(dt)) and bool((wide[:, k:] == 7.0).all())
        for dt in (torch.int32, torch.int64):
            ids = torch.tensor([[n - 1, 0, n // 2, 0]] * 5, dtype=dt, device="cuda")
            for out in (torch.float32, torch.bfloat16):
                assert torch.equal(ops.dequantize_rows(src, t, ids, out).cpu(), want[ids.cpu().long()].to(out))
    assert ops.device_status() == 0
    got = ops.dequantize_rows(src, t, torch.tensor([0, n, -1, n - 1], device="cuda"))
    assert ops.device_status() == 2
    assert torch.equal(got[[0, 3]].cpu(), want[[0, n - 1]])


@pytest.mark.parametrize("parts", [[(1, F.Q4_K)], [(130, F.Q4_K), (64, F.Q8_0), (70, F.IQ1_M)], [(64 * i, F.Q6_K) for i in range(1, 9)]])
def test_descriptor_tables_written_on_the_device(parts):
    n_outs, types = [n for n, _ in parts], [t for _, t in parts]
    for k, splits in [(256, [1]), (5120, [1, 3, 20])]:
        for s, d in zip(splits, ops.build_descs_on("cuda", types, n_outs, k, splits)):
            assert torch.equal(d.cpu(), torch.from_numpy(ops.build_descs(types, n_outs, k, s)))


@pytest.mark.parametrize("t", [F.Q4_K, F.Q6_K, F.Q2_K, F.IQ3_S, F.Q8_0])
@pytest.mark.parametrize("n_out,k", [(64, 256), (70, 768), (1024, 5120), (130, 17408)])
def test_small_launches_that_convert_their_activations(t, n_out, k):
    """One row (two beside it) of a layer without the preparation kernel (the native path) against the prepared call, bit for
    bit: fewer k-blocks than stages, splits of up to four, more than four, rows of odd stride, a block of zeros, an infinity."""
    lin = GGUFLinear(k, [n_out])
    lin.load_shard(synth.random_blocks(n_out, k, t, seed=n_out, device="cuda"), t)
    lin.finalize()
    packed, descs, splits, _, nb, bb = lin.gguf_groups["__all__"]
    for m, bad in ((1, False), (1, True), (2, False)):
        s = ops.grouped_split_for(-(-n_out // 64), nb, m=m, block_bytes=bb, sms=ops.sm_count(packed.device))
        x = synth.activations(m, k, device="cuda")
        x[0, :256] = 0
        if bad:
            x[0, 300 % k] = float("inf")
        wide = torch.zeros((m, k + 3), dtype=torch.bfloat16, device="cuda")
        wide[:, 2:2 + k] = x
        want = ops.grouped_gemm(x, packed, descs[splits.index(s)], s, [t], n_out)
        for _ in range(2):
            assert torch.equal(lin(x).nan_to_num(7.0), want.nan_to_num(7.0))
            assert torch.equal(lin(wide[:, 2:2 + k]).nan_to_num(7.0), want.nan_to_num(7.0))
    assert ops.device_status() == 0
