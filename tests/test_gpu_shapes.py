"""GPU parity at the sizes the benchmark runs (BASELINE configs[1]-[3]) and on the path's corners: every type at the
real projection shapes, the grouped prefill cells, one block of the mixed stack, splits beyond a thread-block
cluster, a wait on a peer that never answers, a one-ulp check of the arithmetic, and extreme block scales.
Full-size outputs are checked on a subset of output columns (and batch rows) against the fp64 oracle."""
import ctypes

import numpy as np
import pytest
import torch

from hyperqwen_rtx4080s32_b200 import _lib, formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from hyperqwen_rtx4080s32_b200 import stack as S
from hyperqwen_rtx4080s32_b200.linear import GGUFLinear
from oracle import oracle

pytestmark = pytest.mark.gpu
TOL_TIGHT = 6e-3      # bf16 output rounding (2^-8 of the value) plus fp32 accumulation; the contract is 1e-2

SHAPES = {"q": (5120, 5120), "k": (1024, 5120), "gate": (17408, 5120), "down": (5120, 17408)}


def dev():
    return torch.device("cuda", 0)


def subset_rows(n_out: int, count: int = 80) -> np.ndarray:
    """Output columns to check: spread over the tensor, both ends of it, and both ends of some 64-row tiles."""
    idx = set(np.linspace(0, n_out - 1, count).astype(np.int64).tolist())
    idx |= {0, 1, 15, 16, 63, 64, n_out - 64, n_out - 17, n_out - 1}
    return np.array(sorted(i for i in idx if 0 <= i < n_out), dtype=np.int64)


def oracle_subset(x: torch.Tensor, raw_rows: torch.Tensor, t: int) -> np.ndarray:
    return oracle.matmul_f64(x.float().cpu().numpy(), raw_rows.cpu().numpy(), t)


@pytest.mark.parametrize("t", sorted(F.SUPPORTED_TYPES))
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_decode_at_the_real_projection_shapes(t, shape):
    """every type at q / k / gate / down of the dense decoder (hidden 5120, intermediate 17408)
    at M = 1, 8 and 64, through the op (so with the library's own split-K and row-count dispatch)."""
    n_out, k = SHAPES[shape]
    raw = synth.random_blocks(n_out, k, t, seed=7000 + t, device=dev())
    tiles = ops.repack_tiles(raw, n_out, t)
    packed, views, descs, splits, nb, bb = ops.prepare_grouped_layer([tiles], [n_out], [t])
    rows = subset_rows(n_out)
    raw_sub = raw[torch.from_numpy(rows).to(dev())]
    del raw, tiles
    for m in (1, 8, 64):
        x = synth.activations(m, k, device=dev())
        y = ops.fused_mul_mat_gguf_tiles_grouped(x, packed, descs, splits, views, [n_out], [t], nb, bb)
        assert not torch.isnan(y).any()
        got = y[:, torch.from_numpy(rows).to(dev())].float().cpu().numpy()
        err = oracle.rel_err(got, oracle_subset(x, raw_sub, t))
        assert err < TOL_TIGHT, f"{F.TYPE_NAMES[t]} {shape} M={m}: {err:.3e}"
    assert ops.device_status() == 0


@pytest.mark.parametrize("t", [F.Q4_K, F.Q6_K])
@pytest.mark.parametrize("m", [512, 2048, 8192])
def test_prefill_grouped_gate_up_and_down_cells(t, m):
    """grouped gate_up (K 5120, N 2 x 17408) and down (K 17408, N 5120) in Q4_K and Q6_K at
    M = 512, 2048, 8192 on the tcgen05 path: a subset of output columns and batch rows against the oracle."""
    for n_outs, k in (([17408, 17408], 5120), ([5120], 17408)):
        raws = [synth.random_blocks(n, k, t, seed=7100 + 3 * i + t, device=dev()) for i, n in enumerate(n_outs)]
        tiles = [ops.repack_tiles(r, n, t) for r, n in zip(raws, n_outs)]
        packed, views, descs, splits, nb, bb = ops.prepare_grouped_layer(tiles, n_outs, [t] * len(n_outs))
        del tiles
        x = synth.activations(m, k, device=dev())
        y = ops.fused_mul_mat_gguf_tiles_grouped(x, packed, descs, splits, views, n_outs, [t] * len(n_outs), nb, bb)
        assert tuple(y.shape) == (m, sum(n_outs))
        brow = torch.from_numpy(np.unique(np.concatenate([np.linspace(0, m - 1, 24).astype(np.int64), [0, 1, 255, 256, m - 1]]))).to(dev())
        col0 = 0
        for raw, n in zip(raws, n_outs):
            rows = subset_rows(n, 40)
            ridx = torch.from_numpy(rows).to(dev())
            got = y[brow][:, col0 + ridx].float().cpu().numpy()
            err = oracle.rel_err(got, oracle_subset(x[brow], raw[ridx], t))
            assert err < TOL_TIGHT, f"{F.TYPE_NAMES[t]} N={n} K={k} M={m}: {err:.3e}"
            col0 += n
        del raws, packed, views, descs, y
        torch.cuda.empty_cache()
    assert ops.device_status() == 0


@pytest.mark.parametrize("m", [1, 8, 64])
def test_one_block_of_the_mixed_stack(m):
    """the four linears of one block of the benchmark's stack (same type draw, same seeds, same
    LinearMethod calls as bench.py) against the oracle."""
    st = S.LinearStack(n_layers=1, device=dev())
    x = st.make_inputs(m)
    t = st.types[0]
    seed = 20261125 % 100000
    for lname, shards in (("qkv", ["q", "k", "v"]), ("o", ["o"]), ("gate_up", ["gate", "up"]), ("down", ["down"])):
        y = st.layers[0][lname](x[lname])
        col0 = 0
        for sname in shards:
            n_out, k = st.full_shapes[sname]
            raw = synth.random_blocks(n_out, k, t[sname], seed=seed + 10 * S.TENSORS.index(sname), device=dev())
            rows = subset_rows(n_out, 48)
            ridx = torch.from_numpy(rows).to(dev())
            got = y[:, col0 + ridx].float().cpu().numpy()
            err = oracle.rel_err(got, oracle_subset(x[lname], raw[ridx], t[sname]))
            assert err < TOL_TIGHT, f"{lname}/{sname} {F.TYPE_NAMES[t[sname]]} M={m}: {err:.3e}"
            col0 += n_out
    assert ops.device_status() == 0


@pytest.mark.parametrize("t", [F.Q4_K, F.IQ3_S, F.Q8_0])
def test_splits_beyond_a_cluster_use_the_partial_sum(t):
    """A split-K factor above 8 cannot reduce inside a thread-block cluster: the kernel writes fp32 partials and the
    sum kernel adds them in split order.  Descriptor tables for such splits are built by hand (the library's own
    policy never asks for them)."""
    n_out, k = 200, 5120
    raw = synth.random_blocks(n_out, k, t, seed=33 + t)
    tl = ops.repack_tiles(raw.to(dev()), n_out, t).reshape(-1)
    for split in (9, 10, 20):
        d = torch.from_numpy(ops.build_descs([t], [n_out], k, split)).to(dev())
        for m in (1, 8, 16, 17, 40):
            x = synth.activations(m, k, device=dev())
            y = ops.grouped_gemm(x, tl, d, split, [t], n_out)
            err = oracle.rel_err(y.float().cpu().numpy(), oracle.matmul_f64(x.float().cpu().numpy(), raw.numpy(), t))
            assert err < TOL_TIGHT, f"{F.TYPE_NAMES[t]} split={split} M={m}: {err:.3e}"
    assert ops.device_status() == 0


class _FakeTwoRanks:
    """A two-rank context whose second rank is a zeroed local buffer nobody writes: rank 0 stores its words into both
    buffers and then waits for rank 1's words, which never come."""

    def __init__(self, max_m, max_n_total):
        L = _lib.lib()
        self.rank, self.world, self.max_m, self.max_n_total = 0, 2, max_m, max_n_total
        nbytes = _lib.check(L.gq_fused_allreduce_buffer_bytes(2, max_m, max_n_total), "gq_fused_allreduce_buffer_bytes")
        self.bufs = [torch.zeros(nbytes, dtype=torch.uint8, device=dev()) for _ in range(2)]
        self.ptrs = (ctypes.c_uint64 * 2)(*[b.data_ptr() for b in self.bufs])
        self.used = False


def test_a_wait_on_a_silent_peer_runs_out_and_the_context_stays_usable():
    """Failure detection without a fault: the fused all-reduce waits for a peer that never writes, with the limit set to
    2 ms; the kernel gives up, the status words say so, and the next ordinary call on the device is correct.  Also: a
    multi-rank buffer is bound to the first output width it is used with."""
    n_out, k, t = 256, 1024, F.Q4_K
    raw = synth.random_blocks(n_out, k, t, seed=91)
    tl = ops.repack_tiles(raw.to(dev()), n_out, t).reshape(-1)
    d = torch.from_numpy(ops.build_descs([t], [n_out], k, 1)).to(dev())
    x = synth.activations(8, k, device=dev())
    want = ops.grouped_gemm(x, tl, d, 1, [t], n_out)
    assert ops.device_status() == 0
    ctx = _FakeTwoRanks(8, n_out)
    L = _lib.lib()
    ws = torch.zeros(L.gq_workspace_bytes(8, k, n_out, 1), dtype=torch.uint8, device=dev())
    ops.set_peer_wait_limit(2e-3)
    try:
        t0 = torch.cuda.Event(enable_timing=True); t1 = torch.cuda.Event(enable_timing=True)
        t0.record()
        ops.grouped_gemm(x, tl, d, 1, [t], n_out, workspace=ws, allreduce=ctx)
        t1.record()
        torch.cuda.synchronize()
        assert t0.elapsed_time(t1) < 500.0            # milliseconds: the wait is bounded by the limit, not by the default 4 s
        assert L.gq_read_status(ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream) == 1
        assert ops.device_status(clear=True) == 1
        assert ops.device_status() == 0
        # the same buffers with another output width are refused on the host (nothing is launched)
        raw2 = synth.random_blocks(128, k, t, seed=92)
        tl2 = ops.repack_tiles(raw2.to(dev()), 128, t).reshape(-1)
        d2 = torch.from_numpy(ops.build_descs([t], [128], k, 1)).to(dev())
        with pytest.raises(_lib.GqError):
            ops.grouped_gemm(x, tl2, d2, 1, [t], 128, allreduce=ctx)
    finally:
        ops.set_peer_wait_limit(4.0)
    got = ops.grouped_gemm(x, tl, d, 1, [t], n_out)
    assert torch.equal(got, want)
    assert ops.device_status() == 0


@pytest.mark.parametrize("m", [1, 8])
def test_a_split_part_that_never_comes_ends_with_a_status(m):
    """Split-K inside a cluster when a part stays away: a descriptor table in which two CTAs of a cluster of three take
    themselves for the receiving one.  Their waits run out after the kernel's own limit (4 s), they leave only after the
    third CTA has, status 1 is read, and the context stays usable.  (Nothing is out of bounds: every CTA stays in its tile.)"""
    k, n_out, t = 5120, 128, F.Q4_K
    raw = synth.random_blocks(n_out, k, t, seed=5, device=dev())
    packed = ops.repack_tiles(raw, n_out, t).reshape(-1)
    table = ops.build_descs([t], [n_out], k, 3)
    good = torch.from_numpy(table.copy()).to(dev())
    table[1::3, 6] = 0
    x = synth.activations(m, k, device=dev())
    want = ops.grouped_gemm(x, packed, good, 3, [t], n_out)
    assert ops.device_status() == 0
    ops.grouped_gemm(x, packed, torch.from_numpy(table).to(dev()), 3, [t], n_out)
    assert ops.device_status() == 1
    assert torch.equal(ops.grouped_gemm(x, packed, good, 3, [t], n_out), want)
    assert ops.device_status() == 0


# what the arithmetic of each form may add to the final bf16 rounding, as a fraction of the 2-norm of the products
# w[n,k] * x[m,k] of an output (99.9th percentile, maximum).  Integer form: activations are 16-bit fixed point per
# 256-block, everything else is exact integer arithmetic — 2^-16; the reference pins its kernel to the same 2e-5
# (gguf-plugin/test_gluon_kq_gpu.py:130-143).  fp16 form: exact weights and activations, fp16 hi + lo run sums in the
# correction MMAs.  tcgen05 form: every dequantised weight is rounded to fp16 (2^-11).
ARITH_BOUNDS = {"integer": (2e-5, 6e-5), "fp16": (2e-4, 4e-4), "tcgen05": (1.5e-3, 3e-3)}


@pytest.mark.parametrize("t", sorted(F.SUPPORTED_TYPES))
def test_arithmetic_error_beyond_the_output_rounding(t):
    """The tight check (the 1e-2 contract and the 6e-3 asserted elsewhere are the bf16 output rounding, which hides an
    arithmetic slip of 1e-3): against the fp64 oracle, what an output is off by BEYOND half a bf16 ulp of the exact
    value must stay within the bound of the form that computed it (ARITH_BOUNDS) — 300 (integer form) to 4 (tcgen05
    form) times tighter than the output rounding."""
    n_out, k = 512, 2048
    raw = synth.random_blocks(n_out, k, t, seed=600 + t)
    tiles = ops.repack_tiles(raw.to(dev()), n_out, t)
    packed, views, descs, splits, nb, bb = ops.prepare_grouped_layer([tiles], [n_out], [t])
    w = oracle.dequantize(raw.numpy(), t).astype(np.float64)
    for m, form in ((1, "integer"), (8, "integer"), (16, "integer"), (17, "fp16"), (32, "fp16"), (64, "tcgen05"), (128, "tcgen05")):
        x = synth.activations(m, k, device=dev())
        y = ops.fused_mul_mat_gguf_tiles_grouped(x, packed, descs, splits, views, [n_out], [t], nb, bb).float().cpu().numpy().astype(np.float64)
        xf = x.float().cpu().numpy().astype(np.float64)
        ref = xf @ w.T
        half_ulp = np.exp2(np.floor(np.log2(np.maximum(np.abs(ref), 1e-300))) - 8)
        norm = np.sqrt((xf ** 2) @ (w ** 2).T)
        extra = np.maximum(np.abs(y - ref) - half_ulp, 0.0) / norm
        p999, worst = ARITH_BOUNDS[form]
        assert np.percentile(extra, 99.9) <= p999 and extra.max() <= worst, \
            f"{F.TYPE_NAMES[t]} M={m} ({form} form): 99.9th percentile {np.percentile(extra, 99.9):.2e}, max {extra.max():.2e}"


@pytest.mark.parametrize("m", [1, 2, 4, 5, 8, 9, 16])
def test_a_block_whose_largest_significand_is_255_keeps_its_small_values(m):
    """The integer form holds every activation within 2^-7 of its block's largest magnitude exactly, also where that magnitude
    is 255 * 2^n of both signs, the edge of what two signed bytes hold.  All products and sums here are bf16 values, so the
    outputs are exact: 129 * 2^-14 beside 255 * 2^-7 lost its last bit (0.8 % of it) at half the scale."""
    k, n_out = 512, 64
    big, small = 255 / 128, 129 / 128 / 128
    blocks = np.zeros((n_out, k // 32, 34), dtype=np.uint8)
    blocks[:, :, :2] = np.frombuffer(np.float16(1.0).tobytes(), dtype=np.uint8)
    q = np.zeros((n_out, k), dtype=np.int8)
    for row, picks in enumerate([{100: 1}, {3: 1}, {7: 1}, {3: 1, 7: 1}, {3: -1}, {356: 1}, {259: 1}, {100: -2, 3: 1, 7: 1}]):
        for i, v in picks.items():
            q[row, i] = v
    blocks[:, :, 2:] = q.view(np.uint8).reshape(n_out, k // 32, 32)
    lin = GGUFLinear(k, [n_out])
    lin.load_shard(torch.from_numpy(blocks.reshape(n_out, -1)).to(dev()), F.Q8_0)
    lin.finalize()
    x = torch.zeros((m, k), dtype=torch.float64)
    for i, v in ((3, big), (7, -big), (100, small), (259, -16 * big), (356, 16 * small)):
        x[:, i] = v * torch.exp2(torch.arange(m) - 4.0)
    want = x @ torch.from_numpy(q.astype(np.float64)).T
    assert torch.equal(lin(x.to(dev(), torch.bfloat16)).double().cpu(), want)


@pytest.mark.parametrize("t", [F.Q4_K, F.Q6_K, F.Q2_K, F.Q8_0, F.IQ3_S])
@pytest.mark.parametrize("d_exp", [-20, -13, 2])
def test_extreme_block_scales(t, d_exp):
    """Block scales far from the usual 2^-6: tiny super-block d (2^-20, seen in real tensors) must not fall into fp16
    subnormals anywhere on the way, and large ones must not overflow — on all three kernels."""
    n_out, k = 256, 1024
    raw = synth.random_blocks(n_out, k, t, seed=700 + t, d_exp=d_exp)
    tiles = ops.repack_tiles(raw.to(dev()), n_out, t)
    packed, views, descs, splits, nb, bb = ops.prepare_grouped_layer([tiles], [n_out], [t])
    for m in (8, 32, 128):
        x = synth.activations(m, k, device=dev())
        y = ops.fused_mul_mat_gguf_tiles_grouped(x, packed, descs, splits, views, [n_out], [t], nb, bb)
        assert torch.isfinite(y).all()
        err = oracle.rel_err(y.float().cpu().numpy(), oracle.matmul_f64(x.float().cpu().numpy(), raw.numpy(), t))
        assert err < TOL_TIGHT, f"{F.TYPE_NAMES[t]} d=2^{d_exp} M={m}: {err:.3e}"


@pytest.mark.parametrize("t", [F.IQ2_S, F.IQ3_S])
def test_a_codebook_type_the_run_info_does_not_announce_is_reported_not_run(t):
    """The kernels keep a codebook type's grid in shared memory sized from run_info.  A caller whose run_info leaves the
    type out gets device status 2 and an unusable result, on both paths; nothing is read or written out of bounds."""
    n_out, k = 128, 512
    raw = synth.random_blocks(n_out, k, t, seed=77, device=dev())
    tiles = ops.repack_tiles(raw, n_out, t).reshape(-1)
    d1 = torch.from_numpy(ops.build_descs([t], [n_out], k, 1)).to(dev())
    assert ops.device_status() == 0
    ops.grouped_gemm(synth.activations(4, k, device=dev()), tiles, d1, 1, [F.Q8_0, F.Q4_K], n_out)      # large enough stages, no table
    assert ops.device_status() == 2
    ops.grouped_gemm(synth.activations(4, k, device=dev()), tiles, d1, 1, [F.Q4_K], n_out)              # a single type that is not the tiles'
    assert ops.device_status() == 2
    ops.prefill_gemm(synth.activations(128, k, device=dev()), tiles, d1, n_out, wtypes=[F.Q8_0])
    assert ops.device_status() == 2
    y = ops.grouped_gemm(synth.activations(4, k, device=dev()), tiles, d1, 1, [t], n_out)
    assert ops.device_status() == 0 and not torch.isnan(y).any()
