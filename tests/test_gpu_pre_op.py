"""The op in front of a layer as a launch of its own (more rows than the preparation folds) and the row norm that both forms share, where a row
ends within, at and beyond what a CTA keeps."""
import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from hyperqwen_rtx4080s32_b200.linear import GGUFLinear

pytestmark = pytest.mark.gpu


def _layer(k, n=96, t=F.Q4_K):
    lin = GGUFLinear(k, [n])
    lin.load_shard(synth.random_blocks(n, k, t, seed=k, device="cuda"), t)
    return lin.finalize()


def _native_only(lin, x, pre):
    y = lin.gguf_native(lin.gguf_groups, x, pre)
    assert y is not None
    return y


@pytest.mark.parametrize("k", [256, 5120, 8192, 8448, 16384, 16640, 24576])
@pytest.mark.parametrize("m", [1, 16, 17, 33, 300])
def test_norm_of_rows_of_any_length(k, m):
    """Beside torch's operations: the mean square is summed in another order, so a normalised value that lies at a rounding edge of bf16 may round the
    other way (one bit of 8): few of them, and no more.  One unit there is up to 2^-7 of the value; the products with the weight are each rounded
    again, by up to 2^-8: 2^-6 in all."""
    lin, x = _layer(k), synth.activations(m, k, device="cuda")
    res = synth.activations(m, k, seed=5, device="cuda") * 3
    w = (1 + 0.1 * torch.randn(k, device="cuda")).to(torch.bfloat16)
    for residual in (res, None):
        pre, ref = ops.PreAddRMSNorm(w, 1e-6, residual), ops.PreAddRMSNorm(w, 1e-6, residual)
        want = ref.unfused(x)
        y = _native_only(lin, x, pre)
        if residual is not None:
            assert torch.equal(pre.residual_out, ref.residual_out)
        err = (y.double() - lin(want).double()).norm() / lin(want).double().norm()
        assert float(err) < 4e-3
        if m > ops.PRE_MAX_ROWS:
            h = torch.empty_like(x)
            out = torch.empty_like(x) if residual is not None else None
            ops.check(ops.lib().gq_pre_op(x.data_ptr(), m, k, k, 2, w.data_ptr(), residual.data_ptr() if residual is not None else None,
                                          out.data_ptr() if out is not None else None, k, 1e-6, h.data_ptr(), k, torch.cuda.current_stream().cuda_stream), "gq_pre_op")
            assert float((h != want).float().mean()) < 2e-3 and float(((h - want).abs() / want.abs().clamp_min(1e-20)).max()) <= 2.0 ** -6
    assert ops.device_status() == 0


@pytest.mark.parametrize("k", [256, 2304, 5120])
@pytest.mark.parametrize("m", [17, 40, 200])
def test_silu_mul_equals_the_unfused_operations(k, m):
    lin = _layer(k)
    wide = synth.activations(m, 2 * k + 7, device="cuda") * 4
    wide[0, 3], wide[1, 5], wide[2, 7] = float("inf"), -100.0, float("nan")
    for gu in (wide[:, :2 * k].contiguous(), wide[:, 1:2 * k + 1]):          # rows that start anywhere
        want = lin(ops.PreSiluMul().unfused(gu))
        assert torch.equal(_native_only(lin, gu, ops.PreSiluMul()).nan_to_num(7.0), want.nan_to_num(7.0))
    assert ops.device_status() == 0


def test_more_rows_than_a_grid_has_and_refused_arguments():
    k, m = 256, 65535 + 9
    x = torch.randn(m, 2 * k, device="cuda").to(torch.bfloat16)
    out = torch.zeros(m, k, dtype=torch.bfloat16, device="cuda")
    st, L = torch.cuda.current_stream().cuda_stream, ops.lib()
    assert L.gq_pre_op(x.data_ptr(), m, k, 2 * k, 1, None, None, None, 0, 0.0, out.data_ptr(), k, st) == 0
    assert torch.equal(out, ops.PreSiluMul().unfused(x))
    assert L.gq_pre_op(x.data_ptr(), 4, k, k, 1, None, None, None, 0, 0.0, out.data_ptr(), k, st) < 0           # rows of K, not 2 K
    assert L.gq_pre_op(x.data_ptr(), 4, k, k, 2, None, None, None, 0, 0.0, out.data_ptr(), k, st) < 0           # no weight
    assert L.gq_pre_op(x.data_ptr(), 4, k + 1, 2 * k, 2, x.data_ptr(), None, None, 0, 0.0, out.data_ptr(), 2 * k, st) < 0
    assert L.gq_pre_op(x.data_ptr(), 4, k, k, 0, None, None, None, 0, 0.0, out.data_ptr(), k, st) < 0


@pytest.mark.parametrize("k", [256, 5120, 16640])
@pytest.mark.parametrize("m", [17, 24, 300])
def test_the_new_residual_in_place_of_the_old_one(k, m):
    """Above 16 rows, also of rows that are read again before they are written (K beyond 16,384), and in memory that the kernel may not share."""
    lin, x = _layer(k), synth.activations(m, k, device="cuda")
    old = synth.activations(m, k, seed=5, device="cuda") * 3
    w = (1 + 0.1 * torch.randn(k, device="cuda")).to(torch.bfloat16)
    apart = ops.PreAddRMSNorm(w, 1e-6, old)
    want = _native_only(lin, x, apart)
    pre = ops.PreAddRMSNorm(w, 1e-6, old.clone())
    pre.residual_out = pre.residual
    for y in (_native_only(lin, x, pre), None):
        if y is None:                   # the same through the layer
            pre.residual.copy_(old)
            y = lin(x, pre=pre)
        assert torch.equal(pre.residual, apart.residual_out) and torch.equal(y, want)
    # beside each other in one buffer: the kernel; a row on, or over the input: read in full first
    both = torch.empty(m, 2 * k, dtype=torch.bfloat16, device="cuda")
    rows = torch.empty(m + 1, k, dtype=torch.bfloat16, device="cuda")
    xc = x.clone()
    for res, out, inp, native in ((both[:, :k], both[:, k:], x, True), (rows[:m], rows[1:], x, False), (old.clone(), xc, xc, False)):
        res.copy_(old)
        pre = ops.PreAddRMSNorm(w, 1e-6, res)
        pre.residual_out = out
        if native:
            y = _native_only(lin, inp, pre)
        else:
            assert lin.gguf_native(lin.gguf_groups, inp, pre) is None
            y = lin(inp, pre=pre)
        assert torch.equal(pre.residual_out, apart.residual_out)
        assert float((y.double() - want.double()).norm() / want.double().norm()) < 4e-3          # torch sums the mean square in another order
    assert ops.device_status() == 0


def _at_odd(t, at=3):
    """The rows of t as a column view that starts at an odd element, in rows of odd stride, and the buffer around it."""
    m, k = t.shape
    buf = torch.full((m, k + 9), 7.0, dtype=torch.bfloat16, device="cuda")
    buf[:, at:at + k].copy_(t)
    return buf[:, at:at + k], buf


def _untouched(buf, k):
    return bool((buf[:, :3] == 7.0).all()) and bool((buf[:, 3 + k:] == 7.0).all())


@pytest.mark.parametrize("k", [256, 5120, 16640])
@pytest.mark.parametrize("m", [4, 17, 200])
def test_norm_of_rows_that_start_anywhere(k, m):
    """Whatever the alignment of the input, the weight and both residuals: the bits of aligned rows, nothing written beside them."""
    lin, x = _layer(k), synth.activations(m, k, device="cuda")
    old = synth.activations(m, k, seed=5, device="cuda") * 3
    w = (1 + 0.1 * torch.randn(k, device="cuda")).to(torch.bfloat16)
    aligned = ops.PreAddRMSNorm(w, 1e-6, old)
    want, plain = _native_only(lin, x, aligned), _native_only(lin, x, ops.PreAddRMSNorm(w, 1e-6))
    xo, wo = _at_odd(x, 2 if m <= ops.PRE_MAX_ROWS else 3)[0], _at_odd(w[None])[0][0]       # (folded, the first row begins at a multiple of four bytes)
    pre = ops.PreAddRMSNorm(wo, 1e-6, _at_odd(old)[0])
    pre.residual_out, buf = _at_odd(torch.zeros_like(old))
    assert torch.equal(_native_only(lin, xo, pre), want)
    assert torch.equal(pre.residual_out, aligned.residual_out) and _untouched(buf, k)
    assert torch.equal(_native_only(lin, xo, ops.PreAddRMSNorm(wo, 1e-6)), plain)
    assert ops.device_status() == 0


@pytest.mark.parametrize("k", [256, 2304, 16640])
@pytest.mark.parametrize("m", [5, 200])
def test_the_op_by_itself_writes_rows_that_start_anywhere(k, m):
    st, call = torch.cuda.current_stream().cuda_stream, lambda *a: ops.check(ops.lib().gq_pre_op(*a), "gq_pre_op")
    gu, w = synth.activations(m, 2 * k, device="cuda") * 4, (1 + 0.1 * torch.randn(k, device="cuda")).to(torch.bfloat16)
    for op, args in ((1, (None, None, None, 0, 0.0)), (2, (w.data_ptr(), None, None, 0, 1e-6))):
        want = torch.empty(m, k, dtype=torch.bfloat16, device="cuda")
        call(gu.data_ptr(), m, k, 2 * k, op, *args, want.data_ptr(), k, st)
        out, buf = _at_odd(torch.zeros_like(want))
        call(gu.data_ptr(), m, k, 2 * k, op, *args, out.data_ptr(), buf.stride(0), st)
        assert torch.equal(out, want) and _untouched(buf, k)
        ref = ops.PreSiluMul().unfused(gu) if op == 1 else ops.PreAddRMSNorm(w, 1e-6).unfused(gu[:, :k])
        assert float((want != ref).float().mean()) < (1e-9 if op == 1 else 2e-3)       # the norm: torch sums the mean square in another order
