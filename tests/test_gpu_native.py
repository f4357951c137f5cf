"""The native call path of GGUFLinearMethod.apply against the custom op, which runs the same kernels: the same bits for
every row count at the edges of the dispatch and every input layout, and the general path where the native one steps aside."""
import copy

import pytest
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import ops, synth
from hyperqwen_rtx4080s32_b200.linear import GGUFLinear

pytestmark = pytest.mark.gpu


def _layer(parts, k):
    lin = GGUFLinear(k, [n for n, _ in parts])
    for sid, (n, t) in zip(["q", "k", "v"], parts):
        lin.load_shard(synth.random_blocks(n, k, t, seed=n + t, device="cuda"), t, sid)
    return lin.finalize()


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64, 65, 300])
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
    assert torch.equal(copy.deepcopy(lin)(x), want)                          # a copy starts without the native run
    assert tuple(lin(x[:0]).shape) == (0, want.shape[1])
