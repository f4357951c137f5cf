"""Calls beside the plain one on the plain stream: what may follow a load at once, what the native path leaves to the custom op,
what a waiting call keeps from other threads, and the lookup's ids and tables in every layout."""
import threading
import time

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


@pytest.mark.parametrize("t", [F.Q6_K, F.IQ2_S])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_lookup_answers_alike_for_every_layout(t, dt):
    """Ids and tables in every layout: the same rows, and an id outside the table gives NaN and status 2 on the device and an
    IndexError from host memory."""
    n, k = 40, 2304
    raw = synth.random_blocks(n, k, t, seed=77, device="cuda")
    want = torch.from_numpy(oracle.dequantize(raw.cpu().numpy(), t)).to(dt)
    good = torch.tensor([[3, 39, 0], [7, 3, 20]], device="cuda")
    bad = torch.tensor([[3, 40, 0], [7, -1, 20]], device="cuda")
    wide = torch.zeros((n, 2 * raw.shape[1]), dtype=torch.uint8, device="cuda")
    wide[:, ::2] = raw
    spread = torch.stack([good, bad], -1)
    for table in (raw, wide[:, ::2], torch.cat([raw, raw], 1)[:, raw.shape[1]:]):
        for ids in (good, good.int(), good.t().contiguous().t(), spread[..., 0], good.cpu()):
            assert torch.equal(ops.dequantize_rows(table, t, ids, dt).cpu(), want[good.cpu()])
        assert ops.device_status() == 0
        for ids in (bad, bad.int(), bad.t().contiguous().t(), spread[..., 1]):
            got = ops.dequantize_rows(table, t, ids, dt).cpu()
            assert bool(got[0, 1].isnan().all()) and bool(got[1, 1].isnan().all())
            assert torch.equal(got[:, [0, 2]], want[bad.cpu()[:, [0, 2]]])
            assert ops.device_status() == 2
        with pytest.raises(IndexError):
            ops.dequantize_rows(table, t, bad.cpu(), dt)
        assert ops.dequantize_rows(table, t, good[:0], dt).shape == (0, 3, k)
    with pytest.raises(RuntimeError):
        ops.dequantize_rows(raw, t, good.float(), dt)
    one = raw[5:6].expand(n, -1)        # a table of one repeated row: row stride 0
    assert torch.equal(ops.dequantize_rows(one, t, good, dt).cpu(), want[5].expand(2, 3, -1))
    assert ops.device_status() == 0


@pytest.mark.parametrize("how", ["vmap", "negative view", "trace", "function mode", "zero tensor"])
def test_native_path_stands_aside_for_what_is_not_a_plain_tensor_call(how):
    """Transforms, tracing, modes and tensors whose memory is not their value go through the custom op, as without the
    native path."""
    k, m = 512, 4
    lin = _layer([(64, F.Q4_K), (64, F.Q6_K), (64, F.IQ3_S)], k)
    x, x2 = synth.activations(m, k, device="cuda"), synth.activations(2 * m, k, device="cuda").reshape(2, m, k)
    if how == "vmap":
        with pytest.raises(RuntimeError, match="Batching rule"):      # the custom op has none
            torch.func.vmap(lin)(x2)
    elif how == "negative view":
        assert torch.equal(lin(torch._neg_view(x)), lin(-x))
    elif how == "trace":
        traced = torch.jit.trace(lin, x, check_trace=False)
        assert torch.equal(traced(x2[0]), lin(x2[0]))
    elif how == "function mode":
        class Seen(torch.overrides.TorchFunctionMode):
            names = []

            def __torch_function__(self, func, types, args=(), kwargs=None):
                self.names.append(str(func))
                return func(*args, **(kwargs or {}))

        want = lin(x)
        with Seen():
            assert torch.equal(lin(x), want)
        assert any("fused_mul_mat_gguf_tiles_grouped" in n for n in Seen.names)
    else:
        assert not lin(torch._efficientzerotensor((m, k), dtype=torch.bfloat16, device="cuda")).any()


def test_other_threads_run_while_a_call_waits_for_the_launch_queue():
    """A full launch queue holds the caller back, not the interpreter."""
    lin = _layer([(64, F.Q4_K), (64, F.Q6_K), (64, F.IQ3_S)], 512)
    x = synth.activations(8, 512, device="cuda")
    lin(x)
    torch.cuda.synchronize()
    torch.cuda._sleep(2_000_000_000)                     # about a second
    took = []

    def calls():
        t0 = time.monotonic()
        for _ in range(4000):
            lin(x)
        took.append(time.monotonic() - t0)

    worker = threading.Thread(target=calls)
    gap, last = 0.0, time.monotonic()
    worker.start()
    while worker.is_alive():
        time.sleep(1e-3)
        now = time.monotonic()
        gap, last = max(gap, now - last), now
    worker.join()
    torch.cuda.synchronize()
    assert took[0] > 0.5 and gap < 0.3, (took, gap)


def test_a_loaded_run_is_complete_when_the_load_returns():
    """A table holds addresses and any stream may call the layer next: the load's stream has nothing left to do."""
    tiles = ops.repack_tiles(synth.random_blocks(64, 512, F.Q4_K, seed=1, device="cuda"), 64, F.Q4_K)
    torch.cuda._sleep(200_000_000)
    assert not torch.cuda.current_stream().query()
    ops.prepare_grouped_layer([tiles], [64], [F.Q4_K])
    assert torch.cuda.current_stream().query()
    torch.cuda._sleep(200_000_000)
    _layer([(64, F.Q4_K), (64, F.Q6_K), (64, F.IQ3_S)], 512)
    assert torch.cuda.current_stream().query()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):       # part of a graph: complete when the graph is
        _, _, descs, splits, _, _ = ops.prepare_grouped_layer([tiles], [64], [F.Q4_K])
    graph.replay()
    assert torch.equal(descs[0].cpu(), torch.from_numpy(ops.build_descs([F.Q4_K], [64], 512, splits[0])))


@pytest.mark.parametrize("writer", ["gq_build_descs_device", "gq_repack"])
def test_load_kernels_are_ordered_in_front_of_programmatic_launches(writer):
    """The matrix kernels read tables and weights before they wait for the kernel in front of them, so no programmatic
    launch may follow directly on a kernel that writes either.  Captured, not run: the edges of the graph tell."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    k, n, t = 512, 64, F.Q4_K
    raw = synth.random_blocks(n, k, t, seed=2, device="cuda")
    tiles = ops.repack_tiles(raw, n, t)
    desc = ops.build_descs_on("cuda", [t], [n], k, [1])[0]
    x, y = synth.activations(8, k, device="cuda"), torch.empty((8, n), dtype=torch.bfloat16, device="cuda")
    ws = torch.empty(_lib.lib().gq_workspace_bytes(8, k, n, 1), dtype=torch.uint8, device="cuda")
    ops.grouped_gemm(x, tiles, desc, 1, [t], n, out=y, workspace=ws)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        if writer == "gq_repack":
            _lib.native().repack(raw, n, t, k // 256, tiles)
        else:
            _lib.native().build_descs([t], [n], k, [1], desc)
        ops.grouped_gemm(x, tiles, desc, 1, [t], n, out=y, workspace=ws)
    raw_graph = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())
    count = rt.cudaGraphGetEdges_v2(raw_graph)[-1]
    err, src, dst, data, count = rt.cudaGraphGetEdges_v2(raw_graph, count)
    assert int(err) == 0 and count >= 2
    src, dst = [int(s) for s in src], [int(d) for d in dst]
    programmatic = [e.type == rt.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic for e in data]
    first = [not p for s, p in zip(src, programmatic) if s not in dst]
    assert any(programmatic) and first and all(first)
