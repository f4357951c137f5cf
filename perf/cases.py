"""The work this framework is used for, as cases that can be timed one by one: quantized linear layers in decode, in
speculative verification and in prefill, the ops folded into them, the LM head, the load of a layer and the embedding
lookup.  Shapes are those of the benchmark's decoder (hidden 5120, 40 / 8 heads of 128, intermediate 17408, vocabulary
248320) and of its tensor-parallel shards; weights are random valid blocks of the sixteen GGML types, activations bf16
N(0, 1), all made on the GPU from the seed.

    listed()            the cases, each a dict of plain values with a name
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the layers and inputs a program holds before the call
    run(state)          one pass through the public entry points, returning its outputs
    work(case)          bytes and flops the pass cannot do without
    tolerance(case)     how far another correct implementation may be off
"""
import torch

from hyperqwen_rtx4080s32_b200 import formats as F
from hyperqwen_rtx4080s32_b200 import loader, ops, synth
from hyperqwen_rtx4080s32_b200.linear import GGUFLinear
from hyperqwen_rtx4080s32_b200.stack import draw_types

HIDDEN, INTER, Q_ROWS, KV_ROWS, VOCAB = 5120, 17408, 5120, 1024, 248320
# rows and K of the decoder's linear layers; a merged layer has one entry per shard
LAYERS = {
    "qkv": ((Q_ROWS, KV_ROWS, KV_ROWS), HIDDEN), "o": ((HIDDEN,), Q_ROWS), "gate_up": ((INTER, INTER), HIDDEN), "down": ((HIDDEN,), INTER),
}
SHARDS = {"qkv": ("q", "k", "v"), "o": ("o",), "gate_up": ("gate", "up"), "down": ("down",)}
ROW_PARALLEL = ("o", "down")       # cut along K under tensor parallelism, the others along their rows
MAX_FLOPS = 2.0 * 8192 * HIDDEN * INTER


def listed():
    return [
        # a key or value projection for one sequence in a program that does not capture graphs: latency and host work
        dict(name="k_proj_m1", kind="linear", types="Q4_K", rows="1024", k=HIDDEN, m=1),
        # the linears of four decoder blocks for one sequence / eight sequences, replayed as a CUDA graph as a serving
        # engine does in decode; the weights are several times the L2
        dict(name="decode_m1", kind="stack", blocks=4, types_seed=20261125, m=1, graph=True),
        dict(name="decode_m8", kind="stack", blocks=4, types_seed=20261125, m=8, graph=True),
        # the same with the batch of a speculative step: 9 sequences of 3 tokens, 16 sequences of 4
        dict(name="verify_m27", kind="stack", blocks=4, types_seed=20261126, m=27, graph=True),
        dict(name="verify_m64", kind="stack", blocks=4, types_seed=20261126, m=64, graph=True),
        # an MLP with the norm and the activation folded in, on one of four tensor-parallel ranks, types of the served checkpoint
        dict(name="mlp_folded_tp4_m13", kind="mlp", types="IQ2_XS,IQ3_XXS,IQ4_XS", inter=INTER // 4, m=13),
        # logits of eight sequences
        dict(name="lm_head_m8", kind="linear", types="Q6_K", rows=str(VOCAB), k=HIDDEN, m=8),
        # a ragged chunk of a prompt through one block's linears, called one by one
        dict(name="prefill_block_m517", kind="stack", blocks=1, types_seed=20261127, m=517, graph=False),
        # prompts of ordinary and of large size through the two widest layers
        dict(name="prefill_gate_up_m2048", kind="linear", types="Q4_K,IQ3_S", rows="17408,17408", k=HIDDEN, m=2048),
        dict(name="prefill_down_m8192", kind="linear", types="IQ4_XS", rows=str(HIDDEN), k=INTER, m=8192),
        # a merged layer of two types as the loader builds it, then its weights as bf16 (a check or a conversion of a checkpoint)
        dict(name="load_gate_up", kind="load", types="IQ3_S,Q5_K", rows="17408,17408", k=HIDDEN),
        # the embedding rows of a prompt chunk
        dict(name="embedding_2048", kind="embed", types="IQ2_S", vocab=VOCAB, k=HIDDEN, m=2048),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _type(rng):
    return F.TYPE_NAMES[rng.choice(sorted(F.SUPPORTED_TYPES))]


def _layer(rng):
    """A layer of the decoder or of one tensor-parallel rank of it: rows per shard and K."""
    name = rng.choice(sorted(LAYERS))
    rows, k = LAYERS[name]
    tp = rng.choice((1, 1, 2, 4))
    if name in ROW_PARALLEL:
        k //= tp
    else:
        rows = tuple(r // tp for r in rows)
    return rows, k


def draw(rng):
    kind = rng.choice(("decode", "decode", "prefill", "prefill", "head", "graph", "graph", "block", "mlp", "load", "embed"))
    if kind in ("decode", "prefill"):
        rows, k = _layer(rng)
        top = 32 if kind == "decode" else min(8192, int(MAX_FLOPS / (2.0 * sum(rows) * k)))
        m = _log_int(rng, 1 if kind == "decode" else 33, top)
        return dict(kind="linear", types=",".join(_type(rng) for _ in rows), rows=",".join(str(r) for r in rows), k=k, m=m)
    if kind == "head":      # whole or cut over the ranks, of a vocabulary of any size
        return dict(kind="linear", types=_type(rng), rows=str(_log_int(rng, VOCAB // 8, VOCAB)), k=HIDDEN, m=_log_int(rng, 1, 16))
    if kind == "graph":
        return dict(kind="stack", blocks=rng.randint(2, 4), types_seed=rng.randrange(1 << 20), m=_log_int(rng, 1, 128), graph=True)
    if kind == "block":
        return dict(kind="stack", blocks=1, types_seed=rng.randrange(1 << 20), m=_log_int(rng, 1, 2048), graph=False)
    if kind == "mlp":
        return dict(kind="mlp", types=",".join(_type(rng) for _ in range(3)), inter=256 * rng.randint(8, INTER // 256), m=_log_int(rng, 1, 48))
    if kind == "load":
        rows, k = _layer(rng)
        return dict(kind="load", types=",".join(_type(rng) for _ in rows), rows=",".join(str(r) for r in rows), k=k)
    return dict(kind="embed", types=_type(rng), vocab=_log_int(rng, 32000, VOCAB), k=HIDDEN, m=_log_int(rng, 1, 8192))


# ---- the layers and inputs ------------------------------------------------------------------------------

def _types(case):
    return [F.TYPE_IDS[t] for t in case["types"].split(",")]


def _rows(case):
    return [int(r) for r in case["rows"].split(",")]


def _shard_ids(n):
    return [None] if n == 1 else [0, 1] if n == 2 else ["q", "k", "v"]


def _raw(rows, k, types, seed):
    return [synth.random_blocks(n, k, t, seed=seed + 17 * i, device="cuda") for i, (n, t) in enumerate(zip(rows, types))]


def _linear(raws, k, types):
    lin = GGUFLinear(k, [r.shape[0] for r in raws])
    for raw, t, sid in zip(raws, types, _shard_ids(len(raws))):
        lin.load_shard(raw, t, sid)
    return lin.finalize()


def _activations(m, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((m, k), device="cuda", generator=g).to(torch.bfloat16)


def _stack_types(case):
    return draw_types(case["blocks"], case["types_seed"])


def _stack_step(layers, x):
    return [lin(x[name]) for blk in layers for name, lin in blk.items()]


def prepare(case, seed):
    kind = case["kind"]
    seed = 1000 * int(seed)
    if kind == "linear":
        types, rows, k = _types(case), _rows(case), case["k"]
        return {"kind": kind, "layer": _linear(_raw(rows, k, types, seed), k, types), "x": _activations(case["m"], k, seed + 500)}
    if kind == "stack":
        layers = []
        for b, t in enumerate(_stack_types(case)):
            blk = {}
            for j, (name, (rows, k)) in enumerate(LAYERS.items()):
                types = [t[s] for s in SHARDS[name]]
                blk[name] = _linear(_raw(rows, k, types, seed + 100 * b + 60 * (j + 1)), k, types)
            layers.append(blk)
        x = {name: _activations(case["m"], k, seed + 500 + j) for j, (name, (_, k)) in enumerate(LAYERS.items())}
        state = {"kind": kind, "layers": layers, "x": x}
        if case["graph"]:
            # warm-up and capture on a side stream; the step's new hidden states are copied into the graph's own input
            state["hidden"] = _activations(case["m"], HIDDEN, seed + 600)
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _stack_step(layers, x)
            torch.cuda.current_stream().wait_stream(side)
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"]):
                state["out"] = _stack_step(layers, x)
        return state
    if kind == "mlp":
        types, inter, m = _types(case), case["inter"], case["m"]
        g = torch.Generator(device="cuda").manual_seed(seed + 700)
        return {"kind": kind,
                "gate_up": _linear(_raw((inter, inter), HIDDEN, types[:2], seed), HIDDEN, types[:2]),
                "down": _linear(_raw((HIDDEN,), inter, types[2:], seed + 50), inter, types[2:]),
                "x": _activations(m, HIDDEN, seed + 500), "residual": _activations(m, HIDDEN, seed + 501),
                "norm": (torch.rand(HIDDEN, device="cuda", generator=g) * 0.02).to(torch.bfloat16)}
    if kind == "load":
        types, rows, k = _types(case), _rows(case), case["k"]
        return {"kind": kind, "raw": _raw(rows, k, types, seed), "types": types, "k": k}
    if kind == "embed":
        t = _types(case)[0]
        g = torch.Generator(device="cuda").manual_seed(seed + 800)
        return {"kind": kind, "table": _raw((case["vocab"],), case["k"], [t], seed)[0], "type": t,
                "ids": torch.randint(0, case["vocab"], (case["m"],), device="cuda", generator=g)}
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "stack":
        if "graph" not in state:
            return _stack_step(state["layers"], state["x"])
        state["x"]["qkv"].copy_(state["hidden"])
        state["graph"].replay()
        return state["out"]
    if kind == "mlp":
        norm = ops.PreAddRMSNorm(state["norm"], residual=state["residual"])
        h = state["gate_up"](state["x"], pre=norm)
        return [state["down"](h, pre=ops.PreSiluMul()), norm.residual_out, h]
    if kind == "load":
        lin = _linear(state["raw"], state["k"], state["types"])
        tiles = lin.gguf_tiles
        return [ops.dequantize_tiles(tiles[key], lin.gguf_tiles_rows[key], state["k"], lin.gguf_tiles_types[key], dtype=torch.bfloat16) for key in tiles]
    return loader.embedding_lookup(state["table"], state["type"], state["ids"])


# ---- what a pass needs, and how exact it is ----------------------------------------------------------------

def _gemm(m, rows, k, types):
    n = sum(rows)
    return {"bytes": sum(F.raw_bytes(t, r, k) for t, r in zip(types, rows)) + 2 * m * (k + n), "flops": 2.0 * m * n * k}


def _add(*works):
    return {key: sum(w[key] for w in works) for key in ("bytes", "flops")}


def work(case):
    kind = case["kind"]
    if kind == "linear":
        return _gemm(case["m"], _rows(case), case["k"], _types(case))
    if kind == "stack":
        return _add(*[_gemm(case["m"], rows, k, [t[s] for s in SHARDS[name]]) for t in _stack_types(case) for name, (rows, k) in LAYERS.items()])
    if kind == "mlp":
        types, inter, m = _types(case), case["inter"], case["m"]
        folded = {"bytes": 2 * (2 * m * HIDDEN + HIDDEN), "flops": 0.0}      # residual in and out, norm weight
        return _add(_gemm(m, (inter, inter), HIDDEN, types[:2]), _gemm(m, (HIDDEN,), inter, types[2:]), folded)
    if kind == "load":
        rows, k = _rows(case), case["k"]
        return {"bytes": sum(F.raw_bytes(t, r, k) for t, r in zip(_types(case), rows)) + 2 * sum(rows) * k, "flops": 0.0}
    return {"bytes": case["m"] * (8 + F.raw_row_bytes(_types(case)[0], case["k"]) + 2 * case["k"]), "flops": 0.0}


def tolerance(case):
    if case["kind"] in ("load", "embed"):
        return "exact"
    # bf16 outputs round at 2^-9 and the prefill path's weights at 2^-11; the MLP's second layer multiplies rounded values
    return {"rel": 1e-2 if case["kind"] == "mlp" else 5e-3, "max": 5e-2}
