"""What the performance of this package is measured on: the calls a model makes of its codebook
linears and routed layers, through the modules an engine drives (``CBLinear``, ``apply_shared_row``,
``CBMoE``), from one decode row to long prefills, in the benchmark's formats and in the product
formats checkpoints ship.

Decode batches of an engine run inside a captured CUDA graph; a case with ``graph`` replays one that
``prepare`` captured.  Prefill and stand-alone use call the modules directly."""
import math

import torch

from gridbook_b200 import formats, synth
from gridbook_b200.linear import CBLinear, apply_shared_row
from gridbook_b200.moe import CBMoE

# name -> (format, weight_global_scale).  The first four are the benchmark's; K12 .. K24 two-tier and
# the ragged FP8 rungs are what mixed-precision checkpoints assign layer by layer.
FORMATS = {
    "literal": (formats.NVFP4_LITERAL, 1.0 / 448.0),
    "k16v2": (formats.NVFP4_CB_K16, 1.0),
    "fp8k32": (formats.FP8_CB_K32, 1.0),
    "fp8lit": (formats.FP8_LITERAL, 1.0),
    "k12v2": (formats.CBFormat("fp4", 12, n_sub=2, scale_coding="v2"), 1.0),
    "k20v2": (formats.CBFormat("fp4", 20, n_sub=2, scale_coding="v2"), 1.0),
    "fp8k30": (formats.CBFormat("fp8", 30, n_sub=4), 1.0),
}

# the decoder layer of the benchmark's dense configurations, and its routed layer
LAYER = dict(hidden=5120, q=6144, kv=2048, inter=17408)
EXPERTS = dict(E=128, topk=8, hidden=2048, inter=768)


def listed():
    return [
        # one linear called on its own: the smallest call, all launch and call overhead
        dict(name="linear_m1_literal", kind="linear", fmt="literal", M=1, N=4096, K=4096, roles=1, graph=False),
        # one decode row through four decoder layers, as an engine replays it: the benchmark's workload
        dict(name="layers_m1_literal", kind="dense", fmt="literal", M=1, layers=4, roles=False, graph=True, **LAYER),
        # a few decode rows of an FP8-grid checkpoint whose fused modules keep one codebook per role
        dict(name="layer_m4_fp8k32_roles", kind="dense", fmt="fp8k32", M=4, layers=1, roles=True, graph=False, **LAYER),
        # the decode batch of a small server, in the product format checkpoints use most
        dict(name="layers_m16_k16v2", kind="dense", fmt="k16v2", M=16, layers=2, roles=False, graph=True, **LAYER),
        # a large decode batch
        dict(name="layer_m64_literal", kind="dense", fmt="literal", M=64, layers=1, roles=False, graph=False, **LAYER),
        # the ragged tail of a chunked prefill, a wider rung, one codebook per role
        dict(name="layer_m333_k20v2_roles", kind="dense", fmt="k20v2", M=333, layers=1, roles=True, graph=False,
             **LAYER),
        # prefill, both grids: configuration 2 of the benchmark
        dict(name="layer_m2048_literal", kind="dense", fmt="literal", M=2048, layers=1, roles=False, graph=False,
             **LAYER),
        dict(name="layer_m8192_fp8lit", kind="dense", fmt="fp8lit", M=8192, layers=1, roles=False, graph=False,
             **LAYER),
        # one token through a routed layer, as an engine replays it
        dict(name="moe_t1_literal", kind="moe", fmt="literal", fmt2="literal", T=1, graph=True, **EXPERTS),
        # a decode batch through a routed layer
        dict(name="moe_t48_k16v2", kind="moe", fmt="k16v2", fmt2="k16v2", T=48, graph=False, **EXPERTS),
        # one rank's share of the large layer with mixed grids: 32 of 256 experts, 512 routed pairs
        dict(name="moe_t64_mixed", kind="moe", fmt="fp8lit", fmt2="literal", T=64, graph=False, E=32, topk=8,
             hidden=7168, inter=2048),
        # prefill of a routed layer
        dict(name="moe_t4096_literal", kind="moe", fmt="literal", fmt2="literal", T=4096, graph=False, **EXPERTS),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    fmt = rng.choice(list(FORMATS))
    kind = rng.choice(["linear", "dense", "dense", "moe"])
    if kind == "linear":
        return dict(kind="linear", fmt=fmt, M=_log(rng, 1, 4096), N=_log(rng, 1024, 16384, 64),
                    K=_log(rng, 1024, 16384, 256), roles=rng.choice([1, 1, 2]), graph=rng.random() < 0.3)
    if kind == "dense":
        M = _log(rng, 1, 8192)
        return dict(kind="dense", fmt=fmt, M=M, layers=rng.choice([1, 2, 3]) if M <= 16 else 1,
                    roles=rng.random() < 0.5, graph=M <= 128 and rng.random() < 0.5,
                    hidden=_log(rng, 1024, 5120, 256), q=_log(rng, 1024, 6144, 256), kv=_log(rng, 256, 2048, 128),
                    inter=_log(rng, 2048, 17408, 256))
    T = _log(rng, 1, 4096)
    return dict(kind="moe", fmt=fmt, fmt2=rng.choice([fmt, fmt, "literal"]), T=T, graph=T <= 128 and rng.random() < 0.5,
                E=_log(rng, 8, 128), topk=rng.choice([2, 4, 8]), hidden=_log(rng, 1024, 2048, 256),
                inter=_log(rng, 256, 768, 256))


# ------------------------------------------------------------------------------------- the cases' parts
def _linears(case):
    """(name, widths of the fused parts, in features, one codebook per part) of the case's linears, in
    call order, one layer."""
    if case["kind"] == "linear":
        r = case["roles"]
        return [("linear", [case["N"] // r] * r, case["K"], r > 1)]
    h, q, kv, inter, roles = case["hidden"], case["q"], case["kv"], case["inter"], case["roles"]
    attn = ([("qkv_proj", [q, kv // 2, kv // 2], h, True)] if roles
            else [("q_proj", [q], h, False), ("kv_proj", [kv // 2, kv // 2], h, False)])
    return attn + [("o_proj", [h], q, False), ("gate_up_proj", [inter, inter], h, roles),
                   ("down_proj", [h], inter, False)]


def _scales(fmt, shape, gen, dev):
    return None if fmt.is_fp4 else (torch.rand(shape, generator=gen, device=dev) + 0.5) * 0.02


def _make_linear(fmt, gscale, name, parts, K, roles, gen, seed, dev):
    books = [synth.codebook_tables(fmt, seed + i) for i in range(len(parts) if roles else 1)]
    lin = CBLinear(fmt, K, parts, books, global_scale=gscale, prefix=name)
    return lin.load(synth.make_packed_device(fmt, sum(parts), K, gen, dev), _scales(fmt, sum(parts), gen, dev), dev)


def _captured(step):
    """A replay of ``step`` as an engine captures it: warmed up on a side stream, then recorded."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    return dict(replay=graph.replay, out=out, step=step)      # the step owns what the graph reads


def _dense_step(layers, inputs):
    outs = []
    for lins in layers:
        xs = inputs
        if len(lins) == 5:                   # q and kv read the same rows
            outs += apply_shared_row(lins[:2], xs[0])
            lins, xs = lins[2:], xs[1:]
        outs += [lin(x) for lin, x in zip(lins, xs)]
    return outs


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)

    def rows(m, k):
        return torch.randn(m, k, generator=gen, device=dev).to(torch.bfloat16)

    fmt, gscale = FORMATS[case["fmt"]]
    if case["kind"] == "moe":
        E, hidden, inter, T = case["E"], case["hidden"], case["inter"], case["T"]
        fmt2 = FORMATS[case["fmt2"]][0]
        moe = CBMoE(fmt, fmt2, E, hidden, inter, synth.codebook_tables(fmt, seed), synth.codebook_tables(fmt2, seed + 1))
        moe.load(synth.make_packed_device(fmt, E * 2 * inter, hidden, gen, dev).view(E, 2 * inter, -1),
                 synth.make_packed_device(fmt2, E * hidden, inter, gen, dev).view(E, hidden, -1),
                 _scales(fmt, (E, 2 * inter), gen, dev), _scales(fmt2, (E, hidden), gen, dev), dev)
        # router: softmax over N(0, 1) logits, top-k, renormalised
        w, ids = torch.softmax(torch.randn(T, E, generator=gen, device=dev), -1).topk(case["topk"], -1)
        w, ids, x = w / w.sum(-1, keepdim=True), ids.to(torch.int32), rows(T, hidden)
        step = lambda: moe(x, w, ids)  # noqa: E731
    else:
        spec, n = _linears(case), case.get("layers", 1)
        layers = [[_make_linear(fmt, gscale, f"layers.{i}.{name}", parts, K, roles, gen, seed + 16 * i, dev)
                   for name, parts, K, roles in spec] for i in range(n)]
        ins = spec[1:] if len(spec) == 5 else spec
        inputs = [rows(case["M"], K) for _, _, K, _ in ins]
        step = lambda: _dense_step(layers, inputs)  # noqa: E731
    return _captured(step) if case["graph"] else dict(step=step)


def run(state):
    if "replay" in state:
        state["replay"]()
        return state["out"]
    return state["step"]()


def work(case):
    """Packed weights and scales of what is read, each once; activations in, results out."""
    fmt = FORMATS[case["fmt"]][0]

    def packed(f, n, k):
        return n * (f.packed_row_bytes(k) + (0 if f.is_fp4 else 4))

    if case["kind"] == "moe":
        E, topk, h, inter, T = case["E"], case["topk"], case["hidden"], case["inter"], case["T"]
        hit = E * (1.0 - (1.0 - topk / E) ** T)          # experts a batch of random routings touches
        per = packed(fmt, 2 * inter, h) + packed(FORMATS[case["fmt2"]][0], h, inter)
        return {"bytes": hit * per + 4 * T * h + 8 * T * topk, "flops": 2.0 * T * topk * 3 * inter * h}
    M, nbytes, flops = case["M"], 0.0, 0.0
    spec, n = _linears(case), case.get("layers", 1)
    for _, parts, K, _ in spec:
        nbytes += packed(fmt, sum(parts), K) + 2 * M * sum(parts)
        flops += 2.0 * M * sum(parts) * K
    nbytes = n * nbytes + 2 * M * sum(K for _, _, K, _ in (spec[1:] if len(spec) == 5 else spec))
    return {"bytes": nbytes, "flops": n * flops}


def tolerance(case):
    """bf16 results of fp32 sums in another order: single roundings to the other neighbour.  In a routed
    layer such a difference can move an activation of the second projection by one step of its
    quantisation grid."""
    if case["kind"] == "moe":
        return {"rel": 1e-2}
    return {"rel": 3e-3, "max": 0.05}
