"""Whole-layer CUDA-graph capture (the engine's FULL decode graphs, docs/KERNELS.md:1018-1071 of the
reference): a decoder block's codebook linears and its routed layer, driven through the plugin
methods, are captured at every decode size AND at prefill sizes - none of the routes reads a
device value on the host - and a replay on new inputs returns what eager execution returns, bit
for bit (capture on == capture off)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def block():
    """q, kv, o, gate_up, down (small shapes with the stack's proportions) + one routed layer."""
    from gridbook_b200 import _native, synth
    from gridbook_b200.formats import NVFP4_LITERAL
    from gridbook_b200.linear import CBLinear
    from gridbook_b200.moe import CBMoE
    _native.prepare(0)
    dev = torch.device("cuda:0")
    fmt = NVFP4_LITERAL
    hidden, inter = 1024, 2048
    gen = torch.Generator(device=dev).manual_seed(3)
    shapes = {"q": ([768], hidden), "kv": ([128, 128], hidden), "o": ([hidden], 768),
              "gate_up": ([inter, inter], hidden), "down": ([hidden], inter)}
    lins = {}
    for i, (name, (parts, K)) in enumerate(shapes.items()):
        lin = CBLinear(fmt, K, parts, [synth.codebook_tables(fmt, i)], global_scale=1.0 / 448.0, prefix=f"blk.{name}")
        lins[name] = lin.load(synth.make_packed_device(fmt, sum(parts), K, gen, dev), None, dev)
    E, topk, minter = 16, 4, 256
    moe = CBMoE(fmt, fmt, E, hidden, minter, synth.codebook_tables(fmt, 7), synth.codebook_tables(fmt, 8))
    moe.load(synth.make_packed_device(fmt, E * 2 * minter, hidden, gen, dev).view(E, 2 * minter, -1),
             synth.make_packed_device(fmt, E * hidden, minter, gen, dev).view(E, hidden, -1), None, None, dev)
    return dev, lins, moe, hidden, inter, E, topk


def _forward(lins, moe, inter, x, tw, ids):
    from gridbook_b200.linear import apply_shared_row
    q, kv = apply_shared_row([lins["q"], lins["kv"]], x)
    a = lins["o"](q)                                     # stands in for attention: shapes only
    h = lins["gate_up"](a)
    y = lins["down"](torch.nn.functional.silu(h[..., :inter]) * h[..., inter:])
    return y + moe(a, tw, ids), kv


@pytest.mark.parametrize("T", [1, 2, 4, 8, 16, 40, 300, 1800])
def test_block_capture_equals_eager(block, T):
    from gridbook_b200 import _native, synth
    dev, lins, moe, hidden, inter, E, topk = block
    ids, tw = synth.make_routing(T, E, topk, seed=T)
    x = synth.bf16_tensor(synth.make_activations(T, hidden, seed=T), dev)
    tw_d, ids_d = torch.from_numpy(tw).to(dev), torch.from_numpy(ids).to(dev)
    _forward(lins, moe, inter, x, tw_d, ids_d)           # warm-up outside the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out, kv = _forward(lins, moe, inter, x, tw_d, ids_d)
    for seed in (100 + T, 200 + T):                      # two replays on new inputs and new routings
        ids2, tw2 = synth.make_routing(T, E, topk, seed=seed)
        x.copy_(synth.bf16_tensor(synth.make_activations(T, hidden, seed=seed), dev))
        tw_d.copy_(torch.from_numpy(tw2).to(dev))
        ids_d.copy_(torch.from_numpy(ids2).to(dev))
        g.replay()
        torch.cuda.synchronize()
        want, want_kv = _forward(lins, moe, inter, x, tw_d, ids_d)
        torch.cuda.synchronize()
        assert torch.equal(out, want) and torch.equal(kv, want_kv), (T, seed)
    assert _native.device_status(0) == 0


def test_first_call_of_a_shape_under_capture(block):
    """Nothing that a capture made is taken by a later call outside the graph: it was recorded, not run."""
    from gridbook_b200 import _native, synth
    dev, lins, moe, hidden, inter, E, _ = block
    from gridbook_b200.linear import apply_shared_row
    T, topk = 6, 3                                       # a top-k that no other test uses
    ids, tw = synth.make_routing(T, E, topk, seed=T)
    x = synth.bf16_tensor(synth.make_activations(T, hidden, seed=T), dev)
    tw_d, ids_d = torch.from_numpy(tw).to(dev), torch.from_numpy(ids).to(dev)
    pair = [lins["kv"], lins["q"]]                       # an order that no other test uses
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = moe(x, tw_d, ids_d)
        rows = apply_shared_row(pair, x[:1])
    want, want_rows = moe(x, tw_d, ids_d), apply_shared_row(pair, x[:1])     # before any replay
    one_by_one = torch.cat([moe(x[t:t + 1], tw_d[t:t + 1], ids_d[t:t + 1]) for t in range(T)])
    torch.cuda.synchronize()
    assert torch.equal(want, one_by_one)
    assert all(torch.equal(a, lin(x[:1])) for a, lin in zip(want_rows, pair))
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and all(torch.equal(a, b) for a, b in zip(rows, want_rows))
    assert _native.device_status(0) == 0


def test_batch_sizes_share_what_a_plan_keeps(block):
    """Every batch size reads the front of one list of tokens, on whichever stream it runs."""
    from gridbook_b200 import synth
    dev, _, moe, hidden, inter, E, _ = block
    topk, x = 2, synth.bf16_tensor(synth.make_activations(200, hidden, seed=9), dev)
    ids, tw = synth.make_routing(200, E, topk, seed=9)
    tw_d, ids_d = torch.from_numpy(tw).to(dev), torch.from_numpy(ids).to(dev)
    moe(x[:8], tw_d[:8], ids_d[:8])
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for T in range(1, 200):
        moe(x[:T], tw_d[:T], ids_d[:T])
        with torch.cuda.stream(side):
            moe(x[:T], tw_d[:T], ids_d[:T])
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() - before <= 16 << 10   # lists of 256 and 512 pairs; one each would be 200 KB
