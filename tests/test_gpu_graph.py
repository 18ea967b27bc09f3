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


def _layer(name, N, K, dev):
    from gridbook_b200 import formats, synth
    from gridbook_b200.linear import CBLinear
    fmt = {"literal": formats.NVFP4_LITERAL, "k16": formats.NVFP4_CB_K16, "fp8k32": formats.FP8_CB_K32}[name]
    gen = torch.Generator(device=dev).manual_seed(N)
    lin = CBLinear(fmt, K, [N], [synth.codebook_tables(fmt, N)], global_scale=1.0 / 448.0 if name == "literal" else 1.0, prefix=f"s{N}")
    scale = None if fmt.is_fp4 else (torch.rand(N, generator=gen, device=dev) + 0.5) * 0.02
    return lin.load(synth.make_packed_device(fmt, N, K, gen, dev), scale, dev)


def _rows(n, M, K, dev):
    gen = torch.Generator(device=dev).manual_seed(n)
    return [torch.randn(M, K, generator=gen, device=dev).to(torch.bfloat16) for _ in range(n)]


@pytest.mark.parametrize("name", ["literal", "k16", "fp8k32"])
def test_one_layer_on_several_streams_and_threads(name):
    """Decode calls of one layer that overlap on the GPU, from two streams and a graph, and calls of two threads that share a
    stream: each has scratch of its own."""
    import threading
    from gridbook_b200 import _native
    _native.prepare(0)
    dev = torch.device("cuda:0")
    lin = _layer(name, 1536, 4096, dev)
    xs = _rows(3, 4, 4096, dev)
    want = [lin(x) for x in xs]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = lin(xs[2])
    torch.cuda.synchronize()
    streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], [], []]
    for _ in range(40):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                if i == 2:
                    g.replay()
                    got[2].append(captured.clone())
                else:
                    got[i].append(lin(xs[i]))
    torch.cuda.synchronize()

    def calls(i):
        got[i] += [lin(xs[i]) for _ in range(100)]

    threads = [threading.Thread(target=calls, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert [len(g) for g in got] == [140, 140, 40]
    for i in range(3):
        assert all(torch.equal(y, want[i]) for y in got[i]), (name, i)


@pytest.mark.parametrize("M", [1, 4, 300])
@pytest.mark.parametrize("name", ["literal", "fp8k32"])
def test_the_first_cuda_call_of_a_thread(name, M):
    """A thread that has made no CUDA call yet has no context, in which the driver encodes a launch's tensor maps."""
    from concurrent.futures import ThreadPoolExecutor
    from gridbook_b200 import _native
    _native.prepare(0)
    dev = torch.device("cuda:0")
    lin = _layer(name, 512, 2048, dev)
    (x,) = _rows(1, M, 2048, dev)
    want = lin(x)
    torch.cuda.synchronize()
    with ThreadPoolExecutor(1) as pool:
        got = pool.submit(lin, x).result()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and _native.device_status(0) == 0


def test_one_row_of_a_layer_on_several_streams():
    """The table kernel's slots are one stream's each, and a graph's: streams past the number that is kept, one layer and two
    that share a row, in turn."""
    from gridbook_b200 import _native
    from gridbook_b200.linear import apply_shared_row
    _native.prepare(0)
    dev = torch.device("cuda:0")
    a, b = _layer("literal", 1024, 2048, dev), _layer("literal", 512, 2048, dev)
    (x,) = _rows(1, 1, 2048, dev)
    want = [a(x), *apply_shared_row([a, b], x)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = [a(x), *apply_shared_row([a, b], x)]
    torch.cuda.synchronize()
    for _ in range(2):
        for s in [torch.cuda.Stream() for _ in range(10)]:
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                g.replay()
                got = [a(x), *apply_shared_row([a, b], x)]
            torch.cuda.current_stream().wait_stream(s)
            torch.cuda.synchronize()
            assert all(torch.equal(u, v) and torch.equal(w, v) for u, w, v in zip(got, captured, want))
    assert _native.device_status(0) == 0
