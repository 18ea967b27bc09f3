"""The decode-batch kernel on the block-scaled FP4 tensor cores: the exact three-term split of the bucketed
activations, edges of the row, tile, slice and pass counts, codebooks that change with the role, scales
of either sign and scales that are no E4M3 value (which must take the other kernel), dense and per expert."""
import numpy as np
import pytest
import torch

from oracle import cb_oracle as O
from oracle import oracle_kwargs
from tests.helpers import assert_close_bf16, f32_of, oracle_linear

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from gridbook_b200 import _native
    _native.prepare(0)
    return torch.device("cuda:0")


def _fmt(name):
    from gridbook_b200 import formats as F
    if name == "lit":
        return F.NVFP4_LITERAL
    return F.CBFormat("fp4", int(name[1:]), n_sub=2, scale_coding="v2")


def _tables(fmt, flat):
    out, pos = [], 0
    for r, d in fmt.table_shapes():
        out.append(torch.from_numpy(flat[pos:pos + r * d].reshape(r, d).copy()))
        pos += r * d
    return out


def _linear(fmt, d, parts, dev, **kw):
    from gridbook_b200.linear import CBLinear
    n = fmt.codebook_elems()
    books = [_tables(fmt, d["cb"][i * n:(i + 1) * n]) for i in range(d["cb"].size // n)]
    lin = CBLinear(fmt, d["K"], parts, books, global_scale=d["global_scale"] or 1.0, **kw)
    return lin.load(torch.from_numpy(d["qw"]), None, dev)


def _wide_rows(M, K, seed):
    """Groups from far below to far above the row's typical magnitude, a zero group and a zero row."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((M, K // 16, 16)).astype(np.float32)
    x *= np.exp2(rng.integers(-9, 3, (M, K // 16, 1))).astype(np.float32)
    x[:, 3] = 0.0
    x = x.reshape(M, K)
    if M > 2:
        x[M // 2] = 0.0
    return O.bf16_round(x)


@pytest.mark.parametrize("name", ["lit", "k12", "k16", "k20", "k24"])
@pytest.mark.parametrize("M,N,K", [(2, 64, 256), (5, 129, 512), (8, 200, 2048), (9, 384, 1280), (16, 640, 5120), (3, 1024, 17408)])
def test_decode_rows_match_the_oracle(dev, name, M, N, K):
    from gridbook_b200 import _native, synth
    fmt = _fmt(name)
    d = synth.make_linear(fmt, N, K, seed=M + N, global_scale=1.0 / 448.0 if name == "lit" else None, super_span=None)
    lin = _linear(fmt, d, [N], dev)
    for x in (synth.make_activations(M, K, seed=K), _wide_rows(M, K, M)):
        y = lin(synth.bf16_tensor(x, dev))
        torch.cuda.synchronize()
        assert _native.device_status(0) == 0
        assert_close_bf16(f32_of(y), oracle_linear(x, d), f"{name} {M}x{N}x{K}", atol_rel=1e-6)


@pytest.mark.parametrize("M,K", [(64, 17408), (80, 8448), (1, 40960)])
def test_rows_split_over_a_cluster(dev, M, K):
    """Rows that two to eight CTAs hold: more clusters than run at once, uneven shares, one row alone; each row's largest
    group in another CTA's share."""
    from gridbook_b200 import _native, kernels, synth
    fmt, N = _fmt("k16"), 136
    d = synth.make_linear(fmt, N, K, seed=M)
    lin = _linear(fmt, d, [N], dev)
    assert M <= kernels.row_batch_max_rows(lin._cb_weight)
    x = _wide_rows(M, K, M).reshape(M, K // 16, 16)
    x[np.arange(M), np.arange(M) * 37 % (K // 16)] *= np.float32(64)
    y = lin(synth.bf16_tensor(x.reshape(M, K), dev))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert_close_bf16(f32_of(y), oracle_linear(x.reshape(M, K), d), f"M={M} K={K}", atol_rel=1e-6)


@pytest.mark.parametrize("name", ["lit", "k16"])
@pytest.mark.parametrize("M", [1, 15, 17, 31, 32, 33, 48, 64, 65, 100, 128])
def test_row_counts_past_sixteen(dev, name, M):
    from gridbook_b200 import _native, kernels, synth
    fmt = _fmt(name)
    N, K = 320, 1536
    d = synth.make_linear(fmt, N, K, seed=M, global_scale=1.0 / 448.0 if name == "lit" else None)
    lin = _linear(fmt, d, [N], dev)
    if M > kernels.row_batch_max_rows(lin._cb_weight):
        pytest.skip("past the decode batches of this format")
    x = _wide_rows(M, K, M)
    y = lin(synth.bf16_tensor(x, dev))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert_close_bf16(f32_of(y), oracle_linear(x, d), f"{name} M={M}", atol_rel=1e-6)


@pytest.mark.parametrize("name", ["lit", "k16", "k20"])
@pytest.mark.parametrize("parts,K", [([96, 96], 1024), ([256, 64, 64], 2560), ([40, 200, 130, 14], 512), ([17408, 17408], 256)])
def test_roles_with_their_own_codebooks(dev, name, parts, K):
    from gridbook_b200 import _native, synth
    fmt = _fmt(name)
    N, M = sum(parts), 7
    d = synth.make_linear(fmt, N, K, seed=N, n_books=len(parts))
    d["cb_row_offset"] = np.repeat(np.arange(len(parts)), parts).astype(np.int32) * fmt.codebook_elems()
    lin = _linear(fmt, d, parts, dev)
    x = synth.make_activations(M, K, seed=5)
    y = lin(synth.bf16_tensor(x, dev))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert_close_bf16(f32_of(y), oracle_linear(x, d), f"{name} roles {parts}")


def test_negative_scale_bytes_and_non_finite_rows(dev):
    from gridbook_b200 import synth
    fmt = _fmt("lit")
    M, N, K = 6, 256, 1024
    d = synth.make_linear(fmt, N, K, seed=4)
    blk = d["qw"].reshape(N, K // 256, 48)
    blk[:, :, 32:] |= (np.random.default_rng(1).integers(0, 2, (N, K // 256, 16)) * 128).astype(np.uint8)
    lin = _linear(fmt, d, [N], dev)
    x = synth.make_activations(M, K, seed=1)
    assert_close_bf16(f32_of(lin(synth.bf16_tensor(x, dev))), oracle_linear(x, d), "negative scales")
    x[2, 40] = np.nan
    x[4, 500] = np.inf
    y = f32_of(lin(synth.bf16_tensor(x, dev)))
    assert np.isnan(y[2]).all() and np.isnan(y[4]).all() and np.isfinite(y[[0, 1, 3, 5]]).all()
    keep = [0, 1, 3, 5]
    assert_close_bf16(y[keep], oracle_linear(x[keep], d), "finite rows beside them")


def test_scales_off_the_e4m3_grid_take_the_other_kernel(dev):
    """Super exponents past the E4M3 range: the block-scaled operand cannot hold them."""
    from gridbook_b200 import synth
    fmt = _fmt("k16")
    M, N, K = 4, 256, 1024
    d = synth.make_linear(fmt, N, K, seed=8)
    d["qw"].reshape(N, K // 256, 73)[:, :, 64] = np.random.default_rng(2).choice([100, 126, 140], (N, K // 256)).astype(np.uint8)
    lin = _linear(fmt, d, [N], dev)
    x = synth.make_activations(M, K, seed=3)
    assert_close_bf16(f32_of(lin(synth.bf16_tensor(x, dev))), oracle_linear(x, d), "scales off the grid")


@pytest.mark.parametrize("f13,f2", [("lit", "lit"), ("k16", "k16"), ("k20", "lit"), ("k12", "k24")])
@pytest.mark.parametrize("T", [3, 40, 150, 700])
def test_routed_layer_matches_the_loop_chain(dev, f13, f2, T):
    """Experts without rows, with a few and with several passes; a dropped (-1) slot."""
    from gridbook_b200 import _native, synth
    from gridbook_b200.moe import CBMoE
    fmt13, fmt2 = _fmt(f13), _fmt(f2)
    E, hidden, inter, topk = 8, 512, 256, 2
    w13d, w2d = synth.make_moe(fmt13, fmt2, E, hidden, inter, seed=T)
    ids, tw = synth.make_routing(T, E - 1, topk, seed=T)
    ids[2, 1] = -1
    x = synth.make_activations(T, hidden, seed=T + 1)
    ref = O.moe_loop_chain(x, np.where(ids < 0, 0, ids), np.where(ids < 0, 0.0, tw).astype(np.float32), w13d, w2d, E=E,
                           hidden=hidden, inter=inter, fmt13=oracle_kwargs(fmt13), fmt2=oracle_kwargs(fmt2), scale_rule="recip")
    moe = CBMoE(fmt13, fmt2, E, hidden, inter, _tables(fmt13, w13d["cb"]), _tables(fmt2, w2d["cb"]))
    moe.load(torch.from_numpy(w13d["qw"]), torch.from_numpy(w2d["qw"]), None, None, dev)
    moe.method.sorted_min_pairs_per_expert = 0
    moe.method.sorted_min_pairs_other = 0
    got = f32_of(moe(synth.bf16_tensor(x, dev), torch.from_numpy(tw).to(dev), torch.from_numpy(ids).to(dev)))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert "sorted rows" in moe._cb_route
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= 3e-3
    assert np.abs(got - ref).max() <= 2e-2 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("name", ["lit", "k16", "k20"])
@pytest.mark.parametrize("T", [40, 60, 300, 1700])
def test_several_tiles_per_cta_with_an_odd_number_of_superblocks(dev, name, T):
    """More expert tiles than SMs, three superblocks of K in the down projection: units change from tile
    to tile; up to sixteen rows a pass, more, and the stack decoded once (1700 tokens: 170 rows an
    expert) against the decoded bf16 stack's grouped GEMM, run to run the same bits."""
    from gridbook_b200 import synth
    from gridbook_b200.moe import CBMoE
    fmt = _fmt(name)
    E, hidden, inter, topk = 40, 1024, 768, 4
    w13d, w2d = synth.make_moe(fmt, fmt, E, hidden, inter, seed=T)
    ids, tw = synth.make_routing(T, E, topk, seed=T)
    x = synth.bf16_tensor(synth.make_activations(T, hidden, seed=T + 1), dev)
    moe = CBMoE(fmt, fmt, E, hidden, inter, _tables(fmt, w13d["cb"]), _tables(fmt, w2d["cb"]))
    moe.load(torch.from_numpy(w13d["qw"]), torch.from_numpy(w2d["qw"]), None, None, dev)
    args = x, torch.from_numpy(tw).to(dev), torch.from_numpy(ids).to(dev)
    got = [moe(*args).float() for _ in range(3)]
    assert "sorted rows" in moe._cb_route
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    moe.method.prefill_min_pairs_per_expert = 1
    ref = moe(*args).float()
    assert "grouped prefill" in moe._cb_route
    assert float((got[0] - ref).norm() / ref.norm()) <= 3e-3


def _zero_first_group(fmt, qw, cb):
    """Entry 0 of every (sub-)table becomes the zero codeword; returns a function that points the first
    group of the given packed rows at it."""
    pos = 0
    for _ in range(cb.size // fmt.codebook_elems()):
        for r, dim in fmt.table_shapes():
            cb[pos:pos + dim] = 0.0
            pos += r * dim

    def clear(rows):
        rows[..., :2 if fmt.mode == "full" else fmt.k // 4] = 0
    return clear


def _outlier_rows(M, K, seed):
    """Every third row: a first group 2^14 and more above all the others, which span 2^20 themselves;
    the next: groups anywhere within 2^30; the third kind is ordinary."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((M, K // 16, 16)).astype(np.float32)
    x[0::3] *= np.exp2(rng.integers(-28, -8, x[0::3].shape[:2] + (1,))).astype(np.float32)
    x[0::3, 0] = rng.standard_normal(x[0::3, 0].shape) * 128.0
    x[1::3] *= np.exp2(rng.integers(-25, 6, x[1::3].shape[:2] + (1,))).astype(np.float32)
    return O.bf16_round(x.reshape(M, K))


@pytest.mark.parametrize("name", ["lit", "k12", "k16", "k20", "k24"])
@pytest.mark.parametrize("M,N,K", [(2, 64, 256), (7, 384, 1280), (16, 200, 5120), (3, 136, 17408), (20, 129, 768), (64, 320, 1536),
                                   (70, 128, 1024)])
def test_groups_far_below_the_rows_largest_keep_their_precision(dev, name, M, N, K):
    """Half of the weight rows are zero under the outlier, so that their result is the small groups' alone;
    every row is held to the oracle by its own magnitude."""
    from gridbook_b200 import _native, kernels, synth
    fmt = _fmt(name)
    d = synth.make_linear(fmt, N, K, seed=M + K, global_scale=1.0 / 448.0 if name == "lit" else None)
    _zero_first_group(fmt, d["qw"], d["cb"])(d["qw"][::2])
    lin = _linear(fmt, d, [N], dev)
    if M > kernels.row_batch_max_rows(lin._cb_weight):
        pytest.skip("past the decode batches of this format")
    x = _outlier_rows(M, K, M)
    y = f32_of(lin(synth.bf16_tensor(x, dev)))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    ref = oracle_linear(x, d)
    for part in (slice(0, None, 2), slice(1, None, 2)):      # weight rows without and with the outlier
        for m in range(M):
            top = np.abs(ref[m, part]).max()
            assert_close_bf16(y[m, part] / top, ref[m, part] / top, f"{name} {M}x{N}x{K} row {m}", atol_rel=1e-6)


def test_left_out_groups_under_codebooks_per_role(dev):
    """The rows of a tile are multiplied by their own role's codebook, also where the CTA has moved on to the next."""
    from gridbook_b200 import _native, synth
    fmt, M, K, parts = _fmt("k16"), 6, 512, [12800, 12800]
    N = sum(parts)
    d = synth.make_linear(fmt, N, K, seed=3, n_books=2)
    d["cb_row_offset"] = np.repeat(np.arange(2), parts).astype(np.int32) * fmt.codebook_elems()
    _zero_first_group(fmt, d["qw"], d["cb"])(d["qw"])
    x = _outlier_rows(M, K, 1)
    y = f32_of(_linear(fmt, d, parts, dev)(synth.bf16_tensor(x, dev)))
    assert _native.device_status(0) == 0
    ref = oracle_linear(x, d)
    for m in range(M):
        top = np.abs(ref[m]).max()
        assert_close_bf16(y[m] / top, ref[m] / top, f"row {m}", atol_rel=1e-6)


@pytest.mark.parametrize("f13,f2", [("lit", "lit"), ("k16", "k16"), ("k20", "lit"), ("lit", "k24")])
@pytest.mark.parametrize("T", [6, 50, 150, 700])
def test_left_out_groups_of_a_routed_layer(dev, f13, f2, T):
    """Outliers in front of both projections whose weights are zero under them (but for the sixteen features
    that carry the outlier into the second): few rows a pass, more, and the stack decoded once."""
    from gridbook_b200 import _native, synth
    from gridbook_b200.moe import CBMoE
    fmt13, fmt2 = _fmt(f13), _fmt(f2)
    E, hidden, inter, topk = 8, 512, 768, 2
    w13d, w2d = synth.make_moe(fmt13, fmt2, E, hidden, inter, seed=T)
    clear13, clear2 = _zero_first_group(fmt13, w13d["qw"], w13d["cb"]), _zero_first_group(fmt2, w2d["qw"], w2d["cb"])
    w13 = w13d["qw"].reshape(E, 2 * inter, -1)
    clear13(w13[:, 16:inter])
    clear13(w13[:, inter + 16:])
    clear2(w2d["qw"].reshape(E, hidden, -1))
    ids, tw = synth.make_routing(T, E, topk, seed=T)
    rng = np.random.default_rng(T)
    x = rng.standard_normal((T, hidden)).astype(np.float32)
    x[:, 16:] *= np.float32(2.0 ** -5)
    x[:, :16] *= np.float32(2.0 ** 11)
    x = O.bf16_round(x)
    ref = O.moe_loop_chain(x, ids, tw, w13d, w2d, E=E, hidden=hidden, inter=inter, fmt13=oracle_kwargs(fmt13),
                           fmt2=oracle_kwargs(fmt2), scale_rule="recip")
    moe = CBMoE(fmt13, fmt2, E, hidden, inter, _tables(fmt13, w13d["cb"]), _tables(fmt2, w2d["cb"]))
    moe.load(torch.from_numpy(w13d["qw"]), torch.from_numpy(w2d["qw"]), None, None, dev)
    moe.method.sorted_min_pairs_per_expert = 0
    moe.method.sorted_min_pairs_other = 0
    got = f32_of(moe(synth.bf16_tensor(x, dev), torch.from_numpy(tw).to(dev), torch.from_numpy(ids).to(dev)))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert "sorted rows" in moe._cb_route
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() <= 1e-2                                 # one step of the second bucket in a few values, as in the test above


@pytest.mark.parametrize("name", ["lit", "k16", "k20", "k24"])
@pytest.mark.parametrize("T", [40, 150, 450])
def test_left_out_groups_between_tiles_of_one_cta(dev, name, T):
    """Sums that groups are added to are read out while the CTA's next tile is decoded: more expert tiles than SMs,
    several passes of a tile, against the decoded bf16 stack's grouped GEMM."""
    from gridbook_b200 import _native, synth
    from gridbook_b200.moe import CBMoE
    fmt = _fmt(name)
    E, hidden, inter, topk = 40, 2048, 768, 4
    w13d, w2d = synth.make_moe(fmt, fmt, E, hidden, inter, seed=T)
    _zero_first_group(fmt, w13d["qw"], w13d["cb"])(w13d["qw"].reshape(E, 2 * inter, -1))
    ids, tw = synth.make_routing(T, E, topk, seed=T)
    moe = CBMoE(fmt, fmt, E, hidden, inter, _tables(fmt, w13d["cb"]), _tables(fmt, w2d["cb"]))
    moe.load(torch.from_numpy(w13d["qw"]), torch.from_numpy(w2d["qw"]), None, None, dev)
    x = _outlier_rows(T, hidden, T)
    args = synth.bf16_tensor(x, dev), torch.from_numpy(tw).to(dev), torch.from_numpy(ids).to(dev)
    moe.method.sorted_min_pairs_per_expert = 0
    moe.method.prefill_min_pairs_per_expert = 1 << 30
    got = moe(*args).float()
    assert "sorted rows" in moe._cb_route
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    moe.method.prefill_min_pairs_per_expert = 1
    ref = moe(*args).float()
    assert "grouped prefill" in moe._cb_route
    # A first projection that rounds to the other bf16 neighbour can move a value of the second bucket by a step,
    # at most a third of the larger neighbour (4 and 6 on the E2M1 grid), so a row that one value dominates moves
    # by up to a third; a row whose small groups were dropped is off by its whole length.
    err = (got - ref).norm(dim=1) / ref.norm(dim=1)
    assert float(err.max()) <= 1 / 3 and float(err.mean()) <= 3e-3


@pytest.mark.parametrize("name,M", [("lit", 16), ("lit", 33), ("lit", 64), ("k12", 16), ("k16", 16), ("k16", 17), ("k16", 64), ("k20", 16)])
def test_rings_wrap_from_tile_to_tile(dev, name, M):
    """More tiles than SMs, an odd number of units per tile: every ring depth (four or eight units, by format and row
    count) goes round, and crosses from one tile to the next, with a half-filled raw stage where one holds two."""
    from gridbook_b200 import _native, synth
    fmt = _fmt(name)
    N, K = 128 * 2 * 148 + 40, 256 * 9
    d = synth.make_linear(fmt, N, K, seed=M, global_scale=1.0 / 448.0 if name == "lit" else None)
    lin = _linear(fmt, d, [N], dev)
    x = _wide_rows(M, K, M)
    y = lin(synth.bf16_tensor(x, dev))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert_close_bf16(f32_of(y), oracle_linear(x, d), f"{name} M={M} {N}x{K}", atol_rel=1e-6)


@pytest.mark.parametrize("M", [1, 2, 16, 17, 64, 100, 128, 300])
@pytest.mark.parametrize("name", ["lit", "k12", "k16", "k20", "fp8lit", "fp8k32", "fp8k30"])
def test_rows_shared_by_several_matrices(dev, name, M):
    """Rows bucketed or quantised once for matrices of different heights, codebooks, scales and outputs (in one launch for the
    decode batches of the fp4 grid): as each layer gives by itself, up to the order of the sum, with misaligned and
    strided rows among them, and nothing replaced where a layer is watched."""
    from gridbook_b200 import _native, formats, synth
    from gridbook_b200.linear import CBLinear, apply_shared_row
    fmt = {"fp8lit": formats.FP8_LITERAL, "fp8k32": formats.FP8_CB_K32, "fp8k30": formats.CBFormat("fp8", 30, n_sub=4)}.get(name) or _fmt(name)
    gen = torch.Generator(device=dev).manual_seed(M)
    K, lins = 1792, []
    for i, N in enumerate((1000, 129, 640)):
        lin = CBLinear(fmt, K, [N], [synth.codebook_tables(fmt, i)], global_scale=(1.0 / 448.0 if name == "lit" else 1.0) * (i + 1), prefix=f"m{i}")
        scale = None if fmt.is_fp4 else (torch.rand(N, generator=gen, device=dev) + 0.5) * 0.02
        lins.append(lin.load(synth.make_packed_device(fmt, N, K, gen, dev), scale, dev))
    wide = torch.randn(M, K + 64, generator=gen, device=dev).to(torch.bfloat16)
    for x in (wide[:, :K].contiguous(), wide[:, 64:], wide.view(-1)[8:8 + M * K].view(M, K)):
        want = [lin(x) for lin in lins]
        got = apply_shared_row(lins, x)
        torch.cuda.synchronize()
        assert _native.device_status(0) == 0
        for a, b in zip(got, want):
            assert a.shape == b.shape and a.is_contiguous()
            assert_close_bf16(f32_of(a), f32_of(b), f"{name} M={M}", atol_rel=1e-6)
    seen = []
    hook = lins[1].register_forward_hook(lambda mod, args, out: seen.append(1))
    assert len(apply_shared_row(lins, x)) == 3 and (M == 1 and name == "lit") != bool(seen)
    hook.remove()


@pytest.mark.parametrize("M", [1, 16, 17, 100, 300])
@pytest.mark.parametrize("name", ["lit", "k16", "fp8lit", "fp8k32", "fp8k30"])
def test_rows_off_the_alignment_shared_by_several_matrices(dev, name, M):
    """Rows that start two or ten bytes into another tensor: as each layer gives by itself, and refused in the same words where a
    layer refuses them (past 16 rows most kernels read sixteen bytes at a time)."""
    from gridbook_b200 import _native, formats, synth
    from gridbook_b200.linear import CBLinear, apply_shared_row
    fmt = {"fp8lit": formats.FP8_LITERAL, "fp8k32": formats.FP8_CB_K32, "fp8k30": formats.CBFormat("fp8", 30, n_sub=4)}.get(name) or _fmt(name)
    K, lins = 2048, []
    gen = torch.Generator(device=dev).manual_seed(M)
    for i, N in enumerate((256, 520)):
        lin = CBLinear(fmt, K, [N], [synth.codebook_tables(fmt, i)], prefix=f"off.{i}")
        scale = None if fmt.is_fp4 else (torch.rand(N, generator=gen, device=dev) + 0.5) * 0.02
        lins.append(lin.load(synth.make_packed_device(fmt, N, K, gen, dev), scale, dev))
    wide = torch.randn(M * K + 64, generator=gen, device=dev).to(torch.bfloat16)
    for at in (1, 5):
        x = wide[at:at + M * K].view(M, K)
        try:
            want = [lin(x) for lin in lins]
        except RuntimeError as e:
            assert M > 16
            with pytest.raises(RuntimeError) as again:
                apply_shared_row(lins, x)
            assert str(again.value) == str(e)
            continue
        got = apply_shared_row(lins, x)
        torch.cuda.synchronize()
        assert _native.device_status(0) == 0
        for a, b in zip(got, want):
            assert_close_bf16(f32_of(a), f32_of(b), f"{name} M={M} at {at}", atol_rel=1e-6)


@pytest.mark.parametrize("name,pass_rows", [("lit", 1), ("lit", 5), ("k16", 7), ("lit", 13), ("k16", 18), ("lit", 33), ("lit", 61)])
def test_any_number_of_rows_per_pass(dev, name, pass_rows):
    """The C entries take every row count up to the one that is named for the stack: what 16 or 64 rows a pass give."""
    import ctypes
    from gridbook_b200 import _native as nat, kernels, synth
    fmt = _fmt(name)
    E, N, K, P = 3, 256, 512, 300
    d = synth.make_linear(fmt, E * N, K, seed=pass_rows, global_scale=1.0 / 448.0 if name == "lit" else None)
    if name == "k16":
        from gridbook_b200 import codec
        d = dict(d, fmt=fmt.padded(80), qw=codec.pad_superblocks(torch.from_numpy(d["qw"]), 73, 80).numpy())
    w = synth.to_device_weight(d, dev)
    nw = w.native()
    nw.rows = N
    gen = torch.Generator(device=dev).manual_seed(pass_rows)
    x = torch.randn(P, K, generator=gen, device=dev).to(torch.bfloat16)
    ids = torch.randint(0, E, (P,), generator=gen, device=dev, dtype=torch.int32)
    inv = torch.argsort(torch.argsort(ids, stable=True)).to(torch.int32)
    seg = torch.zeros(E + 1, dtype=torch.int32, device=dev)
    seg[1:] = torch.bincount(ids, minlength=E).cumsum(0)
    lib, ptr, i64, stream = nat.load(), lambda t: ctypes.c_void_p(t.data_ptr()), ctypes.c_int64, ctypes.c_void_p(nat.stream_ptr(dev))

    def product(rows):
        assert lib.gb_moe_fp4_pass_rows(ctypes.byref(nw), 1, i64(P), i64(E)) >= rows
        op = torch.zeros(lib.gb_moe_fp4_operand_bytes(i64(P), i64(E), i64(K), rows), dtype=torch.uint8, device=dev)
        y = torch.empty(P, N, dtype=torch.bfloat16, device=dev)
        nat.check(lib.gb_moe_fp4_rows(ptr(x), ptr(ids), ptr(inv), ptr(seg), i64(P), i64(1), i64(E), i64(K), rows, 0, ptr(op), stream), lib)
        nat.check(lib.gb_moe_gemv_fp4(ptr(op), ctypes.byref(nw), 1, i64(N * nw.row_stride), i64(E), ptr(seg), None, i64(P), rows, ptr(y), stream), lib)
        return y

    got, want = product(pass_rows), product(16 if pass_rows <= 16 else 64)
    torch.cuda.synchronize()
    assert nat.device_status(0) == 0
    assert_close_bf16(f32_of(got), f32_of(want), f"{name} {pass_rows} rows a pass", atol_rel=1e-6)
