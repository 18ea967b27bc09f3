"""Edges of the row kernels and of the product-format expanders: rows of every register count and the
longer ones, values on and next to the rounding boundaries, codebooks that change inside and between
the row runs of a CTA, one row, ragged row counts."""
import numpy as np
import pytest
import torch

from oracle import cb_oracle as O
from oracle import oracle_kwargs
from tests.helpers import bits_of, nvfp4_quantize_rows_ref, oracle_weight

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from gridbook_b200 import _native
    _native.prepare(0)
    return torch.device("cuda:0")


def _near_boundaries(M, K, seed):
    """Rows whose values sit on, one bf16 step above and one below grid midpoints of their scale."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((M, K)).astype(np.float32) * np.exp2(rng.integers(-12, 12, (M, 1))).astype(np.float32)
    g = x[:, :K // 16 * 16].reshape(M, -1, 16)
    amax = np.abs(g).max(axis=-1)
    mids = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], np.float32) / 6.0
    for j in range(1, 8):
        g[:, ::2, j] = amax[:, ::2] * mids[j - 1] * (1.0 if j % 2 else -1.0)
    b = O.f32_to_bf16_bits(x).astype(np.int64) + rng.integers(-1, 2, (M, K))
    return O.bf16_bits_to_f32(np.clip(b, 0, 65535).astype(np.uint16))


@pytest.mark.parametrize("K", [16, 1040, 4096, 5120, 8192, 17408, 40960, 65536 + 16])
def test_row_buckets_are_bit_exact(dev, K):
    from gridbook_b200 import kernels
    M = 3 if K > 8192 else 33
    x = _near_boundaries(M, K, K)
    x[-1] = 0.0
    x = np.where(np.isfinite(x), x, np.float32(1.0)).astype(np.float32)
    xd = torch.from_numpy(x).to(torch.bfloat16).to(dev)
    for rule in ("recip", "div"):
        assert np.array_equal(bits_of(kernels.fp4_act_qdq(xd, rule)), O.f32_to_bf16_bits(O.fp4_group16_act_qdq(x, rule)))
        want = O.f32_to_bf16_bits(O.fp8_dynamic_act_qdq(x, rule))
        assert np.array_equal(bits_of(kernels.fp8_act_qdq(xd, rule)), want)
        q, s = kernels.fp8_quantize_rows(xd, rule)
        back = (q.float() * s[:, None]).to(torch.bfloat16)
        assert np.array_equal(bits_of(back), want)
    if K % 64 == 0:
        packed, sf, a_scale = kernels.nvfp4_quantize_rows(xd)
        rp, rs, ra = nvfp4_quantize_rows_ref(x)
        assert np.array_equal(packed.cpu().numpy(), rp)
        assert np.array_equal(a_scale.cpu().numpy(), ra)
        assert np.array_equal(sf.cpu().numpy(), O.swizzle_sf_plane(rs))


def _formats():
    from gridbook_b200.formats import CBFormat
    fp4 = [CBFormat("fp4", k, n_sub=2, scale_coding=c) for k, c in ((12, "v2"), (13, "v1"), (16, "v2"), (20, "v2"), (21, "v1"), (24, "v2"))]
    return fp4 + [fp4[2].padded(80)] + [CBFormat("fp8", k, n_sub=4) for k in (28, 30, 33, 48)]


@pytest.mark.parametrize("rows,K,books", [(1, 256, 1), (129, 512, 3), (1000, 1024, 7)])
@pytest.mark.parametrize("idx", range(11))
def test_product_expanders_are_bit_exact(dev, idx, rows, K, books):
    from gridbook_b200 import kernels, synth
    fmt = _formats()[idx]
    if books == 7 and fmt.k > 24 and not fmt.is_fp4 and fmt.k == 48:
        books = 2
    base = fmt if fmt.sb_pad == 0 else fmt.padded(fmt.packed_type_size)
    d = synth.make_linear(base, rows, K, seed=rows + idx, n_books=books, super_span=None)
    up = d
    if fmt.sb_pad:
        from gridbook_b200 import codec
        up = dict(d, fmt=fmt, qw=codec.pad_superblocks(torch.from_numpy(d["qw"]), base.type_size, fmt.type_size).numpy())
    w = synth.to_device_weight(up, dev)
    ref = O.f32_to_bf16_bits(oracle_weight(d))
    lo, n = rows // 3, max(1, rows // 2)
    off = d["cb_row_offset"] if d["cb_row_offset"] is not None else np.zeros(rows, np.int32)
    if fmt.is_fp4:
        assert np.array_equal(bits_of(kernels.expand_fp4_bf16(w)), ref)
        assert np.array_equal(bits_of(kernels.expand_fp4_bf16(w, lo, n)), ref[lo:lo + n])
        rp, rs = O.decode_nvfp4_tile(d["qw"], d["cb"], off, N=rows, K=K, compose=d["compose"],
                                     **{k: v for k, v in oracle_kwargs(base).items() if k != "grid"})
        packed, sf = kernels.expand_fp4_nvfp4(w, swizzled=True)
        assert np.array_equal(packed.cpu().numpy(), rp)
        assert np.array_equal(sf.cpu().numpy(), O.swizzle_sf_plane(rs))
    else:
        vals = O.decode_values(d["qw"], d["cb"], off, N=rows, K=K, k_bits=base.k, n_sub=base.n_sub, type_size=base.type_size)
        assert np.array_equal(kernels.expand_fp8(w).view(torch.uint8).cpu().numpy(), O.f32_to_e4m3(vals))
        assert np.array_equal(bits_of(kernels.expand_fp8_bf16(w)), ref)
        assert np.array_equal(bits_of(kernels.expand_fp8_bf16(w, lo, n)), ref[lo:lo + n])


@pytest.mark.parametrize("T,topk,H", [(1, 1, 2), (3, 8, 2048), (700, 5, 2048), (2500, 8, 258)])
def test_combine_both_widths(dev, T, topk, H):
    from gridbook_b200 import kernels
    gen = torch.Generator(device=dev).manual_seed(T)
    y = torch.randn(T * topk, H, generator=gen, device=dev).to(torch.bfloat16)
    w = torch.rand(T * topk, generator=gen, device=dev)
    ids = torch.randint(-1, 9, (T, topk), generator=gen, device=dev, dtype=torch.int32)
    got = kernels.moe_combine(y, w, T, topk, topk_ids=ids, E=8, round_weights=True).float()
    live = ((ids >= 0) & (ids < 8)).reshape(-1)
    yw = torch.where(live[:, None], y.float() * w.to(torch.bfloat16).float()[:, None], torch.zeros((), device=dev))
    want = yw.reshape(T, topk, H).double().sum(1)
    assert torch.all((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-6)


@pytest.mark.parametrize("rows,K,books", [(1, 256, 1), (129, 512, 3), (1000, 1024, 7), (700, 5120, 1)])
@pytest.mark.parametrize("k", [8, 12, 16, 20, 24])
def test_nvfp4_view_of_resident_slots_is_exact(dev, k, rows, K, books):
    """The expander of aligned superblocks: one superblock a row, fewer superblocks than a step of the
    CTA, rows that end inside a step, a codebook per part."""
    from gridbook_b200 import codec, kernels, synth
    from gridbook_b200.formats import NVFP4_LITERAL, CBFormat
    fmt = NVFP4_LITERAL if k == 8 else CBFormat("fp4", k, n_sub=2, scale_coding="v2")
    d = synth.make_linear(fmt, rows, K, seed=rows + k, n_books=books, super_span=None)
    up, slot = d, codec.resident_slot(fmt)
    if slot is not None:
        up = dict(d, fmt=fmt.padded(slot), qw=codec.pad_superblocks(torch.from_numpy(d["qw"]), fmt.type_size, slot).numpy())
    off = d["cb_row_offset"] if d["cb_row_offset"] is not None else np.zeros(rows, np.int32)
    rp, rs = O.decode_nvfp4_tile(d["qw"], d["cb"], off, N=rows, K=K, compose=d["compose"],
                                 **{a: v for a, v in oracle_kwargs(fmt).items() if a != "grid"})
    packed, sf = kernels.expand_fp4_nvfp4(synth.to_device_weight(up, dev), swizzled=True)
    assert np.array_equal(packed.cpu().numpy(), rp)
    assert np.array_equal(sf.cpu().numpy(), O.swizzle_sf_plane(rs))


@pytest.mark.parametrize("name", ["lit", "k16", "k12", "fp8k32", "fp8k30"])
def test_rows_that_start_in_the_middle_of_another_tensor(dev, name):
    """Contiguous activations whose first element is not at a multiple of sixteen bytes: decode batches and
    routed layers give what they give for a copy of them."""
    from gridbook_b200 import _native, formats as F, kernels, synth
    from gridbook_b200.linear import CBLinear
    from gridbook_b200.moe import CBMoE
    fmt = {"lit": F.NVFP4_LITERAL, "k16": F.NVFP4_CB_K16, "k12": F.CBFormat("fp4", 12, n_sub=2, scale_coding="v2"),
           "fp8k32": F.FP8_CB_K32, "fp8k30": F.CBFormat("fp8", 30, n_sub=4)}[name]
    N, K, E, inter = 256, 1024, 8, 256
    gen = torch.Generator(device=dev).manual_seed(5)
    scale = (lambda *s: None) if fmt.is_fp4 else (lambda *s: torch.rand(s, generator=gen, device=dev) + 0.5)
    lin = CBLinear(fmt, K, [N], [synth.codebook_tables(fmt, 1)]).load(synth.make_packed_device(fmt, N, K, gen, dev), scale(N), dev)
    moe = CBMoE(fmt, fmt, E, K, inter, synth.codebook_tables(fmt, 1), synth.codebook_tables(fmt, 2))
    moe.load(synth.make_packed_device(fmt, E * 2 * inter, K, gen, dev).view(E, 2 * inter, -1),
             synth.make_packed_device(fmt, E * K, inter, gen, dev).view(E, K, -1), scale(E, 2 * inter), scale(E, K), dev)
    for rows, first in ((1, 1), (1, 2), (3, 1), (16, 5)):
        flat = torch.randn(rows * K + 16, generator=gen, device=dev).to(torch.bfloat16)
        x = flat[first:first + rows * K].view(rows, K)
        assert x.is_contiguous() and x.data_ptr() % 16
        assert torch.equal(kernels.fp4_act_qdq(x), kernels.fp4_act_qdq(x.clone()))
        assert torch.equal(kernels.fp8_act_qdq(x), kernels.fp8_act_qdq(x.clone()))
        a, b = lin(x).float(), lin(x.clone()).float()        # another kernel may serve the odd start: sums in another order
        assert float((a - b).norm() / b.norm()) <= 1e-3
        ids = torch.randint(0, E, (rows, 2), generator=gen, device=dev, dtype=torch.int32)
        tw = torch.full((rows, 2), 0.5, device=dev)
        assert torch.equal(moe(x, tw, ids), moe(x.clone(), tw, ids))
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("rows,K,books", [(1, 256, 1), (37, 768, 2), (4099, 512, 3), (1000, 2304, 7)])
@pytest.mark.parametrize("k,n_sub", [(16, 2), (32, 4)])
def test_fp8_expander_rebuilds_its_tables_where_rows_change_codebook(dev, k, n_sub, rows, K, books, shift):
    """Runs of rows that end inside a CTA's share, a window of rows, codebook blocks at any byte."""
    from gridbook_b200 import kernels, synth
    from gridbook_b200.formats import CBFormat
    fmt = CBFormat("fp8", k, n_sub=n_sub)
    d = synth.make_linear(fmt, rows, K, seed=rows + k, n_books=books)
    off = d["cb_row_offset"] if d["cb_row_offset"] is not None else np.zeros(rows, np.int32)
    up = dict(d, cb=np.concatenate([np.zeros(shift, np.float32), d["cb"]]), cb_row_offset=off + np.int32(shift)) if shift or books > 1 else d
    w = synth.to_device_weight(up, dev)
    want = O.f32_to_e4m3(O.decode_values(d["qw"], d["cb"], off, N=rows, K=K, k_bits=k, n_sub=n_sub, type_size=fmt.type_size))
    assert np.array_equal(kernels.expand_fp8(w).view(torch.uint8).cpu().numpy(), want)
    lo, n = rows // 3, max(1, rows // 2)
    assert np.array_equal(kernels.expand_fp8(w, lo, n).view(torch.uint8).cpu().numpy(), want[lo:lo + n])


@pytest.mark.parametrize("M", [20, 140, 333, 1500])
def test_prefill_linears_launched_back_to_back(dev, M):
    """The expander of a linear runs beside the quantiser of its rows and overwrites what the linear before has read: a
    chain without a pause gives the outputs of the same calls one at a time, in every format's expander."""
    from gridbook_b200 import formats, synth
    from gridbook_b200.linear import CBLinear
    fmts = [formats.NVFP4_LITERAL, formats.FP8_LITERAL, formats.CBFormat("fp4", 20, n_sub=2, scale_coding="v2"), formats.FP8_CB_K32,
            formats.CBFormat("fp8", 30, n_sub=4), formats.CBFormat("fp4", 12, n_sub=2, scale_coding="v2"), formats.CBFormat("fp4", 13, n_sub=2, scale_coding="v2")]
    gen = torch.Generator(device=dev).manual_seed(M)
    lins, K = [], 1024
    for i, fmt in enumerate(fmts * 2):
        parts = [640, 384] if i % 2 else [1024]
        lin = CBLinear(fmt, K, parts, [synth.codebook_tables(fmt, i + j) for j in range(len(parts))], prefix=f"chain.{i}")
        lin.method.midm_max_rows = 16
        scale = None if fmt.is_fp4 else (torch.rand(sum(parts), generator=gen, device=dev) + 0.5) * 0.02
        lins.append(lin.load(synth.make_packed_device(fmt, sum(parts), K, gen, dev), scale, dev))
    x = torch.randn(M, K, generator=gen, device=dev).to(torch.bfloat16)

    def chain(pause):
        out = []
        for lin in lins:
            out.append(lin(x))
            if pause:
                torch.cuda.synchronize()
        return out

    one_at_a_time = chain(True)
    for _ in range(5):
        for a, b in zip(chain(False), one_at_a_time):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("name", ["fp8k32", "lit"])
def test_shared_prefill_holds_one_decoded_copy_at_a_time(dev, name):
    """Three linears that read the same rows need no more memory at their peak together than one after the other."""
    from gridbook_b200 import formats as F, synth
    from gridbook_b200.linear import CBLinear, apply_shared_row
    fmt, M, K = {"lit": F.NVFP4_LITERAL, "fp8k32": F.FP8_CB_K32}[name], 300, 2048
    gen = torch.Generator(device=dev).manual_seed(1)
    lins = []
    for i, N in enumerate((2048, 3072, 4096)):               # the largest last: all outputs are there at either peak
        lin = CBLinear(fmt, K, [N], [synth.codebook_tables(fmt, i)], prefix=f"mem.{i}")
        scale = None if fmt.is_fp4 else torch.rand(N, generator=gen, device=dev) + 0.5
        lins.append(lin.load(synth.make_packed_device(fmt, N, K, gen, dev), scale, dev))
    x = torch.randn(M, K, generator=gen, device=dev).to(torch.bfloat16)

    def peak(call):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        out = call()
        torch.cuda.synchronize()
        return torch.cuda.max_memory_allocated() - before, out

    (apart, want), (shared, got) = peak(lambda: [lin(x) for lin in lins]), peak(lambda: apply_shared_row(lins, x))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert shared <= apart + (64 << 10), (shared, apart)
