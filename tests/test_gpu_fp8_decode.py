"""The fp8 formats on the tensor-core decode kernel: one codebook per role, tiles that end inside a role,
row scales for which the two-factor product exists and scales that must keep the fp32 product."""
import numpy as np
import pytest
import torch

from tests.helpers import assert_close_bf16, f32_of, oracle_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n_sub", [(32, 4), (16, 2)])
@pytest.mark.parametrize("M,parts,K", [(1, [128], 1024), (16, [384, 64, 64], 1280), (5, [200, 130], 4096), (9, [1024, 1024], 2560)])
@pytest.mark.parametrize("scales", ["usual", "wide"])
def test_fp8_decode_rows(k, n_sub, M, parts, K, scales):
    from gridbook_b200 import _native, synth
    from gridbook_b200.formats import CBFormat
    from gridbook_b200.linear import CBLinear
    _native.prepare(0)
    dev = torch.device("cuda:0")
    fmt = CBFormat("fp8", k, n_sub=n_sub)
    N = sum(parts)
    d = synth.make_linear(fmt, N, K, seed=N + M, n_books=len(parts))
    d["cb_row_offset"] = np.repeat(np.arange(len(parts)), parts).astype(np.int32) * fmt.codebook_elems()
    rng = np.random.default_rng(M)
    if scales == "wide":        # any significand, far exponents, zero: some rows have no exact pair of factors
        d["weight_scale"] = ((1.0 + rng.random(N)) * np.exp2(rng.integers(-40, 20, N))).astype(np.float32)
        d["weight_scale"][::37] = 0.0
        d["weight_scale"][1::41] = np.float32(1.5e-23)
    n = fmt.codebook_elems()
    books = []
    for i in range(len(parts)):
        out, pos = [], i * n
        for r, c in fmt.table_shapes():
            out.append(torch.from_numpy(d["cb"][pos:pos + r * c].reshape(r, c).copy()))
            pos += r * c
        books.append(out)
    lin = CBLinear(fmt, K, parts, books).load(torch.from_numpy(d["qw"]), torch.from_numpy(d["weight_scale"]), dev)
    x = synth.make_activations(M, K, seed=3)
    got, ref = f32_of(lin(synth.bf16_tensor(x, dev))), oracle_linear(x, d)
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    # row by row magnitudes differ by powers of two: compare every output column on its own scale
    s = np.where(d["weight_scale"] == 0, 1.0, d["weight_scale"])
    assert_close_bf16(got / s, ref / s, f"k={k} M={M} {parts} {scales}", atol_rel=1e-6)


@pytest.mark.parametrize("k,n_sub", [(32, 4), (16, 2)])
@pytest.mark.parametrize("M,N,K", [(1, 128, 8192), (4, 256, 17408), (9, 512, 16384), (33, 130, 5632), (64, 256, 17408), (70, 128, 6400)])
def test_narrow_layers_of_long_rows(k, n_sub, M, N, K):
    """One to four row tiles: K over clusters of nine to sixteen CTAs where the GPU has room for them, more CTAs than groups of eight
    rows to own, a last slice that is short."""
    from gridbook_b200 import _native, kernels, synth
    from gridbook_b200.formats import CBFormat
    _native.prepare(0)
    dev = torch.device("cuda:0")
    fmt = CBFormat("fp8", k, n_sub=n_sub)
    d = synth.make_linear(fmt, N, K, seed=N + M)
    w = synth.to_device_weight(d, dev)
    assert M <= kernels.row_batch_max_rows(w)
    x = synth.make_activations(M, K, seed=3)
    got, ref = f32_of(kernels.gemv(synth.bf16_tensor(x, dev), w, act="fp8")), oracle_linear(x, d)
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    s = np.where(d["weight_scale"] == 0, 1.0, d["weight_scale"])
    assert_close_bf16(got / s, ref / s, f"k={k} M={M} {N}x{K}", atol_rel=1e-6)
