"""The prefill GEMMs on CTA pairs at the edges of their tiles: the fewest rows that take them, ragged
rows and columns, rows of the output that are no multiple of 16 bytes, both tile widths (72 pairs of
256 columns make one wave of (2049, 2048); small outputs take 192), more tiles than pairs."""
import pytest
import torch

from tests.helpers import assert_close_bf16, f32_of

pytestmark = pytest.mark.gpu
SHAPES = [(129, 64, 256), (129, 257, 512), (256, 192, 256), (257, 250, 768), (333, 2056, 1024), (1000, 5121, 256),
          (2049, 2048, 512), (2300, 8200, 256)]


@pytest.fixture(scope="module")
def dev():
    from gridbook_b200 import _native
    _native.prepare(0)
    return torch.device("cuda:0")


def _rand(dev, seed):
    return torch.Generator(device=dev).manual_seed(seed)


def _status(dev):
    from gridbook_b200 import _native
    torch.cuda.synchronize()
    return _native.device_status(0)


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_pair_gemm(dev, kind, M, N, K):
    from gridbook_b200 import kernels
    g = _rand(dev, M + N)
    dt = torch.bfloat16 if kind == "bf16" else torch.float8_e4m3fn
    a = torch.randn(M, K, generator=g, device=dev).to(dt)
    b = torch.randn(N, K, generator=g, device=dev).to(dt)
    rows, cols = torch.rand(M, generator=g, device=dev) + 0.5, torch.rand(N, generator=g, device=dev) + 0.5
    y = kernels.gemm_tn(a, b, a_scale=rows, b_scale=cols, global_scale=0.25)
    ref = (a.double() @ b.double().T * rows[:, None].double() * cols.double() * 0.25).to(torch.bfloat16)
    assert _status(dev) == 0
    assert_close_bf16(f32_of(y), f32_of(ref), f"{kind} {M}x{N}x{K}", atol_rel=1e-6)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_pair_gemm_block_scaled(dev, M, N, K):
    from gridbook_b200 import kernels
    g = _rand(dev, M * N)
    e2m1 = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], device=dev, dtype=torch.float64)
    lut = torch.cat([e2m1, -e2m1])

    def operand(R):
        codes = torch.randint(0, 256, (R, K // 2), generator=g, device=dev, dtype=torch.uint8)
        sf = torch.randint(0x30, 0x48, ((R + 127) // 128 * (K // 64) * 512,), generator=g, device=dev, dtype=torch.uint8)
        plane = sf.view(torch.float8_e4m3fn).double().view(-1, K // 64, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(-1, K // 16)
        vals = lut[torch.stack([codes & 15, codes >> 4], -1).reshape(R, K).long()]
        return codes, sf, vals * plane[:R].repeat_interleave(16, 1)

    (a, sfa, av), (b, sfb, bv) = operand(M), operand(N)
    rows = torch.rand(M, generator=g, device=dev) + 0.5
    y = kernels.gemm_fp4(a, sfa, b, sfb, a_scale=rows, global_scale=0.25)
    ref = (av @ bv.T * rows[:, None].double() * 0.25).to(torch.bfloat16)
    assert _status(dev) == 0
    assert_close_bf16(f32_of(y), f32_of(ref), f"fp4 {M}x{N}x{K}", atol_rel=1e-6)
