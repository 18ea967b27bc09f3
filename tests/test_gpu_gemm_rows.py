"""The prefill GEMM for few rows or narrow layers at the edges of its tiles: one to 256 activation rows a pass, passes that start in the
middle of a 128-row group of scale factors, output features that fill no tile or no 16 bytes, K slices over clusters
of two to eight CTAs (uneven ones among them) and none at all, more tiles than SMs."""
import pytest
import torch

from tests.helpers import assert_close_bf16, f32_of

pytestmark = pytest.mark.gpu
SHAPES = [(1, 128, 256), (17, 40, 512), (16, 200, 1024), (64, 129, 4096), (65, 2056, 2560), (100, 1000, 8192), (128, 20000, 256),
          (129, 300, 8192), (192, 640, 9216), (193, 512, 8192), (256, 250, 16384), (257, 1024, 8192), (333, 384, 9472), (385, 130, 8192),
          (512, 1280, 8448)]


@pytest.fixture(scope="module")
def dev():
    from gridbook_b200 import _native
    _native.prepare(0)
    return torch.device("cuda:0")


def _check(y, ref, tag):
    from gridbook_b200 import _native
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    assert_close_bf16(f32_of(y), f32_of(ref.to(torch.bfloat16)), tag, atol_rel=1e-6)


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_rows_gemm(dev, kind, M, N, K):
    from gridbook_b200 import kernels
    g = torch.Generator(device=dev).manual_seed(M + N)
    dt = torch.bfloat16 if kind == "bf16" else torch.float8_e4m3fn
    a, b = torch.randn(M, K, generator=g, device=dev).to(dt), torch.randn(N, K, generator=g, device=dev).to(dt)
    rows, cols = torch.rand(M, generator=g, device=dev) + 0.5, torch.rand(N, generator=g, device=dev) + 0.5
    y = kernels.gemm_tn(a, b, a_scale=rows, b_scale=cols, global_scale=0.25)
    _check(y, a.double() @ b.double().T * rows[:, None].double() * cols.double() * 0.25, f"{kind} {M}x{N}x{K}")


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_rows_gemm_block_scaled(dev, M, N, K):
    from gridbook_b200 import kernels
    g = torch.Generator(device=dev).manual_seed(M * N)
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
    _check(y, av @ bv.T * rows[:, None].double() * 0.25, f"fp4 {M}x{N}x{K}")


@pytest.mark.parametrize("M,N,K", [(520, 640, 4096), (700, 200, 8192), (1000, 384, 8192), (1024, 130, 2048)])
@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_rows_gemm_in_more_passes(dev, kind, M, N, K):
    """Three to six passes of 192 and 256 rows, which the bf16 and fp8 operands reach."""
    from gridbook_b200 import kernels
    assert kernels.gemm_kernel(M, N, 2 * K if kind == "bf16" else K, False) == "gemm_rows_kernel"
    test_rows_gemm(dev, kind, M, N, K)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_the_shapes_reach_the_rows_kernel(dev, M, N, K):
    from gridbook_b200 import kernels
    assert {kernels.gemm_kernel(M, N, k_bytes, fp4) for k_bytes, fp4 in ((2 * K, False), (K, False), (K // 2, True))} == {"gemm_rows_kernel"}
