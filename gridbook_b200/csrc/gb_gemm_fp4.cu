// Prefill GEMM on the block-scaled FP4 tensor cores: D[M,N] = a_scale[m] * global * sum_k
// (A[m,k] * SFA[m,k/16]) * (B[n,k] * SFB[n,k/16]) with A and B packed E2M1 (two per byte, K-major)
// and UE4M3 scale factors per sixteen elements: tcgen05.mma kind::mxf4nvf4, block16, fp32
// accumulator in tensor memory.  B is the native NVFP4 view of a codebook layer written by the
// expander (gb_expand_fp4_nvfp4: 0.56 bytes per weight instead of the 2-byte bf16 tile), A the
// activations through gb_nvfp4_quantize_rows below.  Replaces the reference's block-scaled
// prefill (gridbook/csrc/cb_fused_fp4_gemm.cu:291-450,758-903) with the operands decoded once.
//
// Scale factors travel in the 128 x 4 atom layout (gridbook/codec.py:353-374): 512 bytes hold the
// scale bytes of 128 rows x 4 groups, row r and group g at (r % 32) * 16 + (r / 32) * 4 + g; the
// atoms of one 128-row tile follow each other along K.  One atom is exactly what one MMA
// (K = 64) needs for 128 rows: four columns of tensor memory, row r's four bytes at lane r % 32
// of every lane quarter, column r / 32.
//
// The kernels: gb_gemm_pair.cu, gb_gemm_rows.cu.  Here are the entry and the activations' quantiser.
#include "gb_common.cuh"

namespace {

// ---- NVFP4 quantisation of activation rows ---------------------------------------------
// The arithmetic of gridbook/codec.py:377-425 with a scale of its own per row, as the
// reference's row quantiser chooses it (gridbook/csrc/cb_fused_fp4_gemm.cu:345-355):
//   gs = (range * 6) / rowmax,  a_scale = 1 / gs,  xs = x * gs,
//   SF = E4M3(min(max|xs| / 6, 448)) per group of sixteen, one rounding,
//   code = E2M1 nearest of clamp(xs / SF, +-6), a tie going to the even code index,
//   sign bit = sign of xs (kept on zeros); a zero SF zeroes its group.
// Every operation is a correctly rounded fp32 one (no approximate reciprocal), so the bytes are
// those of the torch formulation.
// One CTA per row, one to four groups per thread kept in registers: the row is read once
// (2048 x 17408: 38.6 us when it was read twice and every value divided twice).
constexpr int kQuantMaxGroups = 4;

template <int kG>
__global__ void __launch_bounds__(1024)
nvfp4_quantize_rows_kernel(const uint4* __restrict__ x, uint2* __restrict__ packed, uint8_t* __restrict__ sfa,
                           float* __restrict__ a_scale, int64_t M, int groups, float range) {
  gb_pdl_wait();
  gb_pdl_launch_dependents();                            // behind the wait: the weights' expander runs beside this launch
  const int64_t row = blockIdx.x;
  const int64_t k_atoms = (groups + 3) / 4;
  auto sf_offset = [&](int g) {
    return (row % 32) * 16 + ((row / 32) % 4) * 4 + (g % 4) + (int64_t)(g / 4) * 512 + (row / 128) * (512 * k_atoms);
  };
  if (row >= M) {                                        // padding rows of the last 128-row tile: zero scales
    for (int g = threadIdx.x; g < groups; g += blockDim.x) sfa[sf_offset(g)] = 0;
    return;
  }
  const uint4* xr = x + row * 2 * groups;
  __shared__ float red[32];
  uint32_t w[kG][8], gtop[kG];                             // packed magnitude maxima of the groups
  float amax = 0.0f;
  for (int g0 = threadIdx.x; g0 < groups; g0 += kG * blockDim.x) {    // once, unless the row is longer than the registers
#pragma unroll
    for (int j = 0; j < kG; ++j) {
      const int g = g0 + j * blockDim.x;
      const bool in = g < groups;
      gtop[j] = 0u;
      const uint4 a = in ? xr[2 * g] : make_uint4(0u, 0u, 0u, 0u), b = in ? xr[2 * g + 1] : make_uint4(0u, 0u, 0u, 0u);
      w[j][0] = a.x; w[j][1] = a.y; w[j][2] = a.z; w[j][3] = a.w;
      w[j][4] = b.x; w[j][5] = b.y; w[j][6] = b.z; w[j][7] = b.w;
#pragma unroll
      for (int i = 0; i < 8; ++i) gtop[j] = gb_max_bf16x2(gtop[j], w[j][i] & 0x7FFF7FFFu);
      amax = fmaxf(amax, gb_max_of_bf16x2(gtop[j]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = (int)(threadIdx.x & 31) < (int)(blockDim.x >> 5) ? red[threadIdx.x & 31] : 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const bool live = amax > 0.0f && isfinite(amax);
  const float gs = live ? __fdiv_rn(__fmul_rn(range, 6.0f), amax) : 1.0f;
  if (threadIdx.x == 0) a_scale[row] = live ? __fdiv_rn(1.0f, gs) : 0.0f;
  const bool reload = groups > kG * (int)blockDim.x;
  for (int base = 0; base < groups; base += kG * blockDim.x) {        // whole warps stay together: the shuffles below
#pragma unroll
    for (int j = 0; j < kG; ++j) {
      const int g = base + threadIdx.x + j * blockDim.x;
      const unsigned here = __ballot_sync(0xffffffffu, g < groups);
      if (g >= groups) continue;
      if (reload) {
        const uint4 a = xr[2 * g], b = xr[2 * g + 1];
        w[j][0] = a.x; w[j][1] = a.y; w[j][2] = a.z; w[j][3] = a.w;
        w[j][4] = b.x; w[j][5] = b.y; w[j][6] = b.z; w[j][7] = b.w;
        gtop[j] = 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i) gtop[j] = gb_max_bf16x2(gtop[j], w[j][i] & 0x7FFF7FFFu);
      }
      float xs[16];
      const float gmax = __fmul_rn(gb_max_of_bf16x2(gtop[j]), gs);      // rounding keeps the order: the largest |xs|
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        xs[2 * i] = __fmul_rn(gb_bf16_bits_to_f32(w[j][i] & 0xffffu), gs);
        xs[2 * i + 1] = __fmul_rn(gb_bf16_bits_to_f32(w[j][i] >> 16), gs);
      }
      const float sf = live ? fminf(__fdiv_rn(gmax, 6.0f), 448.0f) : 0.0f;
      const uint32_t sf_byte = gb_f32_to_e4m3(sf);
      const float sf_f = gb_e4m3_to_f32(sf_byte);
      // four neighbouring groups share a word of the scale-factor plane
      const uint32_t b1 = __shfl_down_sync(here, sf_byte, 1), b2 = __shfl_down_sync(here, sf_byte, 2);
      const uint32_t b3 = __shfl_down_sync(here, sf_byte, 3);
      if (groups % 4 != 0) sfa[sf_offset(g)] = (uint8_t)sf_byte;
      else if ((g & 3) == 0) *reinterpret_cast<uint32_t*>(sfa + sf_offset(g)) = sf_byte | (b1 << 8) | (b2 << 16) | (b3 << 24);
      const float rinv = sf_f != 0.0f ? __frcp_rn(sf_f) : 0.0f;
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t byte;
        if (sf_f != 0.0f) byte = gb_cvt_e2m1x2(gb_div(xs[2 * i], sf_f, rinv), gb_div(xs[2 * i + 1], sf_f, rinv));
        else byte = ((__float_as_uint(xs[2 * i]) >> 31) << 3) | ((__float_as_uint(xs[2 * i + 1]) >> 31) << 7);
        if (i < 4) lo |= byte << (8 * i);
        else hi |= byte << (8 * (i - 4));
      }
      packed[row * groups + g] = make_uint2(lo, hi);
    }
  }
}

}  // namespace

extern "C" {

int64_t gb_nvfp4_sf_bytes(int64_t rows, int64_t K) {
  if (rows <= 0 || K <= 0) return 0;
  return ((rows + 127) / 128) * ((K / 16 + 3) / 4) * 512;
}

int gb_nvfp4_quantize_rows(const void* x, int64_t M, int64_t K, float range, void* packed, void* sf, float* a_scale,
                           void* stream) {
  GB_REQUIRE(x && packed && sf && a_scale, "null pointer argument");
  GB_REQUIRE(M >= 0 && K > 0 && K % 16 == 0, "bad shape M=%lld K=%lld (K a multiple of 16)", (long long)M, (long long)K);
  GB_REQUIRE(((uintptr_t)x & 15u) == 0 && ((uintptr_t)packed & 7u) == 0, "rows must be 16-byte aligned");
  GB_REQUIRE(range > 0.0f && range <= 448.0f, "range multiplier %g outside (0, 448]", (double)range);
  if (M == 0) return GB_OK;
  GB_REQUIRE(K / 16 < (1ll << 31), "dimension too large");
  const int64_t padded = (M + 127) / 128 * 128, groups = K / 16;
  int per = groups <= 512 ? 1 : groups <= 1024 ? 2 : kQuantMaxGroups;
  if (per == 1 && M >= 8 * gb_sm_count()) per = 2;         // several waves of rows: smaller CTAs, more rows in flight
  int64_t threads = ((groups + per - 1) / per + 31) / 32 * 32;
  if (threads > 1024) threads = 1024;
#define GB_NVFP4_ROWS(G)                                                                                          \
  GB_CUDA_OK(gb_launch(nvfp4_quantize_rows_kernel<G>, dim3((unsigned)padded), dim3((unsigned)threads), 0, (cudaStream_t)stream, \
                       (const uint4*)x, (uint2*)packed, (uint8_t*)sf, a_scale, M, (int)groups, range))
  switch (per) {
    case 1: GB_NVFP4_ROWS(1); break;
    case 2: GB_NVFP4_ROWS(2); break;
    default: GB_NVFP4_ROWS(kQuantMaxGroups); break;
  }
#undef GB_NVFP4_ROWS
  return GB_OK;
}

int gb_gemm_fp4(const void* A, const void* sfa, const void* B, const void* sfb, void* D, int64_t M, int64_t N, int64_t K,
                const float* a_scale, float global_scale, void* stream) {
  GB_REQUIRE(A && sfa && B && sfb && D, "null pointer argument");
  GB_REQUIRE(M >= 0 && N > 0 && K > 0 && K % 256 == 0, "K=%lld must be a multiple of 256", (long long)K);
  GB_REQUIRE(((uintptr_t)A & 15u) == 0 && ((uintptr_t)B & 15u) == 0 && ((uintptr_t)D & 15u) == 0 &&
             ((uintptr_t)sfa & 15u) == 0 && ((uintptr_t)sfb & 15u) == 0, "operands must be 16-byte aligned");
  GB_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "dimension too large");
  if (M == 0) return GB_OK;
  const int sms = gb_sm_count();
  if (sms <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  const float gs = global_scale == 0.0f ? 1.0f : global_scale;
  if (!gb_gemm_rows_applies(true, M, N, K / 256)) {
    const int rc = gb_gemm_fp4_pair(A, sfa, B, sfb, D, M, N, K, a_scale, gs, (cudaStream_t)stream);
    if (rc != GB_EUNSUPPORTED) return rc;
  }
  return gb_gemm_fp4_rows(A, sfa, B, sfb, D, M, N, K, a_scale, gs, (cudaStream_t)stream);
}

}  // extern "C"
