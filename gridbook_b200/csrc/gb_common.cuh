// Shared host/device helpers for the gridbook_b200 kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>

#include <mutex>

#include "../../include/gridbook_b200.h"

#define GB_DEVINL __device__ __forceinline__

// ---------------------------------------------------------------------------
// host-side error plumbing
// ---------------------------------------------------------------------------
void gb_set_error(const char* fmt, ...);
int gb_fail(int code, const char* fmt, ...);
int gb_sm_count();                 // SMs of the current device (cached)
int* gb_status_word();             // device int the kernels raise on a timed-out wait

bool gb_pdl_enabled();             // false when GRIDBOOK_B200_PDL=0 (plain stream order)
void gb_count_launch();            // every kernel launch of this library bumps gb_launch_count()

// Clusters of a kernel's CTAs (along y, up to sixteen) that run at once on the current device, by their size; asked once.
struct GbClusters {
  std::mutex mutex;
  int n[64][17];                   // 0: not asked yet
  int ask(const void* kernel, int threads, size_t smem, int size);
};

// Kernel launch with the programmatic-stream-serialization attribute (see gb_pdl_wait).
template <typename... KArgs, typename... Args>
inline cudaError_t gb_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = gb_pdl_enabled() ? 1 : 0;
  gb_count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

#define GB_REQUIRE(cond, ...)                           \
  do {                                                  \
    if (!(cond)) return gb_fail(GB_EINVAL, __VA_ARGS__); \
  } while (0)

#define GB_CUDA_OK(expr)                                                       \
  do {                                                                         \
    cudaError_t e_ = (expr);                                                   \
    if (e_ != cudaSuccess)                                                     \
      return gb_fail(GB_ECUDA, "%s: %s", #expr, cudaGetErrorString(e_));       \
  } while (0)

#define GB_LAUNCH_OK(name)                                                     \
  do {                                                                         \
    cudaError_t e_ = cudaGetLastError();                                       \
    if (e_ != cudaSuccess)                                                     \
      return gb_fail(GB_ECUDA, "launch of %s: %s", name, cudaGetErrorString(e_)); \
  } while (0)

int gb_check_format(const gb_format& f, int64_t K);
int gb_check_weight(const gb_weight* w);
int gb_prepare_kernels();          // per-device function attributes of the big kernels
int gb_prepare_gemm();
int gb_prepare_dot();
int gb_prepare_umma();
int gb_prepare_tab();
int gb_prepare_gemm_pair();
int gb_prepare_gemm_rows();
int gb_prepare_gemv_fp4();
// Longest a device-side wait may spin before it gives up and raises the status word
// (two seconds unless gb_set_wait_limit_ms changed it).
unsigned long long gb_wait_limit_ns();
// Swizzled (128-byte) operand map over a row-major [rows, K] matrix of 2- or 1-byte elements:
// box = 128 bytes of K x box_rows rows, rows past the end read zero.
int gb_tensor_map_operand(void* map_out, const void* base, int64_t rows, int64_t K, int elem_bytes, int box_rows);
// Row-major bf16 output [M, N] in boxes of 32 x 32 with the 64-byte swizzle (N a multiple of 8).
int gb_tensor_map_out(void* map_out, void* base, int64_t M, int64_t N);
// Activation operand of the grouped GEMM (gb_moe_gemm_fp4): tiles of 64 rows, [tile][64 code rows of q, 64 of the
// correction][K / 2 bytes], then the scale-factor atoms of 192 columns a tile, then the rows' powers of two, then
// the scales of the groups left out as [tile][64][K / 16] (gb_left_out).
// Column 96 (m / 32) + 32 t + m % 32 of a tile is term t of row m.
struct GbFp4Tiles { int64_t tiles, sf_groups, sf_at, scale_at, tail_at, bytes; };
inline GbFp4Tiles gb_fp4_tiles(int64_t P, int64_t E, int64_t K) {
  GbFp4Tiles t;
  auto up = [](int64_t v) { return (v + 255) & ~(int64_t)255; };
  t.tiles = P / 64 + E + 1;
  t.sf_groups = (t.tiles * 192 + 127) / 128;
  t.sf_at = up(t.tiles * 128 * (K / 2));
  t.scale_at = t.sf_at + up(t.sf_groups * (K / 64) * 512);
  t.tail_at = t.scale_at + up(t.tiles * 64 * 4);
  t.bytes = t.tail_at + up(t.tiles * 64 * (K / 16) * 4);
  return t;
}
// The prefill GEMM for few rows or narrow layers (gb_gemm_rows.cu), where gb_gemm_rows_applies says so.
bool gb_gemm_rows_applies(bool fp4, int64_t M, int64_t N, int64_t k_tiles);
int gb_gemm_rows(const void* X, const void* W, void* D, int64_t M, int64_t N, int64_t K, int kind, const float* a_scale,
                 const float* b_scale, float global_scale, cudaStream_t stream);
int gb_gemm_fp4_rows(const void* X, const void* sfx, const void* W, const void* sfw, void* D, int64_t M, int64_t N, int64_t K,
                     const float* a_scale, float global_scale, cudaStream_t stream);
// The prefill GEMMs on CTA pairs (gb_gemm_pair.cu), for the others.
int gb_gemm_pair(const void* A, const void* B, void* D, int64_t M, int64_t N, int64_t K, int kind, const float* a_scale,
                 const float* b_scale, float global_scale, cudaStream_t stream);
int gb_gemm_fp4_pair(const void* A, const void* sfa, const void* B, const void* sfb, void* D, int64_t M, int64_t N, int64_t K,
                     const float* a_scale, float global_scale, cudaStream_t stream);
// 1..128 activation rows of the literal format, the two-tier k = 16 format with 80-byte superblocks
// or the fp8 k = 32 format: decode into tensor memory, tcgen05 MMA with the weights on the M side
// (gb_gemv_umma.cu); GB_EUNSUPPORTED when the format, layout or row count is not its own.
int gb_gemv_umma(const void* x, int64_t M, const gb_weight* w, int n_roles, const int64_t* role_rows, int act, int scale_rule,
                 void* y, void* workspace, int64_t workspace_bytes, void* stream);
int64_t gb_gemv_umma_workspace_bytes(int64_t M, int64_t N, int64_t K);
int gb_gemv_umma_max_rows(const gb_weight* w);
bool gb_gemv_umma_is_literal(const gb_weight* w);
int gb_tensor_map_bytes_2d(void* map_out, const void* base, uint64_t inner_bytes, uint64_t rows,
                           uint64_t pitch_bytes, uint32_t box_bytes, uint32_t box_rows);
// Decode batches of the fp4 grid on the block-scaled FP4 tensor cores (gb_gemv_fp4.cu): the literal format
// and, where the caller knows that every two-tier scale is an exact E4M3 value, the product formats
// k = 12, 16, 20, 24 in 16-byte aligned superblock slots.  `role_rows`: row counts of the parts of a
// fused matrix that carry their own codebook (n_roles <= 1: one codebook).
bool gb_gemv_fp4_applies(const gb_weight* w, bool scales_e4m3);
int64_t gb_gemv_fp4_workspace_bytes(int64_t M, int64_t K);
int gb_gemv_fp4(const void* x, int64_t M, const gb_weight* w, bool scales_e4m3, int n_roles, const int64_t* role_rows,
                int scale_rule, void* y, void* workspace, int64_t workspace_bytes, void* stream);
// M = 1 literal-format linear by per-column inner-product tables (gb_gemv_dot.cu); GB_EUNSUPPORTED when
// the shape or layout is not its own, and the caller falls back to the MMA kernel.
int gb_gemv_dot_rows(const void* x, int64_t M, const gb_weight* w, int act, int scale_rule, void* y, void* workspace,
                     int64_t workspace_bytes, void* stream);
int64_t gb_gemv_dot_rows_workspace_bytes(int64_t M, int64_t N, int64_t K);
int gb_gemv_dot(const void* x, const gb_weight* w, int act, int scale_rule, void* y, void* workspace,
                int64_t workspace_bytes, void* stream);
int64_t gb_gemv_dot_workspace_bytes(int64_t N, int64_t K);

// ---------------------------------------------------------------------------
// scalar formats
// ---------------------------------------------------------------------------
GB_DEVINL float gb_bf16_bits_to_f32(uint32_t b) { return __uint_as_float(b << 16); }

GB_DEVINL uint32_t gb_f32_to_bf16_bits(float v) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// Two fp32 -> one word of two bf16 (a in the low half), round to nearest even: one conversion.
GB_DEVINL uint32_t gb_pack_bf16x2(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// E4M3 byte -> fp32, exact (no NaN handling: 0x7F/0xFF decode as 480, never stored).
GB_DEVINL float gb_e4m3_to_f32(uint32_t b) {
  const uint32_t mag = b & 0x7Fu;
  // place exponent+mantissa at the fp32 exponent, then rebias by 2^120; the
  // multiply also renormalises the subnormal codes (exponent field 0).
  float f = __uint_as_float(mag << 20) * 0x1p120f;
  return (b & 0x80u) ? -f : f;
}

// fp32 -> E4M3 with ONE rounding to nearest even (the hardware cvt may round
// twice through fp16).  |f| must be < 480; callers clamp to 448 first.
GB_DEVINL uint32_t gb_f32_to_e4m3(float f) {
  uint32_t u = __float_as_uint(f);
  const uint32_t sign = (u >> 24) & 0x80u;
  u &= 0x7FFFFFFFu;
  uint32_t r;
  if (u < (121u << 23)) {
    // below 2^-6 the result is subnormal with quantum 2^-9: adding 2^14 makes
    // the fp32 adder do the nearest-even rounding at exactly that quantum.
    const float shifted = __uint_as_float(u) + 16384.0f;
    r = __float_as_uint(shifted) - __float_as_uint(16384.0f);
  } else {
    const uint32_t odd = (u >> 20) & 1u;
    u += 0x7FFFFu + odd;            // round at bit 20
    r = (u >> 20) - (120u << 3);    // rebias exponent 127 -> 7
  }
  return (r & 0x7Fu) | sign;
}

// Round-to-nearest on the signed E2M1 grid {0, +-.5, +-1, +-1.5, +-2, +-3, +-4, +-6} with the
// reference's tie rule (gridbook/codec.py:248-260): the upper neighbour wins only when it is
// STRICTLY closer, so an exact midpoint goes to the lower (more negative) rung.
GB_DEVINL float gb_e2m1_rtn(float v) {
  constexpr float grid[15] = {-6.0f, -4.0f, -3.0f, -2.0f, -1.5f, -1.0f, -0.5f, 0.0f,
                              0.5f,  1.0f,  1.5f,  2.0f,  3.0f,  4.0f,  6.0f};
  // hi = first rung >= v (bucketize, right = false; the top rung when there is none),
  // lo = the rung before it (the bottom rung when hi is the bottom).  Selects only: a
  // dynamically indexed table would live in local memory.
  float hi = grid[14], lo = grid[0];
#pragma unroll
  for (int i = 14; i >= 0; --i)
    if (grid[i] >= v) hi = grid[i];
#pragma unroll
  for (int i = 0; i < 15; ++i)
    if (!(grid[i] >= v)) lo = grid[i];
  return fabsf(__fsub_rn(hi, v)) < fabsf(__fsub_rn(v, lo)) ? hi : lo;
}

// v / d, correctly rounded, given rinv = RN(1 / d): a product and one correction step with an exact
// remainder (Markstein's theorem; it excludes a divisor whose significand is all ones and needs a
// finite quotient, see gb_plain_division).  Three instructions where __fdiv_rn takes about ten.
GB_DEVINL float gb_div(float v, float d, float rinv) {
  const float q = v * rinv;
  return fmaf(fmaf(-q, d, v), rinv, q);
}

// Divisors gb_div does not take.
GB_DEVINL bool gb_plain_division(float d) {
  return (__float_as_uint(d) & 0x7FFFFFu) == 0x7FFFFFu || !(d < __int_as_float(0x7F800000));
}

// Two fp32 -> one byte of two E2M1 codes (a in the low nibble), nearest, |value| clamped to 6.
GB_DEVINL uint32_t gb_cvt_e2m1x2(float a, float b) {
  uint32_t r;
  asm("{ .reg .b8 t;\n  cvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n  cvt.u32.u8 %0, t; }" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

// Two fp32 -> two E4M3 bytes (a in the low byte), nearest, |value| clamped to 448.
GB_DEVINL uint32_t gb_cvt_e4m3x2(float a, float b) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(b), "f"(a));
  return r;
}

// E2M1 codes of v0 / scale and v1 / scale under the reference's tie rule (finite arguments, a divisor
// gb_div takes).  The conversion rounds a tie to the even code; the rule wants the lower value.  Every
// midpoint has its low 21 significand bits clear, so a quotient with those bits clear moves down by
// an ulp first: grid values among them convert as before.  A zero may carry either sign.
// (Midpoints are no rare accident: bf16 values reach them in half a percent of cases, so nearly
// every warp holds one and a slow path for them cost 160 us of the routed SwiGLU launch.)
GB_DEVINL uint32_t gb_e2m1_div2(float v0, float v1, float scale, float rinv) {
  float x0 = gb_div(v0, scale, rinv), x1 = gb_div(v1, scale, rinv);
  if ((__float_as_uint(x0) & 0x1FFFFFu) == 0) x0 = fmaf(fabsf(x0), -0x1p-22f, x0);
  if ((__float_as_uint(x1) & 0x1FFFFFu) == 0) x1 = fmaf(fabsf(x1), -0x1p-22f, x1);
  return gb_cvt_e2m1x2(x0, x1);
}

// E4M3 bytes of clamp(v / scale, +-448), one rounding each (the conversion saturates); NaN gives -448 as fmaxf
// leaves it.
// `plain`: a divisor gb_div does not take.
GB_DEVINL uint32_t gb_e4m3_div2(float v0, float v1, float scale, float rinv, bool plain) {
  float x0, x1;
  if (plain) { x0 = __fdiv_rn(v0, scale); x1 = __fdiv_rn(v1, scale); }
  else { x0 = gb_div(v0, scale, rinv); x1 = gb_div(v1, scale, rinv); }
  return gb_cvt_e4m3x2(fmaxf(x0, -448.0f), fmaxf(x1, -448.0f));
}

// Two E2M1 codes (one byte) -> fp32.
GB_DEVINL float2 gb_e2m1x2_to_f32(uint32_t byte) {
  uint32_t h2;
  asm("{ .reg .b8 t;\n  cvt.u8.u32 t, %1;\n  cvt.rn.f16x2.e2m1x2 %0, t; }" : "=r"(h2) : "r"(byte));
  return __half22float2(*reinterpret_cast<const __half2*>(&h2));
}

// Two E4M3 bytes -> fp32.
GB_DEVINL float2 gb_e4m3x2_to_f32(uint32_t bytes) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)bytes));
  return __half22float2(*reinterpret_cast<const __half2*>(&h2));
}

// The fp32 scale of a group whose largest magnitude is `amax` (already floored at 1e-8).
GB_DEVINL float gb_fp4_group_scale(float amax, int scale_rule) {
  return scale_rule == GB_SCALE_RULE_DIV ? __fdiv_rn(amax, 6.0f) : __fmul_rn(amax, 1.0f / 6.0f);
}

// bf16 pair of the bucket: E2M1(v / scale) * scale, rounded once each; a zero comes out positive.
// `odd` (an infinity or a NaN in the group, which spreads as in the reference's codec, or a scale
// gb_div does not take): the plain formulation.
GB_DEVINL uint32_t gb_fp4_bucket2(float v0, float v1, float scale, float rinv, bool odd) {
  if (odd) {
    const float q0 = __fmul_rn(gb_e2m1_rtn(__fdiv_rn(v0, scale)), scale);
    const float q1 = __fmul_rn(gb_e2m1_rtn(__fdiv_rn(v1, scale)), scale);
    return gb_f32_to_bf16_bits(q0) | (gb_f32_to_bf16_bits(q1) << 16);
  }
  const float2 q = gb_e2m1x2_to_f32(gb_e2m1_div2(v0, v1, scale, rinv));
  return gb_pack_bf16x2(fmaf(q.x, scale, 0.0f), fmaf(q.y, scale, 0.0f));
}

// Larger of two pairs of bf16, a NaN loses; larger of a pair of magnitudes as fp32.
GB_DEVINL uint32_t gb_max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
GB_DEVINL float gb_max_of_bf16x2(uint32_t m) { return fmaxf(__uint_as_float(m << 16), __uint_as_float(m & 0xFFFF0000u)); }

// Largest magnitude of the words' bf16 values, NaNs ignored, and whether one of them is a NaN.
template <int kWords>
GB_DEVINL float gb_amax_bf16(const uint32_t (&w)[kWords], bool* has_nan) {
  uint32_t m = 0u, n = 0u;                                 // packed maxima, the second keeps NaNs
#pragma unroll
  for (int i = 0; i < kWords; ++i) {
    m = gb_max_bf16x2(m, w[i] & 0x7FFF7FFFu);
    asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(n) : "r"(w[i] & 0x7FFF7FFFu));
  }
  *has_nan = (n & 0x7FFFu) > 0x7F80u || (n >> 16 & 0x7FFFu) > 0x7F80u;
  return gb_max_of_bf16x2(m);
}

template <int kWords>
GB_DEVINL void gb_fp4_bucket_words(uint32_t (&w)[kWords], float amax, bool nan, int scale_rule) {
  amax = fmaxf(amax, 1e-8f);
  float scale = gb_fp4_group_scale(amax, scale_rule);
  if (nan) scale = __int_as_float(0x7FC00000);
  const bool odd = gb_plain_division(scale) || nan;
  const float rinv = __frcp_rn(scale);
#pragma unroll
  for (int i = 0; i < kWords; ++i)
    w[i] = gb_fp4_bucket2(gb_bf16_bits_to_f32(w[i] & 0xFFFFu), gb_bf16_bits_to_f32(w[i] >> 16), scale, rinv, odd);
}

// Group-16 E2M1 bucket of sixteen bf16 values (eight packed words), in place.
GB_DEVINL void gb_fp4_group16_qdq(uint32_t (&w)[8], int scale_rule) {
  bool nan;
  const float amax = gb_amax_bf16(w, &nan);
  gb_fp4_bucket_words(w, amax, nan, scale_rule);
}

// The same bucket with the group spread over eight consecutive lanes (lane % 8 = word of the
// group): every lane of the warp must call it.  Bit-identical to gb_fp4_group16_qdq: the
// maximum ignores NaNs and does not depend on the order, everything else is per value.
GB_DEVINL uint32_t gb_fp4_group16_qdq_lanes(uint32_t w, int scale_rule) {
  uint32_t one[1] = {w};
  bool has_nan;
  float amax = gb_amax_bf16(one, &has_nan);
  uint32_t nan = has_nan ? 1u : 0u;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    nan |= __shfl_xor_sync(0xffffffffu, nan, o);
  }
  gb_fp4_bucket_words(one, amax, nan != 0, scale_rule);
  return one[0];
}

// The same bucket with a group split over two adjacent lanes (eight values each, lane ^ 1 holds
// the other half): both lanes must call it.  Bit-identical to gb_fp4_group16_qdq.
GB_DEVINL uint4 gb_fp4_group16_qdq_pair(uint4 in, int scale_rule) {
  uint32_t w[4] = {in.x, in.y, in.z, in.w};
  bool has_nan;
  float amax = gb_amax_bf16(w, &has_nan);
  uint32_t nan = has_nan ? 1u : 0u;
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  nan |= __shfl_xor_sync(0xffffffffu, nan, 1);
  gb_fp4_bucket_words(w, amax, nan != 0, scale_rule);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// The three-term operand of the block-scaled FP4 kernels (gb_gemv_fp4.cu) holds the groups of a row that lie within
// 2^13 of each other.  Other groups are left out: `tail` has their fp32 scales ([row][K / 16], zero for every other
// group), and the low bits of the row's power of two say which sixteenths of the row hold any.  They are
// multiplied on the plain fp32 units: the lane's weight row times groups [g_begin, g_end) of four activation
// rows (those in `rows`), added to acc.  codes(r, g): the E2M1 codes of a group; load(g): what the lane's weight
// row needs of it (some three hundred L1 wavefronts for the 32 rows of a warp, which bound the work where many
// groups are left out; hence four activation rows for each load); dot(raw, x): its sixteen weights times x, which
// lane i (and i + 16) holds element i of.
constexpr uint32_t kGbLeftOutBits = 0xFFFFu, kGbRowScaleMask = 0x7F800000u;
GB_DEVINL int gb_left_out_span(int n_sb) { return (n_sb + 15) / 16; }   // superblocks per bit
template <typename Codes, typename Load, typename Dot>
GB_DEVINL void gb_left_out(float (&acc)[4], const float* tail, int64_t pitch, uint32_t rows, int g_begin, int g_end, Codes codes,
                           Load load, Dot dot) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int g0 = g_begin; g0 < g_end; g0 += 32) {
    float s[4];
    bool any = false;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      s[r] = (rows >> r & 1u) && g0 + lane < g_end ? tail[r * pitch + g0 + lane] : 0.0f;
      any |= s[r] != 0.0f;
    }
#pragma unroll 1
    for (uint32_t have = __ballot_sync(0xffffffffu, any); have != 0; have &= have - 1) {
      const int b = __ffs(have) - 1, g = g0 + b;
      const auto raw = load(g);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float scale = __shfl_sync(0xffffffffu, s[r], b);
        if (scale == 0.0f) continue;                       // the same in every lane
        const uint2 q = codes(r, g);
        const uint32_t c = ((lane & 8) ? q.y : q.x) >> (4 * (lane & 7));   // bucketed value: bf16(q * scale)
        acc[r] += dot(raw, gb_bf16_bits_to_f32(gb_f32_to_bf16_bits(__fmul_rn(gb_e2m1x2_to_f32(c & 0xFu).x, scale))));
      }
    }
  }
}
// What the groups left out of a row add to a sum that still carries the row's normalisation.
GB_DEVINL float gb_normalised(float v, uint32_t x_word) { return v * __uint_as_float((254u << 23) - (x_word & kGbRowScaleMask)); }
// Adds v to four tensor-memory columns of the warp's lanes.
GB_DEVINL void gb_tmem_add(uint32_t taddr, const float (&v)[4]) {
  uint32_t u[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) u[i] = __float_as_uint(__uint_as_float(u[i]) + v[i]);
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// gate / (1 + exp(-gate)) with the quotient taken as a product with the reciprocal and one correction
// step.  The plain division leaves its fast path when the exponential is huge, and gates far below
// zero are common: the routed SwiGLU launch over 32768 x 768 values spent 186 us, four times what
// its bytes take.
GB_DEVINL float gb_silu(float gate) {
  const float d = 1.0f + __expf(-gate);
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = gate * r;
  return d < 0x1p100f && fabsf(gate) < 0x1p100f ? fmaf(fmaf(-q, d, gate), r, q) : q;
}

// ---------------------------------------------------------------------------
// bit-stream extraction (docs/SPEC.md:56-92): codeword c of a superblock
// occupies stream bits [c*k, c*k+k), least significant bit first.
// ---------------------------------------------------------------------------
// p must point at a 4-byte aligned address at or before the first needed byte;
// bit is the offset of the codeword's LSB from p (may exceed 31).
template <typename Ptr>
GB_DEVINL uint64_t gb_extract_bits(Ptr words, uint32_t bit, int k_bits) {
  const uint32_t w = bit >> 5, s = bit & 31u;
  const uint32_t a = words[w], b = words[w + 1];
  uint64_t lo = __funnelshift_r(a, b, s);
  if (k_bits > 32) {
    const uint32_t c = words[w + 2];
    lo |= (uint64_t)__funnelshift_r(b, c, s) << 32;
  }
  return k_bits >= 64 ? lo : (lo & ((1ull << k_bits) - 1ull));
}

// Generic byte-granular version for unaligned global rows (expand kernels).
GB_DEVINL uint64_t gb_extract_bits_bytes(const uint8_t* p, int64_t nbytes_valid,
                                         uint32_t bit, int k_bits) {
  const uint32_t byte0 = bit >> 3, s = bit & 7u;
  const int nb = (int)(s + (uint32_t)k_bits + 7u) >> 3;     // bytes the field touches
  uint64_t win = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t idx = (int64_t)byte0 + i;
    const uint64_t v = (i < nb && idx < nbytes_valid) ? (uint64_t)p[idx] : 0ull;
    win |= v << (8 * i);
  }
  return (win >> s) & ((1ull << k_bits) - 1ull);
}

struct GbSplit {
  int width[4];
  int shift[4];
  int base[4];   // element offset of sub-table i inside one codebook block
  int sub_dim;
  int n_sub;
};

__host__ __device__ inline GbSplit gb_make_split(int k_bits, int n_sub) {
  GbSplit s;
  s.n_sub = n_sub;
  s.sub_dim = 8 / n_sub;
  int off = 0, base = 0;
  for (int i = 0; i < 4; ++i) {
    if (i < n_sub) {
      s.width[i] = k_bits / n_sub + (i < k_bits % n_sub ? 1 : 0);
      s.shift[i] = off;
      s.base[i] = base;
      off += s.width[i];
      base += (1 << s.width[i]) * s.sub_dim;
    } else {
      s.width[i] = 0; s.shift[i] = 0; s.base[i] = 0;
    }
  }
  return s;
}

__host__ __device__ inline int64_t gb_codebook_elems(const gb_format& f) {
  if (f.mode == GB_MODE_FULL) return (int64_t)8 << f.k_bits;
  if (f.mode == GB_MODE_SIGNED) return (int64_t)8 << (f.k_bits - 8);
  GbSplit s = gb_make_split(f.k_bits, f.n_sub);
  return (int64_t)s.base[f.n_sub - 1] + ((int64_t)s.sub_dim << s.width[f.n_sub - 1]);
}

// ---------------------------------------------------------------------------
// mbarrier / bulk-copy primitives (all waits are bounded)
// ---------------------------------------------------------------------------
GB_DEVINL uint32_t gb_smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

GB_DEVINL void gb_mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gb_smem_u32(bar)), "r"(count));
}

// One lane of a warp that has converged.  Warps that load, issue MMAs or copy walk their loops as a whole, with values that
// are the same in every lane, and the elected lane issues: the operands stay in uniform registers.  (In code that only
// lane 0 enters, each is moved there first: 53 clocks to issue an MMA whatever its size, 45 or more a copy.  One dense layer,
// us: 333 rows K20 249 -> 233, 2048 rows literal 522 -> 491, 8192 rows fp8 2853 -> 2677; routed, 4096 tokens, 656 -> 613.)
GB_DEVINL bool gb_elect_one() {
  uint32_t one;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
  return one != 0;
}

// All threads of a thread-block cluster; what was written before, to a peer's shared memory too, is visible behind it.
GB_DEVINL void gb_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

GB_DEVINL void gb_mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(gb_smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

GB_DEVINL void gb_mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gb_smem_u32(bar)) : "memory");
}

// Programmatic dependent launch.  A kernel launched through gb_launch may start while the
// kernel before it on the stream is still running; gb_pdl_wait() returns once that kernel
// (and everything before it) has completed and its writes are visible, so it must come before
// the first read of anything an earlier kernel produced and before the first global write.
// One exception: an expander behind the launch that quantises the rows (gb_expand_*_beside) writes first and waits before it
// exits.  It may, because that launch lets it start only behind its OWN wait - all work further ahead, the last reader of the
// expander's output too, has completed - and neither reads nor writes what the other writes.
// What sits in front of it - barrier setup, the prefetch of weights, tables of constants -
// overlaps the predecessor's tail.  gb_pdl_launch_dependents() lets the successor start.
GB_DEVINL void gb_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
GB_DEVINL void gb_pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

GB_DEVINL uint64_t gb_globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Returns false when the wait ran out of patience (two seconds of wall clock);
// the caller raises the status word and leaves the kernel.
// `tok` (optional) receives a value the compiler cannot see through; loads that must not move
// above the wait take it as an operand.
GB_DEVINL bool gb_mbar_wait(uint64_t* bar, uint32_t parity, uint32_t* tok = nullptr) {
  const uint32_t addr = gb_smem_u32(bar);
  uint64_t t0 = 0;
  if (tok) *tok = 0;
  for (uint32_t spin = 0;; ++spin) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) {
      if (tok) *tok = done;
      return true;
    }
    if ((spin & 255u) == 255u) {
      const uint64_t now = gb_globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > 2000000000ull) return false;
    }
  }
}

// 1-D bulk copy global -> this CTA's shared memory, completion on an mbarrier.
// Both addresses 16-byte aligned, bytes a multiple of 16.
GB_DEVINL void gb_bulk_g2s(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          gb_smem_u32(smem_dst)),
      "l"(gmem_src), "r"(bytes), "r"(gb_smem_u32(bar))
      : "memory");
}

GB_DEVINL void gb_fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// D[16x8] = A[16x8] . B[8x8] (bf16 in, fp32 out, no accumulator input)
GB_DEVINL void gb_mma_bf16_1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0), "f"(0.0f));
}

GB_DEVINL void gb_mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  // not volatile: a pure function of its register operands, free to be interleaved
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
