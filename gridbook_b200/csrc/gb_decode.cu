// Activation buckets and decoded-tile expanders.
//
// The expanders are the bit-exact gate of the whole library: every other kernel's
// decode reduces to "the tile it multiplies equals what these write".
#include "gb_common.cuh"

namespace {

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------
// Activation buckets (gridbook/codec.py:248-260, 428-437)
// ---------------------------------------------------------------------------
// One thread per group of 16: two 16-byte loads, amax, scale, 16 roundings.  kAligned = false: rows that start
// anywhere, value by value.
template <bool kAligned>
__global__ void __launch_bounds__(kThreads)
fp4_group16_qdq_kernel(const uint16_t* __restrict__ x, uint16_t* __restrict__ out,
                       int64_t n_groups, int scale_rule) {
  gb_pdl_launch_dependents();
  gb_pdl_wait();
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_groups) return;
  uint32_t packed[8];
  if (kAligned) {
    const uint4* src = reinterpret_cast<const uint4*>(x + g * 16);
    const uint4 r0 = src[0], r1 = src[1];
    packed[0] = r0.x; packed[1] = r0.y; packed[2] = r0.z; packed[3] = r0.w;
    packed[4] = r1.x; packed[5] = r1.y; packed[6] = r1.z; packed[7] = r1.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) packed[i] = x[g * 16 + 2 * i] | (uint32_t)x[g * 16 + 2 * i + 1] << 16;
  }
  gb_fp4_group16_qdq(packed, scale_rule);
  if (kAligned) {
    uint4* dst = reinterpret_cast<uint4*>(out + g * 16);
    dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      out[g * 16 + 2 * i] = (uint16_t)packed[i];
      out[g * 16 + 2 * i + 1] = (uint16_t)(packed[i] >> 16);
    }
  }
}

// Per-token E4M3 bucket: one CTA per row, the row held in registers (kVec vectors of eight values
// per thread), so it is read once: block-wide amax, then every element is scaled and rounded once
// to E4M3.  kQuantize: the E4M3 bytes and the row's scale; otherwise scaled back to bf16.
// Bound by memory for many rows (8192 x 17408: 257 us when each element was loaded twice on its own
// and divided), by the two round trips for a few.
template <int kVec, bool kQuantize>
__global__ void __launch_bounds__(1024)
fp8_rows_kernel(const uint4* __restrict__ x, void* __restrict__ out, float* __restrict__ scale_out, int vecs,
                int scale_rule) {
  if (!kQuantize) gb_pdl_launch_dependents();
  gb_pdl_wait();
  if (kQuantize) gb_pdl_launch_dependents();               // the weights' expander runs beside this launch (gb_expand_fp8_beside)
  const uint4* row = x + (int64_t)blockIdx.x * vecs;
  __shared__ float red[32];
  uint4 v[kVec];
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    const int i = threadIdx.x + j * blockDim.x;
    v[j] = i < vecs ? row[i] : make_uint4(0u, 0u, 0u, 0u);
  }
  uint32_t top = 0u;
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
    for (int q = 0; q < 4; ++q) top = gb_max_bf16x2(top, w[q] & 0x7FFF7FFFu);
  }
  float amax = gb_max_of_bf16x2(top);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = (int)(threadIdx.x & 31) < (int)(blockDim.x + 31) / 32 ? red[threadIdx.x & 31] : 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float s = scale_rule == GB_SCALE_RULE_DIV ? __fdiv_rn(amax, 448.0f) : __fmul_rn(amax, 1.0f / 448.0f);
  const float scale = fmaxf(s, 1.0f / (448.0f * 512.0f)), rinv = __frcp_rn(scale);
  const bool plain = gb_plain_division(scale);
  if (kQuantize && threadIdx.x == 0) scale_out[blockIdx.x] = scale;
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    const int i = threadIdx.x + j * blockDim.x;
    if (i >= vecs) break;
    const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
    uint32_t q[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) q[c] = gb_e4m3_div2(gb_bf16_bits_to_f32(w[c] & 0xFFFFu), gb_bf16_bits_to_f32(w[c] >> 16), scale, rinv, plain);
    if (kQuantize) {
      reinterpret_cast<uint2*>(out)[(int64_t)blockIdx.x * vecs + i] = make_uint2(q[0] | (q[1] << 16), q[2] | (q[3] << 16));
    } else {
      uint32_t r[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 f = gb_e4m3x2_to_f32(q[c]);
        r[c] = gb_pack_bf16x2(__fmul_rn(f.x, scale), __fmul_rn(f.y, scale));
      }
      reinterpret_cast<uint4*>(out)[(int64_t)blockIdx.x * vecs + i] = make_uint4(r[0], r[1], r[2], r[3]);
    }
  }
}

// The same for rows that are not whole aligned vectors (or longer than the registers of a CTA hold).
template <bool kQuantize>
__global__ void __launch_bounds__(kThreads)
fp8_rows_any_kernel(const uint16_t* __restrict__ x, void* __restrict__ out, float* __restrict__ scale_out, int64_t K,
                    int scale_rule) {
  if (!kQuantize) gb_pdl_launch_dependents();
  gb_pdl_wait();
  if (kQuantize) gb_pdl_launch_dependents();
  const uint16_t* row = x + (int64_t)blockIdx.x * K;
  __shared__ float red[kThreads / 32];
  __shared__ float s_scale;
  float amax = 0.0f;
  for (int64_t i = threadIdx.x; i < K; i += blockDim.x)
    amax = fmaxf(amax, fabsf(gb_bf16_bits_to_f32(row[i])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x == 0) {
    float a = red[0];
    for (int w = 1; w < kThreads / 32; ++w) a = fmaxf(a, red[w]);
    const float s = scale_rule == GB_SCALE_RULE_DIV ? __fdiv_rn(a, 448.0f)
                                                    : __fmul_rn(a, 1.0f / 448.0f);
    s_scale = fmaxf(s, 1.0f / (448.0f * 512.0f));
    if (kQuantize) scale_out[blockIdx.x] = s_scale;
  }
  __syncthreads();
  const float scale = s_scale;
  for (int64_t i = threadIdx.x; i < K; i += blockDim.x) {
    const float v = gb_bf16_bits_to_f32(row[i]);
    const uint32_t q = gb_f32_to_e4m3(fminf(fmaxf(__fdiv_rn(v, scale), -448.0f), 448.0f));
    if (kQuantize) reinterpret_cast<uint8_t*>(out)[(int64_t)blockIdx.x * K + i] = (uint8_t)q;
    else reinterpret_cast<uint16_t*>(out)[(int64_t)blockIdx.x * K + i] = (uint16_t)gb_f32_to_bf16_bits(__fmul_rn(gb_e4m3_to_f32(q), scale));
  }
}

// Rows of up to 8 x 1024 vectors stay in registers; the fewest vectors per thread that 512 threads
// (or, past that, 1024) can hold, since a few long rows are bound by latency.  Rows enough for several waves
// take twice as many: smaller CTAs, more rows in flight per SM (8192 x 5120 33 -> 26 us, 8192 x 17408 100 -> 82).
template <bool kQuantize>
int launch_fp8_rows(const void* x, void* out, float* scale, int64_t M, int64_t K, int scale_rule, void* stream) {
  const int64_t vecs = K / 8;
  cudaStream_t st = (cudaStream_t)stream;
  if (K % 8 != 0 || vecs > 8 * 1024 || ((uintptr_t)x & 15u) != 0 || ((uintptr_t)out & (kQuantize ? 7u : 15u)) != 0) {
    GB_CUDA_OK(gb_launch(fp8_rows_any_kernel<kQuantize>, dim3((unsigned)M), dim3(kThreads), 0, st, (const uint16_t*)x, out,
                         scale, K, scale_rule));
    return GB_OK;
  }
  int per = vecs <= 512 ? 1 : vecs <= 1024 ? 2 : vecs <= 2048 + 512 ? 4 : 8;
  if (per < 8 && M >= 8 * gb_sm_count()) per *= 2;
  const unsigned threads = (unsigned)(((vecs + per - 1) / per + 31) / 32 * 32);
#define GB_FP8_ROWS(V)                                                                                        \
  GB_CUDA_OK(gb_launch(fp8_rows_kernel<V, kQuantize>, dim3((unsigned)M), dim3(threads), 0, st, (const uint4*)x, out, scale, \
                       (int)vecs, scale_rule))
  switch (per) {
    case 1: GB_FP8_ROWS(1); break;
    case 2: GB_FP8_ROWS(2); break;
    case 4: GB_FP8_ROWS(4); break;
    default: GB_FP8_ROWS(8); break;
  }
#undef GB_FP8_ROWS
  return GB_OK;
}

// ---------------------------------------------------------------------------
// Expanders.  One warp per (row, superblock); lane v owns codeword v, i.e. the
// eight weights [8v, 8v+8) of the superblock and half of group v/2.
// ---------------------------------------------------------------------------
struct ExpandArgs {
  const uint8_t* qw;
  int64_t row_stride;
  int64_t valid_bytes;   // bytes that may be read from the first row's start
  const void* codebook;
  const int32_t* cb_row_offset;
  const float* compose;
  const float* weight_scale;   // fp8 grid: per-row scale, indexed by the absolute row
  int64_t row0, nrows, K;
  gb_format fmt;
  GbSplit split;
};

// Codebook values of one codeword as fp32 (exact for both grids).
template <bool kFp8>
GB_DEVINL void gather_values(const ExpandArgs& a, int64_t cb_base, uint64_t code, float (&val)[8]) {
  auto load = [&](int64_t idx) -> float {
    if constexpr (kFp8)
      return gb_e4m3_to_f32(reinterpret_cast<const uint8_t*>(a.codebook)[cb_base + idx]);
    else
      return gb_bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(a.codebook)[cb_base + idx]);
  };
  if (a.fmt.mode == GB_MODE_FULL) {
    if constexpr (!kFp8) {
      // a full codeword is eight consecutive bf16: one 16-byte load when the block is aligned
      const uint16_t* entry = reinterpret_cast<const uint16_t*>(a.codebook) + cb_base + (int64_t)code * 8;
      if ((reinterpret_cast<uintptr_t>(entry) & 15u) == 0) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(entry));
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          val[2 * j] = gb_bf16_bits_to_f32(w[j] & 0xffffu);
          val[2 * j + 1] = gb_bf16_bits_to_f32(w[j] >> 16);
        }
        return;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) val[j] = load((int64_t)code * 8 + j);
  } else if (a.fmt.mode == GB_MODE_SIGNED) {
    const int64_t mag = (int64_t)(code >> 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float m = load(mag * 8 + j);
      val[j] = ((code >> j) & 1ull) ? -m : m;
    }
  } else {
    const int sd = a.split.sub_dim;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int s = j / sd;   // sd is 2 or 4, so s < n_sub
      const int64_t idx = (int64_t)((code >> a.split.shift[s]) & ((1ull << a.split.width[s]) - 1ull));
      val[j] = load(a.split.base[s] + idx * sd + (j - s * sd));
    }
  }
}

// Group scale of codeword v (group v/2) for the fp4 grid, as fp32 and as its E4M3 byte.
GB_DEVINL float fp4_group_scale(const ExpandArgs& a, const uint8_t* sb, int v, uint32_t* byte_out) {
  const int g = v >> 1;
  const uint8_t* plane = sb + 4 * a.fmt.k_bits;
  if (a.fmt.scale_coding == GB_SCALE_V1) {
    const uint32_t b = plane[g];
    *byte_out = b;
    return gb_e4m3_to_f32(b);
  }
  const uint32_t e = plane[0];
  const uint32_t nib = (plane[1 + (g >> 1)] >> ((g & 1) * 4)) & 0xFu;
  const float s = a.compose[e * 16 + nib];
  *byte_out = gb_f32_to_e4m3(fminf(s, 448.0f));   // exact for every legal (E, c) pair
  return s;
}

enum { kOutFp8 = 0, kOutBf16 = 1, kOutNvfp4 = 2, kOutFp8Bf16 = 3 };

// Every warp takes kUnitsPerWarp consecutive (row, superblock) units and runs them in phases:
// all code loads, then all codebook and scale loads, then all stores, so that two independent
// load chains are in flight per lane.  Measured on the 805 MB bf16 tile of a 128-expert stack:
// one unit 327 us, two 291 us, four 372 us (fewer resident warps); at two the kernel writes
// 2.8 TB/s, close to the write half of a device copy.
constexpr int kUnitsPerWarp = 2;

template <int kOut>
__global__ void __launch_bounds__(kThreads)
expand_kernel(ExpandArgs a, void* __restrict__ out0, uint8_t* __restrict__ out_sf, int sf_swizzled) {
  constexpr bool kFp8Grid = kOut == kOutFp8 || kOut == kOutFp8Bf16;
  const int lane = threadIdx.x & 31;
  const int64_t n_sb = a.K / 256, units = a.nrows * n_sb;
  const int64_t unit0 = ((int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * kUnitsPerWarp;
  if (unit0 >= units) return;

  int64_t r[kUnitsPerWarp], s[kUnitsPerWarp];
  const uint8_t* sb[kUnitsPerWarp];
  uint64_t code[kUnitsPerWarp];
#pragma unroll
  for (int u = 0; u < kUnitsPerWarp; ++u) {
    const int64_t unit = unit0 + u < units ? unit0 + u : unit0;     // a dead unit re-reads the first
    // the unit index fits 32 bits whenever the grid does: one short division
    r[u] = unit < (1ll << 32) ? (int64_t)((uint32_t)unit / (uint32_t)n_sb) : unit / n_sb;
    s[u] = unit - r[u] * n_sb;
    const int64_t sb_off = r[u] * a.row_stride + s[u] * a.fmt.type_size;
    sb[u] = a.qw + sb_off;   // a.qw is the first byte of row0
    // byte-wide codes sit at byte `lane` of the superblock; other widths go through the bit window
    code[u] = a.fmt.k_bits == 8 ? (uint64_t)sb[u][lane]
                                : gb_extract_bits_bytes(sb[u], a.valid_bytes - sb_off, (uint32_t)(lane * a.fmt.k_bits),
                                                        a.fmt.k_bits);
  }

  float val[kUnitsPerWarp][8], scale[kUnitsPerWarp];
  uint32_t sbyte[kUnitsPerWarp];
  uint4 raw[kUnitsPerWarp];          // bf16 tile of a full-mode codeword: the eight bf16 as loaded
  bool have_raw[kUnitsPerWarp];
#pragma unroll
  for (int u = 0; u < kUnitsPerWarp; ++u) {
    const int64_t row = a.row0 + r[u];
    const int64_t cb_base = a.cb_row_offset ? (int64_t)a.cb_row_offset[row] : 0;
    have_raw[u] = false;
    if constexpr (kOut == kOutBf16) {
      const uint16_t* entry = reinterpret_cast<const uint16_t*>(a.codebook) + cb_base + (int64_t)code[u] * 8;
      if (a.fmt.mode == GB_MODE_FULL && (reinterpret_cast<uintptr_t>(entry) & 15u) == 0) {
        raw[u] = __ldg(reinterpret_cast<const uint4*>(entry));
        have_raw[u] = true;
      }
    }
    if (!have_raw[u]) gather_values<kFp8Grid>(a, cb_base, code[u], val[u]);
    sbyte[u] = 0;
    if constexpr (kOut == kOutFp8Bf16) scale[u] = a.weight_scale[row];     // the served weight's row scale
    else if constexpr (kOut == kOutFp8) scale[u] = 1.0f;
    else scale[u] = fp4_group_scale(a, sb[u], lane, &sbyte[u]);
  }

#pragma unroll
  for (int u = 0; u < kUnitsPerWarp; ++u) {
    if (unit0 + u >= units) break;
    const int64_t col = s[u] * 256 + lane * 8;
    const int64_t at = r[u] * a.K + col;
    if constexpr (kOut == kOutFp8) {
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        lo |= gb_f32_to_e4m3(val[u][j]) << (8 * j);
        hi |= gb_f32_to_e4m3(val[u][4 + j]) << (8 * j);
      }
      *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(out0) + at) = make_uint2(lo, hi);
    } else if constexpr (kOut == kOutBf16 || kOut == kOutFp8Bf16) {
      // bf16(value * scale): the group scale (fp4 grid) or the row scale (fp8 grid)
      uint32_t p[4];
      const uint32_t sbits = __float_as_uint(scale[u]);
      if (kOut == kOutBf16 && have_raw[u] && (sbits & 0xFFFFu) == 0) {
        // the scale is a bf16 number (every E4M3 byte is): the packed bf16 multiply rounds the
        // exact product once, the same bits as bf16(f32(value) * f32(scale))
        const uint32_t s2 = (sbits >> 16) * 0x10001u;
        const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(p[j]) : "r"(w[j]), "r"(s2));
      } else {
        if (kOut == kOutBf16 && have_raw[u]) {
          const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            val[u][2 * j] = gb_bf16_bits_to_f32(w[j] & 0xffffu);
            val[u][2 * j + 1] = gb_bf16_bits_to_f32(w[j] >> 16);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          p[j] = gb_pack_bf16x2(__fmul_rn(val[u][2 * j], scale[u]), __fmul_rn(val[u][2 * j + 1], scale[u]));
      }
      *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out0) + at) = make_uint4(p[0], p[1], p[2], p[3]);
    } else {
      uint32_t nib = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // E2M1 code: magnitudes {0,.5,1,1.5,2,3,4,6} -> 0..7, bit 3 = sign
        const float m = fabsf(val[u][j]);
        const uint32_t c = m < 2.0f ? (uint32_t)(m * 2.0f) : (m < 4.0f ? (uint32_t)m + 2u : (m < 6.0f ? 6u : 7u));
        nib |= (c | (val[u][j] < 0.0f ? 8u : 0u)) << (4 * j);
      }
      if (sf_swizzled == 2 && (sbyte[u] & 0x80u)) {
        // operand form of the block-scaled MMA, whose scale factors carry no sign: a negative
        // group scale moves its sign into the group's sixteen values, (-s) * v = s * (-v)
        nib ^= 0x88888888u;
        sbyte[u] &= 0x7Fu;
      }
      reinterpret_cast<uint32_t*>(out0)[at >> 3] = nib;
      if ((lane & 1) == 0) {
        const int64_t groups = a.K / 16;
        const int64_t g = s[u] * 16 + (lane >> 1);
        int64_t off = r[u] * groups + g;
        if (sf_swizzled) {
          const int64_t gpad = (groups + 3) / 4 * 4;
          const int64_t rr = r[u];
          off = (rr % 32) * 16 + ((rr / 32) % 4) * 4 + (g % 4) + (g / 4) * 512 + (rr / 128) * (512 * (gpad / 4));
        }
        out_sf[off] = (uint8_t)sbyte[u];
      }
    }
  }
}

int make_expand_args(const gb_weight* w, int64_t row0, int64_t nrows, ExpandArgs* a) {
  int rc = gb_check_weight(w);
  if (rc != GB_OK) return rc;
  GB_REQUIRE(row0 >= 0 && nrows > 0 && row0 + nrows <= w->rows, "rows [%lld, %lld) outside [0, %lld)",
             (long long)row0, (long long)(row0 + nrows), (long long)w->rows);
  a->qw = w->qw;
  a->row_stride = w->row_stride;
  a->codebook = w->codebook;
  a->cb_row_offset = w->cb_row_offset;
  a->compose = w->compose;
  a->weight_scale = w->weight_scale;
  a->row0 = row0;
  a->nrows = nrows;
  a->K = w->K;
  a->fmt = w->fmt;
  a->split = gb_make_split(w->fmt.k_bits, w->fmt.mode == GB_MODE_PRODUCT ? w->fmt.n_sub : 1);
  return GB_OK;
}

}  // namespace

extern "C" {

int gb_fp4_act_qdq(const void* x, void* out, int64_t M, int64_t K, int scale_rule, void* stream) {
  GB_REQUIRE(x && out, "null activation pointer");
  GB_REQUIRE(M >= 0 && K > 0 && K % 16 == 0, "fp4 activation bucket wants K %% 16 == 0, got K=%lld",
             (long long)K);
  if (M == 0) return GB_OK;
  const int64_t groups = M * (K / 16);
  const unsigned blocks = (unsigned)((groups + kThreads - 1) / kThreads);
  const bool aligned = (((uintptr_t)x | (uintptr_t)out) & 15u) == 0;
  GB_CUDA_OK(gb_launch(aligned ? fp4_group16_qdq_kernel<true> : fp4_group16_qdq_kernel<false>, dim3(blocks), dim3(kThreads), 0,
                       (cudaStream_t)stream, (const uint16_t*)x, (uint16_t*)out, groups, scale_rule));
  return GB_OK;
}

int gb_fp8_act_qdq(const void* x, void* out, int64_t M, int64_t K, int scale_rule, void* stream) {
  GB_REQUIRE(x && out, "null activation pointer");
  GB_REQUIRE(M >= 0 && K > 0, "bad shape M=%lld K=%lld", (long long)M, (long long)K);
  if (M == 0) return GB_OK;
  return launch_fp8_rows<false>(x, out, nullptr, M, K, scale_rule, stream);
}

int gb_fp8_quantize_rows(const void* x, void* q, float* scale, int64_t M, int64_t K, int scale_rule, void* stream) {
  GB_REQUIRE(x && q && scale, "null pointer argument");
  GB_REQUIRE(M >= 0 && K > 0, "bad shape M=%lld K=%lld", (long long)M, (long long)K);
  if (M == 0) return GB_OK;
  return launch_fp8_rows<true>(x, q, scale, M, K, scale_rule, stream);
}

}  // extern "C"

namespace {
template <int kOut>
int launch_expand(const gb_weight* w, int64_t row0, int64_t nrows, void* out0, void* out_sf,
                  int sf_swizzled, void* stream) {
  ExpandArgs a;
  int rc = make_expand_args(w, row0, nrows, &a);
  if (rc != GB_OK) return rc;
  GB_REQUIRE(out0 != nullptr, "null output");
  // The kernel addresses rows relative to row0 so that `valid_bytes` bounds every read.
  a.qw = w->qw + row0 * w->row_stride;
  a.valid_bytes = (nrows - 1) * w->row_stride + (w->K / 256) * w->fmt.type_size;
  const int64_t units = nrows * (w->K / 256);
  const int64_t per_cta = (kThreads / 32) * kUnitsPerWarp;
  const unsigned blocks = (unsigned)((units + per_cta - 1) / per_cta);
  gb_count_launch();
  expand_kernel<kOut><<<blocks, kThreads, 0, (cudaStream_t)stream>>>(a, out0, (uint8_t*)out_sf,
                                                                    sf_swizzled);
  GB_LAUNCH_OK("expand_kernel");
  return GB_OK;
}

// The fp8 product formats k = 32 (four sub-tables of two values) and k = 16 (two sub-tables of four
// values) -> the E4M3 value plane, one byte per weight: the sub-table entries are copied through as
// they are.  Eight lanes per (row, superblock); a lane takes two codewords of each half of the
// superblock, so that every store instruction of the eight lanes writes 128 contiguous bytes.  The
// sub-tables sit in shared memory as 32-bit words, eight copies each (copy = lane mod 8: lanes of
// different copies never share a bank).  Memory-bound: 128 or 64 bytes read and 256 written per
// 256 weights.  A CTA takes a contiguous run of rows and rebuilds its tables where they change codebook (k = 16 with
// a codebook per role took the generic kernel before: 8192 x 5120 99.7 -> 10.9 us).
constexpr int kF8Unroll = 4;

// Rows [run, end) from `run` on that share a codebook block; *base: its element offset.  Called by the whole CTA.
GB_DEVINL int64_t codebook_run(const int32_t* offsets, int64_t run, int64_t end, int64_t* base, int* scratch) {
  if (offsets == nullptr) { *base = 0; return end; }
  const int32_t mine = offsets[run];
  *base = mine;
  __syncthreads();
  if (threadIdx.x == 0) *scratch = (int)(end - run);
  __syncthreads();
  for (int64_t r = run + threadIdx.x; r < end; r += blockDim.x)
    if (offsets[r] != mine) { atomicMin(scratch, (int)(r - run)); break; }
  __syncthreads();
  return run + *scratch;
}

// An expander right behind the launch that quantises the rows of the same product (gb_expand_*_beside): nothing of that one
// is read or overwritten, and it lets its successor start only once everything ahead of it has completed, so the
// two run side by side.  The wait moves to the end, so that whoever waits for this launch waits for both.
// One linear, both launches and the GEMM, us, one after the other / side by side: fp8 k = 16, 200 rows of 2048 x 2048 21.6 / 17.4,
// K20 100 rows of 2048 x 2048 19.7 / 17.4 (19.9 before its tables were built from vector loads: they start later
// here), 600 rows of 8192 x 5120 39.6 / 36.5, literal 2048 rows 57.1 / 56.9.
GB_DEVINL void wait_before_output(bool beside) { if (!beside) gb_pdl_wait(); }
GB_DEVINL void wait_at_end(bool beside) { if (beside) gb_pdl_wait(); }

template <bool kK32>
__global__ void __launch_bounds__(kThreads)
expand_fp8_fast_kernel(const uint8_t* __restrict__ qw, int64_t row_stride, const uint8_t* __restrict__ codebook, const int32_t* __restrict__ offsets,
                       int64_t nrows, int n_sb, int rows_per_cta, bool beside, uint4* __restrict__ out) {
  constexpr int kEntries = kK32 ? 1024 : 512;              // 4 x 256 two-byte or 2 x 256 four-byte entries
  constexpr int kSb = kK32 ? 128 : 64;
  __shared__ uint32_t lut[kEntries * 8];
  __shared__ int run_s;
  const int lane = threadIdx.x & 31, sub = lane & 7, which = lane >> 3;
  const uint32_t* my = lut + sub;
  const int64_t r_begin = (int64_t)blockIdx.x * rows_per_cta, r_end = min(r_begin + rows_per_cta, nrows);
  bool waited = false;
  gb_pdl_launch_dependents();
  for (int64_t run = r_begin; run < r_end;) {
    int64_t base;
    const int64_t run_end = codebook_run(offsets, run, r_end, &base, &run_s);
    const uint8_t* book = codebook + base;
    for (int e = threadIdx.x; e < kEntries; e += kThreads) {
      uint32_t v;
      if (((uintptr_t)book & 3u) != 0) {                   // a row's offset may be any
        const uint8_t* c = book + e * (kK32 ? 2 : 4);
        v = c[0] | (uint32_t)c[1] << 8 | (kK32 ? 0u : (uint32_t)c[2] << 16 | (uint32_t)c[3] << 24);
      } else {
        v = kK32 ? (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(book) + e) : __ldg(reinterpret_cast<const uint32_t*>(book) + e);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) lut[e * 8 + j] = v;
    }
    __syncthreads();
    if (!waited) { wait_before_output(beside); waited = true; }
    const uint8_t* rows = qw + run * row_stride;
    uint4* to = out + run * n_sb * 16;
    const uint32_t units = (uint32_t)(run_end - run) * (uint32_t)n_sb;   // fits: rows_per_cta * n_sb is checked
    for (uint32_t u0 = (threadIdx.x >> 5) * (4 * kF8Unroll); u0 < units; u0 += (kThreads / 32) * (4 * kF8Unroll)) {
      uint32_t in[kF8Unroll][kK32 ? 4 : 2];                // two codewords of the first half, two of the second
#pragma unroll
      for (int i = 0; i < kF8Unroll; ++i) {
        const uint32_t u = u0 + 4 * i + which < units ? u0 + 4 * i + which : u0;
        const uint32_t r = u / (uint32_t)n_sb, sb = u - r * (uint32_t)n_sb;
        const uint8_t* p = rows + r * row_stride + sb * kSb;
        if (kK32) {
          const uint2 a = __ldg(reinterpret_cast<const uint2*>(p) + sub), b = __ldg(reinterpret_cast<const uint2*>(p + 64) + sub);
          in[i][0] = a.x; in[i][1] = a.y; in[i][2] = b.x; in[i][3] = b.y;
        } else {
          in[i][0] = __ldg(reinterpret_cast<const uint32_t*>(p) + sub);
          in[i][1] = __ldg(reinterpret_cast<const uint32_t*>(p + 32) + sub);
        }
      }
#pragma unroll
      for (int i = 0; i < kF8Unroll; ++i) {
        const uint32_t u = u0 + 4 * i + which;
        if (u >= units) continue;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint4 o;
          if (kK32) {
            const uint32_t c0 = in[i][2 * half], c1 = in[i][2 * half + 1];
            o.x = my[(c0 & 0xffu) * 8] | (my[(256 + ((c0 >> 8) & 0xffu)) * 8] << 16);
            o.y = my[(512 + ((c0 >> 16) & 0xffu)) * 8] | (my[(768 + (c0 >> 24)) * 8] << 16);
            o.z = my[(c1 & 0xffu) * 8] | (my[(256 + ((c1 >> 8) & 0xffu)) * 8] << 16);
            o.w = my[(512 + ((c1 >> 16) & 0xffu)) * 8] | (my[(768 + (c1 >> 24)) * 8] << 16);
          } else {
            const uint32_t c = in[i][half];                // two 16-bit codewords
            o.x = my[(c & 0xffu) * 8];
            o.y = my[(256 + ((c >> 8) & 0xffu)) * 8];
            o.z = my[((c >> 16) & 0xffu) * 8];
            o.w = my[(256 + (c >> 24)) * 8];
          }
          to[(int64_t)u * 16 + half * 8 + sub] = o;
        }
      }
    }
    run = run_end;
    if (run < r_end) __syncthreads();                      // the next run rebuilds the tables
  }
  wait_at_end(beside);
}

int launch_expand_fp8_fast(const gb_weight* w, int64_t row0, int64_t nrows, void* out, bool beside, void* stream) {
  const int sms = gb_sm_count();
  if (sms <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  const int64_t n_sb = w->K / 256;
  // Eight CTAs per SM where there are rows for them, at least 64 superblocks each so that the tables pay.  Fewer and larger ones
  // pile up on the SMs that the launch ahead leaves first: k = 32, 4096 x 4096 behind the quantiser of 700 rows, both launches / the
  // whole linear, us: 256 superblocks 17.2 / 35.8, 128 11.8 / 29.2, 64 10.8 / 27.5, 32 the same.
  const int64_t least = (64 + n_sb - 1) / n_sb;
  int64_t rows_per = (nrows + (int64_t)sms * 8 - 1) / ((int64_t)sms * 8);
  if (rows_per < least) rows_per = least;
  GB_REQUIRE(rows_per * n_sb < (1ll << 31), "too many superblocks per CTA");
  const unsigned blocks = (unsigned)((nrows + rows_per - 1) / rows_per);
  GB_CUDA_OK(gb_launch(w->fmt.k_bits == 32 ? expand_fp8_fast_kernel<true> : expand_fp8_fast_kernel<false>, dim3(blocks), dim3(kThreads), 0,
                       (cudaStream_t)stream, w->qw + row0 * w->row_stride, w->row_stride, (const uint8_t*)w->codebook,
                       w->cb_row_offset ? w->cb_row_offset + row0 : nullptr, nrows, (int)n_sb, (int)rows_per, beside, (uint4*)out));
  return GB_OK;
}

// ---- product formats of any width, fast -----------------------------------------------------
// fp4 grid, two sub-indices (K12 .. K24, either scale coding) and fp8 grid, four sub-indices (ragged
// rungs included) -> the native NVFP4 pair, the E4M3 plane or the bf16 tile.  The generic kernel
// above gathers eight values one by one from global memory and converts each: 566 us for the NVFP4
// view of a 34816 x 5120 K20 layer (0.29 TB/s of 233 bytes moved per superblock).  Here a sub-index
// is ONE shared-memory lookup of its finished output bits (four E2M1 nibbles or two E4M3 bytes: a
// 16-bit entry; four bf16: an 8-byte entry), the scale byte comes out of a 4096-entry table, and
// eight lanes share a superblock so that every store instruction writes 128 contiguous bytes: bound
// by memory from about K20 down, by the lookups (bank conflicts between random entries; copies
// interleaved per lane where they fit) above.
// A CTA takes a contiguous run of rows; where the rows change codebook (fused modules with one
// book per role) it rebuilds its tables.
constexpr int kProdThreads = 512;
constexpr int kProdLutCap = 64 * 1024;                     // three CTAs per SM keep the loads in flight

GB_DEVINL uint32_t e2m1_nibble(uint32_t bf16_bits) {
  const float v = gb_bf16_bits_to_f32(bf16_bits), m = fabsf(v);
  const uint32_t c = m < 2.0f ? (uint32_t)(m * 2.0f) : (m < 4.0f ? (uint32_t)m + 2u : (m < 6.0f ? 6u : 7u));
  return c | (v < 0.0f ? 8u : 0u);
}

// Two bf16 values of the grid as nibbles, the lower half's in the low one; a zero comes out positive.
GB_DEVINL uint32_t e2m1_pair(uint32_t w) { return gb_cvt_e2m1x2(__uint_as_float(w << 16) + 0.0f, __uint_as_float(w & 0xFFFF0000u) + 0.0f); }

struct ProdArgs {
  ExpandArgs a;
  int entries;        // sub-table entries of one codebook block
  int copies;         // interleaved copies of every entry (a power of two)
  int n_sb;
  int64_t rows_per_cta;
  bool beside;
};

// Bits [bit, bit + n) of the stream at `p` (any alignment), n <= 64: only words that hold a wanted bit are read.
GB_DEVINL uint64_t stream_bits(const uint8_t* p, uint32_t bit, int n) {
  const uintptr_t at = (uintptr_t)p + (bit >> 3);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(at & ~(uintptr_t)3);
  const uint32_t s = ((uint32_t)(at & 3u) << 3) | (bit & 7u);
  const uint32_t w0 = __ldg(w), w1 = s + n > 32 ? __ldg(w + 1) : 0u, w2 = s + n > 64 ? __ldg(w + 2) : 0u;
  const uint64_t lo = __funnelshift_r(w0, w1, s), hi = __funnelshift_r(w1, w2, s);
  const uint64_t v = lo | (hi << 32);
  return n >= 64 ? v : v & ((1ull << n) - 1ull);
}

template <int kOut>
__global__ void __launch_bounds__(kProdThreads)
expand_product_kernel(const __grid_constant__ ProdArgs p, void* __restrict__ out0, uint8_t* __restrict__ out_sf,
                      int fold_sign) {
  constexpr bool kFp8 = kOut == kOutFp8 || kOut == kOutFp8Bf16;
  constexpr bool kWide = kOut == kOutBf16;                 // 8-byte entries
  constexpr int kSubs = kFp8 ? 4 : 2;
  extern __shared__ uint8_t smem[];
  __shared__ int run_end_s;
  const ExpandArgs& a = p.a;
  uint8_t* comp_s = smem;                                  // two-tier scale bytes (NVFP4 output only)
  uint8_t* lut_s = smem + (kOut == kOutNvfp4 ? 4096 : 0);
  const int tid = threadIdx.x, lane = tid & 31, sub = lane & 7, which = lane >> 3;
  const int k = a.fmt.k_bits;
  const bool v2 = a.fmt.scale_coding == GB_SCALE_V2;
  const uint32_t my = (uint32_t)(sub & (p.copies - 1));
  bool waited = false;
  gb_pdl_launch_dependents();
  if (kOut == kOutNvfp4 && v2)
    for (int i = tid; i < 4096; i += kProdThreads) comp_s[i] = (uint8_t)gb_f32_to_e4m3(fminf(__ldg(a.compose + i), 448.0f));

  const int64_t r_begin = (int64_t)blockIdx.x * p.rows_per_cta;
  const int64_t r_end = r_begin + p.rows_per_cta < a.nrows ? r_begin + p.rows_per_cta : a.nrows;
  for (int64_t run = r_begin; run < r_end;) {
    int64_t cb_base;
    const int64_t run_end = codebook_run(a.cb_row_offset ? a.cb_row_offset + a.row0 : nullptr, run, r_end, &cb_base, &run_end_s);
    for (int e = tid; e < p.entries; e += kProdThreads) {
      if constexpr (kFp8) {
        const uint8_t* c = reinterpret_cast<const uint8_t*>(a.codebook) + cb_base + (int64_t)e * 2;
        const uint16_t v = (uint16_t)(c[0] | (c[1] << 8));
        for (int j = 0; j < p.copies; ++j) reinterpret_cast<uint16_t*>(lut_s)[e * p.copies + j] = v;
      } else {
        const uint16_t* c = reinterpret_cast<const uint16_t*>(a.codebook) + cb_base + (int64_t)e * 4;
        const uint32_t c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
        if constexpr (kWide) {
          for (int j = 0; j < p.copies; ++j)
            reinterpret_cast<uint2*>(lut_s)[e * p.copies + j] = make_uint2(c0 | (c1 << 16), c2 | (c3 << 16));
        } else {
          const uint16_t v = (uint16_t)(e2m1_nibble(c0) | (e2m1_nibble(c1) << 4) | (e2m1_nibble(c2) << 8) | (e2m1_nibble(c3) << 12));
          for (int j = 0; j < p.copies; ++j) reinterpret_cast<uint16_t*>(lut_s)[e * p.copies + j] = v;
        }
      }
    }
    __syncthreads();
    if (!waited) { wait_before_output(p.beside); waited = true; }

    // entry offset of sub-index i inside the table
    uint32_t base[kSubs], mask[kSubs];
    int shift[kSubs];
#pragma unroll
    for (int i = 0; i < kSubs; ++i) {
      base[i] = (uint32_t)(a.split.base[i] / a.split.sub_dim);
      mask[i] = (1u << a.split.width[i]) - 1u;
      shift[i] = a.split.shift[i];
    }
    auto entry = [&](uint64_t code, int i) { return (base[i] + ((uint32_t)(code >> shift[i]) & mask[i])) * (uint32_t)p.copies + my; };
    auto lut16 = [&](uint64_t code, int i) { return (uint32_t)reinterpret_cast<const uint16_t*>(lut_s)[entry(code, i)]; };

    const int64_t units = (run_end - run) * p.n_sb;
    for (int64_t u = (int64_t)(tid >> 5) * 4 + which; u < units; u += kProdThreads / 8) {
      const uint32_t rr = (uint32_t)u / (uint32_t)p.n_sb;  // rows_per_cta * n_sb fits 32 bits
      const int s = (int)((uint32_t)u - rr * (uint32_t)p.n_sb);
      const int64_t r = run + rr;
      const uint8_t* sb = a.qw + r * a.row_stride + (int64_t)s * a.fmt.type_size;
      const uint8_t* plane = sb + 4 * k;
      const int64_t at = r * a.K + (int64_t)s * 256;
      if constexpr (kOut == kOutNvfp4) {
        // four neighbouring codewords, one 16-byte store
        const uint64_t ca = stream_bits(sb, (uint32_t)(sub * 4 * k), 2 * k), cb = stream_bits(sb, (uint32_t)(sub * 4 + 2) * k, 2 * k);
        const uint64_t m = (1ull << k) - 1ull;
        const uint64_t code[4] = {ca & m, ca >> k, cb & m, cb >> k};
        uint32_t w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) w[c] = lut16(code[c], 0) | (lut16(code[c], 1) << 16);
        uint32_t sc2, sc4 = 0;                             // the lane's two groups; atom `sub`'s four groups
        if (v2) {
          const uint8_t* t = comp_s + (uint32_t)plane[0] * 16u;
          const uint32_t n2 = plane[1 + sub];
          sc2 = t[n2 & 15u] | ((uint32_t)t[n2 >> 4] << 8);
          if (sub < 4) {
            const uint32_t n0 = plane[1 + 2 * sub], n1 = plane[2 + 2 * sub];
            sc4 = t[n0 & 15u] | ((uint32_t)t[n0 >> 4] << 8) | ((uint32_t)t[n1 & 15u] << 16) | ((uint32_t)t[n1 >> 4] << 24);
          }
        } else {
          sc2 = plane[2 * sub] | ((uint32_t)plane[2 * sub + 1] << 8);
          if (sub < 4)
            sc4 = plane[4 * sub] | ((uint32_t)plane[4 * sub + 1] << 8) | ((uint32_t)plane[4 * sub + 2] << 16) |
                  ((uint32_t)plane[4 * sub + 3] << 24);
        }
        if (fold_sign) {                                   // UE4M3 scale factors carry no sign
          if (sc2 & 0x80u) { w[0] ^= 0x88888888u; w[1] ^= 0x88888888u; }
          if (sc2 & 0x8000u) { w[2] ^= 0x88888888u; w[3] ^= 0x88888888u; }
          sc4 &= 0x7F7F7F7Fu;
        }
        reinterpret_cast<uint4*>(out0)[(at >> 5) + sub] = make_uint4(w[0], w[1], w[2], w[3]);
        if (sub < 4) {
          const int64_t off = (r / 128) * (512 * (int64_t)p.n_sb * 4) + ((int64_t)s * 4 + sub) * 512 + (r % 32) * 16 + ((r / 32) % 4) * 4;
          *reinterpret_cast<uint32_t*>(out_sf + off) = sc4;
        }
      } else if constexpr (kOut == kOutFp8) {
        // two codewords of each half of the superblock: two 16-byte stores
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t w[4];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint64_t code = stream_bits(sb, (uint32_t)(h * 16 + sub * 2 + c) * k, k);
            w[2 * c] = lut16(code, 0) | (lut16(code, 1) << 16);
            w[2 * c + 1] = lut16(code, 2) | (lut16(code, 3) << 16);
          }
          reinterpret_cast<uint4*>(out0)[(at >> 4) + h * 8 + sub] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      } else {
        // bf16(value * scale), the product taken in fp32: one codeword per 16-byte store
        const float rs = kOut == kOutFp8Bf16 ? __ldg(a.weight_scale + a.row0 + r) : 0.0f;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int v = h * 8 + sub;
          const uint64_t code = stream_bits(sb, (uint32_t)(v * k), k);
          uint32_t w[4];
          if constexpr (kOut == kOutFp8Bf16) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t e2 = lut16(code, i);
              w[i] = gb_pack_bf16x2(__fmul_rn(gb_e4m3_to_f32(e2 & 0xFFu), rs), __fmul_rn(gb_e4m3_to_f32(e2 >> 8), rs));
            }
          } else {
            const int g = v >> 1;
            float sc;
            if (v2) sc = __ldg(a.compose + (uint32_t)plane[0] * 16u + ((plane[1 + (g >> 1)] >> ((g & 1) * 4)) & 0xFu));
            else sc = gb_e4m3_to_f32(plane[g]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint2 e = reinterpret_cast<const uint2*>(lut_s)[entry(code, i)];
              w[2 * i] = gb_pack_bf16x2(__fmul_rn(__uint_as_float(e.x << 16), sc), __fmul_rn(__uint_as_float(e.x & 0xFFFF0000u), sc));
              w[2 * i + 1] = gb_pack_bf16x2(__fmul_rn(__uint_as_float(e.y << 16), sc), __fmul_rn(__uint_as_float(e.y & 0xFFFF0000u), sc));
            }
          }
          reinterpret_cast<uint4*>(out0)[(at >> 3) + v] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
    run = run_end;
    if (run < r_end) __syncthreads();                      // the next run rebuilds the tables
  }
  wait_at_end(p.beside);
}

// Whether the product kernel takes the weight: the mode it decodes, sub-tables that fit shared
// memory, 16-byte stores.
bool product_serves(const gb_weight* w, const void* out, int kout) {
  const gb_format& f = w->fmt;
  if (f.mode != GB_MODE_PRODUCT || f.n_sub != (f.grid == GB_GRID_FP8 ? 4 : 2) || ((uintptr_t)out & 15u) != 0) return false;
  if (f.grid == GB_GRID_FP4 && f.k_bits > 32) return false;
  const int64_t entry_bytes = kout == kOutBf16 ? 8 : 2;
  const int64_t entries = gb_codebook_elems(f) / (8 / f.n_sub);
  return entries * entry_bytes <= kProdLutCap;
}

template <int kOut>
int launch_expand_product(const gb_weight* w, int64_t row0, int64_t nrows, void* out0, void* out_sf, int fold_sign,
                          bool beside, void* stream) {
  ProdArgs p = {};
  p.beside = beside;
  int rc = make_expand_args(w, row0, nrows, &p.a);
  if (rc != GB_OK) return rc;
  p.a.qw = w->qw + row0 * w->row_stride;
  p.n_sb = (int)(w->K / 256);
  p.entries = (int)(gb_codebook_elems(w->fmt) / (8 / w->fmt.n_sub));
  const int entry_bytes = kOut == kOutBf16 ? 8 : 2;
  p.copies = 8;
  while (p.copies > 1 && p.entries * entry_bytes * p.copies > kProdLutCap) p.copies >>= 1;
  const int smem = p.entries * entry_bytes * p.copies + (kOut == kOutNvfp4 ? 4096 : 0);
  const int sms = gb_sm_count();
  if (sms <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  const int per_sm = smem * 4 <= 200 * 1024 ? 4 : smem * 3 <= 216 * 1024 ? 3 : 2;
  // one wave of CTAs over the rows, at least 64 superblocks each so that the tables pay
  int64_t rows_per = (nrows + (int64_t)sms * per_sm - 1) / ((int64_t)sms * per_sm);
  const int64_t least = (64 + p.n_sb - 1) / p.n_sb;
  if (rows_per < least) rows_per = least;
  GB_REQUIRE(rows_per * p.n_sb < (1ll << 31), "too many superblocks per CTA");
  p.rows_per_cta = rows_per;
  const unsigned blocks = (unsigned)((nrows + rows_per - 1) / rows_per);
  if (smem > 47 * 1024)                                   // the default limit counts the static words too
    GB_CUDA_OK(cudaFuncSetAttribute((const void*)expand_product_kernel<kOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GB_CUDA_OK(gb_launch(expand_product_kernel<kOut>, dim3(blocks), dim3(kProdThreads), (size_t)smem, (cudaStream_t)stream, p, out0,
                       (uint8_t*)out_sf, fold_sign));
  return GB_OK;
}
// ---- native NVFP4 view, fast ------------------------------------------------------------------
// The literal format (full mode, k = 8, E4M3 scales) and the two-tier product formats k = 12, 16, 20, 24
// whose superblocks start on 4-byte boundaries (the resident slots do).  Eight lanes take one (row,
// superblock): a lane fetches the one to three words that hold its four codewords, cuts them with
// constant shifts, looks every (sub-)index up as its finished E2M1 nibbles and stores sixteen bytes; two
// lanes join their group scales into the word of one 128 x 4 atom.  A CTA takes a run of rows and
// rebuilds its tables where the codebook changes.
//
// Two thirds of the issue slots went to index arithmetic (64-bit divisions, bit windows of any width,
// scale bytes fetched and looked up twice): 175 instructions per 32 lanes and step for the literal
// format, 297 for K20.  34816 x 5120: literal 41 -> 33 us, K20 73 -> 54 us (5120 x 17408: 24 -> 19, 44 -> 31);
// the bytes moved (133 and 178 MB) take 20 and 27 us.
constexpr int kNvThreads = 512;

template <int F>
struct NvFmt {
  static constexpr bool kLit = F == 8;
  static constexpr int kWords = kLit ? 1 : F <= 16 ? 2 : 3;              // words that hold 4 F bits from any 2-byte boundary
  static constexpr int kEntries = kLit ? 256 : 2 << (F / 2);
  static constexpr int kWide = kLit || F == 12 ? 2 : 1;                  // 16-bit halves of an entry
  static constexpr int kCopies = F <= 16 ? 32 : F == 20 ? 8 : 4;
  static constexpr int kShift = F == 20 ? 4 : F == 24 ? 3 : F == 16 ? 6 : 7;   // log2 of an entry's bytes, copies included
  static constexpr int kUnroll = kLit ? 4 : 2;                           // superblocks in flight per lane
  static constexpr int kLutBytes = kEntries << kShift;
  static constexpr int kSmem = kLutBytes + (kLit ? 0 : 4096);            // and the two-tier scale bytes
  static_assert(kCopies * kWide * 2 == 1 << kShift, "entry size");
};

struct NvArgs {
  const uint8_t* qw;           // first row
  int64_t row_stride, row0, nrows;
  int slot, n_sb;              // bytes from superblock to superblock
  int rows_per_cta;
  const uint16_t* codebook;
  const int32_t* cb_row_offset;
  const float* compose;
  uint4* out;
  uint8_t* sf;
  int fold_sign;
  bool beside;
};

template <int F>
__global__ void __launch_bounds__(kNvThreads, 3)
expand_nvfp4_kernel(const __grid_constant__ NvArgs a) {
  using T = NvFmt<F>;
  extern __shared__ uint8_t smem[];
  __shared__ int run_end_s;
  const int tid = threadIdx.x, lane = tid & 31, sub = lane & 7;
  uint8_t* comp_s = smem + T::kLutBytes;
  gb_pdl_launch_dependents();
  if (!T::kLit) {
    if (((uintptr_t)a.compose & 15u) == 0) {               // (scales are no negative numbers: the conversion saturates at 448)
#pragma unroll
      for (int i = tid; i < 1024; i += kNvThreads) {
        const float4 c = __ldg(reinterpret_cast<const float4*>(a.compose) + i);
        reinterpret_cast<uint32_t*>(comp_s)[i] = gb_cvt_e4m3x2(fminf(c.x, 448.0f), fminf(c.y, 448.0f)) | gb_cvt_e4m3x2(fminf(c.z, 448.0f), fminf(c.w, 448.0f)) << 16;
      }
    } else {
#pragma unroll 1
      for (int i = tid; i < 4096; i += kNvThreads) comp_s[i] = (uint8_t)gb_f32_to_e4m3(fminf(__ldg(a.compose + i), 448.0f));
    }
  }

  const int64_t r_begin = (int64_t)blockIdx.x * a.rows_per_cta;
  const int64_t r_end = r_begin + a.rows_per_cta < a.nrows ? r_begin + a.rows_per_cta : a.nrows;
  const uint8_t* lut = smem + (lane & (T::kCopies - 1)) * T::kWide * 2;
  const uint32_t n_sb = (uint32_t)a.n_sb;
  const uint32_t dr = (kNvThreads / 32) / n_sb, ds = (kNvThreads / 32) % n_sb;   // a step of the CTA's warps
  const int code_at = T::kLit ? 4 * sub : (sub * F / 2) & ~3;
  const int cut = (sub * F / 2 & 2) * 8;                   // odd lanes of F = 12 and 20 start in mid-word

  for (int64_t run = r_begin; run < r_end;) {
    int64_t cb_base = 0, run_end = r_end;
    if (a.cb_row_offset) {                                 // rows [run, run_end) use one codebook block
      cb_base = a.cb_row_offset[a.row0 + run];
      __syncthreads();
      if (tid == 0) run_end_s = (int)(r_end - run);
      __syncthreads();
      for (int64_t r = run + tid; r < r_end; r += kNvThreads)
        if (a.cb_row_offset[a.row0 + r] != (int32_t)cb_base) { atomicMin(&run_end_s, (int)(r - run)); break; }
      __syncthreads();
      run_end = run + run_end_s;
    }
    // an entry is converted once; its copies go out as 8 or 16 bytes a store, rotated by lane over the banks
#pragma unroll 4
    for (int e = tid; e < T::kEntries; e += kNvThreads) {
      const uint16_t* c = a.codebook + cb_base + (int64_t)e * (T::kLit ? 8 : 4);
      uint32_t nib = 0;
      if (((uintptr_t)c & 7u) == 0) {
#pragma unroll
        for (int j = 0; j < (T::kLit ? 2 : 1); ++j) {
          const uint2 v = __ldg(reinterpret_cast<const uint2*>(c) + j);
          nib |= (e2m1_pair(v.x) | e2m1_pair(v.y) << 8) << (16 * j);
        }
      } else {
#pragma unroll 1
        for (int j = 0; j < (T::kLit ? 8 : 4); ++j) nib |= e2m1_nibble(__ldg(c + j)) << (4 * j);
      }
      if (T::kWide == 1) nib |= nib << 16;
      constexpr int kVec = 1 << T::kShift >= 16 ? (1 << T::kShift) / 16 : 1;
      if (T::kShift == 3) reinterpret_cast<uint2*>(smem)[e] = make_uint2(nib, nib);
#pragma unroll
      for (int q = 0; q < (T::kShift == 3 ? 0 : kVec); ++q)
        reinterpret_cast<uint4*>(smem)[e * kVec + ((q + lane) & (kVec - 1))] = make_uint4(nib, nib, nib, nib);
    }
    __syncthreads();
    if (run == r_begin) wait_before_output(a.beside);

    // a warp's unit: one superblock of four neighbouring rows, whose scale words lie 16 bytes apart
    const uint32_t rows = (uint32_t)(run_end - run), units = (rows + 3) / 4 * n_sb;
    uint32_t u = (uint32_t)(tid >> 5);
    uint32_t rr = u / n_sb, s = u - rr * n_sb;
    for (; u < units; u += T::kUnroll * (kNvThreads / 32)) {
      uint32_t w[T::kUnroll][T::kWords], sc[T::kUnroll], sup[T::kUnroll], row[T::kUnroll], col[T::kUnroll];
#pragma unroll
      for (int i = 0; i < T::kUnroll; ++i) {
        row[i] = rr * 4 + (uint32_t)(lane >> 3);
        col[i] = s;
        const uint8_t* sb = a.qw + (run + min(row[i], rows - 1)) * a.row_stride + (int64_t)col[i] * a.slot;
#pragma unroll
        for (int q = 0; q < T::kWords; ++q) w[i][q] = __ldg(reinterpret_cast<const uint32_t*>(sb + code_at) + q);
        if (T::kLit) sc[i] = __ldg(reinterpret_cast<const uint16_t*>(sb + 32) + sub);     // groups 2 sub, 2 sub + 1
        else { sup[i] = __ldg(sb + 4 * F); sc[i] = __ldg(sb + 4 * F + 1 + sub); }
        rr += dr;
        s += ds;
        if (s >= n_sb) { s -= n_sb; ++rr; }
      }
#pragma unroll
      for (int i = 0; i < T::kUnroll; ++i) {
        uint32_t v[4];
        if (T::kLit) {
          v[0] = *reinterpret_cast<const uint32_t*>(lut + ((w[i][0] & 0xFFu) << 7));
          v[1] = *reinterpret_cast<const uint32_t*>(lut + ((w[i][0] >> 1) & 0x7F80u));
          v[2] = *reinterpret_cast<const uint32_t*>(lut + ((w[i][0] >> 9) & 0x7F80u));
          v[3] = *reinterpret_cast<const uint32_t*>(lut + ((w[i][0] >> 17) & 0x7F80u));
        } else {
          uint32_t b[3] = {w[i][0], w[i][1], T::kWords == 3 ? w[i][T::kWords - 1] : 0u};
          if (F == 12 || F == 20) {
            b[0] = __funnelshift_r(b[0], b[1], cut);
            b[1] = __funnelshift_r(b[1], b[2], cut);
            b[2] >>= cut;
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t half[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              constexpr uint32_t kMask = ((1u << (F / 2)) - 1u) << T::kShift;
              const int bit = c * F + h * (F / 2), wd = bit >> 5, at = bit & 31;
              uint32_t x;                                  // the sub-index shifted to its entry's byte offset
              if (at + F / 2 > 32) x = __funnelshift_r(b[wd], b[wd + 1 < 3 ? wd + 1 : 2], at) << T::kShift;
              else x = at >= T::kShift ? b[wd] >> (at - T::kShift) : b[wd] << (T::kShift - at);
              const uint8_t* at_p = lut + (h * T::kLutBytes / 2) + (x & kMask);
              half[h] = T::kWide == 2 ? *reinterpret_cast<const uint32_t*>(at_p) : *reinterpret_cast<const uint16_t*>(at_p);
            }
            v[c] = half[0] | (half[1] << 16);
          }
        }
        uint32_t sc2 = sc[i];
        if (!T::kLit) {
          const uint8_t* t = comp_s + sup[i] * 16u;
          sc2 = t[sc[i] & 15u] | ((uint32_t)t[sc[i] >> 4] << 8);
        }
        if (a.fold_sign) {                                 // UE4M3 scale factors carry no sign
          if (sc2 & 0x80u) { v[0] ^= 0x88888888u; v[1] ^= 0x88888888u; }
          if (sc2 & 0x8000u) { v[2] ^= 0x88888888u; v[3] ^= 0x88888888u; }
          sc2 &= 0x7F7Fu;
        }
        const uint32_t sc4 = sc2 | (__shfl_down_sync(0xffffffffu, sc2, 1) << 16);
        if (row[i] < rows) {
          const int64_t r = run + row[i];
          a.out[(r * n_sb + col[i]) * 8 + sub] = make_uint4(v[0], v[1], v[2], v[3]);
          if ((sub & 1) == 0)
            *reinterpret_cast<uint32_t*>(a.sf + (r >> 7) * (int64_t)(2048u * n_sb) + (int64_t)(col[i] * 2048u) +
                                         (uint32_t)(sub * 256) + ((uint32_t)r & 31u) * 16u + (((uint32_t)r >> 5) & 3u) * 4u) = sc4;
        }
      }
    }
    run = run_end;
    if (run < r_end) __syncthreads();                      // the next run rebuilds the tables
  }
  wait_at_end(a.beside);
}

// GB_EUNSUPPORTED: the weight is not the kernel's.
int launch_expand_nvfp4(const gb_weight* w, int64_t row0, int64_t nrows, void* out, void* sf, int fold_sign, bool beside, void* stream) {
  const gb_format& f = w->fmt;
  const bool lit = f.mode == GB_MODE_FULL && f.k_bits == 8 && f.scale_coding == GB_SCALE_V1;
  const bool prod = f.mode == GB_MODE_PRODUCT && f.n_sub == 2 && f.scale_coding == GB_SCALE_V2 &&
                    (f.k_bits == 12 || f.k_bits == 16 || f.k_bits == 20 || f.k_bits == 24);
  if (!(lit || prod) || f.type_size % 4 != 0 || w->row_stride % 4 != 0 || ((uintptr_t)w->qw & 3u) != 0 ||
      ((uintptr_t)out & 15u) != 0 || ((uintptr_t)sf & 3u) != 0 || ((uintptr_t)w->codebook & 1u) != 0)
    return GB_EUNSUPPORTED;
  ExpandArgs e;
  if (lit && nrows == 0 && row0 >= 0 && row0 <= w->rows) return GB_OK;
  int rc = make_expand_args(w, row0, nrows, &e);
  if (rc != GB_OK) return rc;
  GB_REQUIRE(out != nullptr, "null output");
  if (prod && (e.split.width[0] != f.k_bits / 2 || e.split.width[1] != f.k_bits / 2 || e.split.shift[0] != 0 ||
               e.split.shift[1] != f.k_bits / 2 || e.split.base[0] != 0 || e.split.base[1] != 4 << (f.k_bits / 2)))
    return GB_EUNSUPPORTED;
  NvArgs a = {};
  a.qw = w->qw + row0 * w->row_stride;
  a.row_stride = w->row_stride; a.row0 = row0; a.nrows = nrows;
  a.slot = f.type_size;
  a.n_sb = (int)(w->K / 256);
  a.codebook = (const uint16_t*)w->codebook;
  a.cb_row_offset = w->cb_row_offset;
  a.compose = w->compose;
  a.out = (uint4*)out; a.sf = (uint8_t*)sf; a.fold_sign = fold_sign; a.beside = beside;
  // one wave of three CTAs per SM over the rows, at least 128 superblocks each so that the tables pay
  const int64_t ctas = (int64_t)gb_sm_count() * 3;
  if (ctas <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  int64_t rows_per = (nrows + ctas - 1) / ctas;
  const int64_t least = (128 + a.n_sb - 1) / a.n_sb;
  if (rows_per < least) rows_per = least;
  rows_per = (rows_per + 3) / 4 * 4;
  GB_REQUIRE(rows_per * a.n_sb < (1ll << 30), "too many superblocks per CTA");
  a.rows_per_cta = (int)rows_per;
  const unsigned blocks = (unsigned)((nrows + rows_per - 1) / rows_per);
#define GB_EXPAND_NVFP4(F)                                                                                              \
  GB_CUDA_OK(cudaFuncSetAttribute((const void*)expand_nvfp4_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, NvFmt<F>::kSmem)); \
  GB_CUDA_OK(gb_launch(expand_nvfp4_kernel<F>, dim3(blocks), dim3(kNvThreads), NvFmt<F>::kSmem, (cudaStream_t)stream, a))
  switch (f.k_bits) {
    case 8: GB_EXPAND_NVFP4(8); break;
    case 12: GB_EXPAND_NVFP4(12); break;
    case 16: GB_EXPAND_NVFP4(16); break;
    case 20: GB_EXPAND_NVFP4(20); break;
    default: GB_EXPAND_NVFP4(24); break;
  }
#undef GB_EXPAND_NVFP4
  return GB_OK;
}

}  // namespace

static int expand_fp8(const gb_weight* w, int64_t row0, int64_t nrows, void* out, bool beside, void* stream) {
  GB_REQUIRE(w && w->fmt.grid == GB_GRID_FP8, "gb_expand_fp8 wants an fp8-grid weight");
  const gb_format& f = w->fmt;
  if (f.mode == GB_MODE_PRODUCT && ((f.k_bits == 32 && f.n_sub == 4 && f.type_size == 128) ||
                                    (f.k_bits == 16 && f.n_sub == 2 && f.type_size == 64)) &&
      ((uintptr_t)w->codebook & 3u) == 0 && ((uintptr_t)out & 15u) == 0 && ((uintptr_t)w->qw & 15u) == 0 && w->row_stride % 16 == 0) {
    int rc = gb_check_weight(w);
    if (rc != GB_OK) return rc;
    GB_REQUIRE(out != nullptr, "null output pointer");
    GB_REQUIRE(row0 >= 0 && nrows >= 0 && row0 + nrows <= w->rows, "rows [%lld, %lld) outside [0, %lld)",
               (long long)row0, (long long)(row0 + nrows), (long long)w->rows);
    if (nrows == 0) return GB_OK;
    return launch_expand_fp8_fast(w, row0, nrows, out, beside, stream);
  }
  if (product_serves(w, out, kOutFp8)) return launch_expand_product<kOutFp8>(w, row0, nrows, out, nullptr, 0, beside, stream);
  return launch_expand<kOutFp8>(w, row0, nrows, out, nullptr, 0, stream);
}

static int expand_nvfp4(const gb_weight* w, int64_t row0, int64_t nrows, void* out_packed, void* out_sf, int sf_swizzled, bool beside,
                        void* stream) {
  GB_REQUIRE(w && w->fmt.grid == GB_GRID_FP4, "gb_expand_fp4_nvfp4 wants an fp4-grid weight");
  GB_REQUIRE(out_sf != nullptr, "null scale-factor output");
  if (sf_swizzled != 0) {
    const int rc = launch_expand_nvfp4(w, row0, nrows, out_packed, out_sf, sf_swizzled == 2, beside, stream);
    if (rc != GB_EUNSUPPORTED) return rc;
  }
  if (sf_swizzled != 0 && ((uintptr_t)out_sf & 3u) == 0 && product_serves(w, out_packed, kOutNvfp4))
    return launch_expand_product<kOutNvfp4>(w, row0, nrows, out_packed, out_sf, sf_swizzled == 2, beside, stream);
  return launch_expand<kOutNvfp4>(w, row0, nrows, out_packed, out_sf, sf_swizzled, stream);
}

extern "C" {

int gb_expand_fp8(const gb_weight* w, int64_t row0, int64_t nrows, void* out, void* stream) {
  return expand_fp8(w, row0, nrows, out, false, stream);
}

int gb_expand_fp8_beside(const gb_weight* w, int64_t row0, int64_t nrows, void* out, void* stream) {
  return expand_fp8(w, row0, nrows, out, true, stream);
}

int gb_expand_fp8_bf16(const gb_weight* w, int64_t row0, int64_t nrows, void* out, void* stream) {
  GB_REQUIRE(w && w->fmt.grid == GB_GRID_FP8 && w->weight_scale, "gb_expand_fp8_bf16 wants an fp8-grid weight with its row scales");
  if (product_serves(w, out, kOutFp8Bf16)) return launch_expand_product<kOutFp8Bf16>(w, row0, nrows, out, nullptr, 0, false, stream);
  return launch_expand<kOutFp8Bf16>(w, row0, nrows, out, nullptr, 0, stream);
}

int gb_expand_fp4_bf16(const gb_weight* w, int64_t row0, int64_t nrows, void* out, void* stream) {
  GB_REQUIRE(w && w->fmt.grid == GB_GRID_FP4, "gb_expand_fp4_bf16 wants an fp4-grid weight");
  if (product_serves(w, out, kOutBf16)) return launch_expand_product<kOutBf16>(w, row0, nrows, out, nullptr, 0, false, stream);
  return launch_expand<kOutBf16>(w, row0, nrows, out, nullptr, 0, stream);
}

int gb_expand_fp4_nvfp4(const gb_weight* w, int64_t row0, int64_t nrows, void* out_packed,
                        void* out_sf, int sf_swizzled, void* stream) {
  return expand_nvfp4(w, row0, nrows, out_packed, out_sf, sf_swizzled, false, stream);
}

int gb_expand_fp4_nvfp4_beside(const gb_weight* w, int64_t row0, int64_t nrows, void* out_packed, void* out_sf, int sf_swizzled,
                               void* stream) {
  return expand_nvfp4(w, row0, nrows, out_packed, out_sf, sf_swizzled, true, stream);
}

}  // extern "C"
