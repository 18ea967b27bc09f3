// Decode-batch linear of the fp4 grid on the block-scaled FP4 tensor cores, the decode contract kept:
// y[M, N] = bucket(x)[M, K] . W^T for 1 <= M <= 64 rows per pass, dense and per expert.
//
// A weight of the fp4 grid IS E2M1 x (E4M3 group scale), so the packed rows only have to be turned
// into the MMA's own operand format: one 32-bit word of nibbles per codeword, one scale byte per group
// (the kernel of gb_gemv_umma.cu multiplies every weight out to bf16 first: four times the
// operand bytes, sixteen MMAs per superblock instead of four).  What does not fit the format is the
// ACTIVATION: the contract's value is bf16(q * s) with q on the E2M1 grid and a full fp32 group scale
// s.  It is split exactly into three E2M1 x UE4M3 terms, i.e. three columns of the N side per row:
//   * the eight magnitudes of q share two significands: m1 = bf16(s) (q = 0.5, 1, 2, 4) and
//     bf16(1.5 s) (q = 1.5, 3, 6), each times a power of two;
//   * hi  : q x (m1 rounded down to four significant bits),
//   * lo  : q x (the other four bits of m1), its own power of two on the column,
//   * dlt : bf16(1.5 s) - 1.5 m1 is n half-ulps of m1 with |n| <= 3, so for q = 1.5, 3, 6 the missing
//           part is (n q / 3) half-ulps: again an E2M1 value times a power of two.
// Every term is normalised per row by a power of two that puts the row's largest m1 into [128, 256).
// UE4M3 is normal down to 2^-6, so the split is exact for groups within 2^13 of the row's largest.  A row that
// spans more is normalised around its mean exponent instead; what is still out of range - an outlier channel,
// or groups far below the rest - is left out of the operand and added while the sums are read out
// (gb_left_out).  No group may be dropped: a weight row may be zero wherever the activations are large, and
// its result is then the small groups' alone.
//
// Up to sixteen rows the three terms are columns of one MMA (N <= 48).  Past them two MMAs share the
// codes of q: N = 2 R with the scale factors [hi | dlt] over the code rows [q | e], N = R with lo over
// [q], so a row costs two code rows of shared memory and L2 traffic instead of three.
//
// Work split as in gb_gemv_umma.cu: a CTA owns 128 weight rows (the M side) and a K slice; one warp
// streams the packed rows (tiled TMA), one the operand of the activations (one bulk copy per superblock:
// the rows kernel below writes it swizzled, scale factors in front), two issue MMAs, four move the activations'
// scale factors to tensor memory, sixteen decode.  A UNIT is one superblock of K (256 weights): unit u is
// decoded by warpgroup u mod 4 into operand buffer u mod 4 of TENSOR MEMORY (32 columns of nibbles, 16 of scale
// factors) and multiplied by four MMAs of K = 64 (or eight).
// Bound by the instructions of the decoders, who wait little: a unit of the literal format takes 570 clocks (HBM
// 260), of K16 660 (430); without loads, lookups and MMAs it would still take 430.  What was tried for the scale factors of
// the activations: by the decoders (320 of the 2300 clocks a unit then took its warpgroup); tcgen05.cp from two to four
// warps (shares the tensor pipe with the MMAs: eight copies and eight MMAs of a wide unit 900 clocks).
// us, before those warps, the uniform issue below, rings of four or eight units for every format and the present
// stores / now, launches back to back, rows kernel included: 34816 x 5120, 16 rows literal 21.5 / 18.6, K12 26.4 / 22.7, K16 26.6 / 21.9,
// K20 40.9 / 26.2; 64 rows literal 29.7 / 24.5, 48 rows K16 32.9 / 26.6; 5120 x 17408, 16 rows K16 20.6 / 17.3.
//
// A layer with few 128-row tiles is sliced along K over a thread-block cluster: every CTA of the
// cluster pushes its fp32 sums into the shared memory of the CTA that owns the activation row, which
// adds them in slice order - no partial sums in HBM and no second launch.
#include "gb_common.cuh"

#include <cuda.h>
#include <type_traits>

namespace {

constexpr int kBM = 128;
constexpr int kDecWarps = 16;
constexpr int kCtlWarps = 8;                              // packed rows, activations, two MMA issuers, four for the scale factors
constexpr int kThreads = 32 * (kCtlWarps + kDecWarps);
constexpr int kMaxRows = 64;                              // activation rows per pass (three columns each)
constexpr int kMaxRaw = 8, kMaxX = 8;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kDynBase = 0x400u;                     // dynamic shared memory starts here (checked); in a
                                                          // cluster the CTA's rank sits in the address's top byte
constexpr uint32_t kSmemMax = 227 * 1024;
constexpr uint32_t kSmemEnd = kDynBase + kSmemMax;
constexpr uint32_t kLut = 0x800u;                         // shared-window address of the lookup tables, behind the barriers
constexpr int kMaxRoles = GB_MAX_ROLES;                     // and no fewer than matrices, which count as roles
constexpr int kMaxSlices = 8;

enum { kLit = 8 };                                        // other formats: the product format's k

// Packed superblocks as they sit in memory and the lookup tables of a format.
template <int F> struct Fmt {                             // two-tier product format, k = F
  static constexpr int kW0 = (F + 1) / 2, kW1 = F / 2;    // sub-index widths
  static constexpr int kSb = (4 * F + 9 + 15) / 16 * 16;  // slot of a superblock
  static constexpr int kSbPerStage = 1;
  static constexpr int kEntries = 1 << kW0;
  static constexpr int kCopies = kEntries <= 512 ? 32 : 16 * 1024 / kEntries;
  static constexpr uint32_t kStride = kCopies * 4;        // bytes between entries: both sub-tables in one word
  static constexpr uint32_t kLutBytes = kEntries * kStride;
  static constexpr uint32_t kScaleTab = 4096;             // E4M3 byte of every (super, sub) pair
};
template <> struct Fmt<kLit> {
  static constexpr int kSb = 48, kSbPerStage = 2;
  static constexpr uint32_t kStride = 256;                // a code dropped into byte 1 is the entry's offset
  static constexpr uint32_t kLutBytes = 256 * 256, kScaleTab = 0;
};
template <int F> struct Geo {
  static constexpr int kPitch0 = Fmt<F>::kSbPerStage * Fmt<F>::kSb;
  static constexpr int kPitch = kPitch0 + ((kPitch0 / 16) % 2 ? 32 : 16);   // an odd number of 16-byte units
  static constexpr int kBoxBytes = kBM * kPitch;
  static_assert(kPitch <= 256 && (kPitch / 16) % 2 == 1, "row pitch");
};

constexpr int kMaxMatrices = 4;
// A matrix of the launch: several that read the same activation rows go out together.
struct Matrix {
  const uint8_t* qw;         // packed rows, once more for groups left out
  int64_t row_stride, N;
  const void* codebook;      // bf16 flat
  const float* compose;
  float global_scale;
  uint16_t* y;
};
struct Maps { CUtensorMap m[kMaxMatrices]; };
struct Role { int mat, row0, rows, tile0; int64_t cb; };   // rows of a matrix that share a codebook; first tile; element offset

struct Fp4Params {
  Matrix mat[kMaxMatrices];  // grouped: the first is the stack, N the rows of an expert
  int64_t K;
  int M;                     // dense: activation rows
  int n_sb, units;           // superblocks per row / per K slice (the last slice may have fewer)
  int slices;                // = cluster size along y
  int pass_rows;             // most rows per pass (dense: M)
  int x_stages, raw_stages;  // ring depths: 4 or 8, 2 or 4
  uint32_t x_off, raw_off, sf_off, red_off;
  const uint8_t* xop;        // activation operand: [tile][superblock][scale factors | codes]
  int64_t x_unit;            // bytes of one superblock of it
  const float* x_scale;      // [tile][scale_pitch(pass_rows)] power of two of every row; low bits: where groups are left out
  const float* tail;         // [tile][pass_rows][K / 16] scales of the groups left out, of the rows that have any
  int* status;
  int n_roles, n_tiles;
  Role role[kMaxRoles];
  const int32_t* seg;        // grouped: [E + 1]
  const int32_t* row_map;
  int tiles_n;
  int E;
  uint32_t seg_off;          // their copy in shared memory, 0: no room
};

// Columns.  Narrow (up to 16 rows per pass): term t of row m in column 12 (m / 4) + 4 t + m % 4, so that the
// twelve columns of four rows are read out together; one MMA of N = 3 R rounded up to 16.  Wide: R code
// rows of q, then R of the correction, scale factors [hi | dlt] and [lo].  R = rows rounded up to 8
// (narrow) or 16.
constexpr int kNarrowRows = 16;
__host__ __device__ constexpr bool is_wide(int pass_rows) { return pass_rows > kNarrowRows; }
// Distance between the row scales of two tiles: they are read four and eight at a time.
__host__ __device__ constexpr int scale_pitch(int pass_rows) { return (pass_rows + 7) / 8 * 8; }
__host__ __device__ constexpr int term_rows(bool wide, int rows) { return wide ? (rows + 15) / 16 * 16 : (rows + 7) / 8 * 8; }
__host__ __device__ constexpr int narrow_col(int t, int m) { return 12 * (m >> 2) + 4 * t + (m & 3); }
__host__ __device__ constexpr int mma_cols(bool wide, int rows) {
  return wide ? 2 * term_rows(true, rows) : (3 * term_rows(false, rows) + 15) / 16 * 16;
}
// Bytes in front of the codes of a unit: scale-factor atoms of 128 columns (wide: two sets).
__host__ __device__ constexpr int sf_bytes(bool wide) { return wide ? 4096 : 2048; }
__host__ __device__ constexpr int unit_bytes(bool wide, int rows) { return sf_bytes(wide) + mma_cols(wide, rows) * 128; }
// Offset of group gi of code row n behind them (128-byte swizzle).
__host__ __device__ constexpr int code_at(int n, int gi) { return (n >> 3) * 1024 + (n & 7) * 128 + (((gi >> 1) ^ (n & 7)) << 4) + (gi & 1) * 8; }

// ---- PTX ---------------------------------------------------------------------------------------
GB_DEVINL void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
GB_DEVINL void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
GB_DEVINL void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
GB_DEVINL bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// Acquire at cluster scope: the arrivals come from other CTAs of the cluster.
GB_DEVINL bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// A bounded wait that remembers a timeout for the rest of the CTA: later waits return at once.  The
// spin is kept out of line: a dozen inlined copies crowd the instruction cache.
template <bool kCluster>
__device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  uint64_t t0 = 0;
  for (uint32_t spin = 0; !*abort_flag; ++spin) {
    if (kCluster ? mbar_try_cluster(bar, parity) : mbar_try(bar, parity)) return;
    if ((spin & 255u) == 255u) {
      const uint64_t now = gb_globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > 2000000000ull) { *abort_flag = 1; atomicExch(status, code); }
    }
  }
}
template <bool kCluster = false>
GB_DEVINL void wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (!(kCluster ? mbar_try_cluster(bar, parity) : mbar_try(bar, parity))) wait_slow<kCluster>(bar, parity, abort_flag, status, code);
}
// The same for a whole warp that goes on together; false: given up.
GB_DEVINL bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  wait_slow<false>(bar, parity, abort_flag, status, code);
  return !__any_sync(0xffffffffu, *abort_flag != 0);
}
GB_DEVINL void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
GB_DEVINL void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
GB_DEVINL bool mbar_test(uint32_t bar, uint32_t parity) {   // never suspends: for a look ahead of the wait
  uint32_t done;
  asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
GB_DEVINL uint64_t desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D[tmem] (+)= (A SFA)[tmem] . (B SFB)[smem]: A holds 128 rows (lanes) x 64 E2M1 in 8 columns.
GB_DEVINL void umma_fp4_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, bool acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], [%1], %2, %3, [%5], [%6], p;\n}\n"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"((uint32_t)acc), "r"(sfa), "r"(sfb) : "memory");
}
GB_DEVINL void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
GB_DEVINL void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
GB_DEVINL void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
GB_DEVINL void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}
GB_DEVINL void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                 "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr));
}
GB_DEVINL uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
GB_DEVINL void sts128(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
template <uint32_t kImm>
GB_DEVINL uint32_t lds_imm(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kImm));
  return v;
}
template <uint32_t kImm>
GB_DEVINL uint32_t lds_imm16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1+%2];" : "=h"(v) : "r"(a), "n"(kImm));
  return v;
}

// Four E2M1 nibbles of four bf16 codebook values.
GB_DEVINL uint32_t nib4(uint2 w) {
  uint32_t r = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float v = gb_bf16_bits_to_f32(((j < 2 ? w.x : w.y) >> (16 * (j & 1))) & 0xFFFFu), m = fabsf(v);
    const uint32_t c = m < 2.0f ? (uint32_t)(m * 2.0f) : (m < 4.0f ? (uint32_t)m + 2u : (m < 6.0f ? 6u : 7u));
    r |= (c | (v < 0.0f ? 8u : 0u)) << (4 * j);
  }
  return r;
}

// Sub-indices that are whole bytes (k = 16): a byte permutation drops one into byte 1 of a lookup's address, one
// instruction instead of two, and the second sub-table's entries are kept in place (bits 16 to 31).  Their
// tables take 256 bytes an entry, which the wide passes have no room for.  34816 x 5120, 16 rows: 22.9 -> 22.5 us.
template <int F, bool kWide> constexpr bool kByteCodes = F == 16 && !kWide;

// Lookup tables of one codebook, built by the 512 decoder threads; the order of a thread's stores rotates
// with it, since the entries of neighbouring threads start in the same bank.
template <int F, bool kWide>
GB_DEVINL void build_lut(const uint16_t* cb, int d, uint32_t lut) {
  if constexpr (F == kLit) {
    const int e = d & 255, half = d >> 8;
    const uint4 q = *reinterpret_cast<const uint4*>(cb + e * 8);
    const uint32_t w = nib4(make_uint2(q.x, q.y)) | (nib4(make_uint2(q.z, q.w)) << 16);
#pragma unroll
    for (int j = 0; j < 4; ++j) sts128(lut + (uint32_t)e * 256u + (uint32_t)((half * 4 + j + d) & 7) * 16u, make_uint4(w, w, w, w));
  } else if constexpr (kByteCodes<F, kWide>) {
    const int e = d & 255, second = d >> 8;
    const uint32_t w = nib4(reinterpret_cast<const uint2*>(cb)[d]) << (16 * second);
#pragma unroll
    for (int j = 0; j < 8; ++j) sts128(lut + (uint32_t)e * 256u + (uint32_t)second * 128u + (uint32_t)((j + d) & 7) * 16u, make_uint4(w, w, w, w));
  } else {
    using T = Fmt<F>;
    const uint2* t0 = reinterpret_cast<const uint2*>(cb);
    const uint2* t1 = t0 + T::kEntries;
    for (int e = d; e < T::kEntries; e += 32 * kDecWarps) {
      uint32_t w = nib4(t0[e]);
      if (e < (1 << T::kW1)) w |= nib4(t1[e]) << 16;
#pragma unroll
      for (int j = 0; j < T::kCopies / 4; ++j)
        sts128(lut + (uint32_t)e * T::kStride + (uint32_t)((j + e / (128 / T::kStride)) & (T::kCopies / 4 - 1)) * 16u, make_uint4(w, w, w, w));
    }
  }
}

// Byte offset of the sub-index at bits [bit, bit + width) of the code words, times the entry stride.
template <int F, int kWidth>
GB_DEVINL uint32_t entry_offset(const uint32_t* w, int bit, uint32_t lane4) {
  constexpr int kShift = F == kLit ? 8 : (Fmt<F>::kStride == 128 ? 7 : Fmt<F>::kStride == 64 ? 6 : 4);
  static_assert(F == kLit || Fmt<F>::kStride == 1 << kShift, "entry stride");
  constexpr uint32_t kMask = ((1u << kWidth) - 1u) << kShift;
  const int i = bit >> 5, s = bit & 31;
  uint32_t x;
  if (s + kWidth <= 32) x = s >= kShift ? w[i] >> (s - kShift) : w[i] << (kShift - s);
  else x = s >= kShift ? __funnelshift_r(w[i], w[i + 1], s - kShift) : 0u;
  return (x & kMask) | lane4;
}

// Eight weights of codeword c as nibbles.
template <int F, bool kWide>
GB_DEVINL uint32_t codeword(const uint32_t* w, int c, uint32_t lane4) {
  if constexpr (F == kLit) {
    // [lane4's byte 0, code, lane4's bytes 2 and 3]: lane offset, entry, the window's rank byte
    const uint32_t a = c % 4 == 0 ? __byte_perm(w[c / 4], lane4, 0x7604) : c % 4 == 1 ? __byte_perm(w[c / 4], lane4, 0x7614)
                     : c % 4 == 2 ? __byte_perm(w[c / 4], lane4, 0x7624) : __byte_perm(w[c / 4], lane4, 0x7634);
    return lds_imm<kLut>(a);
  } else if constexpr (kByteCodes<F, kWide>) {
    const uint32_t a0 = c % 2 == 0 ? __byte_perm(w[c / 2], lane4, 0x7604) : __byte_perm(w[c / 2], lane4, 0x7624);
    const uint32_t a1 = c % 2 == 0 ? __byte_perm(w[c / 2], lane4, 0x7614) : __byte_perm(w[c / 2], lane4, 0x7634);
    return lds_imm<kLut>(a0) | lds_imm<kLut + 128>(a1);
  } else {
    using T = Fmt<F>;
    const uint32_t a0 = entry_offset<F, T::kW0>(w, c * F, lane4), a1 = entry_offset<F, T::kW1>(w, c * F + T::kW0, lane4);
    return lds_imm16<kLut>(a0) | (lds_imm16<kLut + 2>(a1) << 16);
  }
}

// Two-tier scales: four E4M3 bytes of four nibble codes (low 16 bits of c) from the sixteen bytes t.
GB_DEVINL uint32_t four_scales(uint4 t, uint32_t c) {
  const uint32_t sel = c & 0x7777u;
  const uint32_t lo = __byte_perm(t.x, t.y, sel), hi = __byte_perm(t.z, t.w, sel);
  uint32_t m;                                              // 0xFF where the code is 8..15 (sign replication), else 0x80
  asm("prmt.b32 %0, %1, %1, %2;" : "=r"(m) : "r"(0x80808080u), "r"(c & 0x8888u));
  return lo ^ ((lo ^ hi) & m & 0x7F7F7F7Fu);
}

// The E4M3 byte of every (super, sub) pair of the two-tier formats.
template <int F>
GB_DEVINL void build_scale_tab(const float* compose, int d, uint32_t scale_tab) {
  if constexpr (F != kLit) {
    for (int i = d * 4; i < 4096; i += 4 * 32 * kDecWarps) {
      uint32_t w = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) w |= gb_f32_to_e4m3(fminf(__ldg(compose + i + j), 448.0f)) << (8 * j);
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(scale_tab + (uint32_t)i), "r"(w) : "memory");
    }
  }
}

// Group g of a packed row (sixteen bf16 codebook values and their scale), from global memory: the tables in shared
// memory may already be another role's.
struct RowGroup { uint2 v[4]; float scale; };
template <int F>
GB_DEVINL RowGroup row_group(const uint8_t* row, const uint16_t* cb, const float* compose, int g) {
  const uint8_t* sb = row + (g >> 4) * Fmt<F>::kSb;
  const int gi = g & 15;
  RowGroup r;
  if constexpr (F == kLit) {
    r.scale = gb_e4m3_to_f32(sb[32 + gi]);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const uint4 e = *reinterpret_cast<const uint4*>(cb + 8 * sb[2 * gi + c]);
      r.v[2 * c] = make_uint2(e.x, e.y);
      r.v[2 * c + 1] = make_uint2(e.z, e.w);
    }
  } else {
    using T = Fmt<F>;
    const uint32_t* words = reinterpret_cast<const uint32_t*>(sb);
    r.scale = fminf(compose[sb[4 * F] * 16 + (sb[4 * F + 1 + (gi >> 1)] >> (4 * (gi & 1)) & 0xF)], 448.0f);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int bit = (2 * gi + c) * F;
      const uint32_t x = __funnelshift_r(words[bit >> 5], words[(bit >> 5) + 1], bit & 31);
      r.v[2 * c] = reinterpret_cast<const uint2*>(cb)[x & ((1u << T::kW0) - 1u)];
      r.v[2 * c + 1] = reinterpret_cast<const uint2*>(cb)[T::kEntries + (x >> T::kW0 & ((1u << T::kW1) - 1u))];
    }
  }
  return r;
}
GB_DEVINL float dot16(const RowGroup& r, float x) {
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint32_t w = i & 2 ? r.v[i >> 2].y : r.v[i >> 2].x;
    s = fmaf(__shfl_sync(0xffffffffu, x, i), i & 1 ? __uint_as_float(w & 0xFFFF0000u) : __uint_as_float(w << 16), s);
  }
  return s * r.scale;
}

template <bool kGrouped, bool kWide, int F>
__global__ void __launch_bounds__(kThreads, 1)
fp4_decode_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Fp4Params p) {
  using T = Fmt<F>;
  using G = Geo<F>;
  extern __shared__ uint8_t smem_raw[];
  // barriers and small state
  const uint32_t win = gb_smem_u32(smem_raw) & 0xFF000000u;
  const uint32_t misc = kDynBase | win;
  const uint32_t raw_full = misc, raw_empty = misc + 8 * kMaxRaw;
  // per unit slot: activations landed / operand complete / multiplied
  const uint32_t x_full = raw_empty + 8 * kMaxRaw, full = x_full + 8 * kMaxX, done = full + 8 * kMaxX;
  const uint32_t acc_full = done + 8 * kMaxX, acc_empty = acc_full + 8, red_full = acc_full + 16;
  const uint32_t slot_addr = acc_full + 24;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_raw + (slot_addr - misc));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + (slot_addr - misc) + 4);
  const uint32_t scale_tab = p.sf_off | win;               // two-tier: the scale table, then
  const uint32_t sfa_stage = scale_tab + 4096u;            // scale bytes of a unit, two buffers of 2 KiB per warpgroup

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slice = blockIdx.y;
  const int sb_begin = slice * p.units;
  const int units = min(p.units, p.n_sb - sb_begin);
  // Units are numbered over all items, an item's count rounded up to whole raw stages: a unit without weights
  // passes every barrier and multiplies nothing.  So the warpgroup, the raw slot and the activation slot of a
  // unit follow from its number alone.  A warp must see every phase of a barrier it waits for (a parity wait cannot
  // tell a phase from the one two before); with four or eight units in a ring, a slot's units are always the same
  // warpgroup's, so only that one waits for it.
  const int span = (units + T::kSbPerStage - 1) / T::kSbPerStage * T::kSbPerStage;
  // Layout of tensor memory.  Narrow: four accumulators of 64 columns, one per warpgroup, two issuers in turn; wide:
  // [hi | dlt] in columns [0, 128), [lo] in [128, 192), one issuer each.  Then the four operand
  // buffers: nibbles (32), weight scale factors (16), activation scale factors (16 per set).
  constexpr bool wide = kWide;
  constexpr int n_iss = 2;
  constexpr uint32_t acc_stride = wide ? 128u : 64u;
  constexpr uint32_t buf_col0 = wide ? 192u : 256u, buf_stride = wide ? 80u : 64u;
  constexpr int sfx = sf_bytes(wide);
  // each ring holds four units or eight
  const int raw_stages = p.raw_stages, raw_two = raw_stages * T::kSbPerStage == 8 ? 1 : 0, raw_log = raw_stages == 8 ? 3 : raw_stages == 4 ? 2 : 1;
  const uint32_t raw_ring = p.raw_off | win;
  const int x_two = p.x_stages == 8 ? 1 : 0, x_mask = p.x_stages - 1, x_log = 2 + x_two;
  const uint32_t x_ring = p.x_off | win, x_stage = (uint32_t)p.x_unit;

  gb_pdl_launch_dependents();
  if ((gb_smem_u32(smem_raw) ^ win) != kDynBase) {                 // the addresses above assume it
    if (threadIdx.x == 0) atomicExch(p.status, 41);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxRaw; ++s) {
      mbar_init(raw_full + 8 * s, 1);
      mbar_init(raw_empty + 8 * s, 4 * T::kSbPerStage);
    }
    for (int s = 0; s < kMaxX; ++s) {
      mbar_init(x_full + 8 * s, 1);
      mbar_init(full + 8 * s, 8);                            // four warps that decode the unit, four that store the scale factors
      mbar_init(done + 8 * s, wide ? 2 : 1);
    }
    mbar_init(acc_full, (uint32_t)n_iss);
    mbar_init(acc_empty, kDecWarps);
    mbar_init(red_full, (uint32_t)(p.slices * kDecWarps));
    *abort_flag = 0;
    gb_fence_barrier_init();
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (p.slices > 1) {
    uint32_t size, rank;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    if (threadIdx.x == 0 && ((int)size != p.slices || (int)rank != slice)) {
      *abort_flag = 1;
      atomicExch(p.status, 51);
    }
    gb_cluster_sync();                                        // peers write into this CTA's shared memory later: all must have started
  }
  const uint32_t tmem_base = *tmem_slot;

  int have_role = -1;
  if (kGrouped) {
    // the tables need nothing of an earlier launch, the segment offsets do: every role looks through the
    // experts for its tiles, so they are copied next to it (ten tiles a CTA, 500 clocks each from L2)
    if (warp >= kCtlWarps) {
      build_scale_tab<F>(p.mat[0].compose, threadIdx.x - 32 * kCtlWarps, scale_tab);
      build_lut<F, kWide>(reinterpret_cast<const uint16_t*>(p.mat[0].codebook), threadIdx.x - 32 * kCtlWarps, kLut | win);
      have_role = 0;
    }
    gb_pdl_wait();
    if (p.seg_off != 0)
      for (int i = threadIdx.x; i <= p.E; i += kThreads)
        asm volatile("st.shared.s32 [%0], %1;" ::"r"((p.seg_off | win) + 4u * (uint32_t)i), "r"(p.seg[i]) : "memory");
    __syncthreads();
  }
  auto seg_at = [&](int e) {
    if (p.seg_off == 0) return p.seg[e];
    int v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"((p.seg_off | win) + 4u * (uint32_t)e));
    return v;
  };
  struct Tile { int n0, n_end, w_row0, lo, cnt, n_pass, x_tile, role; };   // role 0: grouped
  auto tile_at = [&](int t) {
    Tile R;
    if (kGrouped) {
      const int e = t / p.tiles_n;
      R.n0 = (t - e * p.tiles_n) * kBM;
      R.n_end = (int)p.mat[0].N;
      R.w_row0 = e * (int)p.mat[0].N + R.n0;
      R.lo = seg_at(e);
      R.cnt = seg_at(e + 1) - R.lo;
      R.n_pass = R.cnt > 0 ? (R.cnt + p.pass_rows - 1) / p.pass_rows : 0;
      R.x_tile = R.lo / p.pass_rows + e;                   // tiles of different (expert, pass) never coincide
      R.role = 0;
    } else {
      int r = 0;
      while (r + 1 < p.n_roles && t >= p.role[r + 1].tile0) ++r;
      R.n0 = p.role[r].row0 + (t - p.role[r].tile0) * kBM;
      R.n_end = p.role[r].row0 + p.role[r].rows;
      R.w_row0 = R.n0;
      R.lo = 0; R.cnt = p.M; R.n_pass = 1; R.x_tile = 0; R.role = r;
    }
    return R;
  };

  // The loading and issuing warps walk their loops whole, with values that are the same in every lane, and one elected
  // lane issues: the operands then stay in uniform registers.  In code that only lane 0 enters an MMA takes 53 clocks to
  // issue whatever its N; this way 11 (N = 16), 22 (48), 60 (128), and four of N = 48 have completed after 180 clocks instead of 413.
  if (warp == 0) {
    // ------------------------- packed weight rows -------------------------
    const bool leader = gb_elect_one();
    int n = 0;                                             // stages since the start
    bool ok = true;
    for (int t = blockIdx.x; t < p.n_tiles && ok; t += gridDim.x) {
      const Tile R = tile_at(t);
      const int n_pass = kGrouped ? __shfl_sync(0xffffffffu, R.n_pass, 0) : 1;
      for (int pass = 0; pass < n_pass && ok; ++pass)
        for (int u = 0; u < units; u += T::kSbPerStage, ++n) {
          const int s = n & (raw_stages - 1);
          ok = warp_wait(raw_empty + 8 * s, ((uint32_t)(n >> raw_log) & 1u) ^ 1u, abort_flag, p.status, 42);
          if (!ok) break;                                  // no copy may be in flight when the CTA leaves
          if (leader) {
            mbar_expect(raw_full + 8 * s, G::kBoxBytes);
            tma_load_2d(raw_ring + (uint32_t)s * G::kBoxBytes, &maps.m[kGrouped ? 0 : p.role[R.role].mat], (sb_begin + u) * T::kSb, R.w_row0, raw_full + 8 * s);
          }
          __syncwarp();
        }
    }
  } else if (warp == 1) {
    // ------------------------- activation operand --------------------------
    gb_pdl_wait();
    const bool leader = gb_elect_one();
    int g = 0;                                             // units since the start, over all tiles and passes
    bool ok = true;
    for (int t = blockIdx.x; t < p.n_tiles && ok; t += gridDim.x) {
      const Tile R = tile_at(t);
      const int n_pass = kGrouped ? __shfl_sync(0xffffffffu, R.n_pass, 0) : 1, cnt = kGrouped ? __shfl_sync(0xffffffffu, R.cnt, 0) : p.M;
      const int x_tile = kGrouped ? __shfl_sync(0xffffffffu, R.x_tile, 0) : 0;
      for (int pass = 0; pass < n_pass && ok; ++pass) {
        const int rows = min(p.pass_rows, cnt - pass * p.pass_rows);
        const uint32_t bytes = (uint32_t)unit_bytes(wide, rows);
        const uint8_t* src = p.xop + ((int64_t)(x_tile + pass) * p.n_sb + sb_begin) * p.x_unit;
        for (int u = 0; u < span; ++u, ++g, src += p.x_unit) {
          const int s = g & x_mask;
          ok = warp_wait(done + 8 * s, ((uint32_t)(g >> x_log) & 1u) ^ 1u, abort_flag, p.status, 43);
          if (!ok) break;
          if (leader) {
            if (T::kSbPerStage > 1 && u >= units) {
              mbar_arrive(x_full + 8 * s);
            } else {
              mbar_expect(x_full + 8 * s, bytes);
              bulk_load(x_ring + (uint32_t)s * x_stage, src, bytes, x_full + 8 * s);
            }
          }
          __syncwarp();
        }
      }
    }
  } else if (warp < 4) {
    // ------------------------- MMA issuers ---------------------------------
    // Narrow: issuer i takes every other unit, into the accumulator of its warpgroup.  Wide: issuer 0 multiplies
    // every unit with [hi | dlt], issuer 1 with [lo].
    const int i = __shfl_sync(0xffffffffu, warp, 0) - 2;
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    const bool leader = gb_elect_one();
    constexpr int u_step = wide ? 1 : 2;
    const uint32_t sf_col = 48u + (wide ? (uint32_t)i * 16u : 0u);
    const uint64_t db0 = desc_sw128(x_ring + (uint32_t)sfx);
    int g0 = 0, item = 0;                                  // units / (tile, pass) items since the start
    bool gone = false;
    for (int t = blockIdx.x; t < p.n_tiles && !gone; t += gridDim.x) {
      const Tile R = tile_at(t);
      const int n_pass = kGrouped ? __shfl_sync(0xffffffffu, R.n_pass, 0) : 1, cnt = kGrouped ? __shfl_sync(0xffffffffu, R.cnt, 0) : p.M;
      for (int pass = 0; pass < n_pass && !gone; ++pass, ++item, g0 += span) {
        const int rows = min(p.pass_rows, cnt - pass * p.pass_rows);
        const int n = wide && i == 1 ? term_rows(true, rows) : mma_cols(wide, rows);
        // E2M1 x E2M1, UE4M3 scale factors, both K-major, fp32 accumulate; N >> 3, M >> 4
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
        if (item > 0) {
          wait(acc_empty, (item - 1) & 1, abort_flag, p.status, 44);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        for (int u = wide ? 0 : (i - g0) & 1; u < span; u += u_step) {
          const int g = g0 + u, s = g & x_mask;
          const uint32_t acc = tmem + (uint32_t)(wide ? i : g & 3) * acc_stride;
          const uint32_t a = tmem + buf_col0 + (uint32_t)(g & 3) * buf_stride, off = (uint32_t)s * x_stage;
          const uint64_t db = db0 + (uint64_t)(off >> 4);
          if (!warp_wait(full + 8 * s, (uint32_t)(g >> x_log) & 1u, abort_flag, p.status, 45)) { gone = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (leader) {
            if (T::kSbPerStage == 1 || u < units) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_fp4_ts(acc, a + 8u * k, db + (uint64_t)(2 * k), idesc, a + 32u + 4u * k, a + sf_col + 4u * k, u >= (wide ? 1 : 4) || k > 0);
            }
            umma_commit(done + 8 * s);
          }
          __syncwarp();
        }
        if (leader) umma_commit(acc_full);
        __syncwarp();
      }
    }
  } else if (warp < kCtlWarps) {
    // ------------------------- activation scale factors ---------------------
    // From shared to tensor memory, one warp per lane quarter: atom k is what MMA k reads, its line l the four columns
    // of lane l of every quarter.
    // The next unit's are read while the stores of this one complete: every unit passes these four warps.
    const uint32_t sf_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + buf_col0 + 48u;
    int64_t total = 0;                                     // units of the CTA
    for (int t = blockIdx.x; t < p.n_tiles; t += gridDim.x) total += (kGrouped ? tile_at(t).n_pass : 1) * span;
    const int n_units = (int)total;
    uint32_t v[wide ? 2 : 1][16];
    auto arrived = [&](int g) { return mbar_test(x_full + 8 * (g & x_mask), (uint32_t)(g >> x_log) & 1u); };
    auto fetch = [&](int g) {                              // (a unit without weights reads what an earlier one left)
      const uint32_t sx = x_ring + (uint32_t)(g & x_mask) * x_stage + (uint32_t)lane * 16u;
#pragma unroll
      for (int k = 0; k < (wide ? 8 : 4); ++k) {
        const uint4 q = lds128(sx + 512u * k);
        uint32_t* o = &v[k >> 2][4 * (k & 3)];
        o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w;
      }
    };
    bool have = false;
    for (int g = 0; g < n_units; ++g) {
      const int s = g & x_mask;
      const bool free = g < 4 || mbar_test(done + 8 * ((g - 4) & x_mask), (uint32_t)((g - 4) >> x_log) & 1u);
      if (!have) {
        wait(x_full + 8 * s, (uint32_t)(g >> x_log) & 1u, abort_flag, p.status, 46);
        fetch(g);
      }
      if (!free) wait(done + 8 * ((g - 4) & x_mask), (uint32_t)((g - 4) >> x_log) & 1u, abort_flag, p.status, 52);
      const uint32_t col = sf_base + (uint32_t)(g & 3) * buf_stride;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tmem_st16(col, v[0]);
      if constexpr (wide) tmem_st16(col + 16u, v[1]);
      have = __all_sync(0xffffffffu, arrived(g + 1)) && g + 1 < n_units;
      if (have) fetch(g + 1);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * s);
    }
  } else {
    // ------------------------- decoders -------------------------------------
    const int d = threadIdx.x - 32 * kCtlWarps;              // 0 .. 511
    const int quarter = warp & 3, wg = (warp - kCtlWarps) >> 2;
    const int row = quarter * 32 + lane;                     // weight row of the tile = tensor-memory lane
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t buf = lane_base + buf_col0 + (uint32_t)wg * buf_stride;
    const uint32_t lane4 = win | (F == kLit || kByteCodes<F, kWide> ? (uint32_t)lane * 4u : (uint32_t)(lane & ((int)(T::kStride / 4) - 1)) * 4u);
    int have_mat = kGrouped ? 0 : -1;                        // whose scale table it is
    bool waited = false;
    float xs0 = 0.0f, xs1 = 0.0f;                            // scale words of rows lane, lane + 32
    int item = 0, g0 = 0;                                    // items and units so far
    // This warpgroup's units are wg, wg + 4, ..; the j-th of them:
    int g = wg, j = 0;
    const uint32_t raw_slot = (uint32_t)(wg / T::kSbPerStage), raw_step = 4u / T::kSbPerStage;   // raw slots: first, to the second
    const uint32_t raw_row = raw_ring + raw_slot * G::kBoxBytes + (uint32_t)(wg % T::kSbPerStage) * T::kSb;
    auto raw_bar = [&](uint32_t base, int n) { return base + 8u * (raw_slot + raw_step * (uint32_t)(n & raw_two)); };
    auto raw_phase = [&](int n) { return (uint32_t)(n >> raw_two) & 1u; };
    auto x_bar = [&](uint32_t base, int n) { return base + 8u * ((uint32_t)wg + 4u * (uint32_t)(n & x_two)); };
    auto x_phase = [&](int n) { return (uint32_t)(n >> x_two) & 1u; };
    bool raw_ok = false;                                     // the next unit's rows have been seen to be there
    // An item's accumulators are read out after the warpgroup has decoded its first unit of the NEXT item:
    // the last multiplications, their completion and the read-out then overlap decoding, and the next
    // item's multiplications find their operands ready.  (Nothing that first unit waits for needs this
    // read-out: its buffer, its activations' slot and its raw stage were last used by earlier items.)
    int t = blockIdx.x, pass = 0, out_t = -1, out_pass = 0;  // current item; the item to be read out
    Tile R = {};
    auto settle = [&]() {                                    // t: the next tile with rows, from t on
      for (; t < p.n_tiles; t += gridDim.x) {
        R = tile_at(t);
        if (R.n_pass > 0) break;
      }
    };
    settle();
    while (t < p.n_tiles || out_t >= 0) {
      const bool live = t < p.n_tiles;
      if (live && R.role != have_role) {                     // the CTA's rows change codebook
        if (have_role >= 0) asm volatile("bar.sync 1, %0;" ::"n"(32 * kDecWarps) : "memory");
        const Matrix& W = p.mat[p.role[R.role].mat];
        if (F != kLit && p.role[R.role].mat != have_mat) build_scale_tab<F>(W.compose, d, scale_tab);
        have_mat = p.role[R.role].mat;
        build_lut<F, kWide>(reinterpret_cast<const uint16_t*>(W.codebook) + p.role[R.role].cb, d, kLut | win);
        have_role = R.role;
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kDecWarps) : "memory");
      }
      {
        const int g_end = live ? g0 + span : g0;
#pragma unroll 1
        do {
          if (g < g_end) {
            if (!raw_ok) wait(raw_bar(raw_full, j), raw_phase(j), abort_flag, p.status, 47);
            // The buffer's last unit has been multiplied: looked at early, waited for where it matters.  The slot's next
            // completion is a later unit of this warpgroup, so it cannot run ahead of this wait.
            bool free = j == 0;
            if (T::kSbPerStage == 1 || g - g0 < units) {
              const uint32_t stage = raw_row + (uint32_t)(j & raw_two) * (raw_step * G::kBoxBytes);
              const uint32_t rp = stage + (uint32_t)row * G::kPitch;
              uint32_t v[32], sfa[16], sg;                   // sfa: scale words of rows lane, lane + 32, lane + 64, lane + 96
              constexpr uint32_t sg_step = F == kLit ? 32u * G::kPitch : 512u;
              if constexpr (F == kLit) {
                const uint4 c0 = lds128(rp), c1 = lds128(rp + 16), own = lds128(rp + 32);
                if (j > 0) free = mbar_test(x_bar(done, j - 1), x_phase(j - 1));
                const uint32_t cw[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
                for (int c = 0; c < 32; ++c) v[c] = codeword<F, kWide>(cw, c, lane4);
                if (__builtin_expect((own.x | own.y | own.z | own.w) & 0x80808080u, 0)) {
                  // scale factors carry no sign: it moves into the nibbles
                  const uint32_t os[4] = {own.x, own.y, own.z, own.w};
#pragma unroll
                  for (int q = 0; q < 16; ++q) {
                    const uint32_t neg = (os[q >> 2] >> (8 * (q & 3))) & 0x80u ? 0x88888888u : 0u;
                    v[2 * q] ^= neg;
                    v[2 * q + 1] ^= neg;
                  }
                }
                sg = stage + (uint32_t)lane * G::kPitch + 32u;
              } else {
                uint32_t w[T::kSb / 4];
#pragma unroll
                for (int q = 0; q < T::kSb / 16; ++q) {
                  const uint4 x = lds128(rp + 16u * q);
                  w[4 * q] = x.x; w[4 * q + 1] = x.y; w[4 * q + 2] = x.z; w[4 * q + 3] = x.w;
                }
                if (j > 0) free = mbar_test(x_bar(done, j - 1), x_phase(j - 1));
                // the super byte sits right behind the 4k index bytes, then sixteen nibbles
                const uint4 tb = lds128(scale_tab + (w[F] & 0xFFu) * 16u);
                __syncwarp();
                if (lane == 0) mbar_arrive(raw_bar(raw_empty, j));  // the whole superblock is in registers
                const uint32_t n0s = __funnelshift_r(w[F], w[F + 1], 8), n1s = __funnelshift_r(w[F + 1], w[F + 2], 8);
                // two buffers: a warp that writes the next unit's bytes has passed this unit's barrier,
                // which no warp reaches before it has read the unit before
                const uint32_t st = sfa_stage + (uint32_t)(wg * 4096) + (uint32_t)(j & 1) * 2048u;
                sts128(st + (uint32_t)(row * 16),
                       make_uint4(four_scales(tb, n0s), four_scales(tb, n0s >> 16), four_scales(tb, n1s), four_scales(tb, n1s >> 16)));
#pragma unroll
                for (int c = 0; c < 32; ++c) v[c] = codeword<F, kWide>(w, c, lane4);
                asm volatile("bar.sync %0, 128;" ::"r"(2 + wg) : "memory");   // the four warps of this warpgroup
                sg = st + (uint32_t)lane * 16u;
              }
              if (!free) wait(x_bar(done, j - 1), x_phase(j - 1), abort_flag, p.status, 48);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              tmem_st32(buf, v);
              uint32_t any = 0;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 s = lds128(sg + (uint32_t)q * sg_step);
                sfa[q] = s.x; sfa[4 + q] = s.y; sfa[8 + q] = s.z; sfa[12 + q] = s.w;
                any |= s.x | s.y | s.z | s.w;
              }
              if (F == kLit && __builtin_expect(any & 0x80808080u, 0)) {
#pragma unroll
                for (int q = 0; q < 16; ++q) sfa[q] &= 0x7F7F7F7Fu;
              }
              tmem_st16(buf + 32u, sfa);
              raw_ok = mbar_test(raw_bar(raw_full, j + 1), raw_phase(j + 1));
              asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            } else {                                         // a stage's missing second superblock
              if (!free) wait(x_bar(done, j - 1), x_phase(j - 1), abort_flag, p.status, 48);
              raw_ok = false;
            }
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(x_bar(full, j));
              if (F == kLit) mbar_arrive(raw_bar(raw_empty, j));
            }
            g += 4;
            ++j;
          }
          if (out_t >= 0) {
            // ------------------------- read-out ------------------------------------
            // Sums into registers, the accumulators handed back, then the stores.
            if (!waited) {                                   // the rows' scales come from the launch ahead, which may still read y
              gb_pdl_wait();
              waited = true;
              if (!kGrouped) {
                xs0 = lane < p.M ? p.x_scale[lane] : 0.0f;
                xs1 = lane + 32 < p.M ? p.x_scale[lane + 32] : 0.0f;
              }
            }
            const Tile Q = tile_at(out_t);
            const Matrix& W = p.mat[kGrouped ? 0 : p.role[Q.role].mat];
            const int rows = min(p.pass_rows, Q.cnt - out_pass * p.pass_rows);
            int to0 = lane, to1 = lane + 32;                 // output rows
            if (kGrouped) {
              const float* xsc = p.x_scale + (int64_t)(Q.x_tile + out_pass) * scale_pitch(p.pass_rows);
              xs0 = lane < rows ? xsc[lane] : 0.0f;
              xs1 = lane + 32 < rows ? xsc[lane + 32] : 0.0f;
              to0 += Q.lo + out_pass * p.pass_rows;          // sorted positions
              to1 = to0 + 32;
              if (p.row_map) {
                to0 = lane < rows ? p.row_map[to0] : 0;
                to1 = lane + 32 < rows ? p.row_map[to1] : 0;
              }
            }
            const int q_pass = out_pass;
            out_t = -1;
            wait(acc_full, (item - 1) & 1, abort_flag, p.status, 49);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool ok = *abort_flag == 0;
            if (__builtin_expect(__any_sync(0xffffffffu, (__float_as_uint(xs0) | __float_as_uint(xs1)) & kGbLeftOutBits), 0)) {
              // Groups left out: added to the sums in tensor memory, by the warps that read those out.  (Spread over the
              // warpgroups they would have to wait for each other here.)  17408 x 5120, K16, 16 rows, 15.6 us: one tiny group in
              // one row 17.1, an outlier channel in all rows 19.0, one row over 2^30 165, all of them 556.  Inline and
              // with nothing held over it: as a function, or with the sums in registers, it cost the ordinary read-out
              // its registers (two layers at 16 rows 164 -> 188..208 us, this way 167..169).
              const int64_t tile = Q.x_tile + (kGrouped ? q_pass : 0);
              const uint8_t* w_row = W.qw + (Q.w_row0 + (kGrouped ? row : min(row, (int)W.N - 1 - Q.n0))) * W.row_stride;
              const uint16_t* cb = reinterpret_cast<const uint16_t*>(W.codebook) + p.role[Q.role].cb;
              const int per = gb_left_out_span(p.n_sb);
#pragma unroll 1
              for (int j = 0; j < (wide ? 4 : 1); ++j) {
                const int m0 = wide ? (wg + 4 * (j >> 1)) * 8 + 4 * (j & 1) : wg * 4;
                if (m0 >= rows) break;
                uint32_t word[4], bits = 0u, marked = 0u;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                  word[r] = __float_as_uint(__shfl_sync(0xffffffffu, m0 < 32 ? xs0 : xs1, (m0 + r) & 31));
                  bits |= word[r] & kGbLeftOutBits;
                  marked |= (word[r] & kGbLeftOutBits) != 0 ? 1u << r : 0u;
                }
                if (bits == 0) continue;
                float add[4] = {};
                const int n0 = wide ? m0 : narrow_col(0, m0);
#pragma unroll 1
                for (; bits != 0; bits &= bits - 1) {
                  const int b = __ffs(bits) - 1;
                  gb_left_out(
                      add, p.tail + (tile * p.pass_rows + m0) * (p.K / 16), p.K / 16, marked, max(b * per, sb_begin) * 16,
                      min((b + 1) * per, sb_begin + units) * 16,
                      [&](int r, int g) {
                        return *reinterpret_cast<const uint2*>(p.xop + (tile * p.n_sb + (g >> 4)) * p.x_unit + sfx + code_at(n0 + r, g & 15));
                      },
                      [&](int g) { return row_group<F>(w_row, cb, W.compose, g); }, [](const RowGroup& r, float x) { return dot16(r, x); });
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) add[r] = gb_normalised(add[r], word[r]);
                gb_tmem_add(lane_base + (wide ? 0u : (uint32_t)((g0 - span) & 3) * acc_stride) + (uint32_t)n0, add);
              }
            }
            const int64_t col = (int64_t)Q.n0 + row;
            const uint32_t Rt = (uint32_t)term_rows(wide, rows);
            float sum[16];
            if (wide) {
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const int c = wg + 4 * j;
                if (c * 8 >= rows) break;
                uint32_t h[8], l[8], e[8];
                const uint32_t at = lane_base + (uint32_t)(c * 8);
                tmem_ld8(at, h);
                tmem_ld8(at + 128u, l);
                tmem_ld8(at + Rt, e);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  sum[8 * j + i] = fmaf(__uint_as_float(e[i]), 0x1p-7f, fmaf(__uint_as_float(l[i]), 0x1p-4f, __uint_as_float(h[i])));
              }
            } else if (wg * 4 < rows) {
              // four rows per warpgroup; issuers without a unit leave their accumulator untouched.  Units 0, 4, ..
              // of the item first, then 1, 5, ..: the order does not depend on where the item's first unit fell
              const int accs = min(4, units), a_first = g0 - span;
#pragma unroll
              for (int i = 0; i < 4; ++i) sum[i] = 0.0f;
#pragma unroll
              for (int a0 = 0; a0 < 4; a0 += 2) {
                if (a0 >= accs) break;
                uint32_t v[2][16];
                const uint32_t at = lane_base + (uint32_t)(wg * 12);
                tmem_ld16(at + (uint32_t)((a_first + a0) & 3) * acc_stride, v[0]);
                tmem_ld16(at + (uint32_t)((a_first + min(a0 + 1, accs - 1)) & 3) * acc_stride, v[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                  for (int i = 0; i < 4; ++i)
                    if (a0 + a < accs)
                      sum[i] += fmaf(__uint_as_float(v[a][8 + i]), 0x1p-7f, fmaf(__uint_as_float(v[a][4 + i]), 0x1p-4f, __uint_as_float(v[a][i])));
              }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty);
            // kRows rows from m0 on.  Their scales in one or two loads: a shuffle, a mask and a selection per row, and a division by the
            // slice count, made 190 clocks a row of these stores (64 rows, 34816 x 5120: 3 us of each tile).
            auto emit = [&](auto n_rows, int m0, const float* total) {
              constexpr int kRows = decltype(n_rows)::value;
              if (m0 >= rows) return;
              const uint4* words = reinterpret_cast<const uint4*>(p.x_scale + (kGrouped ? (int64_t)(Q.x_tile + q_pass) * scale_pitch(p.pass_rows) : 0) + m0);
              float val[kRows];
#pragma unroll
              for (int q = 0; q < kRows / 4; ++q) {
                const uint4 w = words[q];
                val[4 * q] = total[4 * q] * __uint_as_float(w.x & kGbRowScaleMask);
                val[4 * q + 1] = total[4 * q + 1] * __uint_as_float(w.y & kGbRowScaleMask);
                val[4 * q + 2] = total[4 * q + 2] * __uint_as_float(w.z & kGbRowScaleMask);
                val[4 * q + 3] = total[4 * q + 3] * __uint_as_float(w.w & kGbRowScaleMask);
              }
              if (!kGrouped && p.slices > 1) {
                // into the shared memory of the row's owner: slot [row / slices][slice][128 weight rows]
                int own = m0 / p.slices, to = m0 - own * p.slices;
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                  if (m0 + i < rows) {
                    uint32_t dst;
                    const uint32_t local = (p.red_off | win) + (uint32_t)((own * p.slices + slice) * kBM + row) * 4u;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(local), "r"(to));
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(val[i]) : "memory");
                  }
                  if (++to == p.slices) { to = 0; ++own; }
                }
              } else {
                const bool mine = ok && col < Q.n_end;
                uint16_t* y = W.y + (kGrouped ? 0 : (int64_t)m0 * W.N) + col;
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                  const int m = m0 + i;
                  const uint16_t b = (uint16_t)gb_f32_to_bf16_bits(val[i] * W.global_scale);
                  if (kGrouped) {
                    const int orow = __shfl_sync(0xffffffffu, m < 32 ? to0 : to1, m & 31);
                    if (m < rows && mine) y[(int64_t)orow * W.N] = b;
                  } else {
                    if (m < rows && mine) *y = b;
                    y += W.N;
                  }
                }
              }
            };
            if (wide) {
              emit(std::integral_constant<int, 8>(), wg * 8, sum);
              emit(std::integral_constant<int, 8>(), wg * 8 + 32, sum + 8);
            } else {
              emit(std::integral_constant<int, 4>(), wg * 4, sum);
            }
            if (!kGrouped && p.slices > 1) {
              // every warp tells every CTA of the cluster that its sums are in place, then the owners add
              __syncwarp();
              if (lane < p.slices) {
                uint32_t dst;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(red_full), "r"(lane));
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(dst) : "memory");
              }
              wait<true>(red_full, 0, abort_flag, p.status, 50);
              for (int i = d; ; i += 32 * kDecWarps) {
                const int own = i / kBM, r = i % kBM, m = own * p.slices + slice;
                if (m >= rows) break;
                float s = 0.0f;
                for (int q = 0; q < p.slices; ++q) {
                  float f;
                  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"((p.red_off | win) + (uint32_t)((own * p.slices + q) * kBM + r) * 4u));
                  s += f;
                }
                if (*abort_flag == 0 && Q.n0 + r < Q.n_end) W.y[(int64_t)m * W.N + Q.n0 + r] = (uint16_t)gb_f32_to_bf16_bits(s * W.global_scale);
              }
            }
          }
        } while (g < g_end);
      }
      if (!live) break;
      out_t = t;
      out_pass = pass;
      ++item;
      g0 += span;
      if (++pass >= R.n_pass) {
        pass = 0;
        t += gridDim.x;
        settle();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag) __nanosleep(1000000);                   // loads and MMAs still in flight end before the memory goes
  if (p.slices > 1)                                        // no CTA leaves while a peer may still reach its shared memory
    gb_cluster_sync();
  if (warp == 4)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

// ---- the activations' operand ------------------------------------------------------------------
struct Group { uint32_t q[2], e[2]; uint32_t hi, lo, dl; float tail; };   // codes of q, of the correction, three scale bytes; the scale, if left out

// The three terms of one group of sixteen bf16 values; `shift` normalises the row.
constexpr int kMinExp = -6, kMaxExp = 7;                   // normalised exponents of m1 whose terms are all exact
GB_DEVINL Group split_group(const uint32_t (&w)[8], float amax, bool nan, int scale_rule, int shift) {
  Group r;
  r.tail = 0.0f;
  amax = fmaxf(amax, 1e-8f);
  const float scale = gb_fp4_group_scale(amax, scale_rule);
  if (nan || !(scale < __int_as_float(0x7F800000))) {       // the whole group is NaN (and with it the row's results)
    r.q[0] = r.q[1] = r.e[0] = r.e[1] = 0x22222222u;
    r.hi = r.lo = r.dl = 0x7Fu;
    return r;
  }
  if (__builtin_expect(gb_plain_division(scale), 0)) {
    // one significand in 2^23: rolled up, since sixteen divisions and roundings by comparison in line were 40% of a
    // kernel that runs cold (2744 -> 1656 instructions; 34816 x 5120, rows kernel included, us: 16 rows K16 21.9 -> 21.4,
    // literal 18.6 -> 18.2, 64 rows 24.5 -> 24.0)
    uint32_t v[8], q0 = 0u, q1 = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = w[i];
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
      const uint32_t x = v[0];
      const uint32_t c = gb_cvt_e2m1x2(gb_e2m1_rtn(__fdiv_rn(gb_bf16_bits_to_f32(x & 0xFFFFu), scale)), gb_e2m1_rtn(__fdiv_rn(gb_bf16_bits_to_f32(x >> 16), scale)));
      q0 = __funnelshift_r(q0, q1, 8);
      q1 = (q1 >> 8) | (c << 24);
#pragma unroll
      for (int k = 0; k < 7; ++k) v[k] = v[k + 1];
    }
    r.q[0] = q0;
    r.q[1] = q1;
  } else {
    const float rinv = __frcp_rn(scale);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t q = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t x = w[4 * h + i];
        q |= gb_e2m1_div2(gb_bf16_bits_to_f32(x & 0xFFFFu), gb_bf16_bits_to_f32(x >> 16), scale, rinv) << (8 * i);
      }
      r.q[h] = q;
    }
  }
  const float m1 = gb_bf16_bits_to_f32(gb_f32_to_bf16_bits(scale));
  const float m3 = gb_bf16_bits_to_f32(gb_f32_to_bf16_bits(__fmul_rn(1.5f, scale)));
  const int e1 = (int)((__float_as_uint(m1) >> 23) & 0xFFu) - 127;      // m1 is normal: scale >= 1e-8 / 6
  // half-ulps of m1 by which bf16(1.5 s) misses 1.5 m1 (exact in fp32)
  const int n = (int)((m3 - 1.5f * m1) * __uint_as_float((uint32_t)(127 + 8 - e1 > 254 ? 254 : 127 + 8 - e1) << 23));
  // m1 normalised, its upper four significant bits (truncated to UE4M3), the rest times 16
  const int e = e1 + shift;
  if (e >= kMinExp && e <= kMaxExp) {
    const uint32_t vb = (__float_as_uint(m1) & 0x007FFFFFu) | ((uint32_t)(127 + e) << 23);
    r.hi = (vb >> 20) - (120u << 3);
    r.lo = gb_f32_to_e4m3((__uint_as_float(vb) - gb_e4m3_to_f32(r.hi)) * 16.0f);
    r.dl = (uint32_t)(e + 7) << 3;
  } else {                                                             // left out of the operand
    r.hi = r.lo = r.dl = 0u;
    if (((r.q[0] | r.q[1]) & 0x77777777u) != 0) r.tail = scale;
  }
  const uint32_t an = (uint32_t)(n < 0 ? -n : n), flip = n < 0 ? 0x88888888u : 0u;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t q = r.q[h];
    const uint32_t b0 = q & 0x11111111u, b1 = (q >> 1) & 0x11111111u, b2 = (q >> 2) & 0x11111111u;
    const uint32_t on = b0 & (b1 | b2), m = (on << 4) - on;            // nibbles with q = +-1.5, 3, 6: 0xF
    const uint32_t one = (b1 & ~b2) | ((b2 & ~b1) << 1) | ((b1 & b2) << 2);      // n = 1: 0.5, 1, 2
    const uint32_t mag = an == 3 ? q & 0x77777777u : an == 2 ? q & 0x66666666u : an == 1 ? one : 0u;
    r.e[h] = (mag | ((q ^ flip) & 0x88888888u)) & m;
  }
  return r;
}

// Stores one group's terms for row m of a tile with `rows` rows; called by whole quads of lanes (four
// neighbouring groups) so that the scale bytes leave as words.
GB_DEVINL void store_group(const Group& G, uint8_t* tile, int64_t unit_stride, bool wide, int rows, int m, int g, unsigned mask) {
  const int sb = g >> 4, gi = g & 15;
  uint8_t* unit = tile + sb * unit_stride;
  uint8_t* codes = unit + sf_bytes(wide);
  const int R = term_rows(wide, rows);
  auto put = [&](int n, uint2 c) {
    *reinterpret_cast<uint2*>(codes + code_at(n, gi)) = c;
  };
  const uint2 q = make_uint2(G.q[0], G.q[1]), e = make_uint2(G.e[0], G.e[1]);
  if (wide) {
    put(m, q);
    put(R + m, e);
  } else {
    put(narrow_col(0, m), q);
    put(narrow_col(1, m), q);
    put(narrow_col(2, m), e);
  }
#pragma unroll
  for (int t = 0; t < 3; ++t) {                             // hi, lo, dlt
    const uint32_t b = t == 0 ? G.hi : t == 1 ? G.lo : G.dl;
    const uint32_t b1 = __shfl_down_sync(mask, b, 1), b2 = __shfl_down_sync(mask, b, 2), b3 = __shfl_down_sync(mask, b, 3);
    const int n = !wide ? narrow_col(t, m) : t == 2 ? R + m : m;
    if ((gi & 3) == 0)
      *reinterpret_cast<uint32_t*>(unit + (wide && t == 1 ? 2048 : 0) + (gi >> 2) * 512 + (n & 31) * 16 + ((n >> 5) & 3) * 4) =
          b | (b1 << 8) | (b2 << 16) | (b3 << 24);
  }
}

// The same as the grouped GEMM's operand (gb_fp4_tiles): row m of tile `tile`.
GB_DEVINL void store_group_matrix(const Group& G, uint8_t* xop, uint8_t* sf, int K, int64_t tile, int m, int g, unsigned mask) {
  uint8_t* codes = xop + ((tile * 128 + m) * (int64_t)K) / 2 + g * 8;
  *reinterpret_cast<uint2*>(codes) = make_uint2(G.q[0], G.q[1]);
  *reinterpret_cast<uint2*>(codes + (int64_t)K * 32) = make_uint2(G.e[0], G.e[1]);
#pragma unroll
  for (int t = 0; t < 3; ++t) {                             // hi, lo, dlt
    const uint32_t b = t == 0 ? G.hi : t == 1 ? G.lo : G.dl;
    const uint32_t b1 = __shfl_down_sync(mask, b, 1), b2 = __shfl_down_sync(mask, b, 2), b3 = __shfl_down_sync(mask, b, 3);
    const int64_t c = tile * 192 + (m >> 5) * 96 + t * 32 + (m & 31);
    if ((g & 3) == 0)
      *reinterpret_cast<uint32_t*>(sf + (c >> 7) * ((int64_t)K * 8) + (g >> 2) * 512 + (c & 31) * 16 + ((c >> 5) & 3) * 4) =
          b | (b1 << 8) | (b2 << 16) | (b3 << 24);
  }
}

struct RowsParams {
  const uint4* x;            // bf16 rows [*, K]
  uint8_t* xop;
  float* x_scale;
  float* tail;
  uint8_t* sf;               // matrix form (x_unit = 0): the scale-factor plane
  int64_t x_unit;
  int K, n_sb, scale_rule, pass_rows;
  int split;                 // dense: CTAs per row
  int rows;                  // dense: M
  // grouped: sorted row j = blockIdx.x belongs to expert ids[order[j]]
  const int32_t* ids;
  const int32_t* order;
  const int32_t* seg;
  int E, topk;
  int swiglu;                // x holds [gate | up] rows in sorted order
  const int32_t* inv;        // token mode: sorted position of every pair
};

constexpr int kRowsMaxGroups = 4;
constexpr int kMaxRowSplit = 8;
constexpr int kMaxCopies = 32;                             // destinations looked up ahead
constexpr int kRowSplitGroups = 320;                       // groups of a row per CTA of its cluster

// Exponent of the bf16 group scale of a group whose largest magnitude is amax: -30 .. 125.
GB_DEVINL int scale_exponent(float amax, int scale_rule) {
  const float m1 = gb_bf16_bits_to_f32(gb_f32_to_bf16_bits(gb_fp4_group_scale(fmaxf(amax, 1e-8f), scale_rule)));
  return (int)((__float_as_uint(m1) >> 23) & 0xFFu) - 127;
}
constexpr uint32_t kZeroCodes = (127u - 32u) << 23;        // 2^-32: below this every code is zero (the scale's floor is 1e-8 / 6)

// A value of this CTA into its slot of every CTA of the cluster, all of which must have started.
GB_DEVINL void to_peers(uint32_t* slots, uint32_t v, int split) {
  if ((int)threadIdx.x < split) {
    uint32_t dst;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(gb_smem_u32(&slots[(int)blockIdx.x % split])), "r"(threadIdx.x));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst), "r"(v) : "memory");
  }
}

// kMode 0: dense, a cluster of `split` CTAs per row (a single CTA holding 1088 groups of a 17408-wide row took
// 16 us for 64 rows: 64 SMs, four groups a thread in turn).  1: one CTA per token, its row goes to each of its experts' tiles.
// 2: one CTA per sorted row of [gate | up]: SwiGLU (with the bf16 roundings of F.silu(gate) * up), then the split.
template <int kG, int kMode>
__global__ void __launch_bounds__(1024)
fp4_rows_kernel(const __grid_constant__ RowsParams p) {
  // the grouped GEMM's operand (no unit size): the stack's expander runs beside this launch and needs what is ahead to
  // have completed; the decode kernel waits for it all the same, and starts early
  const bool late = kMode != 0 && p.x_unit == 0;
  if (!late) gb_pdl_launch_dependents();
  // A peer's shared memory may be written only once its CTA has started.  Said here, waited for in front of the first such
  // store: the row's load and the CTA's own maximum lie in between.
  if (kMode == 0 && p.split > 1) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
  gb_pdl_wait();
  if (late) gb_pdl_launch_dependents();
  const int groups = p.K / 16;
  const int j = kMode == 0 ? (int)blockIdx.x / p.split : (int)blockIdx.x;
  const int g_first = (kMode == 0 ? (int)blockIdx.x % p.split * (int)blockDim.x : 0) + (int)threadIdx.x;
  // Where the row goes, looked up first and by the last warp: three or four dependent loads per copy, which
  // one after the other behind the split cost more than the split (4096 tokens x 8 experts 42 -> 36 us)
  __shared__ int dest_tile[kMaxCopies], dest_m[kMaxCopies], dest_rows[kMaxCopies];
  const int copies = kMode == 1 ? p.topk : 1;
  auto place = [&](int s, int& tile, int& m, int& rows) {
    tile = -1;
    if (kMode == 2 && j >= p.seg[p.E]) return;
    const int pair = kMode == 1 ? j * p.topk + s : p.order[j];
    const int e = p.ids[pair];
    const int at = kMode == 1 ? p.inv[pair] : j;
    if (e < 0 || e >= p.E) return;                           // a dropped pair
    const int lo = p.seg[e], cnt = p.seg[e + 1] - lo;
    const int r = at - lo, pass = r / p.pass_rows;
    m = r - pass * p.pass_rows;
    rows = min(p.pass_rows, cnt - pass * p.pass_rows);
    tile = lo / p.pass_rows + e + pass;
  };
  if (kMode != 0) {
    const int s = (int)(blockDim.x - 1 - threadIdx.x);
    if (s < min(copies, kMaxCopies)) {
      int tile, m = 0, rows = 0;
      place(s, tile, m, rows);
      dest_tile[s] = tile; dest_m[s] = m; dest_rows[s] = rows;   // read behind the barrier of the row's maximum
    }
  }
  const uint4* xr = p.x + (int64_t)j * (kMode == 2 ? 4 : 2) * groups;
  __shared__ uint2 red[32];                                // magnitudes order as their bits do
  uint32_t w[kG][8];
  float amax[kG];
  bool nan[kG];
  uint32_t top = 0u, low = 0x7F800000u;                    // largest and smallest group of the row
#pragma unroll
  for (int i = 0; i < kG; ++i) {
    const int g = g_first + i * (int)blockDim.x;
    amax[i] = 0.0f;
    nan[i] = false;
    if (g < groups) {
      if (kMode == 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 a = xr[2 * g + h], b = xr[2 * groups + 2 * g + h];
          const uint32_t gw[4] = {a.x, a.y, a.z, a.w}, uw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float s0 = gb_bf16_bits_to_f32(gb_f32_to_bf16_bits(gb_silu(gb_bf16_bits_to_f32(gw[q] & 0xFFFFu))));
            const float s1 = gb_bf16_bits_to_f32(gb_f32_to_bf16_bits(gb_silu(gb_bf16_bits_to_f32(gw[q] >> 16))));
            w[i][4 * h + q] = gb_pack_bf16x2(s0 * gb_bf16_bits_to_f32(uw[q] & 0xFFFFu), s1 * gb_bf16_bits_to_f32(uw[q] >> 16));
          }
        }
      } else {
        const uint4 a = xr[2 * g], b = xr[2 * g + 1];
        w[i][0] = a.x; w[i][1] = a.y; w[i][2] = a.z; w[i][3] = a.w;
        w[i][4] = b.x; w[i][5] = b.y; w[i][6] = b.z; w[i][7] = b.w;
      }
      amax[i] = gb_amax_bf16(w[i], &nan[i]);
      const uint32_t bits = __float_as_uint(amax[i]);
      if (bits < 0x7F800000u) {
        top = max(top, bits);
        if (bits >= kZeroCodes) low = min(low, bits);
      }
    }
  }
  auto reduce = [&]() {
    top = __reduce_max_sync(0xffffffffu, top);
    low = __reduce_min_sync(0xffffffffu, low);
  };
  reduce();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_uint2(top, low);
  __syncthreads();
  if ((int)(threadIdx.x & 31) < (int)(blockDim.x >> 5)) {
    top = red[threadIdx.x & 31].x;
    low = red[threadIdx.x & 31].y;
  }
  reduce();
  if (kMode == 0 && p.split > 1) {                         // over the row's CTAs
    __shared__ uint32_t peer_top[kMaxRowSplit], peer_low[kMaxRowSplit];
    asm volatile("barrier.cluster.wait;" ::: "memory");
    to_peers(peer_top, top, p.split);
    to_peers(peer_low, low, p.split);
    gb_cluster_sync();                                        // the last access to another CTA's memory lies in front of it
    for (int q = 0; q < p.split; ++q) {
      top = max(top, peer_top[q]);
      low = min(low, peer_low[q]);
    }
  }
  int anchor = scale_exponent(__uint_as_float(top), p.scale_rule);   // exponent of m1 that becomes kMaxExp
  const bool marked = low < 0x7F800000u && anchor - scale_exponent(__uint_as_float(low), p.scale_rule) > kMaxExp - kMinExp;
  if (__builtin_expect(marked, 0)) {                       // half the range above the mean exponent of the groups with codes
    __shared__ int sums[2];
    if (threadIdx.x < 2) sums[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kG; ++i)
      if (__float_as_uint(amax[i]) >= kZeroCodes && __float_as_uint(amax[i]) < 0x7F800000u) {
        atomicAdd(&sums[0], scale_exponent(amax[i], p.scale_rule));
        atomicAdd(&sums[1], 1);
      }
    __syncthreads();
    int sum = sums[0], count = sums[1];
    if (kMode == 0 && p.split > 1) {
      __shared__ uint32_t peer_sum[kMaxRowSplit], peer_count[kMaxRowSplit];
      to_peers(peer_sum, (uint32_t)sum, p.split);
      to_peers(peer_count, (uint32_t)count, p.split);
      gb_cluster_sync();
      sum = count = 0;
      for (int q = 0; q < p.split; ++q) {
        sum += (int)peer_sum[q];
        count += (int)peer_count[q];
      }
    }
    // at most 2^60 below the largest: what is left out is added in the row's normalised units
    anchor = max(min(anchor, sum / count + (kMaxExp - kMinExp) / 2), anchor - 60);
  }
  Group grp[kG];
#pragma unroll
  for (int i = 0; i < kG; ++i)
    if (g_first + i * (int)blockDim.x < groups) grp[i] = split_group(w[i], amax[i], nan[i], p.scale_rule, kMaxExp - anchor);
  uint32_t left_out = 0u;                                  // one bit for each sixteenth of the row
  if (__builtin_expect(marked, 0)) {
    __shared__ uint32_t all;
    if (threadIdx.x == 0) all = 0u;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kG; ++i) {
      const int g = g_first + i * (int)blockDim.x;
      if (g < groups && grp[i].tail != 0.0f) atomicOr(&all, 1u << ((g >> 4) / gb_left_out_span(p.n_sb)));
    }
    __syncthreads();
    left_out = all;
    if (kMode == 0 && p.split > 1) {
      __shared__ uint32_t peer_all[kMaxRowSplit];
      to_peers(peer_all, left_out, p.split);
      gb_cluster_sync();
      for (int q = 0; q < p.split; ++q) left_out |= peer_all[q];
    }
    for (int s = 0; s < copies; ++s) {
      int tile = 0, m = j, rows = 0;
      if (kMode != 0) place(s, tile, m, rows);
#pragma unroll
      for (int i = 0; i < kG; ++i) {
        const int g = g_first + i * (int)blockDim.x;
        if (tile >= 0 && g < groups) p.tail[((int64_t)tile * p.pass_rows + m) * groups + g] = grp[i].tail;
      }
    }
  }
  const float back = __uint_as_float(((uint32_t)(127 - kMaxExp + anchor) << 23) | left_out);

  for (int s = 0; s < copies; ++s) {
    int tile = 0, m = j, rows = p.rows;
    if (kMode != 0) {
      if (s < kMaxCopies) { tile = dest_tile[s]; m = dest_m[s]; rows = dest_rows[s]; }
      else place(s, tile, m, rows);
      if (tile < 0) continue;                                // uniform over the CTA
    }
    if (threadIdx.x == 0 && (kMode != 0 || blockIdx.x % p.split == 0)) p.x_scale[(int64_t)tile * scale_pitch(p.pass_rows) + m] = back;
    uint8_t* dst = p.xop + (int64_t)tile * p.n_sb * p.x_unit;
#pragma unroll
    for (int i = 0; i < kG; ++i) {
      const int g = g_first + i * (int)blockDim.x;
      const unsigned here = __ballot_sync(0xffffffffu, g < groups);
      if (g >= groups) continue;
      if (kMode != 0 && p.x_unit == 0) store_group_matrix(grp[i], p.xop, p.sf, p.K, tile, m, g, here);
      else store_group(grp[i], dst, p.x_unit, is_wide(p.pass_rows), rows, m, g, here);
    }
  }
}

// ---- host side -----------------------------------------------------------------------------------
int fp4_format(const gb_weight* w, bool scales_e4m3) {
  const gb_format& f = w->fmt;
  if (f.grid != GB_GRID_FP4 || (w->row_stride % 16) != 0 || ((uintptr_t)w->qw & 15u) != 0 || ((uintptr_t)w->codebook & 15u) != 0)
    return -1;
  if (f.mode == GB_MODE_FULL && f.k_bits == 8 && f.scale_coding == GB_SCALE_V1 && f.type_size == 48) return kLit;
  if (f.mode == GB_MODE_PRODUCT && f.n_sub == 2 && f.scale_coding == GB_SCALE_V2 && w->compose != nullptr && scales_e4m3) {
    switch (f.k_bits) {
      case 12: return f.type_size == Fmt<12>::kSb ? 12 : -1;
      case 16: return f.type_size == Fmt<16>::kSb ? 16 : -1;
      case 20: return f.type_size == Fmt<20>::kSb ? 20 : -1;
      case 24: return f.type_size == Fmt<24>::kSb ? 24 : -1;
      default: return -1;
    }
  }
  return -1;
}

struct Info { int sb, per_stage, pitch; uint32_t box, lut, extra; };
template <int F> Info info_of(bool wide) {
  const uint32_t lut = (wide ? kByteCodes<F, true> : kByteCodes<F, false>) ? 256 * 256 : Fmt<F>::kLutBytes;
  return {Fmt<F>::kSb, Fmt<F>::kSbPerStage, Geo<F>::kPitch, (uint32_t)Geo<F>::kBoxBytes, lut,
          Fmt<F>::kScaleTab + (F == kLit ? 0u : 16384u)};
}
Info info(int F, bool wide) {
  switch (F) {
    case kLit: return info_of<kLit>(wide);
    case 12: return info_of<12>(wide);
    case 16: return info_of<16>(wide);
    case 20: return info_of<20>(wide);
    default: return info_of<24>(wide);
  }
}

// Shared memory: barriers, tables, then the rings and what else the launch needs.  Both rings hold eight units
// where they fit, else four (kernel: only these keep a slot's units with one warpgroup); the activations'
// first, whose way round (multiplied, asked for, loaded) is the longer one.
bool layout(const Info& f, Fp4Params& p) {
  const uint32_t red = p.slices > 1 ? (uint32_t)((p.M + p.slices - 1) / p.slices * p.slices * kBM * 4) : 0u;
  for (p.x_stages = 8; p.x_stages >= 4; p.x_stages -= 4)
    for (p.raw_stages = 8 / f.per_stage; p.raw_stages * f.per_stage >= 4; p.raw_stages >>= 1) {
      uint32_t at = kLut + f.lut;
      auto take = [&](uint32_t bytes, uint32_t align) {
        const uint32_t a = (at + align - 1) & ~(align - 1);
        at = a + bytes;
        return a;
      };
      p.x_off = take((uint32_t)(p.x_stages * p.x_unit), 1024);
      p.raw_off = take(f.box * (uint32_t)p.raw_stages, 128);
      p.sf_off = take(f.extra, 128);
      p.red_off = take(red, 128);
      if (at > kSmemEnd) continue;
      p.seg_off = p.E > 0 ? take(4u * (uint32_t)(p.E + 1), 128) : 0;
      if (at > kSmemEnd) p.seg_off = 0;
      return true;
    }
  return false;
}

GbClusters g_clusters;
int max_clusters(int size) { return g_clusters.ask((const void*)fp4_decode_kernel<false, false, kLit>, kThreads, kSmemMax, size); }

template <bool kGrouped>
cudaError_t launch(int F, dim3 grid, cudaStream_t stream, const Maps& maps, const Fp4Params& p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemMax;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (gb_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (p.slices > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 1; attr[n].val.clusterDim.y = (unsigned)p.slices; attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  gb_count_launch();
  const bool wide = is_wide(p.pass_rows);
  switch (F) {
#define GB_FP4_LAUNCH(f)                                                                       \
  return wide ? cudaLaunchKernelEx(&cfg, fp4_decode_kernel<kGrouped, true, f>, maps, p)       \
              : cudaLaunchKernelEx(&cfg, fp4_decode_kernel<kGrouped, false, f>, maps, p)
    case kLit: GB_FP4_LAUNCH(kLit);
    case 12: GB_FP4_LAUNCH(12);
    case 16: GB_FP4_LAUNCH(16);
    case 20: GB_FP4_LAUNCH(20);
    default: GB_FP4_LAUNCH(24);
#undef GB_FP4_LAUNCH
  }
}

template <int kMode>
int launch_rows(int64_t rows, int64_t K, cudaStream_t stream, RowsParams p) {
  const int64_t groups = K / 16;
  p.split = 1;
  if (kMode == 0) {
    p.split = groups > 512 ? (int)((groups + kRowSplitGroups - 1) / kRowSplitGroups) : 1;   // 384 groups: 1 us slower in two
    if (p.split > kMaxRowSplit) p.split = kMaxRowSplit;
  }
  const int64_t share = (groups + p.split - 1) / p.split;
  const int per = kMode == 0 || share <= 512 ? 1 : share <= 1024 ? 2 : kRowsMaxGroups;
  const int64_t threads = ((share + per - 1) / per + 31) / 32 * 32;
  if (threads > 1024) return GB_EUNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(rows * p.split));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (gb_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (p.split > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)p.split; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  gb_count_launch();
  if constexpr (kMode == 0) {
    GB_CUDA_OK(cudaLaunchKernelEx(&cfg, fp4_rows_kernel<1, kMode>, p));
  } else {
    switch (per) {
      case 1: GB_CUDA_OK(cudaLaunchKernelEx(&cfg, fp4_rows_kernel<1, kMode>, p)); break;
      case 2: GB_CUDA_OK(cudaLaunchKernelEx(&cfg, fp4_rows_kernel<2, kMode>, p)); break;
      default: GB_CUDA_OK(cudaLaunchKernelEx(&cfg, fp4_rows_kernel<kRowsMaxGroups, kMode>, p)); break;
    }
  }
  return GB_OK;
}

int64_t align256(int64_t v) { return (v + 255) & ~255ll; }

}  // namespace

int gb_prepare_gemv_fp4() {
#define GB_FP4_ATTR1(G, W, F) GB_CUDA_OK(cudaFuncSetAttribute((const void*)fp4_decode_kernel<G, W, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax))
#define GB_FP4_ATTR(F) GB_FP4_ATTR1(false, false, F); GB_FP4_ATTR1(false, true, F); GB_FP4_ATTR1(true, false, F); GB_FP4_ATTR1(true, true, F)
  GB_FP4_ATTR(kLit);
  GB_FP4_ATTR(12);
  GB_FP4_ATTR(16);
  GB_FP4_ATTR(20);
  GB_FP4_ATTR(24);
#undef GB_FP4_ATTR
#undef GB_FP4_ATTR1
  return GB_OK;
}

// Whether the kernel takes the weight (any row count; 64 rows per launch).
bool gb_gemv_fp4_applies(const gb_weight* w, bool scales_e4m3) {
  return fp4_format(w, scales_e4m3) >= 0 && w->rows >= 64 && w->K / 16 <= 1024 * kRowsMaxGroups;
}

// The operand of up to 64 rows, the rows' scales, the scales of groups left out.
int64_t gb_gemv_fp4_workspace_bytes(int64_t M, int64_t K) {
  const int rows = (int)(M > kMaxRows ? kMaxRows : M);
  return align256((K / 256) * unit_bytes(is_wide(rows), rows)) + align256(rows * 4) + align256(rows * (K / 16) * 4);
}

namespace {
// y_i[M, N_i] for matrices of one format and width: the rows' operand once, then one launch.  Roles: of a single matrix.
int gemv_fp4(const void* x, int64_t M, const gb_weight* const* w, int n_mat, bool scales_e4m3, int n_roles, const int64_t* role_rows,
             int scale_rule, void* const* y, void* workspace, int64_t workspace_bytes, void* stream_) {
  const int F = fp4_format(w[0], scales_e4m3);
  const int sms = gb_sm_count();
  if (sms <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  if (workspace == nullptr || workspace_bytes < gb_gemv_fp4_workspace_bytes(M, w[0]->K))
    return gb_fail(GB_EWORKSPACE, "workspace of %lld bytes is too small (need %lld)", (long long)workspace_bytes,
                   (long long)gb_gemv_fp4_workspace_bytes(M, w[0]->K));
  cudaStream_t stream = (cudaStream_t)stream_;
  const int64_t K = w[0]->K;
  Maps maps;
  for (int i = 0; i < n_mat; ++i) {
    const Info f = info(F, false);                         // the packed rows are read alike
    const int rc = gb_tensor_map_bytes_2d(&maps.m[i], w[i]->qw, (uint64_t)(K / 256) * f.sb, (uint64_t)w[i]->rows, (uint64_t)w[i]->row_stride, f.pitch, kBM);
    if (rc != GB_OK) return rc;
  }
  for (int i = n_mat; i < kMaxMatrices; ++i) maps.m[i] = maps.m[0];
  for (int64_t m0 = 0; m0 < M; m0 += kMaxRows) {
    Fp4Params p = {};
    p.K = K;
    p.M = (int)(M - m0 < kMaxRows ? M - m0 : kMaxRows);
    p.n_sb = (int)(K / 256);
    p.pass_rows = p.M;
    p.x_unit = unit_bytes(is_wide(p.M), p.M);
    p.xop = (const uint8_t*)workspace;
    p.x_scale = (const float*)((const uint8_t*)workspace + align256(p.n_sb * p.x_unit));
    p.tail = (const float*)((const uint8_t*)p.x_scale + align256(p.M * 4));
    p.status = gb_status_word();
    for (int i = 0; i < n_mat; ++i) {
      p.mat[i] = {w[i]->qw, w[i]->row_stride, w[i]->rows, w[i]->codebook, w[i]->compose, w[i]->global_scale == 0.0f ? 1.0f : w[i]->global_scale,
                  (uint16_t*)y[i] + m0 * w[i]->rows};
      int64_t row = 0;
      for (int r = 0; r < (n_roles < 1 ? 1 : n_roles); ++r) {
        const int64_t rows = n_roles < 1 ? w[i]->rows : role_rows[r];
        p.role[p.n_roles++] = {i, (int)row, (int)rows, p.n_tiles, r * gb_codebook_elems(w[i]->fmt)};
        p.n_tiles += (int)((rows + kBM - 1) / kBM);
        row += rows;
      }
      GB_REQUIRE(row == w[i]->rows, "the roles hold %lld rows, the matrix %lld", (long long)row, (long long)w[i]->rows);
    }
    const Info f = info(F, is_wide(p.M));
    // K slices: enough CTAs for the SMs when there are few tiles; no more clusters than run at once,
    // at least two superblocks per slice
    int want = 1;
    for (int s = 2; s <= kMaxSlices && p.n_tiles * s <= sms && s * 2 <= p.n_sb; ++s)
      if (p.n_tiles <= max_clusters(s)) want = s;
    p.units = (p.n_sb + want - 1) / want;
    p.units = (p.units + f.per_stage - 1) / f.per_stage * f.per_stage;
    p.slices = (p.n_sb + p.units - 1) / p.units;
    if (!layout(f, p)) return gb_fail(GB_EUNSUPPORTED, "no shared-memory layout for %d rows", p.M);
    RowsParams rp = {};
    rp.x = (const uint4*)((const uint16_t*)x + m0 * K);
    rp.xop = (uint8_t*)workspace;
    rp.x_scale = const_cast<float*>(p.x_scale);
    rp.tail = const_cast<float*>(p.tail);
    rp.x_unit = p.x_unit;
    rp.K = (int)K; rp.n_sb = p.n_sb; rp.scale_rule = scale_rule; rp.pass_rows = p.pass_rows; rp.rows = p.M;
    const int rc = launch_rows<0>(p.M, K, stream, rp);
    if (rc != GB_OK) return rc;
    const int ctas = p.slices > 1 || p.n_tiles <= sms ? p.n_tiles : sms;
    GB_CUDA_OK(launch<false>(F, dim3((unsigned)ctas, (unsigned)p.slices), stream, maps, p));
  }
  return GB_OK;
}
}  // namespace

int gb_gemv_fp4(const void* x, int64_t M, const gb_weight* w, bool scales_e4m3, int n_roles, const int64_t* role_rows,
                int scale_rule, void* y, void* workspace, int64_t workspace_bytes, void* stream) {
  if (fp4_format(w, scales_e4m3) < 0 || ((uintptr_t)x & 15u) != 0 || n_roles > kMaxRoles || (n_roles <= 1 && w->cb_row_offset != nullptr))
    return GB_EUNSUPPORTED;
  return gemv_fp4(x, M, &w, 1, scales_e4m3, n_roles, role_rows, scale_rule, &y, workspace, workspace_bytes, stream);
}

// ---- routed experts ------------------------------------------------------------------------------
namespace {

// Every scale of the two-tier weight an exact positive E4M3 value?  Raises *flag otherwise.
__global__ void __launch_bounds__(256)
scales_exact_kernel(const uint8_t* qw, int64_t row_stride, int64_t rows, int n_sb, int type_size, int super_at,
                    const float* compose, int* flag) {
  __shared__ uint8_t bad[256];
  {
    bool ok = true;
    for (int i = 0; i < 16; ++i) {
      const float v = compose[threadIdx.x * 16 + i];
      ok &= v >= 0.0f && v <= 448.0f && gb_e4m3_to_f32(gb_f32_to_e4m3(fminf(v, 448.0f))) == v;
    }
    bad[threadIdx.x] = ok ? 0 : 1;
  }
  __syncthreads();
  bool any = false;
  const int64_t units = rows * n_sb;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = u / n_sb;
    any |= bad[qw[r * row_stride + (u - r * n_sb) * type_size + super_at]] != 0;
  }
  if (any) *flag = 1;
}

// Rows per pass of a grouped launch: more rows per pass decode the weights less often, fewer leave
// room for more accumulators and deeper rings.  From the average number of rows per expert.
int pass_rows_for(int F, int64_t P, int64_t E) {
  const int64_t avg = P / (E > 0 ? E : 1);
  if (F == 20 || F == 24) return 16;                       // their tables leave no more room
  return avg <= 8 ? 16 : avg <= 24 ? 32 : 64;
}

}  // namespace

extern "C" {

int gb_scales_e4m3(const gb_weight* w, int64_t rows, int32_t* flag, void* stream) {
  int rc = gb_check_weight(w);
  if (rc != GB_OK) return rc;
  GB_REQUIRE(flag != nullptr && w->compose != nullptr && rows >= 1, "gb_scales_e4m3 wants a two-tier weight and a flag");
  const int sms = gb_sm_count();
  if (sms <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  GB_CUDA_OK(cudaMemsetAsync(flag, 0, sizeof(int32_t), (cudaStream_t)stream));
  gb_count_launch();
  scales_exact_kernel<<<sms * 4, 256, 0, (cudaStream_t)stream>>>(w->qw, w->row_stride, rows, (int)(w->K / 256), w->fmt.type_size,
                                                                 4 * w->fmt.k_bits, w->compose, flag);
  GB_LAUNCH_OK("scales_exact_kernel");
  return GB_OK;
}

int gb_gemv_hinted(const void* x, int64_t M, const gb_weight* w, const gb_hints* hints, int scale_rule, void* y,
                   void* workspace, int64_t workspace_bytes, void* stream) {
  int rc = gb_check_weight(w);
  if (rc != GB_OK) return rc;
  GB_REQUIRE(x && y && hints, "null pointer argument");
  GB_REQUIRE(M >= 1 && M <= 128, "decode-batch kernels take 1..128 rows, got M=%lld", (long long)M);
  GB_REQUIRE(hints->n_roles >= 0 && hints->n_roles <= GB_MAX_ROLES, "%d roles", hints->n_roles);
  const int act = w->fmt.grid == GB_GRID_FP4 ? GB_ACT_FP4_GROUP16 : GB_ACT_FP8_TOKEN;
  if (act == GB_ACT_FP4_GROUP16 && gb_gemv_fp4_applies(w, hints->scales_e4m3 != 0)) {
    rc = gb_gemv_fp4(x, M, w, hints->scales_e4m3 != 0, hints->n_roles, hints->role_rows, scale_rule, y, workspace,
                     workspace_bytes, stream);
    if (rc != GB_EUNSUPPORTED) return rc;
  }
  if (hints->n_roles > 1) {                                // parts with their own codebook: the per-row offsets alone hide them
    rc = gb_gemv_umma(x, M, w, hints->n_roles, hints->role_rows, act, scale_rule, y, workspace, workspace_bytes, stream);
    if (rc != GB_EUNSUPPORTED) return rc;
  }
  return gb_gemv(x, M, w, act, scale_rule, y, workspace, workspace_bytes, stream);
}

int gb_gemv_shared_applies(const gb_weight* const* w, int n_weights, int scales_e4m3) {
  if (w == nullptr || n_weights < 1 || n_weights > kMaxMatrices) return 0;
  for (int i = 0; i < n_weights; ++i)
    if (gb_check_weight(w[i]) != GB_OK || w[i]->K != w[0]->K || !gb_gemv_fp4_applies(w[i], scales_e4m3 != 0) ||
        fp4_format(w[i], scales_e4m3 != 0) != fp4_format(w[0], scales_e4m3 != 0) || w[i]->cb_row_offset != nullptr)
      return 0;
  return 1;
}

int gb_gemv_shared(const void* x, int64_t M, const gb_weight* const* w, int n_weights, int scales_e4m3, int scale_rule, void* const* y,
                   void* workspace, int64_t workspace_bytes, void* stream) {
  GB_REQUIRE(x && w && y, "null pointer argument");
  GB_REQUIRE(n_weights >= 1 && n_weights <= kMaxMatrices, "1..%d matrices per call, got %d", kMaxMatrices, n_weights);
  GB_REQUIRE(M >= 1 && M <= 128, "decode-batch kernels take 1..128 rows, got M=%lld", (long long)M);
  for (int i = 0; i < n_weights; ++i) {
    const int rc = gb_check_weight(w[i]);
    if (rc != GB_OK) return rc;
    GB_REQUIRE(y[i] != nullptr, "null output %d", i);
    GB_REQUIRE(w[i]->K == w[0]->K, "matrix %d has K=%lld, matrix 0 K=%lld: they must read the same rows", i, (long long)w[i]->K, (long long)w[0]->K);
  }
  if (!gb_gemv_shared_applies(w, n_weights, scales_e4m3) || ((uintptr_t)x & 15u) != 0) return GB_EUNSUPPORTED;
  return gemv_fp4(x, M, w, n_weights, scales_e4m3 != 0, 0, nullptr, scale_rule, y, workspace, workspace_bytes, stream);
}

int gb_moe_fp4_pass_rows(const gb_weight* w, int scales_e4m3, int64_t P, int64_t E) {
  if (gb_check_weight(w) != GB_OK) return 0;
  const int F = fp4_format(w, scales_e4m3 != 0);
  if (F < 0 || w->cb_row_offset != nullptr || w->rows % kBM != 0 || w->K / 16 > 1024 * kRowsMaxGroups) return 0;
  return pass_rows_for(F, P, E);
}

int64_t gb_moe_fp4_operand_bytes(int64_t P, int64_t E, int64_t K, int pass_rows) {
  if (pass_rows == 0) return gb_fp4_tiles(P, E, K).bytes;
  if (pass_rows < 1) return 0;
  const int64_t tiles = P / pass_rows + E + 1;
  return align256(tiles * (K / 256) * unit_bytes(is_wide(pass_rows), pass_rows)) + align256(tiles * scale_pitch(pass_rows) * 4) +
         align256(tiles * pass_rows * (K / 16) * 4);
}

static int rows_params(RowsParams* p, const void* x, int64_t P, int64_t E, int64_t K, int pass_rows, const int32_t* ids,
                       const int32_t* seg, int scale_rule, void* operand) {
  GB_REQUIRE(x && ids && seg && operand, "null pointer argument");
  GB_REQUIRE(P >= 1 && P < (1ll << 30) && E >= 1 && K > 0 && K % 256 == 0 && pass_rows >= 0 && pass_rows <= kMaxRows,
             "bad shape P=%lld E=%lld K=%lld", (long long)P, (long long)E, (long long)K);
  GB_REQUIRE(((uintptr_t)x & 15u) == 0 && ((uintptr_t)operand & 255u) == 0, "rows must be 16-byte aligned, the operand 256-byte");
  p->x = (const uint4*)x;
  p->xop = (uint8_t*)operand;
  if (pass_rows == 0) {
    const GbFp4Tiles op = gb_fp4_tiles(P, E, K);
    p->sf = (uint8_t*)operand + op.sf_at;
    p->x_scale = (float*)((uint8_t*)operand + op.scale_at);
    p->tail = (float*)((uint8_t*)operand + op.tail_at);
    pass_rows = 64;
  } else {
    const int64_t tiles = P / pass_rows + E + 1;
    p->x_unit = unit_bytes(is_wide(pass_rows), pass_rows);
    p->x_scale = (float*)((uint8_t*)operand + align256(tiles * (K / 256) * p->x_unit));
    p->tail = (float*)((uint8_t*)p->x_scale + align256(tiles * scale_pitch(pass_rows) * 4));
  }
  p->K = (int)K; p->n_sb = (int)(K / 256); p->scale_rule = scale_rule; p->pass_rows = pass_rows;
  p->ids = ids; p->seg = seg; p->E = (int)E;
  return GB_OK;
}

int gb_moe_fp4_rows(const void* x, const int32_t* ids, const int32_t* inv, const int32_t* seg, int64_t T, int64_t topk,
                    int64_t E, int64_t K, int pass_rows, int scale_rule, void* operand, void* stream) {
  RowsParams p = {};
  int rc = rows_params(&p, x, T * topk, E, K, pass_rows, ids, seg, scale_rule, operand);
  if (rc != GB_OK) return rc;
  GB_REQUIRE(inv != nullptr, "null pointer argument");
  p.inv = inv; p.topk = (int)topk;
  return launch_rows<1>(T, K, (cudaStream_t)stream, p);
}

int gb_moe_fp4_swiglu_rows(const void* h, const int32_t* ids, const int32_t* order, const int32_t* seg, int64_t P, int64_t E,
                           int64_t inter, int pass_rows, int scale_rule, void* operand, void* stream) {
  RowsParams p = {};
  int rc = rows_params(&p, h, P, E, inter, pass_rows, ids, seg, scale_rule, operand);
  if (rc != GB_OK) return rc;
  GB_REQUIRE(order != nullptr, "null pointer argument");
  p.order = order;
  return launch_rows<2>(P, inter, (cudaStream_t)stream, p);
}

int gb_moe_gemv_fp4(const void* operand, const gb_weight* w, int scales_e4m3, int64_t expert_stride, int64_t E,
                    const int32_t* seg, const int32_t* row_map, int64_t P, int pass_rows, void* y, void* stream_) {
  GB_REQUIRE(operand && w && seg && y, "null pointer argument");
  GB_REQUIRE(P >= 1 && P < (1ll << 30) && E >= 1 && pass_rows >= 1 && pass_rows <= kMaxRows, "bad shape P=%lld E=%lld, %d rows per pass",
             (long long)P, (long long)E, pass_rows);
  int rc = gb_check_weight(w);
  if (rc != GB_OK) return rc;
  const int64_t N = w->rows, K = w->K;
  const int F = fp4_format(w, scales_e4m3 != 0);
  if (F < 0 || gb_moe_fp4_pass_rows(w, scales_e4m3, P, E) < pass_rows || expert_stride != N * w->row_stride || E * N >= (1ll << 31))
    return gb_fail(GB_EUNSUPPORTED, "not a stack the fp4 expert kernel takes");
  const int sms = gb_sm_count();
  if (sms <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  const Info f = info(F, is_wide(pass_rows));
  const int64_t tiles = P / pass_rows + E + 1;
  Fp4Params p = {};
  p.K = K; p.n_sb = (int)(K / 256); p.units = p.n_sb; p.slices = 1;
  p.pass_rows = pass_rows;
  p.x_unit = unit_bytes(is_wide(pass_rows), pass_rows);
  p.xop = (const uint8_t*)operand;
  p.x_scale = (const float*)((const uint8_t*)operand + align256(tiles * p.n_sb * p.x_unit));
  p.tail = (const float*)((const uint8_t*)p.x_scale + align256(tiles * scale_pitch(pass_rows) * 4));
  p.mat[0] = {w->qw, w->row_stride, N, w->codebook, w->compose, w->global_scale == 0.0f ? 1.0f : w->global_scale, (uint16_t*)y};
  p.status = gb_status_word();
  p.n_roles = 1;
  p.seg = seg; p.row_map = row_map;
  p.tiles_n = (int)(N / kBM);
  p.n_tiles = (int)(E * p.tiles_n);
  p.E = (int)E;
  if (!layout(f, p)) return gb_fail(GB_EUNSUPPORTED, "no shared-memory layout for %d rows per pass", pass_rows);
  Maps maps;
  rc = gb_tensor_map_bytes_2d(&maps.m[0], w->qw, (uint64_t)p.n_sb * f.sb, (uint64_t)(E * N), (uint64_t)w->row_stride, f.pitch, kBM);
  if (rc != GB_OK) return rc;
  for (int i = 1; i < kMaxMatrices; ++i) maps.m[i] = maps.m[0];
  GB_CUDA_OK(launch<true>(F, dim3((unsigned)(p.n_tiles < sms ? p.n_tiles : sms)), (cudaStream_t)stream_, maps, p));
  return GB_OK;
}

}  // extern "C"
