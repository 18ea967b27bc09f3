// Prefill GEMMs on CTA pairs: D[M,N] = A[M,K] . B[N,K]^T, both operands K-major, bf16 (kind::f16),
// E4M3 (kind::f8f6f4) or block-scaled E2M1 (kind::mxf4nvf4, UE4M3 scale factors per sixteen), fp32
// accumulators in tensor memory, scaled bf16 epilogue.
//
// A single CTA's 128 x 256 tile takes 48 KiB of operands per 128-byte K slab into shared memory and
// reads them out again for the tensor core: 192 bytes a clock at the full fp8 or fp4 rate, more than
// the 128 that shared memory moves, and 28 TB/s out of L2 over the GPU.  A pair (tcgen05
// cta_group::2) works on a 256 x 256 tile together: each CTA loads its own 128 rows of A and its own
// half of the B rows, the tensor cores exchange the B halves, and a slab is 32 KiB per CTA for the
// same work.  Every CTA fetches its own operands (the pair's loads report to the leader's barriers).
//
// The pair walks output tiles persistently.  Warps 0-7 drain the CTA's own 128 rows, warp 8 of each CTA
// loads, warp 9 of the leader issues the MMAs of both tensor cores; two accumulators, so that draining
// overlaps the next tile.
//
// The fp4 form has one accumulator: the columns beside it hold five or six sets of scale factors, which
// warps 10-13 of the leader copy from both CTAs' shared memory (tcgen05.cp, one warp per MMA of a stage)
// that many stages ahead of the MMAs: a stage needs twelve copies, and from one warp they took longer than the
// stage's MMAs (8192 x 34816 x 5120, issued as one lane's code: 759 us with one warp, 647 with two, 635 with four,
// 559 with none at all).  The accumulator is drained into
// registers in one go, so that the next tile's MMAs start early.
//
// Measured, us, one CTA per tile -> pairs, launches back to back (N x K of the four linears of a 5120-wide layer;
// lowest and highest of three runs on different boxes, which differ in what the power cap leaves):
//   fp8, 8192 rows: 34816 x 5120 1434 -> 1081..1247, 5120 x 17408 729 -> 544..558, 6144 x 5120 263 -> 200..205, 2048 x 5120 101 -> 83..94
//   fp8, 2048 rows: 370 -> 278..281, 218 -> 167..187, 80 -> 56..68, 36 -> 26..32
//   fp4, 8192 rows: 960 -> 604..624, 437 -> 295..390, 184 -> 114..138, 66 -> 49..55
//   fp4, 2048 rows: 253 -> 159..191, 145 -> 102..133, 54 -> 34..43, 21 -> 15..21
// The fp8 gate_up at 8192 rows under a profiler: 2.7 PFLOP/s, tensor pipe 79% busy at the 1.45 GHz that the power cap leaves.
#include "gb_common.cuh"

#include <cuda.h>
#include <mutex>

namespace {

enum Kind { kBf16 = 0, kFp8 = 1, kFp4 = 2 };

constexpr int kPairM = 256, kBM = 128;               // rows of a tile, rows of a CTA
constexpr int kSlabBytes = 128;                      // K bytes per row and stage (one swizzle span)
constexpr int kTmemCols = 512;
constexpr int kEpiWarps = 8;                         // two per lane quarter, half of the columns each
constexpr int kOutChunk = 2048;                      // 32 rows x 32 bf16 columns on their way out
constexpr int kMaxGroups = 1024;                     // experts of one grouped launch
constexpr int kTileRows = 64;                        // grouped: activation rows of a tile, three columns each
constexpr int kGroupM = 16;                          // row tiles walked together before the next columns

template <Kind kKind, int kBN, bool kGrouped = false>
struct Shape {
  static constexpr int kABytes = kBM * kSlabBytes;
  static constexpr int kBBytes = kBN / 2 * kSlabBytes;
  static constexpr int kAtoms = 2048;                                    // scale bytes of 128 rows x 16 groups
  static constexpr int kSfBytes = kKind == kFp4 ? 3 * kAtoms : 0;        // A's rows, two 128-row groups of B
  static constexpr int kStageBytes = kABytes + kBBytes + kSfBytes;
  // output chunks on their way out; grouped: segment offsets and the prefix of the row tiles
  static constexpr int kOutBytes = kGrouped ? 2 * (kMaxGroups + 1) * 4 + 8 : kEpiWarps * 2 * kOutChunk;
  static constexpr int kStages = (227 * 1024 - 2048 - kOutBytes) / kStageBytes;
  static constexpr int kSmem = kStages * kStageBytes + kOutBytes + 2048;
  static constexpr int kThreads = kKind == kFp4 ? 448 : 320;
  static constexpr int kAccs = kKind == kFp4 && !kGrouped ? 1 : 2;
  static constexpr uint32_t kAcc1 = kKind == kFp4 ? kBN : 256;           // column of the second accumulator
  static constexpr uint32_t kSf0 = kKind == kFp4 ? kAccs * kBN : 0;      // first column of the scale factors
  static constexpr uint32_t kSfCols = 48;                                // columns of a set: 16 of A, 32 of B
  static constexpr int kSets = kKind == kFp4 ? (kTmemCols - kAccs * kBN) / (int)kSfCols : 1;
};

struct PairParams {
  int64_t M, N, K;
  int k_tiles, m_tiles, n_tiles;
  uint32_t idesc;
  const float* a_scale;        // [M] or null
  const float* b_scale;        // [N] or null
  float global_scale;
  int out_tma;                 // rows of D are a multiple of 16 bytes
  uint16_t* D;
  int* status;
  // grouped: a tile is 256 weight rows of an expert times up to 64 of its activation rows
  const int32_t* seg;          // [E + 1]
  const int32_t* row_map;      // output row of a sorted row, or null
  const float* x_scale;        // [row tile][64]
  const float* tail;           // [row tile][64][K / 16], and the operands as they lie in memory: for groups left out
  const uint8_t *codes, *packed, *sf;
  int E;
};

GB_DEVINL uint32_t leader_addr(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
// An accumulator goes back from the epilogue warps of both CTAs to the leader's MMA issuer.  What the pair of arrive
// and wait hands over is tensor memory alone, so the tensor-memory fences order it and the arrive may be
// relaxed (the PTX pattern for tcgen05 instructions of different threads: tcgen05.ld, wait::ld,
// fence::before_thread_sync, arrive.relaxed.cluster | try_wait.relaxed.cluster or stronger,
// fence::after_thread_sync, tcgen05.mma) - at cluster scope on both sides, since the threads may be of different
// CTAs; so are the other waits that the peer's arrivals end.  An arrive that released would wait for the output stores in flight, once a tile: 4096 tokens of a routed layer 637 -> 664 us,
// 333 rows of a dense one 248 -> 254; one thread of the peer that collects its warps' arrives and releases them
// together: 640, 252.
GB_DEVINL void arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
template <bool kOfPair>
GB_DEVINL bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  if (kOfPair)
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  else
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// A bounded wait that remembers a timeout for the rest of the CTA: later waits return at once.
template <bool kOfPair>
__device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  uint64_t t0 = 0;
  for (uint32_t spin = 0; !*abort_flag; ++spin) {
    if (try_wait<kOfPair>(bar, parity)) return;
    if ((spin & 255u) == 255u) {
      const uint64_t now = gb_globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > 2000000000ull) { *abort_flag = 1; atomicExch(status, code); }
    }
  }
}
template <bool kOfPair = false>
GB_DEVINL void wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (!try_wait<kOfPair>(bar, parity)) wait_slow<kOfPair>(bar, parity, abort_flag, status, code);
}
// The same for a whole warp that goes on together; false: given up.
template <bool kOfPair = false>
GB_DEVINL bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (__all_sync(0xffffffffu, try_wait<kOfPair>(bar, parity))) return true;
  wait_slow<kOfPair>(bar, parity, abort_flag, status, code);
  return !__any_sync(0xffffffffu, *abort_flag != 0);
}
// A value that is the same in every lane, for a warp that walks its loop whole (gb_elect_one).
GB_DEVINL int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
// Tile load into this CTA's shared memory that reports to a barrier of the pair.
GB_DEVINL void tma_load_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
GB_DEVINL void expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
GB_DEVINL void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
// K-major operand tile stored as rows of 128 bytes with the 128-byte swizzle.
GB_DEVINL uint64_t desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(1024u >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// One scale-factor atom: 32 rows of 16 bytes, unswizzled, the 8-row groups 128 bytes apart; the copy
// repeats it in the four lane quarters of both CTAs' tensor memory, each from its own shared memory.
GB_DEVINL void sf_to_tmem(uint32_t tmem_col, uint32_t smem_addr) {
  const uint64_t d = (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(16u >> 4) << 16 | (uint64_t)(128u >> 4) << 32 | (uint64_t)1 << 46;
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_col), "l"(d) : "memory");
}
template <Kind kKind>
GB_DEVINL void mma_pair(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sfa, uint32_t sfb, bool accumulate) {
  if (kKind == kFp4)
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n}\n"
        ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate), "r"(sfa), "r"(sfb) : "memory");
  else if (kKind == kFp8)
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
  else
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
// Completion of the MMAs (or copies) issued so far, told to a barrier of either CTA.
GB_DEVINL void commit_to(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
GB_DEVINL void commit_pair(uint32_t bar, uint32_t to_peer) {
  commit_to(bar);
  commit_to(bar + to_peer);
}
GB_DEVINL void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}

// 32 accumulator columns of one output row, scaled and rounded to bf16 pairs.
template <bool kColScale>
GB_DEVINL void pack_chunk(const PairParams& p, const uint32_t (&v)[32], uint32_t* w, float rs, int col0) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float lo = __uint_as_float(v[2 * j]) * rs, hi = __uint_as_float(v[2 * j + 1]) * rs;
    if (kColScale && p.b_scale) {
      const int c = col0 + 2 * j;
      lo *= c < (int)p.N ? p.b_scale[c] : 0.0f;
      hi *= c + 1 < (int)p.N ? p.b_scale[c + 1] : 0.0f;
    }
    w[j] = gb_pack_bf16x2(lo, hi);
  }
}

// Output tile of a step: groups of kGroupM row tiles, inside a group the rows fastest.  The pairs that
// run together (74) then share sixteen row tiles of A and about five column tiles of B, which stay in L2
// while the group sweeps N (rows fastest over all of M re-read a 142 MB activation matrix from HBM for
// every two or three columns of tiles).  8192 x 34816 x 5120 fp8 / fp4: groups of 4 1111 / 687 us, 8
// 1065 / 652, 16 1041 / 632.
GB_DEVINL void tile_at(const PairParams& p, int tile, int& mt, int& nt) {
  const int per = kGroupM * p.n_tiles, g = tile / per, in = tile - g * per;
  const int rows = min(kGroupM, p.m_tiles - g * kGroupM);
  mt = g * kGroupM + in % rows;
  nt = in / rows;
}

// The tiles of a pair, first, first + stride, ..: first row of A, first row of B; grouped: the expert's weight row and
// its activation rows.  The expert is found by stepping on from the last tile's (a few experts per step of 74 tiles).
template <int kBN, bool kGrouped>
struct Tiles {
  int m0 = 0, n0 = 0, w0 = 0, lo = 0, rows = 0, x_tile = 0;
  int tile, gp = 0, mt = 0, e = 0;
  int step, step_gp = 0, step_mt = 0;
  GB_DEVINL Tiles(const PairParams& p, int first, int stride) : tile(first - stride), step(stride) {
    if (kGrouped) {                                          // the expert's weight tiles run fastest
      step_gp = stride / p.m_tiles;
      step_mt = stride - step_gp * p.m_tiles;
      gp = first / p.m_tiles;
      mt = first - gp * p.m_tiles;
      gp -= step_gp;
      mt -= step_mt;
      if (mt < 0) { mt += p.m_tiles; --gp; }
    }
  }
  GB_DEVINL bool next(const PairParams& p, int total, const int* seg_s, const int* base_s) {
    tile += step;
    if (tile >= total) return false;
    if (!kGrouped) {
      int tm, tn;
      tile_at(p, tile, tm, tn);
      m0 = tm * kPairM;
      n0 = tn * kBN;
      return true;
    }
    gp += step_gp;
    mt += step_mt;
    if (mt >= p.m_tiles) { mt -= p.m_tiles; ++gp; }
    while (base_s[e + 1] <= gp) ++e;                         // experts without rows are stepped over
    const int pass = gp - base_s[e], first_row = seg_s[e];
    w0 = mt * kPairM;
    m0 = e * (int)p.N + w0;
    lo = first_row + pass * kTileRows;
    rows = min(kTileRows, seg_s[e + 1] - lo);
    x_tile = first_row / kTileRows + e + pass;               // tiles of different (expert, pass) never coincide
    n0 = x_tile * kBN;
    return true;
  }
};

template <Kind kKind, int kBN, bool kGrouped>
__global__ void __launch_bounds__(Shape<kKind, kBN, kGrouped>::kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_d,
                 const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb, const PairParams p) {
  using S = Shape<kKind, kBN, kGrouped>;
  constexpr int kStages = S::kStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t ring = (gb_smem_u32(smem_raw) + 1023u) & ~1023u;        // the same offset in both CTAs
  uint8_t* ring_ptr = smem_raw + (ring - gb_smem_u32(smem_raw));
  const uint32_t out_ring = ring + kStages * S::kStageBytes;             // two chunks per epilogue warp
  const uint32_t full_bar = out_ring + (S::kOutBytes + 7) / 8 * 8;             // leader: both CTAs' operand tiles have landed
  const uint32_t empty_bar = full_bar + 8 * kStages;                     // the MMAs that read the stage are done
  const uint32_t acc_full = empty_bar + 8 * kStages;                     // [2] accumulator complete
  const uint32_t acc_empty = acc_full + 16;                              // [2] leader: drained by both CTAs
  const uint32_t sf_full = acc_empty + 16;                               // [kSets] leader: column set written in both CTAs
  const uint32_t sf_empty = sf_full + 8 * S::kSets;                      // [kSets] leader: the MMAs that read the set are done
  const uint32_t slot = sf_empty + 8 * S::kSets;
  volatile uint32_t* slot_ptr = reinterpret_cast<volatile uint32_t*>(ring_ptr + (slot - ring));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  gb_pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      bar_init(full_bar + 8 * s, 1);
      bar_init(empty_bar + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      bar_init(acc_full + 8 * b, 1);
      bar_init(acc_empty + 8 * b, 2 * kEpiWarps);
    }
    for (int t = 0; t < S::kSets; ++t) {
      bar_init(sf_full + 8 * t, 4);
      bar_init(sf_empty + 8 * t, 1);
    }
    *abort_flag = 0;
    gb_fence_barrier_init();
  }
  if (warp == kEpiWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"((uint32_t)kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  gb_cluster_sync();                                                        // both CTAs' barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *slot_ptr;
  gb_pdl_wait();
  int* seg_s = reinterpret_cast<int*>(ring_ptr + (out_ring - ring));
  int* base_s = seg_s + kMaxGroups + 1;                                  // row tiles in front of an expert
  if (kGrouped) {
    if (warp == 0) {
      int carry = 0;
      for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        const int lo = e < p.E ? p.seg[e] : 0, hi = e < p.E ? p.seg[e + 1] : 0;
        const int tiles = (hi - lo + kTileRows - 1) / kTileRows;
        int incl = tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (e < p.E) {
          seg_s[e] = lo;
          base_s[e] = carry + incl - tiles;
          if (e == p.E - 1) { seg_s[p.E] = hi; base_s[p.E] = carry + incl; }
        }
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    __syncthreads();
  }
  const int total_tiles = kGrouped ? base_s[p.E] * p.m_tiles : p.m_tiles * p.n_tiles;
  const int stride = (int)(gridDim.x >> 1), first = (int)(blockIdx.x >> 1);
  const int my_tiles = total_tiles > first ? (total_tiles - first + stride - 1) / stride : 0;

  if (warp == kEpiWarps) {
    // ------------------------------- producer (each CTA) -------------------------------
    constexpr int slab_elems = kKind == kBf16 ? kSlabBytes / 2 : kSlabBytes;   // E2M1 pairs and E4M3 go by bytes
    const uint32_t full_pair = (uint32_t)uniform((int)leader_addr(full_bar));
    const int me = uniform((int)rank);
    const bool one = gb_elect_one();
    int s = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (Tiles<kBN, kGrouped> T(p, first, stride); ok && T.next(p, total_tiles, seg_s, base_s);) {
      const int m0 = uniform(T.m0) + me * kBM, n0 = uniform(T.n0), x_tile = uniform(T.x_tile);
      for (int kt = 0; kt < p.k_tiles; ++kt) {
        ok = warp_wait<true>(empty_bar + 8 * s, ph, abort_flag, p.status, 71);
        if (!ok) break;
        if (one) {
          const uint32_t st = ring + (uint32_t)s * S::kStageBytes;
          if (me == 0) expect_tx(full_bar + 8 * s, 2 * S::kStageBytes);
          tma_load_pair(st, &map_a, kt * slab_elems, m0, full_pair + 8 * s);
          if (kGrouped) {                                    // 32 rows: codes of q for hi and for lo, of the correction
            const uint32_t b = st + S::kABytes;
            const int r0 = x_tile * 2 * kTileRows + me * 32;
            tma_load_pair(b, &map_b, kt * slab_elems, r0, full_pair + 8 * s);
            tma_load_pair(b + 4096, &map_b, kt * slab_elems, r0, full_pair + 8 * s);
            tma_load_pair(b + 8192, &map_b, kt * slab_elems, r0 + kTileRows, full_pair + 8 * s);
          } else {
            tma_load_pair(st + S::kABytes, &map_b, kt * slab_elems, n0 + me * (kBN / 2), full_pair + 8 * s);
          }
          if (kKind == kFp4) {                               // row groups past the end read zero
            const uint32_t sf = st + S::kABytes + S::kBBytes;
            tma_load_pair(sf, &map_sfa, 0, (m0 / 128 * p.k_tiles + kt) * 8, full_pair + 8 * s);
            tma_load_pair(sf + S::kAtoms, &map_sfb, 0, (n0 / 128 * p.k_tiles + kt) * 8, full_pair + 8 * s);
            tma_load_pair(sf + 2 * S::kAtoms, &map_sfb, 0, ((n0 / 128 + 1) * p.k_tiles + kt) * 8, full_pair + 8 * s);
          }
        }
        __syncwarp();
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == kEpiWarps + 1) {
    // --------------------------- MMA issuer (the leader's) ------------------------------
    if (uniform((int)rank) == 0) {
      uint32_t to_peer;                                      // distance of the peer's barriers
      asm volatile("mapa.shared::cluster.u32 %0, %1, 1;" : "=r"(to_peer) : "r"(full_bar));
      to_peer = (uint32_t)uniform((int)(to_peer - full_bar));
      const uint32_t tmem = (uint32_t)uniform((int)tmem_base);
      const int tiles = uniform(my_tiles);
      const bool one = gb_elect_one();
      int s = 0, set = 0;
      uint32_t ph = 0, sf_ph = 0;
      bool ok = true;
      Tiles<kBN, kGrouped> T(p, first, stride);
      for (int it = 0; ok && it < tiles; ++it) {
        const int buf = S::kAccs == 2 ? it & 1 : 0;
        const uint32_t use = (uint32_t)(S::kAccs == 2 ? it >> 1 : it);
        bool shifted = false;
        if (kKind == kFp4 && kBN % 128 != 0) {
          T.next(p, total_tiles, seg_s, base_s);
          shifted = uniform(T.n0) % 128 != 0;
        }
        ok = warp_wait<true>(acc_empty + 8 * buf, (use & 1) ^ 1, abort_flag, p.status, 72);   // its last tile is drained
        if (!ok) break;
        const uint32_t acc = tmem + (buf ? S::kAcc1 : 0u);
        for (int kt = 0; kt < p.k_tiles; ++kt) {
          ok = kKind == kFp4 ? warp_wait(sf_full + 8 * set, sf_ph, abort_flag, p.status, 73)
                             : warp_wait(full_bar + 8 * s, ph, abort_flag, p.status, 74);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t st = ring + (uint32_t)s * S::kStageBytes;
          const uint64_t da = desc_sw128(st), db = desc_sw128(st + S::kABytes);
          // 192 columns start in the middle of a 128-row group every other time: two columns on
          const uint32_t sfa_t = tmem + S::kSf0 + S::kSfCols * set, sfb_t = sfa_t + 16u + (shifted ? 2u : 0u);
          if (one) {
#pragma unroll
            for (int k = 0; k < 4; ++k)                      // 32 bytes of K per instruction
              mma_pair<kKind>(acc, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), p.idesc, sfa_t + 4u * k, sfb_t + 8u * k,
                              kt > 0 || k > 0);
            commit_pair(empty_bar + 8 * s, to_peer);
            if (kKind == kFp4) commit_to(sf_empty + 8 * set);
          }
          __syncwarp();
          if (kKind == kFp4 && ++set == S::kSets) { set = 0; sf_ph ^= 1; }
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
        if (ok && one) commit_pair(acc_full + 8 * buf, to_peer);
        __syncwarp();
      }
    }
  } else if (warp >= kEpiWarps + 2) {
    // ------------ scale factors -> tensor memory (the leader's, fp4): warp k the k-th MMA's ------------
    const uint32_t k = (uint32_t)(uniform(warp) - kEpiWarps - 2);
    if (uniform((int)rank) == 0) {
      const uint32_t tmem = (uint32_t)uniform((int)tmem_base);
      const bool one = gb_elect_one();
      int s = 0, set = 0;
      uint32_t ph = 0, sf_ph = 1;
      const int total = uniform(my_tiles) * p.k_tiles;
      for (int g = 0; g < total; ++g) {
        if (!warp_wait(full_bar + 8 * s, ph, abort_flag, p.status, 75) || !warp_wait(sf_empty + 8 * set, sf_ph, abort_flag, p.status, 76)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sf = ring + (uint32_t)s * S::kStageBytes + S::kABytes + S::kBBytes;
        const uint32_t col = tmem + S::kSf0 + S::kSfCols * set;
        if (one) {
          sf_to_tmem(col + 4u * k, sf + 512u * k);
          sf_to_tmem(col + 16u + 8u * k, sf + S::kAtoms + 512u * k);
          sf_to_tmem(col + 20u + 8u * k, sf + 2 * S::kAtoms + 512u * k);
          commit_to(sf_full + 8 * set);
        }
        __syncwarp();
        if (++set == S::kSets) { set = 0; sf_ph ^= 1; }
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp < kEpiWarps) {
    // ------------------------------- epilogue (each CTA) --------------------------------
    // The warp's columns go into registers, scaled and rounded, before anything is stored: the MMAs of the
    // next tile (fp4) wait for them.  Then out through shared memory, 32 x 32 values a TMA store; rows of
    // 16-byte pieces straight from the registers reach L2 as half-written sectors.
    const uint32_t acc_empty_pair = leader_addr(acc_empty);
    constexpr int kCols = kBN / 2, kChunks = kCols / 32;
    const int quarter = warp & 3, c_lo = (warp >> 2) * kCols;
    const uint32_t out = out_ring + (uint32_t)warp * 2 * kOutChunk;
    int it = 0, flip = 0;
    if constexpr (kGrouped) {
      // Lane = weight row, i.e. output feature; column 96 h + 32 t + i = term t of activation row 32 h + i.  A
      // warp takes its half's three terms, adds them and stores 64 contiguous bytes per activation row.
      const int half = warp >> 2;
      for (Tiles<kBN, kGrouped> T(p, first, stride); T.next(p, total_tiles, seg_s, base_s); ++it) {
        const int buf = S::kAccs == 2 ? it & 1 : 0, w = T.w0 + (int)rank * kBM + quarter * 32 + lane, m = half * 32 + lane;
        const float xs = m < T.rows ? p.x_scale[(int64_t)T.x_tile * kTileRows + m] : 0.0f;
        const int to = m < T.rows ? (p.row_map ? p.row_map[T.lo + m] : T.lo + m) : 0;
        wait<true>(acc_full + 8 * buf, (uint32_t)(S::kAccs == 2 ? it >> 1 : it) & 1, abort_flag, p.status, 77);
        if (__any_sync(0xffffffffu, *abort_flag)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t at = tmem_base + ((uint32_t)(quarter * 32) << 16) + (buf ? S::kAcc1 : 0u) + (uint32_t)(half * 96);
        if (__builtin_expect(__any_sync(0xffffffffu, __float_as_uint(xs) & kGbLeftOutBits), 0)) {
          // groups left out: added to the sums in tensor memory
          const int64_t w_row = T.m0 - T.w0 + min(w, (int)p.N - 1);
          const uint8_t* wp = p.packed + w_row * (p.K / 2);
          const uint8_t* sf = p.sf + (w_row >> 7) * (p.K * 8) + (w_row & 31) * 16 + (w_row >> 5 & 3) * 4;
          const int n_sb = (int)(p.K / 256), per = gb_left_out_span(n_sb);
          struct Raw { uint2 c; float scale; };
#pragma unroll 1
          for (int i0 = 0; i0 < 32; i0 += 4) {
            uint32_t word[4], bits = 0u, marked = 0u;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              word[r] = __float_as_uint(__shfl_sync(0xffffffffu, xs, i0 + r));
              bits |= word[r] & kGbLeftOutBits;
              marked |= (word[r] & kGbLeftOutBits) != 0 ? 1u << r : 0u;
            }
            if (bits == 0) continue;
            const int64_t m0 = (int64_t)T.x_tile * kTileRows + half * 32 + i0;
            const uint8_t* codes = p.codes + (m0 + (int64_t)T.x_tile * kTileRows) * (p.K / 2);
            float add[4] = {};
#pragma unroll 1
            for (; bits != 0; bits &= bits - 1) {
              const int b = __ffs(bits) - 1;
              gb_left_out(
                  add, p.tail + m0 * (p.K / 16), p.K / 16, marked, b * per * 16, min((b + 1) * per, n_sb) * 16,
                  [&](int r, int g) { return *reinterpret_cast<const uint2*>(codes + r * (p.K / 2) + g * 8); },
                  [&](int g) { return Raw{*reinterpret_cast<const uint2*>(wp + g * 8), gb_e4m3_to_f32(sf[(g >> 2) * 512 + (g & 3)])}; },
                  [](const Raw& q, float x) {
                    float s = 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                      const float2 v = gb_e2m1x2_to_f32((j < 4 ? q.c.x : q.c.y) >> (8 * (j & 3)) & 0xFFu);
                      s = fmaf(__shfl_sync(0xffffffffu, x, 2 * j), v.x, s);
                      s = fmaf(__shfl_sync(0xffffffffu, x, 2 * j + 1), v.y, s);
                    }
                    return s * q.scale;
                  });
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) add[r] = gb_normalised(add[r], word[r]);
            gb_tmem_add(at + (uint32_t)i0, add);
          }
        }
        uint32_t hi[32], lo[32], dl[32];
        tmem_ld32(at, hi);
        tmem_ld32(at + 32u, lo);
        tmem_ld32(at + 64u, dl);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive_cluster(acc_empty_pair + 8 * buf);
        const int n = T.rows - half * 32;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float v = fmaf(__uint_as_float(dl[i]), 0x1p-7f, fmaf(__uint_as_float(lo[i]), 0x1p-4f, __uint_as_float(hi[i])));
          const float r = v * __uint_as_float(__float_as_uint(__shfl_sync(0xffffffffu, xs, i)) & kGbRowScaleMask) * p.global_scale;
          const int64_t row = __shfl_sync(0xffffffffu, to, i);
          if (i < n && w < p.N) p.D[row * p.N + w] = (uint16_t)gb_f32_to_bf16_bits(r);
        }
      }
    } else {
    for (int tile = first; tile < total_tiles; tile += stride, ++it) {
      int mt, nt;
      tile_at(p, tile, mt, nt);
      const int buf = S::kAccs == 2 ? it & 1 : 0, n0 = nt * kBN + c_lo;
      const int row0 = mt * kPairM + (int)rank * kBM + quarter * 32, row = row0 + lane;
      const bool row_ok = row < p.M;
      const float rs = (p.a_scale && row_ok ? p.a_scale[row] : 1.0f) * p.global_scale;
      wait<true>(acc_full + 8 * buf, (uint32_t)(S::kAccs == 2 ? it >> 1 : it) & 1, abort_flag, p.status, 77);
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16) + (buf ? S::kAcc1 : 0u) + (uint32_t)c_lo;
      uint32_t w[kCols / 2], va[32];
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        tmem_ld32(tbase + 32u * c, va);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c == kChunks - 1) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_cluster(acc_empty_pair + 8 * buf);
        }
        pack_chunk<kKind != kFp4>(p, va, &w[16 * c], rs, n0 + 32 * c);
      }
      if (p.out_tma) {
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          const uint32_t dst = out + (uint32_t)flip * kOutChunk;       // in turn across tiles: their chunks may be odd in number
          flip ^= 1;
          asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");       // the chunk before last has left its buffer
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 4; ++q)                        // 64-byte swizzle: eight rows touch eight bank groups
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                         ::"r"(dst + (uint32_t)lane * 64u + (uint32_t)((q ^ ((lane >> 1) & 3)) * 16)), "r"(w[16 * c + 4 * q]),
                           "r"(w[16 * c + 4 * q + 1]), "r"(w[16 * c + 4 * q + 2]), "r"(w[16 * c + 4 * q + 3]) : "memory");
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0 && row0 < p.M && n0 + 32 * c < p.N)  // what sticks out is not written
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                         ::"l"(reinterpret_cast<uint64_t>(&map_d)), "r"(n0 + 32 * c), "r"(row0), "r"(dst) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      } else if (row_ok) {
        uint16_t* d = p.D + (int64_t)row * p.N + n0;
        const int cols = (int)p.N - n0;
#pragma unroll
        for (int c = 0; c < kCols; ++c)
          if (c < cols) d[c] = (uint16_t)(w[c / 2] >> (16 * (c & 1)));
      }
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag) __nanosleep(1000000);                   // loads and MMAs still in flight end before the memory goes
  gb_cluster_sync();                                            // the peer may still signal barriers here
  if (warp == kEpiWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
}

std::mutex g_mutex;
int g_pairs[64][8];                                          // pairs that run at once, per device and kernel (0: not asked)

template <Kind kKind, int kBN, bool kGrouped = false>
int resident_pairs() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(g_mutex);
  int& n = g_pairs[dev][kGrouped ? 6 : (int)kKind * 2 + (kBN == 256)];
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * 256);
    cfg.blockDim = dim3(Shape<kKind, kBN, kGrouped>::kThreads);
    cfg.dynamicSmemBytes = Shape<kKind, kBN, kGrouped>::kSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<kKind, kBN, kGrouped>, &cfg) != cudaSuccess) { n = 0; cudaGetLastError(); }
  }
  return n;
}

template <Kind kKind, int kBN>
int run(const void* A, const void* B, const void* sfa, const void* sfb, PairParams p, int row_bytes_elem, cudaStream_t stream) {
  using S = Shape<kKind, kBN>;
  const int pairs = resident_pairs<kKind, kBN>();
  if (pairs <= 0) return GB_EUNSUPPORTED;
  p.m_tiles = (int)((p.M + kPairM - 1) / kPairM);
  p.n_tiles = (int)((p.N + kBN - 1) / kBN);
  p.idesc |= ((uint32_t)(kBN >> 3) << 17) | ((uint32_t)(kPairM >> 4) << 24);
  CUtensorMap map_a, map_b, map_d = {}, map_sfa = {}, map_sfb = {};
  const int64_t row = kKind == kFp4 ? p.K / 2 : p.K;
  int rc = gb_tensor_map_operand(&map_a, A, p.M, row, row_bytes_elem, kBM);
  if (rc != GB_OK) return rc;
  rc = gb_tensor_map_operand(&map_b, B, p.N, row, row_bytes_elem, kBN / 2);
  if (rc != GB_OK) return rc;
  p.out_tma = p.N % 8 == 0;
  if (p.out_tma) {
    rc = gb_tensor_map_out(&map_d, p.D, p.M, p.N);
    if (rc != GB_OK) return rc;
  }
  if (kKind == kFp4) {                                       // the planes as rows of 256 bytes: eight are four atoms
    const int64_t a_rows = (p.M + 127) / 128 * p.k_tiles * 8, b_rows = (p.N + 127) / 128 * p.k_tiles * 8;
    rc = gb_tensor_map_bytes_2d(&map_sfa, sfa, 256, (uint64_t)a_rows, 256, 256, 8);
    if (rc != GB_OK) return rc;
    rc = gb_tensor_map_bytes_2d(&map_sfb, sfb, 256, (uint64_t)b_rows, 256, 256, 8);
    if (rc != GB_OK) return rc;
  }
  const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles;
  GB_REQUIRE(tiles < (1ll << 31), "too many output tiles");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs)));
  cfg.blockDim = dim3(S::kThreads);
  cfg.dynamicSmemBytes = S::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = gb_pdl_enabled() ? 2 : 1;
  gb_count_launch();
  GB_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_pair_kernel<kKind, kBN, false>, map_a, map_b, map_d, map_sfa, map_sfb, p));
  return GB_OK;
}

}  // namespace

int gb_prepare_gemm_pair() {
#define GB_ATTR(K, N) \
  GB_CUDA_OK(cudaFuncSetAttribute((const void*)gemm_pair_kernel<K, N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<K, N>::kSmem))
  GB_ATTR(kBf16, 256);
  GB_ATTR(kBf16, 192);
  GB_ATTR(kFp8, 256);
  GB_ATTR(kFp8, 192);
  GB_ATTR(kFp4, 256);
  GB_ATTR(kFp4, 192);
#undef GB_ATTR
  GB_CUDA_OK(cudaFuncSetAttribute((const void*)gemm_pair_kernel<kFp4, 192, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  Shape<kFp4, 192, true>::kSmem));
  return GB_OK;
}

namespace {
// Width of a tile: 256 columns, or 192 where that saves more of the last wave than the sixth of extra
// operand traffic costs (columns per pair and wave, 5% in favour of 256: 333 x 5120 x 17408 fp4 34 -> 32 us
// with 192, 2048 x 34816 x 5120 165 -> 201).
bool narrow_tiles(int64_t M, int64_t N) {
  const int64_t pairs = gb_sm_count() / 2, mt = (M + kPairM - 1) / kPairM;
  const int64_t w256 = (mt * ((N + 255) / 256) + pairs - 1) / pairs * 256, w192 = (mt * ((N + 191) / 192) + pairs - 1) / pairs * 192;
  return w192 * 21 < w256 * 20;
}
}  // namespace

int gb_gemm_pair(const void* A, const void* B, void* D, int64_t M, int64_t N, int64_t K, int kind, const float* a_scale,
                 const float* b_scale, float global_scale, cudaStream_t stream) {
  PairParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.k_tiles = (int)(K * (kind == GB_GEMM_BF16 ? 2 : 1) / kSlabBytes);
  p.idesc = (1u << 4) | (kind == GB_GEMM_BF16 ? (1u << 7) | (1u << 10) : 0u);
  p.a_scale = a_scale; p.b_scale = b_scale;
  p.global_scale = global_scale;
  p.D = (uint16_t*)D;
  p.status = gb_status_word();
  const bool narrow = narrow_tiles(M, N);
  if (kind == GB_GEMM_BF16)
    return narrow ? run<kBf16, 192>(A, B, nullptr, nullptr, p, 2, stream) : run<kBf16, 256>(A, B, nullptr, nullptr, p, 2, stream);
  return narrow ? run<kFp8, 192>(A, B, nullptr, nullptr, p, 1, stream) : run<kFp8, 256>(A, B, nullptr, nullptr, p, 1, stream);
}

int gb_gemm_fp4_pair(const void* A, const void* sfa, const void* B, const void* sfb, void* D, int64_t M, int64_t N, int64_t K,
                     const float* a_scale, float global_scale, cudaStream_t stream) {
  PairParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.k_tiles = (int)(K / 256);
  p.idesc = (1u << 7) | (1u << 10);
  p.a_scale = a_scale;
  p.global_scale = global_scale;
  p.D = (uint16_t*)D;
  p.status = gb_status_word();
  const bool narrow = narrow_tiles(M, N);
  return narrow ? run<kFp4, 192>(A, B, sfa, sfb, p, 1, stream) : run<kFp4, 256>(A, B, sfa, sfb, p, 1, stream);
}

extern "C" {

int gb_moe_gemm_fp4(const void* operand, const void* packed, const void* sf, int64_t N, int64_t K, int64_t E, const int32_t* seg,
                    const int32_t* row_map, int64_t P, float global_scale, void* y, void* stream) {
  using S = Shape<kFp4, 192, true>;
  GB_REQUIRE(operand && packed && sf && seg && y, "null pointer argument");
  GB_REQUIRE(N > 0 && N % kBM == 0 && K > 0 && K % 256 == 0, "N=%lld must be a multiple of %d, K=%lld of 256", (long long)N, kBM, (long long)K);
  GB_REQUIRE(P >= 1 && P < (1ll << 30) && E >= 1 && E <= kMaxGroups && E * N < (1ll << 31) && K < (1ll << 31),
             "bad shape P=%lld E=%lld N=%lld", (long long)P, (long long)E, (long long)N);
  GB_REQUIRE(((uintptr_t)operand & 255u) == 0 && ((uintptr_t)packed & 15u) == 0 && ((uintptr_t)sf & 15u) == 0,
             "operands must be aligned: 256 and 16 bytes");
  const int pairs = resident_pairs<kFp4, 192, true>();
  if (pairs <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  const GbFp4Tiles op = gb_fp4_tiles(P, E, K);
  PairParams p = {};
  p.M = E * N; p.N = N; p.K = K;
  p.k_tiles = (int)(K / 256);
  p.m_tiles = (int)((N + kPairM - 1) / kPairM);
  p.idesc = (1u << 7) | (1u << 10) | ((uint32_t)(192 >> 3) << 17) | ((uint32_t)(kPairM >> 4) << 24);
  p.global_scale = global_scale == 0.0f ? 1.0f : global_scale;
  p.D = (uint16_t*)y;
  p.status = gb_status_word();
  p.seg = seg; p.row_map = row_map; p.E = (int)E;
  p.x_scale = (const float*)((const uint8_t*)operand + op.scale_at);
  p.tail = (const float*)((const uint8_t*)operand + op.tail_at);
  p.codes = (const uint8_t*)operand;
  p.packed = (const uint8_t*)packed;
  p.sf = (const uint8_t*)sf;
  CUtensorMap map_a, map_b, map_d = {}, map_sfa, map_sfb;
  int rc = gb_tensor_map_operand(&map_a, packed, E * N, K / 2, 1, kBM);
  if (rc != GB_OK) return rc;
  rc = gb_tensor_map_operand(&map_b, operand, op.tiles * 2 * kTileRows, K / 2, 1, 32);
  if (rc != GB_OK) return rc;
  rc = gb_tensor_map_bytes_2d(&map_sfa, sf, 256, (uint64_t)(E * N / 128 * p.k_tiles * 8), 256, 256, 8);
  if (rc != GB_OK) return rc;
  rc = gb_tensor_map_bytes_2d(&map_sfb, (const uint8_t*)operand + op.sf_at, 256, (uint64_t)(op.sf_groups * p.k_tiles * 8), 256, 256, 8);
  if (rc != GB_OK) return rc;
  const int64_t tiles = op.tiles * p.m_tiles;                // at least as many as the routing can make
  GB_REQUIRE(tiles < (1ll << 31), "too many output tiles");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs)));
  cfg.blockDim = dim3(S::kThreads);
  cfg.dynamicSmemBytes = S::kSmem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = gb_pdl_enabled() ? 2 : 1;
  gb_count_launch();
  GB_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_pair_kernel<kFp4, 192, true>, map_a, map_b, map_d, map_sfa, map_sfb, p));
  return GB_OK;
}

}  // extern "C"
