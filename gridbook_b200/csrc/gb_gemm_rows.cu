// Prefill GEMM for the calls that leave most of the GPU idle in 256-row tiles: few activation rows, or narrow
// layers.  D[M, N] = a_scale[m] * b_scale[n] * global * sum_k X[m, k] W[n, k], the same operands as gb_gemm_pair.cu.
//
// The WEIGHTS are the M side of the MMA: a CTA takes 128 weight rows and up to 256 activation rows (the N side, rounded
// up to 16 only), so a layer has a tile per 128 output features whatever the number of rows, and a few
// rows cost a few columns.  Where these are fewer than the SMs, K is sliced over a thread-block cluster: every CTA
// pushes its fp32 sums into the shared memory of the one that owns the activation row, which adds them in slice order.
//
// Warps 0-7 read the accumulator out (lane = output feature, column = activation row), warp 8
// loads, warp 9 issues the MMAs and, for the fp4 operands, the copies of their scale factors to tensor memory in
// front of them (in order on one thread; a stage has a column set of its own, free once the stage is).
//
// Bound by the operand loads: 16 KiB of weights and 128 bytes per activation row for every 128-byte K slab, of which an
// SM takes in 42 bytes a clock behind the expander (128 rows of 8192 x 5120 fp8, 160 of 5120 x 17408 fp4; 31 and 38 where they come
// from HBM, which, the tensor pipe and the issue slots are then at 30, 25 and 13 %); by launch and prologue (2 us) where K is short.
#include "gb_common.cuh"

#include <cuda.h>

namespace {

enum Kind { kBf16 = 0, kFp8 = 1, kFp4 = 2 };

constexpr int kBM = 128;                             // weight rows of a tile
constexpr int kMaxRows = 256;                        // activation rows of a tile
constexpr int kSlabBytes = 128;                      // K bytes per row and stage (one swizzle span)
constexpr int kEpiWarps = 8;
constexpr int kThreads = 32 * (kEpiWarps + 2);
constexpr int kMaxStages = 8, kMaxSlices = 8;
constexpr uint32_t kTmemCols = 512, kSf0 = 256, kSfCols = 48;   // fp4: column sets of 16 (weights) + 32 (activations)
constexpr int kSfSets = (kTmemCols - kSf0) / kSfCols;
constexpr int kAtoms = 2048;                         // scale bytes of 128 rows x 16 groups
constexpr int kSmemMax = 224 * 1024;

struct GemmRowsParams {
  int64_t M, N;
  int k_tiles, per_slice, slices;                    // K slabs, per slice, slices = cluster size along y
  int n_tiles, rows_per_pass;
  int box_rows;                                      // rows of an activation box
  int stages;
  uint32_t idesc;                                    // without N
  const float* a_scale;                              // [M] or null
  const float* b_scale;                              // [N] or null
  float global_scale;
  const uint8_t* sfw;                                // fp4: scale-factor planes
  const uint8_t* sfx;
  uint16_t* D;
  int out16;                                         // rows of D are a multiple of 16 bytes
  int* status;
};

GB_DEVINL bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// A bounded wait that remembers a timeout for the rest of the CTA: later waits return at once.
__device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  uint64_t t0 = 0;
  for (uint32_t spin = 0; !*abort_flag; ++spin) {
    if (try_wait(bar, parity)) return;
    if ((spin & 255u) == 255u) {
      const uint64_t now = gb_globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > 2000000000ull) { *abort_flag = 1; atomicExch(status, code); }
    }
  }
}
// By a whole warp that goes on together; false: given up.
GB_DEVINL bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (__all_sync(0xffffffffu, try_wait(bar, parity))) return true;
  wait_slow(bar, parity, abort_flag, status, code);
  return !__any_sync(0xffffffffu, *abort_flag != 0);
}
GB_DEVINL void expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
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
GB_DEVINL uint64_t desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(1024u >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// One scale-factor atom: 32 rows of 16 bytes, the 8-row groups 128 bytes apart, into four columns of every lane quarter.
GB_DEVINL void sf_to_tmem(uint32_t tmem_col, uint32_t smem_addr) {
  const uint64_t d = (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(16u >> 4) << 16 | (uint64_t)(128u >> 4) << 32 | (uint64_t)1 << 46;
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem_col), "l"(d) : "memory");
}
template <Kind kKind>
GB_DEVINL void mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sfa, uint32_t sfb, bool accumulate) {
  if (kKind == kFp4)
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n}\n"
        ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate), "r"(sfa), "r"(sfb) : "memory");
  else if (kKind == kFp8)
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
  else
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
GB_DEVINL void commit_to(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
GB_DEVINL void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr));
}

template <Kind kKind>
__global__ void __launch_bounds__(kThreads, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ GemmRowsParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_s[kMaxStages], empty_s[kMaxStages], acc_s;
  __shared__ float rs_s[kMaxRows];
  __shared__ uint32_t slot_s;
  __shared__ volatile int abort_s;
  const uint32_t ring = (gb_smem_u32(smem_raw) + 1023u) & ~1023u;        // the same offset in every CTA of a cluster
  const uint32_t full_bar = gb_smem_u32(full_s), empty_bar = gb_smem_u32(empty_s), acc_bar = gb_smem_u32(&acc_s);
  const uint32_t x_bytes = (uint32_t)p.box_rows * kSlabBytes;
  const uint32_t stage_bytes = kBM * kSlabBytes + x_bytes + (kKind == kFp4 ? 3u * kAtoms : 0u);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int pass = (int)blockIdx.x / p.n_tiles, tile = (int)blockIdx.x - pass * p.n_tiles, slice = (int)blockIdx.y;
  const int n0 = tile * kBM, m0 = pass * p.rows_per_pass;
  const int rows = (int)min((int64_t)p.rows_per_pass, p.M - m0), cols = (rows + 15) / 16 * 16;
  const int k_begin = slice * p.per_slice, k_end = min(p.k_tiles, k_begin + p.per_slice);

  gb_pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      gb_mbar_init(&full_s[s], 1);
      gb_mbar_init(&empty_s[s], 1);
    }
    gb_mbar_init(&acc_s, 1);
    abort_s = 0;
    gb_fence_barrier_init();
  }
  if (warp == kEpiWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gb_smem_u32(&slot_s)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, slot_s, 0);
  gb_pdl_wait();

  // The loading and issuing warps walk their loops whole with one elected lane issuing (gb_elect_one).
  if (warp == kEpiWarps) {
    // ------------------------------- producer -----------------------------------
    constexpr int slab_elems = kKind == kBf16 ? kSlabBytes / 2 : kSlabBytes;   // E2M1 pairs and E4M3 go by bytes
    const bool one = gb_elect_one();
    const int g0 = m0 / 128, groups = kKind == kFp4 ? (m0 + rows - 1) / 128 - g0 + 1 : 0;   // 128-row groups of the pass: one or two
    const uint32_t bytes = kBM * kSlabBytes + x_bytes + (kKind == kFp4 ? (uint32_t)(1 + groups) * kAtoms : 0u);
    int s = 0;
    uint32_t ph = 1;
    for (int kt = k_begin; kt < k_end; ++kt) {
      if (!warp_wait(empty_bar + 8 * s, ph, &abort_s, p.status, 81)) break;
      if (one) {
        const uint32_t st = ring + (uint32_t)s * stage_bytes, bar = full_bar + 8 * s;
        expect_tx(bar, bytes);
        tma_load_2d(st, &map_w, kt * slab_elems, n0, bar);
        tma_load_2d(st + kBM * kSlabBytes, &map_x, kt * slab_elems, m0, bar);
        if (kKind == kFp4) {
          const uint32_t sf = st + kBM * kSlabBytes + x_bytes;
          bulk_load(sf, p.sfw + ((int64_t)tile * p.k_tiles + kt) * kAtoms, kAtoms, bar);
          for (int g = 0; g < groups; ++g) bulk_load(sf + (uint32_t)(1 + g) * kAtoms, p.sfx + ((int64_t)(g0 + g) * p.k_tiles + kt) * kAtoms, kAtoms, bar);
        }
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == kEpiWarps + 1) {
    // ------------------------------- MMA issuer ---------------------------------
    const bool one = gb_elect_one();
    const uint32_t idesc = p.idesc | (uint32_t)(cols >> 3) << 17 | (uint32_t)(kBM >> 4) << 24;
    const bool two = kKind == kFp4 && (m0 + rows - 1) / 128 > m0 / 128;
    const uint32_t shift = kKind == kFp4 && m0 % 128 != 0 ? 2u : 0u;         // a pass that starts in the middle of a 128-row group
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int kt = k_begin; kt < k_end; ++kt) {
      ok = warp_wait(full_bar + 8 * s, ph, &abort_s, p.status, 82);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (one) {
        const uint32_t st = ring + (uint32_t)s * stage_bytes, sf = st + kBM * kSlabBytes + x_bytes;
        const uint64_t dw = desc_sw128(st), dx = desc_sw128(st + kBM * kSlabBytes);
        const uint32_t set = tmem + kSf0 + kSfCols * (uint32_t)s;
        if (kKind == kFp4) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            sf_to_tmem(set + 4u * k, sf + 512u * k);
            sf_to_tmem(set + 16u + 8u * k, sf + kAtoms + 512u * k);
            if (two) sf_to_tmem(set + 20u + 8u * k, sf + 2 * kAtoms + 512u * k);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)                        // 32 bytes of K per instruction
          mma<kKind>(tmem, dw + (uint64_t)(2 * k), dx + (uint64_t)(2 * k), idesc, set + 4u * k, set + 16u + shift + 8u * k, kt > k_begin || k > 0);
        commit_to(empty_bar + 8 * s);
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    if (ok && one) commit_to(acc_bar);
    __syncwarp();
  } else {
    for (int m = threadIdx.x; m < rows; m += 32 * kEpiWarps) rs_s[m] = (p.a_scale ? p.a_scale[m0 + m] : 1.0f) * p.global_scale;
    if (!warp_wait(acc_bar, 0, &abort_s, p.status, 83)) abort_s = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // The row scales are there, and all eight warps see the same flag behind it: the wait may run out in one and end in
    // another, and they meet at barriers below.  (The other two warps raise it only where the accumulator is never complete.)
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
  }

  const bool live = warp < kEpiWarps && !abort_s;
  const int quarter = warp & 3, feature = quarter * 32 + lane;
  const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16);
  if (p.slices == 1) {
    // Out through shared memory, over the operand ring: rows of 16-byte pieces instead of 64 bytes per warp and row
    if (live) {
      const float bs = p.b_scale && n0 + feature < p.N ? p.b_scale[n0 + feature] : 1.0f;
      for (int c = (warp >> 2) * 16; c < cols; c += 32) {
        uint32_t v[16];
        tmem_ld16(acc + (uint32_t)c, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint16_t o = (uint16_t)gb_f32_to_bf16_bits(__uint_as_float(v[i]) * rs_s[c + i] * bs);
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(ring + (uint32_t)((c + i) * kBM + feature) * 2u), "h"(o) : "memory");
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
      const int left = (int)min((int64_t)kBM, p.N - n0);
      uint16_t* d = p.D + (int64_t)m0 * p.N + n0;
      if (p.out16) {
        for (int i = threadIdx.x; i < rows * (kBM / 8); i += 32 * kEpiWarps) {
          const int r = i >> 4, c = (i & 15) * 8;
          uint4 v;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(ring + (uint32_t)(r * kBM + c) * 2u));
          if (c < left) *reinterpret_cast<uint4*>(d + (int64_t)r * p.N + c) = v;
        }
      } else {
        for (int i = threadIdx.x; i < rows * kBM; i += 32 * kEpiWarps) {
          const int r = i >> 7, c = i & (kBM - 1);
          uint16_t v;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(ring + (uint32_t)i * 2u));
          if (c < left) d[(int64_t)r * p.N + c] = v;
        }
      }
    }
  } else {
    // Sums into the shared memory of the CTA that owns the activation row, [slice][own row][feature], over the operand ring:
    // every CTA of the cluster has finished its MMAs, and with them its loads.  Rows are owned in sixteens.
    const int own = (cols / 16 + p.slices - 1) / p.slices * 16;
    gb_cluster_sync();
    if (live) {
      for (int c = (warp >> 2) * 16; c < cols; c += 32) {
        uint32_t v[16];
        tmem_ld16(acc + (uint32_t)c, v);
        const int to = c / own, at = c - to * own;
        uint32_t dst;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(dst) : "r"(ring + (uint32_t)((slice * own + at) * kBM + feature) * 4u), "r"(to));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i)                         // rows past the last are sums of zeros
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst + (uint32_t)i * kBM * 4u), "r"(v[i]) : "memory");
      }
    }
    gb_cluster_sync();                                          // the last access to another CTA's memory lies in front of it
    if (live) {
      const int f = lane * 4, left = (int)min((int64_t)kBM, p.N - n0) - f;
      float bs[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) bs[i] = p.b_scale && i < left ? p.b_scale[n0 + f + i] : 1.0f;
      const int last = min(own, rows - slice * own);
      for (int r = warp; r < last; r += kEpiWarps) {
        float sum[4] = {};
#pragma unroll 4
        for (int q = 0; q < p.slices; ++q) {
          float v[4];
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(ring + (uint32_t)((q * own + r) * kBM + f) * 4u));
#pragma unroll
          for (int i = 0; i < 4; ++i) sum[i] += v[i];
        }
        const float rs = rs_s[slice * own + r];
        uint16_t* d = p.D + (int64_t)(m0 + slice * own + r) * p.N + n0 + f;
        if (p.out16) {
          if (left > 0)
            *reinterpret_cast<uint2*>(d) = make_uint2(gb_pack_bf16x2(sum[0] * rs * bs[0], sum[1] * rs * bs[1]), gb_pack_bf16x2(sum[2] * rs * bs[2], sum[3] * rs * bs[3]));
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i < left) d[i] = (uint16_t)gb_f32_to_bf16_bits(sum[i] * rs * bs[i]);
        }
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_s) __nanosleep(1000000);                   // loads and MMAs still in flight end before the memory goes
  if (warp == kEpiWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

GbClusters g_clusters;
int max_clusters(int size) { return g_clusters.ask((const void*)gemm_rows_kernel<kFp8>, kThreads, kSmemMax, size); }

// Rows of a pass: all of them, else 192 or 256 (starts stay multiples of 64, and a pass within two 128-row
// groups of scale factors), whichever leaves fewer passes, then fewer empty rows.
int pass_rows(int64_t M) {
  if (M <= kMaxRows) return (int)M;
  return (M + 191) / 192 == (M + 255) / 256 ? 192 : 256;
}

struct Split { int rows, slices, per_slice; int64_t tiles; };     // rows of a pass, K slices, slabs of each, (tile, pass) pairs

// K slices: as many as the SMs take, at least four slabs each; adding the sums up costs more the more rows there are, so no
// more than four past 64 (2048 x 8192 fp4, 256 rows: eight 13.4 us, four 11.7; 20 rows fp8: 6.0, 6.3).
Split split_of(int64_t M, int64_t N, int64_t k_tiles) {
  Split s;
  s.rows = pass_rows(M);
  s.tiles = (N + kBM - 1) / kBM * ((M + s.rows - 1) / s.rows);
  const int64_t sms = gb_sm_count();
  int want = 1;
  for (int n = 2; n <= (s.rows <= 64 ? kMaxSlices : 4) && s.tiles * n <= sms && n * 4 <= k_tiles; ++n)
    if (s.tiles <= max_clusters(n)) want = n;
  s.per_slice = (int)((k_tiles + want - 1) / want);
  s.slices = (int)((k_tiles + s.per_slice - 1) / s.per_slice);
  return s;
}

template <Kind kKind>
int run(const void* W, const void* sfw, const void* X, const void* sfx, int64_t K, int elem_bytes, GemmRowsParams p, cudaStream_t stream) {
  if (gb_sm_count() <= 0) return gb_fail(GB_ECUDA, "no usable CUDA device: %s", gb_last_error());
  const Split split = split_of(p.M, p.N, p.k_tiles);
  const int64_t tiles = split.tiles;
  GB_REQUIRE(tiles < (1ll << 31), "too many output tiles");
  p.rows_per_pass = split.rows;
  p.box_rows = (p.rows_per_pass + 15) / 16 * 16;
  p.n_tiles = (int)((p.N + kBM - 1) / kBM);
  p.per_slice = split.per_slice;
  p.slices = split.slices;
  const int stage = kBM * kSlabBytes + p.box_rows * kSlabBytes + (kKind == kFp4 ? 3 * kAtoms : 0);
  p.stages = (kSmemMax - 1024) / stage;
  const int most = kKind == kFp4 ? kSfSets : kMaxStages;
  if (p.stages > most) p.stages = most;
  int bytes = p.stages * stage;
  p.out16 = p.N % 8 == 0;
  const int sums = p.slices > 1 ? (p.box_rows / 16 + p.slices - 1) / p.slices * 16 * p.slices * kBM * 4 : p.box_rows * kBM * 2;
  if (bytes < sums) bytes = sums;
  CUtensorMap map_w, map_x;
  const int64_t row = kKind == kFp4 ? K / 2 : K;
  int rc = gb_tensor_map_operand(&map_w, W, p.N, row, elem_bytes, kBM);
  if (rc != GB_OK) return rc;
  rc = gb_tensor_map_operand(&map_x, X, p.M, row, elem_bytes, p.box_rows);
  if (rc != GB_OK) return rc;
  p.sfw = (const uint8_t*)sfw;
  p.sfx = (const uint8_t*)sfx;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, (unsigned)p.slices);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)bytes + 1024;
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
  GB_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_rows_kernel<kKind>, map_w, map_x, p));
  return GB_OK;
}

}  // namespace

int gb_prepare_gemm_rows() {
  GB_CUDA_OK(cudaFuncSetAttribute((const void*)gemm_rows_kernel<kBf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
  GB_CUDA_OK(cudaFuncSetAttribute((const void*)gemm_rows_kernel<kFp8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
  GB_CUDA_OK(cudaFuncSetAttribute((const void*)gemm_rows_kernel<kFp4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
  return GB_OK;
}

// Where this kernel is the faster one.  us, pairs (to 128 rows: the one-CTA tiles of 128 x 256 that this kernel
// replaced) / this, launches back to back:
//   fp8, bf16   to 192 rows always: 20 rows of 2048 x 2048 19.7 / 4.2, of 5120 x 17408 75 / 12.9, 128 rows of 8192 x 5120 33.2 / 10.3, 160 rows of
//               34816 x 5120 43.5 / 40.3.  Past them where the tiles are one wave and a slice's K no longer than 64 slabs: 256 rows
//               of 2048 x 8192 21.8 / 13.7, 333 of 8192 x 5120 22.7 / 15.3, 1024 of 4096 x 4096 20.5 / 16.9; but 256 of
//               34816 x 5120 45.4 / 51.9, of 12288 x 14336 (112 slabs) 43.5 / 54.8, 512 of 5120 x 17408 42.2 / 54.2.
//   fp4         to 128 rows always: 20 rows of 2048 x 2048 11.1 / 5.0, 128 rows of 5120 x 17408 48.8 / 12.9 (64 rows of 34816 x 5120 20.3 / 21.5).
//               Past them the pairs copy scale factors for twice the rows at a time: only for long K over few tiles, up to 512 rows (160 rows of
//               5120 x 17408 24.0 / 14.5, 333 of 2048 x 8192 13.0 / 10.3, 512 12.9 / 12.7; 256 of 8192 x 5120 10.6 / 12.2, 333 of 5120 x 17408 24.5 / 26.8).
bool gb_gemm_rows_applies(bool fp4, int64_t M, int64_t N, int64_t k_tiles) {
  if (M <= kBM) return true;
  const Split s = split_of(M, N, k_tiles);
  if (fp4) return M <= 512 && k_tiles >= 32 && s.slices >= 3;
  return M <= 192 || (M <= 1024 && s.tiles <= gb_sm_count() && s.per_slice <= 64);
}

extern "C" int gb_gemm_uses_rows(int fp4, int64_t M, int64_t N, int64_t k_bytes) {
  return M >= 1 && N >= 1 && k_bytes >= kSlabBytes && gb_gemm_rows_applies(fp4 != 0, M, N, k_bytes / kSlabBytes) ? 1 : 0;
}

int gb_gemm_rows(const void* X, const void* W, void* D, int64_t M, int64_t N, int64_t K, int kind, const float* a_scale,
                 const float* b_scale, float global_scale, cudaStream_t stream) {
  GemmRowsParams p = {};
  p.M = M; p.N = N;
  p.k_tiles = (int)(K * (kind == GB_GEMM_BF16 ? 2 : 1) / kSlabBytes);
  p.idesc = (1u << 4) | (kind == GB_GEMM_BF16 ? (1u << 7) | (1u << 10) : 0u);
  p.a_scale = a_scale; p.b_scale = b_scale;
  p.global_scale = global_scale;
  p.D = (uint16_t*)D;
  p.status = gb_status_word();
  return kind == GB_GEMM_BF16 ? run<kBf16>(W, nullptr, X, nullptr, K, 2, p, stream) : run<kFp8>(W, nullptr, X, nullptr, K, 1, p, stream);
}

int gb_gemm_fp4_rows(const void* X, const void* sfx, const void* W, const void* sfw, void* D, int64_t M, int64_t N, int64_t K,
                     const float* a_scale, float global_scale, cudaStream_t stream) {
  GemmRowsParams p = {};
  p.M = M; p.N = N;
  p.k_tiles = (int)(K / 256);
  p.idesc = (1u << 7) | (1u << 10);
  p.a_scale = a_scale;
  p.global_scale = global_scale;
  p.D = (uint16_t*)D;
  p.status = gb_status_word();
  return run<kFp4>(W, sfw, X, sfx, K, 1, p, stream);
}
