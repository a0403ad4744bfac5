// Products of many token rows with bf16 weights (prefill):  out[t, n] = W[n, :] . x[t, :].
//
//   gemm_tc_kernel<BM, BN, GATED>   bf16 rows on the tensor cores, an SM on a tile: few tokens, small groups
//   gemm_pair_kernel<GATED>     the same, a pair of SMs on a tile
//   gemm_f32_kernel<.., GATED>  f32 rows, f32 arithmetic (the exact mode)
//
// GATED: the weight holds gate rows, then up rows, and the result is their clamped gated unit.
// Grouped launches have one weight per group (expert) and the token rows sorted by group; the number of rows per
// group is device data, so the tiles are enumerated on the device and the grid is the SM count.
//
// Tensor-core kernel: persistent, warp-specialised, one CTA per SM.  The 128 or 64 weight rows of a tile are M (so a TMEM
// lane is an output feature and a store covers consecutive features), 64 or 32 token rows are N.  One thread
// issues the TMA loads (128-byte swizzle) into a ring of stages, one thread issues the tcgen05.mma, eight warps read
// the accumulators back; two accumulators alternate so that the epilogue of a tile overlaps the products of the next.
#pragma once

#include <cuda.h>

#include "act.cuh"
#include "cluster.cuh"
#include "tcgen05.cuh"

namespace tb {

constexpr int kMaxGroups = 1024;

struct GemmRowsParams {
  int n;                 // output features
  int k;
  int rows;              // token rows; grouped with counts: an upper bound is not needed, the counts say how many
  int n_groups;          // 0: one weight for all rows
  const int* counts;     // [n_groups] device; null: `rows` rows in every group
  float limit, alpha;    // GATED
  const float* bias;     // optional [n] (one weight only)
  void* out;
  long long ldo;
  int out_bf16;
  int* status;
  // the exact mode reads its operands directly
  const __nv_bfloat16* w;
  long long ldw;
  const float* x;
  long long ldx;
};

// Enumeration of (group, feature tile, token tile); token tiles vary fastest, so that CTAs running together share a
// weight tile, or, with `tokens_outer`, feature tiles do.  `rows0` / `tiles0` are exclusive prefix sums over the groups in shared
// memory.
struct TileWalk {
  const int* rows0;
  const int* tiles0;
  int n_groups, ft, bn;
  int bf = 128;          // features of a tile
  bool tokens_outer = false;
  int group = 0;

  struct Tile {
    int group, feature0, row0, row1;
  };
  __device__ __forceinline__ Tile at_warp(int i) {  // the same by a whole warp
    const Tile t = at(i);
    return {warp_uniform(t.group), warp_uniform(t.feature0), warp_uniform(t.row0), warp_uniform(t.row1)};
  }
  __device__ __forceinline__ Tile at(int i) {  // i must not decrease between calls
    while (i >= tiles0[group + 1]) ++group;
    const int local = i - tiles0[group], r0 = rows0[group], r1 = rows0[group + 1];
    const int tt = (r1 - r0 + bn - 1) / bn;
    int f, t;
    if (tokens_outer) {
      t = local / ft;
      f = local - t * ft;
    } else {
      f = local / tt;
      t = local - f * tt;
    }
    return {group, f * bf, r0 + t * bn, min(r0 + (t + 1) * bn, r1)};
  }
};

// Fills the prefix sums (all threads of the CTA; s_rows / s_tiles hold max(n_groups, 1) + 1 entries).
__device__ __forceinline__ void tile_prefix(const GemmRowsParams& p, int bn, int ft, int* s_rows, int* s_tiles) {
  if (p.n_groups == 0) {
    if (threadIdx.x == 0) {
      s_rows[0] = s_tiles[0] = 0;
      s_rows[1] = p.rows;
      s_tiles[1] = (p.rows + bn - 1) / bn * ft;
    }
  } else if (threadIdx.x < 32) {
    int r0 = 0, t0 = 0;
    for (int b = 0; b < p.n_groups; b += 32) {
      const int e = b + static_cast<int>(threadIdx.x);
      const int c = e >= p.n_groups ? 0 : (p.counts != nullptr ? p.counts[e] : p.rows);
      int r = c, t = (c + bn - 1) / bn * ft;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int ra = __shfl_up_sync(0xffffffffu, r, o), ta = __shfl_up_sync(0xffffffffu, t, o);
        if (static_cast<int>(threadIdx.x) >= o) {
          r += ra;
          t += ta;
        }
      }
      if (e < p.n_groups) {
        s_rows[e + 1] = r0 + r;
        s_tiles[e + 1] = t0 + t;
      }
      r0 += __shfl_sync(0xffffffffu, r, 31);
      t0 += __shfl_sync(0xffffffffu, t, 31);
    }
    if (threadIdx.x == 0) s_rows[0] = s_tiles[0] = 0;
  }
  __syncthreads();
}

// ------------------------------------------------------------------ tensor cores
constexpr int kTcEpiWarps = 8;  // two per quarter of the TMEM lanes, each with half of the columns
constexpr int kTcThreads = 64 + 32 * kTcEpiWarps;  // and a producer warp, an MMA warp
constexpr int kTcK = 64;

// BM features x BN token rows.  Few tiles leave most SMs idle, and a tile's time is that of its steps along K.  A step is bound by
// shared memory: 64 x 64 x 16 is 32 cycles of the tensor core, in which it reads 4 KB, as much as that memory gives, and what the
// copies write comes on top; and waiting for a stage and releasing it takes 120 to 170 cycles in which no product is issued.
// So tiles are small where there are few, and a stage is four blocks of 64 along K, two or one where fewer than three stages would
// fit.  B200, stages of two blocks -> of four -> and tiles of 32 rows: 37 rows, 2048 features, K 5632 16.4 -> 14.1 -> 11.8 us; K 2048
// 8.3 -> 7.4 -> 6.4; 2048 rows, 64 features, K 4096 12.5 -> 10.3 -> 8.9; 173 x 3072 x 2048, which keeps tiles of 64 rows, 8.7 -> 7.9.
// Three blocks: 14.4 and 12.9 us at the first of these.
template <int BM, int BN, bool GATED>
struct TcShape {
  static constexpr int kBlocks = GATED ? 128 / BM : (BM == 64 ? 4 : 2);
  static constexpr int kWBytes = BM * kTcK * 2;
  static constexpr int kXBytes = BN * kTcK * 2;
  static constexpr int kBlockBytes = (GATED ? 2 : 1) * kWBytes + kXBytes;
  static constexpr int kStageBytes = kBlocks * kBlockBytes;
  static constexpr int kStages = 196608 / kStageBytes < 8 ? 196608 / kStageBytes : 8;
  static constexpr int kAccCols = GATED ? 2 * BN : BN;
  static constexpr int kTmemCols = 2 * kAccCols;
  static_assert(kTmemCols >= 32 && kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "TMEM allocation size");
  static constexpr size_t kSmemBytes = static_cast<size_t>(kStages) * kStageBytes + 1024;  // + alignment of the ring
};

// K-major operand in 128-byte swizzled rows (the layout a 64-element wide TMA box leaves): eight-row groups are
// 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3fffu) | (1ull << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}
// D = f32, A = B = bf16, both K-major
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// Completion of the loads issued so far; the registers are operands so that no use moves above it.
__device__ __forceinline__ void tmem_ld16_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// Lane l holds v[t], t = 0 .. 7, of feature l; returns the eight features of the lane's group of eight lanes for token
// l & 7.  Three exchanges, each between lanes one bit apart, each sending what the partner keeps.
__device__ __forceinline__ uint4 turn_eight(const float* v, int lane) {
  const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4;
  uint32_t w[4];         // two features; w[k] of token 2 k + b0
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float got = __shfl_xor_sync(0xffffffffu, b0 ? v[2 * k] : v[2 * k + 1], 1);
    w[k] = b0 ? pack_bf16x2(got, v[2 * k + 1]) : pack_bf16x2(v[2 * k], got);
  }
  uint32_t lo[2], hi[2];  // four features; of token 4 m + 2 b1 + b0
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const uint32_t got = __shfl_xor_sync(0xffffffffu, b1 ? w[2 * m] : w[2 * m + 1], 2);
    lo[m] = b1 ? got : w[2 * m];
    hi[m] = b1 ? w[2 * m + 1] : got;
  }
  const uint32_t g0 = __shfl_xor_sync(0xffffffffu, b2 ? lo[0] : lo[1], 4), g1 = __shfl_xor_sync(0xffffffffu, b2 ? hi[0] : hi[1], 4);
  return b2 ? make_uint4(g0, g1, lo[1], hi[1]) : make_uint4(lo[0], hi[0], g0, g1);
}

enum StoreForm : int { STORE_F32, STORE_EIGHTS, STORE_PAIRS, STORE_ONES };
__device__ __forceinline__ StoreForm store_form(const GemmRowsParams& p) {
  if (!p.out_bf16) return STORE_F32;
  if ((p.n & 7) == 0 && (p.ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0) return STORE_EIGHTS;
  return (p.n & 1) == 0 && (p.ldo & 1) == 0 ? STORE_PAIRS : STORE_ONES;
}
// Stores v[j], feature f of row `row0 + j` (below row1); eight lanes that begin at a multiple of eight have eight features
// in a row and the same rows.
__device__ __forceinline__ void store_eight(const GemmRowsParams& p, StoreForm how, const float* v, int f, bool f_ok, int row0, int row1, int lane) {
  const int left = row1 - row0;
  const long long at = static_cast<long long>(row0) * p.ldo;
  if (how == STORE_F32) {
    float* o = reinterpret_cast<float*>(p.out) + at + f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (f_ok && j < left) o[j * p.ldo] = v[j];
  } else if (how == STORE_EIGHTS) {
    // the lanes turn their eight features of eight rows over: a lane stores eight features of one row
    const uint4 w = turn_eight(v, lane);
    const int j = lane & 7;
    if (f_ok && j < left) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + at + j * p.ldo + (f & ~7)) = w;
  } else if (how == STORE_PAIRS) {
    // neighbouring lanes exchange one value, so that a lane stores two features of one row
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at + (f & ~1);
    const bool odd = lane & 1;
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
      const int jj = j + (odd ? 1 : 0);
      const uint32_t w = odd ? pack_bf16x2(got, v[j + 1]) : pack_bf16x2(v[j], got);
      if (f_ok && jj < left) *reinterpret_cast<uint32_t*>(o + jj * p.ldo) = w;
    }
  } else {
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at + f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (f_ok && j < left) o[j * p.ldo] = f2bf(v[j]);
  }
}

template <int BM, int BN, bool GATED>
__global__ void __launch_bounds__(kTcThreads, 1)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const GemmRowsParams p) {
  using S = TcShape<BM, BN, GATED>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[S::kStages], empty[S::kStages], acc_full[2], acc_empty[2], drain;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ int s_rows[kMaxGroups + 1], s_tiles[kMaxGroups + 1];
  uint8_t* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < S::kStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], kTcEpiWarps);
    }
    mbar_init(&drain, 1);
    s_abort = 0;
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(S::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*reinterpret_cast<volatile uint32_t*>(&s_tmem));
  pdl_wait();
  const int ft = (p.n + BM - 1) / BM;
  tile_prefix(p, BN, ft, s_rows, s_tiles);
  const int groups = p.n_groups > 0 ? p.n_groups : 1;
  const int n_tiles = warp_uniform(s_tiles[groups]);
  const int n_blocks = (p.k + kTcK - 1) / kTcK;  // (what lies beyond K in the last one is zero)
  volatile int* abort = &s_abort;
  TileWalk walk{s_rows, s_tiles, groups, ft, BN, BM};

  if (warp == 0) {
    uint32_t it = 0, s = 0, ph = 0;
    bool ok = true;
    for (int i = blockIdx.x; ok && i < n_tiles; i += gridDim.x) {
      const TileWalk::Tile t = walk.at_warp(i);
      const int wrow = t.group * (GATED ? 2 : 1) * p.n + t.feature0;
      for (int kb = 0; kb < n_blocks; kb += S::kBlocks, ++it) {
        if (!mbar_wait_warp(&empty[s], ph ^ 1u, abort)) {
          set_status(p.status, ST_WAIT_EMPTY_TIMEOUT);
          ok = false;
          break;
        }
        uint8_t* st = ring + s * S::kStageBytes;
        if (elect_one()) {
          const int blocks = min(S::kBlocks, n_blocks - kb);
          mbar_expect_tx(&full[s], blocks * S::kBlockBytes);
#pragma unroll
          for (int b = 0; b < S::kBlocks; ++b, st += S::kBlockBytes) {
            if (b >= blocks) break;
            const int k0 = (kb + b) * kTcK;
            tma_load_2d(st, &wmap, k0, wrow, &full[s]);
            if (GATED) tma_load_2d(st + S::kWBytes, &wmap, k0, wrow + p.n, &full[s]);
            tma_load_2d(st + (GATED ? 2 : 1) * S::kWBytes, &xmap, k0, t.row0, &full[s]);
          }
        }
        if (++s == S::kStages) s = 0, ph ^= 1u;
      }
    }
    if (!ok) *abort = 1;
    // copies still in flight must land before this CTA's shared memory goes away
    for (uint32_t j = it > S::kStages ? it - S::kStages : 0; j < it; ++j) mbar_wait(&full[j % S::kStages], (j / S::kStages) & 1u);
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc_bf16(BM, BN);
    const uint32_t base0 = smem_u32(ring);
    uint32_t s = 0, ph = 0, base = base0, n_done = 0;
    bool ok = true, seen = false;
    for (int i = blockIdx.x; ok && i < n_tiles; i += gridDim.x, ++n_done) {
      const uint32_t buf = n_done & 1u, aph = (n_done >> 1) & 1u;
      if (!mbar_wait_warp(&acc_empty[buf], aph ^ 1u, abort)) {
        set_status(p.status, ST_WAIT_EMPTY_TIMEOUT);
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem + buf * S::kAccCols;
      for (int kb = 0; kb < n_blocks; kb += S::kBlocks) {
        if (!mbar_wait_warp(&full[s], ph, abort, seen)) {
          set_status(p.status, ST_WAIT_FULL_TIMEOUT);
          ok = false;
          break;
        }
        uint64_t* const done = &empty[s];
        if (++s == S::kStages) s = 0, ph ^= 1u;
        seen = mbar_test(&full[s], ph);  // (known by the time it is asked for)
        const int blocks = n_blocks - kb;
        const uint64_t wd = umma_desc_sw128(base), ud = umma_desc_sw128(base + S::kWBytes);
        const uint64_t xd = umma_desc_sw128(base + (GATED ? 2 : 1) * S::kWBytes);
        if (elect_one()) {
#pragma unroll
          for (int b = 0; b < S::kBlocks; ++b) {
            if (b >= blocks) break;
#pragma unroll
            for (int q = 0; q < kTcK / 16; ++q) {  // 32 bytes along K per instruction
              const uint32_t off = (b * S::kBlockBytes + q * 32) >> 4;
              umma_bf16(d, wd + off, xd + off, idesc, (kb | b | q) != 0);
              if (GATED) umma_bf16(d + BN, ud + off, xd + off, idesc, (kb | b | q) != 0);
            }
          }
          umma_commit(done);
          if (blocks <= S::kBlocks) umma_commit(&acc_full[buf]);
        }
        base = s == 0 ? base0 : base + S::kStageBytes;
      }
    }
    if (!ok) *abort = 1;
    __syncwarp();
    if (elect_one()) umma_commit(&drain);  // products still running read shared memory and write TMEM
    mbar_wait(&drain, 0);
  } else {
    const int quad = warp & 3;  // TMEM lanes this warp may read
    constexpr int kCols = BN / (kTcEpiWarps / 4);
    const int c0 = (warp - 2) / 4 * kCols;  // its columns
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const StoreForm how = store_form(p);
    uint32_t n_done = 0;
    for (int i = blockIdx.x; i < n_tiles; i += gridDim.x, ++n_done) {
      const TileWalk::Tile t = walk.at_warp(i);
      const uint32_t buf = n_done & 1u, aph = (n_done >> 1) & 1u;
      const bool ok = mbar_wait(&acc_full[buf], aph, abort);
      if (__any_sync(0xffffffffu, !ok)) {  // warp-uniform: tcgen05.ld needs every lane
        if (!ok) set_status(p.status, ST_WAIT_FULL_TIMEOUT);
        *abort = 1;
        break;
      }
      tc_fence_after();
      // 64 features: sixteen in the first half of every quarter of the lanes
      const int f = t.feature0 + (BM == 64 ? quad * 16 : quad * 32) + lane;
      const bool f_ok = f < p.n && (BM == 128 || lane < 16);
      const float bias = p.bias != nullptr && f_ok ? p.bias[f] : 0.f;
      const uint32_t acc = tmem + buf * S::kAccCols + lane_off;
      for (int c = c0; c < c0 + kCols && t.row0 + c < t.row1; c += 16) {
        float v[16];
        uint32_t r[16];
        tmem_ld16(acc + c, r);
        if (GATED) {
          uint32_t u[16];
          tmem_ld16(acc + BN + c, u);
          tmem_ld16_wait(r);
          tmem_ld16_wait(u);
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = clamped_gate(__uint_as_float(r[j]), __uint_as_float(u[j]), p.limit, p.alpha);
        } else {
          tmem_ld16_wait(r);
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + bias;
        }
        store_eight(p, how, v, f, f_ok, t.row0 + c, t.row1, lane);
        store_eight(p, how, v + 8, f, f_ok, t.row0 + c + 8, t.row1, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::kTmemCols) : "memory");
  }
}

// ------------------------------------------------------------------ tensor cores, a pair of SMs on one tile
// The same roles on clusters of two CTAs: the pair's tile is 256 weight rows x up to 256 token rows, either CTA has 128 of
// the weight rows (its TMEM lanes) and half of the token rows in its shared memory, and the products of both
// (tcgen05.mma.cta_group::2) are issued by the first.  A step of 64 along K then moves 32 KB into an SM where a tile of
// 128 x 256 of its own moves 48, which is what paced that kernel.  A gated tile is 128 features: a CTA's 128 weight rows
// are 64 gate rows and their 64 up rows in turns of sixteen, so that a warp has both of sixteen features and half-warps
// exchange halves.  Sums run along K in the same order as in the kernel above: the results have the same bits.
//
// 2048 rows, K 4096, gated 11264 features: 250 us (1.51 PFLOP/s), on single SMs in tiles of 128 rows 332; 4096 features, K
// 11264: 133 us (1.41), 149 in tiles of 256; 1357 rows, gated 18432 features, K 7168: 507 (639); 7168 features, K 8192: 126
// (152).
//
// A group whose count is on the device multiplies its last token tile with as many rows as that has, in steps of 32, and up to half
// a tile loads only those.  Its feature tiles come in turns of one token tile: with token tiles fastest, of which a group has
// one or two, every other pair would get short tiles only.  256 rows each (+- 16) of 64 experts: gated, 1536 features, K 4096 427 us
// (965 TFLOP/s), with whole tiles 463; 4096 features, K 1536 214 (234); 341 rows of 48, spread by a factor of three, gated, 2048 x 7168
// 864 (935); 75 to 310 rows 1 to 10 % faster.  Without groups short tiles gave nothing (0.97 to 1.01): one pair of 74 has them.
constexpr int kPairMaxStages = 8;
constexpr int kPairBox = 16;  // token rows of a copy for a short tile

struct PairTiles {
  int bn;                // token rows of a tile: a multiple of 32, at most 256
  int blocks;            // of 64 along K in a stage
  int stages, stage_bytes;
};

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// loads into this CTA's shared memory that complete on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives at the barrier at this place in both CTAs when the products issued so far are complete
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}

template <bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kTcThreads, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap shortmap,
                     const GemmRowsParams p, const PairTiles q) {
  constexpr int kWBytes = 128 * kTcK * 2, kFeats = GATED ? 64 : 128;  // of a CTA
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[kPairMaxStages], empty[kPairMaxStages], acc_full[2], acc_empty[2], drain;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ int s_rows[kMaxGroups + 1], s_tiles[kMaxGroups + 1];
  uint8_t* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank(), stages = q.stages;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPairMaxStages; ++i) {
      mbar_init(&full[i], 1);   // (the first CTA's counts the bytes of both)
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 2 * kTcEpiWarps);
    }
    mbar_init(&drain, 1);
    s_abort = 0;
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are there
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*reinterpret_cast<volatile uint32_t*>(&s_tmem));
  pdl_wait();
  const int ft = (p.n + 2 * kFeats - 1) / (2 * kFeats);
  tile_prefix(p, q.bn, ft, s_rows, s_tiles);
  const int groups = p.n_groups > 0 ? p.n_groups : 1;
  const int n_tiles = warp_uniform(s_tiles[groups]);
  const int n_kb = (p.k + kTcK * q.blocks - 1) / (kTcK * q.blocks);  // (what lies beyond K is zero)
  const int block_bytes = kWBytes + q.bn / 2 * kTcK * 2;
  volatile int* abort = &s_abort;
  auto give_up = [&] {  // a wait that ran out ends both CTAs' roles
    *abort = 1;
    cluster_store(cluster_addr(&s_abort, rank ^ 1u), 1u);
  };
  TileWalk walk{s_rows, s_tiles, groups, ft, q.bn, 2 * kFeats, p.counts != nullptr};
  const int first = blockIdx.x >> 1, stride = gridDim.x >> 1;
  auto tokens_of = [&](const TileWalk::Tile& t) { return p.counts != nullptr ? min(q.bn, (t.row1 - t.row0 + 31) & ~31) : q.bn; };

  if (warp == 0) {
    uint32_t it = 0, s = 0, ph = 0;
    bool ok = true;
    for (int i = first; ok && i < n_tiles; i += stride) {
      const TileWalk::Tile t = walk.at_warp(i);
      const int f0 = t.feature0 + static_cast<int>(rank) * kFeats;
      const int bn = tokens_of(t), half = bn / 2;  // token rows of a CTA
      const bool few = 2 * bn <= q.bn;             // so few that copies of them alone are worth their number
      const int loaded = few ? half : q.bn / 2;
      const int x0 = t.row0 + static_cast<int>(rank) * half;
      for (int kb = 0; kb < n_kb; ++kb, ++it) {
        if (!mbar_wait_warp(&empty[s], ph ^ 1u, abort)) {
          set_status(p.status, ST_WAIT_EMPTY_TIMEOUT);
          ok = false;
          break;
        }
        uint8_t* st = ring + s * q.stage_bytes;
        if (elect_one()) {
          const uint32_t bar = cluster_addr(&full[s], 0);
          if (rank == 0) mbar_expect_tx(&full[s], 2 * q.blocks * (kWBytes + loaded * kTcK * 2));
          for (int k0 = kb * q.blocks * kTcK, b = 0; b < q.blocks; ++b, k0 += kTcK, st += block_bytes) {
            if (GATED) {
#pragma unroll
              for (int g = 0; g < 4; ++g) tma_load_3d_pair(st + g * (kWBytes / 4), &wmap, k0, f0 + 16 * g, 2 * t.group, bar);
            } else {
              tma_load_2d_pair(st, &wmap, k0, t.group * p.n + f0, bar);
            }
            if (!few)
              tma_load_2d_pair(st + kWBytes, &xmap, k0, x0, bar);
            else
              for (int r = 0; r < half; r += kPairBox) tma_load_2d_pair(st + kWBytes + r * kTcK * 2, &shortmap, k0, x0 + r, bar);
          }
        }
        if (++s == stages) s = 0, ph ^= 1u;
      }
    }
    if (!ok) give_up();
    // What is under way into shared memory lands before the pair goes: copies, which the first CTA waits for on behalf of both
    // and whatever has failed, and arrivals of the other CTA's products.  After a failure one CTA may have requested a stage
    // that the other has not; no barrier tells when such a copy lands, so a wait that runs out gives it its time, once.
    const uint32_t from = it > stages ? it - stages : 0;
    if (rank == 0) {
      bool landed = true;
      for (uint32_t j = from; landed && j < it; ++j) landed = mbar_wait(&full[j % stages], (j / stages) & 1u);
      if (landed && !ok) mbar_wait(&full[it % stages], (it / stages) & 1u);
    }
    for (uint32_t j = from; j < it; ++j) mbar_wait(&empty[j % stages], (j / stages) & 1u, abort);
  } else if (warp == 1) {
    if (rank == 0) {
      uint32_t s = 0, ph = 0, n_done = 0;
      bool ok = true, seen = false;
      for (int i = first; ok && i < n_tiles; i += stride, ++n_done) {
        const uint32_t idesc = umma_idesc_bf16(256, tokens_of(walk.at_warp(i)));
        const uint32_t buf = n_done & 1u, aph = (n_done >> 1) & 1u;
        if (!mbar_wait_warp(&acc_empty[buf], aph ^ 1u, abort)) {
          set_status(p.status, ST_WAIT_EMPTY_TIMEOUT);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + buf * 256;
        for (int kb = 0; kb < n_kb; ++kb) {
          if (!mbar_wait_warp(&full[s], ph, abort, seen)) {
            set_status(p.status, ST_WAIT_FULL_TIMEOUT);
            ok = false;
            break;
          }
          const bool wrap = s + 1 == stages;
          seen = mbar_test(&full[wrap ? 0 : s + 1], ph ^ (wrap ? 1u : 0u));  // (known by the time it is asked for)
          const uint32_t base = smem_u32(ring + s * q.stage_bytes);
          uint64_t wd = umma_desc_sw128(base), xd = umma_desc_sw128(base + kWBytes);
          if (elect_one()) {
            for (int b = 0; b < q.blocks; ++b, wd += block_bytes >> 4, xd += block_bytes >> 4) {
#pragma unroll
              for (int c = 0; c < kTcK / 16; ++c) umma_bf16_pair(d, wd + 2 * c, xd + 2 * c, idesc, (kb | b | c) != 0);
            }
            umma_commit_pair(&empty[s]);
            if (kb == n_kb - 1) umma_commit_pair(&acc_full[buf]);
          }
          if (++s == stages) s = 0, ph ^= 1u;
        }
      }
      if (!ok) give_up();
      __syncwarp();
      // products still running read shared memory and write TMEM
      if (elect_one()) asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&drain)) : "memory");
      mbar_wait(&drain, 0);
    }
  } else {
    const int quad = warp & 3;  // TMEM lanes this warp may read
    const int part = (warp - 2) / 4;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const StoreForm how = store_form(p);
    uint32_t n_done = 0;
    for (int i = first; i < n_tiles; i += stride, ++n_done) {
      const TileWalk::Tile t = walk.at_warp(i);
      const uint32_t buf = n_done & 1u, aph = (n_done >> 1) & 1u;
      const bool ok = mbar_wait(&acc_full[buf], aph, abort);
      if (__any_sync(0xffffffffu, !ok)) {  // warp-uniform: tcgen05.ld needs every lane
        if (!ok) set_status(p.status, ST_WAIT_FULL_TIMEOUT);
        give_up();
        break;
      }
      tc_fence_after();
      const int f = t.feature0 + static_cast<int>(rank) * kFeats + (GATED ? quad * 16 + (lane & 15) : quad * 32 + lane);
      const bool f_ok = f < p.n;
      const float bias = p.bias != nullptr && f_ok ? p.bias[f] : 0.f;
      const uint32_t acc = tmem + buf * 256 + lane_off;
      const int half = tokens_of(t) / 2, c0 = part * half;  // (columns in multiples of sixteen)
      for (int c = c0; c < c0 + half && t.row0 + c < t.row1; c += 16) {
        uint32_t r[16];
        tmem_ld16(acc + c, r);
        tmem_ld16_wait(r);
        float v[16];
        if (GATED) {
          // lanes 0-15 have gates, 16-31 the ups of the same features: the first half-warp takes rows 0-7, the other 8-15
          const bool up = lane & 16;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float got = __uint_as_float(__shfl_xor_sync(0xffffffffu, up ? r[j] : r[8 + j], 16));
            v[j] = clamped_gate(up ? got : __uint_as_float(r[j]), up ? __uint_as_float(r[8 + j]) : got, p.limit, p.alpha);
          }
          store_eight(p, how, v, f, f_ok, t.row0 + c + (up ? 8 : 0), t.row1, lane);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + bias;
          store_eight(p, how, v, f, f_ok, t.row0 + c, t.row1, lane);
          store_eight(p, how, v + 8, f, f_ok, t.row0 + c + 8, t.row1, lane);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[buf], 0));
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA's memory goes while the other may signal it or compute from it
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// ------------------------------------------------------------------ f32
// Tiles of BF features x BT tokens, K by KB through shared memory; a thread has 4 features x 8 tokens (gated: 4 pairs x 4) of one of
// KG equal parts of every step of K, and the parts' sums are added pairwise at the end, by all threads.  The next KB of both operands
// are in registers while a step is computed, and the reads of a step are 16 bytes along K from rows an odd number of 16-byte
// units apart (no bank conflicts).  Two shapes: 64 x 64 where such tiles fill the SMs twice, else 32 x 32 with a warp or two a part
// of K: few rows leave a walk along K bound by latency.
// Bound by the reads from shared memory and the instructions around the multiplications: 16 bytes a lane take four cycles of the one
// load path even where lanes share them, so 4 x 2 outputs a thread, as it was, took 24 of them for 32 multiplications of a warp, 12
// loads for 128 take 48.  B200, 4 x 2 -> now: 97 rows, 1088 features, K 1024 17.7 -> 14.1 us; 388 rows over 16 experts, gated 704
// features, K 1024 78.7 -> 59.3, 1024 features, K 704 53.0 -> 40.7; 200 x 2048 x 1024 on 64 x 64 tiles 65.8 -> 50.0; 64 x 4000 x 1600,
// gated, 78.6 -> 61.8.  (Three stages by cp.async with the weights kept as bf16: as fast, gated 5 % slower for the conversions of
// every read.  Eight tokens a thread where gated: 70 us in place of 59.)
template <int BF, int BT, int KB, int KG, bool GATED>
struct F32Shape {
  static constexpr int kRt = GATED ? 4 : 8;              // tokens of a thread
  static constexpr int kFt = BF / 4, kTt = BT / kRt;     // threads along the features, along the tokens
  static constexpr int kGroup = kFt * kTt;               // threads of a part of K
  static constexpr int kThreads = kGroup * KG;
  static constexpr int kW = GATED ? 2 : 1;
  static constexpr int kPitch = KB + 4;                  // (KB / 4 + 1) units of 16 bytes
  static constexpr int kWPieces = (BF * KB / 8 + kThreads - 1) / kThreads, kXPieces = (BT * KB / 4 + kThreads - 1) / kThreads;  // loads of a thread
  static constexpr int kOperands = (kW * BF + BT) * kPitch, kSums = KG / 2 * kW * BF * BT;  // floats, one in the other's place
  static constexpr size_t kSmemBytes = sizeof(float) * (kOperands > kSums ? kOperands : kSums);
  static_assert((KB / 4) % 2 == 0 && KB % (4 * KG) == 0 && kThreads == 512 && (KG & (KG - 1)) == 0, "odd pitch, whole parts, pairs of parts");
};

template <int BF, int BT, int KB, int KG, bool GATED>
__global__ void __launch_bounds__(F32Shape<BF, BT, KB, KG, GATED>::kThreads, 1) gemm_f32_kernel(const GemmRowsParams p) {
  using S = F32Shape<BF, BT, KB, KG, GATED>;
  constexpr int kW = S::kW, RT = S::kRt;
  extern __shared__ __align__(16) float buf[];
  float(*ws)[BF][S::kPitch] = reinterpret_cast<float(*)[BF][S::kPitch]>(buf);
  float(*xs)[S::kPitch] = reinterpret_cast<float(*)[S::kPitch]>(buf + kW * BF * S::kPitch);
  __shared__ int s_rows[kMaxGroups + 1], s_tiles[kMaxGroups + 1];
  pdl_launch_dependents();
  pdl_wait();
  const int ft = (p.n + BF - 1) / BF;
  tile_prefix(p, BT, ft, s_rows, s_tiles);
  const int groups = p.n_groups > 0 ? p.n_groups : 1;
  const int n_tiles = s_tiles[groups];
  TileWalk walk{s_rows, s_tiles, groups, ft, BT, BF};
  const int kg = threadIdx.x / S::kGroup, th = threadIdx.x - kg * S::kGroup;
  const int tf = th % S::kFt, tt = th / S::kFt;  // features tf + kFt i, tokens tt + kTt i
  for (int i = blockIdx.x; i < n_tiles; i += gridDim.x) {
    const TileWalk::Tile t = walk.at(i);
    // this thread's pieces of a step: eight along K of weight rows, four of token rows, the same place along K in all of them
    constexpr int kWRows = S::kThreads / (KB / 8), kXRows = S::kThreads / (KB / 4);  // rows apart
    const int wr0 = threadIdx.x / (KB / 8), wk = threadIdx.x % (KB / 8) * 8, xr0 = threadIdx.x / (KB / 4), xk = threadIdx.x % (KB / 4) * 4;
    const __nv_bfloat16* wp = p.w + (static_cast<long long>(t.group) * kW * p.n + t.feature0 + wr0) * p.ldw + wk;
    const float* xp = p.x + static_cast<long long>(t.row0 + xr0) * p.ldx + xk;
    uint4 wr[kW][S::kWPieces];
    float4 xr[S::kXPieces];
    auto request = [&](int k0) {
#pragma unroll
      for (int e = 0; e < S::kWPieces; ++e) {
        const bool ok = k0 + wk < p.k && wr0 + e * kWRows < min(BF, p.n - t.feature0);
#pragma unroll
        for (int h = 0; h < kW; ++h)
          wr[h][e] = ok ? __ldg(reinterpret_cast<const uint4*>(wp + (static_cast<long long>(h) * p.n + e * kWRows) * p.ldw + k0)) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int e = 0; e < S::kXPieces; ++e) {
        const bool ok = k0 + xk < p.k && xr0 + e * kXRows < min(BT, t.row1 - t.row0);
        xr[e] = ok ? *reinterpret_cast<const float4*>(xp + e * kXRows * p.ldx + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    auto deposit = [&](int k0) {  // (a piece may reach past K)
      const bool whole = k0 + KB <= p.k;
#pragma unroll
      for (int e = 0; e < S::kWPieces; ++e) {
        if (wr0 + e * kWRows >= BF) break;
#pragma unroll
        for (int h = 0; h < kW; ++h) {
          float f[8];
          bf16x8_to_f32(wr[h][e], f);
          if (!whole) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (k0 + wk + j >= p.k) f[j] = 0.f;
          }
          act_st8(&ws[h][wr0 + e * kWRows][wk], f);
        }
      }
#pragma unroll
      for (int e = 0; e < S::kXPieces; ++e) {
        if (xr0 + e * kXRows >= BT) break;
        float4 v = xr[e];
        if (!whole) {
          if (k0 + xk + 1 >= p.k) v.y = 0.f;
          if (k0 + xk + 2 >= p.k) v.z = 0.f;
          if (k0 + xk + 3 >= p.k) v.w = 0.f;
        }
        *reinterpret_cast<float4*>(&xs[xr0 + e * kXRows][xk]) = v;
      }
    };
    float acc[kW][4][RT];
#pragma unroll
    for (int h = 0; h < kW; ++h)
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < RT; ++b) acc[h][a][b] = 0.f;
    request(0);
    for (int k0 = 0; k0 < p.k; k0 += KB) {
      __syncthreads();  // the step before has been read
      deposit(k0);
      __syncthreads();
      if (k0 + KB < p.k) request(k0 + KB);
#pragma unroll
      for (int c = kg * (KB / KG); c < (kg + 1) * (KB / KG); c += 4) {
        float4 xv[RT];
#pragma unroll
        for (int b = 0; b < RT; ++b) xv[b] = *reinterpret_cast<const float4*>(&xs[tt + S::kTt * b][c]);
#pragma unroll
        for (int h = 0; h < kW; ++h)
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const float4 wv = *reinterpret_cast<const float4*>(&ws[h][tf + S::kFt * a][c]);
#pragma unroll
            for (int b = 0; b < RT; ++b) {
              acc[h][a][b] += wv.x * xv[b].x;
              acc[h][a][b] += wv.y * xv[b].y;
              acc[h][a][b] += wv.z * xv[b].z;
              acc[h][a][b] += wv.w * xv[b].w;
            }
          }
      }
    }
    // the parts' sums, half of the parts at a time into shared memory and onto the other half's
    float4* sums = reinterpret_cast<float4*>(buf);
#pragma unroll
    for (int half = KG / 2; half > 0; half /= 2) {
      __syncthreads();  // the last step, or the sums of the round before, have been read
      if (kg >= half && kg < 2 * half) {
#pragma unroll
        for (int h = 0; h < kW; ++h)
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < RT; b += 4)
              sums[((((kg - half) * kW + h) * 4 + a) * (RT / 4) + b / 4) * S::kGroup + th] =
                  make_float4(acc[h][a][b], acc[h][a][b + 1], acc[h][a][b + 2], acc[h][a][b + 3]);
      }
      __syncthreads();
      if (kg < half) {
#pragma unroll
        for (int h = 0; h < kW; ++h)
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < RT; b += 4) {
              const float4 v = sums[(((kg * kW + h) * 4 + a) * (RT / 4) + b / 4) * S::kGroup + th];
              acc[h][a][b] += v.x;
              acc[h][a][b + 1] += v.y;
              acc[h][a][b + 2] += v.z;
              acc[h][a][b + 3] += v.w;
            }
      }
    }
    // the first part's threads have them now: out through shared memory, by all
    __syncthreads();
    if (kg == 0) {
#pragma unroll
      for (int h = 0; h < kW; ++h)
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < RT; ++b) buf[(h * BT + tt + S::kTt * b) * BF + tf + S::kFt * a] = acc[h][a][b];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < BF * BT; e += S::kThreads) {
      const int r = e / BF, f = e - r * BF;
      if (t.feature0 + f >= p.n || t.row0 + r >= t.row1) continue;
      const float v = buf[e];
      reinterpret_cast<float*>(p.out)[static_cast<long long>(t.row0 + r) * p.ldo + t.feature0 + f] =
          GATED ? clamped_gate(v, buf[(kW - 1) * BF * BT + e], p.limit, p.alpha) : v + (p.bias != nullptr ? p.bias[t.feature0 + f] : 0.f);
    }
  }
}

}  // namespace tb
