// Attention of a portion of tokens over expanded keys and values (every head has its own) on tcgen05.
//
// A CTA has NQ tiles of 128 queries of one head and walks over the keys they see in tiles of 128.  Two threads issue the
// TMA loads, one per query tile the products, and a warpgroup per query tile does the softmax with a row per thread (a TMEM
// lane): no exchange between lanes anywhere.  Scores are f32 in TMEM; the probabilities go back, as bf16, over the scores they
// come from and are the A operand of the value product straight from TMEM.  Either half of a tile's keys has its own scores,
// probabilities and hand-over: the products of one half run under the softmax of the other, and of the other query tile, with
// which the keys and values in shared memory are shared.
//
// The reference of the exponentials is the largest score so far, taken anew for every 64 keys, so that the largest probability
// of a row is an exact one in bf16; a warp rescales its rows' sums in TMEM where one has grown, once the half before has been
// added to them.  (One reference for 128 keys: errors up to 0.8 % larger, 275 us in place of 263 for the first size below, with
// the products of a whole tile handed over at once.  A reference that lags behind by up to 2^8 saves most of the rescaling, 2 to
// 8 % of the time, but rounds the largest probability too: errors up to a quarter larger for peaked scores.)
//
// Bound by the chain of a half's scores, softmax (64 exponentials of a row) and value product, several of which run under each
// other, and by the loads of keys and values, 80 KB a tile of 128 keys at 192 + 128 columns.  Against the mma.sync kernel of
// window_attention.cuh (64 rows a CTA), which keeps portions of less than a tile and heads whose tiles do not fit: 32 heads of
// 128 + 64 / 128 columns, 2048 queries behind 4096 keys 263 us (817 TFLOP/s), was 1724; a window of 1024 93 (461), was 375; 64
// heads, 1357 queries from the start 88 (429), was 375; 16 heads, 300 queries 17 (27), was 31; 32 heads, 128 queries 14 (12),
// was 17.  The error against 64 bits is that kernel's to 0.1 %, 0.0016 to 0.0023 over sizes and spreads of scores.
//
// Keys lie in a ring.  A tile ends at the last key, after 128 keys, or at the ring's end, so that its rows are consecutive; 128
// rows are loaded, from the first key at the ring's end and up to the last key elsewhere, and what is no key of the tile is
// hidden.  Those rows are outside of the ring (and zeros), or hold tokens of this portion, which has at least 128: a hidden
// value has a probability of zero, but is multiplied by it, and a row that no query may see can hold anything.
#pragma once

#include "act.cuh"
#include "gemm_rows.cuh"
#include "tcgen05.cuh"

namespace tb {

constexpr int kXaTile = 128;                       // queries, and keys, of a tile
constexpr int kXaBox = kXaTile * 64 * 2;           // bytes of 128 rows x 64 columns, 128-byte swizzle
constexpr int kXaHalf = 64;                        // keys whose exponentials have a common reference
constexpr int kXaKeyStages = 2;

struct ExpandedAttnParams {
  int rows, heads;
  int dimp, rotp, vdim, vdimp;  // a query and a key row: dimp elements, then rotp
  int dim_boxes, v_boxes, k_boxes, v_stages;  // boxes of 64 columns: unrotated part, values, whole key; tiles of values in flight
  int rankp;                    // column of the rotated key part in a cache row
  int ring, window;             // window 0: none
  const int* pos;               // position of row 0
  float scale;                  // > 0
  const float* sink;            // optional [heads]
  HeadGate gate;
  __nv_bfloat16* out;           // [rows, ldo]
  long long ldo;
  int eights;                   // the output (and an element-wise gate) in pieces of eight: sizes and addresses allow it
  int* status;
};

__host__ __device__ inline size_t expanded_attn_smem(int nq, int k_boxes, int v_boxes, int v_stages) {
  return static_cast<size_t>(kXaBox) * (k_boxes * (nq + kXaKeyStages) + v_boxes * v_stages) + 1024;  // + alignment
}

// Tile of keys [a, b) in box rows row0 ..; box row r holds key `key0 + r`.
struct XaKeyTile {
  int a, b, row0, key0;
  __device__ __forceinline__ XaKeyTile(int a_, int hi, int ring) : a(a_) {
    const int slot = a % ring;
    b = min(min(a + kXaTile, hi), a + ring - slot);
    row0 = b - a == ring - slot ? slot : slot + (b - a) - kXaTile;  // rows outside of [0, ring) are loaded as zeros
    key0 = a - (slot - row0);
  }
};

// B operand with its columns (here: value columns) contiguous: rows of 64 columns in 128-byte swizzle, eight-row groups
// 1024 bytes apart, the next 64 columns in the next box.
__device__ __forceinline__ uint64_t umma_desc_sw128_columns(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3fffu) | (static_cast<uint64_t>(kXaBox >> 4) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// A from TMEM (lane = row, two bf16 along K per 32-bit column)
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

#define TB_R8(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])
#define TB_RW8(r, o) "+r"(r[o]), "+r"(r[o + 1]), "+r"(r[o + 2]), "+r"(r[o + 3]), "+r"(r[o + 4]), "+r"(r[o + 5]), "+r"(r[o + 6]), "+r"(r[o + 7])
#define TB_I8(r, o) "r"(r[o]), "r"(r[o + 1]), "r"(r[o + 2]), "r"(r[o + 3]), "r"(r[o + 4]), "r"(r[o + 5]), "r"(r[o + 6]), "r"(r[o + 7])
// 32 columns; the registers may be used after tmem_wait_ld and tmem_use32
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : TB_R8(r, 0), TB_R8(r, 8), TB_R8(r, 16), TB_R8(r, 24)
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_use32(uint32_t (&r)[32]) {  // no use of the registers moves above this
  asm volatile("" : TB_RW8(r, 0), TB_RW8(r, 8), TB_RW8(r, 16), TB_RW8(r, 24));
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,"
      "%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::TB_I8(r, 0), TB_I8(r, 8), TB_I8(r, 16), TB_I8(r, 24), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::TB_I8(r, 0), TB_I8(r, 8),
      "r"(taddr)
      : "memory");
}
#undef TB_R8
#undef TB_RW8
#undef TB_I8
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int NQ>
__global__ void __launch_bounds__(128 + 128 * NQ, 1)
    expanded_attn_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kvmap,
                         const __grid_constant__ CUtensorMap rotmap, const ExpandedAttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kMaxV = 3;
  __shared__ __align__(8) uint64_t q_full, k_full[kXaKeyStages], k_empty[kXaKeyStages], v_full[kMaxV], v_empty[kMaxV], s_full[NQ][2],
      p_full[NQ][2], v_done[NQ][2], o_full[NQ], drain[NQ];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int k_bytes = p.k_boxes * kXaBox, v_bytes = p.v_boxes * kXaBox;
  uint8_t* qs = base;
  uint8_t* ks = qs + NQ * k_bytes;
  uint8_t* vs = ks + kXaKeyStages * k_bytes;
  constexpr int kTmemCols = NQ * 256;  // a score tile and a sum of each query tile

  // heads vary fastest and the tokens with the longest key ranges come first
  const int head = blockIdx.x, t0 = (gridDim.y - 1 - blockIdx.y) * (NQ * kXaTile);
  const int nq = NQ > 1 && t0 + kXaTile < p.rows ? NQ : 1;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int i = 0; i < kXaKeyStages; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], nq);
    }
    for (int i = 0; i < kMaxV; ++i) {
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], nq);
    }
    for (int i = 0; i < NQ; ++i) {
      for (int h = 0; h < 2; ++h) {
        mbar_init(&s_full[i][h], 1);
        mbar_init(&p_full[i][h], 4);
        mbar_init(&v_done[i][h], 1);
      }
      mbar_init(&o_full[i], 1);
      mbar_init(&drain[i], 1);
    }
    s_abort = 0;
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*reinterpret_cast<volatile uint32_t*>(&s_tmem));
  pdl_wait();

  const int pos0 = warp_uniform(*p.pos);
  const int win = p.window > 0 ? p.window : 0x7fffffff;
  // keys that query tile i sees: [lo(i), hi(i)); tile 0 always has tokens
  auto lo_of = [&](int i) { return p.window > 0 ? max(0, pos0 + t0 + i * kXaTile - p.window + 1) : 0; };
  auto hi_of = [&](int i) { return pos0 + min(t0 + (i + 1) * kXaTile, p.rows); };
  const int lo = lo_of(0), hi = hi_of(nq - 1);
  auto sees = [&](int i, const XaKeyTile& t) { return i < nq && t.a < hi_of(i) && t.b > lo_of(i); };
  volatile int* abort = &s_abort;

  if (warp == 0) {  // queries and keys
    if (elect_one()) {
      mbar_expect_tx(&q_full, nq * k_bytes);
      for (int i = 0; i < nq; ++i)
        for (int c = 0; c < p.k_boxes; ++c) {
          const int x = head * (p.dimp + p.rotp) + (c < p.dim_boxes ? c * 64 : p.dimp + (c - p.dim_boxes) * 64);
          tma_load_2d(qs + i * k_bytes + c * kXaBox, &qmap, x, t0 + i * kXaTile, &q_full);
        }
    }
    uint32_t it = 0;
    for (int a = lo; a < hi; ++it) {
      const XaKeyTile t(a, hi, p.ring);
      a = t.b;
      const uint32_t s = it % kXaKeyStages;
      if (!mbar_wait_warp(&k_empty[s], ((it / kXaKeyStages) & 1u) ^ 1u, abort)) {
        set_status(p.status, ST_WAIT_EMPTY_TIMEOUT);
        *abort = 1;
        break;
      }
      if (elect_one()) {
        mbar_expect_tx(&k_full[s], k_bytes);
        for (int c = 0; c < p.k_boxes; ++c) {
          uint8_t* dst = ks + s * k_bytes + c * kXaBox;
          if (c < p.dim_boxes)
            tma_load_2d(dst, &kvmap, head * p.dimp + c * 64, t.row0, &k_full[s]);
          else
            tma_load_2d(dst, &rotmap, p.rankp + (c - p.dim_boxes) * 64, t.row0, &k_full[s]);
        }
      }
    }
    // copies still in flight must land before this CTA's shared memory goes away
    mbar_wait(&q_full, 0);
    for (uint32_t j = it > kXaKeyStages ? it - kXaKeyStages : 0; j < it; ++j) mbar_wait(&k_full[j % kXaKeyStages], (j / kXaKeyStages) & 1u);
  } else if (warp == 2) {  // values, on their own: they wait for other products than the keys do
    const uint32_t stages = p.v_stages;
    uint32_t it = 0;
    for (int a = lo; a < hi; ++it) {
      const XaKeyTile t(a, hi, p.ring);
      a = t.b;
      const uint32_t s = it % stages;
      if (!mbar_wait_warp(&v_empty[s], ((it / stages) & 1u) ^ 1u, abort)) {
        set_status(p.status, ST_WAIT_EMPTY_TIMEOUT);
        *abort = 1;
        break;
      }
      if (elect_one()) {
        mbar_expect_tx(&v_full[s], v_bytes);
        for (int c = 0; c < p.v_boxes; ++c)
          tma_load_2d(vs + s * v_bytes + c * kXaBox, &kvmap, p.heads * p.dimp + head * p.vdimp + c * 64, t.row0, &v_full[s]);
      }
    }
    for (uint32_t j = it > stages ? it - stages : 0; j < it; ++j) mbar_wait(&v_full[j % stages], (j / stages) & 1u);
  } else if (warp == 1 || (warp == 3 && nq == 2)) {  // the products of a query tile
    const int i = warp >> 1;
    const uint32_t s_idesc = umma_idesc_bf16(kXaTile, kXaHalf), v_idesc = umma_idesc_bf16(kXaTile, p.vdimp) | (1u << 16);
    const uint64_t qd0 = umma_desc_sw128(smem_u32(qs + i * k_bytes)), kd0 = umma_desc_sw128(smem_u32(ks));
    const uint64_t vd0 = umma_desc_sw128_columns(smem_u32(vs));
    const uint32_t ts = tmem + i * kXaTile, to = tmem + (NQ + i) * kXaTile;
    auto scores = [&](int h, uint32_t stage) {
      uint64_t qd = qd0, kd = kd0 + ((stage * k_bytes + h * kXaHalf * 128) >> 4);
      const uint32_t d = ts + h * kXaHalf;
      for (int c = 0; c < p.k_boxes; ++c, qd += kXaBox >> 4, kd += kXaBox >> 4) {
        const int left = c < p.dim_boxes ? p.dimp / 16 - c * 4 : p.rotp / 16 - (c - p.dim_boxes) * 4;  // steps of 16 columns, 32 bytes
        if (left >= 4) {
          if (elect_one()) {
#pragma unroll
            for (int q = 0; q < 4; ++q) umma_bf16(d, qd + 2 * q, kd + 2 * q, s_idesc, c | q);
          }
        } else if (elect_one()) {
          for (int q = 0; q < left; ++q) umma_bf16(d, qd + 2 * q, kd + 2 * q, s_idesc, c | q);
        }
      }
      if (elect_one()) umma_commit(&s_full[i][h]);
    };
    auto values = [&](int h, uint32_t stage, bool first) {
      const uint64_t vd = vd0 + ((stage * v_bytes + h * kXaHalf * 128) >> 4);
      if (elect_one()) {
#pragma unroll
        for (int c = 0; c < kXaHalf / 16; ++c)  // sixteen keys: eight columns of probabilities, sixteen rows of values
          umma_bf16_ta(to, ts + h * kXaHalf + c * 8, vd + c * (2048 >> 4), v_idesc, !first || c != 0);
        umma_commit(&v_done[i][h]);
      }
    };
    bool ok = mbar_wait_warp(&q_full, 0, abort);
    uint32_t n_p = 0;  // tiles whose probabilities have been taken
    uint32_t it = 0;
    int prev = -1;     // beginning of the tile before
    for (int a = lo; ok; ++it) {
      const bool more = a < hi;
      const XaKeyTile t(more ? a : hi - 1, hi, p.ring), u(prev < 0 ? lo : prev, hi, p.ring);
      const uint32_t ksg = it % kXaKeyStages, vsg = (it - 1) % p.v_stages;
      const bool take = prev >= 0 && sees(i, u), give = more && sees(i, t);
      if (prev >= 0) ok = mbar_wait_warp(&v_full[vsg], ((it - 1) / p.v_stages) & 1u, abort);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (ok && take) {
          ok = mbar_wait_warp(&p_full[i][h], n_p & 1u, abort);
          if (ok) {
            tc_fence_after();
            values(h, vsg, (n_p | h) == 0);
          }
        }
        if (ok && more && h == 0) ok = mbar_wait_warp(&k_full[ksg], (it / kXaKeyStages) & 1u, abort);
        if (ok && give) scores(h, ksg);
      }
      if (!ok) break;
      if (take) {
        ++n_p;
        if (u.b >= hi_of(i) && elect_one()) umma_commit(&o_full[i]);
      }
      if (prev >= 0 && elect_one()) umma_commit(&v_empty[vsg]);
      if (!more) break;
      if (elect_one()) umma_commit(&k_empty[ksg]);
      prev = a;
      a = t.b;
    }
    if (!ok) {
      set_status(p.status, ST_WAIT_FULL_TIMEOUT);
      *abort = 1;
    }
    __syncwarp();
    if (elect_one()) umma_commit(&drain[i]);  // products still running read shared memory and write TMEM
    mbar_wait(&drain[i], 0);
  } else if (warp >= 4 && (warp - 4) / 4 < nq) {
    const int i = (warp - 4) / 4, quad = warp & 3;
    const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t sc = tmem + i * kXaTile + lanes, so = tmem + (NQ + i) * kXaTile + lanes;
    const int t = t0 + i * kXaTile + quad * 32 + lane;
    const int first_q = pos0 + t0 + i * kXaTile, last_q = first_q + kXaTile - 1;
    const int qpos = t < p.rows ? pos0 + t : -1;  // a row without a token sees nothing
    const float c = p.scale * 1.4426950408889634f;
    float m = -INFINITY, l[4] = {0.f, 0.f, 0.f, 0.f};
    auto rescale = [&](float corr) {
      int v = 0;
      for (; v + 32 <= p.vdimp; v += 32) {
        uint32_t o[32];
        tmem_ld32_issue(so + v, o);
        tmem_wait_ld();
        tmem_use32(o);
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
        tmem_st32(so + v, o);
      }
      if (v < p.vdimp) {
        uint32_t o[16];
        tmem_ld16(so + v, o);
        tmem_ld16_wait(o);
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
        tmem_st16(so + v, o);
      }
    };
    uint32_t n = 0;
    bool ok = true;
    for (int a = lo; a < hi;) {
      const XaKeyTile kt(a, hi, p.ring);
      a = kt.b;
      if (!sees(i, kt)) continue;
      // every key of an inner tile is visible to every row (rows without a token are never stored)
      const bool inner = kt.key0 == kt.a && kt.b == kt.a + kXaTile && kt.b - 1 <= first_q && last_q - kt.a < win;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ok = mbar_wait(&s_full[i][h], n & 1u, abort);
        if (__any_sync(0xffffffffu, !ok)) {  // warp-uniform: tcgen05.ld needs every lane
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t r[2][32];
#pragma unroll
        for (int q = 0; q < 2; ++q) tmem_ld32_issue(sc + h * kXaHalf + q * 32, r[q]);
        tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 2; ++q) tmem_use32(r[q]);
        if (!inner) {
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int key = kt.key0 + h * kXaHalf + q * 32 + j;
              const bool hidden = key < kt.a || key >= kt.b || key > qpos || qpos - key >= win;
              if (hidden) r[q][j] = 0xff800000u;
            }
        }
        float top = m;
#pragma unroll
        for (int j = 0; j < 32; ++j) top = fmaxf(top, fmaxf(__uint_as_float(r[0][j]), __uint_as_float(r[1][j])));
        const float corr = top == m ? 1.f : exp2_approx((m - top) * c);
        m = top;
        const float mc = m == -INFINITY ? 0.f : m * c;
#pragma unroll
        for (int q = 0; q < 4; ++q) l[q] *= corr;
        uint32_t w[32];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float e0 = exp2_approx(fmaf(__uint_as_float(r[q][j]), c, -mc));
            const float e1 = exp2_approx(fmaf(__uint_as_float(r[q][j + 1]), c, -mc));
            l[2 * q] += e0;
            l[2 * q + 1] += e1;
            w[q * 16 + j / 2] = pack_bf16x2(e0, e1);
          }
        tmem_st32(sc + h * kXaHalf, w);
        if ((n > 0 || h > 0) && __any_sync(0xffffffffu, corr != 1.f)) {
          // the product of the half before writes the sums too
          ok = mbar_wait(&v_done[i][h ^ 1], (n - (h ^ 1)) & 1u, abort);
          if (__any_sync(0xffffffffu, !ok)) {
            ok = false;
            break;
          }
          tc_fence_after();
          rescale(corr);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[i][h]);
      }
      if (!ok) break;
      ++n;
    }
    if (ok) ok = mbar_wait(&o_full[i], 0, abort);
    if (__any_sync(0xffffffffu, !ok)) {
      set_status(p.status, ST_WAIT_FULL_TIMEOUT);
      *abort = 1;
    } else {
      tc_fence_after();
      const float sum = (l[0] + l[1]) + (l[2] + l[3]);
      float inv = 1.f / sum;
      if (p.sink != nullptr) {
        const float mm = m * p.scale, sk = p.sink[head], top = fmaxf(mm, sk), e = expf(mm - top);
        inv = e / (sum * e + expf(sk - top));
      }
      if (p.gate.per_head && t < p.rows) inv *= p.gate(t, head, p.vdim, 0);
      const bool gated = p.gate.z != nullptr && !p.gate.per_head;
      __nv_bfloat16* dst = p.out + static_cast<long long>(t) * p.ldo + static_cast<long long>(head) * p.vdim;
      const float* z = gated ? p.gate.z + static_cast<long long>(t) * p.gate.ld + static_cast<long long>(head) * p.vdim : nullptr;
      for (int v = 0; v < p.vdimp; v += 16) {
        uint32_t o[16];
        tmem_ld16(so + v, o);
        tmem_ld16_wait(o);
        float f[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(o[j]) * inv;
        if (t < p.rows && p.eights) {
#pragma unroll
          for (int q = 0; q < 16; q += 8) {
            if (v + q >= p.vdim) break;
            float g[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] = f[q + j];
            if (gated) {
              float zz[8];
              act_ld8(z + v + q, zz);
#pragma unroll
              for (int j = 0; j < 8; ++j) g[j] *= 1.f / (1.f + expf(-zz[j]));
            }
            act_st8(dst + v + q, g);
          }
        } else if (t < p.rows) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (v + j < p.vdim) dst[v + j] = f2bf(gated ? f[j] * (1.f / (1.f + expf(-z[v + j]))) : f[j]);
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

}  // namespace tb
