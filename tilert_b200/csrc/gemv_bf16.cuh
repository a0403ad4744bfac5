// bf16-weight GEMV with f32 accumulation for the products that are not FP8 in the checkpoint:
// the MoE router gate, the indexer head-weight projection and the vocabulary head.
// HBM-bound on the weight stream: each warp keeps several 16-byte loads per lane in flight; the (optionally
// RMS-normalised) activations sit in shared memory.
#pragma once

#include "common.cuh"

namespace tb {

struct GemvBf16Params {
  const void* w;                 // [n, k] bf16 (w_is_f32 = 0) or f32 (w_is_f32 = 1), row-major
  int w_is_f32;
  int n, k;                      // k multiple of 256
  const __nv_bfloat16* x;        // [tokens, k]
  long long x_stride;
  int n_tokens;                  // 1..4
  const float* gamma;            // optional RMSNorm gain
  float eps;
  int round_norm_bf16;           // 1: normalised activations are rounded to bf16 before the product
  __nv_bfloat16* xnorm_out;      // optional [tokens, k] (written by CTA 0)
  long long xnorm_stride;
  // Optional second segment (row-per-warp kernel only): activations [k1, k) come from x2 and are
  // normalised on their own with gamma2 -- the MTP input "concat(enorm(e), hnorm(h))".
  const __nv_bfloat16* x2;       // [tokens, k - k1]; nullptr = one segment
  long long x2_stride;
  int k1;
  const float* gamma2;
  __nv_bfloat16* xnorm2_out;     // optional [tokens, k - k1] (written by CTA 0)
  long long xnorm2_stride;
  void* out;                     // [tokens, n] f32 (out_bf16 = 0) or bf16 (out_bf16 = 1)
  int out_bf16;
  long long out_stride;
  int aligned;                   // x, x2, their rows and the gains are 16-byte aligned
};

constexpr int kGemvBf16Threads = 512;

// Eight activations (a piece) of a token as staged in shared memory: bf16 where they are bf16 values (rounded, or not
// normalised), else f32 with the halves of a piece apart -- a warp's 16-byte reads are free of bank conflicts either way.
template <typename X>
struct GemvX;
template <>
struct GemvX<__nv_bfloat16> {
  static __host__ __device__ size_t bytes(int k) { return static_cast<size_t>(k) * 2; }
  static __device__ __forceinline__ void get(const uint8_t* base, int, int piece, float (&f)[8]) {
    const uint4 u = reinterpret_cast<const uint4*>(base)[piece];
    f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
    f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
    f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
  }
  static __device__ __forceinline__ float4 four(const uint8_t* base, int, int i) {
    const uint2 u = *reinterpret_cast<const uint2*>(base + i * 2);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
  }
  static __device__ __forceinline__ void put(uint8_t* base, int, int piece, const float (&f)[8]) {
    reinterpret_cast<uint4*>(base)[piece] = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
  }
};
template <>
struct GemvX<float> {
  static __host__ __device__ size_t bytes(int k) { return static_cast<size_t>(k) * 4; }
  static __device__ __forceinline__ void get(const uint8_t* base, int k, int piece, float (&f)[8]) {
    const float4 a = reinterpret_cast<const float4*>(base)[piece], b = reinterpret_cast<const float4*>(base)[k / 8 + piece];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  static __device__ __forceinline__ float4 four(const uint8_t* base, int k, int i) {
    return reinterpret_cast<const float4*>(base)[(i & 4 ? k / 8 : 0) + (i >> 3)];
  }
  static __device__ __forceinline__ void put(uint8_t* base, int k, int piece, const float (&f)[8]) {
    reinterpret_cast<float4*>(base)[piece] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4*>(base)[k / 8 + piece] = make_float4(f[4], f[5], f[6], f[7]);
  }
};
// A lane's eight weights, as loaded, and activations of a step of 256 elements: a piece of eight bf16 weights, or two pieces of
// four f32 ones 128 elements apart.  A piece's products are summed first, then added to the lane's sum.
template <typename W>
struct GemvW;
template <>
struct GemvW<__nv_bfloat16> {
  uint4 u;
  __device__ __forceinline__ void load(const void* w, long long step_at, int lane) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                 : "l"(reinterpret_cast<const __nv_bfloat16*>(w) + step_at + lane * 8));
  }
  template <typename X>
  static __device__ __forceinline__ void operand(const uint8_t* base, int k, int step, int lane, float (&f)[8]) {
    GemvX<X>::get(base, k, step * 32 + lane, f);
  }
  static __device__ __forceinline__ void add(float& acc, const float (&w)[8], const float (&f)[8]) {
    acc += w[0] * f[0] + w[1] * f[1] + w[2] * f[2] + w[3] * f[3] + w[4] * f[4] + w[5] * f[5] + w[6] * f[6] + w[7] * f[7];
  }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
    f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
    f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
  }
};
template <>
struct GemvW<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const void* w, long long step_at, int lane) {
    const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(w) + step_at) + lane;
    a = __ldg(p);
    b = __ldg(p + 32);
  }
  template <typename X>
  static __device__ __forceinline__ void operand(const uint8_t* base, int k, int step, int lane, float (&f)[8]) {
    const float4 x = GemvX<X>::four(base, k, step * 256 + lane * 4), y = GemvX<X>::four(base, k, step * 256 + 128 + lane * 4);
    f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
    f[4] = y.x; f[5] = y.y; f[6] = y.z; f[7] = y.w;
  }
  static __device__ __forceinline__ void add(float& acc, const float (&w)[8], const float (&f)[8]) {
    acc += w[0] * f[0] + w[1] * f[1] + w[2] * f[2] + w[3] * f[3];
    acc += w[4] * f[4] + w[5] * f[5] + w[6] * f[6] + w[7] * f[7];
  }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
};

// Sums v[0 .. N) over the warp, N a power of two up to 32: while there are several, lanes an offset apart exchange the
// halves they do not keep, so N sums cost about N + 4 shuffles.  Lane l ends with the sum of v[l >> (5 - log2 N)].
template <int N>
__device__ __forceinline__ float warp_sums(float (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int cnt = N;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (cnt > 1) {
      cnt >>= 1;
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        if (i < cnt) {
          const float got = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + cnt], o);
          v[i] = (up ? v[i + cnt] : v[i]) + got;
        }
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

// Long weights (vocabulary head, eh_proj).  A warp owns four rows at a time, so that a staged piece of the activations
// serves four weights, and keeps the next two steps of 256 elements requested: 12 sixteen-byte loads per lane.  (With a
// row per warp the reads of the activations are the bound for several tokens.)  Rows that are no more than the warps go one
// to a warp with seven steps requested: nothing is shared, and a walk along K is all there is to wait for.
// Statistics and products are summed in the order of a row per warp and an element per thread in every form, so that the
// results have the same bits.  Back to back, head 16160 x 7168, one / two / four tokens: 46.4 / 48.6 / 53.5 us (a row per
// warp, without steps requested, 64.9 / 114.9 / 147.5); eh_proj 7168 x 14336: 44.4 / 46.4 / 53.1 (69.1 / 91.7 / 183.4).
// Every CTA normalises the vector for itself: gains in 16-byte loads take 0.7 to 1.3 us off any size (512 rows of 14336, one
// token: 28.7 us, an element at a time 29.9).
template <int TOK, int ROWS, typename X, typename W>
__global__ void __launch_bounds__(kGemvBf16Threads, 1) gemv_bf16_kernel(const GemvBf16Params p) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t gsm[];  // [TOK] GemvX<X>
  __shared__ float red[2][TOK][16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kWarps = kGemvBf16Threads / 32;
  constexpr int kAhead = ROWS == 1 ? (sizeof(W) == 2 ? 7 : 3) : 2;  // steps (256 elements of the warp's rows) requested beyond the current one
  const size_t x_bytes = GemvX<X>::bytes(p.k);
  const int pieces = p.k / 8, steps = pieces / 32;
  const int groups = (p.n + ROWS - 1) / ROWS, stride = gridDim.x * kWarps;

  GemvW<W> w[kAhead + 1][ROWS];
  auto request = [&](int group, int step, GemvW<W> (&dst)[ROWS]) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r)  // rows past the end: the last one, dropped below
      dst[r].load(p.w, static_cast<long long>(min(group * ROWS + r, p.n - 1)) * p.k + step * 256, lane);
  };
  int group = warp * gridDim.x + blockIdx.x;  // neighbouring CTAs read neighbouring rows
  int pg = group, ps = 0;                     // the next step to request
  auto advance = [&] {
    if (++ps == steps) {
      ps = 0;
      pg += stride;
    }
  };
  // the weights do not depend on the predecessor
#pragma unroll
  for (int d = 0; d < kAhead; ++d) {
    if (pg < groups) request(pg, ps, w[d]);
    advance();
  }

  // stage (and normalise) the activations; with a second segment each one has its own statistics
  pdl_wait();
  const int k1 = p.x2 != nullptr ? p.k1 : p.k;
  for (int i = threadIdx.x; i < pieces; i += kGemvBf16Threads) {
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      float f[8] = {};
      if (t < p.n_tokens) {
        const __nv_bfloat16* src = i * 8 < k1 ? p.x + t * p.x_stride + i * 8 : p.x2 + t * p.x2_stride + i * 8 - k1;
        if (p.aligned) {
          const uint4 u = *reinterpret_cast<const uint4*>(src);
          const uint32_t q[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            f[2 * j] = __uint_as_float(q[j] << 16);
            f[2 * j + 1] = __uint_as_float(q[j] & 0xffff0000u);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = bf2f(src[j]);
        }
      }
      GemvX<X>::put(gsm + t * x_bytes, p.k, i, f);
    }
  }
  if (p.gamma != nullptr) {
    // Four warps per token.  A thread sums the squares of four neighbouring elements of every 512, each on its own, and 32 such
    // sums are added as a warp that holds one each would add them.
    __syncthreads();
    if (warp / 4 < TOK) {
      const int t = warp / 4, q = threadIdx.x & 127;
      float ss[4] = {}, ss2[4] = {};
#pragma unroll 7
      for (int i = q * 4; i < p.k; i += 512) {
        const float4 v = GemvX<X>::four(gsm + t * x_bytes, p.k, i);
        const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (i < k1) ss[j] += f[j] * f[j]; else ss2[j] += f[j] * f[j];
        }
      }
      auto thirty_two = [](float (&v)[4]) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        return (v[0] + v[2]) + (v[1] + v[3]);
      };
      const float s = thirty_two(ss), s2 = thirty_two(ss2);
      if (q % 8 == 0) {
        red[0][t][q / 8] = s;
        red[1][t][q / 8] = s2;
      }
    }
    __syncthreads();
    float rinv[TOK], rinv2[TOK];
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      const float tot = warp_sum(lane < 16 ? red[0][t][lane] : 0.f), tot2 = warp_sum(lane < 16 ? red[1][t][lane] : 0.f);
      rinv[t] = rsqrtf(tot / static_cast<float>(k1) + p.eps);
      rinv2[t] = rsqrtf(tot2 / static_cast<float>(p.k - k1 > 0 ? p.k - k1 : 1) + p.eps);
    }
    for (int i = threadIdx.x; i < pieces; i += kGemvBf16Threads) {  // every thread rescales what it wrote
      const bool first = i * 8 < k1;
      const float* gains = first ? p.gamma + i * 8 : p.gamma2 + i * 8 - k1;
      float g[8];
      if (p.aligned) {
        const float4 lo = __ldg(reinterpret_cast<const float4*>(gains)), hi = __ldg(reinterpret_cast<const float4*>(gains) + 1);
        g[0] = lo.x; g[1] = lo.y; g[2] = lo.z; g[3] = lo.w;
        g[4] = hi.x; g[5] = hi.y; g[6] = hi.z; g[7] = hi.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = gains[j];
      }
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        float f[8];
        GemvX<X>::get(gsm + t * x_bytes, p.k, i, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * (first ? rinv[t] : rinv2[t]) * g[j];
        GemvX<X>::put(gsm + t * x_bytes, p.k, i, f);
        __nv_bfloat16* out = first ? p.xnorm_out : p.xnorm2_out;
        if (blockIdx.x == 0 && t < p.n_tokens && out != nullptr) {
          out += first ? t * p.xnorm_stride + i * 8 : t * p.xnorm2_stride + i * 8 - k1;
#pragma unroll
          for (int j = 0; j < 8; ++j) out[j] = f2bf(f[j]);
        }
      }
    }
  }
  __syncthreads();

  for (; group < groups; group += stride) {
    float acc[ROWS * TOK];
#pragma unroll
    for (int i = 0; i < ROWS * TOK; ++i) acc[i] = 0.f;
#pragma unroll (kAhead + 1)
    for (int s = 0; s < steps; ++s) {
      if (pg < groups) request(pg, ps, w[kAhead]);
      advance();
      float wf[ROWS][8];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) w[0][r].get(wf[r]);
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        float f[8];
        GemvW<W>::template operand<X>(gsm + t * x_bytes, p.k, s, lane, f);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) GemvW<W>::add(acc[r * TOK + t], wf[r], f);
      }
#pragma unroll
      for (int d = 0; d < kAhead; ++d)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) w[d][r] = w[d + 1][r];
    }
    constexpr int kSums = ROWS * TOK, kLanes = 32 / kSums;  // lanes that hold the same sum
    const float sum = warp_sums<kSums>(acc);
    const int i = lane / kLanes, row = group * ROWS + i / TOK, t = i % TOK;
    if (lane % kLanes == 0 && row < p.n && t < p.n_tokens) {
      if (p.out_bf16)
        reinterpret_cast<__nv_bfloat16*>(p.out)[t * p.out_stride + row] = f2bf(sum);
      else
        reinterpret_cast<float*>(p.out)[t * p.out_stride + row] = sum;
    }
  }
}

// Variant for few rows (router gate, indexer head weights): one CTA per pair of rows, the warps
// split K, so the dependent load chain is K / (8 warps * 256) iterations instead of K / 256.
// Latency: a few round trips to L2 and what four tokens move through shared memory.  The activations stay in registers until they
// are normalised, go to shared memory once, in pieces with their halves apart (scalar stores eight floats apart met in four
// banks), and are read once for both rows.  Scalar staging, a pass per row -> now: 64 rows of 7168, four tokens 11.5 -> 9.0 us,
// inside attn_prep_kernel 10.8 -> 7.8; one token 256 rows 5.9 -> 5.2.
constexpr int kGemvBf16SmallThreads = 256;
constexpr int kGemvBf16SmallRows = 2;

// `block` = index of the row pair; `xs` = [TOK][k] floats of shared memory.  The weights of the
// block's two rows are requested before the wait for the predecessor kernel: they are static, and
// their DRAM latency then overlaps the activation staging and the normalisation.
template <int TOK>
__device__ __forceinline__ void gemv_bf16_ksplit_body(const GemvBf16Params& p, int block, float* xs) {
  __shared__ float red[TOK][8];
  __shared__ float part[kGemvBf16SmallRows][TOK][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kslice = p.k / 8;  // per warp; multiple of 8 elements (k % 256 == 0); at most 1024 (k <= 8192)
  uint4 wpre[kGemvBf16SmallRows][4][2];  // [row][iteration][bf16: .0 only | f32: two halves]
#pragma unroll
  for (int r = 0; r < kGemvBf16SmallRows; ++r) {
    const int row = block * kGemvBf16SmallRows + r;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int k0 = warp * kslice + lane * 8 + it * 256;
      wpre[r][it][0] = make_uint4(0u, 0u, 0u, 0u);
      wpre[r][it][1] = make_uint4(0u, 0u, 0u, 0u);
      if (row < p.n && k0 < (warp + 1) * kslice) {
        if (p.w_is_f32) {
          const float* wr = reinterpret_cast<const float*>(p.w) + static_cast<long long>(row) * p.k + k0;
          wpre[r][it][0] = __ldg(reinterpret_cast<const uint4*>(wr));
          wpre[r][it][1] = __ldg(reinterpret_cast<const uint4*>(wr + 4));
        } else {
          const __nv_bfloat16* wr = reinterpret_cast<const __nv_bfloat16*>(p.w) + static_cast<long long>(row) * p.k + k0;
          wpre[r][it][0] = __ldg(reinterpret_cast<const uint4*>(wr));
        }
      }
    }
  }
  pdl_wait();
  // all of this thread's activation loads first (k <= 8192: at most four pieces of eight per token) and, behind them, the gains of
  // the same elements: a plain loop would pay one memory round trip per iteration
  uint4 xraw[4][TOK];
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int i = (it * kGemvBf16SmallThreads + threadIdx.x) * 8;
#pragma unroll
    for (int t = 0; t < TOK; ++t)
      xraw[it][t] = (i < p.k && t < p.n_tokens) ? *reinterpret_cast<const uint4*>(p.x + t * p.x_stride + i)
                                                : make_uint4(0, 0, 0, 0);
  }
  auto piece_of = [&](int it, int t, float (&f)[8]) {
    const uint32_t wv[4] = {xraw[it][t].x, xraw[it][t].y, xraw[it][t].z, xraw[it][t].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[2 * j] = __uint_as_float(wv[j] << 16);
      f[2 * j + 1] = __uint_as_float(wv[j] & 0xffff0000u);
    }
  };
  float rinv[TOK];
  float4 gm[4][2];
  if (p.gamma != nullptr) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = (it * kGemvBf16SmallThreads + threadIdx.x) * 8;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        gm[it][h] = i < p.k ? __ldg(reinterpret_cast<const float4*>(p.gamma + i) + h) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      float ss = 0.f;
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        float f[8];
        piece_of(it, t, f);
#pragma unroll
        for (int j = 0; j < 4; ++j) ss += f[2 * j] * f[2 * j] + f[2 * j + 1] * f[2 * j + 1];
      }
      const float s = warp_sum(ss);
      if (lane == 0) red[t][warp] = s;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      float tot = lane < 8 ? red[t][lane] : 0.f;
      tot = warp_sum(tot);
      rinv[t] = rsqrtf(tot / static_cast<float>(p.k) + p.eps);
    }
  }
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int piece = it * kGemvBf16SmallThreads + threadIdx.x, i = piece * 8;
    if (i < p.k) {
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        float f[8];
        piece_of(it, t, f);
        if (p.gamma != nullptr) {
          const float g[8] = {gm[it][0].x, gm[it][0].y, gm[it][0].z, gm[it][0].w, gm[it][1].x, gm[it][1].y, gm[it][1].z, gm[it][1].w};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            f[j] = f[j] * rinv[t] * g[j];
            if (p.round_norm_bf16) f[j] = bf2f(f2bf(f[j]));
          }
          if (p.xnorm_out != nullptr && block == 0 && t < p.n_tokens) {
            uint2* out = reinterpret_cast<uint2*>(p.xnorm_out + t * p.xnorm_stride + i);
            out[0] = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
            out[1] = make_uint2(pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          }
        }
        GemvX<float>::put(reinterpret_cast<uint8_t*>(xs + t * p.k), p.k, piece, f);
      }
    }
  }
  __syncthreads();

  float acc[kGemvBf16SmallRows][TOK];
#pragma unroll
  for (int r = 0; r < kGemvBf16SmallRows; ++r)
#pragma unroll
    for (int t = 0; t < TOK; ++t) acc[r][t] = 0.f;
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int k0 = warp * kslice + lane * 8 + it * 256;
    if (k0 < (warp + 1) * kslice) {
      float wf[kGemvBf16SmallRows][8];  // (rows past the end: zeros)
#pragma unroll
      for (int r = 0; r < kGemvBf16SmallRows; ++r) {
        const uint4 w0 = wpre[r][it][0], w1 = wpre[r][it][1];
        if (p.w_is_f32) {
          wf[r][0] = __uint_as_float(w0.x); wf[r][1] = __uint_as_float(w0.y); wf[r][2] = __uint_as_float(w0.z);
          wf[r][3] = __uint_as_float(w0.w); wf[r][4] = __uint_as_float(w1.x); wf[r][5] = __uint_as_float(w1.y);
          wf[r][6] = __uint_as_float(w1.z); wf[r][7] = __uint_as_float(w1.w);
        } else {
          const uint32_t ww[4] = {w0.x, w0.y, w0.z, w0.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            wf[r][2 * j] = __uint_as_float(ww[j] << 16);
            wf[r][2 * j + 1] = __uint_as_float(ww[j] & 0xffff0000u);
          }
        }
      }
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        float x[8];
        GemvX<float>::get(reinterpret_cast<const uint8_t*>(xs + t * p.k), p.k, k0 / 8, x);
#pragma unroll
        for (int r = 0; r < kGemvBf16SmallRows; ++r)
          acc[r][t] += wf[r][0] * x[0] + wf[r][1] * x[1] + wf[r][2] * x[2] + wf[r][3] * x[3] + wf[r][4] * x[4] + wf[r][5] * x[5] +
                       wf[r][6] * x[6] + wf[r][7] * x[7];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kGemvBf16SmallRows; ++r)
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      const float s = warp_sum(acc[r][t]);
      if (lane == 0) part[r][t][warp] = s;
    }
  __syncthreads();
  if (threadIdx.x < kGemvBf16SmallRows * TOK) {
    const int r = threadIdx.x / TOK, t = threadIdx.x % TOK;
    const int row = block * kGemvBf16SmallRows + r;
    if (row < p.n && t < p.n_tokens) {
      float s = 0.f;
#pragma unroll
      for (int w2 = 0; w2 < 8; ++w2) s += part[r][t][w2];
      if (p.out_bf16)
        reinterpret_cast<__nv_bfloat16*>(p.out)[t * p.out_stride + row] = f2bf(s);
      else
        reinterpret_cast<float*>(p.out)[t * p.out_stride + row] = s;
    }
  }
}

template <int TOK>
__global__ void __launch_bounds__(kGemvBf16SmallThreads) gemv_bf16_ksplit_kernel(const GemvBf16Params p) {
  extern __shared__ __align__(16) float xs[];  // [TOK][k]
  pdl_launch_dependents();
  gemv_bf16_ksplit_body<TOK>(p, blockIdx.x, xs);
}

}  // namespace tb
