// Row kernels around the norms of a residual stream kept in f32: embedding + norm, sublayer output -> norm ->
// residual (-> norm of the next sublayer's input), and the norm in front of the vocabulary head.  One CTA per token; the
// gain vectors are f32 and already hold the factor the norm multiplies with (a weight that is an offset from one arrives
// as 1 + w).  A norm is the RMS norm, or with `centered` the layer norm (mean taken off first); biases are optional.
//
// The embedding and the residual kernels are bound by memory (14 bytes per element of a residual step with a norm behind
// it) and have two forms.  Up to 8192 wide, in multiples of eight and with aligned rows, a thread owns one or two pieces
// of eight elements and keeps them in registers from the loads to the stores: every operand is requested in 16-byte
// pieces before the first reduction, and memory sees each element once.  Other shapes take an element at a time through
// shared memory.  Both forms of an RMS norm sum the squares in one order, so that a row has the same bits in either: what
// follows such a norm may be a choice of experts, where a last bit can decide a near tie.
#pragma once

#include "act.cuh"

namespace tb {

constexpr int kNormThreads = 256;

struct RowStat {
  float mean, rinv;
};

// Statistics of n values that get(i) returns, the calling thread owning i = threadIdx.x, + blockDim.x, ...  The squared
// deviations are summed in a pass of their own (no cancellation).
template <class Get>
__device__ __forceinline__ RowStat row_stat(int n, float eps, int centered, float* red, Get get) {
  float mean = 0.f;
  if (centered) {
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += get(i);
    mean = cta_sum(s, red) / static_cast<float>(n);
  }
  float ss = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float d = get(i) - mean;
    ss += d * d;
  }
  return {mean, 1.f / sqrtf(cta_sum(ss, red) / static_cast<float>(n) + eps)};
}
__device__ __forceinline__ float row_norm(float v, const RowStat& st, const float* gain, const float* bias, int i) {
  return (v - st.mean) * st.rinv * gain[i] + (bias != nullptr ? bias[i] : 0.f);
}

// ------------------------------------------------------------------ rows in registers
// NJ pieces of eight elements per thread: piece j of thread i is elements (i + j * TH) * 8 ..  The threads are as many as
// give one piece each up to 4096: a row then has the most loads under way for the registers it holds.
constexpr int kRowThreads = 512, kRowPieces = 2;  // most of both

template <int TH, int NJ, class Each>
__device__ __forceinline__ void each_piece(int dim, Each each) {
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int e = (static_cast<int>(threadIdx.x) + j * TH) * 8;
    if (e < dim) each(j, e);
  }
}
// Pieces beyond dim hold zeros.  The RMS norm turns the row over in shared memory (`vals`, [dim]) and sums as row_stat with
// kNormThreads threads does.
template <int TH, int NJ>
__device__ __forceinline__ RowStat piece_stat(const float (&v)[NJ][8], int dim, float eps, int centered, float* red, float* vals) {
  float ss = 0.f;
  if (!centered) {
    static_assert(TH >= kNormThreads, "every partial sum has its thread");
    each_piece<TH, NJ>(dim, [&](int j, int e) { act_st8(vals + e, v[j]); });
    __syncthreads();
    if (threadIdx.x < kNormThreads) {
#pragma unroll 8
      for (int i = threadIdx.x; i < dim; i += kNormThreads) ss += vals[i] * vals[i];
    }
    return {0.f, 1.f / sqrtf(cta_sum(ss, red) / static_cast<float>(dim) + eps)};
  }
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int q = 0; q < 8; ++q) s += v[j][q];
  const float mean = cta_sum(s, red) / static_cast<float>(dim);
  each_piece<TH, NJ>(dim, [&](int j, int) {
#pragma unroll
    for (int q = 0; q < 8; ++q) ss += (v[j][q] - mean) * (v[j][q] - mean);
  });
  return {mean, 1.f / sqrtf(cta_sum(ss, red) / static_cast<float>(dim) + eps)};
}
// v = norm(v) * gain + bias, one piece
__device__ __forceinline__ void norm_piece(float (&v)[8], const RowStat& st, const float* gain, const float* bias, int e) {
  float g[8], b[8];
  act_ld8(gain + e, g);
  if (bias != nullptr) act_ld8(bias + e, b);
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = (v[q] - st.mean) * st.rinv * g[q] + (bias != nullptr ? b[q] : 0.f);
}

struct EmbedNormParams {
  const long long* tokens;      // [rows]
  const __nv_bfloat16* table;   // [vocab, ld_table]
  long long ld_table;
  int vocab;
  const float* gain;            // null: the embedding as it is
  float eps;
  int dim;
  float* x;                     // [rows, ldx] f32 residual
  long long ldx;
  void* xh;                     // optional [rows, ldh] activations
  long long ldh;
  int* status;
};

template <typename T>
__global__ void __launch_bounds__(kNormThreads) embed_norm_kernel(const EmbedNormParams p) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[32];
  const int t = blockIdx.x;
  const long long tok = p.tokens[t];
  if (tok < 0 || tok >= p.vocab) {  // uniform over the CTA
    if (threadIdx.x == 0) set_status(p.status, ST_BAD_ARGUMENT);
    return;
  }
  const __nv_bfloat16* row = p.table + tok * p.ld_table;
  RowStat st{0.f, 1.f};
  if (p.gain != nullptr) st = row_stat(p.dim, p.eps, 0, red, [&](int i) { return bf2f(row[i]); });
  for (int i = threadIdx.x; i < p.dim; i += kNormThreads) {
    const float v = p.gain != nullptr ? row_norm(bf2f(row[i]), st, p.gain, nullptr, i) : bf2f(row[i]);
    p.x[t * p.ldx + i] = v;
    if (p.xh != nullptr) act_st(reinterpret_cast<T*>(p.xh) + t * p.ldh + i, v);
  }
}

template <typename T, int TH, int NJ>
__global__ void __launch_bounds__(TH) embed_norm_pieces_kernel(const EmbedNormParams p) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float vals[];  // [dim], with a gain
  __shared__ float red[32];
  const int t = blockIdx.x;
  const long long tok = p.tokens[t];
  if (tok < 0 || tok >= p.vocab) {  // uniform over the CTA
    if (threadIdx.x == 0) set_status(p.status, ST_BAD_ARGUMENT);
    return;
  }
  const __nv_bfloat16* row = p.table + tok * p.ld_table;
  float v[NJ][8] = {};
  each_piece<TH, NJ>(p.dim, [&](int j, int e) { act_ld8(row + e, v[j]); });
  if (p.gain != nullptr) {
    const RowStat st = piece_stat<TH, NJ>(v, p.dim, p.eps, 0, red, vals);
    each_piece<TH, NJ>(p.dim, [&](int j, int e) { norm_piece(v[j], st, p.gain, nullptr, e); });
  }
  each_piece<TH, NJ>(p.dim, [&](int j, int e) {
    act_st8(p.x + t * p.ldx + e, v[j]);
    if (p.xh != nullptr) act_st8(reinterpret_cast<T*>(p.xh) + t * p.ldh + e, v[j]);
  });
}

// x[t] += norm(y[t]) (+ add), where the sublayer output y is either one row, or a weighted sum of rows of expert
// outputs (row slot_row[t, j], weight slot_w[t, j]) plus an optional further row (a shared expert), or absent.  xh is
// x, or its norm with gain2.
struct ResidualNormParams {
  const float* y;               // [rows, ldy] f32, or null with slots
  long long ldy;
  const void* ye;               // expert outputs [*, lde], element type T
  long long lde;
  const int* slot_row;          // [rows, top]
  const float* slot_w;          // [rows, top]
  int top;
  const void* ysh;              // optional [rows, ldsh], element type T
  long long ldsh;
  const float* gain;            // null: no sublayer output
  const float* bias;            // optional
  const float* add;             // optional [dim], the same for every row
  const float* gain2;           // optional norm of the new x, for xh alone
  const float* bias2;           // optional
  int centered;                 // both norms
  float eps;
  int dim;
  float* x;                     // [rows, ldx] f32, updated
  long long ldx;
  void* xh;                     // optional [rows, ldh] x (or its norm) as activations
  long long ldh;
};

template <typename T>
__global__ void __launch_bounds__(kNormThreads) residual_norm_kernel(const ResidualNormParams p) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float vals[];  // [dim]
  __shared__ float red[32];
  const int t = blockIdx.x;
  if (p.y != nullptr) {
    const float* y = p.y + t * p.ldy;
    for (int i = threadIdx.x; i < p.dim; i += kNormThreads) vals[i] = y[i];
  } else if (p.ye != nullptr) {
    const int n8 = pad_to(p.dim, 8) / 8;
    for (int c = threadIdx.x; c < n8; c += kNormThreads) {
      float acc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = 0.f;
      for (int j = 0; j < p.top; ++j) {
        const float w = p.slot_w[t * p.top + j];
        float f[8];
        act_ld8(reinterpret_cast<const T*>(p.ye) + static_cast<long long>(p.slot_row[t * p.top + j]) * p.lde + c * 8, f);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] += w * f[q];
      }
      if (p.ysh != nullptr) {
        float f[8];
        act_ld8(reinterpret_cast<const T*>(p.ysh) + t * p.ldsh + c * 8, f);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] += f[q];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (c * 8 + q < p.dim) vals[c * 8 + q] = acc[q];
    }
    __syncthreads();  // the pieces were eight wide
  }
  RowStat st{0.f, 0.f};
  if (p.gain != nullptr) st = row_stat(p.dim, p.eps, p.centered, red, [&](int i) { return vals[i]; });
  float* x = p.x + t * p.ldx;
  T* xh = p.xh != nullptr ? reinterpret_cast<T*>(p.xh) + t * p.ldh : nullptr;
  for (int i = threadIdx.x; i < p.dim; i += kNormThreads) {
    float v = x[i];
    if (p.gain != nullptr) v += row_norm(vals[i], st, p.gain, p.bias, i);
    if (p.add != nullptr) v += p.add[i];
    x[i] = v;
    if (p.gain2 != nullptr)
      vals[i] = v;
    else if (xh != nullptr)
      act_st(xh + i, v);
  }
  if (p.gain2 == nullptr) return;
  const RowStat s2 = row_stat(p.dim, p.eps, p.centered, red, [&](int i) { return vals[i]; });
  for (int i = threadIdx.x; i < p.dim; i += kNormThreads) act_st(xh + i, row_norm(vals[i], s2, p.gain2, p.bias2, i));
}

// The same from registers.  With a norm behind the step, B200, back to back: 2048 rows of 4096 in 31.8 us (3.7 TB/s), an
// element at a time 42.9; 2048 x 7168 53.2 (72.4); 173 x 2048 4.7 (8.2).  Eight experts and a shared one combined into
// 2048 x 4096: 53.3 (56.9).
template <typename T, int TH, int NJ>
__global__ void __launch_bounds__(TH, NJ == 1 ? 1536 / TH : 1024 / TH) residual_norm_pieces_kernel(const ResidualNormParams p) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float vals[];  // [dim], not centered
  __shared__ float red[32];
  const int t = blockIdx.x;
  float* x = p.x + t * p.ldx;
  float v[NJ][8] = {}, r[NJ][8] = {};  // the sublayer's output, the residual
  each_piece<TH, NJ>(p.dim, [&](int j, int e) { act_ld8(x + e, r[j]); });
  if (p.y != nullptr) {
    each_piece<TH, NJ>(p.dim, [&](int j, int e) { act_ld8(p.y + t * p.ldy + e, v[j]); });
  } else if (p.ye != nullptr) {
    const T* ye = reinterpret_cast<const T*>(p.ye);
#pragma unroll 4
    for (int s = 0; s < p.top; ++s) {
      const float w = p.slot_w[t * p.top + s];
      const T* src = ye + static_cast<long long>(p.slot_row[t * p.top + s]) * p.lde;
      each_piece<TH, NJ>(p.dim, [&](int j, int e) {
        float f[8];
        act_ld8(src + e, f);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[j][q] += w * f[q];
      });
    }
    if (p.ysh != nullptr)
      each_piece<TH, NJ>(p.dim, [&](int j, int e) {
        float f[8];
        act_ld8(reinterpret_cast<const T*>(p.ysh) + t * p.ldsh + e, f);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[j][q] += f[q];
      });
  }
  if (p.gain != nullptr) {
    const RowStat st = piece_stat<TH, NJ>(v, p.dim, p.eps, p.centered, red, vals);
    each_piece<TH, NJ>(p.dim, [&](int j, int e) {
      norm_piece(v[j], st, p.gain, p.bias, e);
#pragma unroll
      for (int q = 0; q < 8; ++q) r[j][q] += v[j][q];
    });
  }
  if (p.add != nullptr)
    each_piece<TH, NJ>(p.dim, [&](int j, int e) {
      float f[8];
      act_ld8(p.add + e, f);
#pragma unroll
      for (int q = 0; q < 8; ++q) r[j][q] += f[q];
    });
  each_piece<TH, NJ>(p.dim, [&](int j, int e) { act_st8(x + e, r[j]); });
  if (p.xh == nullptr) return;
  T* xh = reinterpret_cast<T*>(p.xh) + t * p.ldh;
  if (p.gain2 != nullptr) {
    const RowStat st = piece_stat<TH, NJ>(r, p.dim, p.eps, p.centered, red, vals);
    each_piece<TH, NJ>(p.dim, [&](int j, int e) { norm_piece(r[j], st, p.gain2, p.bias2, e); });
  }
  each_piece<TH, NJ>(p.dim, [&](int j, int e) { act_st8(xh + e, r[j]); });
}

// out[r] = norm(x[rows[r]])
struct GatherNormParams {
  const float* x;
  long long ldx;
  const int* rows;              // [n]
  const float* gain;
  const float* bias;            // optional
  int centered;
  float eps;
  int dim;
  void* out;                    // [n, ldo]
  long long ldo;
};

template <typename T>
__global__ void __launch_bounds__(kNormThreads) gather_norm_kernel(const GatherNormParams p) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[32];
  const float* x = p.x + static_cast<long long>(p.rows[blockIdx.x]) * p.ldx;
  const RowStat st = row_stat(p.dim, p.eps, p.centered, red, [&](int i) { return x[i]; });
  T* o = reinterpret_cast<T*>(p.out) + blockIdx.x * p.ldo;
  for (int i = threadIdx.x; i < p.dim; i += kNormThreads) act_st(o + i, row_norm(x[i], st, p.gain, p.bias, i));
}

}  // namespace tb
