// Token sampling from the vocabulary logits: temperature, top-k, top-p (nucleus), seeded; plus the
// top-256 log-probabilities a serving front end exports.  Eight CTAs per token.
//
//   config = (temperature, top_p, top_k, use_top_p) as four floats in device memory (the layout of
//   the reference's SAMPLING_CONFIG scratch tensor, modules/end2end.py:282-289).
//   temperature == 0: greedy (arg-max, ties to the lower token id).
//   Otherwise candidates are the 1024 largest logits (exact, ties to the lower id), sorted by value;
//   top_k in [1, 1024] keeps the first top_k of them (any other value keeps all 1024); with
//   use_top_p the shortest prefix whose probability mass (under the temperature-scaled softmax over
//   the WHOLE vocabulary) reaches top_p is kept; one uniform number picks a token from what is left,
//   in proportion to its probability.  Mass outside the 1024 candidates is never sampled.
//   Log-probabilities are those of the unscaled softmax over the whole vocabulary.
#pragma once

#include "cluster.cuh"
#include "common.cuh"
#include "topk_radix.cuh"

namespace tb {

constexpr int kSampleThreads = 1024;
constexpr int kSampleCandidates = kSampleThreads;  // one candidate per thread
constexpr int kSampleTopN = 256;
constexpr int kGreedyThreads = 512;
constexpr int kRowCtas = 8;       // on a row of logits: a portable cluster
constexpr int kDigitBins = 2048;  // eleven bits
constexpr int kHeldBytes = 128 * 1024;  // parts up to this size stay in shared memory

struct SampleParams {
  const float* logits;  // [tokens, stride]
  long long stride;
  int vocab;
  const float* config;  // (temperature, top_p, top_k, use_top_p)
  unsigned long long seed;
  unsigned long long* step;  // optional device state {step index, CTAs done}: the launch reads the step index
                             // and its last CTA increments it, so a replayed CUDA graph draws new numbers
  unsigned long long step_value;  // used when `step` is null
  bool held;            // the parts are kept in shared memory
  int* token;           // [tokens]
  float* token_logprob; // optional [tokens]
  float* topn_logprob;  // optional [tokens, 256]
  int* topn_index;      // optional [tokens, 256]
  long long* token_out; // optional [tokens]: the token once more
  int* pos;             // optional: advanced by `advance`
  int advance;
};

// uniform in [0, 1) from (seed, step, token): splitmix64 finaliser, top 24 bits
__host__ __device__ inline float sample_uniform(unsigned long long seed, unsigned long long step, unsigned long long tok) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (step + 1) + 0xD1B54A32D192ED03ull * (tok + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return static_cast<float>(z >> 40) * (1.0f / 16777216.0f);
}

// Sum of `v` over the CTA, in every thread (`red`: one float a warp).
__device__ __forceinline__ float block_reduce_sum(float v, float* red) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_sum(red[threadIdx.x & 31]);
}

// The place of this CTA's part of a row of `n` values: whole pieces of four, the last CTAs' parts may be short or empty.
struct RowPart {
  int lo, n;
};
__host__ __device__ inline int row_part_len(int n) { return (n + kRowCtas * 4 - 1) / (kRowCtas * 4) * 4; }
__device__ __forceinline__ RowPart row_part(int n, int rank) {
  const int per = row_part_len(n), lo = min(rank * per, n);
  return {lo, min(per, n - lo)};
}
// visit(i, value) of the part's elements, sixteen bytes a load where the address allows it
template <int THREADS, class Visit>
__device__ __forceinline__ void each_of_part(const float* part, int n, Visit visit) {
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(part) & 15) == 0) {
    const float4* p4 = reinterpret_cast<const float4*>(part);
    done = n / 4 * 4;
#pragma unroll 4
    for (int i = threadIdx.x; i < n / 4; i += THREADS) {
      const float4 v = __ldcg(p4 + i);
      visit(4 * i, v.x);
      visit(4 * i + 1, v.y);
      visit(4 * i + 2, v.z);
      visit(4 * i + 3, v.w);
    }
  }
  for (int i = done + threadIdx.x; i < n; i += THREADS) visit(i, __ldcg(part + i));
}

// (value, index) as one number: larger values first, equal ones by lower index; zero below all of them
__device__ __forceinline__ unsigned long long pair_of(uint32_t key, int index) {
  return static_cast<unsigned long long>(key) << 32 | static_cast<uint32_t>(~index);
}
__device__ __forceinline__ float value_of_key(uint32_t key) { return __uint_as_float((key & 0x80000000u) ? key ^ 0x80000000u : ~key); }

// ------------------------------------------------------------------ arg-max
struct GreedyParams {
  const float* logits;  // [tokens, stride]
  long long stride;
  int vocab;
  long long* token;  // [tokens]
  int* pos;          // optional: advanced by `advance`
  int advance;
};

// The index of a row's largest value, the lowest of equal ones; a value that is no number counts as the largest of all.
// Latency: two 16-byte loads a thread at 32768 values on eight SMs.  A reduction on one SM, a copy of its result and a kernel that
// advances the position took 11.6 us there and 29.3 at 129280 values, this launch 2.2 and 4.0.
__global__ void __cluster_dims__(kRowCtas, 1, 1) __launch_bounds__(kGreedyThreads) greedy_kernel(const GreedyParams p) {
  __shared__ unsigned long long s_warp[kGreedyThreads / 32], s_cta[kRowCtas];
  cluster_arrive();
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, rank = static_cast<int>(cluster_rank()), tok = blockIdx.x / kRowCtas;
  const RowPart part = row_part(p.vocab, rank);
  uint32_t key = 0;
  int index = 0x7fffffff;
  each_of_part<kGreedyThreads>(p.logits + tok * p.stride + part.lo, part.n, [&](int i, float v) {
    const uint32_t k = v == v ? f32_order_key(v) : 0xffffffffu;
    if (k > key) key = k, index = part.lo + i;  // (a thread's elements come in order)
  });
  const uint32_t best = __reduce_max_sync(0xffffffffu, key);
  const uint32_t first = __reduce_min_sync(0xffffffffu, key == best ? static_cast<uint32_t>(index) : 0x7fffffffu);
  if (lane == 0) s_warp[tid >> 5] = pair_of(best, static_cast<int>(first));
  __syncthreads();
  cluster_wait();  // the first CTA runs
  if (tid == 0) {
    unsigned long long top = s_warp[0];
    for (int w = 1; w < kGreedyThreads / 32; ++w) top = max(top, s_warp[w]);
    cluster_store(cluster_addr(&s_cta[rank], 0), top);
  }
  cluster_sync_all();
  if (rank == 0 && tid == 0) {
    unsigned long long top = s_cta[0];
    for (int c = 1; c < kRowCtas; ++c) top = max(top, s_cta[c]);
    p.token[tok] = static_cast<int>(~static_cast<uint32_t>(top));
    if (p.pos != nullptr && tok == 0) *p.pos += p.advance;
  }
}

// ------------------------------------------------------------------ sampling
// A row over a cluster of eight CTAs, its parts in shared memory (read again from L2 where they do not fit): the maximum, the
// two sums and the counts of each digit meet over distributed shared memory, and the first CTA finds the digits, sorts the
// candidates and picks.  The sums are those of the parts, added in the parts' order: log-probabilities and the ends of a nucleus have
// last bits of their own, the order of the candidates has none.  Eleven bits a digit: with eight, nearly all of a vocabulary's logits
// count into the same few words.
// Bound by the instructions of the passes, some ten cluster barriers and the sort: 15.8 us for 32768 values, 22.4 for 129280; the
// same steps on one CTA a token took 47.5 and 138.
__global__ void __cluster_dims__(kRowCtas, 1, 1) __launch_bounds__(kSampleThreads) sample_kernel(const SampleParams p) {
  extern __shared__ float s_part[];
  __shared__ __align__(16) int s_hist[kDigitBins], s_all[kDigitBins];  // this CTA's counts; in the first CTA everyone's
  __shared__ unsigned long long s_pick_pair[2][kSampleCandidates];     // candidates of this CTA; [0] of the first CTA: all of them
  __shared__ float red[32], s_max[kRowCtas], s_sum[2][kRowCtas];
  __shared__ int s_warp_tot_i[32], s_eq[kRowCtas];
  __shared__ uint32_t s_digit[4];  // prefix, values equal to it that are wanted, as many as there are, whether all values are wanted
  __shared__ int s_mine, s_total, s_base, s_pick, s_keep;
  __shared__ float s_warp_tot[32];
  cluster_arrive();
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = static_cast<int>(cluster_rank()), tok = blockIdx.x / kRowCtas;
  const RowPart part = row_part(p.vocab, rank);
  const float* row = p.logits + tok * p.stride + part.lo;
  const float temperature = p.config[0], top_p = p.config[1];
  const int top_k_cfg = static_cast<int>(p.config[2]);
  const bool use_top_p = p.config[3] != 0.f;
  const unsigned long long step =
      rank != 0 ? 0 : (p.step != nullptr ? *reinterpret_cast<volatile unsigned long long*>(p.step) : p.step_value);

  // ---- the part, its maximum, the row's ----
  float m = -INFINITY;
  each_of_part<kSampleThreads>(row, part.n, [&](int i, float v) {
    if (p.held) s_part[i] = v;
    m = fmaxf(m, v);
  });
  for (int i = tid; i < kDigitBins; i += kSampleThreads) s_hist[i] = s_all[i] = 0;
  if (tid == 0) s_mine = s_total = 0;
  m = warp_max(m);
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = warp_max(red[lane]);
  cluster_wait();  // all CTAs run
  if (tid < kRowCtas) cluster_store(cluster_addr(&s_max[rank], tid), __float_as_uint(m));
  cluster_sync_all();
  m = s_max[0];
#pragma unroll
  for (int c = 1; c < kRowCtas; ++c) m = fmaxf(m, s_max[c]);
  auto value = [&](int i) { return p.held ? s_part[i] : __ldcg(row + i); };

  // ---- softmax normalisers over the whole vocabulary, the counts of the first digit ----
  const float inv_t = temperature > 0.f ? 1.0f / temperature : 1.0f;
  float s1 = 0.f, st = 0.f;
  for (int i = tid; i < part.n; i += kSampleThreads) {
    const float v = value(i), d = v - m;
    s1 += __expf(d);
    st += __expf(d * inv_t);
    const uint32_t key = f32_order_key(v);
    if (key > kNegInfKey) atomicAdd(&s_hist[key >> 21], 1);
  }
  s1 = block_reduce_sum(s1, red);
  st = block_reduce_sum(st, red);
  if (tid < 2) cluster_store(cluster_addr(&s_sum[tid][rank], 0), __float_as_uint(tid == 0 ? s1 : st));

  // ---- the 1024th largest value, digit by digit ----
  uint32_t prefix = 0, mask = 0;
  int want = kSampleCandidates;  // of the values with the prefix
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int shift = d == 0 ? 21 : (d == 1 ? 10 : 0), bits = d == 2 ? 10 : 11, bins = 1 << bits;
    if (d > 0) {
      for (int i = tid; i < part.n; i += kSampleThreads) {
        const uint32_t key = f32_order_key(value(i));
        if (key > kNegInfKey && (key & mask) == prefix) atomicAdd(&s_hist[(key >> shift) & (bins - 1)], 1);
      }
      __syncthreads();
    }
    for (int i = tid; i < bins; i += kSampleThreads) {
      if (s_hist[i] != 0) cluster_add(cluster_addr(&s_all[i], 0), s_hist[i]);
      s_hist[i] = 0;
    }
    cluster_sync_all();
    if (rank == 0) {
      // counts of this thread's bins and above: within the warp, then of the warps above
      const int per = bins / kSampleThreads;  // 2 or 1
      const int hi = s_all[tid * per + per - 1], lo = per == 2 ? s_all[tid * per] : 0;
      int suf = hi + lo;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += v;
      }
      if (lane == 0) s_warp_tot_i[warp] = suf;
      __syncthreads();
      for (int w = warp + 1; w < kSampleThreads / 32; ++w) suf += s_warp_tot_i[w];
      const int above = suf - hi - lo;
      const bool few = tid == 0 && suf < want;  // (of the first digit only: fewer values than candidates)
      if ((suf >= want && above < want) || few) {
        const bool upper = !few && above + hi >= want;
        const uint32_t next = prefix | static_cast<uint32_t>(tid * per + (upper ? per - 1 : 0)) << shift;
        const uint32_t say[4] = {next, static_cast<uint32_t>(want - above - (upper ? 0 : per == 2 ? hi : 0)),
                                 static_cast<uint32_t>(upper || per == 1 ? hi : lo), few ? 1u : 0u};
        for (int c = 0; c < kRowCtas; ++c)
          for (int j = 0; j < 4; ++j) cluster_store(cluster_addr(&s_digit[j], c), say[j]);
      }
      __syncthreads();
      for (int i = tid; i < bins; i += kSampleThreads) s_all[i] = 0;
    }
    cluster_sync_all();
    prefix = s_digit[0];
    want = static_cast<int>(s_digit[1]);
    mask |= static_cast<uint32_t>(bins - 1) << shift;
    if (s_digit[3] != 0) break;
  }
  const bool all = s_digit[3] != 0, all_equal = !all && static_cast<uint32_t>(want) == s_digit[2];
  const uint32_t below = all ? kNegInfKey : (all_equal ? prefix - 1 : prefix);  // all values above it are candidates

  // ---- the candidates, in any order ----
  auto take = [&](uint32_t key, int i) { s_pick_pair[1][atomicAdd(&s_mine, 1)] = pair_of(key, part.lo + i); };
  int equal = 0;
  for (int i = tid; i < part.n; i += kSampleThreads) {
    const uint32_t key = f32_order_key(value(i));
    if (key > below) take(key, i);
    equal += key == prefix;
  }
  if (!all && !all_equal) {
    // of the values equal to the last one wanted, those with the lowest indices
    equal = __reduce_add_sync(0xffffffffu, equal);
    if (lane == 0) s_warp_tot_i[warp] = equal;
    __syncthreads();
    if (warp == 0) {
      const int n = __reduce_add_sync(0xffffffffu, s_warp_tot_i[lane]);
      if (lane < kRowCtas) cluster_store(cluster_addr(&s_eq[rank], lane), static_cast<uint32_t>(n));
    }
    cluster_sync_all();
    int left = want;
    for (int c = 0; c < rank; ++c) left -= s_eq[c];
    for (int base = 0; base < part.n && left > 0; base += kSampleThreads) {
      const int i = base + tid;
      const bool hit = i < part.n && f32_order_key(value(i)) == prefix;
      const uint32_t hits = __ballot_sync(0xffffffffu, hit);
      __syncthreads();
      if (lane == 0) s_warp_tot_i[warp] = __popc(hits);
      __syncthreads();
      int before = __popc(hits & ((1u << lane) - 1)), there = 0;
      for (int w = 0; w < kSampleThreads / 32; ++w) {
        if (w < warp) before += s_warp_tot_i[w];
        there += s_warp_tot_i[w];
      }
      if (hit && before < left) take(prefix, i);
      left -= there;
    }
  }
  __syncthreads();
  if (tid == 0 && s_mine > 0) s_base = cluster_add_get(cluster_addr(&s_total, 0), s_mine);
  __syncthreads();
  if (tid < s_mine) cluster_store(cluster_addr(&s_pick_pair[0][s_base + tid], 0), s_pick_pair[1][tid]);
  cluster_sync_all();
  if (rank != 0) return;

  // ---- sorted by (value descending, index ascending) ----
  unsigned long long mine = tid < s_total ? s_pick_pair[0][tid] : 0;
  int turn = 1;
  for (int size = 2; size <= kSampleCandidates; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      unsigned long long other;
      if (stride >= 32) {
        s_pick_pair[turn][tid] = mine;
        __syncthreads();
        other = s_pick_pair[turn][tid ^ stride];
        turn ^= 1;
      } else {
        other = __shfl_xor_sync(0xffffffffu, mine, stride);
      }
      const bool larger = ((tid & size) == 0) == ((tid & stride) == 0);  // this place keeps the larger one
      mine = larger == (mine > other) ? mine : other;
    }
  }
  __syncthreads();
  const float my_val = mine != 0 ? value_of_key(static_cast<uint32_t>(mine >> 32)) : -INFINITY;
  const int my_idx = mine != 0 ? static_cast<int>(~static_cast<uint32_t>(mine)) : 0x7fffffff;
  s1 = st = 0.f;
#pragma unroll
  for (int c = 0; c < kRowCtas; ++c) s1 += s_sum[0][c], st += s_sum[1][c];
  const float log_s1 = __logf(s1);

  // ---- exported log-probabilities ----
  if (p.topn_logprob != nullptr && tid < kSampleTopN) {
    p.topn_logprob[tok * kSampleTopN + tid] = mine != 0 ? my_val - m - log_s1 : -INFINITY;
    p.topn_index[tok * kSampleTopN + tid] = mine != 0 ? my_idx : -1;
  }

  float* s_cum = reinterpret_cast<float*>(s_hist);
  // ---- pick ----
  if (tid == 0) {
    s_pick = 0;
    s_keep = 0;
  }
  if (temperature > 0.f) {
    const int k_eff = (top_k_cfg >= 1 && top_k_cfg <= kSampleCandidates) ? top_k_cfg : kSampleCandidates;
    const float w = (tid < k_eff && mine != 0) ? __expf((my_val - m) * inv_t) : 0.f;
    // inclusive scan of w over the CTA
    float sc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float a = __shfl_up_sync(0xffffffffu, sc, o);
      if (lane >= o) sc += a;
    }
    if (lane == 31) s_warp_tot[warp] = sc;
    __syncthreads();
    float pre = 0.f;
    for (int w2 = 0; w2 < warp; ++w2) pre += s_warp_tot[w2];
    const float cum = pre + sc;
    s_cum[tid] = cum;
    __syncthreads();
    // nucleus: the shortest prefix whose mass reaches top_p of the whole distribution
    const float need = top_p * st;
    if (use_top_p) {
      const float before = tid > 0 ? s_cum[tid - 1] : 0.f;
      if (cum >= need && before < need) s_keep = tid + 1;
    }
    __syncthreads();
    int n_keep = (use_top_p && s_keep > 0) ? s_keep : k_eff;  // never reached: keep every candidate
    if (n_keep > k_eff) n_keep = k_eff;
    const float u = sample_uniform(p.seed, step, static_cast<unsigned long long>(tok));
    const float target = u * s_cum[n_keep - 1];
    {
      const float before = tid > 0 ? s_cum[tid - 1] : 0.f;
      if (tid < n_keep && cum > target && before <= target) s_pick = tid;
    }
    __syncthreads();
  }
  __syncthreads();
  if (tid == s_pick) {
    p.token[tok] = my_idx;
    if (p.token_logprob != nullptr) p.token_logprob[tok] = my_val - m - log_s1;
    if (p.token_out != nullptr) p.token_out[tok] = my_idx;
    if (p.pos != nullptr && tok == 0) *p.pos += p.advance;
  }
  if (p.step != nullptr && tid == 0) {
    // this CTA has read the step index (above, or it is greedy and does not care): count it done;
    // the last one advances the index for the next launch
    const unsigned long long prev = atomicAdd(p.step + 1, 1ull);
    if (prev == static_cast<unsigned long long>(gridDim.x / kRowCtas) - 1ull) {
      p.step[1] = 0ull;
      __threadfence();
      p.step[0] = p.step[0] + 1ull;
    }
  }
}

}  // namespace tb
