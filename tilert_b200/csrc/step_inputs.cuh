// What a pass of a model begins with: the tokens' embedding rows and the rotary rows of their positions, one launch.  Latency: a
// gather, a conversion of the position, an addition and a second gather took 8 us at one token (rows of 7168), with nothing of the
// first product under way; as one launch that lets its successor start, a step is 6 us shorter (420 -> 414 us with two layers).
#pragma once

#include "common.cuh"

namespace tb {

constexpr int kStepInputThreads = 512;

struct StepInputsParams {
  const long long* tokens;     // [n]; negative ones count from the end
  const __nv_bfloat16* table;  // [vocab, dim]
  int vocab, dim;
  const int* pos;              // position of token 0
  const float* freqs;          // [positions, freq_len]
  int positions, freq_len;
  __nv_bfloat16* x;            // [n, dim]
  float* fr;                   // [n, freq_len]
  int* status;
};

// grid = tokens.  A token or position outside of its table is refused: status 4, and rows that are no number, so that nothing computed
// from them passes for a result.
__global__ void __launch_bounds__(kStepInputThreads) step_inputs_kernel(const StepInputsParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, tid = threadIdx.x;
  long long tok = p.tokens[t];
  if (tok < 0) tok += p.vocab;
  const long long pos = static_cast<long long>(*p.pos) + t;
  __nv_bfloat16* dst = p.x + static_cast<long long>(t) * p.dim;
  if (tok < 0 || tok >= p.vocab || pos < 0 || pos >= p.positions) {  // uniform over the CTA
    if (tid == 0) set_status(p.status, ST_BAD_ARGUMENT);
    const float none = __int_as_float(0x7fc00000);
    for (int i = tid; i < p.freq_len; i += kStepInputThreads) p.fr[t * p.freq_len + i] = none;
    for (int i = tid; i < p.dim; i += kStepInputThreads) dst[i] = f2bf(none);
    return;
  }
  const __nv_bfloat16* src = p.table + tok * p.dim;
  for (int i = tid; i < p.freq_len; i += kStepInputThreads) p.fr[t * p.freq_len + i] = p.freqs[pos * p.freq_len + i];
  if (p.dim % 8 == 0 && ((reinterpret_cast<uintptr_t>(p.table) | reinterpret_cast<uintptr_t>(p.x)) & 15) == 0) {
#pragma unroll 2
    for (int i = tid; i < p.dim / 8; i += kStepInputThreads) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
  } else {
    for (int i = tid; i < p.dim; i += kStepInputThreads) dst[i] = src[i];
  }
}

}  // namespace tb
