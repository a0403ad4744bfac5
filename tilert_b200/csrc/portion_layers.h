// A layer of a portion of tokens as one call: the operators of the C ABI in the layer's order, their sizes and strides worked out here.
// A short prompt was bound by the host: an operator called from Python took 11 us of it, called from here 3 us.  37 tokens behind
// 4000 cached positions through four layers of attention over a latent cache, 62 launches: 704 -> 539 us, of which the host
// has 340 now.
#pragma once

#include "../../include/tilert_gqa.h"
#include "host_util.h"

#define TB_STEP(call)               \
  do {                              \
    const int rc__ = (call);        \
    if (rc__ != TB_OK) return rc__; \
  } while (0)

extern "C" int tilert_gqa_routed_layer_op(TgContext* ctx, const TgRoutedLayer* layer, int rows, const int* pos, float* x, void* xh, void* stream) {
  TB_REQUIRE(ctx != nullptr && layer != nullptr && rows >= 1 && rows <= layer->portion && x != nullptr && xh != nullptr);
  const TgRoutedLayer& l = *layer;
  const int dimp = pad_to(l.dim, 8), n_qkv = (l.heads + l.kv_heads) * l.head_dim + l.kv_heads * l.vdim, n_att = l.heads * l.vdim;
  auto gemm = [&](const void* in, int k, const void* w, int n, const float* bias, void* out, bool out_f32) {
    return tilert_gqa_gemm_op(ctx, in, pad_to(k, 8), rows, w, pad_to(k, 8), n, k, 0, 0.f, 0.f, 0, nullptr, bias, out, pad_to(n, 8), out_f32 || l.f32, l.f32,
                              stream);
  };
  TB_STEP(gemm(xh, l.dim, l.w_qkv, n_qkv, nullptr, l.qkv, true));
  TB_STEP(tilert_gqa_qkv_rows_op(ctx, l.qkv, pad_to(n_qkv, 8), l.q_gain, l.k_gain, l.eps, l.v_mode, l.lambda, l.v_first, rows, l.heads, l.kv_heads,
                                 l.head_dim, l.vdim, pos, l.q, l.k_cache, l.v_cache, l.ring, l.f32, stream));
  TB_STEP(tilert_gqa_attn_rows_op(ctx, l.q, l.k_cache, l.v_cache, rows, l.heads, l.kv_heads, l.head_dim, l.vdim, pos, l.window, l.ring, l.scale, l.att,
                                  pad_to(n_att, 8), l.f32, stream));
  TB_STEP(gemm(l.att, n_att, l.w_o, l.dim, nullptr, l.y, true));
  TB_STEP(tilert_gqa_residual_norm_op(ctx, l.y, dimp, nullptr, 0, nullptr, nullptr, 0, nullptr, 0, l.norm1, nullptr, nullptr, nullptr, nullptr, 0, l.eps,
                                      rows, l.dim, x, dimp, xh, dimp, l.f32, stream));
  if (l.experts == 0) return TB_OK;
  TB_STEP(gemm(xh, l.dim, l.w_router, l.experts, l.router_bias, l.logits, true));
  TB_STEP(tilert_gqa_route_rows_op(ctx, l.logits, pad_to(l.experts, 8), rows, l.experts, l.top, l.ids, l.slot_w, l.rank, l.counts, stream));
  TB_STEP(tilert_gqa_gather_rows_op(ctx, xh, dimp, rows, l.dim, l.experts, l.top, l.ids, l.rank, l.counts, l.xs, l.slot_row, l.f32, stream));
  const int ffp = pad_to(l.ff, 8);
  TB_STEP(tilert_gqa_gemm_op(ctx, l.xs, dimp, rows * l.top, l.w_gate_up, dimp, l.ff, l.dim, 1, l.limit, l.alpha, l.experts, l.counts, nullptr, l.hid, ffp,
                             l.f32, l.f32, stream));
  TB_STEP(tilert_gqa_gemm_op(ctx, l.hid, ffp, rows * l.top, l.w_down, ffp, l.dim, l.ff, 0, 0.f, 0.f, l.experts, l.counts, nullptr, l.ye, dimp, l.f32,
                             l.f32, stream));
  if (l.shared_ff > 0) {
    TB_STEP(tilert_gqa_gemm_op(ctx, xh, dimp, rows, l.w_shared_gate_up, dimp, l.shared_ff, l.dim, 1, l.shared_limit, l.alpha, 0, nullptr, nullptr,
                               l.shared_hid, pad_to(l.shared_ff, 8), l.f32, l.f32, stream));
    TB_STEP(gemm(l.shared_hid, l.shared_ff, l.w_shared_down, l.dim, nullptr, l.shared_y, false));
  }
  return tilert_gqa_residual_norm_op(ctx, nullptr, 0, l.ye, dimp, l.slot_row, l.slot_w, l.top, l.shared_ff > 0 ? l.shared_y : nullptr,
                                     l.shared_ff > 0 ? dimp : 0, l.norm2, nullptr, nullptr, nullptr, nullptr, 0, l.eps, rows, l.dim, x, dimp, xh, dimp,
                                     l.f32, stream);
}

extern "C" int tilert_gqa_latent_layer_op(TgContext* ctx, const TgLatentLayer* layer, int rows, int cached, int n_splits, const int* pos, float* x,
                                          void* xh, const float* y, const float* y_gain, const float* y_bias, const float* add, void* stream) {
  TB_REQUIRE(ctx != nullptr && layer != nullptr && rows >= 1 && x != nullptr && xh != nullptr && cached >= 0);
  const TgLatentLayer& l = *layer;
  TB_REQUIRE(rows <= l.portion && rows <= l.work_rows && l.cache != nullptr && l.z != nullptr && l.cq != nullptr && l.q != nullptr && l.att != nullptr &&
             l.y != nullptr && (l.ff == 0 || l.hid != nullptr));
  if (cached > 0)
    TB_REQUIRE(!l.f32 && l.w_kv != nullptr && l.qe != nullptr && l.kv != nullptr && cached <= l.work_cached && cached <= l.ring);
  else
    TB_REQUIRE(l.qn != nullptr && l.lat != nullptr && l.part != nullptr && l.c != nullptr && l.o != nullptr && n_splits >= 1 && n_splits <= l.work_splits);
  const int dimp = pad_to(l.dim, 8), n_att = l.heads * l.vdim, rankp = pad_to(l.kv_rank, 8);
  const int off_c = pad_to(l.q_rank, 8), off_r = off_c + rankp, off_g = off_r + pad_to(l.rot, 8), z_len = off_g + l.gate_rows, ldz = pad_to(z_len, 8);
  const int ldh = pad_to(l.head_dim, 8) + pad_to(l.rot, 8), per_head = l.gate_rows == l.heads;
  const float* gate = l.z + off_g;
  // a product of `k` columns; heads > 0: one weight and `rows` rows a head
  auto gemm = [&](const void* in, int k, const void* w, int n, int heads, void* out, long long ldo, bool out_f32) {
    return tilert_gqa_gemm_op(ctx, in, pad_to(k, 8), rows, w, pad_to(k, 8), n, k, 0, 0.f, 0.f, heads, nullptr, nullptr, out, ldo, out_f32 || l.f32, l.f32,
                              stream);
  };
  auto settle = [&](const float* out, const float* gain, const float* bias, const float* added, const float* gain2, const float* bias2) {
    return tilert_gqa_residual_norm_op(ctx, gain != nullptr ? out : nullptr, gain != nullptr ? dimp : 0, nullptr, 0, nullptr, nullptr, 0, nullptr, 0, gain, bias,
                                       added, gain2, bias2, 1, l.eps, rows, l.dim, x, dimp, xh, dimp, l.f32, stream);
  };
  TB_STEP(settle(y, y_gain, y_bias, add, l.norm1_gain, l.norm1_bias));
  TB_STEP(gemm(xh, l.dim, l.w_z, z_len, 0, l.z, ldz, true));
  TB_STEP(tilert_gqa_latent_tokens_op(ctx, l.z, ldz, l.q_rank, off_c, off_r, l.q_gain, l.c_gain, l.eps, rows, l.kv_rank, l.rot, l.rope, l.positions,
                                      l.rope_dims, l.interleaved, pos, l.ring, l.cq, off_c, l.cache, l.f32, stream));
  TB_STEP(gemm(l.cq, l.q_rank, l.w_uq, l.heads * ldh, 0, l.q, l.heads * ldh, true));
  const int ldq = l.heads * ldh;
  if (cached > 0) {
    const int n_kv = l.heads * (pad_to(l.head_dim, 16) + pad_to(l.vdim, 16)), row = latent_row(l.kv_rank, l.rot).row;
    TB_STEP(tilert_gqa_latent_queries_op(ctx, l.q, ldq, rows, l.heads, l.head_dim, l.rot, l.rope, l.positions, l.rope_dims, l.interleaved, pos, l.qe, nullptr,
                                         l.kv_rank, l.f32, stream));
    TB_STEP(tilert_gqa_gemm_op(ctx, l.cache, row, cached, l.w_kv, rankp, n_kv, l.kv_rank, 0, 0.f, 0.f, 0, nullptr, nullptr, l.kv, n_kv, 0, 0, stream));
    TB_STEP(tilert_gqa_expanded_attn_op(ctx, l.qe, l.kv, l.cache, rows, l.heads, l.head_dim, l.rot, l.vdim, l.kv_rank, pos, l.window, l.ring, l.scale, l.sink,
                                        gate, ldz, per_head, l.att, pad_to(n_att, 8), stream));
  } else {
    const int row = latent_row(l.kv_rank, l.rot).row;
    TB_STEP(tilert_gqa_latent_queries_op(ctx, l.q, ldq, rows, l.heads, l.head_dim, l.rot, l.rope, l.positions, l.rope_dims, l.interleaved, pos, l.qn, l.lat,
                                         l.kv_rank, l.f32, stream));
    TB_STEP(gemm(l.qn, l.head_dim, l.w_uk_t, l.kv_rank, l.heads, l.lat, row, true));
    TB_STEP(tilert_gqa_latent_attn_op(ctx, l.lat, l.cache, rows, l.heads, l.kv_rank, l.rot, pos, l.window, l.ring, l.scale, n_splits, l.part, l.f32, stream));
    TB_STEP(tilert_gqa_latent_merge_op(ctx, l.part, rows, l.heads, n_splits, l.kv_rank, l.rot, l.sink, l.c, rankp, l.f32, stream));
    TB_STEP(gemm(l.c, l.kv_rank, l.w_uv, l.vdim, l.heads, l.o, pad_to(l.vdim, 8), true));
    TB_STEP(tilert_gqa_gate_heads_op(ctx, l.o, pad_to(l.vdim, 8), rows, l.heads, l.vdim, gate, ldz, per_head, l.att, pad_to(n_att, 8), l.f32, stream));
  }
  TB_STEP(gemm(l.att, n_att, l.w_o, l.dim, 0, l.y, dimp, true));
  if (l.ff == 0) return TB_OK;
  TB_STEP(settle(l.y, l.norm1b_gain, l.norm1b_bias, nullptr, l.norm2_gain, l.norm2_bias));
  TB_STEP(tilert_gqa_gemm_op(ctx, xh, dimp, rows, l.w_gate_up, dimp, l.ff, l.dim, 1, l.limit, l.alpha, 0, nullptr, nullptr, l.hid, pad_to(l.ff, 8), l.f32, l.f32,
                             stream));
  return gemm(l.hid, l.ff, l.w_down, l.dim, 0, l.y, dimp, true);
}
