// Whole forward passes: the launches of a network's kernels in order on one stream, issued from
// C++. A pass over a small tile is paced by the host - a block is seven kernels of 3-10 us each -
// so nothing but the launches is left between them: no Python call, allocation, weight cast or
// table per kernel. 32 x 32 pixels, two 128-wide blocks: 20 launches in 90 us; the same kernels with a
// Python call each, as for a model with hooks, take 260 us and more.
#pragma once
#include "../../include/strata_b200.h"

#include <algorithm>

namespace strata {

// Hands out 256-byte aligned pieces of the caller's workspace, or only counts them (base null).
struct ScratchPlan {
  uint8_t* base;
  int64_t used = 0;
  explicit ScratchPlan(void* b) : base(static_cast<uint8_t*>(b)) {}
  void* take(int64_t bytes) {
    void* p = base ? base + used : nullptr;
    used += (bytes + 255) / 256 * 256;
    return p;
  }
};

// Pixel rows whose conditioning matrix [rows, Cb] exists at a time: whole groups of `factor` image
// rows (no cell straddles two chunks), about 2^18 of them (0.5 GB at Cb = 1024).
inline int64_t cond_chunk_rows(int64_t pixels, int64_t width, int factor) {
  const int64_t band = width * factor;
  return std::min(pixels, std::max(band, (int64_t{1} << 18) / band * band));
}

struct NetworkPlan {
  // sizes
  int64_t M, Mp;              // backbone tokens, pixel tokens (0: single stage)
  int d, h, w;                // token grid
  // pieces
  float *lat0, *lon0;
  double* sums;
  float4 *px_fwd, *px_inv;
  float2* px_lat;
  void *rope, *rope_px;
  void *tokens, *patches, *block_ws;                   // backbone
  void *px, *px_patches, *mod, *cond, *xn, *qkv, *attn, *y, *hid;   // pixel stage
  void *head_n, *head_y;
  int64_t cond_rows;
  int64_t bytes;
};

inline bool network_plan(const strata_backbone_desc& b, const strata_pixel_desc* px, int B, int D,
                         int H, int W, void* ws, NetworkPlan& n) {
  n = NetworkPlan{};
  n.d = D / b.patch_v; n.h = H / b.patch_h; n.w = W / b.patch_w;
  n.M = static_cast<int64_t>(B) * n.d * n.h * n.w;
  n.Mp = px ? static_cast<int64_t>(B) * D * H * W : 0;
  if (n.M > 0x7fffffffLL || n.Mp > 0x7fffffffLL) return false;
  ScratchPlan s(ws);
  n.lat0 = static_cast<float*>(s.take(4LL * B));
  n.lon0 = static_cast<float*>(s.take(4LL * B));
  n.sums = static_cast<double*>(s.take(strata_tile_tables_workspace_bytes(B, H, W)));
  const int64_t columns = static_cast<int64_t>(B) * H * W;
  if (b.u_idx >= 0) {
    n.px_fwd = static_cast<float4*>(s.take(16 * columns));
    n.px_inv = static_cast<float4*>(s.take(16 * columns));
  }
  if (b.concat_lat) n.px_lat = static_cast<float2*>(s.take(8 * columns));
  if (b.rope_mode != STRATA_ROPE_NONE) n.rope = s.take(4LL * B * n.h * n.w * (b.dim / b.heads / 2));
  n.tokens = s.take(2 * n.M * b.dim);
  // what follows is shared by phases that do not overlap in time
  const int64_t mark = s.used;
  n.patches = s.take(2 * n.M * b.k_embed);
  int64_t most = s.used;
  s.used = mark;
  n.block_ws = s.take(strata_block_workspace_bytes(n.M, b.dim, b.hidden));
  most = std::max(most, s.used);
  s.used = mark;
  const int64_t rows = px ? n.Mp : n.M;
  if (px) {
    const int C = px->dim;
    n.px = s.take(2 * n.Mp * C);
    if (px->rope_mode != STRATA_ROPE_NONE) n.rope_px = s.take(4LL * B * H * W * (C / px->heads / 2));
    const int64_t pmark = s.used;
    n.px_patches = s.take(2 * n.Mp * px->k_embed);
    most = std::max(most, s.used);
    s.used = pmark;
    n.mod = s.take(2 * n.Mp * 6 * C);
    const int64_t bmark = s.used;
    n.cond_rows = cond_chunk_rows(n.Mp, W, b.patch_h);
    n.cond = s.take(2 * n.cond_rows * b.dim);
    most = std::max(most, s.used);
    s.used = bmark;
    n.xn = s.take(2 * n.Mp * C);
    n.qkv = s.take(2 * n.Mp * 3 * C);
    n.attn = s.take(2 * n.Mp * C);
    n.y = s.take(2 * n.Mp * C);
    n.hid = s.take(2 * n.Mp * px->hidden);
    most = std::max(most, s.used);
    s.used = pmark;
  }
  n.head_n = s.take(2 * rows * (px ? px->dim : b.dim));
  n.head_y = s.take(2 * rows * (px ? px->n_head : b.n_head));
  n.bytes = std::max(most, s.used);
  return true;
}

#define STRATA_TRY(call)            \
  do {                              \
    const int r_ = (call);          \
    if (r_ != 0) return r_;         \
  } while (0)

// x (bf16 rows [Mp, C]) through one AdaLN pixel block, in place; n.mod is overwritten.
inline int pixel_block(const strata_backbone_desc& b, const strata_pixel_desc& px, int i, int B,
                       int D, int H, int W, const NetworkPlan& n, void* stream) {
  const strata_pixel_block_weights& w = px.h_blocks[i];
  const int C = px.dim, M = static_cast<int>(n.Mp), hd = C / px.heads;
  const __nv_bfloat16* mod = nullptr;
  if (w.w_mod) {
    mod = static_cast<const __nv_bfloat16*>(n.mod);
    for (int64_t r0 = 0; r0 < n.Mp; r0 += n.cond_rows) {
      const int64_t rows = std::min(n.cond_rows, n.Mp - r0);
      STRATA_TRY(strata_adaln_cond_ready_bf16(n.tokens, B, n.d, n.h, n.w, b.dim, b.patch_h, w.w_dw,
                                              w.b_dw, px.cond_ks, r0, rows, n.cond, w.cond_table,
                                              stream));
      STRATA_TRY(strata_linear_bf16(n.cond, b.dim, w.w_mod, b.dim, w.b_mod,
                                    static_cast<__nv_bfloat16*>(n.mod) + r0 * 6 * C, 6 * C,
                                    static_cast<int>(rows), 6 * C, b.dim, STRATA_EPI_BIAS, nullptr,
                                    0, stream));
    }
  }
  auto part = [&](int k) { return mod ? mod + k * C : nullptr; };   // shift, scale, gate, shift, scale, gate
  const int ldm = 6 * C;
  void* x = n.px;
  const strata_block_weights& a = w.block;
  STRATA_TRY(strata_adaln_rows_bf16(x, C, nullptr, 0, nullptr, 0, nullptr, 0, part(0), part(1), ldm, n.xn,
                                    C, M, C, 1e-6f, stream));
  STRATA_TRY(strata_qkv_rope_bf16(n.xn, C, a.w_qkv, C, a.b_qkv, n.qkv, 3 * C, M, C, hd, n.rope_px,
                                  D * H * W, H * W, px.qk_norm, 1e-6f, stream));
  const auto* q = static_cast<const __nv_bfloat16*>(n.qkv);
  const int32_t* k3 = px.h_kernels + 3 * i;
  STRATA_TRY(strata_na3d_fwd_bf16(q, 3 * C, q + C, 3 * C, q + 2 * C, 3 * C, n.attn, C, B, D, H, W,
                                  px.heads, hd, k3[0], k3[1], k3[2], 0.f, stream));
  if (a.w_gate)
    STRATA_TRY(strata_linear_bf16(n.xn, C, a.w_gate, C, a.b_gate, n.attn, C, M, C, C, STRATA_EPI_GATE,
                                  n.attn, C, stream));
  STRATA_TRY(strata_linear_bf16(n.attn, C, a.w_proj, C, a.b_proj, n.y, C, M, C, C, STRATA_EPI_BIAS,
                                nullptr, 0, stream));
  STRATA_TRY(strata_adaln_rows_bf16(x, C, n.y, C, part(2), ldm, x, C, part(3), part(4), ldm, n.xn, C, M, C,
                                    1e-6f, stream));
  if (mod && mlp_fused_pays(M, C, px.hidden, current_sm_count()))
    return strata_mlp_bf16(n.xn, C, a.w_fc1, a.b_fc1, a.w_fc2, a.b_fc2, x, C, part(5), ldm, x, C, M, C, px.hidden,
                           stream);
  STRATA_TRY(strata_linear_bf16(n.xn, C, a.w_fc1, C, a.b_fc1, n.hid, px.hidden, M, px.hidden, C,
                                STRATA_EPI_GELU, nullptr, 0, stream));
  STRATA_TRY(strata_linear_bf16(n.hid, px.hidden, a.w_fc2, px.hidden, a.b_fc2, n.y, C, M, C, px.hidden,
                                STRATA_EPI_BIAS, nullptr, 0, stream));
  return strata_adaln_rows_bf16(x, C, n.y, C, part(5), ldm, x, C, nullptr, nullptr, 0, nullptr, 0, M, C,
                                1e-6f, stream);
}

inline int network_forward(const strata_backbone_desc& b, const strata_pixel_desc* px, const float* x,
                           const float* lat, const float* lon, int B, int D, int H, int W, float* out,
                           const NetworkPlan& n, void* stream) {
  const bool wind = b.u_idx >= 0;
  const int hd = b.dim / b.heads, M = static_cast<int>(n.M);
  float* lat0 = wind ? n.lat0 : nullptr;
  float* lon0 = wind ? n.lon0 : nullptr;
  STRATA_TRY(tile_tables_impl(lat, lon, B, H, W, lat0, lon0, b.rope_mode, b.patch_h, b.patch_w,
                              b.rope_length_scale, b.rope_base, hd, n.rope, n.sums, n.bytes, n.px_fwd, n.px_inv, n.px_lat,
                              stream));
  STRATA_TRY(preprocess_impl(x, B, b.in_channels, D, H, W, lat, lon, lat0, lon0, b.u_idx, b.v_idx,
                             b.concat_lat, b.patch_v, b.patch_h, b.patch_w, n.patches, b.k_embed, n.px_fwd,
                             n.px_lat, stream));
  STRATA_TRY(strata_linear_bf16(n.patches, b.k_embed, b.w_embed, b.k_embed, b.b_embed, n.tokens, b.dim, M,
                                b.dim, static_cast<int>(b.k_embed), STRATA_EPI_BIAS, nullptr, 0, stream));
  const int64_t ws_bytes = strata_block_workspace_bytes(n.M, b.dim, b.hidden);
  // a narrow block writes the norm that the next one, or the head, begins with
  bool normed = false;
  for (int i = 0; i < b.n_blocks; ++i) {
    const int32_t* k3 = b.h_kernels + 3 * i;
    void* next = i + 1 < b.n_blocks ? n.block_ws : (px ? nullptr : n.head_n);
    bool done = false;
    STRATA_TRY(block_impl(n.tokens, n.tokens, B, n.d, n.h, n.w, b.dim, b.heads, b.hidden, k3[0], k3[1], k3[2],
                          b.h_blocks + i, n.rope, b.qk_norm, 1e-6f, 1e-6f, n.block_ws, ws_bytes, normed, next, &done,
                          stream));
    normed = done;
  }
  const void *rows = n.tokens, *w_head = b.w_head;
  const float* b_head = b.b_head;
  int C = b.dim, n_head = b.n_head, R = M, pv = b.patch_v, ph = b.patch_h, pw = b.patch_w;
  if (px) {
    if (px->rope_mode != STRATA_ROPE_NONE)
      STRATA_TRY(strata_tile_tables(lat, lon, B, H, W, nullptr, nullptr, px->rope_mode, 1,
                                    px->rope_length_scale, px->rope_base, px->dim / px->heads, n.rope_px,
                                    n.sums, n.bytes, stream));
    STRATA_TRY(preprocess_impl(x, B, b.in_channels, D, H, W, lat, lon, lat0, lon0, b.u_idx, b.v_idx,
                               b.concat_lat, 1, 1, 1, n.px_patches, px->k_embed, n.px_fwd, n.px_lat, stream));
    STRATA_TRY(strata_linear_bf16(n.px_patches, px->k_embed, px->w_embed, px->k_embed, px->b_embed, n.px,
                                  px->dim, static_cast<int>(n.Mp), px->dim, static_cast<int>(px->k_embed),
                                  STRATA_EPI_BIAS, nullptr, 0, stream));
    for (int i = 0; i < px->n_blocks; ++i) STRATA_TRY(pixel_block(b, *px, i, B, D, H, W, n, stream));
    normed = false;
    rows = n.px; w_head = px->w_head; b_head = px->b_head;
    C = px->dim; n_head = px->n_head; R = static_cast<int>(n.Mp); pv = ph = pw = 1;
  }
  if (!normed) STRATA_TRY(strata_layernorm_bf16(rows, C, n.head_n, C, R, C, 1e-6f, stream));
  STRATA_TRY(strata_linear_bf16(n.head_n, C, w_head, C, b_head, n.head_y, n_head, R, n_head, C,
                                STRATA_EPI_BIAS, nullptr, 0, stream));
  return postprocess_impl(n.head_y, n_head, B, b.out_channels, D, H, W, lat, lon, lat0, lon0, b.u_idx,
                          b.v_idx, pv, ph, pw, out, n.px_inv, stream);
}

#undef STRATA_TRY

}  // namespace strata
