// Kernels of the AdaLN-conditioned pixel blocks (stage 2 of the two-stage model: 128-channel
// tokens at full pixel resolution, modulated per pixel by the backbone's tokens).
//
//   adaln_rows_kernel     x' = x + gate * y ;  out = LN(x') * (1 + scale) + shift
//                         (either half optional) - one pass over the token rows, HBM-bound:
//                         up to 5 row reads + 2 row writes of 2*C bytes per token
//   qk_norm_rows_kernel   RMS norm of every 64-channel q and k head of a packed qkv row, in place
//   adaln_cond_kernel     GELU(depthwise KSxKS conv(bilinear upsample(backbone tokens)) + b)
//                         as bf16 rows [pixels, Cb] - the A operand of the modulation projection
#pragma once
#include "common.cuh"

namespace strata {

struct AdalnRowsParams {
  const __nv_bfloat16* x;      long long ldx;
  const __nv_bfloat16* y;      long long ldy;     // nullable: no residual update
  const __nv_bfloat16* gate;   long long ldg;     // nullable with y: x' = x + y
  __nv_bfloat16* xo;           long long ldxo;    // x' (may alias x); required when y != null
  const __nv_bfloat16* shift;  const __nv_bfloat16* scale;  long long ldm;  // nullable: plain LN
  __nv_bfloat16* out;          long long ldo;     // nullable: residual update only
  int M, C;
  float eps;
};

__device__ __forceinline__ void unpack8(const uint4& r, float (&v)[8]) {
  v[0] = bf16_lo(r.x); v[1] = bf16_hi(r.x); v[2] = bf16_lo(r.y); v[3] = bf16_hi(r.y);
  v[4] = bf16_lo(r.z); v[5] = bf16_hi(r.z); v[6] = bf16_lo(r.w); v[7] = bf16_hi(r.w);
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint4 o;
  o.x = pack_bf16(v[0], v[1]); o.y = pack_bf16(v[2], v[3]);
  o.z = pack_bf16(v[4], v[5]); o.w = pack_bf16(v[6], v[7]);
  return o;
}

// LPR lanes (16 or 32) share one row; each holds VPL 16-byte vectors of it.
template <int LPR, int VPL>
__global__ void __launch_bounds__(256) adaln_rows_kernel(const AdalnRowsParams p) {
  chain_begin();
  constexpr int ROWS_PER_WARP = 32 / LPR;
  const int lane = threadIdx.x & 31;
  const int sub = lane % LPR;
  const int nvec = p.C >> 3;
  const long long rows_per_block = static_cast<long long>(blockDim.x >> 5) * ROWS_PER_WARP;
  const long long first = static_cast<long long>(blockIdx.x) * rows_per_block +
                          (threadIdx.x >> 5) * ROWS_PER_WARP + lane / LPR;
  // every lane of a warp runs the same number of iterations (the shuffles below need the
  // whole warp): rows past M are computed on row M-1 and not stored
  const long long row_iters =
      (p.M + rows_per_block * gridDim.x - 1) / (rows_per_block * gridDim.x);
  for (long long it = 0; it < row_iters; ++it) {
    const long long row_raw = first + it * rows_per_block * gridDim.x;
    const bool live = row_raw < p.M;
    const long long row = live ? row_raw : p.M - 1;
    float v[VPL][8];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int vi = sub + LPR * i;
      if (vi < nvec) {
        unpack8(__ldg(reinterpret_cast<const uint4*>(p.x + row * p.ldx) + vi), v[i]);
        if (p.y != nullptr) {
          float yv[8];
          unpack8(__ldg(reinterpret_cast<const uint4*>(p.y + row * p.ldy) + vi), yv);
          if (p.gate != nullptr) {
            float g[8];
            unpack8(__ldg(reinterpret_cast<const uint4*>(p.gate + row * p.ldg) + vi), g);
#pragma unroll
            for (int t = 0; t < 8; ++t) v[i][t] = fmaf(g[t], yv[t], v[i][t]);
          } else {
#pragma unroll
            for (int t = 0; t < 8; ++t) v[i][t] += yv[t];
          }
          const uint4 o = pack8(v[i]);
          if (live) reinterpret_cast<uint4*>(p.xo + row * p.ldxo)[vi] = o;
          unpack8(o, v[i]);   // the norm sees the stored (bf16) residual stream
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) sum += v[i][t];
      } else {
#pragma unroll
        for (int t = 0; t < 8; ++t) v[i][t] = 0.f;
      }
    }
    if (p.out == nullptr) continue;
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum / static_cast<float>(p.C);
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (sub + LPR * i < nvec) {
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const float d = v[i][t] - mean;
          sq += d * d;
        }
      }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rstd = rsqrtf(sq / static_cast<float>(p.C) + p.eps);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int vi = sub + LPR * i;
      if (vi < nvec) {
        float o[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) o[t] = (v[i][t] - mean) * rstd;
        if (p.scale != nullptr) {
          float sc[8], sh[8];
          unpack8(__ldg(reinterpret_cast<const uint4*>(p.scale + row * p.ldm) + vi), sc);
          unpack8(__ldg(reinterpret_cast<const uint4*>(p.shift + row * p.ldm) + vi), sh);
#pragma unroll
          for (int t = 0; t < 8; ++t) o[t] = fmaf(o[t], 1.0f + sc[t], sh[t]);
        }
        if (live) reinterpret_cast<uint4*>(p.out + row * p.ldo)[vi] = pack8(o);
      }
    }
  }
}

inline int launch_adaln_rows(const AdalnRowsParams& p, int sm_count, cudaStream_t stream) {
  if (p.C % 8 != 0 || p.C <= 0 || p.C > 2048) return -2;
  if (p.M <= 0) return 0;
  const int nvec = p.C / 8;
  const int lpr = nvec <= 16 ? 16 : 32;
  const int threads = 256;
  const long long rows_per_block = (threads / 32) * (32 / lpr);
  long long blocks = (p.M + rows_per_block - 1) / rows_per_block;
  const long long cap = static_cast<long long>(sm_count) * 16;
  if (blocks > cap) blocks = cap;
  const int g = static_cast<int>(blocks);
  const int vpl = (nvec + lpr - 1) / lpr;
  auto kern = lpr == 16 ? adaln_rows_kernel<16, 1>
              : vpl <= 1 ? adaln_rows_kernel<32, 1>
              : vpl <= 2 ? adaln_rows_kernel<32, 2>
              : vpl <= 4 ? adaln_rows_kernel<32, 4> : adaln_rows_kernel<32, 8>;
  return launch_chained(kern, dim3(g), threads, 0, stream, 1, p);
}

// RMS norm of the q and k heads (64 channels each) of packed qkv rows [M, 3C], in place:
// t <- t * rsqrt(mean(t^2) + eps). Eight lanes share a head (one 16-byte vector each).
__global__ void __launch_bounds__(256)
qk_norm_rows_kernel(__nv_bfloat16* __restrict__ qkv, long long ld, long long M, int C, float eps) {
  chain_begin();
  const int heads2 = 2 * (C >> 6);                      // q heads then k heads: columns [0, 2C)
  const long long groups = M * heads2;                  // one 8-lane group per (row, head)
  const long long n_thr = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long iters = (groups * 8 + n_thr - 1) / n_thr;
  long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (long long it = 0; it < iters; ++it, t += n_thr) {
    const long long g_raw = t >> 3;
    const bool live = g_raw < groups;
    const long long g = live ? g_raw : groups - 1;
    const long long row = g / heads2;
    const int head = static_cast<int>(g - row * heads2);
    uint4* ptr = reinterpret_cast<uint4*>(qkv + row * ld + head * 64) + (t & 7);
    float v[8];
    unpack8(*ptr, v);
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) sq = fmaf(v[i], v[i], sq);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float r = rsqrtf(sq * (1.0f / 64.0f) + eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= r;
    if (live) *ptr = pack8(v);
  }
}

inline int launch_qk_norm_rows(__nv_bfloat16* qkv, long long ld, long long M, int C, float eps,
                               int sm_count, cudaStream_t stream) {
  if (C % 64 != 0 || C <= 0 || ld % 8 != 0 || ld < 3LL * C) return -2;
  if (M <= 0) return 0;
  const long long thr = M * 2 * (C / 64) * 8;
  long long blocks = (thr + 255) / 256;
  const long long cap = static_cast<long long>(sm_count) * 16;
  if (blocks > cap) blocks = cap;
  return launch_chained(qk_norm_rows_kernel, dim3(static_cast<unsigned>(blocks)), 256, 0, stream, 1, qkv, ld, M, C, eps);
}

// Source index and weights of a 1-D bilinear upsample by an integer factor (half-pixel
// centres, negative source coordinates clamped to 0, upper neighbour clamped to n-1).
__device__ __forceinline__ void bilinear_tap(int p, int factor, int n, int& i0, int& i1, float& l0,
                                             float& l1) {
  float s = (static_cast<float>(p) + 0.5f) / static_cast<float>(factor) - 0.5f;
  s = s < 0.f ? 0.f : s;
  i0 = static_cast<int>(s);
  if (i0 > n - 1) i0 = n - 1;
  i1 = i0 + 1 < n ? i0 + 1 : n - 1;
  l1 = s - static_cast<float>(i0);
  l0 = 1.0f - l1;
}

struct AdalnCondParams {
  const __nv_bfloat16* tok;   // backbone tokens [B, D, h, w, Cb], token-major
  const float* wdw;           // depthwise weights [Cb, KS*KS]
  const float* bdw;           // [Cb] or null
  __nv_bfloat16* out;         // rows [n_rows, Cb] for pixels row0 .. row0+n_rows of (b, d, y, x)
  long long row0, n_rows;
  int D, h, w, Cb, factor, ks;
};

// Direct evaluation of one pixel x 8 channels: every conv tap is an upsampled value, i.e. four
// token reads; taps outside the H x W image are the convolution's zero padding.
__device__ __forceinline__ void cond_direct_pixel(const AdalnCondParams& p, const uint4* base,
                                                  int nvec, int H, int W, int y, int x, int cv,
                                                  float (&acc)[8]) {
  const int r = p.ks >> 1;
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = p.bdw ? __ldg(p.bdw + cv * 8 + c) : 0.f;
  for (int dy = -r; dy <= r; ++dy) {
    const int py = y + dy;
    if (py < 0 || py >= H) continue;
    int r0, r1;
    float ly0, ly1;
    bilinear_tap(py, p.factor, p.h, r0, r1, ly0, ly1);
    for (int dx = -r; dx <= r; ++dx) {
      const int px = x + dx;
      if (px < 0 || px >= W) continue;
      int c0, c1;
      float lx0, lx1;
      bilinear_tap(px, p.factor, p.w, c0, c1, lx0, lx1);
      float a[8], b[8], c[8], d[8];
      unpack8(__ldg(base + (static_cast<long long>(r0) * p.w + c0) * nvec), a);
      unpack8(__ldg(base + (static_cast<long long>(r0) * p.w + c1) * nvec), b);
      unpack8(__ldg(base + (static_cast<long long>(r1) * p.w + c0) * nvec), c);
      unpack8(__ldg(base + (static_cast<long long>(r1) * p.w + c1) * nvec), d);
      const int tap = (dy + r) * p.ks + (dx + r);
#pragma unroll
      for (int ch = 0; ch < 8; ++ch) {
        const float u = ly0 * (lx0 * a[ch] + lx1 * b[ch]) + ly1 * (lx0 * c[ch] + lx1 * d[ch]);
        acc[ch] = fmaf(__ldg(p.wdw + (cv * 8 + ch) * p.ks * p.ks + tap), u, acc[ch]);
      }
    }
  }
}

__device__ __forceinline__ void gelu8(float (&acc)[8]) {
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) {
    const float v = acc[ch];
    const float u = 0.7978845608028654f * (v + 0.044715f * v * v * v);
    acc[ch] = 0.5f * v * (1.0f + fast_tanh(u));
  }
}

// One thread: one pixel x 8 channels, direct evaluation (any factor and kernel size).
__global__ void __launch_bounds__(256) adaln_cond_kernel(const AdalnCondParams p) {
  chain_begin();
  const int nvec = p.Cb >> 3;
  const int H = p.h * p.factor, W = p.w * p.factor;
  const long long total = p.n_rows * nvec;
  for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long pix = p.row0 + t / nvec;
    const int cv = static_cast<int>(t % nvec);
    const int x = static_cast<int>(pix % W);
    const int y = static_cast<int>((pix / W) % H);
    const long long plane = pix / (static_cast<long long>(W) * H);   // b * D + d
    const uint4* base = reinterpret_cast<const uint4*>(p.tok + plane * p.h * p.w * p.Cb) + cv;
    float acc[8];
    cond_direct_pixel(p, base, nvec, H, W, y, x, cv, acc);
    gelu8(acc);
    reinterpret_cast<uint4*>(p.out + (pix - p.row0) * p.Cb)[cv] = pack8(acc);
  }
}

// Upsample followed by the depthwise conv is linear in the tokens: a pixel of the
// factor x factor cell of token (R, Cc) reads a 3 x 3 block of tokens with weights that depend
// only on the channel and on the pixel's position class along each axis - 3 * factor classes:
// the `factor` pixels of the first cell (clamped upsample source, conv taps cut by the zero
// padding), the `factor` phases of an interior cell, the `factor` pixels of the last cell.
// The token block starts at row R-1 (0 for the first cell, h-3 for the last), same for columns.
// This kernel folds the ks x ks taps into that table, [3f][3f][9][Cb] fp32. Valid for
// factor >= 4, ks <= 5 and at least 3 cells per axis (then every tap falls inside the block).
__device__ __forceinline__ void cond_class_ref(int cls, int f, int& pos, int& base) {
  // representative pixel position and token-block base on a reference axis of 4 cells
  if (cls < f) { pos = cls; base = 0; }
  else if (cls < 2 * f) { pos = cls; base = 0; }             // cell 1, phase cls - f
  else { pos = 3 * f + (cls - 2 * f); base = 1; }            // cell 3 (last)
}

__global__ void adaln_cond_table_kernel(const float* __restrict__ wdw, int Cb, int factor, int ks,
                                        float* __restrict__ table) {
  chain_begin();
  const int ncls = 3 * factor;
  const int n = ncls * ncls * Cb;
  const int r = ks >> 1;
  const int n_ref = 4 * factor;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int ch = t % Cb;
    const int cls = t / Cb;
    int y, rb, x, cb;
    cond_class_ref(cls / ncls, factor, y, rb);
    cond_class_ref(cls % ncls, factor, x, cb);
    float acc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k] = 0.f;
    for (int dy = -r; dy <= r; ++dy) {
      if (y + dy < 0 || y + dy >= n_ref) continue;
      int r0, r1;
      float ly0, ly1;
      bilinear_tap(y + dy, factor, 4, r0, r1, ly0, ly1);
      r0 -= rb; r1 -= rb;
      for (int dx = -r; dx <= r; ++dx) {
        if (x + dx < 0 || x + dx >= n_ref) continue;
        int c0, c1;
        float lx0, lx1;
        bilinear_tap(x + dx, factor, 4, c0, c1, lx0, lx1);
        c0 -= cb; c1 -= cb;
        const float wt = wdw[ch * ks * ks + (dy + r) * ks + (dx + r)];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const int j = k / 3, i = k % 3;
          const float wy = (j == r0 ? ly0 : 0.f) + (j == r1 ? ly1 : 0.f);
          const float wx = (i == c0 ? lx0 : 0.f) + (i == c1 ? lx1 : 0.f);
          acc[k] = fmaf(wt, wy * wx, acc[k]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) table[(static_cast<long long>(cls) * 9 + k) * Cb + ch] = acc[k];
  }
}

// GELU(stencil) of the cells of a row, through the table. One warp = a run of up to COND_RUN
// neighbouring cells of one cell row x 64 channels: lane l owns channels 2l, 2l+1 of the group, so
// a token read and a pixel write are 128 contiguous bytes per warp. The first and the last cell
// of a row are runs of their own (their table classes differ), the cells between share one block
// of classes; the row's own class follows from R. A lane keeps the 3 x (COND_RUN + 2) tokens its
// cells touch as fp32 pairs in registers and reads the 9 table entries of a phase once for all
// its cells (L1: a group's classes are 37 KB at factor 4).
//
// Bound: instruction issue and the FMA pipe - 9 packed multiply-adds for the stencil and 5 for
// the GELU per pixel and channel pair. With 2 cells x 4 channels a lane the entries came from a
// shared-memory slab, nine 16-byte reads per 36 multiply-adds, and those reads set the pace; a run
// of 6 cells x 2 channels needs nine 8-byte reads per 54 with fewer token registers, because
// neighbouring cells share six of their nine tokens (runs of 7 and 8 spill and are no faster).
// No slab, so no block-wide item either: small images spread over the chip, and where the runs
// alone are too few for it (psplit) the f phase rows of a run are separate warps. 2^18 pixels x 1024
// channels: 0.40 -> 0.29 ms; 4 x 64 x 64 pixels x 128 channels: 88 -> 12 us (edges included).
constexpr int COND_RUN = 6;

__global__ void __launch_bounds__(256, 2)
adaln_cond_runs_kernel(const AdalnCondParams p, const float* __restrict__ table, int psplit) {
  chain_begin();
  const int f = p.factor;
  const int ncls = 3 * f;
  const int H = p.h * f, W = p.w * f;
  const int groups = (p.Cb + 63) >> 6;
  const int runs = 2 + (p.w - 2 + COND_RUN - 1) / COND_RUN;     // first cell, last cell, the rest
  const long long gR0 = p.row0 / W / f;
  const long long gR1 = (p.row0 + p.n_rows - 1) / W / f;
  const long long n_items = (gR1 - gR0 + 1) * runs * psplit;
  const int lane = threadIdx.x & 31;
  const int phys = psplit > 1 ? 1 : f;                          // phase rows of an item
  // a block stays with one channel group, whose table entries then fit its L1; neighbouring blocks
  // take the other groups of the same pixels, so that whole output rows are written at about one time
  const int grp = static_cast<int>(blockIdx.x) % groups;
  const int ch = grp * 64 + 2 * lane;
  if (ch >= p.Cb) return;
  const long long stride = static_cast<long long>(gridDim.x / groups) * 8;
  for (long long item = static_cast<long long>(blockIdx.x / groups) * 8 + (threadIdx.x >> 5);
       item < n_items; item += stride) {
    long long t = item;
    const int run = static_cast<int>(t % runs); t /= runs;
    const int phy0 = psplit > 1 ? static_cast<int>(t % psplit) : 0;
    if (psplit > 1) t /= psplit;
    const long long gR = gR0 + t;
    const long long plane = gR / p.h;
    const int R = static_cast<int>(gR - plane * p.h);
    // (the last full run ends at the last inner cell: it repeats some cells of the one before it
    // rather than being a short run)
    const int inner = p.w - 2;
    const int c0 = run == 0 ? 0 : (run == 1 ? p.w - 1
                                            : 1 + max(0, min((run - 2) * COND_RUN, inner - COND_RUN)));
    const int n = run < 2 ? 1 : min(COND_RUN, inner);
    const int rb = R == 0 ? 0 : (R == p.h - 1 ? p.h - 3 : R - 1);
    const int cb = run == 0 ? 0 : (run == 1 ? p.w - 3 : c0 - 1);
    const int ycls0 = R == 0 ? 0 : (R == p.h - 1 ? 2 * f : f);
    const int xcls0 = run == 0 ? 0 : (run == 1 ? 2 * f : f);
    uint64_t tk[3][COND_RUN + 2];
    const __nv_bfloat16* base = p.tok + ((plane * p.h + rb) * p.w + cb) * static_cast<long long>(p.Cb) + ch;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < COND_RUN + 2; ++i) {
        const uint32_t v = i < n + 2 ? __ldg(reinterpret_cast<const uint32_t*>(
                                           base + (static_cast<long long>(j) * p.w + i) * p.Cb)) : 0u;
        tk[j][i] = pack2(bf16_lo(v), bf16_hi(v));
        // keep the pair: the compiler would hold the bf16 word and convert it again at every use
        asm volatile("" : "+l"(tk[j][i]));
      }
    uint64_t bias = 0ull;
    if (p.bdw != nullptr) {
      const float2 b2 = __ldg(reinterpret_cast<const float2*>(p.bdw + ch));
      bias = pack2(b2.x, b2.y);
    }
    const float k0 = 0.7978845608028654f, k01 = 0.7978845608028654f * 0.044715f;
    const uint64_t K0 = pack2(k0, k0), K01 = pack2(k01, k01), HALF = pack2(0.5f, 0.5f);
    const int step = f * p.Cb;                                  // one cell to the right
    for (int phy = phy0; phy < phy0 + phys; ++phy) {
      // first pixel of the run in this image row, and the part of the run the call asks for
      const long long pix0 = (plane * H + static_cast<long long>(R) * f + phy) * W +
                             static_cast<long long>(c0) * f - p.row0;
      if (pix0 >= p.n_rows || pix0 + static_cast<long long>(n) * f <= 0) continue;
      const bool whole = pix0 >= 0 && pix0 + static_cast<long long>(n) * f <= p.n_rows;
      const float* tb = table + (static_cast<long long>(ycls0 + phy) * ncls + xcls0) * 9 * p.Cb + ch;
      __nv_bfloat16* op = p.out + pix0 * p.Cb + ch;
      for (int phx = 0; phx < f; ++phx) {
        uint64_t wt[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const float2 w2 = __ldg(reinterpret_cast<const float2*>(tb));
          wt[k] = pack2(w2.x, w2.y);
          tb += p.Cb;
        }
        auto pixel = [&](int i) -> uint32_t {
          uint64_t x = bias;
#pragma unroll
          for (int k = 0; k < 9; ++k) x = ffma2(wt[k], tk[k / 3][i + k % 3], x);
          // tanh GELU, the polynomial part on packed fp32x2
          const uint64_t u = fmul2(x, ffma2(fmul2(x, x), K01, K0));
          float u0, u1, v0, v1;
          unpack2(u, u0, u1);
          const uint64_t hx = fmul2(x, HALF);
          unpack2(ffma2(hx, pack2(fast_tanh(u0), fast_tanh(u1)), hx), v0, v1);
          return pack_bf16(v0, v1);
        };
        __nv_bfloat16* q = op;
        if (whole && n == COND_RUN) {          // straight-line: the cells' chains overlap
#pragma unroll
          for (int i = 0; i < COND_RUN; ++i) {
            *reinterpret_cast<uint32_t*>(q) = pixel(i);
            q += step;
          }
        } else {
#pragma unroll
          for (int i = 0; i < COND_RUN; ++i) {
            const long long pix = pix0 + i * f + phx;
            if (i < n && pix >= 0 && pix < p.n_rows) *reinterpret_cast<uint32_t*>(q) = pixel(i);
            q += step;
          }
        }
        op += p.Cb;
      }
    }
  }
}

// Number of floats of the table the cell kernel needs, or 0 when the geometry takes the
// direct kernel (small factor, wide conv kernel, channel count not a multiple of 32).
inline long long adaln_cond_table_floats(int Cb, int factor, int ks) {
  if (factor < 4 || factor > 8 || ks > 5 || Cb % 32 != 0) return 0;
  return 9LL * factor * factor * 9 * Cb;
}

inline int launch_adaln_cond_table(const float* wdw, int Cb, int factor, int ks, float* table,
                                   cudaStream_t stream) {
  const int n = 9 * factor * factor * Cb;
  return launch_chained(adaln_cond_table_kernel, dim3((n + 255) / 256), 256, 0, stream, 1, wdw, Cb, factor, ks, table);
}

// table: what launch_adaln_cond_table wrote for these weights (adaln_cond_table_floats() floats),
// or null for the direct kernel.
inline int launch_adaln_cond(const AdalnCondParams& p, const float* table, int sm_count,
                             cudaStream_t stream) {
  if (p.Cb % 8 != 0 || p.Cb <= 0 || p.factor <= 0 || p.ks <= 0 || (p.ks & 1) == 0 || p.ks > 9 ||
      p.D <= 0 || p.h <= 0 || p.w <= 0 || p.row0 < 0)
    return -2;
  if (p.n_rows <= 0) return 0;
  if (table != nullptr && p.h >= 3 && p.w >= 3 &&
      adaln_cond_table_floats(p.Cb, p.factor, p.ks) > 0) {
    const long long W = static_cast<long long>(p.w) * p.factor;
    const long long cell_rows = (p.row0 + p.n_rows - 1) / W / p.factor - p.row0 / W / p.factor + 1;
    const int groups = (p.Cb + 63) / 64;
    long long warps = cell_rows * (2 + (p.w - 2 + COND_RUN - 1) / COND_RUN);
    // 16 warps of this kernel fill an SM; below two such waves a run's phase rows go to separate warps
    const int psplit = warps * groups < 32LL * sm_count ? p.factor : 1;
    warps *= psplit;
    long long blocks = (warps + 7) / 8;
    const long long cap = (static_cast<long long>(sm_count) * 16 + groups - 1) / groups;
    if (blocks > cap) blocks = cap;
    blocks *= groups;
    return launch_chained(adaln_cond_runs_kernel, dim3(static_cast<unsigned>(blocks)), 256, 0, stream, 1, p, table, psplit);
  }
  const long long total = p.n_rows * (p.Cb / 8);
  long long blocks = (total + 255) / 256;
  const long long cap = static_cast<long long>(sm_count) * 32;
  if (blocks > cap) blocks = cap;
  return launch_chained(adaln_cond_kernel, dim3(static_cast<unsigned>(blocks)), 256, 0, stream, 1, p);
}

}  // namespace strata
