// Per-tile geometry of the model's input: the tile centre the winds are rotated about and the
// packed rotary table of the tile's tokens, from the per-pixel latitudes and longitudes.
//
//   tile_sums_kernel   partial sums over a tile's pixels (latitude, longitude circle, unit
//                      vector); only launched when a tile has more pixels than one block of the
//                      second kernel should walk by itself
//   tile_tables_kernel tile centre from the sums; per pixel, where asked for, the wind rotation
//                      about it and the latitude channels; per token the stereographic
//                      coordinates of its patch x patch pixels about the tile's spherical
//                      centroid, their mean, and the (cos, sin) half pair of every frequency
//
// Everything is evaluated in double precision and rounded once. Bound: launch and dependent
// latency - the table is 4 * head_dim / 2 bytes per token, the arithmetic two sincos per pixel and
// one per table entry: 7 us for 32 x 32 pixels, 17 us for 256 x 256. (Written with tensor operations,
// rope.py, the tables are some 45 launches: 150 us of the GPU and 400 us of the host at 32 x 32.)
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "prepost.cuh"

namespace strata {

constexpr int GEO_SUMS = 6;            // lat, sin lon, cos lon, and the unit vector's x, y, z
constexpr int GEO_MAX_PARTS = 64;      // partial sums per tile
// Pixels up to which every block of the table kernel sums the tile itself (256 threads, so 4
// pixels a thread): below that the walk is shorter than another launch.
constexpr int GEO_SELF_SUM_PIXELS = 1024;

enum RopeMode : int { ROPE_NONE = 0, ROPE_AXIAL = 1, ROPE_STEREO = 2 };

__device__ __forceinline__ void geo_add_pixel(double lat, double lon, double (&s)[GEO_SUMS]) {
  double sl, cl, so, co;
  sincos(lat, &sl, &cl);
  sincos(lon, &so, &co);
  s[0] += lat; s[1] += so; s[2] += co;
  s[3] += cl * co; s[4] += cl * so; s[5] += sl;
}

// Sum over the block's 256 threads, result in thread 0 (fixed order: the same on every run).
__device__ __forceinline__ void geo_block_sum(double (&s)[GEO_SUMS], double (*sh)[GEO_SUMS]) {
#pragma unroll
  for (int k = 0; k < GEO_SUMS; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < GEO_SUMS; ++k) sh[threadIdx.x >> 5][k] = s[k];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 0; k < GEO_SUMS; ++k) {
      s[k] = 0.0;
      for (int w = 0; w < 8; ++w) s[k] += sh[w][k];
    }
}

__global__ void __launch_bounds__(256)
tile_sums_kernel(const float* __restrict__ lat, const float* __restrict__ lon, int HW,
                 double* __restrict__ parts) {
  chain_begin();
  __shared__ double sh[8][GEO_SUMS];
  const long long base = static_cast<long long>(blockIdx.y) * HW;
  double s[GEO_SUMS] = {0, 0, 0, 0, 0, 0};
  for (int i = blockIdx.x * 256 + threadIdx.x; i < HW; i += gridDim.x * 256)
    geo_add_pixel(static_cast<double>(__ldg(lat + base + i)), static_cast<double>(__ldg(lon + base + i)), s);
  geo_block_sum(s, sh);
  if (threadIdx.x == 0)
    for (int k = 0; k < GEO_SUMS; ++k)
      parts[(static_cast<long long>(blockIdx.y) * gridDim.x + blockIdx.x) * GEO_SUMS + k] = s[k];
}

struct TileTablesParams {
  const float* lat;          // [B, H, W] radians
  const float* lon;
  int H, W, patch, h, w;     // h x w tokens of patch x patch pixels
  int mode, pairs;           // pairs = head_dim / 2
  double inv_scale;          // 1 / (length_scale * patch * patch): mean and unit in one factor
  double freq[32];           // theta^(-i / (pairs / 2)), i < pairs / 2
  const double* parts;       // [B, n_parts, GEO_SUMS], or null: sum the tile here
  int n_parts;
  float* lat0;               // [B] tile centre (nullable)
  float* lon0;
  uint32_t* table;           // [B, h*w, pairs] (cos, sin) half pairs; unused for ROPE_NONE
  // per-pixel geometry for the pre- and post-processing kernels, each nullable: wind rotation
  // into the tile frame and back (need lat0), (cos lat, sin lat)
  float4 *px_fwd, *px_inv;   // [B, H, W]
  float2* px_lat;
};

__host__ __device__ constexpr int geo_tokens_per_warp(int mode, int patch) {
  return mode != ROPE_STEREO || patch > 4 || patch == 3 ? 1 : (patch == 1 ? 32 : (patch == 2 ? 8 : 2));
}

__global__ void __launch_bounds__(256) tile_tables_kernel(const TileTablesParams p) {
  chain_begin();
  __shared__ double sh[8][GEO_SUMS];
  __shared__ double centre[4];         // sin / cos of the centroid's latitude, of its longitude
  __shared__ float wind0[2];           // tile centre of the wind rotation
  const int HW = p.H * p.W;
  const long long base = static_cast<long long>(blockIdx.y) * HW;
  if (p.mode == ROPE_STEREO || (p.lat0 != nullptr && (blockIdx.x == 0 || p.px_fwd != nullptr))) {
    double s[GEO_SUMS] = {0, 0, 0, 0, 0, 0};
    if (p.parts == nullptr) {
      for (int i = threadIdx.x; i < HW; i += 256)
        geo_add_pixel(static_cast<double>(__ldg(p.lat + base + i)),
                      static_cast<double>(__ldg(p.lon + base + i)), s);
    } else if (threadIdx.x < p.n_parts) {
      const double* q = p.parts + (static_cast<long long>(blockIdx.y) * p.n_parts + threadIdx.x) * GEO_SUMS;
#pragma unroll
      for (int k = 0; k < GEO_SUMS; ++k) s[k] = q[k];
    }
    geo_block_sum(s, sh);
    if (threadIdx.x == 0) {
      if (p.lat0 != nullptr) {
        double l = atan2(s[1] / HW, s[2] / HW);
        if (l < 0.0) l += 6.283185307179586476925;
        wind0[0] = static_cast<float>(s[0] / HW);
        wind0[1] = static_cast<float>(l);
        if (blockIdx.x == 0) {
          p.lat0[blockIdx.y] = wind0[0];
          p.lon0[blockIdx.y] = wind0[1];
        }
      }
      const double n = sqrt(s[3] * s[3] + s[4] * s[4] + s[5] * s[5]), r = sqrt(s[3] * s[3] + s[4] * s[4]);
      centre[0] = s[5] / n;
      centre[1] = r / n;
      centre[2] = r > 0.0 ? s[4] / r : 0.0;
      centre[3] = r > 0.0 ? s[3] / r : 1.0;
    }
    __syncthreads();
  }
  if (p.px_fwd != nullptr || p.px_lat != nullptr) {
    Basis q0{};
    if (p.px_fwd != nullptr) {
      double s0, c0, so0, co0;
      sincos(static_cast<double>(wind0[0]), &s0, &c0);
      sincos(static_cast<double>(wind0[1]), &so0, &co0);
      q0 = local_basis_enr(s0, c0, so0, co0);
    }
    for (int i = blockIdx.x * 256 + threadIdx.x; i < HW; i += gridDim.x * 256) {
      double sl, cl, so, co;
      sincos(static_cast<double>(__ldg(p.lat + base + i)), &sl, &cl);
      if (p.px_lat != nullptr) p.px_lat[base + i] = make_float2(static_cast<float>(cl), static_cast<float>(sl));
      if (p.px_fwd == nullptr) continue;
      sincos(static_cast<double>(__ldg(p.lon + base + i)), &so, &co);
      const Basis q = local_basis_enr(sl, cl, so, co);
      p.px_fwd[base + i] = wind_matrix(q, q0, true);
      p.px_inv[base + i] = wind_matrix(q, q0, false);
    }
  }
  if (p.mode == ROPE_NONE) return;
  const int lane = threadIdx.x & 31;
  const int tokens = p.h * p.w, half = p.pairs >> 1;
  // A warp takes TPW tokens at a time: first 32 / TPW lanes per token share its pixels, then all
  // lanes write the tokens' rows one after the other. (With one token per warp 31 lanes wait for
  // the one pixel of a patch-1 token: 64 us for 24 tiles of 48 x 48, 24 this way.)
  const int tpw = geo_tokens_per_warp(p.mode, p.patch), lpt = 32 / tpw;
  for (int t0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * tpw; t0 < tokens; t0 += gridDim.x * 8 * tpw) {
    const int t = min(t0 + lane / lpt, tokens - 1);
    const int ti = t / p.w, tj = t - ti * p.w;
    double x = tj, y = ti;
    if (p.mode == ROPE_STEREO) {
      const double s0 = centre[0], c0 = centre[1];
      x = 0.0; y = 0.0;
      for (int q = lane % lpt; q < p.patch * p.patch; q += lpt) {
        const int dy = q / p.patch, dx = q - dy * p.patch;
        const long long pix = base + static_cast<long long>(ti * p.patch + dy) * p.W + tj * p.patch + dx;
        double sl, cl, so, co;
        sincos(static_cast<double>(__ldg(p.lat + pix)), &sl, &cl);
        sincos(static_cast<double>(__ldg(p.lon + pix)), &so, &co);
        // sin / cos of the longitude difference to the centroid
        const double sd = so * centre[3] - co * centre[2], cd = co * centre[3] + so * centre[2];
        const double k = 2.0 / (1.0 + s0 * sl + c0 * cl * cd);
        x += k * cl * sd;
        y += k * (c0 * sl - s0 * cl * cd);
      }
      for (int o = lpt >> 1; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
      }
      x *= p.inv_scale;
      y *= p.inv_scale;
    }
    const int n = min(tpw, tokens - t0);
    uint32_t* row = p.table + (static_cast<long long>(blockIdx.y) * tokens + t0) * p.pairs;
    for (int i = 0; i < n; ++i, row += p.pairs) {
      const double xi = __shfl_sync(0xffffffffu, x, i * lpt), yi = __shfl_sync(0xffffffffu, y, i * lpt);
      for (int j = lane; j < p.pairs; j += 32) {
        double s, c;
        sincos(j < half ? xi * p.freq[j] : yi * p.freq[j - half], &s, &c);
        const __half2 v = __floats2half2_rn(static_cast<float>(c), static_cast<float>(s));
        row[j] = *reinterpret_cast<const uint32_t*>(&v);
      }
    }
  }
}

inline int geo_parts(int HW) {
  if (HW <= GEO_SELF_SUM_PIXELS) return 0;
  const int n = (HW + 1023) / 1024;
  return n < GEO_MAX_PARTS ? n : GEO_MAX_PARTS;
}
inline long long tile_tables_ws_bytes(int B, int H, int W) {
  return static_cast<long long>(B) * geo_parts(H * W) * GEO_SUMS * 8;
}

// ws: tile_tables_ws_bytes() of scratch, 8-byte aligned (null when that is 0).
inline int launch_tile_tables(TileTablesParams p, int B, double* ws, cudaStream_t stream) {
  p.n_parts = geo_parts(p.H * p.W);
  p.parts = nullptr;
  if (p.n_parts > 0 && (p.mode == ROPE_STEREO || p.lat0 != nullptr)) {
    const int r = launch_chained(tile_sums_kernel, dim3(p.n_parts, B), 256, 0, stream, 1, p.lat, p.lon, p.H * p.W, ws);
    if (r != 0) return r;
    p.parts = ws;
  }
  // one round of tokens per warp, one pixel per thread
  const int tpb = 8 * geo_tokens_per_warp(p.mode, p.patch);
  int bx = p.mode == ROPE_NONE ? 1 : (p.h * p.w + tpb - 1) / tpb;
  if (p.px_fwd != nullptr || p.px_lat != nullptr) bx = std::max(bx, (p.H * p.W + 255) / 256);
  if (bx > 1024) bx = 1024;
  return launch_chained(tile_tables_kernel, dim3(bx, B), 256, 0, stream, 1, p);
}

}  // namespace strata
