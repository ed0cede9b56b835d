// Fused pre- and post-processing of the Strata wrapper around the token path.
//
// Pre (one pass over the input fields instead of ~40 elementwise kernels, three concatenations
// and a transposing copy): for every pixel
//   * rotate the horizontal wind (U, V) from the pixel's east / north basis into the tangent
//     basis of the tile centre,
//   * append cos(lat), sin(lat) as two more channels,
//   * write the pixel's channel values, cast to bf16, into its slot of the patch-embedding
//     GEMM operand A[token, (c, dv, dh, dw)] (non-overlapping patches: a pure permutation).
// Post: the final linear layer's output Y[token, (dv, dh, dw, c)] is un-patchified to
// [B, C_out, D, H, W] fp32 and the wind channels are rotated back to east / north.
//
// Both directions are transposes between rows of pixels and rows of tokens, so a block takes a run
// of neighbouring tokens of one token row (NT tokens, ph image rows of NT * pw pixels, a few
// levels) through a tile in shared memory: fields are read and written along image rows, token
// rows as whole 16-byte vectors. The wind rotation is a 2 x 2 matrix per pixel in double precision
// (its values are then independent of the fast-math setting), from the caller's table or worked
// out once per block for its levels: two double sincos per pixel, which otherwise set the pace.
// Bound: HBM, 4 bytes of field and 2 of token per value, and in practice the latency of a block's
// load - barrier - store sequence. 13 fields of 24 x 256 x 256 at patch 4 (126 MB): in 60 us, out 48;
// of 13 x 88 x 120, three tiles: in 20, out 15. (A thread that walks one pixel's levels and channels,
// storing two bytes at a time into token rows that its neighbours share, takes 212 and 51, 90 and 25.)
#pragma once
#include <algorithm>

#include "common.cuh"

namespace strata {

struct Basis {
  double e[3], n[3], r[3];
};
__device__ __forceinline__ Basis local_basis_enr(double sl, double cl, double so, double co) {
  Basis b;
  b.e[0] = -so; b.e[1] = co; b.e[2] = 0.0;
  b.n[0] = -sl * co; b.n[1] = -sl * so; b.n[2] = cl;
  b.r[0] = cl * co; b.r[1] = cl * so; b.r[2] = sl;
  return b;
}
__device__ __forceinline__ double dot3(const double (&a)[3], const double (&b)[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

struct PrePostParams {
  int B, C, D, H, W;      // field tensor [B, C, D, H, W] (C = channels of x resp. of the output)
  int pv, ph, pw;         // patch extents
  int u_idx, v_idx;       // wind channels, -1: no rotation
  int concat_lat;         // pre only: append cos(lat), sin(lat)
  const float* lat;       // [B, H, W] radians
  const float* lon;
  const float* lat0;      // [B] tile-centre latitude / longitude (rotation only)
  const float* lon0;
  long long ld;           // row stride of the token matrix (elements)
  // the block's share (host-chosen, prepost_plan)
  int NT;                 // tokens of a run
  int DL;                 // token levels a block walks
  int LT;                 // of them side by side in the tile (tile row = level * nt + token)
  int chunk;              // pre: channels, post: (dv, dh) rows of a token that the tile holds
  int rs;                 // tile row stride (elements)
  // per-pixel geometry where the caller has it (tile_tables_kernel): rotation matrices of this
  // direction and (cos lat, sin lat); null: worked out by the block
  const float4* px_rot;
  const float2* px_lat;
};

constexpr int PREPOST_THREADS = 256;
constexpr int PREPOST_MAX_SMEM = 220 * 1024;

// Position of a block: tokens [tw0, tw0 + nt) of token row th of batch entry b, levels [td0, td1).
struct PrePostBlock {
  int b, th, tw0, nt, td0, td1;
};
__device__ __forceinline__ PrePostBlock prepost_block(const PrePostParams& p) {
  const int w_tok = p.W / p.pw, h_tok = p.H / p.ph, d_tok = p.D / p.pv;
  const int runs = (w_tok + p.NT - 1) / p.NT, dch = (d_tok + p.DL - 1) / p.DL;
  unsigned t = blockIdx.x;
  PrePostBlock k;
  k.tw0 = static_cast<int>(t % runs) * p.NT; t /= runs;
  k.th = static_cast<int>(t % h_tok); t /= h_tok;
  k.td0 = static_cast<int>(t % dch) * p.DL;
  k.b = static_cast<int>(t / dch);
  k.td1 = min(k.td0 + p.DL, d_tok);
  k.nt = min(p.NT, w_tok - k.tw0);
  return k;
}

// Wind rotation of a pixel: forward from its east / north basis into the tangent basis of the
// tile centre, inverse the way back (reference: forward_uv_to_tile / inverse_tile_to_uv,
// screamcast/wind_rotation.py:49-144); rows (u, v), columns (first, second component).
__device__ __forceinline__ float4 wind_matrix(const Basis& q, const Basis& q0, bool forward) {
  float4 m;
  if (forward) {   // the component along the centre's radial drops out: e0, n0 are normal to r0
    m.x = static_cast<float>(dot3(q.e, q0.e)); m.y = static_cast<float>(dot3(q.n, q0.e));
    m.z = static_cast<float>(dot3(q.e, q0.n)); m.w = static_cast<float>(dot3(q.n, q0.n));
  } else {
    const double rr = dot3(q0.r, q.r);
    const double bu = dot3(q0.e, q.r) / rr, bv = dot3(q0.n, q.r) / rr;
    const double re = dot3(q0.r, q.e), rn = dot3(q0.r, q.n);
    m.x = static_cast<float>(dot3(q0.e, q.e) - bu * re);
    m.y = static_cast<float>(dot3(q0.n, q.e) - bv * re);
    m.z = static_cast<float>(dot3(q0.e, q.n) - bu * rn);
    m.w = static_cast<float>(dot3(q0.n, q.n) - bv * rn);
  }
  return m;
}

// The block's pixels: rotation matrices rot[i] (nullable), i = dh * (nt*pw) + x, and cos / sin of
// their latitudes (nullable) - copied from the caller's tables or worked out here.
__device__ __forceinline__ void prepost_geometry(const PrePostParams& p, const PrePostBlock& k,
                                                 bool forward, float4* rot, float2* latcs) {
  const int npx = k.nt * p.pw;
  auto pixel = [&](int i) {
    const int dh = i / npx, x = i - dh * npx;
    return (static_cast<long long>(k.b) * p.H + k.th * p.ph + dh) * p.W + k.tw0 * p.pw + x;
  };
  if (rot && p.px_rot) {
    for (int i = threadIdx.x; i < p.ph * npx; i += PREPOST_THREADS) rot[i] = __ldg(p.px_rot + pixel(i));
    rot = nullptr;
  }
  if (latcs && p.px_lat) {
    for (int i = threadIdx.x; i < p.ph * npx; i += PREPOST_THREADS) latcs[i] = __ldg(p.px_lat + pixel(i));
    latcs = nullptr;
  }
  if (!rot && !latcs) return;
  Basis q0{};
  if (rot) {
    double s0, c0, so0, co0;
    sincos(static_cast<double>(__ldg(p.lat0 + k.b)), &s0, &c0);
    sincos(static_cast<double>(__ldg(p.lon0 + k.b)), &so0, &co0);
    q0 = local_basis_enr(s0, c0, so0, co0);
  }
  for (int i = threadIdx.x; i < p.ph * npx; i += PREPOST_THREADS) {
    const long long pix = pixel(i);
    double sl, cl;
    sincos(static_cast<double>(__ldg(p.lat + pix)), &sl, &cl);
    if (latcs) latcs[i] = make_float2(static_cast<float>(cl), static_cast<float>(sl));
    if (!rot) continue;
    double so, co;
    sincos(static_cast<double>(__ldg(p.lon + pix)), &so, &co);
    rot[i] = wind_matrix(local_basis_enr(sl, cl, so, co), q0, forward);
  }
}

template <int V>
__device__ __forceinline__ void load_px(const float* p, float (&v)[V]) {
  if constexpr (V == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else if constexpr (V == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(p));
    v[0] = t.x; v[1] = t.y;
  } else {
    v[0] = __ldg(p);
  }
}

// Counts in mixed radix (n0, n1, n2, unbounded), advancing by a fixed step: the digits of a running
// index without a division per step.
struct Digits {
  int n0, n1, n2;
  int d0, d1, d2, d3;      // current digits, least significant first
  int s0, s1, s2, s3;      // the step's
  __device__ __forceinline__ Digits(int start, int step, int r0, int r1, int r2)
      : n0(r0), n1(r1), n2(r2) {
    split(start, d0, d1, d2, d3);
    split(step, s0, s1, s2, s3);
  }
  __device__ __forceinline__ void split(int v, int& a, int& b, int& c, int& d) const {
    a = v % n0; v /= n0;
    b = v % n1; v /= n1;
    c = v % n2;
    d = v / n2;
  }
  __device__ __forceinline__ void next() {
    d0 += s0; d1 += s1; d2 += s2; d3 += s3;
    if (d0 >= n0) { d0 -= n0; ++d1; }
    if (d1 >= n1) { d1 -= n1; ++d2; }
    if (d2 >= n2) { d2 -= n2; ++d3; }
  }
};

// x [B, C, D, H, W] fp32 -> A [B*d*h*w, ld] bf16, columns (c, dv, dh, dw), zero beyond K.
// V: pixels of a row a thread handles together (4 or 2: pw and W are multiples of it).
template <int V>
__global__ void __launch_bounds__(PREPOST_THREADS, 3)
preprocess_patches_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ a,
                          const PrePostParams p) {
  chain_begin();
  extern __shared__ __align__(16) uint8_t pp_smem[];
  constexpr int UR = 4;
  const PrePostBlock k = prepost_block(p);
  const int npx = k.nt * p.pw, pvol = p.pv * p.ph * p.pw, prow = p.pv * p.ph;
  const int c_all = p.C + (p.concat_lat ? 2 : 0);
  const bool rotate = p.u_idx >= 0;
  float4* rot = reinterpret_cast<float4*>(pp_smem);
  float2* latcs = reinterpret_cast<float2*>(rot + (rotate ? p.ph * p.NT * p.pw : 0));
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(
      pp_smem + (((rotate ? 16 : 0) + (p.concat_lat ? 8 : 0)) * p.ph * p.NT * p.pw + 15) / 16 * 16);
  if (rotate || p.concat_lat)
    prepost_geometry(p, k, true, rotate ? rot : nullptr, p.concat_lat ? latcs : nullptr);
  const long long plane = static_cast<long long>(p.H) * p.W, cstep = p.D * plane;
  // threads: TX columns of V pixels x TY (level, channel, dv, dh) rows
  const int TX = min(npx / V, PREPOST_THREADS), TY = PREPOST_THREADS / TX;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const float* xb = x + static_cast<long long>(k.b) * p.C * cstep +
                    static_cast<long long>(k.th * p.ph) * p.W + k.tw0 * p.pw;
  const int w_tok = p.W / p.pw, h_tok = p.H / p.ph, d_tok = p.D / p.pv;
  const bool a_vec = (reinterpret_cast<uintptr_t>(a) & 15u) == 0 && (p.ld & 7) == 0;
  const long long lstep = static_cast<long long>(h_tok) * w_tok * p.ld;   // one level up
  for (int td = k.td0; td < k.td1; td += p.LT) {
    const int nl = min(p.LT, k.td1 - td);
    __nv_bfloat16* arow = a + (((static_cast<long long>(k.b) * d_tok + td) * h_tok + k.th) * w_tok + k.tw0) * p.ld;
    for (int c0 = 0; c0 < c_all; c0 += p.chunk) {
      const int nc = min(p.chunk, c_all - c0);
      __syncthreads();          // geometry written / the previous tile has been copied out
      if (ty < TY)
        for (int xi = tx * V; xi < npx; xi += TX * V) {
          const int tok = xi / p.pw, dw = xi - tok * p.pw;
          __nv_bfloat16* trow = tile + tok * p.rs + dw;
          Digits r(ty, TY, p.ph, p.pv, nc);     // dh, dv, channel, level
          const int n_rows = nl * nc * prow;
          for (int rl = ty; rl < n_rows; rl += UR * TY) {
            // UR independent loads first: a block is paced by their latency
            float v[UR][V];
            int col[UR], ch[UR], dh[UR];
            const float* src[UR];
#pragma unroll
            for (int u = 0; u < UR; ++u) {
              ch[u] = rl + u * TY < n_rows ? c0 + r.d2 : -1;
              dh[u] = r.d0;
              // column (channel, dv, dh, dw) of the tile row (level, token)
              col[u] = r.d3 * k.nt * p.rs + ((r.d2 * p.pv + r.d1) * p.ph + r.d0) * p.pw;
              src[u] = xb + (c0 + r.d2) * cstep + ((td + r.d3) * p.pv + r.d1) * plane +
                       static_cast<long long>(r.d0) * p.W + xi;
              if (ch[u] >= 0 && ch[u] < p.C) load_px<V>(src[u], v[u]);
              r.next();
            }
#pragma unroll
            for (int u = 0; u < UR; ++u) {
              if (ch[u] < 0) continue;
              if (ch[u] >= p.C) {
#pragma unroll
                for (int i = 0; i < V; ++i) {
                  const float2 cs = latcs[dh[u] * npx + xi + i];
                  v[u][i] = ch[u] == p.C ? cs.x : cs.y;
                }
              } else if (rotate && (ch[u] == p.u_idx || ch[u] == p.v_idx)) {
                float o[V];
                load_px<V>(src[u] + (ch[u] == p.u_idx ? p.v_idx - p.u_idx : p.u_idx - p.v_idx) * cstep, o);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                  const float4 m = rot[dh[u] * npx + xi + i];
                  v[u][i] = ch[u] == p.u_idx ? v[u][i] * m.x + o[i] * m.y : o[i] * m.z + v[u][i] * m.w;
                }
              }
              __nv_bfloat16* t = trow + col[u];
              if constexpr (V == 4) {
                uint2 o;
                o.x = pack_bf16(v[u][0], v[u][1]);
                o.y = pack_bf16(v[u][2], v[u][3]);
                *reinterpret_cast<uint2*>(t) = o;
              } else if constexpr (V == 2) {
                *reinterpret_cast<uint32_t*>(t) = pack_bf16(v[u][0], v[u][1]);
              } else {
                *t = __float2bfloat16(v[u][0]);
              }
            }
          }
        }
      // the tile's columns of the token rows; the last chunk also carries the padding columns
      const int cols = nc * pvol;
      const bool last = c0 + nc == c_all;
      const int wcols = last ? static_cast<int>(p.ld - static_cast<long long>(c0) * pvol) : cols;
      __syncthreads();
      __nv_bfloat16* dst = arow + static_cast<long long>(c0) * pvol;
      if (a_vec && ((wcols | (c0 * pvol)) & 7) == 0) {
        const int vec = wcols >> 3;
        Digits i(threadIdx.x, PREPOST_THREADS, vec, k.nt, 1 << 30);      // vector, token, level
        for (; i.d2 < nl; i.next()) {
          uint4 o = make_uint4(0u, 0u, 0u, 0u);
          const __nv_bfloat16* t = tile + (i.d2 * k.nt + i.d1) * p.rs + i.d0 * 8;
          if (i.d0 * 8 + 8 <= cols) {
            if constexpr (V == 4) {
              const uint2 lo = reinterpret_cast<const uint2*>(t)[0], hi = reinterpret_cast<const uint2*>(t)[1];
              o = make_uint4(lo.x, lo.y, hi.x, hi.y);
            } else {
              const uint32_t* w = reinterpret_cast<const uint32_t*>(t);
              o = make_uint4(w[0], w[1], w[2], w[3]);
            }
          } else if (i.d0 * 8 < cols) {        // the vector that holds the last live column
            __nv_bfloat16 e[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) e[j] = i.d0 * 8 + j < cols ? t[j] : __float2bfloat16(0.f);
            memcpy(&o, e, 16);
          }
          *reinterpret_cast<uint4*>(dst + i.d2 * lstep + i.d1 * p.ld + i.d0 * 8) = o;
        }
      } else {
        Digits i(threadIdx.x, PREPOST_THREADS, wcols, k.nt, 1 << 30);
        for (; i.d2 < nl; i.next())
          dst[i.d2 * lstep + i.d1 * p.ld + i.d0] =
              i.d0 < cols ? tile[(i.d2 * k.nt + i.d1) * p.rs + i.d0] : __float2bfloat16(0.f);
      }
    }
  }
}

// Y [B*d*h*w, ld] bf16, columns (dv, dh, dw, c) -> out [B, C, D, H, W] fp32, wind rotated back.
template <int V>
__global__ void __launch_bounds__(PREPOST_THREADS)
postprocess_fields_kernel(const __nv_bfloat16* __restrict__ y, float* __restrict__ out,
                          const PrePostParams p) {
  chain_begin();
  extern __shared__ __align__(16) uint8_t pp_smem[];
  const PrePostBlock k = prepost_block(p);
  const int npx = k.nt * p.pw, prow = p.pv * p.ph;
  const bool rotate = p.u_idx >= 0;
  float4* rot = reinterpret_cast<float4*>(pp_smem);
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(rot + (rotate ? p.ph * p.NT * p.pw : 0));
  if (rotate) prepost_geometry(p, k, false, rot, nullptr);
  const long long plane = static_cast<long long>(p.H) * p.W, cstep = p.D * plane;
  const int TX = min(npx / V, PREPOST_THREADS), TY = PREPOST_THREADS / TX;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  float* ob = out + static_cast<long long>(k.b) * p.C * cstep +
              static_cast<long long>(k.th * p.ph) * p.W + k.tw0 * p.pw;
  const int w_tok = p.W / p.pw, h_tok = p.H / p.ph, d_tok = p.D / p.pv;
  const bool vec_ok = (p.ld & 7) == 0 && (reinterpret_cast<uintptr_t>(y) & 15u) == 0;
  const long long lstep = static_cast<long long>(h_tok) * w_tok * p.ld;
  for (int td = k.td0; td < k.td1; td += p.LT) {
    const int nl = min(p.LT, k.td1 - td);
    const __nv_bfloat16* yrow = y + (((static_cast<long long>(k.b) * d_tok + td) * h_tok + k.th) * w_tok + k.tw0) * p.ld;
    for (int q0 = 0; q0 < prow; q0 += p.chunk) {
      const int nq = min(p.chunk, prow - q0);
      const int cols = nq * p.pw * p.C, col0 = q0 * p.pw * p.C;
      __syncthreads();
      if (vec_ok && (col0 & 7) == 0) {
        // (a row is at least its columns rounded up to 8 long)
        Digits i(threadIdx.x, PREPOST_THREADS, (cols + 7) >> 3, k.nt, 1 << 30);
#pragma unroll 2
        for (; i.d2 < nl; i.next()) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(yrow + i.d2 * lstep + i.d1 * p.ld + col0 + i.d0 * 8));
          uint32_t* t = reinterpret_cast<uint32_t*>(tile + (i.d2 * k.nt + i.d1) * p.rs + i.d0 * 8);
          t[0] = v.x; t[1] = v.y; t[2] = v.z; t[3] = v.w;
        }
      } else {
        Digits i(threadIdx.x, PREPOST_THREADS, cols, k.nt, 1 << 30);
        for (; i.d2 < nl; i.next())
          tile[(i.d2 * k.nt + i.d1) * p.rs + i.d0] = yrow[i.d2 * lstep + i.d1 * p.ld + col0 + i.d0];
      }
      __syncthreads();
      if (ty < TY)
        for (int xi = tx * V; xi < npx; xi += TX * V) {
          const int tok = xi / p.pw, dw = xi - tok * p.pw;
          Digits r(ty, TY, nq, p.C, 1 << 30);       // (dv, dh) row of the chunk, channel, level
          for (int rl = ty; rl < nl * nq * p.C; rl += TY, r.next()) {
            const int q = q0 + r.d0, dv = prow == p.ph ? 0 : q / p.ph, dh = q - dv * p.ph, c = r.d1;
            const __nv_bfloat16* t = tile + (r.d2 * k.nt + tok) * p.rs + (r.d0 * p.pw + dw) * p.C;
            float v[V];
#pragma unroll
            for (int i = 0; i < V; ++i) v[i] = __bfloat162float(t[i * p.C + c]);
            if (rotate && (c == p.u_idx || c == p.v_idx)) {
              const int other = c == p.u_idx ? p.v_idx : p.u_idx;
#pragma unroll
              for (int i = 0; i < V; ++i) {
                const float o = __bfloat162float(t[i * p.C + other]);
                const float4 m = rot[dh * npx + xi + i];
                v[i] = c == p.u_idx ? v[i] * m.x + o * m.y : o * m.z + v[i] * m.w;
              }
            }
            float* dst = ob + c * cstep + ((td + r.d2) * p.pv + dv) * plane +
                         static_cast<long long>(dh) * p.W + xi;
            if constexpr (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            else if constexpr (V == 2) *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
            else *dst = v[0];
          }
        }
    }
  }
}

// Patch 1 x 1 x 1: a token is a pixel and both sides are rows of pixels already, so one thread
// takes a pixel through p.DL levels, eight channels at a time (one 16-byte piece of the token row;
// eight independent field accesses, each contiguous over the warp). Needs ld % 8 == 0 and a
// 16-byte aligned token matrix. Through the shared-memory tile the same rows took two to four
// times as long (8 fields of 24 tiles 8 x 48 x 48: 9 us in, 8 out, against 36 and 29): two barriers
// per tile for a transpose that is not there.
__device__ __forceinline__ void pixel_geometry(const PrePostParams& p, long long pix, int b, bool forward,
                                               float4& m, float2& cs) {
  const bool rotate = p.u_idx >= 0;
  if (rotate && p.px_rot) m = __ldg(p.px_rot + pix);
  if (p.concat_lat && p.px_lat) cs = __ldg(p.px_lat + pix);
  const bool need_m = rotate && !p.px_rot, need_cs = p.concat_lat && !p.px_lat;
  if (!need_m && !need_cs) return;
  double sl, cl;
  sincos(static_cast<double>(__ldg(p.lat + pix)), &sl, &cl);
  if (need_cs) cs = make_float2(static_cast<float>(cl), static_cast<float>(sl));
  if (!need_m) return;
  double so, co, s0, c0, so0, co0;
  sincos(static_cast<double>(__ldg(p.lon + pix)), &so, &co);
  sincos(static_cast<double>(__ldg(p.lat0 + b)), &s0, &c0);
  sincos(static_cast<double>(__ldg(p.lon0 + b)), &so0, &co0);
  m = wind_matrix(local_basis_enr(sl, cl, so, co), local_basis_enr(s0, c0, so0, co0), forward);
}

__global__ void __launch_bounds__(PREPOST_THREADS)
preprocess_pixels_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ a, const PrePostParams p) {
  chain_begin();
  const long long plane = static_cast<long long>(p.H) * p.W, cstep = p.D * plane;
  const long long pix = static_cast<long long>(blockIdx.x) * PREPOST_THREADS + threadIdx.x;
  if (pix >= p.B * plane) return;
  const int b = static_cast<int>(pix / plane);
  float4 m = make_float4(1.f, 0.f, 0.f, 1.f);
  float2 cs = make_float2(0.f, 0.f);
  pixel_geometry(p, pix, b, true, m, cs);
  const bool rotate = p.u_idx >= 0;
  const int c_lat = p.concat_lat ? p.C : -8;
  const int d1 = min(p.D, static_cast<int>(blockIdx.y + 1) * p.DL);
  for (int d = blockIdx.y * p.DL; d < d1; ++d) {
    const float* src = x + b * p.C * cstep + d * plane + (pix - b * plane);
    uint4* row = reinterpret_cast<uint4*>(a + ((static_cast<long long>(b) * p.D + d) * plane + (pix - b * plane)) * p.ld);
    float ur = 0.f, vr = 0.f;
    if (rotate) {
      const float U = __ldg(src + p.u_idx * cstep), V = __ldg(src + p.v_idx * cstep);
      ur = U * m.x + V * m.y;
      vr = U * m.z + V * m.w;
    }
    for (int c0 = 0; c0 < p.ld; c0 += 8) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = c0 + j < p.C ? __ldg(src + (c0 + j) * cstep) : 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (c0 + j == c_lat) v[j] = cs.x;
        if (c0 + j == c_lat + 1) v[j] = cs.y;
        if (rotate && c0 + j == p.u_idx) v[j] = ur;
        if (rotate && c0 + j == p.v_idx) v[j] = vr;
      }
      uint4 o;
      o.x = pack_bf16(v[0], v[1]); o.y = pack_bf16(v[2], v[3]);
      o.z = pack_bf16(v[4], v[5]); o.w = pack_bf16(v[6], v[7]);
      row[c0 >> 3] = o;
    }
  }
}

__global__ void __launch_bounds__(PREPOST_THREADS)
postprocess_pixels_kernel(const __nv_bfloat16* __restrict__ y, float* __restrict__ out, const PrePostParams p) {
  chain_begin();
  const long long plane = static_cast<long long>(p.H) * p.W, cstep = p.D * plane;
  const long long pix = static_cast<long long>(blockIdx.x) * PREPOST_THREADS + threadIdx.x;
  if (pix >= p.B * plane) return;
  const int b = static_cast<int>(pix / plane);
  float4 m = make_float4(1.f, 0.f, 0.f, 1.f);
  float2 cs;
  pixel_geometry(p, pix, b, false, m, cs);
  const bool rotate = p.u_idx >= 0;
  const int d1 = min(p.D, static_cast<int>(blockIdx.y + 1) * p.DL);
  for (int d = blockIdx.y * p.DL; d < d1; ++d) {
    float* dst = out + b * p.C * cstep + d * plane + (pix - b * plane);
    const __nv_bfloat16* row = y + ((static_cast<long long>(b) * p.D + d) * plane + (pix - b * plane)) * p.ld;
    float ug = 0.f, vg = 0.f;
    if (rotate) {
      const float U = __bfloat162float(row[p.u_idx]), V = __bfloat162float(row[p.v_idx]);
      ug = U * m.x + V * m.y;
      vg = U * m.z + V * m.w;
    }
    for (int c0 = 0; c0 < p.C; c0 += 8) {
      const uint4 r = __ldg(reinterpret_cast<const uint4*>(row + c0));
      float v[8] = {bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y),
                    bf16_lo(r.z), bf16_hi(r.z), bf16_lo(r.w), bf16_hi(r.w)};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (rotate && c0 + j == p.u_idx) v[j] = ug;
        if (rotate && c0 + j == p.v_idx) v[j] = vg;
        if (c0 + j < p.C) dst[(c0 + j) * cstep] = v[j];
      }
    }
  }
}

// Levels per thread of the two kernels above: one, until the chip is filled four times over.
inline dim3 pixels_grid(PrePostParams& p, int sms) {
  const long long blocks = (static_cast<long long>(p.B) * p.H * p.W + PREPOST_THREADS - 1) / PREPOST_THREADS;
  long long dl = blocks * p.D / (static_cast<long long>(sms) * 32);
  dl = std::max<long long>(1, std::min<long long>(dl, p.D));
  dl = std::max<long long>(dl, (p.D + 65534) / 65535);
  p.DL = static_cast<int>(dl);
  return dim3(static_cast<unsigned>(blocks), static_cast<unsigned>((p.D + p.DL - 1) / p.DL));
}

// Fills in the block's share. unit: tile columns of one chunk element (a channel's patch volume
// going in, one (dv, dh) row of all channels coming out), n_units of them per token. word: bytes
// of the tile's accesses (8: four pixels going in; 4).
inline int prepost_plan(PrePostParams& p, int unit, int n_units, int word, bool lat_too, int sms,
                        long long* blocks, int* smem) {
  const int geo = ((p.u_idx >= 0 ? 16 : 0) + (lat_too ? 8 : 0)) * p.ph;   // bytes per pixel column
  const int w_tok = p.W / p.pw, h_tok = p.H / p.ph, d_tok = p.D / p.pv;
  // The whole token row in a tile of at most 40 KB and 256 pixel columns (then 4 blocks or more
  // share an SM); when a single token is larger than that, pieces of it.
  constexpr int TILE = 40960;
  const long long row = 2LL * unit * n_units + 32;
  long long nt = std::min<long long>(TILE / std::min<long long>(row, TILE), std::max(1, 256 / p.pw));
  p.NT = static_cast<int>(std::min<long long>(nt, w_tok));
  p.chunk = n_units;
  if (row > TILE) {
    p.chunk = static_cast<int>(std::max<long long>(1, (TILE - 32) / (2LL * unit)));
    if (p.chunk > 8) p.chunk = p.chunk / 8 * 8;      // 16-byte pieces
    if (p.chunk > n_units) p.chunk = n_units;
  }
  // row stride: an odd number of `word`-byte words, so that a warp's accesses to one column of
  // neighbouring tokens spread over all banks
  const int e = word / 2;
  long long rs = (static_cast<long long>(p.chunk) * unit + 7) / 8 * 8 + e;
  if (rs / e % 2 == 0) rs += e;
  if (rs > (1 << 24)) return -2;
  p.rs = static_cast<int>(rs);
  // levels per block: enough blocks for two waves of four per SM first, then up to 8 levels that
  // share the block's geometry - side by side in the tile as far as it holds them
  const long long base = static_cast<long long>(p.B) * h_tok * ((w_tok + p.NT - 1) / p.NT);
  long long dl = base * d_tok / (static_cast<long long>(sms) * 8);
  dl = std::max<long long>(1, std::min<long long>(dl, 8));
  p.DL = static_cast<int>(std::min<long long>(dl, d_tok));
  p.LT = static_cast<int>(std::max<long long>(1, std::min<long long>(p.DL, TILE / (2 * rs * p.NT))));
  const long long bytes = (static_cast<long long>(geo) * p.NT * p.pw + 15) / 16 * 16 + 2 * rs * p.NT * p.LT;
  if (bytes > PREPOST_MAX_SMEM) return -2;
  *smem = static_cast<int>(bytes);
  *blocks = base * ((d_tok + p.DL - 1) / p.DL);
  return *blocks > 0x7fffffffLL ? -2 : 0;
}

// De-aliased patch gathering (reference: screamcast/dealias.py:28-143). The reference runs the
// patch convolution at stride 1 without padding, pads its output by replication, low-pass
// filters it per decimated axis and decimates by the patch size. Filtering commutes with the
// convolution, so the same tokens come from ONE strided GEMM whose operand rows are filtered
// patches:  A[token, (c, v, y, x)] = sum_k f[k] * X[c, s_d(k) + v, s_h(k) + y, s_w(k) + x]  with
// s_axis(k) = clamp(token_axis * patch + k_axis - (K_axis - 1) / 2, 0, size - patch) - the clamp
// is the replicate padding of the stride-1 output. X: pixel rows [B, D, H, W, ldx] bf16
// (channels last, the output of preprocess_patches at patch 1); A: [tokens, lda] bf16, zero
// beyond the C * pv * ph * pw valid columns.
struct DealiasParams {
  int B, C, D, H, W, pv, ph, pw;
  int kd, kh, kw;
  float fd[8], fh[8], fw[8];     // per-axis taps, each already divided by its sum
  long long ldx, lda;
};

__global__ void __launch_bounds__(256)
dealias_patches_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ a,
                       const DealiasParams p) {
  chain_begin();
  const int d_tok = p.D / p.pv, h_tok = p.H / p.ph, w_tok = p.W / p.pw;
  const int pvol = p.pv * p.ph * p.pw;
  const int K = p.C * pvol;
  const long long total = static_cast<long long>(p.B) * d_tok * h_tok * w_tok * p.lda;
  for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int col = static_cast<int>(t % p.lda);
    const long long tok = t / p.lda;
    if (col >= K) {
      a[t] = __float2bfloat16(0.f);
      continue;
    }
    const int c = col / pvol;
    int rem = col - c * pvol;
    const int v = rem / (p.ph * p.pw);
    rem -= v * p.ph * p.pw;
    const int yy = rem / p.pw, xx = rem - yy * p.pw;
    const int tw = static_cast<int>(tok % w_tok);
    const int th = static_cast<int>((tok / w_tok) % h_tok);
    const int td = static_cast<int>((tok / (static_cast<long long>(w_tok) * h_tok)) % d_tok);
    const long long b = tok / (static_cast<long long>(w_tok) * h_tok * d_tok);
    float acc = 0.f;
    for (int id = 0; id < p.kd; ++id) {
      int sd = td * p.pv + id - (p.kd - 1) / 2;
      sd = sd < 0 ? 0 : (sd > p.D - p.pv ? p.D - p.pv : sd);
      for (int ih = 0; ih < p.kh; ++ih) {
        int sh = th * p.ph + ih - (p.kh - 1) / 2;
        sh = sh < 0 ? 0 : (sh > p.H - p.ph ? p.H - p.ph : sh);
        const float fdh = p.fd[id] * p.fh[ih];
        const long long row = ((b * p.D + sd + v) * p.H + sh + yy) * p.W;
        for (int iw = 0; iw < p.kw; ++iw) {
          int sw = tw * p.pw + iw - (p.kw - 1) / 2;
          sw = sw < 0 ? 0 : (sw > p.W - p.pw ? p.W - p.pw : sw);
          acc = fmaf(fdh * p.fw[iw], __bfloat162float(x[(row + sw + xx) * p.ldx + c]), acc);
        }
      }
    }
    a[t] = __float2bfloat16(acc);
  }
}

}  // namespace strata
