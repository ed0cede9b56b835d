// Persistent, warp-specialised bf16 GEMM for sm_100a:  D[M,N] = A[M,K] * W[N,K]^T  with a
// fused epilogue. One CTA per SM; each CTA walks output tiles of 128 x BN.
//
//   warp 0      TMA producer: streams 128x64 A tiles and BNx64 W tiles (128-byte swizzle)
//               into a ring of shared-memory stages.
//   warp 1      MMA issuer: one thread issues tcgen05.mma (M=128, N=BN, K=16) from the smem
//               stages into one of two TMEM accumulators (2 x BN fp32 columns), and commits
//               stage-free / accumulator-full mbarriers.
//   warps 2-17  epilogue (16 warps: four per SM sub-partition, because the epilogue of a
//               128 x 256 tile is bound by the latency of each warp's instruction stream
//               rather than by issue slots): read the finished accumulator with tcgen05.ld
//               (as matrix fragments, or each thread one output row, 16 columns at a time), apply bias
//               and the selected epilogue, store bf16. The other accumulator is being filled meanwhile.
//
// BN = 256, 128 or 64 by the rule of launch_gemm. PAIR variant (large problems): two CTAs of a cluster share every MMA
// (tcgen05 cta_group::2,
// M = 256): each CTA loads its own 128 rows of A and HALF of the W tile, the instruction reads
// both halves, and each CTA's tensor memory receives its 128 rows x BN accumulator. A CTA then
// moves 32 KB per k-block through shared memory instead of 48 KB, which matters because the
// one-CTA mainloop is bound by shared-memory bandwidth (operand reads + TMA writes), not by the
// tensor pipe. The first CTA of the pair issues the MMAs; TMA loads of both CTAs signal its
// stage barriers, its commits arrive on both CTAs' barriers, and both CTAs' epilogue warps hand
// the accumulator back on its barrier. Everything else (epilogues, staging, stores) is per CTA.
//
// Epilogues (the operator each one serves in the Strata block):
//   EPI_BIAS           y = acc + b                                   (generic Linear)
//   EPI_GELU           y = gelu_tanh(acc + b)                        (mlp.layers.0 + tanh GELU)
//   EPI_RESIDUAL       y = acc + b + R[m,n]                          (attn.proj / mlp.layers.2)
//   EPI_RESIDUAL_LN    the same, and layernorm(y) besides            (attn.proj and the norm behind it)
//   EPI_QKV_ROPE       y = rope(acc + b) on q,k columns              (attn.qkv + RoPE + pack)
//   EPI_QKV_NORM       y = rope(rmsnorm(acc + b)) on q,k columns     (the same with the q/k norm)
//   EPI_GATE           y = G[m,n] * sigmoid(acc + b)                 (attn.gate_proj)
#pragma once
#include <cuda_fp16.h>

#include <atomic>

#include "common.cuh"
#include "tensormap.cuh"

namespace strata {

enum GemmEpilogue : int {
  EPI_BIAS = 0,
  EPI_GELU = 1,
  EPI_RESIDUAL = 2,
  EPI_QKV_ROPE = 3,
  EPI_GATE = 4,
  EPI_QKV_NORM = 5,   // EPI_QKV_ROPE with the q/k norm
  EPI_RESIDUAL_LN = 6,   // EPI_RESIDUAL, and the LayerNorm of the result into a second matrix (N <= 256)
};

struct GemmParams {
  int M, N, K;
  __nv_bfloat16* out;
  long long ldo;
  const float* bias;          // [N] or nullptr
  const __nv_bfloat16* aux;   // residual (EPI_RESIDUAL) or gated operand (EPI_GATE)
  long long ldaux;
  // EPI_QKV_ROPE: table [n_tiles, hw, head_dim/2] of (cos, sin) pairs in IEEE half (4 bytes per
  // rotated channel pair); token row m belongs to tile m / tokens_per_tile and to horizontal
  // position m % hw (depth levels share a table row).
  const uint32_t* rope_cs;
  int tokens_per_tile;
  int hw;
  int head_dim;
  int rope_cols;   // columns [0, rope_cols) are q and k
  float qk_eps;
  float ln_eps;    // EPI_RESIDUAL_LN
  // Output row remap (pad_T > 0): the M input rows are the interior tokens of tiles
  // [tile, d, i, j] with i, j < pad_T (pad_T a multiple of 32), and row m is stored at row
  // ((tile*pad_D + d)*P + i + pad_h)*P + j + pad_h of the output, P = pad_T + 2*pad_h: the
  // interior of halo-padded tiles. A 32-row store box never leaves one interior row.
  int pad_T, pad_h, pad_D;
};

// Output row of input row m under the padded-tile remap (identity when it is off).
__device__ __forceinline__ int gemm_out_row(int m, const GemmParams& p) {
  if (p.pad_T == 0) return m;
  const int T = p.pad_T, P = T + 2 * p.pad_h;
  const int j = m % T;
  int t = m / T;
  const int i = t % T;
  t /= T;   // tile*pad_D + d
  return (t * P + i + p.pad_h) * P + j + p.pad_h;
}

constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;
constexpr int GEMM_EPI_WARPS = 16;
constexpr int GEMM_THREADS = 64 + 32 * GEMM_EPI_WARPS;

template <int BN, bool PAIR, bool TABLE>
struct GemmSmem {
  static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;
  static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * GEMM_BK * 2;   // a pair splits the W tile
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 256 && !PAIR ? (TABLE ? 3 : 4) : (TABLE ? 5 : 6);   // (BN = 64: 8 gain nothing)
  static constexpr int STAGING_BYTES = 32 * 32 * 2;             // one 32-row x 32-col bf16 box
  // TABLE: the rotary table rows of a tile's 128 output rows, 128 bytes each, twice (QKV epilogues), or the
  // LayerNorm's sums of 8 columns of every row, for the mean and the variance
  static constexpr int TABLE_BYTES = TABLE ? 2 * GEMM_BM * 128 : 0;
  static constexpr int STAGING_OFF = STAGES * STAGE_BYTES;      // per epilogue warp
  static constexpr int TABLE_OFF = STAGING_OFF + GEMM_EPI_WARPS * STAGING_BYTES;
  static constexpr int BAR_OFF = TABLE_OFF + TABLE_BYTES;
  static constexpr int BAR_BYTES = 512;
  static constexpr int TOTAL = BAR_OFF + BAR_BYTES + 1024;      // + alignment slack
  static_assert(TOTAL <= 232448, "shared memory of an SM");
};

// TMA store of a shared-memory box to global memory (bulk async group of the issuing thread).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tm, uint32_t src, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
      ::"l"(tm), "r"(src), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_read0() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// tanh GELU of a pair: the polynomial part runs on packed fp32x2 instructions.
__device__ __forceinline__ uint64_t gelu_pair(uint64_t x) {
  const float k0 = 0.7978845608028654f, k01 = 0.7978845608028654f * 0.044715f;
  const uint64_t K0 = pack2(k0, k0), K01 = pack2(k01, k01), HALF = pack2(0.5f, 0.5f);
  const uint64_t u = fmul2(x, ffma2(fmul2(x, x), K01, K0));
  float u0, u1;
  unpack2(u, u0, u1);
  const uint64_t t = pack2(fast_tanh(u0), fast_tanh(u1));
  const uint64_t hx = fmul2(x, HALF);
  return ffma2(hx, t, hx);
}

// Epilogue math of the row-per-lane form on 16 consecutive columns of output row m, in place. Lane `src_lane0 + j` of
// the warp holds the bias of column j of the group; cs: this row's (cos, sin) half pairs for the 8 channel pairs of
// these 16 columns.
template <int EPI>
__device__ __forceinline__ void gemm_epilogue_16(float (&v)[16], bool rotate, float b_lane, int src_lane0,
                                                 const uint32_t (&cs)[8], const GemmParams& p, const float* bias16) {
  if (p.bias != nullptr) {
    if (bias16 != nullptr) {
      // the 16 biases of this column group, the same for every row: four 16-byte loads at an
      // address that is uniform over the warp (one L1 line, broadcast) instead of one shuffle
      // per output element
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias16) + q);
        v[4 * q] += b4.x; v[4 * q + 1] += b4.y; v[4 * q + 2] += b4.z; v[4 * q + 3] += b4.w;
      }
    } else {   // ragged right edge of the matrix: lane j of the group holds column j's bias
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += __shfl_sync(0xffffffffu, b_lane, src_lane0 + j);
    }
  }
  if constexpr (EPI == EPI_QKV_ROPE) {
    if (rotate) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 t =
            __half22float2(*reinterpret_cast<const __half2*>(&cs[j]));  // (cos, sin)
        const float a = v[2 * j], b = v[2 * j + 1];
        v[2 * j] = a * t.x - b * t.y;
        v[2 * j + 1] = a * t.y + b * t.x;
      }
    }
  }
}

// The other epilogues read the accumulator as matrix fragments, 16 rows x 32 columns a load: registers 4 i + {0, 1}
// hold row lane / 4, columns 8 i + 2 (lane % 4) + {0, 1}, registers 4 i + {2, 3} the same of row lane / 4 + 8. A lane
// then needs eight
// biases for 32 columns (with a row per lane all 32) and holds the pairs that the rotation turns, a row's
// squares are summed within a quad, and 8 x 8 pieces go to the staging boxes and come from them with stmatrix and
// ldmatrix.
__device__ __forceinline__ void tmem_ld_16x256_x4(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void stmatrix_x4(uint32_t addr, const uint32_t* w) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]),
               "r"(w[2]), "r"(w[3]) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t* w) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr) : "memory");
}

// The biases of this lane's columns in the 32 from n0 (zero without a bias, and behind column N).
__device__ __forceinline__ void gemm_lane_bias(const GemmParams& p, int n0, int lane, uint64_t (&bias)[4]) {
  const int n = n0 + 2 * (lane & 3);
  if (p.bias != nullptr && n0 + 32 <= p.N) {
#pragma unroll
    for (int i = 0; i < 4; ++i) bias[i] = __ldg(reinterpret_cast<const unsigned long long*>(p.bias + n + 8 * i));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = n + 8 * i;
      bias[i] = p.bias == nullptr ? 0ull
                                  : pack2(k < p.N ? __ldg(p.bias + k) : 0.f, k + 1 < p.N ? __ldg(p.bias + k + 1) : 0.f);
    }
  }
}

// Epilogue math on a pair of neighbouring columns of one row (bias added); aux: the residual / gated operand of the
// pair (bf16); cs: its (cos, sin) half pair; scale: the RMS factor of the row's head.
template <int EPI>
__device__ __forceinline__ uint32_t gemm_epilogue_pair(uint64_t x, uint32_t aux, bool rotate, uint32_t cs,
                                                       float scale) {
  float a, b;
  if constexpr (EPI == EPI_GELU) {
    unpack2(gelu_pair(x), a, b);
  } else {
    unpack2(x, a, b);
    if constexpr (EPI == EPI_RESIDUAL) {
      a += bf16_lo(aux);
      b += bf16_hi(aux);
    } else if constexpr (EPI == EPI_GATE) {
      a = bf16_lo(aux) / (1.0f + __expf(-a));
      b = bf16_hi(aux) / (1.0f + __expf(-b));
    } else if constexpr (EPI == EPI_QKV_NORM) {
      if (rotate) {
        a *= scale;
        b *= scale;
        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&cs));   // (cos, sin)
        // (spelled out: the row form's contractions, so that both give the same bits)
        const float r0 = __fmaf_rn(a, t.x, -__fmul_rn(b, t.y));
        b = __fmaf_rn(a, t.y, __fmul_rn(b, t.x));
        a = r0;
      }
    }
  }
  return pack_bf16(a, b);
}

// Per-head RMS factors of the q/k norm for one output row: one extra pass over the warp's
// WARP_COLS accumulator columns (+ bias). head_dim 64: the warp's 64 columns are one head, both
// components carry its factor; head_dim 32: one factor per 32-column sub-chunk. Called by a
// whole warp (tensor-memory loads).
template <int NSUB>
__device__ __noinline__ float2 gemm_qk_norm_scales(uint32_t taddr, const float* bias, int n_warp0,
                                                   int N, int lane, int head_dim, float eps) {
  static_assert(NSUB == 1 || NSUB == 2, "one or two 32-column sub-chunks per warp");
  float ss[NSUB];
#pragma unroll
  for (int cc = 0; cc < NSUB; ++cc) {
    float acc = 0.f;
    float bl = 0.f;
    if (bias != nullptr && n_warp0 + 32 * cc + lane < N) bl = __ldg(bias + n_warp0 + 32 * cc + lane);
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      uint32_t r[16];
      tmem_ld_32x16(taddr + 32 * cc + 16 * g, r);
      tmem_ld_wait();
      const int nb0 = n_warp0 + 32 * cc + 16 * g;
      if (bias != nullptr && nb0 + 16 <= N) {
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias + nb0) + q4);
          const float x0 = __uint_as_float(r[4 * q4]) + b4.x;
          const float x1 = __uint_as_float(r[4 * q4 + 1]) + b4.y;
          const float x2 = __uint_as_float(r[4 * q4 + 2]) + b4.z;
          const float x3 = __uint_as_float(r[4 * q4 + 3]) + b4.w;
          acc += x0 * x0 + x1 * x1 + x2 * x2 + x3 * x3;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float x = __uint_as_float(r[j]) + __shfl_sync(0xffffffffu, bl, 16 * g + j);
          acc += x * x;
        }
      }
    }
    ss[cc] = acc;
  }
  if (head_dim == 64 && NSUB == 2) {
    const float f = rsqrtf((ss[0] + ss[NSUB - 1]) * (1.0f / 64.0f) + eps);
    return make_float2(f, f);
  }
  return make_float2(rsqrtf(ss[0] * (1.0f / 32.0f) + eps), rsqrtf(ss[NSUB - 1] * (1.0f / 32.0f) + eps));
}

// LayerNorm of a row that four warps (a lane quarter) hold in parts, a row per lane, bf16 in and out: what
// layernorm_rows_kernel computes, with its order of additions - pairs, the four pairs of 8 columns in turn, then the
// 8-column sums i with i ^ 16, i ^ 8, ... - so that the result is the same bits. Each warp leaves its 8-column sums
// in shared memory ([groups][32 rows] of its quarter, one buffer for the mean and one for the variance) and reads all
// of them.
__device__ __forceinline__ float ln_group_sum(const uint32_t* w) {   // 8 columns
  float s = 0.f;
#pragma unroll
  for (int t = 0; t < 4; ++t) s += bf16_lo(w[t]) + bf16_hi(w[t]);
  return s;
}
__device__ __forceinline__ float ln_group_squares(const uint32_t* w, float mean) {
  float s = 0.f;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    float d = bf16_lo(w[t]) - mean;
    s += d * d;
    d = bf16_hi(w[t]) - mean;
    s += d * d;
  }
  return s;
}
__device__ __forceinline__ void ln_put(uint32_t buf, int group, int lane, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(buf + static_cast<uint32_t>(group * 32 + lane) * 4u), "f"(v) : "memory");
}
// GROUPS: 32, or 16 where group i stands for the sum of i and i + 16 already.
template <int GROUPS>
__device__ __forceinline__ float ln_total(uint32_t buf, int lane) {
  float g[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(g[i])
                 : "r"(buf + static_cast<uint32_t>(i * 32 + lane) * 4u) : "memory");
    if constexpr (GROUPS == 32) {
      float h;
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(h)
                   : "r"(buf + static_cast<uint32_t>((i + 16) * 32 + lane) * 4u) : "memory");
      g[i] += h;
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) g[i] += g[i + o];
  return g[0];
}
__device__ __forceinline__ uint32_t ln_pair(uint32_t w, float mean, float rstd) {
  return pack_bf16((bf16_lo(w) - mean) * rstd, (bf16_hi(w) - mean) * rstd);
}

// mbar_wait with the (bounded) polling loop out of line, for the epilogue warps: the phase has
// usually completed, and rare code left inline in their loop costs registers and schedule.
__device__ __noinline__ bool gemm_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                            int code) {
  return mbar_wait(bar, parity, abort_flag, code);
}
__device__ __forceinline__ bool gemm_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int code) {
  if (mbar_try_wait(bar, parity)) return true;
  return gemm_wait_slow(bar, parity, abort_flag, code);
}

// Requests one warp's eight rows [r0, r0 + 8) of the rotary table part of a lane quarter (the 32
// output rows from m_warp) into shared memory at `tab`, 128 bytes a row, 16-byte chunks swizzled over the
// banks: one cp.async group. one_row: every row reads the same line, through L1.
__device__ __forceinline__ void gemm_fetch_table(const GemmParams& p, int m_warp, int r0, uint32_t tab, bool one_row) {
  const int lane = threadIdx.x & 31;
  const int half = p.head_dim >> 1;
  const int r = r0 + (lane >> 2);           // a row's chunks: four lanes, two each
  const int m = min(m_warp + r, p.M - 1);
  const uint32_t* src = p.rope_cs + (static_cast<long long>(m / p.tokens_per_tile) * p.hw + m % p.hw) * half;
#pragma unroll
  for (int ch = lane & 3; ch < 8; ch += 4)
    if (ch * 4 < half) {
      const uint32_t dst = tab + r * 128u + ((ch ^ (r & 7)) << 4);
      if (one_row) asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + ch * 4) : "memory");
      else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + ch * 4) : "memory");
    }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int BN, int EPI, bool PAIR>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmOut,
                    const __grid_constant__ CUtensorMap tmAux, const __grid_constant__ CUtensorMap tmLn,
                    const GemmParams p) {
  constexpr bool LN = EPI == EPI_RESIDUAL_LN;
  constexpr bool TABLE = EPI == EPI_QKV_ROPE || EPI == EPI_QKV_NORM;
  // The accumulator as matrix fragments (see above) or a row per lane. Fragments / rows, microseconds: residual
  // 262144 x 512, K = 512 115 / 121, 442368 x 256, K = 256 91 / 101; GELU 442368 x 1024, K = 256 231 / 267, 103000 x
  // 1536, K = 384 103 / 110, level from K = 512 on; q/k norm and rotation 262144 x 1536, K = 512 377 / 383, 98304
  // x 2304, K = 768 243 / 267, 103000 x 1152, K = 384 150 / 167. The other way: rotation alone 346 / 338, 252 / 246,
  // 121 / 120 (without the norm's code in the kernel rows take 324, 245, 121); bias alone 295 / 291, 171 / 166.
  constexpr bool FRAG = EPI != EPI_BIAS && EPI != EPI_QKV_ROPE && !LN;
  using S = GemmSmem<BN, PAIR, TABLE || LN>;
  // PAIR: this CTA is rank 0 or 1 of a cluster of two that computes 256 x BN tiles together
  const uint32_t pair_rank = PAIR ? cluster_ctarank() : 0u;
  const int unit = PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int n_units = PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  constexpr int TILE_M = PAIR ? 2 * GEMM_BM : GEMM_BM;
  constexpr bool HAS_AUX = (EPI == EPI_RESIDUAL || EPI == EPI_GATE || LN);
  // Epilogues without an operand to prefetch wait for the staging box as late as possible.
  constexpr bool LATE_WAIT = !HAS_AUX;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

  const uint32_t bar_base = smem_base + S::BAR_OFF;
  // barriers (8 bytes each): full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], aux[warps]; the QKV
  // epilogue has no aux operand and uses four of those for its table, one per lane quarter
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (S::STAGES + s); };
  auto accf_bar = [&](int b) { return bar_base + 8u * (2 * S::STAGES + b); };
  auto acce_bar = [&](int b) { return bar_base + 8u * (2 * S::STAGES + 2 + b); };
  auto aux_bar = [&](int w) { return bar_base + 8u * (2 * S::STAGES + 4 + w); };
  [[maybe_unused]] auto tabf_bar = [&](int q) { return aux_bar(q); };
  uint8_t* tail = smem_gen + S::BAR_OFF + 8 * (2 * S::STAGES + 4 + GEMM_EPI_WARPS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8);
  // one per lane quarter
  [[maybe_unused]] const uint32_t ln_bar0 = bar_base + 8u * (2 * S::STAGES + 4 + GEMM_EPI_WARPS) + 16u;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  const int tiles_m = (p.M + TILE_M - 1) / TILE_M;
  const int tiles_n = (p.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  // Tile t of the order (row block, then column tile), walked t = unit, unit + n_units, ...: units side by
  // side share their row block's A and their column tile's W while both are on their way through L2
  // (one contiguous range per unit, A kept in shared memory over a row block's column tiles, ran 5 %
  // slower at K = 512, and 10 to 30 % at K = 2048 and 3072 without the keeping). Where the last column
  // tile is narrower, the column order turns with every round, so that no unit gets only wide ones.
  const bool ragged = p.N % BN != 0;
  auto tile_of = [&](int t, int& mt, int& jt) {
    mt = t / tiles_n;
    jt = t - mt * tiles_n;
    if (ragged) jt = (jt + static_cast<int>(static_cast<long long>(mt) * tiles_n / n_units)) % tiles_n;
  };
  // columns of column tile j that the MMA computes (the last tile may be narrower)
  auto tile_cols = [&](int j) { return min(BN, (p.N - j * BN + 31) / 32 * 32); };
  const int num_kb = (p.K + GEMM_BK - 1) / GEMM_BK;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accf_bar(b), 1);
      mbar_init(acce_bar(b), PAIR ? 2 * GEMM_EPI_WARPS : GEMM_EPI_WARPS);
    }
    // (a rotary table part is written by the four warps of a lane quarter)
    for (int w = 0; w < GEMM_EPI_WARPS; ++w) mbar_init(aux_bar(w), TABLE ? 4 : 1);
    if constexpr (LN)
      for (int q = 0; q < 4; ++q) mbar_init(ln_bar0 + 8u * q, 4);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // the partner's barriers exist before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  chain_begin();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = unit; t < num_tiles && ok; t += n_units) {
        int mt, jt;
        tile_of(t, mt, jt);
        const int m0 = mt * TILE_M + static_cast<int>(pair_rank) * GEMM_BM;
        // the pair's CTAs supply half of the MMA's columns each
        const int n0 = jt * BN + (PAIR ? static_cast<int>(pair_rank) * (tile_cols(jt) / 2) : 0);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, ST_TIMEOUT_PRODUCER)) {
            ok = false;
            break;
          }
          const uint32_t a_dst = smem_base + stage * S::STAGE_BYTES;
          const uint32_t b_dst = a_dst + S::A_BYTES;
          if constexpr (PAIR) {
            // both CTAs' loads complete on the FIRST CTA's stage barrier (it issues the MMAs);
            // that CTA's producer announces the bytes of both (a transaction count may run
            // ahead of its announcement within a phase)
            const uint32_t fb = map_to_cta(full_bar(stage), 0);
            if (pair_rank == 0) mbar_expect_tx(full_bar(stage), 2 * S::STAGE_BYTES);
            tma_load_2d_pair(a_dst, &tmA, kb * GEMM_BK, m0, fb);
            tma_load_2d_pair(b_dst, &tmB, kb * GEMM_BK, n0, fb);
          } else {
            mbar_expect_tx(full_bar(stage), S::STAGE_BYTES);
            tma_load_2d(a_dst, &tmA, kb * GEMM_BK, m0, full_bar(stage));
            tma_load_2d(b_dst, &tmB, kb * GEMM_BK, n0, full_bar(stage));
          }
          if (++stage == S::STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        // Give loads already in flight time to land before the CTA retires.
#pragma unroll 1
        for (int i = 0; i < 2000; ++i) __nanosleep(100);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (pair_rank == 0 && elect_one()) {
      constexpr uint32_t idesc0 = umma_idesc_bf16(TILE_M, 0, false, false);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int t = unit; t < num_tiles && ok; t += n_units, ++it) {
        int mt, jt;
        tile_of(t, mt, jt);
        const uint32_t idesc = idesc0 | (static_cast<uint32_t>(tile_cols(jt) >> 3) << 17);
        const int buf = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1u;
        if (!mbar_wait(acce_bar(buf), acc_phase ^ 1u, abort_flag, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, ST_TIMEOUT_MMA)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_src = smem_base + stage * S::STAGE_BYTES;
          const uint32_t b_src = a_src + S::A_BYTES;
          const uint64_t adesc = umma_smem_desc_sw128(a_src);
          const uint64_t bdesc = umma_smem_desc_sw128(b_src);
#pragma unroll
          for (int k = 0; k < GEMM_BK / 16; ++k) {
            // advance 16 bf16 = 32 bytes along K inside the 128-byte swizzle span
            if constexpr (PAIR)
              umma_ss_pair(d_tmem, adesc + 2u * k, bdesc + 2u * k, idesc, (kb | k) != 0 ? 1u : 0u);
            else
              umma_ss(d_tmem, adesc + 2u * k, bdesc + 2u * k, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          if constexpr (PAIR) umma_commit_pair(empty_bar(stage)); else umma_commit(empty_bar(stage));
          if (++stage == S::STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok) {
          if constexpr (PAIR) umma_commit_pair(accf_bar(buf)); else umma_commit(accf_bar(buf));
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps
    // Each warp owns 32 output rows (its TMEM lane quarter) x BN/4 columns of the tile and
    // walks them in 32-column sub-chunks of two 16-column groups: TMEM -> registers -> math ->
    // 64-byte-swizzled staging box (32 rows x 32 columns) in shared memory -> TMA store
    // (clipped at the matrix edge by the tensor map). The residual / gated operand of a
    // sub-chunk is TMA-loaded into the same staging box beforehand.
    const int e = warp - 2;
    const int quarter = warp & 3;            // TMEM lane quarter this warp may read
    const int cg = e >> 2;                   // which quarter of the BN columns
    // (the q/k norm takes a head to a warp; in narrow tiles the warps of the upper quarters have no columns)
    constexpr int WARP_COLS = EPI == EPI_QKV_NORM ? 64 : BN < 128 ? 32 : BN / 4;
    constexpr int NSUB = WARP_COLS / 32;
    const uint32_t stage_s = smem_base + S::STAGING_OFF + e * S::STAGING_BYTES;
    [[maybe_unused]] const uint32_t my_row_s = stage_s + lane * 64;   // (row form: this lane's row, its swizzle)
    [[maybe_unused]] const uint32_t sw = static_cast<uint32_t>((lane >> 1) & 3);
    // this lane's row of the four 8 x 8 pieces (rows 16 hf + {0, 8}, columns 16 q + {0, 8}) of a staging box: 64-byte
    // rows, 64-byte swizzle
    const uint32_t box_row = stage_s + static_cast<uint32_t>(((lane >> 3) & 1) * 8 + (lane & 7)) * 64u;
    auto box_addr = [&](int hf, int q) -> uint32_t {
      return box_row + hf * 1024u +
             ((static_cast<uint32_t>(2 * q + (lane >> 4)) ^ static_cast<uint32_t>((lane >> 1) & 3)) << 4);
    };
    const uint32_t acce_remote0 = PAIR ? map_to_cta(acce_bar(0), 0) : 0u;
    const uint32_t acce_remote1 = PAIR ? map_to_cta(acce_bar(1), 0) : 0u;
    uint32_t aux_phase = 0;
    int it = 0;
    bool ok = true;
    // EPI_QKV_ROPE: the rotation table rows (one 4-byte (cos, sin) pair per channel pair of a head: 128
    // bytes for head_dim 64) are the same for every q / k head. The four warps of a lane quarter bring
    // the 32 rows of a tile into shared memory together, eight each, while they work on the tile
    // before; a row is then read by its lane, 16 bytes at a time. (Read from global memory, 32
    // lanes with 32 different rows take 32 L1 cycles per 16 bytes, over a tile as many as its whole
    // matrix work: 262144 x 1536, K = 512 took 0.50 ms instead of 0.45.)
    const uint32_t tab_quarter = smem_base + S::TABLE_OFF + static_cast<uint32_t>(quarter) * 32u * 128u;
    const bool rope = TABLE && p.rope_cs != nullptr;
    // (a table of one row - the identity that a q/k norm without rotation runs with - is fetched into both
    // buffers once: every SM asking L2 for the same line, tile after tile, made QKV of 393216 x 256 take
    // 0.74 ms instead of 0.27)
    const bool one_row = p.hw == 1 && p.tokens_per_tile >= p.M;
    auto tile_rows = [&](int t) {        // first output row of this warp's quarter in tile t
      int mt, jt;
      tile_of(t, mt, jt);
      return mt * TILE_M + static_cast<int>(pair_rank) * GEMM_BM + quarter * 32;
    };
    // EPI_RESIDUAL_LN: one tile (N <= BN: a tile has whole rows)
    [[maybe_unused]] auto ln_tile = [&](int it_, int m_warp, int n_warp0) -> bool {
      const int buf = it_ & 1;
      const uint32_t sums = smem_base + S::TABLE_OFF + static_cast<uint32_t>(quarter) * 4096u, squares = sums + 16384u;
      const uint32_t ln_bar = ln_bar0 + 8u * quarter;
      uint32_t w[NSUB][16];
#pragma unroll
      for (int c = 0; c < NSUB; ++c) {
        const int n0 = n_warp0 + c * 32;
        const bool live = n0 < p.N && m_warp < p.M;           // warp-uniform
        if (live && elect_one()) {
          tma_store_wait_read0();
          mbar_expect_tx(aux_bar(e), S::STAGING_BYTES);
          tma_load_2d(stage_s, &tmAux, n0, m_warp, aux_bar(e));
        }
        if (c == 0) {
          if (!gemm_wait(accf_bar(buf), (it_ >> 1) & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
          tc_fence_after();
        }
        if (live) {
          if (!gemm_wait(aux_bar(e), aux_phase, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
          aux_phase ^= 1u;
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t r[16];
          if (live) {
            tmem_ld_32x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                              static_cast<uint32_t>(buf * BN + cg * WARP_COLS + c * 32 + 16 * g), r);
            tmem_ld_wait();
          }
          if (g == 1 && c == NSUB - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              if constexpr (PAIR) mbar_arrive_cluster(buf ? acce_remote1 : acce_remote0);
              else mbar_arrive(acce_bar(buf));
            }
          }
          if (live) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const uint32_t addr = my_row_s + ((static_cast<uint32_t>(2 * g + q) ^ sw) << 4);
              uint32_t ax[4];
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(ax[0]), "=r"(ax[1]), "=r"(ax[2]), "=r"(ax[3]) : "r"(addr) : "memory");
#pragma unroll
              for (int h = 0; h < 2; ++h) {       // four columns: N is a multiple of 64
                float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
                if (p.bias != nullptr)
                  b4 = __ldg(reinterpret_cast<const float4*>(p.bias + n0 + 16 * g + 8 * q + 4 * h));
                const int k = 8 * q + 4 * h;
                w[c][8 * g + 4 * q + 2 * h] = pack_bf16(__uint_as_float(r[k]) + b4.x + bf16_lo(ax[2 * h]),
                                                        __uint_as_float(r[k + 1]) + b4.y + bf16_hi(ax[2 * h]));
                w[c][8 * g + 4 * q + 2 * h + 1] = pack_bf16(__uint_as_float(r[k + 2]) + b4.z + bf16_lo(ax[2 * h + 1]),
                                                            __uint_as_float(r[k + 3]) + b4.w + bf16_hi(ax[2 * h + 1]));
              }
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[c][8 * g + 4 * q]),
                           "r"(w[c][8 * g + 4 * q + 1]), "r"(w[c][8 * g + 4 * q + 2]), "r"(w[c][8 * g + 4 * q + 3])
                           : "memory");
            }
          }
        }
        if (live) {
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            tma_store_2d(&tmOut, stage_s, n0, m_warp);
            tma_store_commit();
          }
        }
        if (m_warp < p.M) {                        // (columns behind N count as zero)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ln_put(sums, cg * (WARP_COLS / 8) + 4 * c + k, lane, live ? ln_group_sum(&w[c][4 * k]) : 0.f);
        }
      }
      if (m_warp >= p.M) return true;              // all four warps of the quarter
      __syncwarp();
      if (lane == 0) mbar_arrive(ln_bar);
      if (!gemm_wait(ln_bar, 0u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
      const float mean = ln_total<BN / 8>(sums, lane) / static_cast<float>(p.N);
#pragma unroll
      for (int c = 0; c < NSUB; ++c)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ln_put(squares, cg * (WARP_COLS / 8) + 4 * c + k, lane,
                 n_warp0 + 32 * c < p.N ? ln_group_squares(&w[c][4 * k], mean) : 0.f);
      __syncwarp();
      if (lane == 0) mbar_arrive(ln_bar);
      if (!gemm_wait(ln_bar, 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
      const float rstd = rsqrtf(ln_total<BN / 8>(squares, lane) / static_cast<float>(p.N) + p.ln_eps);
#pragma unroll
      for (int c = 0; c < NSUB; ++c) {
        if (n_warp0 + 32 * c >= p.N) break;
        if (elect_one()) tma_store_wait_read0();
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t addr = my_row_s + ((static_cast<uint32_t>(q) ^ sw) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(ln_pair(w[c][4 * q], mean, rstd)),
                       "r"(ln_pair(w[c][4 * q + 1], mean, rstd)), "r"(ln_pair(w[c][4 * q + 2], mean, rstd)),
                       "r"(ln_pair(w[c][4 * q + 3], mean, rstd)) : "memory");
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (elect_one()) {
          tma_store_2d(&tmLn, stage_s, n_warp0 + 32 * c, m_warp);
          tma_store_commit();
        }
      }
      return true;
    };
    if (rope && unit < num_tiles) gemm_fetch_table(p, tile_rows(unit), cg * 8, tab_quarter, one_row);
    for (int t = unit; t < num_tiles && ok; t += n_units, ++it) {
      const int buf = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1u;
      int mt, jt;
      tile_of(t, mt, jt);
      const int m0 = mt * TILE_M + static_cast<int>(pair_rank) * GEMM_BM;
      const int n_tile0 = jt * BN;
      const int m_warp = m0 + quarter * 32;
      const int n_warp0 = n_tile0 + cg * WARP_COLS;
      [[maybe_unused]] uint32_t tab_base = 0;   // the tile's table rows of this lane quarter
      if constexpr (TABLE) {
        if (rope) {
          tab_base = tab_quarter + static_cast<uint32_t>(buf) * (GEMM_BM * 128u);
          // this warp's part of the tile's table has arrived; when all four warps say so, the whole has,
          // and none of them reads the tile before's any more: the next tile's goes there
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(tabf_bar(quarter));
          if (!gemm_wait(tabf_bar(quarter), it & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) {
            ok = false;
            break;
          }
          if (t + n_units < num_tiles && !(one_row && it != 0))
            gemm_fetch_table(p, tile_rows(t + n_units), cg * 8,
                             tab_quarter + static_cast<uint32_t>(buf ^ 1) * (GEMM_BM * 128u), one_row);
        }
      }
      if constexpr (LN) {
        if (!ln_tile(it, m_warp, n_warp0)) {
          ok = false;
          break;
        }
        continue;
      }
      bool acc_ready = false;
      float qk_scale[4] = {1.f, 1.f, 1.f, 1.f};   // RMS factors of this lane's four rows
      [[maybe_unused]] float2 row_scale = make_float2(1.f, 1.f);   // of row `lane`, for the warp's two sub-chunks
#pragma unroll 1
      for (int c = 0; c < NSUB; ++c) {
        const int n0 = n_warp0 + c * 32;
        const bool chunk_live = (n0 < p.N) && (m_warp < p.M) && cg * WARP_COLS < BN;   // warp-uniform
        if constexpr (FRAG) {
          uint64_t bias[4];
          gemm_lane_bias(p, n0, lane, bias);
          if constexpr (!LATE_WAIT) {
            if (chunk_live) {
              // staging box free again? (previous TMA store has finished reading it) - a
              // residual / gated operand is fetched into it right away
              if (elect_one()) tma_store_wait_read0();
              __syncwarp();
              if constexpr (HAS_AUX) {
                if (elect_one()) {
                  mbar_expect_tx(aux_bar(e), S::STAGING_BYTES);
                  tma_load_2d(stage_s, &tmAux, n0, m_warp, aux_bar(e));
                }
              }
            }
          }
          if (!acc_ready) {
            if (!gemm_wait(accf_bar(buf), acc_phase, abort_flag, ST_TIMEOUT_EPILOGUE)) {
              ok = false;
              break;
            }
            tc_fence_after();
            acc_ready = true;
          }
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                 static_cast<uint32_t>(buf * BN + cg * WARP_COLS + c * 32);
          const bool rotate = rope && n0 < p.rope_cols;           // warp-uniform
          if constexpr (EPI == EPI_QKV_NORM) {
            // q/k norm: one extra pass over the warp's columns with a row per lane (a row's squares are then summed in
            // column order by one lane); the factors of this lane's fragment rows come from the lanes that have them
            if (c == 0 && rotate && chunk_live)
              row_scale = gemm_qk_norm_scales<NSUB>(taddr, p.bias, n_warp0, p.N, lane, p.head_dim, p.qk_eps);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              qk_scale[k] = __shfl_sync(0xffffffffu, c == 0 ? row_scale.x : row_scale.y, 8 * k + (lane >> 2));
          }
          if constexpr (HAS_AUX) {
            if (chunk_live) {
              if (!gemm_wait(aux_bar(e), aux_phase, abort_flag, ST_TIMEOUT_EPILOGUE)) {
                ok = false;
                break;
              }
              aux_phase ^= 1u;
            }
          }
          uint32_t acc[2][16];
          if (chunk_live) {
            tmem_ld_16x256_x4(taddr, acc[0]);
            tmem_ld_16x256_x4(taddr + (16u << 16), acc[1]);
            tmem_ld_wait();
          }
          if (c == NSUB - 1) {
            // the accumulator is in registers (or not needed): hand it back to the MMA warp
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              if constexpr (PAIR) mbar_arrive_cluster(buf ? acce_remote1 : acce_remote0);
              else mbar_arrive(acce_bar(buf));
            }
          }
          if (chunk_live) {
            // head_dim 64: the 32-column sub-chunks of a head use table pairs [0, 16) and [16, 32); head_dim
            // 32: each sub-chunk is a whole head and uses pairs [0, 16). The table's 16-byte pieces hold four pairs.
            [[maybe_unused]] const uint32_t piece0 = p.head_dim == 64 ? static_cast<uint32_t>(n0 & 63) >> 3 : 0u;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              uint32_t aux[8], w[8];
              if constexpr (HAS_AUX) {
#pragma unroll
                for (int q = 0; q < 2; ++q) ldmatrix_x4(box_addr(hf, q), &aux[4 * q]);
              }
              // (a pair of the table is four bytes, a piece four pairs: the words of an 8 x 8 matrix of halves)
              uint32_t cs[8];
              if constexpr (TABLE) {
                if (rotate) {
#pragma unroll
                  for (int q = 0; q < 2; ++q)
                    ldmatrix_x4(tab_base + (16 * hf + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128u +
                                    (((piece0 + 2 * q + (lane >> 4)) ^ (lane & 7u)) << 4),
                                &cs[4 * q]);
                }
              }
#pragma unroll
              for (int i = 0; i < 8; ++i) {       // columns 8 (i / 2), row + 8 (i % 2)
                w[i] = gemm_epilogue_pair<EPI>(fadd2(pack2u(acc[hf][2 * i], acc[hf][2 * i + 1]), bias[i >> 1]),
                                               HAS_AUX ? aux[i] : 0u, rotate, TABLE ? cs[i] : 0u,
                                               qk_scale[2 * hf + (i & 1)]);
              }
              if constexpr (LATE_WAIT) {
                if (hf == 0) {
                  // the previous sub-chunk's TMA store must have finished reading the staging
                  // box before it is overwritten; waiting only now lets that drain overlap with
                  // the TMEM load and the arithmetic above
                  if (elect_one()) tma_store_wait_read0();
                  __syncwarp();
                }
              }
#pragma unroll
              for (int q = 0; q < 2; ++q) stmatrix_x4(box_addr(hf, q), &w[4 * q]);
            }
          }
        } else {
          float b_lane = 0.f;
          if (p.bias != nullptr && n0 + lane < p.N) b_lane = __ldg(p.bias + n0 + lane);
          if (!acc_ready) {
            if (!gemm_wait(accf_bar(buf), acc_phase, abort_flag, ST_TIMEOUT_EPILOGUE)) {
              ok = false;
              break;
            }
            tc_fence_after();
            acc_ready = true;
          }
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                 static_cast<uint32_t>(buf * BN + cg * WARP_COLS + c * 32);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            // head_dim 64: the 32-column sub-chunks of a head use table pairs [0,16) and
            // [16,32); head_dim 32: each sub-chunk is a whole head and uses pairs [0,16).
            // The table words are requested before the TMEM load so that the two latencies overlap.
            const bool rotate = rope && n0 < p.rope_cols;
            uint32_t cs[8];
            if constexpr (EPI == EPI_QKV_ROPE) {
              if (rotate && chunk_live) {
                const int pair0 = ((p.head_dim == 64) ? (n0 & 63) >> 1 : 0) + 8 * g;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                  const uint32_t addr =
                      tab_base + lane * 128u + ((static_cast<uint32_t>((pair0 >> 2) + q) ^ (lane & 7u)) << 4);
                  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                               : "=r"(cs[4 * q]), "=r"(cs[4 * q + 1]), "=r"(cs[4 * q + 2]), "=r"(cs[4 * q + 3])
                               : "r"(addr) : "memory");
                }
              }
            }
            uint32_t r[16];
            if (chunk_live) {
              tmem_ld_32x16(taddr + 16 * g, r);
              tmem_ld_wait();
            }
            if (g == 1 && c == NSUB - 1) {
              // the accumulator is in registers (or not needed): hand it back to the MMA warp
              tc_fence_before();
              __syncwarp();
              if (lane == 0) {
                if constexpr (PAIR) mbar_arrive_cluster(buf ? acce_remote1 : acce_remote0);
                else mbar_arrive(acce_bar(buf));
              }
            }
            if (chunk_live) {
              float v[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
              // (the bias group is read directly when all its 16 columns exist; p.bias is
              // 16-byte aligned and n0 a multiple of 32)
              const float* bias16 = (p.bias != nullptr && n0 + 16 * g + 16 <= p.N)
                                        ? p.bias + n0 + 16 * g : nullptr;
              gemm_epilogue_16<EPI>(v, rotate, b_lane, 16 * g, cs, p, bias16);
              if (g == 0) {
                // the previous sub-chunk's TMA store must have finished reading the staging
                // box before it is overwritten; waiting only now lets that drain overlap with
                // the TMEM load and the arithmetic above
                if (elect_one()) tma_store_wait_read0();
                __syncwarp();
              }
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const uint32_t addr = my_row_s + ((static_cast<uint32_t>(2 * g + q) ^ sw) << 4);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
                             "r"(pack_bf16(v[8 * q], v[8 * q + 1])),
                             "r"(pack_bf16(v[8 * q + 2], v[8 * q + 3])),
                             "r"(pack_bf16(v[8 * q + 4], v[8 * q + 5])),
                             "r"(pack_bf16(v[8 * q + 6], v[8 * q + 7]))
                             : "memory");
              }
            }
          }
        }
        if (!chunk_live) continue;
        fence_proxy_async_smem();
        __syncwarp();
        if (elect_one()) {
          tma_store_2d(&tmOut, stage_s, n0, gemm_out_row(m_warp, p));
          tma_store_commit();
        }
      }
    }
    if (elect_one()) tma_store_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // no signal may reach a CTA that has already left
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// Host launcher. A: [M,K] bf16 row-major with row stride lda (elements); W: [N,K] bf16
// row-major with row stride ldw. Returns 0, or a negative argument error / CUDA error code.
template <int BN, int EPI, bool PAIR>
inline int launch_gemm_t(const __nv_bfloat16* A, long long lda, const __nv_bfloat16* W,
                         long long ldw, const GemmParams& p, int sm_count, cudaStream_t stream,
                         __nv_bfloat16* ln_out = nullptr, long long ldln = 0) {
  CUtensorMap tmA, tmB;
  {
    uint64_t dims[2] = {static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.M)};
    uint64_t str[1] = {static_cast<uint64_t>(lda) * 2};
    uint32_t box[2] = {GEMM_BK, GEMM_BM};
    if (make_tmap_bf16(&tmA, A, 2, dims, str, box) != 0) return -20;
  }
  {
    uint64_t dims[2] = {static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.N)};
    uint64_t str[1] = {static_cast<uint64_t>(ldw) * 2};
    uint32_t box[2] = {GEMM_BK, static_cast<uint32_t>(PAIR ? BN / 2 : BN)};
    if (make_tmap_bf16(&tmB, W, 2, dims, str, box) != 0) return -21;
  }
  CUtensorMap tmOut, tmAux, tmLn;
  {
    uint64_t dims[2] = {static_cast<uint64_t>(p.N), static_cast<uint64_t>(p.M)};
    uint64_t str[1] = {static_cast<uint64_t>(p.ldo) * 2};
    uint32_t box[2] = {32, 32};
    uint64_t odims[2] = {dims[0], dims[1]};
    if (p.pad_T > 0) {
      const uint64_t P = static_cast<uint64_t>(p.pad_T + 2 * p.pad_h);
      odims[1] = dims[1] / (static_cast<uint64_t>(p.pad_T) * p.pad_T) * P * P;
    }
    if (make_tmap_bf16(&tmOut, p.out, 2, odims, str, box, TMAP_SWIZZLE_64B) != 0) return -22;
    tmAux = tmOut;
    if (EPI == EPI_RESIDUAL || EPI == EPI_GATE || EPI == EPI_RESIDUAL_LN) {
      uint64_t astr[1] = {static_cast<uint64_t>(p.ldaux) * 2};
      if (make_tmap_bf16(&tmAux, p.aux, 2, dims, astr, box, TMAP_SWIZZLE_64B) != 0) return -23;
    }
    tmLn = tmOut;
    if (EPI == EPI_RESIDUAL_LN) {
      uint64_t lstr[1] = {static_cast<uint64_t>(ldln) * 2};
      if (make_tmap_bf16(&tmLn, ln_out, 2, dims, lstr, box, TMAP_SWIZZLE_64B) != 0) return -25;
    }
  }
  using S = GemmSmem<BN, PAIR, EPI == EPI_QKV_ROPE || EPI == EPI_QKV_NORM || EPI == EPI_RESIDUAL_LN>;
  auto kern = gemm_tcgen05_kernel<BN, EPI, PAIR>;
  static std::atomic<uint64_t> smem_set;
  if (const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), S::TOTAL, smem_set); e != cudaSuccess)
    return -static_cast<int>(e) - 1000;
  if constexpr (PAIR) {
    const int tiles = ((p.M + 2 * GEMM_BM - 1) / (2 * GEMM_BM)) * ((p.N + BN - 1) / BN);
    // A persistent grid must be resident at once: not every SM has a partner for a pair, so the
    // number of clusters that fit is asked for (once per kernel and device), not assumed.
    static std::atomic<int> max_clusters[64];   // per device; concurrent first calls store the same value
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return -24;
    int fit = max_clusters[dev].load(std::memory_order_relaxed);
    if (fit == 0) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(static_cast<unsigned>(sm_count & ~1));
      cfg.blockDim = dim3(GEMM_THREADS);
      cfg.dynamicSmemBytes = S::TOTAL;
      cfg.stream = stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess || fit <= 0) return -24;
      max_clusters[dev].store(fit, std::memory_order_relaxed);
    }
    const int clusters = tiles < fit ? tiles : fit;
    return launch_chained(kern, dim3(static_cast<unsigned>(2 * clusters)), GEMM_THREADS, S::TOTAL, stream, 2,
                          tmA, tmB, tmOut, tmAux, tmLn, p);
  }
  const int tiles = ((p.M + GEMM_BM - 1) / GEMM_BM) * ((p.N + BN - 1) / BN);
  const int grid = tiles < sm_count ? tiles : sm_count;
  return launch_chained(kern, dim3(grid), GEMM_THREADS, S::TOTAL, stream, 1, tmA, tmB, tmOut, tmAux, tmLn, p);
}

template <int EPI>
inline int launch_gemm(const __nv_bfloat16* A, long long lda, const __nv_bfloat16* W, long long ldw,
                       const GemmParams& p, int sm_count, cudaStream_t stream) {
  // CTA pairs share each MMA (less shared-memory and L2 traffic per SM) from 1024 rows on, for every N that
  // one 128-wide tile does not cover; the last column tile is as narrow as it needs to be.
  // Except where the last tile is half one and a tile has two k-blocks at most: it is then all epilogue, the
  // pair's two column tiles of 256 and 128 take turns at unequal lengths, and equal 128-wide tiles of one
  // CTA run faster - as long as A's rows are whole pieces of a line (K = 32, 64, 128), for A is read once
  // per column tile. Microseconds of pairs / of 128-wide tiles, at 1572864, 196608 and 24576 rows:
  //   N = 384: K = 32 309 / 233, 51 / 40, 10.2 / 7.7; K = 64 314 / 231, 45 / 34, 10.0 / 7.3;
  //            K = 128 318 / 293, 47 / 41, 10.6 / 8.3
  //   N = 640: K = 64 487 / 378, 68 / 53, 12.0 / 10.1; K = 128 510 / 483, 69 / 64, 12.8 / 11.6
  //   the other way: K = 8 N = 384 465 / 679, 76 / 85, 13.4 / 14.8; K = 120 395 / 630, 55 / 72, 12.7 / 11.6;
  //            K = 192 372 / 388, 54 / 54, 12.3 / 10.2; N = 448 K = 128 339 / 458, 52 / 65, 11.8 / 12.3
  // And except where the chip is not filled: a launch that is a few turns of the persistent CTAs long costs what its
  // longest CTA does, and a CTA's 128-wide tile is half a pair's share. Times as fast, by turns with 128-wide tiles /
  // with pairs (M = 1024 ... 24576, C = 192 ... 1024, a block's four shapes; least, mean, most):
  //   1 / 1  1.31 1.49 1.72 (1024 x 512, K = 512 8.2 / 5.3 us; 4096 x 512, K = 2048 15.5 / 10.2)
  //   2 / 2  1.18 1.34 1.50 (4096 x 1152, K = 384 with rotation 11.3 / 7.5)
  //   2 / 1, 3 / 2, 4 / 3  up to K = 1024 0.95 1.10 1.27, beyond 0.88 0.98 1.10; N <= 256, K > 512 0.86 - 0.95
  //   4 / 2, 5 / 3  up to K = 1024 0.83 0.93 1.10, beyond 0.8 - 0.9
  // Equal work's operands are twice as many bytes in 128-wide tiles: from K = 512 on a further turn of them takes as
  // long as one of pairs, and with N <= 256 a pair reads A once. The norm of q and k keeps a head to a warp, so that
  // half the warps of a 128-wide tile have none: 1 / 1 1.21 - 1.25 (1536 x 1536, K = 512 9.6 / 7.9), 2 / 2 1.21, 2 / 1
  // and 3 / 2 0.83 - 0.97.
  constexpr bool QKV = EPI == EPI_QKV_ROPE || EPI == EPI_QKV_NORM;
  const int tiles128 = ((p.M + GEMM_BM - 1) / GEMM_BM) * ((p.N + 127) / 128);
  // One tile per SM at most, as narrow as 64: a launch is the latency of one tile, and half as wide a one has half
  // the epilogue and two thirds of the bytes for each k-block. 128-wide tiles / these, microseconds: 256 x 384 with
  // rotation, K = 128 4.4 / 4.2; 1024 x 512, K = 512 5.3 / 4.6; 1024 x 256, K = 1024 6.5 / 5.5; 256 x 1024,
  // K = 4096 13.5 / 11.6; 1.03 - 1.2 times as fast at 64 to 4096 rows, 64 to 1024 channels. A QKV launch is
  // 0.97 - 1.16 times as fast with rotation and 1.16 - 1.35 with the norm, but the attention behind it, whose CTAs come
  // up while it runs, has no room beside it: from half the SMs on a model is slower with these tiles (five blocks
  // on 1512 x 192 204 -> 214 us, eight on 864 x 320 with the norm 302 -> 314).
  if (((p.M + GEMM_BM - 1) / GEMM_BM) * ((p.N + 63) / 64) <= (QKV ? sm_count / 2 : sm_count))
    return launch_gemm_t<64, EPI, false>(A, lda, W, ldw, p, sm_count, stream);
  if (p.M >= 1024 && (p.N > 128 || QKV)) {
    const int pairs = sm_count / 2, tiles_pair = ((p.M + 2 * GEMM_BM - 1) / (2 * GEMM_BM)) * ((p.N + 255) / 256);
    const int turns = (tiles128 + sm_count - 1) / sm_count, turns_pair = (tiles_pair + pairs - 1) / pairs;
    const bool few = turns <= turns_pair || (EPI != EPI_QKV_NORM && turns == turns_pair + 1 && turns <= 4 &&
                                             p.K <= (p.N > 256 ? 1024 : 512));
    if (few || (!QKV && p.N % 256 == 128 && p.K >= 32 && 128 % p.K == 0))
      return launch_gemm_t<128, EPI, false>(A, lda, W, ldw, p, sm_count, stream);
    return launch_gemm_t<256, EPI, true>(A, lda, W, ldw, p, sm_count, stream);
  }
  // Few rows of many columns: the same against 256-wide tiles, as long as there are SMs for twice as many.
  if (tiles128 > sm_count && (QKV || p.N % 256 == 0 || p.N > 512))
    return launch_gemm_t<256, EPI, false>(A, lda, W, ldw, p, sm_count, stream);
  return launch_gemm_t<128, EPI, false>(A, lda, W, ldw, p, sm_count, stream);
}

// y = A W^T + bias + aux and layernorm(y) into ln_out, for whole rows in a tile: N a multiple of 64, at most 256.
// For calls of many rows: pairs of CTAs where one 128-wide tile does not hold a row.
inline int launch_gemm_residual_ln(const __nv_bfloat16* A, long long lda, const __nv_bfloat16* W, long long ldw,
                                   __nv_bfloat16* ln_out, long long ldln, const GemmParams& p, int sm_count,
                                   cudaStream_t stream) {
  if (p.N % 64 != 0 || p.N > 256) return -2;
  if (p.N <= 128) return launch_gemm_t<128, EPI_RESIDUAL_LN, false>(A, lda, W, ldw, p, sm_count, stream, ln_out, ldln);
  return launch_gemm_t<256, EPI_RESIDUAL_LN, true>(A, lda, W, ldw, p, sm_count, stream, ln_out, ldln);
}

}  // namespace strata
