// The MLP of a block in one kernel for narrow models (C = 64, 128, 192, 256 channels):
//
//   y = aux + [gate *] (W2 gelu(W1 x + b1) + b2)        x, aux, gate, y: [M, C] bf16; W1 [H, C], W2 [C, H]
//
// As two GEMMs the hidden rows [M, H] are written and read again: at C = 256, H = 1024 that is 4 of every 5
// bytes the two move, and they are bound by it. Here a CTA keeps 128 rows: the hidden channels are made 128 at a time
// in tensor memory, leave it as bf16 through the GELU into shared memory and are multiplied on from there.
//
//   warp 0      TMA producer: the x tile, and the weights of every chunk of 128 hidden channels through two
//               rings (W1: 128 x 64 boxes, W2: C x 64 boxes); the weights come from L2, 16 C^2 bytes per tile.
//   warp 1      MMA issuer: chunk c + 1 of W1 x goes to one of two accumulators while the epilogue warps work on
//               chunk c, then W2 times the bf16 chunk c accumulates into the output columns.
//   warps 2-17  epilogue: each takes 32 rows x 32 hidden channels of a chunk (bias, GELU, bf16, into the 128-byte
//               swizzled layout the second product reads), and at a tile's end 32 x 32 boxes of the output
//               (bias, gate, aux) through 64-byte-swizzled staging boxes to TMA stores, and for C <= 128, where a
//               warp has one box of a tile, the LayerNorm of the rows besides (the next block begins with it:
//               of one block on 8 x 32 x 32 tokens of 128 channels the two norms that the kernels before them write
//               are 39.6 -> 38.3 us, of three blocks on 19000 220 -> 204; at C = 256 the second box and the
//               wait for the sums cost more than the pass they save, 3.33 -> 3.48 ms in two blocks on 442368).
//
// Every element sees the arithmetic of the two GEMMs - products accumulated over k in the same order, the
// hidden channels rounded to bf16, the output too before it meets a gate - so the results are the same bits.
//
// Tensor memory: two chunk accumulators of 128 columns and the output, for C <= 128 twice: the epilogue warps then
// form two sets that take the chunks in turn (a hidden buffer each), and the GELU of a tile's first chunk comes
// before the last tile's output is read, which hides the last product.
// Bound: C <= 128 by the epilogue warps (tanh on the special-function unit alone: 128 x 512 per tile take
// 4096 cycles at C = 128, the products as many; a tile takes 11000), C = 256 by shared memory (operands,
// weights coming in and the hidden chunk: 1.5 times what it moves in the products' own time) and the same warps.
// 442368 rows, one call from a cold L2 (back to back: at the rule below), two GEMMs -> this kernel: C = 64 132 -> 80
// us, 128 232 -> 145, 192 345 -> 301, 256 480 -> 412; with the gated residual of the pixel blocks, which was a third
// kernel, C = 128 296 -> 180.
#pragma once
#include "gemm_tcgen05.cuh"

namespace strata {

struct MlpParams {
  int M, H;
  const float* b1;              // [H] or nullptr
  const float* b2;              // [C] or nullptr
  const __nv_bfloat16* aux;     // [M, C] or nullptr
  long long ldaux;
  const __nv_bfloat16* gate;    // [M, C] or nullptr: the output is rounded to bf16 and multiplied by it
  long long ldgate;
  __nv_bfloat16* ln_out;        // [M, C] or nullptr: layernorm(y), for C = 64 and 128 (may be x)
  long long ldln;
  float ln_eps;
};

constexpr int MLP_CHUNK = 128;             // hidden channels of a chunk
constexpr int MLP_MAX_C = 256;

template <int C, bool LN>
struct MlpSmem {
  static constexpr bool AHEAD = C <= 128;                        // see the top: two outputs, staging boxes of their own
  static constexpr int SETS = AHEAD ? 2 : 1;                     // sets of epilogue warps, taking chunks in turn
  static constexpr int KB = C / 64;                              // k-blocks of the first product
  static constexpr int X_BYTES = KB * 128 * 128;
  static constexpr int X_BUFS = 1;
  static constexpr int H_BYTES = 2 * 128 * 128;                  // one chunk, a buffer per set
  static constexpr int W1_BYTES = 128 * 128, W2_BYTES = C * 128; // one stage
  static_assert(!LN || C == 64 || C == 128, "the norm of a tile's rows comes out of one box per warp");
  static constexpr int S1 = C == 256 ? 4 : 3, S2 = C == 256 || (C == 128 && LN) ? 2 : 3;
  static constexpr int STAGING_BYTES = 32 * 32 * 2;
  static constexpr int H_OFF = X_BUFS * X_BYTES;
  static constexpr int W1_OFF = H_OFF + SETS * H_BYTES;
  static constexpr int W2_OFF = W1_OFF + S1 * W1_BYTES;
  static constexpr int STAGING_OFF = AHEAD ? W2_OFF + S2 * W2_BYTES : H_OFF;
  // LN: sums over 8 columns of every row, for the mean and the variance: [quarter][16 groups][32 rows] each
  static constexpr int LN_OFF = W2_OFF + S2 * W2_BYTES + (AHEAD ? GEMM_EPI_WARPS * STAGING_BYTES : 0);
  static constexpr int BAR_OFF = LN_OFF + (LN ? 2 * 4 * 16 * 32 * 4 : 0);
  static constexpr int TOTAL = BAR_OFF + 512 + 1024;             // + alignment slack
  static constexpr int OUT_COL = 256, OUT_BUFS = AHEAD ? 2 : 1, OUT_STRIDE = 128;
  // Warps that read a tile's output: those whose box of 32 columns begins below C (16 warps, four boxes side by side).
  static constexpr int OUT_READERS = C < 128 ? 4 * (C / 32) : GEMM_EPI_WARPS;
  static_assert(GEMM_EPI_WARPS * STAGING_BYTES <= H_BYTES, "the staging boxes fit the hidden chunk's buffer");
  static_assert(TOTAL <= 232448, "shared memory of an SM");
};

template <int C, bool LN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
mlp_tcgen05_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW1,
                   const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmOut,
                   const __grid_constant__ CUtensorMap tmAux, const __grid_constant__ CUtensorMap tmLn,
                   const MlpParams p) {
  using S = MlpSmem<C, LN>;
  constexpr bool AHEAD = S::AHEAD;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar = smem_base + S::BAR_OFF;
  const uint32_t x_full = bar, x_empty = bar + 8u;
  auto w1_full = [&](int s) { return bar + 32u + 8u * s; };
  auto w1_empty = [&](int s) { return bar + 64u + 8u * s; };
  auto w2_full = [&](int s) { return bar + 96u + 8u * s; };
  auto w2_empty = [&](int s) { return bar + 120u + 8u * s; };
  auto acc_full = [&](int b) { return bar + 144u + 8u * b; };
  auto acc_free = [&](int b) { return bar + 160u + 8u * b; };
  auto out_full = [&](int b) { return bar + 176u + 8u * b; };
  auto out_free = [&](int b) { return bar + 192u + 8u * b; };
  auto h_full = [&](int b) { return bar + 208u + 8u * b; };
  auto h_empty = [&](int b) { return bar + 224u + 8u * b; };
  const uint32_t staged = bar + 240u;
  auto aux_full = [&](int w) { return bar + 256u + 8u * w; };
  [[maybe_unused]] auto ln_bar = [&](int q) { return bar + 400u + 8u * q; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_gen + S::BAR_OFF + 384);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + S::BAR_OFF + 392);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int tiles = (p.M + 127) / 128;
  const int nj = p.H / MLP_CHUNK;
  const int ctas = static_cast<int>(gridDim.x);
  const int n_my = (tiles - static_cast<int>(blockIdx.x) + ctas - 1) / ctas;
  const int chunks = n_my * nj;              // of this CTA, numbered through its tiles

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW1);
    tma_prefetch_desc(&tmW2);
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_free(b), GEMM_EPI_WARPS / S::SETS);
      mbar_init(h_full(b), GEMM_EPI_WARPS / S::SETS);
      mbar_init(h_empty(b), 1);
      mbar_init(out_full(b), 1);
      mbar_init(out_free(b), S::OUT_READERS);
    }
    for (int s = 0; s < S::S1; ++s) { mbar_init(w1_full(s), 1); mbar_init(w1_empty(s), 1); }
    for (int s = 0; s < S::S2; ++s) { mbar_init(w2_full(s), 1); mbar_init(w2_empty(s), 1); }
    mbar_init(x_full, 1);
    mbar_init(x_empty, 1);
    mbar_init(staged, GEMM_EPI_WARPS);
    for (int w = 0; w < GEMM_EPI_WARPS; ++w) mbar_init(aux_full(w), 1);
    for (int q = 0; q < 4; ++q) mbar_init(ln_bar(q), S::OUT_READERS / 4);   // the warps of a quarter that have columns
    *abort_flag = 0;
    fence_mbar_init();
  }
  if constexpr (LN && C == 64)   // groups that no warp has
    for (int i = threadIdx.x; i < 2 * 4 * 16 * 32; i += GEMM_THREADS)
      *reinterpret_cast<float*>(smem_gen + S::LN_OFF + 4 * i) = 0.f;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  chain_begin();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      bool ok = true;
      int s1 = 0, s2 = 0;
      uint32_t ph1 = 0, ph2 = 0;
      // in the order of use: W1 of chunk c, then W2 of chunk c - 1
      for (int c = 0; c <= chunks && ok; ++c) {
        const int t = c / nj, j = c - t * nj;
        if (c < chunks) {
          if (j == 0) {
            if (!mbar_wait(x_empty, (t & 1u) ^ 1u, abort_flag, ST_TIMEOUT_PRODUCER)) break;
            mbar_expect_tx(x_full, S::X_BYTES);
            const int m0 = (static_cast<int>(blockIdx.x) + t * static_cast<int>(gridDim.x)) * 128;
            for (int kb = 0; kb < S::KB; ++kb)
              tma_load_2d(smem_base + kb * 16384, &tmX, kb * 64, m0, x_full);
          }
          for (int kb = 0; kb < S::KB && ok; ++kb) {
            ok = mbar_wait(w1_empty(s1), ph1 ^ 1u, abort_flag, ST_TIMEOUT_PRODUCER);
            if (!ok) break;
            mbar_expect_tx(w1_full(s1), S::W1_BYTES);
            tma_load_2d(smem_base + S::W1_OFF + s1 * S::W1_BYTES, &tmW1, kb * 64, j * MLP_CHUNK, w1_full(s1));
            if (++s1 == S::S1) { s1 = 0; ph1 ^= 1u; }
          }
        }
        if (c > 0) {
          const int jp = j == 0 ? nj - 1 : j - 1;
          for (int hb = 0; hb < 2 && ok; ++hb) {
            ok = mbar_wait(w2_empty(s2), ph2 ^ 1u, abort_flag, ST_TIMEOUT_PRODUCER);
            if (!ok) break;
            mbar_expect_tx(w2_full(s2), S::W2_BYTES);
            tma_load_2d(smem_base + S::W2_OFF + s2 * S::W2_BYTES, &tmW2, jp * MLP_CHUNK + hb * 64, 0, w2_full(s2));
            if (++s2 == S::S2) { s2 = 0; ph2 ^= 1u; }
          }
        }
      }
      if (*abort_flag)   // loads in flight must land before the CTA retires
#pragma unroll 1
        for (int i = 0; i < 2000; ++i) __nanosleep(100);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc1 = umma_idesc_bf16(128, MLP_CHUNK, false, false);
      constexpr uint32_t idesc2 = umma_idesc_bf16(128, C, false, false);
      int s1 = 0, s2 = 0;
      uint32_t ph1 = 0, ph2 = 0;
      int t1 = 0, j1 = 0;                   // tile and chunk of the next first product
      auto first = [&](int c) -> bool {     // W1 x of chunk c
        if (j1 == 0 && !mbar_wait(x_full, t1 & 1u, abort_flag, ST_TIMEOUT_MMA)) return false;
        if (!mbar_wait(acc_free(c & 1), ((c >> 1) & 1u) ^ 1u, abort_flag, ST_TIMEOUT_MMA)) return false;
        tc_fence_after();
        for (int kb = 0; kb < S::KB; ++kb) {
          if (!mbar_wait(w1_full(s1), ph1, abort_flag, ST_TIMEOUT_MMA)) return false;
          tc_fence_after();
          const uint64_t a = umma_smem_desc_sw128(smem_base + kb * 16384);
          const uint64_t b = umma_smem_desc_sw128(smem_base + S::W1_OFF + s1 * S::W1_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ss(tmem_base + (c & 1) * MLP_CHUNK, a + 2u * k, b + 2u * k, idesc1, (kb | k) != 0 ? 1u : 0u);
          umma_commit(w1_empty(s1));
          if (++s1 == S::S1) { s1 = 0; ph1 ^= 1u; }
        }
        umma_commit(acc_full(c & 1));
        if (++j1 == nj) {                   // the x tile has been read
          umma_commit(x_empty);
          j1 = 0;
          ++t1;
        }
        return true;
      };
      bool ok = chunks > 0 && first(0);
      int t = 0, j = 0;
      for (int c = 0; c < chunks && ok; ++c) {
        if (c + 1 < chunks && !first(c + 1)) break;
        const int ob = AHEAD ? t & 1 : 0;
        if (j == 0 && !mbar_wait(out_free(ob), ((AHEAD ? t >> 1 : t) & 1u) ^ 1u, abort_flag, ST_TIMEOUT_MMA)) break;
        const int hbuf = c % S::SETS;
        if (!mbar_wait(h_full(hbuf), (c / S::SETS) & 1u, abort_flag, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        for (int hb = 0; hb < 2; ++hb) {
          if (!mbar_wait(w2_full(s2), ph2, abort_flag, ST_TIMEOUT_MMA)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a = umma_smem_desc_sw128(smem_base + S::H_OFF + hbuf * S::H_BYTES + hb * 16384);
          const uint64_t b = umma_smem_desc_sw128(smem_base + S::W2_OFF + s2 * S::W2_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ss(tmem_base + S::OUT_COL + ob * S::OUT_STRIDE, a + 2u * k, b + 2u * k, idesc2,
                    (j | hb | k) != 0 ? 1u : 0u);
          umma_commit(w2_empty(s2));
          if (++s2 == S::S2) { s2 = 0; ph2 ^= 1u; }
        }
        if (!ok) break;
        umma_commit(h_empty(hbuf));
        if (++j == nj) {
          umma_commit(out_full(ob));
          j = 0;
          ++t;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps
    const int e = warp - 2;
    const int quarter = warp & 3;            // TMEM lane quarter this warp may read
    constexpr int SETS = S::SETS;
    const int set = SETS == 2 ? e >> 3 : 0;
    const int cg = SETS == 2 ? (e >> 2) & 1 : e >> 2;   // which 32 * SETS hidden channels of a chunk
    const int box0 = (e >> 2) * 32;          // output columns of its (first) box
    const uint32_t lane_taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t stage_s = smem_base + S::STAGING_OFF + e * S::STAGING_BYTES;
    const uint32_t my_row_s = stage_s + lane * 64;
    const uint32_t sw = static_cast<uint32_t>((lane >> 1) & 3);   // 64-byte swizzle of a staging box's row
    // the quarter's rows of the hidden chunk
    const uint32_t h_row0 = smem_base + S::H_OFF + set * S::H_BYTES + quarter * 32 * 128;
    auto tile_row = [&](int t) { return (static_cast<int>(blockIdx.x) + t * ctas) * 128 + quarter * 32; };

    // A chunk's accumulator is read as matrix fragments (lane: rows lane / 4 and + 8, columns 2 (lane % 4) and + 1
    // of every 8): a lane then needs two biases per 8 columns, eight for its 32 channels, which are asked for before
    // the accumulator is ready - with a row per lane all 32, read when they were needed, which cost 16 % at
    // C = 128 - and stmatrix puts the 8 x 8 pieces where the second product wants them.
    const uint32_t st_row = h_row0 + static_cast<uint32_t>(((lane >> 3) & 1) * 8 + (lane & 7)) * 128;
    auto gelu_chunk = [&](int c, int j) -> bool {
      const int buf = c & 1, use = c / SETS;
      uint64_t bias[SETS][4];
#pragma unroll
      for (int pc = 0; pc < SETS; ++pc)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          bias[pc][i] = p.b1 == nullptr ? 0ull
                                        : __ldg(reinterpret_cast<const unsigned long long*>(
                                              p.b1 + j * MLP_CHUNK + (cg * SETS + pc) * 32 + 8 * i + 2 * (lane & 3)));
      if (!gemm_wait(acc_full(buf), (c >> 1) & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
      tc_fence_after();
#pragma unroll
      for (int pc = 0; pc < SETS; ++pc) {    // 32 hidden channels at a time
        const int col = (cg * SETS + pc) * 32;
        uint32_t acc[2][16], h[2][8];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf)
          tmem_ld_16x256_x4(lane_taddr + (static_cast<uint32_t>(16 * hf) << 16) + buf * MLP_CHUNK + col, acc[hf]);
        tmem_ld_wait();
        if (pc == SETS - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_free(buf));
        }
#pragma unroll
        for (int hf = 0; hf < 2; ++hf)
#pragma unroll
          for (int i = 0; i < 8; ++i) {      // columns 8 (i / 2), rows + 8 (i % 2)
            float g0, g1;
            unpack2(gelu_pair(fadd2(pack2u(acc[hf][2 * i], acc[hf][2 * i + 1]), bias[pc][i >> 1])), g0, g1);
            h[hf][i] = pack_bf16(g0, g1);
          }
        // the product of the chunk before that used this buffer has read it
        if (pc == 0 && !gemm_wait(h_empty(set), (use & 1u) ^ 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf)
#pragma unroll
          for (int q = 0; q < 2; ++q) {      // columns 16 q: k-block col / 64, 16-byte pieces (col % 64) / 8 + 2 q, + 1
            const uint32_t piece = static_cast<uint32_t>((col & 32) / 8 + 2 * q + (lane >> 4));
            const uint32_t addr = st_row + hf * 2048 + (col >> 6) * 16384 + ((piece ^ (lane & 7u)) << 4);
            stmatrix_x4(addr, &h[hf][4 * q]);
          }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(h_full(set));
      return true;
    };

    // 64 bytes of this thread's row (a box's columns from n0) of an [M, C] operand
    auto fetch = [&](uint4 (&v)[4], const __nv_bfloat16* base, long long ld, int t, int n0) {
      const long long m = tile_row(t) + lane;
      if (base != nullptr && m < p.M && n0 < C) {
        const uint4* src = reinterpret_cast<const uint4*>(base + m * ld + n0);
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = src[q];
      }
    };
    // AHEAD: aux of a tile's box waits in the staging box, fetched while the tile is computed
    auto fetch_aux_box = [&](int t) {
      if (AHEAD && p.aux != nullptr && box0 < C && tile_row(t) < p.M && elect_one()) {
        tma_store_wait_read0();
        mbar_expect_tx(aux_full(e), S::STAGING_BYTES);
        tma_load_2d(stage_s, &tmAux, box0, tile_row(t), aux_full(e));
      }
    };

    // The tile's output boxes, columns box0 + 128 i. pre: requested ahead of a chunk's work, the first box's gate
    // (AHEAD) or aux.
    int aux_uses = 0;
    auto store_tile = [&](int t, uint4 (&pre)[4]) -> bool {
      const int ob = AHEAD ? t & 1 : 0;
      const int m_warp = tile_row(t);
      bool ready = false;
      [[maybe_unused]] uint32_t keep[16];          // LN: the row's columns of this warp
      [[maybe_unused]] const uint32_t sums = smem_base + S::LN_OFF + static_cast<uint32_t>(quarter) * 2048u;
      [[maybe_unused]] const uint32_t squares = sums + 8192u;
#pragma unroll 1
      for (int n0 = box0; n0 < C; n0 += 128) {
        uint4 aux[4], gate[4];
        if constexpr (AHEAD) {
#pragma unroll
          for (int q = 0; q < 4; ++q) gate[q] = pre[q];
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) aux[q] = pre[q];
          fetch(gate, p.gate, p.ldgate, t, n0);
          fetch(pre, p.aux, p.ldaux, t, n0 + 128);   // the next box's
        }
        if (!ready) {
          if (!gemm_wait(out_full(ob), (AHEAD ? t >> 1 : t) & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
          tc_fence_after();
          ready = true;
        }
        if (m_warp >= p.M) break;             // (warp-uniform; the hand-over below is still owed)
        if constexpr (AHEAD) {
          if (p.aux != nullptr) {
            if (!gemm_wait(aux_full(e), aux_uses & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
            ++aux_uses;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t addr = my_row_s + ((static_cast<uint32_t>(q) ^ sw) << 4);
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(aux[q].x), "=r"(aux[q].y), "=r"(aux[q].z), "=r"(aux[q].w) : "r"(addr) : "memory");
            }
          } else {
            if (elect_one()) tma_store_wait_read0();
            __syncwarp();
          }
        } else {
          if (elect_one()) tma_store_wait_read0();   // the staging box has been read
          __syncwarp();
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t acc[16];
          tmem_ld_32x16(lane_taddr + S::OUT_COL + ob * S::OUT_STRIDE + n0 + 16 * g, acc);
          tmem_ld_wait();
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(acc[i]);
          if (p.b2 != nullptr) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 b4 = __ldg(reinterpret_cast<const float4*>(p.b2 + n0 + 16 * g) + q);
              v[4 * q] += b4.x; v[4 * q + 1] += b4.y; v[4 * q + 2] += b4.z; v[4 * q + 3] += b4.w;
            }
          }
          if (p.aux != nullptr) {
            const uint32_t ax[8] = {aux[2 * g].x, aux[2 * g].y, aux[2 * g].z, aux[2 * g].w,
                                    aux[2 * g + 1].x, aux[2 * g + 1].y, aux[2 * g + 1].z, aux[2 * g + 1].w};
            if (p.gate != nullptr) {
              const uint32_t gt[8] = {gate[2 * g].x, gate[2 * g].y, gate[2 * g].z, gate[2 * g].w,
                                      gate[2 * g + 1].x, gate[2 * g + 1].y, gate[2 * g + 1].z, gate[2 * g + 1].w};
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint32_t yb = pack_bf16(v[2 * i], v[2 * i + 1]);
                v[2 * i] = fmaf(bf16_lo(gt[i]), bf16_lo(yb), bf16_lo(ax[i]));
                v[2 * i + 1] = fmaf(bf16_hi(gt[i]), bf16_hi(yb), bf16_hi(ax[i]));
              }
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                v[2 * i] += bf16_lo(ax[i]);
                v[2 * i + 1] += bf16_hi(ax[i]);
              }
            }
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const uint32_t addr = my_row_s + ((static_cast<uint32_t>(2 * g + q) ^ sw) << 4);
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              w[i] = pack_bf16(v[8 * q + 2 * i], v[8 * q + 2 * i + 1]);
              if constexpr (LN) keep[8 * g + 4 * q + i] = w[i];
            }
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                         "r"(w[3]) : "memory");
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (elect_one()) {
          tma_store_2d(&tmOut, stage_s, n0, m_warp);
          tma_store_commit();
        }
      }
      // The output columns may be accumulated into again. Every arrival follows its warp's own wait for out_full of
      // this tile, so a phase of out_free is made of one tile's readers. A warp without columns waits for nothing here
      // and runs ahead by as many tiles as its chunks let it, so it has no say: else two of its tiles would fill a
      // phase before the readers of the first are done (C = 64, one chunk a tile, from the fourth tile of a CTA on).
      if (box0 < C) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(out_free(ob));
      }
      if constexpr (LN) {
        if (box0 < C && m_warp < p.M) {      // (the whole quarter has rows or none)
#pragma unroll
          for (int k = 0; k < 4; ++k) ln_put(sums, box0 / 8 + k, lane, ln_group_sum(&keep[4 * k]));
          __syncwarp();
          if (lane == 0) mbar_arrive(ln_bar(quarter));
          if (!gemm_wait(ln_bar(quarter), 0u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
          const float mean = ln_total<16>(sums, lane) / static_cast<float>(C);
#pragma unroll
          for (int k = 0; k < 4; ++k) ln_put(squares, box0 / 8 + k, lane, ln_group_squares(&keep[4 * k], mean));
          __syncwarp();
          if (lane == 0) mbar_arrive(ln_bar(quarter));
          if (!gemm_wait(ln_bar(quarter), 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
          const float rstd = rsqrtf(ln_total<16>(squares, lane) / static_cast<float>(C) + p.ln_eps);
          if (elect_one()) tma_store_wait_read0();
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t addr = my_row_s + ((static_cast<uint32_t>(q) ^ sw) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(ln_pair(keep[4 * q], mean, rstd)),
                         "r"(ln_pair(keep[4 * q + 1], mean, rstd)), "r"(ln_pair(keep[4 * q + 2], mean, rstd)),
                         "r"(ln_pair(keep[4 * q + 3], mean, rstd)) : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            tma_store_2d(&tmLn, stage_s, box0, m_warp);
            tma_store_commit();
          }
        }
      }
      if constexpr (!AHEAD) {
        // the staging boxes lie in the hidden chunk's buffer: nobody writes there before all have been read
        if (elect_one()) tma_store_wait_read0();
        __syncwarp();
        if (lane == 0) mbar_arrive(staged);
        if (!gemm_wait(staged, t & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
      }
      return true;
    };

    bool ok = true;
    uint4 pre[4] = {};
    if constexpr (AHEAD) {
      // a set's first chunk of a tile comes before the store of the tile before
      int c0 = 0;
      for (int t = 0; t <= n_my && ok; ++t, c0 += nj) {
        int j = (set + c0) & 1;              // the set's first chunk of this tile (chunk numbers run through the tiles)
        if (t > 0) fetch(pre, p.gate, p.ldgate, t - 1, box0);
        if (t < n_my && j < nj) {
          ok = gelu_chunk(c0 + j, j);
          j += 2;
        }
        if (t > 0 && ok) ok = store_tile(t - 1, pre);
        if (t == n_my || !ok) break;
        fetch_aux_box(t);
        for (; j < nj && ok; j += 2) ok = gelu_chunk(c0 + j, j);
      }
    } else {
      int c = 0;
      for (int t = 0; t < n_my && ok; ++t) {
        for (int j = 0; j < nj && ok; ++j, ++c) {
          if (j == nj - 1) fetch(pre, p.aux, p.ldaux, t, box0);
          ok = gelu_chunk(c, j);
        }
        if (ok) ok = store_tile(t, pre);
      }
    }
    if (elect_one()) tma_store_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int C, bool LN>
inline int launch_mlp_t(const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w1, const __nv_bfloat16* w2,
                        __nv_bfloat16* y, long long ldy, const MlpParams& p, int sm_count, cudaStream_t stream) {
  using S = MlpSmem<C, LN>;
  CUtensorMap tmX, tmW1, tmW2, tmOut, tmAux, tmLn;
  auto make = [&](CUtensorMap* tm, const __nv_bfloat16* base, uint64_t cols, uint64_t rows, long long ld, uint32_t bc,
                  uint32_t br, TmapSwizzle swz) {
    const uint64_t dims[2] = {cols, rows}, str[1] = {static_cast<uint64_t>(ld) * 2};
    const uint32_t box[2] = {bc, br};
    return make_tmap_bf16(tm, base, 2, dims, str, box, swz);
  };
  const uint64_t M = static_cast<uint64_t>(p.M), H = static_cast<uint64_t>(p.H);
  if (make(&tmX, x, C, M, ldx, 64, 128, TMAP_SWIZZLE_128B) != 0 ||
      make(&tmW1, w1, C, H, C, 64, MLP_CHUNK, TMAP_SWIZZLE_128B) != 0 ||
      make(&tmW2, w2, H, C, p.H, 64, C, TMAP_SWIZZLE_128B) != 0 ||
      make(&tmOut, y, C, M, ldy, 32, 32, TMAP_SWIZZLE_64B) != 0)
    return -20;
  tmAux = tmOut;
  if (p.aux != nullptr && make(&tmAux, p.aux, C, M, p.ldaux, 32, 32, TMAP_SWIZZLE_64B) != 0) return -20;
  tmLn = tmOut;
  if (LN && make(&tmLn, p.ln_out, C, M, p.ldln, 32, 32, TMAP_SWIZZLE_64B) != 0) return -20;
  auto kern = mlp_tcgen05_kernel<C, LN>;
  static std::atomic<uint64_t> smem_set;
  if (const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), S::TOTAL, smem_set); e != cudaSuccess)
    return -static_cast<int>(e) - 1000;
  const int tiles = (p.M + 127) / 128;
  return launch_chained(kern, dim3(static_cast<unsigned>(tiles < sm_count ? tiles : sm_count)), GEMM_THREADS, S::TOTAL,
                        stream, 1, tmX, tmW1, tmW2, tmOut, tmAux, tmLn, p);
}

// Whether the kernel takes these sizes (weights contiguous, everything else as the GEMMs want it).
inline bool mlp_fused_sizes(int C, int H) {
  return C % 64 == 0 && C > 0 && C <= MLP_MAX_C && H % MLP_CHUNK == 0 && H > 0;
}

// Whether it is the faster way. Two GEMMs/this kernel, microseconds with a residual, passes back to back on inputs and
// outputs that do not stay in L2, by row blocks of 128 (148 of them are one turn of the chip):
//              16        75        148       149       222       296       352       445       592       3456
//   C = 192 H = 2C 8.0/11.2  13.6/12.8 15.9/14.0 17.7/21.2 22.8/22.6 26.9/23.4 31.5/32.0 37.8/39.2 42.7/41.7 218/220
//           H = 4C 9.6/15.0  18.7/16.5 21.7/17.8 25.6/28.4 29.1/29.9 32.6/30.8 40.9/42.6 51.6/53.5 64.5/56.2 329/311
//           H = 8C 12.7/22.0 24.5/23.5 31.1/25.1 37.3/41.9 47.9/44.5 60.5/45.3 75.3/63.6 94.1/81.0 116/84.8  612/490
//   C = 256 H = 2C 9.1/13.9  15.5/15.2 20.0/16.6 22.8/25.6 25.2/27.5 29.4/28.6 34.9/38.9 42.1/48.2 50.9/52.0 272/274
//           H = 4C 10.7/18.7 22.6/20.5 26.9/22.1 32.2/35.9 36.5/38.3 45.3/39.3 58.1/54.3 73.6/69.0 90.7/76.2 473/435
//           H = 8C 14.5/29.1 32.0/31.2 42.8/33.1 52.8/56.2 68.0/61.7 85.4/62.2 104/87.5  138/130   163/135   915/705
//              1         16        48        64        149       296       592       3456
//   C = 64  H = 2C 6.5/5.2   7.0/5.3   7.1/5.3   7.5/5.6   10.7/7.5  12.6/8.3  18.6/12.6 81.9/57.7
//           H = 4C 6.8/6.1   7.3/6.1   8.2/6.4   8.4/6.7   12.4/9.2  16.5/10.2 25.0/16.5 122/78.3
//           H = 8C 7.3/8.3   7.9/8.4   9.8/8.8   10.3/9.0  17.6/13.5 22.4/14.6 38.9/25.0 211/131
//   C = 128 H = 2C 6.9/6.6   7.4/6.8   8.8/7.3   9.3/7.5   13.7/11.2 18.4/12.2 26.9/19.1 132/87.6
//           H = 4C 7.3/8.8   8.2/9.0   10.6/9.6  10.9/9.8  18.6/15.3 22.8/16.8 40.8/28.1 219/141
//           H = 8C 8.8/13.1  9.9/13.4  13.1/13.9 15.3/14.3 25.1/24.0 36.5/25.9 74.7/46.0 390/249
// The kernel's time goes by turns of the chip, each a fixed part and one for every chunk of hidden channels, however
// many row blocks the turn has; the GEMMs spread columns over the SMs too, and theirs goes by row blocks and chunks.
// Up to half a turn the kernel leaves SMs idle through all of its chunks; from there to the turn's end it is ahead. Of
// two turns the second has to be half full, a quarter where the chunks are many. From three on a 192-wide block of few
// chunks, whose turn takes as long as the GEMMs' share of one, wants two thirds of the last turn full (H = 2C: at 370
// blocks 31.9/32.2, at 400 33.7/32.4, at 520 41.0/41.3, at 560 42.2/41.6); elsewhere the two lines compare the times,
// in units of their own, as fitted to 22 numbers of blocks from 297 to 3456: the slower way by more than 2.4 % nowhere.
// Narrower blocks have the kernel ahead from few rows on; with more than four chunks its chain is longer than the two
// GEMMs' until a third of the SMs have work, and with four the two are within 1.5 us there, where the host, which
// launches one kernel less, is what a small model waits for.
inline bool mlp_fused_pays(int M, int C, int H, int sm_count) {
  if (!mlp_fused_sizes(C, H)) return false;
  const int blocks = (M + GEMM_BM - 1) / GEMM_BM, turns = (blocks + sm_count - 1) / sm_count, chunks = H / MLP_CHUNK;
  if (C <= 128) return chunks <= 4 || 3 * blocks > sm_count;
  if (turns <= 1) return 2 * blocks > sm_count;
  if (turns == 2) return 4 * blocks > (chunks >= 10 ? 5 : 6) * sm_count;
  if (C <= 192 && chunks <= 4) return 3 * (turns * sm_count - blocks) <= sm_count;
  const float passes = static_cast<float>(blocks) / static_cast<float>(sm_count);
  return C <= 192 ? turns * (4.5f + 1.1f * chunks) <= 2.5f + passes * 2.15f * chunks
                  : turns * (5.75f + 1.1f * chunks) <= 2.f + passes * 2.35f * chunks;
}

inline int launch_mlp(int C, const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w1, const __nv_bfloat16* w2,
                      __nv_bfloat16* y, long long ldy, const MlpParams& p, int sm_count, cudaStream_t stream) {
  if (p.ln_out != nullptr) switch (C) {
    case 64: return launch_mlp_t<64, true>(x, ldx, w1, w2, y, ldy, p, sm_count, stream);
    case 128: return launch_mlp_t<128, true>(x, ldx, w1, w2, y, ldy, p, sm_count, stream);
    default: return -2;
  }
  switch (C) {
    case 64: return launch_mlp_t<64, false>(x, ldx, w1, w2, y, ldy, p, sm_count, stream);
    case 128: return launch_mlp_t<128, false>(x, ldx, w1, w2, y, ldy, p, sm_count, stream);
    case 192: return launch_mlp_t<192, false>(x, ldx, w1, w2, y, ldy, p, sm_count, stream);
    case 256: return launch_mlp_t<256, false>(x, ldx, w1, w2, y, ldy, p, sm_count, stream);
    default: return -2;
  }
}

}  // namespace strata
