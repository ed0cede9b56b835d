// 3-D neighbourhood attention forward for NARROW windows (head_dim 64, bf16): same operator and
// same arguments as na3d_fwd_kernel, for windows of at most five columns.
//
// Why another kernel: tcgen05 multiplies 128 query rows by whole (plane, 4 rows, 8 or 16 columns) key
// units, so a 3 x 3 x 3 window costs every query several hundred key columns of matrix work and
// exponentials for its 27 keys. The warp-level mma.sync has a quarter of the rate (557 TFLOP/s
// measured on this part) but works on 16 queries x 8 keys: 16 queries that are neighbours
// (2 depths x 2 rows x 4 columns) see 4 * 4 = 16 groups of 8 keys of that window, a
// sixth of the work, and P stays in registers - no trip through tensor memory, no barrier between
// Q K^T, softmax and P V.
//
//   block      persistent, two per SM; an item is 2 x 8 x 8 queries (depth x rows x columns) of one
//              head: eight warps of 16 queries. The halves of an m16 tile (rows 0-7 and 8-15) are the
//              two depths, so that what differs between them - the planes they see - is uniform
//              over the warp, and the lanes' row and column masks serve both. Heads change fastest
//              over the items: the blocks that run at one time then read whole cache lines of a
//              few tiles' tokens (heads of one token are neighbours in memory).
//   keys       the box of kd+1 planes x (kh+7) rows x (kw+7) columns, one TMA box per plane for K
//              and one for V (128-byte swizzle, 128 bytes per key), in a ring of slots of up to
//              one item. The last warp to leave a slot fetches the ring's next plane into it -
//              usually the next item's - so loads run while the item is computed; nobody waits
//              for a slot to become free.
//   softmax    online, per chunk of at most CR key rows of a plane; the reference moves only when the
//              maximum has grown by more than 2^8 (the sum absorbs what lies below that as well).
//   masks      an additive -1e30 per key column, folded with the row's; planes: skipped.
//              Border clamping is exact per query.
//
// Bound: instruction issue (some 1100 instructions per 16 queries of a 3 x 3 x 3 window, 190 of them
// matrix instructions and their loads). Measured, the tcgen05 kernel -> this one: 12 heads of
// 24 x 64 x 64 tokens, window 3 x 3 x 3: 295 -> 189 us; 24 tiles of 8 x 48 x 48, 4 heads, 3 x 5 x 5:
// 439 -> 348 us; 16 heads of 24 x 64 x 64, 3 x 1 x 1: 213 -> 194 us. Windows of seven columns (16 queries
// as 1 x 8 per depth, two groups per key row) were slower, 3 x 7 x 7 by a half: tcgen05's work per
// useful key has halved by then, so the line lies at five.
// (Two m16 tiles per warp halve the ldmatrix traffic but leave eight warps per SM, each waiting out
// its own latencies; blocks of one item each wait for their loads: both no faster than tcgen05.)
#pragma once
#include <algorithm>
#include <type_traits>

#include "na3d.cuh"

namespace strata {

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

struct NaNarrowParams {
  int B, D, H, W, heads;
  int kd, kh;
  int tiles_d, tiles_h, tiles_w, n_tiles;
  int q_h0, q_H, q_w0, q_W;         // query region and output window: as in Na3dParams
  int o_h0, o_H, o_w0, o_W;
  const __nv_bfloat16* q;
  long long ldq;
  __nv_bfloat16* out;
  long long ldo;
  float scale_log2e;
  int slots;                        // ring slots, at most 2 * (kd + 1)
  int slot_bytes;                   // one K or V plane, a multiple of 1024, at least 8 spare rows
};

template <int KW>
struct NaNarrowCfg {
  static_assert(4 + KW - 1 <= 8, "the windows of 4 neighbouring queries fit one group of 8 keys");
  static constexpr int BW = 8 + KW - 1;                        // box columns
  static constexpr int THREADS = 256;
};
constexpr int NA_NARROW_MAX_KW = 5;
constexpr int NA_NARROW_Q_BYTES = 128 * 128;
constexpr int NA_NARROW_MAX_SLOTS = 32;
constexpr int NA_NARROW_SMEM = 112 * 1024;                     // per block: two per SM
constexpr int NA_NARROW_TAIL = 1024;                           // behind the slots: barriers, counters, coordinates

struct NaNarrowItem {
  int b, head, d0, h0, w0, bd0, bh0, bw0;
};

// CR: key rows of a chunk, a group of 8 keys each. ONE: the chunk is the whole plane (kh + 1 == CR).
template <int KW, int CR, bool ONE>
__global__ void __launch_bounds__(NaNarrowCfg<KW>::THREADS, 2)
na3d_narrow_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const NaNarrowParams p) {
  using Cfg = NaNarrowCfg<KW>;
  constexpr int BW = Cfg::BW;
  static_assert(CR % 2 == 0, "P V takes two key rows at a time");
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  uint8_t* tail = smem + p.slots * p.slot_bytes + NA_NARROW_Q_BYTES;
  const uint32_t q_smem = sbase + p.slots * p.slot_bytes;
  const uint32_t bar = q_smem + NA_NARROW_Q_BYTES;
  auto full = [&](int s) { return bar + 8u * s; };
  auto left = [&](int s) { return bar + 8u * NA_NARROW_MAX_SLOTS + 4u * s; };     // warps that have left a slot
  // Coordinates of the block's items n, n + 1, n + 2 (index & 3). Item n + 2 is entered by thread 0 while
  // it works on item n, before its warp leaves that item's first slot: a warp may run one item ahead of
  // thread 0 (all of an item's planes can be in the ring), but not enter item n + 1's first plane - nor
  // look at item n + 2 - before every warp has left item n's; and every warp has then read item n - 1.
  NaNarrowItem* coords = reinterpret_cast<NaNarrowItem*>(tail + 12 * NA_NARROW_MAX_SLOTS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 12 * NA_NARROW_MAX_SLOTS + 128);
  const uint32_t q_full = bar + 12 * NA_NARROW_MAX_SLOTS + 136, q_left = q_full + 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_my = (p.n_tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) /
                   static_cast<int>(gridDim.x);
  const int per_tile = 2 * (p.kd + 1);                         // ring items: K and V of every plane in turn
  const int box_bytes = BW * (p.kh + 7) * 128;

  auto decode = [&](int n) {
    unsigned t = blockIdx.x + static_cast<unsigned>(n) * gridDim.x;
    NaNarrowItem it;
    it.head = static_cast<int>(t % p.heads); t /= p.heads;
    it.w0 = p.q_w0 + static_cast<int>(t % p.tiles_w) * 8; t /= p.tiles_w;
    it.h0 = p.q_h0 + static_cast<int>(t % p.tiles_h) * 8; t /= p.tiles_h;
    it.d0 = static_cast<int>(t % p.tiles_d) * 2;
    it.b = static_cast<int>(t / p.tiles_d);
    it.bd0 = na_window_start(it.d0, p.D, p.kd);
    it.bh0 = na_window_start(it.h0, p.H, p.kh);
    it.bw0 = na_window_start(it.w0, p.W, KW);
    return it;
  };
  // plane i >> 1 of item `it` (K for even i, V for odd) into a slot
  auto fetch = [&](const NaNarrowItem& it, int i, int slot) {
    mbar_expect_tx(full(slot), box_bytes);
    tma_load_5d(sbase + slot * p.slot_bytes, (i & 1) ? &tmV : &tmK, it.head * 64, it.bw0, it.bh0,
                it.bd0 + (i >> 1), it.b, full(slot));
  };

  auto fetch_q = [&](const NaNarrowItem& it) {
    mbar_expect_tx(q_full, NA_NARROW_Q_BYTES);
    tma_load_5d(q_smem, &tmQ, it.head * 64, it.w0, it.h0, it.d0, it.b, q_full);
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    for (int s = 0; s < p.slots; ++s) {
      mbar_init(full(s), 1);
      asm volatile("st.shared.u32 [%0], 0;" ::"r"(left(s)) : "memory");
    }
    mbar_init(q_full, 1);
    asm volatile("st.shared.u32 [%0], 0;" ::"r"(q_left) : "memory");
    *abort_flag = 0;
    fence_mbar_init();
    coords[0] = decode(0);
    coords[1] = decode(1);
  }
  // the rows behind each slot's box may be read (and multiplied by zero) by the last key row's group
  for (int i = threadIdx.x; i < p.slots * 64; i += Cfg::THREADS)
    *reinterpret_cast<uint4*>(smem + (i >> 6) * p.slot_bytes + box_bytes + (i & 63) * 16) = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  chain_begin();
  if (threadIdx.x == 0) {
    fetch_q(coords[0]);
    for (int i = 0; i < p.slots; ++i) fetch(coords[0], i, i);
  }

  const int g = lane >> 2, tq = lane & 3;
  // the warp's plane position within the 8 x 8 tile, and this lane's query (both depths)
  const int zh0 = (warp >> 1) * 2, zw0 = (warp & 1) * 4;
  const int zh = zh0 + (g >> 2), zw = zw0 + (g & 3);
  // the row of the Q tile (d, h, w) this lane supplies to ldmatrix: lane 8i + j query j of depth i & 1
  const int q_row = (((lane >> 3) & 1) * 8 + zh0 + ((lane & 7) >> 2)) * 8 + zw0 + (lane & 3);
  const int n_rows = p.kh + 1;                                 // key rows of a plane the warp's queries see
  const uint64_t c2 = pack2(p.scale_log2e, p.scale_log2e);
  // Byte offset in a slot of a lane's row of an ldmatrix: key `key` of the box, 16-byte chunk `chunk` of
  // its 64 channels (128-byte swizzle). Other chunks of the same key are an XOR away: chunk ^ x is
  // offset ^ (x << 4), and slots are multiples of 1024 bytes, so the XOR may come after the slot.
  auto row_off = [&](int key, int chunk) -> uint32_t { return key * 128 + ((chunk ^ (key & 7)) << 4); };

  bool ok = true;
  int st = 0;               // slot of the plane's K, and the parity of its barrier
  uint32_t ph = 0;
#pragma unroll 1
  for (int n = 0; n < n_my && ok; ++n) {
    const NaNarrowItem it = coords[n & 3];
    const int ih = min(it.h0 + zh, p.H - 1), iw = min(it.w0 + zw, p.W - 1);
    // Q: A fragments (rows 0-7: depth d0, rows 8-15: depth d0 + 1); the last warp fetches the next item's
    uint32_t qf[4][4];
    if (!na_wait(q_full, n & 1u, abort_flag, ST_TIMEOUT_SOFTMAX)) { ok = false; break; }
#pragma unroll
    for (int s = 0; s < 4; ++s) ldsm_x4(q_smem + q_row * 128 + (((2 * s + (lane >> 4)) ^ (q_row & 7)) << 4), qf[s]);
    __syncwarp();
    if (lane == 0) {
      uint32_t cnt;
      asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(cnt) : "r"(q_left) : "memory");
      if (cnt == 7u) {
        asm volatile("st.shared.u32 [%0], 0;" ::"r"(q_left) : "memory");
        if (n + 1 < n_my) fetch_q(coords[(n + 1) & 3]);
      }
    }
    // box coordinates of the first key row / column any of the warp's queries sees
    const int rb = na_window_start(min(it.h0 + zh0, p.H - 1), p.H, p.kh) - it.bh0;
    const int cb = na_window_start(min(it.w0 + zw0, p.W - 1), p.W, KW) - it.bw0;
    const uint32_t rows = ((1u << p.kh) - 1u) << (na_window_start(ih, p.H, p.kh) - it.bh0 - rb);
    const int ww = na_window_start(iw, p.W, KW) - it.bw0 - cb;
    // the masks as addends of the scaled scores of this lane's two keys of a group
    const uint64_t colb = pack2(static_cast<unsigned>(2 * tq - ww) < static_cast<unsigned>(KW) ? 0.f : -1e30f,
                                static_cast<unsigned>(2 * tq + 1 - ww) < static_cast<unsigned>(KW) ? 0.f : -1e30f);
    const uint64_t NEG2 = pack2(-1e30f, -1e30f);
    uint64_t rowb[CR];
    if constexpr (ONE) {
#pragma unroll
      for (int r = 0; r < CR; ++r) rowb[r] = (rows >> r) & 1u ? colb : NEG2;
    }
    // first plane of each depth's window (the second depth may not exist)
    const int pd0 = 0, pd1 = it.d0 + 1 < p.D ? na_window_start(it.d0 + 1, p.D, p.kd) - it.bd0 : 1 << 20;
    // ldmatrix rows. K: lane 8i + j supplies key j, chunk i (the other four chunks: ^ 64). V
    // (transposed): two key rows, lane 8i + j supplies key j of row i & 1, chunk i >> 1 (the next two: ^ 32 ...)
    const int kkey = rb * BW + cb + (lane & 7);
    auto k_off = [&](int r) { return row_off(kkey + r * BW, lane >> 3); };
    auto v_off = [&](int r) { return row_off(kkey + (r + ((lane >> 3) & 1)) * BW, lane >> 4); };

    float o[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
    float mx[2] = {-5e29f, -5e29f}, l[2] = {0.f, 0.f};   // reference (scaled), this lane's part of the sum

#pragma unroll 1
    for (int pl = 0; pl <= p.kd; ++pl) {
      const int st_v = st + 1 == p.slots ? 0 : st + 1;
      const uint32_t ph_v = st + 1 == p.slots ? ph ^ 1u : ph;
      const bool act[2] = {static_cast<unsigned>(pl - pd0) < static_cast<unsigned>(p.kd),
                           static_cast<unsigned>(pl - pd1) < static_cast<unsigned>(p.kd)};
      // (a plane this warp does not see is waited for too: it may only leave the slots once they
      // hold that plane, or it would count towards an earlier or later one)
      if (!na_wait(full(st), ph, abort_flag, ST_TIMEOUT_SOFTMAX)) { ok = false; break; }
      if (pl == 0 && threadIdx.x == 0) coords[(n + 2) & 3] = decode(n + 2);
      const uint32_t ks = sbase + st * p.slot_bytes, vs = sbase + st_v * p.slot_bytes;
#pragma unroll 1
      for (int r0 = 0; r0 < (ONE ? 1 : n_rows); r0 += CR) {
        if (!act[0] && !act[1]) break;
        // ---- scores of the chunk
        float s[CR][4];
#pragma unroll
        for (int i = 0; i < CR; ++i) {
#pragma unroll
          for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
          if (ONE || r0 + i < n_rows) {
            uint32_t k0[4], k1[4];
            const uint32_t addr = ks + k_off(r0 + i);
            ldsm_x4(addr, k0);
            ldsm_x4(addr ^ 64u, k1);
            mma_16816(s[i], qf[0], k0[0], k0[1]);
            mma_16816(s[i], qf[1], k0[2], k0[3]);
            mma_16816(s[i], qf[2], k1[0], k1[1]);
            mma_16816(s[i], qf[3], k1[2], k1[3]);
          }
        }
        // ---- softmax of the depths that see the plane (both in the middle planes: their chains of
        // dependent instructions then overlap); P as bf16 A fragments (two key rows = 16 keys)
        uint32_t pf[CR / 2][4];
        auto softmax = [&](auto lo, auto hi) {
          constexpr int H0 = decltype(lo)::value, H1 = decltype(hi)::value;
          if constexpr (H1 - H0 == 1) {
#pragma unroll
            for (int i = 0; i < CR; ++i) pf[i / 2][(i & 1) * 2 + 1 - H0] = 0u;
          }
          uint64_t x[2][CR];
          float cm[2] = {-1e30f, -1e30f};
#pragma unroll
          for (int i = 0; i < CR; ++i) {
            uint64_t bias;
            if constexpr (ONE) bias = rowb[i];
            else bias = (rows >> (r0 + i)) & 1u ? colb : NEG2;
#pragma unroll
            for (int h = H0; h < H1; ++h) {
              x[h][i] = ffma2(pack2(s[i][2 * h], s[i][2 * h + 1]), c2, bias);
              float x0, x1;
              unpack2(x[h][i], x0, x1);
              cm[h] = fmax3(cm[h], x0, x1);
            }
          }
#pragma unroll
          for (int h = H0; h < H1; ++h) cm[h] = fmaxf(cm[h], __shfl_xor_sync(0xffffffffu, cm[h], 1));
#pragma unroll
          for (int h = H0; h < H1; ++h) cm[h] = fmaxf(cm[h], __shfl_xor_sync(0xffffffffu, cm[h], 2));
          bool moves = false;
#pragma unroll
          for (int h = H0; h < H1; ++h) moves |= cm[h] > mx[h] + 8.f;
          if (__any_sync(0xffffffffu, moves)) {
#pragma unroll
            for (int h = H0; h < H1; ++h) {
              const float nm = cm[h] > mx[h] + 8.f ? cm[h] : mx[h], alpha = fast_exp2(mx[h] - nm);
              mx[h] = nm;
              l[h] *= alpha;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                o[i][2 * h] *= alpha;
                o[i][2 * h + 1] *= alpha;
              }
            }
          }
          uint64_t sum[2] = {0ull, 0ull};
#pragma unroll
          for (int i = 0; i < CR; ++i)
#pragma unroll
            for (int h = H0; h < H1; ++h) {
              float t0, t1;
              unpack2(fadd2(x[h][i], pack2(-mx[h], -mx[h])), t0, t1);
              const float e0 = fast_exp2(t0), e1 = fast_exp2(t1);
              sum[h] = fadd2(sum[h], pack2(e0, e1));
              pf[i / 2][(i & 1) * 2 + h] = pack_bf16(e0, e1);
            }
#pragma unroll
          for (int h = H0; h < H1; ++h) {
            float s0, s1;
            unpack2(sum[h], s0, s1);
            l[h] += s0 + s1;
          }
        };
        using C0 = std::integral_constant<int, 0>;
        using C1 = std::integral_constant<int, 1>;
        using C2 = std::integral_constant<int, 2>;
        if (act[0] && act[1]) softmax(C0{}, C2{});
        else if (act[0]) softmax(C0{}, C1{});
        else softmax(C1{}, C2{});
        // ---- O += P V
        if (r0 == 0 && !na_wait(full(st_v), ph_v, abort_flag, ST_TIMEOUT_SOFTMAX)) { ok = false; break; }
#pragma unroll
        for (int i = 0; i < CR / 2; ++i) {
          if (ONE || r0 + 2 * i < n_rows) {
            const uint32_t addr = vs + v_off(r0 + 2 * i);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t v[4];
              ldsm_x4_t(addr ^ (32u * j), v);
              mma_16816(o[2 * j], pf[i], v[0], v[1]);
              mma_16816(o[2 * j + 1], pf[i], v[2], v[3]);
            }
          }
        }
      }
      if (!ok) break;
      if (!act[0] && !act[1] && !na_wait(full(st_v), ph_v, abort_flag, ST_TIMEOUT_SOFTMAX)) { ok = false; break; }
      // ---- leave the two slots; the last warp out fetches the ring's next plane into each
      __syncwarp();
      if (lane < 2) {
        const int slot = lane ? st_v : st;
        int next = 2 * pl + lane + p.slots, tile = n;
        if (next >= per_tile) { next -= per_tile; ++tile; }
        uint32_t cnt;
        asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(cnt) : "r"(left(slot)) : "memory");
        if (cnt == 7u) {
          asm volatile("st.shared.u32 [%0], 0;" ::"r"(left(slot)) : "memory");
          if (tile < n_my) fetch(coords[tile & 3], next, slot);
        }
      }
      st = st_v + 1 == p.slots ? 0 : st_v + 1;
      ph = st_v + 1 == p.slots ? ph_v ^ 1u : ph_v;
    }
    if (!ok) break;

    // ---------------------------------------------------------------- normalise and store
    const bool live = it.w0 + zw < p.q_w0 + p.q_W && it.h0 + zh < p.q_h0 + p.q_H;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && it.d0 + 1 >= p.D) break;
      float sum = l[h];
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      const float inv = 1.0f / sum;
      const long long tok = ((static_cast<long long>(it.b) * p.D + it.d0 + h) * p.o_H + (it.h0 + zh - p.o_h0)) * p.o_W +
                            (it.w0 + zw - p.o_w0);
      __nv_bfloat16* op = p.out + tok * p.ldo + it.head * 64;
      // the quad's four lanes hold words t of every 8-channel chunk: transpose 4 chunks x 4 words so
      // that each lane stores whole 16-byte chunks
      const bool odd = tq & 1, hi = tq & 2;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t w[4], x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          w[i] = pack_bf16(o[4 * half + i][2 * h] * inv, o[4 * half + i][2 * h + 1] * inv);
        const uint32_t s0 = __shfl_xor_sync(0xffffffffu, odd ? w[0] : w[1], 1);
        const uint32_t s1 = __shfl_xor_sync(0xffffffffu, odd ? w[2] : w[3], 1);
        x[0] = odd ? s0 : w[0]; x[1] = odd ? w[1] : s0;
        x[2] = odd ? s1 : w[2]; x[3] = odd ? w[3] : s1;
        const uint32_t u0 = __shfl_xor_sync(0xffffffffu, hi ? x[0] : x[2], 2);
        const uint32_t u1 = __shfl_xor_sync(0xffffffffu, hi ? x[1] : x[3], 2);
        if (live)
          *reinterpret_cast<uint4*>(op + (4 * half + tq) * 8) =
              hi ? make_uint4(u0, u1, x[2], x[3]) : make_uint4(x[0], x[1], u0, u1);
      }
    }
  }
  if (!ok) {   // loads in flight must land before the block retires
#pragma unroll 1
    for (int k = 0; k < 2000; ++k) __nanosleep(100);
  }
}

template <int KW, int CR, bool ONE>
inline int launch_na3d_narrow_t(const __nv_bfloat16* k, long long ldk, const __nv_bfloat16* v, long long ldv,
                                NaNarrowParams p, int sm_count, cudaStream_t stream) {
  using Cfg = NaNarrowCfg<KW>;
  auto make = [&](CUtensorMap* tm, const __nv_bfloat16* base, long long ld, uint32_t bw, uint32_t bh, uint32_t bd) {
    const uint64_t w = static_cast<uint64_t>(p.W), h = static_cast<uint64_t>(p.H), d = static_cast<uint64_t>(p.D);
    uint64_t dims[5] = {static_cast<uint64_t>(p.heads) * 64, w, h, d, static_cast<uint64_t>(p.B)};
    const uint64_t row = static_cast<uint64_t>(ld) * 2;
    uint64_t str[4] = {row, row * w, row * w * h, row * w * h * d};
    uint32_t box[5] = {64, bw, bh, bd, 1};
    return make_tmap_bf16(tm, base, 5, dims, str, box);
  };
  CUtensorMap tmQ, tmK, tmV;
  const uint32_t bh = static_cast<uint32_t>(p.kh + 7);
  if (make(&tmQ, p.q, p.ldq, 8, 8, 2) != 0 || make(&tmK, k, ldk, Cfg::BW, bh, 1) != 0 ||
      make(&tmV, v, ldv, Cfg::BW, bh, 1) != 0)
    return -20;
  p.slot_bytes = (Cfg::BW * (p.kh + 7) * 128 + 1024 + 1023) / 1024 * 1024;
  const int fit = (NA_NARROW_SMEM - NA_NARROW_Q_BYTES - NA_NARROW_TAIL) / p.slot_bytes;
  p.slots = std::min(std::min(2 * (p.kd + 1), fit), NA_NARROW_MAX_SLOTS);
  if (p.slots < 2) return -2;
  const long long items = static_cast<long long>(p.tiles_d) * p.tiles_h * p.tiles_w * p.heads * p.B;
  if (items > 0x3fffffffLL) return -2;
  p.n_tiles = static_cast<int>(items);
  auto kern = na3d_narrow_kernel<KW, CR, ONE>;
  static std::atomic<uint64_t> smem_set;
  if (const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), NA_NARROW_SMEM, smem_set); e != cudaSuccess)
    return -static_cast<int>(e) - 1000;
  const int grid = p.n_tiles < 2 * sm_count ? p.n_tiles : 2 * sm_count;
  return launch_chained(kern, dim3(static_cast<unsigned>(grid)), Cfg::THREADS,
                        static_cast<size_t>(p.slots) * p.slot_bytes + NA_NARROW_Q_BYTES + NA_NARROW_TAIL, stream, 1, tmQ, tmK,
                        tmV, p);
}

// The chunk is the whole plane for the common heights (its row masks then stay in registers), eight
// key rows otherwise.
inline int launch_na3d_narrow(const __nv_bfloat16* k, long long ldk, const __nv_bfloat16* v, long long ldv,
                              int kw, const NaNarrowParams& p, int sms, cudaStream_t st) {
  switch (kw) {
    case 1: return p.kh == 1 ? launch_na3d_narrow_t<1, 2, true>(k, ldk, v, ldv, p, sms, st)
                             : launch_na3d_narrow_t<1, 8, false>(k, ldk, v, ldv, p, sms, st);
    case 3: return p.kh == 3 ? launch_na3d_narrow_t<3, 4, true>(k, ldk, v, ldv, p, sms, st)
                             : launch_na3d_narrow_t<3, 8, false>(k, ldk, v, ldv, p, sms, st);
    case 5: return p.kh == 5 ? launch_na3d_narrow_t<5, 6, true>(k, ldk, v, ldv, p, sms, st)
                             : launch_na3d_narrow_t<5, 8, false>(k, ldk, v, ldv, p, sms, st);
    default: return -2;
  }
}

}  // namespace strata
