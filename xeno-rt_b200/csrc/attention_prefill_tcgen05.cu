// Causal grouped-query attention for prompts on the fifth-generation tensor cores (head size 128).
// (The reference's prefill form: crates/xrt-models/src/llama.rs:728-770: for token t the keys
// 0 .. start + t, read from the cache so that earlier context is included.)
//
// A block owns two tiles of 128 query rows that need the same keys: 128 consecutive new tokens of one sequence for two
// query heads of one kv head, or, where a kv head's query heads are odd in number, 256 consecutive new tokens for one query
// head; or one tile of 128 rows, where two would leave multiprocessors empty (two_tiles, below).  It walks the sequence's keys in steps of 128 (two cache blocks of 64) from the cache block of the first row's
// first visible key (KeyRange in common.cuh: all keys, a window, or the query's own chunk of positions).  A head may have
// a sink: one more term of the softmax's denominator, added to the row's sum at the end.  Ten warps (one tile: six):
//   warp 0    TMA: the Q tiles once, then for each step its K and V tiles ([128 keys x 128], as boxes
//             of 64 keys x 64 dims, 128-byte swizzle), fetched once for both query tiles, into rings of two stages
//             (one tile: three).
//   warp 1    owns TMEM and issues the MMAs: S = Q K^T (128 x 128, eight tcgen05.mma over the head
//             size) and O += P V (128 x 128, eight tcgen05.mma over the step's keys) accumulated in TMEM over all
//             steps.  K is a K-major operand as stored; V ([key][dim]) is an MN-major operand as stored: no
//             transposition anywhere.  The two query tiles take turns: while one's softmax runs, the tensor core has
//             the other's products (P V of a step, at once followed by Q K^T of the next).  A single tile has two S of its
//             own: while the softmax of a step runs, the tensor core has the Q K^T of the next.
//   warps 2-9 softmax and output, four warps a query tile, one thread a query row (TMEM lane).  A thread reads its row
//             of S (tcgen05.ld), masks (only steps that reach the diagonal), keeps the row's sum in 32-bit,
//             and writes P as bfloat16 pairs over the S it has read (tcgen05.st), from where P V reads it as its A
//             operand; the next S overwrites it after that product, in the order in which the products are issued.
//             The exponents are taken
//             against a reference value m of the row that only moves when the row's maximum has
//             grown by more than 8 (a factor 256) beyond it: softmax does not depend on m as long as
//             P and the sum use the same one, P stays within 2^8 (bfloat16 keeps its 8 bits of
//             precision at any magnitude), and the accumulated O in TMEM has to be rescaled (read,
//             multiplied, written back by the row's thread) only on those rare moves instead of once a step.
// What bounds a step of one tile is the chain of its softmax (the exponentials alone take 1,024 clocks of the special-function
// units, as long as the tile's products take the tensor core): with one tile a block that chain is all a multiprocessor
// does.  Measured, microseconds a layer of 32 + 8 heads, one tile a block -> two: a prompt of 7,999
// tokens 814 -> 714 (734 TFLOP/s), 16 prompts of 64 to 2,047 582 -> 404, one of 2,048 58 -> 50.  With two tiles neither unit is
// the bound yet: the products of 7,999 tokens are 333 us at the burst rate and the exponentials 235, and a prompt of 4,096 keeps
// the tensor core busy 43 percent of the clocks, the special-function units 43 and the issue slots 34, so the two tiles' chains
// overlap only in part.  What a step waits for is not known; two threads a row (eight warps a tile, halves of the keys) were no
// faster (718 and 420), so it is not the length of one thread's chain.
// Every mbarrier wait is bounded; a wait that runs out raises the error flag and an abort flag, all
// roles leave their loops, TMEM is freed and the block returns.
#include "tcgen05.cuh"

namespace xrt {

using namespace sm100;

constexpr int FA_ROWS = 128, FA_KEYS = 128, FA_HD = 128;
constexpr int FA_Q_BYTES = FA_ROWS * FA_HD * 2;        // 32 KB (two halves of 16 KB)
constexpr int FA_BOX = 64 * 64 * 2;                    // 8 KB: what one tensor copy brings, 64 keys x 64 dims
constexpr int FA_KV_HALF = FA_KEYS * 64 * 2;           // 16 KB: 128 keys (two cache blocks) x 64 dims
constexpr int FA_STAGE_BYTES = 4 * FA_KV_HALF;         // K halves, then V halves: 64 KB
template <int TILES> struct FaShape {
  static constexpr int STAGES = TILES == 2 ? 2 : 3, THREADS = 64 + 128 * TILES;
  static constexpr int SMEM = TILES * FA_Q_BYTES + STAGES * FA_STAGE_BYTES + 512 + 1024;
};

// 2^x by the special-function unit; exp2(-inf) = 0.  Inputs are differences to a running maximum
// (at most 0) and the result feeds a bfloat16 product or a 32-bit sum: the unit's 2 ulp are far
// inside bfloat16's 8 bits.
__device__ __forceinline__ float fa_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// HEADS: the block's two tiles are the same rows of two query heads of one kv head; else its tiles are consecutive rows of one
// query head.
template <int TILES, bool HEADS>
__global__ void __launch_bounds__(FaShape<TILES>::THREADS, 1)
attention_prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                 const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out,
                                 const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot,
                                 const int* __restrict__ seq_start, const int* __restrict__ block_table, int max_blocks,
                                 int n_heads, int n_kv_heads, float scale_log2, int* __restrict__ error_flag,
                                 const KeyRange range, const float* __restrict__ sinks) {
  static_assert(TILES == 2 || !HEADS, "one tile is of one head");
  constexpr int FA_TILES = TILES, FA_STAGES = FaShape<TILES>::STAGES;
  constexpr int S_BUFFERS = TILES == 1 ? 2 : 1;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* q_tiles = smem;                                   // [FA_TILES] x 32 KB
  unsigned char* kv_ring = smem + FA_TILES * FA_Q_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(kv_ring + FA_STAGES * FA_STAGE_BYTES);
  uint64_t* q_full = bars;                 // [1]
  uint64_t* k_full = bars + 1;             // [FA_STAGES] each: K and V of a step have barriers of their own,
  uint64_t* k_empty = k_full + FA_STAGES;  //   since a step's K is free again (after its QK^T) a whole step
  uint64_t* v_full = k_empty + FA_STAGES;  //   before its V (after its PV): the next K is fetched that much earlier
  uint64_t* v_empty = v_full + FA_STAGES;
  uint64_t* s_full = v_empty + FA_STAGES;  // [2]: of a tile, or of a single tile's buffer of S (whose next step but one comes
  uint64_t* p_full = s_full + 2;           //   first when its waits have passed); p_full also says that S was read
  uint64_t* o_done = p_full + 2;           // [FA_TILES]: once, after the tile's last product; one tile: after every step's
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + FA_TILES);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // later query tiles walk more keys: they are scheduled first, the longest tiles of ALL heads before any shorter one
  // (the heads are the grid's fastest dimension).  With the query tiles fastest, the last heads' long tiles started
  // when most multiprocessors were already idle: a prompt of 2,048 tokens is 512 blocks of 1 to 16 steps on 148
  // multiprocessors, 42 steps on the busiest that way against 33 this way (71.5 -> 61.2 us a layer).
  // Of several prompts, every prompt's tiles at a query index come before any tile at a lower one (a tile beyond a
  // shorter prompt's end leaves at once): the prompts are the grid's second dimension, the query tiles its slowest.
  const int q_index = gridDim.z - 1 - blockIdx.z, head0 = blockIdx.x * (HEADS ? 2 : 1), seq = blockIdx.y;
  const int slot = seq_slot[seq];
  const int tok0 = cu_seqlens[seq];
  const int n_new = cu_seqlens[seq + 1] - tok0;
  const int row0 = q_index * (HEADS ? FA_ROWS : FA_TILES * FA_ROWS);
  if (slot < 0 || row0 >= n_new) return;  // the whole block leaves before any barrier or allocation
  const int start = seq_start[seq];
  const int kv_head = head0 / (n_heads / n_kv_heads);  // the same for both heads: their number a kv head is even
  // keys from the cache block of the first row's first visible key to a tile's last row's position
  const int first_block = range.first(start + row0) / XRT_BLOCK_TOKENS;
  const int key_base = first_block * XRT_BLOCK_TOKENS;
  auto row0_of = [&](int u) { return HEADS ? row0 : row0 + u * FA_ROWS; };
  auto last_row_of = [&](int u) { return min(row0_of(u) + FA_ROWS, n_new) - 1; };
  auto steps_of = [&](int u) {  // 0: the second tile lies beyond the sequence
    return row0_of(u) < n_new ? (start + last_row_of(u) + 1 - key_base + FA_KEYS - 1) / FA_KEYS : 0;
  };
  const int steps0 = steps_of(0), steps1 = TILES == 2 ? steps_of(1) : 0;
  const int n_steps = max(steps0, steps1);
  const int last_row = steps1 > 0 ? last_row_of(1) : last_row_of(0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int TMEM_COLS = 512;  // S (and P over it) and O of every tile: all of TMEM, or 384 columns of it
  static_assert(FA_TILES * (S_BUFFERS * FA_KEYS + FA_HD) <= TMEM_COLS, "S and O must fit in TMEM");

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(q_full), 1);
    for (int s = 0; s < FA_STAGES; ++s) {
      mbar_init(smem_u32(&k_full[s]), 1); mbar_init(smem_u32(&k_empty[s]), 1);
      mbar_init(smem_u32(&v_full[s]), 1); mbar_init(smem_u32(&v_empty[s]), 1);
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(smem_u32(&s_full[u]), 1);
      // the softmax warps arrive once each (lane 0, after the warp has synchronised): a hundred
      // arrivals on one shared-memory word would serialise
      mbar_init(smem_u32(&p_full[u]), 4);
    }
    for (int u = 0; u < FA_TILES; ++u) mbar_init(smem_u32(&o_done[u]), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_s = tmem_base;                            // [tile or buffer] x 128 columns; P: the first 64 of them
  const uint32_t tmem_o = tmem_base + 2 * FA_KEYS;              // [tile] x 128 columns
  auto s_place = [](int j, int u) { return TILES == 2 ? u : j & 1; };  // which S (and barrier) tile u has at step j
  auto s_parity = [](int j) { return (uint32_t)(TILES == 2 ? j : j >> 1) & 1u; };

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
      mbar_arrive_expect_tx(smem_u32(q_full), FA_TILES * FA_Q_BYTES);
#pragma unroll
      for (int u = 0; u < FA_TILES; ++u) {
        const uint32_t dst = smem_u32(q_tiles + u * FA_Q_BYTES);
        const int col = (HEADS ? head0 + u : head0) * FA_HD;
        tma_load_2d(dst, &map_q, col, tok0 + row0_of(u), smem_u32(q_full));
        tma_load_2d(dst + FA_Q_BYTES / 2, &map_q, col + 64, tok0 + row0_of(u), smem_u32(q_full));
      }
      const int* blocks = block_table + (size_t)slot * max_blocks;
      const int n_blocks = (start + last_row + 1 + XRT_BLOCK_TOKENS - 1) / XRT_BLOCK_TOKENS;  // cache blocks the rows see
      bool ok = true;
      for (int j = 0; j < n_steps && ok; ++j) {
        const int s = j % FA_STAGES;
        unsigned char* stage = kv_ring + s * FA_STAGE_BYTES;
        int pool_row[2];  // the step's two cache blocks; beyond the last one the last again (masked)
#pragma unroll
        for (int part = 0; part < 2; ++part)
          pool_row[part] = (blocks[min(first_block + 2 * j + part, n_blocks - 1)] * n_kv_heads + kv_head) * XRT_BLOCK_TOKENS;
        ok = mbar_wait(smem_u32(&k_empty[s]), ((j / FA_STAGES) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_arrive_expect_tx(smem_u32(&k_full[s]), 2 * FA_KV_HALF);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          tma_load_2d(smem_u32(stage + part * FA_BOX), &map_k, 0, pool_row[part], smem_u32(&k_full[s]));
          tma_load_2d(smem_u32(stage + FA_KV_HALF + part * FA_BOX), &map_k, 64, pool_row[part], smem_u32(&k_full[s]));
        }
        ok = mbar_wait(smem_u32(&v_empty[s]), ((j / FA_STAGES) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_arrive_expect_tx(smem_u32(&v_full[s]), 2 * FA_KV_HALF);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          tma_load_2d(smem_u32(stage + 2 * FA_KV_HALF + part * FA_BOX), &map_v, 0, pool_row[part], smem_u32(&v_full[s]));
          tma_load_2d(smem_u32(stage + 3 * FA_KV_HALF + part * FA_BOX), &map_v, 64, pool_row[part], smem_u32(&v_full[s]));
        }
      }
      if (!ok) { *abort_flag = 1; if (error_flag != nullptr) atomicExch(error_flag, 5); }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issue
    if (lane == 0) {
      constexpr uint32_t idesc_qk = instr_desc(FA_ROWS, FA_KEYS, false);
      constexpr uint32_t idesc_pv = instr_desc(FA_ROWS, FA_HD, true);
      bool ok = mbar_wait(smem_u32(q_full), 0, abort_flag);
      // The tile that uses a step's K and V last: the second, while it has steps left (or has any: the first tile of 256
      // rows never has more steps than the second).
      auto last_tile = [&](int j) { return j < steps1 ? 1 : 0; };
      auto issue_qk = [&](int j, int u) {
        const int s = j % FA_STAGES;
        if (!mbar_wait(smem_u32(&k_full[s]), (j / FA_STAGES) & 1, abort_flag)) return false;
        fence_after();
        unsigned char* stage = kv_ring + s * FA_STAGE_BYTES;
#pragma unroll
        for (int ks = 0; ks < FA_HD / 16; ++ks) {  // 16 dims a step; 4 steps a 64-dim half
          const uint64_t a = desc_k_major(smem_u32(q_tiles + u * FA_Q_BYTES + (ks / 4) * (FA_Q_BYTES / 2))) + 2 * (ks % 4);
          const uint64_t bd = desc_k_major(smem_u32(stage + (ks / 4) * FA_KV_HALF)) + 2 * (ks % 4);
          mma_f16(tmem_s + s_place(j, u) * FA_KEYS, a, bd, idesc_qk, ks > 0);
        }
        commit(smem_u32(&s_full[s_place(j, u)]));
        if (u == last_tile(j)) commit(smem_u32(&k_empty[s]));
        return true;
      };
#pragma unroll 1
      for (int u = 0; u < FA_TILES && ok; ++u)
        if (0 < (u == 0 ? steps0 : steps1)) ok = issue_qk(0, u);
      for (int j = 0; j < n_steps && ok; ++j) {
        const int s = j % FA_STAGES;
        unsigned char* stage = kv_ring + s * FA_STAGE_BYTES;
        // one tile: the next S goes into the other buffer, whose P was used up by a product issued before
        if (TILES == 1 && j + 1 < n_steps) {
          ok = issue_qk(j + 1, 0);
          if (!ok) break;
        }
#pragma unroll 1
        for (int u = 0; u < FA_TILES && ok; ++u) {
          const int steps = u == 0 ? steps0 : steps1;
          if (j >= steps) continue;
          ok = mbar_wait(smem_u32(&p_full[s_place(j, u)]), s_parity(j), abort_flag) &&  // P is written, and O rescaled if it had to be
               mbar_wait(smem_u32(&v_full[s]), (j / FA_STAGES) & 1, abort_flag);
          if (!ok) break;
          fence_after();
#pragma unroll
          for (int ks = 0; ks < FA_KEYS / 16; ++ks) {  // 16 keys a step
            const uint64_t bd = desc_mn_major(smem_u32(stage + 2 * FA_KV_HALF + ks * 2048), FA_KV_HALF);
            mma_f16_a_tmem(tmem_o + u * FA_HD, tmem_s + s_place(j, u) * FA_KEYS + ks * 8, bd, idesc_pv,
                           j > 0 || ks > 0);
          }
          if (u == last_tile(j)) commit(smem_u32(&v_empty[s]));
          // two tiles: the next S takes the place of this step's P: products run in the order in which they are issued
          if (TILES == 2 && j + 1 < steps) ok = issue_qk(j + 1, u);
          else commit(smem_u32(&o_done[u]));
        }
      }
      if (!ok) { *abort_flag = 1; if (error_flag != nullptr) atomicExch(error_flag, 5); }
    }
  } else {
    // ---------------------------------------------------------------- softmax and output: one thread a row and head
    const int quarter = warp & 3;
    const int u = (warp - 2) >> 2;               // which of the block's tiles
    const int head = HEADS ? head0 + u : head0;
    const int r = quarter * 32 + lane;           // row of the tile = TMEM lane
    const int tile_row0 = row0_of(u), n_tiles = u == 0 ? steps0 : steps1;
    const int row = tile_row0 + r;               // new-token index in the sequence
    const bool row_live = row < n_new;
    const int key_hi = row_live ? start + row + 1 : 0;  // keys [key_lo, key_hi) are visible
    const int key_lo = range.first(start + row);
    const int all_lo = range.first(start + last_row_of(u));  // from here on no row's range has yet to begin
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t my_o = tmem_o + lane_base + u * FA_HD;
    float m_ref = -INFINITY, l_run = 0.f;  // the reference value of the exponents (scaled, base 2) and the sum
    bool ok = true;

    for (int j = 0; j < n_tiles && ok; ++j) {
      ok = mbar_wait(smem_u32(&s_full[s_place(j, u)]), s_parity(j), abort_flag);
      if (!ok) break;
      fence_after();
      const uint32_t my_s = tmem_s + lane_base + s_place(j, u) * FA_KEYS;
      const int key0 = key_base + j * FA_KEYS;
      // Only steps that reach past the first row's last visible key, or begin before the last row's first one, can
      // hide a key from a row (uniform over the tile); every other step skips the comparisons.
      const bool early = key0 < all_lo, late = key0 + FA_KEYS > start + tile_row0 + 1;
      // Half of the row at a time, twice: for the maximum, and again from tensor memory for the exponents.  (The whole row
      // in registers beside P does not fit the 168 that ten warps leave each thread; six warps keep it.)
      float s[TILES == 2 ? 1 : 2][FA_KEYS / 2];
      auto read_half = [&](float (&s)[FA_KEYS / 2], int half) {
        uint32_t v0[32], v1[32];
        tmem_ld32(v0, my_s + half * 64);
        tmem_ld32(v1, my_s + half * 64 + 32);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) { s[i] = __uint_as_float(v0[i]); s[32 + i] = __uint_as_float(v1[i]); }
        if (early) {
#pragma unroll
          for (int i = 0; i < 64; ++i) s[i] = (key0 + half * 64 + i >= key_lo) ? s[i] : -INFINITY;
        }
        if (late) {
#pragma unroll
          for (int i = 0; i < 64; ++i) s[i] = (key0 + half * 64 + i < key_hi) ? s[i] : -INFINITY;
        }
      };
      // the maximum of the raw scores (the scale is positive and is applied inside the exponent)
      float part_max[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float (&row)[FA_KEYS / 2] = s[TILES == 2 ? 0 : half];
        read_half(row, half);
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
#pragma unroll
          for (int k = 0; k < 4; ++k) part_max[k] = fmaxf(part_max[k], row[i + k]);
        }
      }
      const float m_tile = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3])) * scale_log2;
      // move the reference only when the maximum has outgrown it by more than 8; the first visible key sets it
      const bool moves = m_tile > m_ref + 8.0f || (m_ref == -INFINITY && m_tile != -INFINITY);
      if (__any_sync(0xffffffffu, moves)) {
        const float factor = (moves && m_ref != -INFINITY) ? fa_exp2(m_ref - m_tile) : 1.0f;
        if (j > 0) {  // O holds the products of the steps so far: two tiles' were issued before this step's S, which is complete
          if (TILES == 1) {
            ok = mbar_wait(smem_u32(&o_done[u]), (uint32_t)(j - 1) & 1u, abort_flag);
            if (!ok) break;
            fence_after();
          }
          if (__any_sync(0xffffffffu, factor != 1.0f)) {
#pragma unroll
            for (int c = 0; c < FA_HD; c += 32) {
              uint32_t v[32];
              tmem_ld32(v, my_o + c);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * factor);
              tmem_st32(my_o + c, v);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            fence_before();
          }
        }
        l_run *= factor;
        if (moves) m_ref = m_tile;
      }
      const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;  // a row without visible keys: exp2(-inf) = 0 all the same
      float part_sum[4] = {0.f, 0.f, 0.f, 0.f};
      // P goes into tensor memory as the A operand of P V, over the S that this thread has read: the row's lane, bfloat16
      // pairs of consecutive keys a column (the first half's P over columns of the first half, the second's likewise over
      // columns that the first half has left behind)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float (&row)[FA_KEYS / 2] = s[TILES == 2 ? 0 : half];
        if (TILES == 2) read_half(row, half);
        uint32_t packed[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float p0 = fa_exp2(fmaf(row[2 * i], scale_log2, neg_m));
          const float p1 = fa_exp2(fmaf(row[2 * i + 1], scale_log2, neg_m));
          part_sum[i & 3] += p0 + p1;
          __nv_bfloat162 pair = __floats2bfloat162_rn(p0, p1);
          packed[i] = *reinterpret_cast<uint32_t*>(&pair);
        }
        tmem_st32(my_s + half * 32, packed);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[s_place(j, u)]));
      l_run += (part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3]);
    }
    if (ok && n_tiles > 0) ok = mbar_wait(smem_u32(&o_done[u]), TILES == 1 ? (uint32_t)(n_tiles - 1) & 1u : 0u, abort_flag);
    if (ok && n_tiles > 0) {
      fence_after();
      if (sinks != nullptr) l_run += exp2f(sinks[head] * 1.4426950408889634f - m_ref);
      const float inv = row_live ? 1.0f / l_run : 0.f;
      __nv_bfloat16* dst = out + ((size_t)(tok0 + row) * n_heads + head) * FA_HD;
#pragma unroll
      for (int c = 0; c < FA_HD; c += 32) {
        uint32_t v[32];
        tmem_ld32(v, my_o + c);  // all lanes take part; rows beyond the sequence store nothing
        tmem_wait_ld();
        if (row_live) {
#pragma unroll
          for (int d = 0; d < 32; d += 8) {
            uint32_t packed[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              __nv_bfloat162 pair = __floats2bfloat162_rn(__uint_as_float(v[d + 2 * i]) * inv,
                                                          __uint_as_float(v[d + 2 * i + 1]) * inv);
              packed[i] = *reinterpret_cast<uint32_t*>(&pair);
            }
            *reinterpret_cast<uint4*>(dst + c + d) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
          }
        }
      }
      fence_before();
    }
    if (!ok && lane == 0) { *abort_flag = 1; if (error_flag != nullptr) atomicExch(error_flag, 5); }
  }

  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS));
  }
}

// Whether blocks of two query tiles take the step.  A two-tile block's step takes 1.6 to 1.8 times a one-tile block's, so two
// tiles a block are faster only while the blocks are many: not where the one-tile blocks all run at once (at most one a
// multiprocessor; measured, microseconds, one tile -> two: 128 new tokens of 32 heads behind 8,000 keys 82 -> 149, 2,000 tokens of
// 8 heads 27 -> 43, 512 of 32 heads 13.4 -> 18.4), nor where a long prompt's few blocks run at most about twice a
// multiprocessor, since its last tiles, which are the longest, then decide (2,000 tokens of 16 heads 31 -> 43, 1,024 of 32 heads
// 22.6 -> 26.7, 1,100 of 32 heads with a kv head each 24.7 -> 28.7; but 8 prompts of 128 tokens 16.4 -> 14.0, 600 tokens of 64
// heads, 2.2 a multiprocessor, 26.7 -> 20.6).  Consecutive tiles of one head share their keys only where every row begins
// at the first key: under a window or a chunk the second tile's steps would begin where the first's do, so that its sums could
// depend on the form (and there is nothing to gain: 4,000 tokens of 24 + 8 heads in a window of 1,024 88 either way).
static bool two_tiles(long long n_tokens, long long n_seqs, long long tiles, int n_heads, bool heads, bool bounded, int sms) {
  if (!heads && bounded) return false;
  if (tuning().prefill_tiles != 0) return tuning().prefill_tiles == 2;
  const long long most = n_tokens / FA_ROWS + n_seqs;  // of sequences of unequal lengths
  const long long blocks = (n_seqs * tiles < most ? n_seqs * tiles : most) * n_heads;
  return blocks > (tiles >= 5 ? 2 : 1) * (long long)sms;
}

// A map over a row-major bfloat16 matrix [rows, cols], boxes of box_rows x 64 columns, 128-byte swizzle.
static bool fa_make_map(CUtensorMap* map, const void* base, long long rows, int cols, int box_rows) {
  return sm100::make_map_bf16_2d(map, base, rows, cols, cols, box_rows);
}

template <int TILES, bool HEADS>
static int launch_prefill(dim3 grid, const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v,
                          __nv_bfloat16* out, const int* cu_seqlens, const int* seq_slot, const int* seq_start,
                          const int* block_table, int max_blocks, int n_heads, int n_kv_heads, float scale_log2,
                          int* error_flag, KeyRange range, const float* sinks, cudaStream_t stream) {
  constexpr auto kernel = attention_prefill_tcgen05_kernel<TILES, HEADS>;
  const cudaError_t err = allow_shared_memory_once<kernel>(FaShape<TILES>::SMEM);
  if (err != cudaSuccess) return (int)err;
  // launched without programmatic dependent launch: a block needs a multiprocessor to itself, so nothing of it can
  // run beside the kernel before it, and the early launch was measured slower (28.2 against 27.8 ms a prompt of 2,048)
  kernel<<<grid, FaShape<TILES>::THREADS, FaShape<TILES>::SMEM, stream>>>(
      map_q, map_k, map_v, out, cu_seqlens, seq_slot, seq_start, block_table, max_blocks, n_heads, n_kv_heads, scale_log2,
      error_flag, range, sinks);
  return launch_status();
}

}  // namespace xrt

// q, out: bfloat16 [n_tokens, n_heads * 128], the sequences' new tokens end to end (cu_seqlens[n_seqs + 1]);
// pools: bfloat16 [n_blocks, n_kv_heads, 64, 128]; seq_slot[n_seqs] (< 0: skipped), seq_start[n_seqs] = tokens each
// sequence held before this step; max_new = the most new tokens any sequence brings.  Head size 128 only.  `window` and `mask_chunk` bound
// the keys a query sees (KeyRange; 0 = no bound); sinks: float32 [n_heads] or null.
// error_flag (may be null) is set to 5 if a bounded wait ran out.
XRT_EXPORT int xrt_attention_prefill_tcgen05(void* out, const void* q, const void* k_pool, const void* v_pool,
                                             const int* cu_seqlens, const int* seq_slot, const int* seq_start,
                                             const int* block_table, int max_blocks, int n_blocks, int n_tokens,
                                             int n_seqs, int max_new, int n_heads, int n_kv_heads, int head_dim,
                                             float scale, int* error_flag, const float* sinks, int window,
                                             int mask_chunk, cudaStream_t stream) {
  if (n_seqs < 0 || max_new < 0 || n_tokens < 0 || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads != 0 ||
      n_blocks <= 0)
    return XRT_ERR_ARGUMENT;
  if (head_dim != xrt::FA_HD || n_seqs > 65535 || (max_new + xrt::FA_ROWS - 1) / xrt::FA_ROWS > 65535) return XRT_ERR_UNSUPPORTED;
  if (((uintptr_t)q & 15) || ((uintptr_t)k_pool & 15) || ((uintptr_t)v_pool & 15) || ((uintptr_t)out & 15))
    return XRT_ERR_UNSUPPORTED;
  if (n_seqs == 0 || max_new == 0 || n_tokens == 0) return XRT_OK;
  CUtensorMap map_q, map_k, map_v;
  const long long pool_rows = (long long)n_blocks * n_kv_heads * XRT_BLOCK_TOKENS;
  if (!xrt::fa_make_map(&map_q, q, n_tokens, n_heads * xrt::FA_HD, xrt::FA_ROWS) ||
      !xrt::fa_make_map(&map_k, k_pool, pool_rows, xrt::FA_HD, XRT_BLOCK_TOKENS) ||
      !xrt::fa_make_map(&map_v, v_pool, pool_rows, xrt::FA_HD, XRT_BLOCK_TOKENS))
    return XRT_ERR_UNSUPPORTED;
  const int tiles = (max_new + xrt::FA_ROWS - 1) / xrt::FA_ROWS;
  const bool heads = (n_heads / n_kv_heads) % 2 == 0;
  const bool two = xrt::two_tiles(n_tokens, n_seqs, tiles, n_heads, heads, window > 0 || mask_chunk > 0, xrt::multiprocessors());
  auto launch = two ? (heads ? xrt::launch_prefill<2, true> : xrt::launch_prefill<2, false>) : xrt::launch_prefill<1, false>;
  const dim3 grid(two && heads ? n_heads / 2 : n_heads, n_seqs, two && !heads ? (tiles + 1) / 2 : tiles);
  return launch(grid, map_q, map_k, map_v, (__nv_bfloat16*)out, cu_seqlens, seq_slot, seq_start, block_table, max_blocks,
                n_heads, n_kv_heads, scale * 1.4426950408889634f, error_flag, xrt::key_range(window, mask_chunk), sinks, stream);
}
