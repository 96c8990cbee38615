// The experts' products for steps of many tokens, bfloat16: rows sorted by expert (xrt_moe_group in moe.cu), ONE
// launch for all experts.  C[r] = A[r] . W_e^T for the rows r of expert e, with A [rows, K] and W [experts, N, K] both
// K-contiguous; on the fifth-generation tensor cores, with the pieces of gemm_tcgen05.cu's single blocks (TMA into a ring, one
// thread that issues tcgen05.mma, two accumulators in TMEM, four epilogue warps) over a walk that finds its tiles from
// the experts' row offsets on the device.
//   first product   N = 2 ff (an expert's gate rows, then its up rows): the block computes the gate columns and the
//                   matching up columns and writes act = g * sigmoid(alpha g) * (u + 1), g = min(gate, limit),
//                   u = clamp(up, -limit, limit), in bfloat16
//   second product  N = width: 32-bit results
//   first product of experts without a gate (MODE 2): N = ff, act = gelu(W_up h) with the exact (erf) gelu, bfloat16
//
// A persistent block a multiprocessor takes tiles of 128 rows of one expert x 256 of its weight rows (the first product of gated
// experts: 128 gate rows and the 128 matching up rows).  A tile's loads may reach into the next expert's rows or weights, or
// beyond the matrices (zeros): those rows and columns of the accumulator are never written.  Tiles are numbered expert
// after expert, inside an expert the row tiles of a column of tiles first, so that the weights of a column are read
// by neighbouring blocks at the same time.  A row's result does not depend on which other rows share its tile, nor on how
// many rows there are.
// Measured, microseconds, tiles of 64 x 64 with mma.sync (bound by their loads and ldmatrix, 180 to 250 TFLOP/s) -> this:
// 16 experts of 1,024 x 2,048, 250 rows each: gated first product 163 -> 74, second 97 -> 41 (410 TFLOP/s), gelu 109 -> 44;
// 4 rows each: 89 -> 49, 39 -> 14, 58 -> 22; 64 experts of 512, 250 rows each: 299 -> 110, 221 -> 97.  With 250 rows an expert
// the second of its two row tiles is all but full; what is left is the ramp of two or three tiles a block.
// Every wait is bounded as in gemm_tcgen05.cu.
#include "tcgen05.cuh"

namespace xrt {

using namespace sm100;

constexpr int MG_ROWS = 128, MG_COLS = 256, MG_BK = 64, MG_STAGES = 4, MG_THREADS = 192;
constexpr int MG_A_BYTES = MG_ROWS * MG_BK * 2, MG_STAGE_BYTES = 3 * MG_A_BYTES;
constexpr int MG_STAGING_BYTES = 4 * 32 * 33 * 4;
constexpr int MG_SMEM = MG_STAGES * MG_STAGE_BYTES + MG_STAGING_BYTES + 256 + 1024;

struct MoeTiles {
  const int* offsets;  // [experts + 1]
  void* out;
  int n_experts, n, k, ff;  // n weight rows an expert
  int col_tiles;
  float limit, alpha, up_shift;
};

// This block's tiles in turn.
struct MoeWalk {
  int tile, e, first;  // the next tile; the expert that the walk has come to, and the number of its first tile
  int row0, row1, row_tiles;
  __device__ void expert(const MoeTiles& g) {
    row0 = g.offsets[e];
    row1 = g.offsets[e + 1];
    row_tiles = (row1 - row0 + MG_ROWS - 1) / MG_ROWS;
  }
  __device__ void begin(const MoeTiles& g) {
    tile = blockIdx.x;
    e = first = 0;
    expert(g);
  }
  // the place of tile `tile`: rows row .. of expert e, column tile col; false if there are no more tiles
  __device__ bool place(const MoeTiles& g, int& row, int& col) {
    while (e < g.n_experts && tile >= first + row_tiles * g.col_tiles) {
      first += row_tiles * g.col_tiles;
      if (++e < g.n_experts) expert(g);
    }
    if (e >= g.n_experts) return false;
    const int inside = tile - first;
    col = inside / row_tiles;
    row = row0 + (inside - col * row_tiles) * MG_ROWS;
    return true;
  }
};

// Columns col .. col + 3 of a row of n, those beyond it left out; in one piece where it is aligned.
template <typename T>
__device__ __forceinline__ void store_four(T* row, int col, int n, const float* src) {
  T* dst = row + col;
  if (col + 3 < n && (reinterpret_cast<uintptr_t>(dst) & (4 * sizeof(T) - 1)) == 0) {
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(dst) = make_float4(src[0], src[1], src[2], src[3]);
    } else {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(src[0], src[1]), hi = __floats2bfloat162_rn(src[2], src[3]);
      *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (col + e < n) dst[e] = from_float<T>(src[e]);
  }
}

// MODE 0: second product, 32-bit results; 1: first product of gated experts; 2: first product of experts without a gate.
template <int MODE>
__global__ void __launch_bounds__(MG_THREADS, 1)
moe_grouped_product_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                           const MoeTiles g, int* __restrict__ error_flag) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* staging = reinterpret_cast<float*>(smem + MG_STAGES * MG_STAGE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + MG_STAGES * MG_STAGE_BYTES + MG_STAGING_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + MG_STAGES;
  uint64_t* acc_full = bars + 2 * MG_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  constexpr int COLS = MODE == 1 ? MG_COLS / 2 : MG_COLS;  // output columns a tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slabs = (g.k + MG_BK - 1) / MG_BK;
  const int out_cols = MODE == 1 ? g.ff : g.n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MG_STAGES; ++s) { mbar_init(smem_u32(&full[s]), 1); mbar_init(smem_u32(&empty[s]), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(smem_u32(&acc_full[a]), 1); mbar_init(smem_u32(&acc_empty[a]), 128); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * MG_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = *tmem_slot;
  MoeWalk walk;
  walk.begin(g);
  int row, col;
  bool ok = true;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (lane == 0) {
      int it = 0;
      for (; ok && walk.place(g, row, col); walk.tile += gridDim.x) {
        const int w0 = walk.e * g.n + col * COLS, w1 = MODE == 1 ? w0 + g.ff : w0 + 128;
        for (int kb = 0; kb < slabs; ++kb, ++it) {
          const int s = it % MG_STAGES;
          ok = mbar_wait(smem_u32(&empty[s]), ((it / MG_STAGES) & 1) ^ 1, abort_flag);
          if (!ok) break;
          const uint32_t bar = smem_u32(&full[s]), dst = smem_u32(smem + s * MG_STAGE_BYTES);
          mbar_arrive_expect_tx(bar, MG_STAGE_BYTES);
          tma_load_2d(dst, &map_a, kb * MG_BK, row, bar);
          tma_load_2d(dst + MG_A_BYTES, &map_w, kb * MG_BK, w0, bar);
          tma_load_2d(dst + 2 * MG_A_BYTES, &map_w, kb * MG_BK, w1, bar);
        }
      }
      if (!ok) { *abort_flag = 1; if (error_flag != nullptr) atomicExch(error_flag, 3); }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issue
    if (lane == 0) {
      constexpr uint32_t idesc = instr_desc(MG_ROWS, MG_COLS);
      int it = 0, tile_i = 0;
      for (; ok && walk.place(g, row, col); walk.tile += gridDim.x, ++tile_i) {
        const int a = tile_i & 1;
        ok = mbar_wait(smem_u32(&acc_empty[a]), ((tile_i >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        fence_after();
        for (int i = 0; i < slabs; ++i, ++it) {
          const int s = it % MG_STAGES;
          ok = mbar_wait(smem_u32(&full[s]), (it / MG_STAGES) & 1, abort_flag);
          if (!ok) break;
          fence_after();
          const uint64_t desc_a = desc_k_major(smem_u32(smem + s * MG_STAGE_BYTES));
          const uint64_t desc_b = desc_k_major(smem_u32(smem + s * MG_STAGE_BYTES + MG_A_BYTES));
#pragma unroll
          for (int k = 0; k < MG_BK / 16; ++k)
            mma_f16(tmem_base + a * MG_COLS, desc_a + 2 * k, desc_b + 2 * k, idesc, (i | k) != 0);
          commit(smem_u32(&empty[s]));
        }
        if (ok) commit(smem_u32(&acc_full[a]));
      }
      if (!ok) { *abort_flag = 1; if (error_flag != nullptr) atomicExch(error_flag, 3); }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3;
    float* patch = staging + (warp - 2) * 32 * 33;  // a 32 x 32 patch of the tile, turned around so that stores are whole lines
    int tile_i = 0;
    for (; ok && walk.place(g, row, col); walk.tile += gridDim.x, ++tile_i) {
      const int a = tile_i & 1, row_end = walk.row1;
      ok = mbar_wait(smem_u32(&acc_full[a]), (tile_i >> 1) & 1, abort_flag);
      if (!ok) break;
      fence_after();
      const uint32_t tmem_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + a * MG_COLS;
      // Rows beyond the expert's and columns beyond the matrix are left out.  (A row of zeros, beyond the last expert, takes the
      // division's slow way, and its warp with it: gated, 3 experts of 64 x 128 with 8 rows each 31 us, of which 20 for that.)
      const int row0 = row + quarter * 32;  // the warp's first row
      const bool live = row0 + lane < row_end;
      const int cols = row0 < row_end ? min(COLS, out_cols - col * COLS) : 0;
#pragma unroll 1
      for (int c = 0; c < cols; c += 32) {
        uint32_t v[32];
        tmem_ld32(v, tmem_row + c);
        if (MODE == 1) {
          uint32_t u[32];
          tmem_ld32(u, tmem_row + MG_COLS / 2 + c);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float gate = live ? fminf(__uint_as_float(v[j]), g.limit) : 1.0f;
            const float up = fminf(fmaxf(__uint_as_float(u[j]), -g.limit), g.limit);
            patch[lane * 33 + j] = gate / (1.0f + expf(-g.alpha * gate)) * (up + g.up_shift);
          }
        } else {
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float x = __uint_as_float(v[j]);
            patch[lane * 33 + j] = MODE == 2 ? 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)) : x;
          }
        }
        __syncwarp();
        // four rows at a time, eight lanes a row, four neighbouring columns a lane
        const int out_col = col * COLS + c + (lane & 7) * 4;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int r = it * 4 + (lane >> 3), out_row = row0 + r;
          const float* src = patch + r * 33 + (lane & 7) * 4;
          if (out_row >= row_end) continue;
          if (MODE == 0) store_four(reinterpret_cast<float*>(g.out) + (size_t)out_row * out_cols, out_col, out_cols, src);
          else store_four(reinterpret_cast<__nv_bfloat16*>(g.out) + (size_t)out_row * out_cols, out_col, out_cols, src);
        }
        __syncwarp();
      }
      fence_before();
      mbar_arrive(smem_u32(&acc_empty[a]));
    }
    if (!ok && lane == 0) { *abort_flag = 1; if (error_flag != nullptr) atomicExch(error_flag, 3); }
  }

  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * MG_COLS));
  }
}

template <int MODE>
static int launch_moe_grouped(const CUtensorMap& map_a, const CUtensorMap& map_w, const MoeTiles& g, int blocks, int* error_flag,
                              cudaStream_t stream) {
  const cudaError_t err = allow_shared_memory_once<moe_grouped_product_kernel<MODE>>(MG_SMEM);
  if (err != cudaSuccess) return (int)err;
  launch_kernel_alone(moe_grouped_product_kernel<MODE>, dim3(blocks), dim3(MG_THREADS), (size_t)MG_SMEM, stream, map_a, map_w, g,
                      error_flag);
  return launch_status();
}

}  // namespace xrt

// first == 2: act [rows, n] bfloat16 = gelu(a . w^T) from w [experts, n, k] (experts without a gate).
// first == 3: as first == 1 with act = silu(gate) * up.
// first == 1: act [rows, ff] bfloat16 from a [rows, k] and w [experts, 2 ff, k]; else out [rows, n] float32 from
// a [rows, k] and w [experts, n, k].  offsets [experts + 1] int32 on the device; `rows` is their last entry's bound
// (the number of (token, choice) pairs).  k must be a multiple of 8 and the bases 16-byte aligned.  error_flag (may be null) is
// set to 3 if a bounded wait ran out.
XRT_EXPORT int xrt_moe_grouped_product(void* out, const void* a, const void* w, const int* offsets, int rows, int n_experts,
                                       int n, int k, int ff, float limit, float alpha, int first, int* error_flag,
                                       cudaStream_t stream) {
  float up_shift = 1.0f;
  if (first == 3) {  // gated silu experts: the gated form without limits and without the one added to the up rows
    first = 1;
    limit = INFINITY;
    alpha = 1.0f;
    up_shift = 0.0f;
  }
  if (rows < 0 || n_experts <= 0 || n <= 0 || k <= 0 || (first == 1 && (ff <= 0 || n != 2 * ff))) return XRT_ERR_ARGUMENT;
  if (k % 8 || (((uintptr_t)a | (uintptr_t)w) & 15)) return XRT_ERR_UNSUPPORTED;
  if (rows == 0) return XRT_OK;
  const int sms = xrt::multiprocessors();
  if (sms <= 0) return XRT_ERR_UNSUPPORTED;
  CUtensorMap map_a, map_w;
  if (!xrt::sm100::make_map_bf16_2d(&map_a, a, rows, k, k, xrt::MG_ROWS) ||
      !xrt::sm100::make_map_bf16_2d(&map_w, w, (long long)n_experts * n, k, k, 128))
    return XRT_ERR_UNSUPPORTED;
  xrt::MoeTiles g;
  g.offsets = offsets; g.out = out; g.n_experts = n_experts; g.n = n; g.k = k; g.ff = ff;
  g.limit = limit; g.alpha = alpha; g.up_shift = up_shift;
  const int cols = first == 1 ? ff : n, per_tile = first == 1 ? xrt::MG_COLS / 2 : xrt::MG_COLS;
  g.col_tiles = (cols + per_tile - 1) / per_tile;
  // every expert may leave one tile partly empty
  const long long tiles = ((long long)rows / xrt::MG_ROWS + n_experts) * g.col_tiles;
  const int blocks = tiles < sms ? (int)tiles : sms;
  if (first == 1) return xrt::launch_moe_grouped<1>(map_a, map_w, g, blocks, error_flag, stream);
  if (first == 2) return xrt::launch_moe_grouped<2>(map_a, map_w, g, blocks, error_flag, stream);
  return xrt::launch_moe_grouped<0>(map_a, map_w, g, blocks, error_flag, stream);
}
