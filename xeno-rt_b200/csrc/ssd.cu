// A state-space recurrence with ONE scalar decay per head and token (the "state-space duality" form), and the
// gated group norm that follows it.  Everything here is 32-bit: step sizes, decays, the state, the norm.
//
//   step size   dt_t = softplus(raw_t + dt_bias[h])                      (no clamp)
//   scan        S_t = exp(-exp(a_log[h]) dt_t) S_(t-1) + dt_t b_t x_t^T,   y_t = S_t^T c_t + d_skip[h] x_t
//               S is [state, vdim] per head; b and c belong to the head's group (n_heads / n_groups heads share them)
//   group norm  v = y * silu(z); every one of `groups` equal stretches of the row is divided by its own root mean
//               square; times a weight
//
// A sequence is a row of the step's cu_seqlens / seq_slot arrays; a row with slot -1 or no tokens is skipped, so
// padding rows of a captured step leave every state alone.  The state is kept [slot][head][vdim][state]: a column
// of S is contiguous.  A token's arithmetic is the same whether it comes alone or inside a prompt, so results do
// not depend on how a sequence was cut into steps.
#include "recurrence.cuh"

namespace xrt {

struct SsdArgs {
  float* out;                       // [T, heads * vdim]
  const float *x, *b, *c, *dt;      // rows of x_stride / bc_stride / dt_stride floats
  int x_stride, bc_stride, dt_stride;
  const float *dt_bias, *a_log, *d_skip;  // [heads]
  float* state;                     // [slots, heads, vdim, state]
  const int *cu_seqlens, *seq_slot;
  int n_heads, heads_per_group, n_state, vdim;
  int parts, cols, tile_tokens;
  int zero_padding;  // rows beyond the step's tokens, one a sequence that brings none, are cleared (single tokens only)
};

// One block: one sequence, one head, `cols` value columns.  A column's state (n_state rows) is held in registers by
// `parts` neighbouring lanes, R rows each (which rows: `row_of` in the kernel; rows beyond n_state stay zero);
// the read-out's sum over rows is finished by a butterfly among those lanes, so its order is fixed.  Tiles of
// `tile_tokens` tokens' b, c, x and raw step sizes are brought into shared memory by cp.async, two tiles in flight:
// the next tile lands while this one is worked on.
// VEC: 16-byte copies (n_state, cols, vdim and every row stride are multiples of 4 floats, every base 16-byte aligned).
template <int R, bool VEC>
__global__ void __launch_bounds__(128) ssd_scan_kernel(const SsdArgs a) {
  extern __shared__ __align__(16) float tile[];
  pdl_trigger();
  const int parts = a.parts, cols = a.cols, TT = a.tile_tokens, n_state = a.n_state, vdim = a.vdim;
  const int padded = parts * R;
  // a stage: b | c, each [TT][padded]; x [TT][cols]; raw step sizes [TT] (padded to 4); then step size and decay [TT] each
  const int stage_floats = 2 * TT * padded + TT * cols + ((TT + 3) & ~3);
  float* sdt = tile + 2 * stage_floats;
  float* sdecay = sdt + TT;
  if (padded != n_state || vdim % cols != 0)  // rows and columns beyond the head's stay zero
    for (int e = threadIdx.x; e < 2 * stage_floats; e += blockDim.x) tile[e] = 0.f;
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y;
  const int slot = a.seq_slot[s];
  const int begin = a.cu_seqlens[s], end = a.cu_seqlens[s + 1];
  if (slot < 0 || end <= begin) {
    if (a.zero_padding && s >= a.cu_seqlens[gridDim.x])
      for (int c = blockIdx.z * cols + threadIdx.x; c < min((int)(blockIdx.z + 1) * cols, vdim); c += blockDim.x)
        a.out[((size_t)s * a.n_heads + h) * vdim + c] = 0.f;
    return;
  }
  __syncthreads();
  const int part = threadIdx.x % parts, jl = threadIdx.x / parts;
  const int col0 = blockIdx.z * cols, j = col0 + jl;
  const int g = h / a.heads_per_group;
  const bool live = j < vdim;
  const float rate = expf(a.a_log[h]), dt_bias = a.dt_bias[h], d_skip = a.d_skip[h];
  constexpr int B = VEC ? 16 : 4, E = VEC ? 4 : 1;
  // the lane's i-th row: with four rows or more a lane, every parts-th group of four (the lanes of a column then read
  // neighbouring 16 bytes of b, c and the state: whole lines, all banks), else R neighbouring rows
  auto row_of = [&](int i) { return R % 4 == 0 ? 4 * ((i >> 2) * parts + part) + (i & 3) : part * R + i; };

  auto issue = [&](int t0, int stage) {
    float* sb = tile + stage * stage_floats;
    float* sc = sb + TT * padded;
    float* sx = sc + TT * padded;
    float* sraw = sx + TT * cols;
    const int nt = min(TT, end - t0);
    const int per = n_state / E;
    if (blockDim.x % per == 0) {  // a thread keeps its piece of the row and steps down the tokens: no division a copy
      const int d = (threadIdx.x % per) * E;
      for (int tt = threadIdx.x / per; tt < nt; tt += blockDim.x / per) {
        const size_t at = (size_t)(t0 + tt) * a.bc_stride + g * n_state + d;
        cp_async<B>(sb + tt * padded + d, a.b + at);
        cp_async<B>(sc + tt * padded + d, a.c + at);
      }
    } else {
      for (int e = threadIdx.x; e < nt * per; e += blockDim.x) {
        const int tt = e / per, d = (e - tt * per) * E;
        const size_t at = (size_t)(t0 + tt) * a.bc_stride + g * n_state + d;
        cp_async<B>(sb + tt * padded + d, a.b + at);
        cp_async<B>(sc + tt * padded + d, a.c + at);
      }
    }
    const int xper = cols / E;
    for (int e = threadIdx.x; e < nt * xper; e += blockDim.x) {
      const int tt = e / xper, cc = (e - tt * xper) * E;
      if (col0 + cc < vdim) cp_async<B>(sx + tt * cols + cc, a.x + (size_t)(t0 + tt) * a.x_stride + h * vdim + col0 + cc);
    }
    for (int tt = threadIdx.x; tt < nt; tt += blockDim.x)
      cp_async<4>(sraw + tt, a.dt + (size_t)(t0 + tt) * a.dt_stride + h);
    cp_async_commit();
  };

  float S[R];
  float* sp = a.state + (((size_t)slot * a.n_heads + h) * vdim + j) * n_state;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = row_of(i);
    S[i] = (live && row < n_state) ? sp[row] : 0.f;
  }
  issue(begin, 0);
  int stage = 0;
  for (int t0 = begin; t0 < end; t0 += TT, stage ^= 1) {
    const int nt = min(TT, end - t0);
    if (t0 + TT < end) {
      issue(t0 + TT, stage ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float* sb = tile + stage * stage_floats;
    const float* sc = sb + TT * padded;
    const float* sx = sc + TT * padded;
    const float* sraw = sx + TT * cols;
    for (int tt = threadIdx.x; tt < nt; tt += blockDim.x) {
      const float z = sraw[tt] + dt_bias;
      const float dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
      sdt[tt] = dt;
      sdecay[tt] = expf(-rate * dt);
    }
    __syncthreads();
#pragma unroll 4
    for (int tt = 0; tt < nt; ++tt) {
      const float xv = sx[tt * cols + jl];
      const float decay = sdecay[tt], u = sdt[tt] * xv;
      float bt[R], ct[R];
      if (R % 4 == 0) {  // a lane's rows of b and c as whole 16 bytes
#pragma unroll
        for (int i = 0; i < R; i += 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(sb + tt * padded + row_of(i));
          const float4 c4 = *reinterpret_cast<const float4*>(sc + tt * padded + row_of(i));
          bt[i] = b4.x; bt[i + 1] = b4.y; bt[i + 2] = b4.z; bt[i + 3] = b4.w;
          ct[i] = c4.x; ct[i + 1] = c4.y; ct[i + 2] = c4.z; ct[i + 3] = c4.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i) {
          bt[i] = sb[tt * padded + part * R + i];
          ct[i] = sc[tt * padded + part * R + i];
        }
      }
      float y0 = 0.f, y1 = 0.f;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        S[i] = fmaf(decay, S[i], u * bt[i]);
        if (i & 1) y1 = fmaf(S[i], ct[i], y1);
        else y0 = fmaf(S[i], ct[i], y0);
      }
      float y = y0 + y1;
      for (int o = parts >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      if (part == 0 && live) a.out[(size_t)(t0 + tt) * a.n_heads * vdim + h * vdim + j] = fmaf(d_skip, xv, y);
    }
    __syncthreads();  // the stage is written again by the copies of the tile after the next
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = row_of(i);
    if (live && row < n_state) sp[row] = S[i];
  }
}

// The scan of prompts whose state has 128 rows: 16 lanes a column of the state as above, 8 rows each, but C2 neighbouring
// columns a lane.  The kernel above is bound by shared memory (every lane reads 8 bytes of b and c for each element of the
// state and token; a multiprocessor delivers 128 bytes a clock) and by its butterflies; here what a lane reads serves C2
// columns, the multiply-adds are the packed 2 x fp32 ones, and the read-outs of four tokens are summed over the lanes
// together (lane_sums).  Each sum has the same terms in the same order as above, so a token's result is the same bit for
// bit.  A ring of SSD_STAGES tiles of SSD_TOKENS tokens is filled by cp.async.
// Measured, microseconds, the kernel above -> this one, 64 heads of 64 x 128: one prompt of 2,000 tokens 719 -> 319, prompts of
// 1,000 and 1,100 tokens 741 -> 271, 16 of 300 1,230 -> 406.  At two columns a lane shared memory was 78 percent busy (301 us for
// the two prompts).
constexpr int SSD_TOKENS = 16, SSD_STAGES = 3, SSD_GROUP = 4;

template <int C2>
__global__ void __launch_bounds__(128) ssd_scan_wide_kernel(const SsdArgs a) {
  constexpr int PARTS = 16, ROWS = 128, COLS = 128 / PARTS * C2, TT = SSD_TOKENS;
  constexpr int STAGE = 2 * TT * ROWS + TT * COLS + TT;  // b | c, each [TT][ROWS]; x [TT][COLS]; raw step sizes [TT]
  extern __shared__ __align__(16) float tile[];
  __shared__ float sdt[TT], sdecay[TT];
  pdl_trigger();
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * COLS;
  const int slot = a.seq_slot[s];
  const int begin = a.cu_seqlens[s], end = a.cu_seqlens[s + 1];
  if (slot < 0 || end <= begin) return;
  const int vdim = a.vdim;
  const int part = threadIdx.x % PARTS, jl = (threadIdx.x / PARTS) * C2, j = col0 + jl;
  const int g = h / a.heads_per_group;
  const float rate = expf(a.a_log[h]), dt_bias = a.dt_bias[h], d_skip = a.d_skip[h];

  auto issue = [&](int t0, int stage) {
    float* sb = tile + stage * STAGE;
    const int nt = min(TT, end - t0);
    const int d = (threadIdx.x % 32) * 4;
    for (int tt = threadIdx.x / 32; tt < nt; tt += 4) {
      const size_t at = (size_t)(t0 + tt) * a.bc_stride + g * ROWS + d;
      cp_async<16>(sb + tt * ROWS + d, a.b + at);
      cp_async<16>(sb + TT * ROWS + tt * ROWS + d, a.c + at);
    }
    constexpr int XPER = COLS / 4;
    const int c = (threadIdx.x % XPER) * 4;
    if (col0 + c < vdim)
      for (int tt = threadIdx.x / XPER; tt < nt; tt += 128 / XPER)
        cp_async<16>(sb + 2 * TT * ROWS + tt * COLS + c, a.x + (size_t)(t0 + tt) * a.x_stride + h * vdim + col0 + c);
    if ((int)threadIdx.x < nt)
      cp_async<4>(sb + 2 * TT * ROWS + TT * COLS + threadIdx.x, a.dt + (size_t)(t0 + threadIdx.x) * a.dt_stride + h);
  };

  float2 S[C2][4];
  float* sp = a.state + (((size_t)slot * a.n_heads + h) * vdim + j) * ROWS;
#pragma unroll
  for (int c = 0; c < C2; ++c)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j + c < vdim) t = *reinterpret_cast<const float4*>(sp + (size_t)c * ROWS + 4 * (i * PARTS + part));
      S[c][2 * i] = make_float2(t.x, t.y);
      S[c][2 * i + 1] = make_float2(t.z, t.w);
    }

  // one token: its write into the state; `read` gets this lane's part of what the token reads, column by column
  auto token = [&](const float* sb, int tt, float (&read)[C2]) {
    const float4* pb = reinterpret_cast<const float4*>(sb + tt * ROWS) + part;
    const float4* pc = reinterpret_cast<const float4*>(sb + TT * ROWS + tt * ROWS) + part;
    const float4 b0 = pb[0], b1 = pb[PARTS], c0 = pc[0], c1 = pc[PARTS];
    const float2 bb[4] = {{b0.x, b0.y}, {b0.z, b0.w}, {b1.x, b1.y}, {b1.z, b1.w}};
    const float2 cc[4] = {{c0.x, c0.y}, {c0.z, c0.w}, {c1.x, c1.y}, {c1.z, c1.w}};
    const float dt = sdt[tt], decay = sdecay[tt];
    const float* sx = sb + 2 * TT * ROWS + tt * COLS + jl;
    float xv[C2];
    if constexpr (C2 == 4) {
      const float4 x4 = *reinterpret_cast<const float4*>(sx);
      xv[0] = x4.x; xv[1] = x4.y; xv[2] = x4.z; xv[3] = x4.w;
    } else {
#pragma unroll
      for (int c = 0; c < C2; ++c) xv[c] = sx[c];
    }
#pragma unroll
    for (int c = 0; c < C2; ++c) {
      const float u = dt * xv[c];
      float2 y = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        S[c][i] = __ffma2_rn(make_float2(decay, decay), S[c][i], __fmul2_rn(make_float2(u, u), bb[i]));
        y = __ffma2_rn(S[c][i], cc[i], y);
      }
      read[c] = y.x + y.y;
    }
  };
  // sum number `value` of a group of tokens that begins at place tt of the tile belongs to this lane
  auto store = [&](const float* sb, int t0, int tt, int value, int per_value, float sum) {
    const int at = tt + value / C2, c = value % C2;
    if (part % per_value == 0 && j + c < vdim)
      a.out[(size_t)(t0 + at) * a.n_heads * vdim + h * vdim + j + c] = fmaf(d_skip, sb[2 * TT * ROWS + at * COLS + jl + c], sum);
  };

  const int n_tiles = (end - begin + TT - 1) / TT;
  for (int p = 0; p < SSD_STAGES - 1; ++p) {
    if (p < n_tiles) issue(begin + p * TT, p);
    cp_async_commit();
  }
  for (int tile_i = 0; tile_i < n_tiles; ++tile_i) {
    const int t0 = begin + tile_i * TT, nt = min(TT, end - t0);
    cp_async_wait<SSD_STAGES - 2>();
    const float* sb = tile + (tile_i % SSD_STAGES) * STAGE;
    __syncthreads();  // the tile is there, and everybody has left the tile before it
    if ((int)threadIdx.x < nt) {
      const float dt = softplusf_(sb[2 * TT * ROWS + TT * COLS + threadIdx.x] + dt_bias);
      sdt[threadIdx.x] = dt;
      sdecay[threadIdx.x] = expf(-rate * dt);
    }
    if (tile_i + SSD_STAGES - 1 < n_tiles) issue(t0 + (SSD_STAGES - 1) * TT, (tile_i + SSD_STAGES - 1) % SSD_STAGES);
    cp_async_commit();
    __syncthreads();
    int tt = 0;
#pragma unroll 1
    for (; tt + SSD_GROUP <= nt; tt += SSD_GROUP) {
      float read[SSD_GROUP * C2];
#pragma unroll
      for (int i = 0; i < SSD_GROUP; ++i) {
        float one[C2];
        token(sb, tt + i, one);
#pragma unroll
        for (int c = 0; c < C2; ++c) read[i * C2 + c] = one[c];
      }
      const float sum = lane_sums<PARTS>(read, part);
      store(sb, t0, tt, part * (SSD_GROUP * C2) / PARTS, PARTS / (SSD_GROUP * C2), sum);
    }
#pragma unroll 1
    for (; tt < nt; ++tt) {
      float read[C2];
      token(sb, tt, read);
      store(sb, t0, tt, part * C2 / PARTS, PARTS / C2, lane_sums<PARTS>(read, part));
    }
  }
#pragma unroll
  for (int c = 0; c < C2; ++c)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (j + c < vdim)
        *reinterpret_cast<float4*>(sp + (size_t)c * ROWS + 4 * (i * PARTS + part)) =
            make_float4(S[c][2 * i].x, S[c][2 * i].y, S[c][2 * i + 1].x, S[c][2 * i + 1].y);
}

template <int C2>
int launch_ssd_scan_wide(const SsdArgs& a, int n_seqs, cudaStream_t stream) {
  constexpr int COLS = 8 * C2;
  constexpr size_t smem = (size_t)SSD_STAGES * (2 * SSD_TOKENS * 128 + SSD_TOKENS * COLS + SSD_TOKENS) * sizeof(float);
  const cudaError_t err = allow_shared_memory_once<ssd_scan_wide_kernel<C2>>((int)smem);
  if (err != cudaSuccess) return (int)err;
  launch_kernel_alone(ssd_scan_wide_kernel<C2>, dim3(n_seqs, a.n_heads, (a.vdim + COLS - 1) / COLS), dim3(128), smem, stream, a);
  return launch_status();
}

// v = y * silu(z); each of `groups` stretches of the row by its own root mean square; times w.  One block a
// (token, group).  A row's numbers are all asked for at once (PER a thread, the weights before the wait) and v is kept: the
// kernel is a chain of latencies in a decode step (alone, the loop over memory below -> this: 4 tokens of 2 x 2,048 5.2 -> 2.2 us, of
// 2 x 4,096 9.1 -> 3.2; 4,000 tokens of 2 x 2,048 66 -> 43).
template <typename TO, int PER>
__global__ void __launch_bounds__(256)
gated_group_norm_rows_kernel(TO* __restrict__ out, const float* __restrict__ y, const float* __restrict__ z, int z_stride,
                             const float* __restrict__ w, int width, int groups, float eps) {
  __shared__ float scratch[33];
  pdl_trigger();
  const int t = blockIdx.x, g = blockIdx.y;
  const int per = width / groups;
  float wv[PER], v[PER], zv[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    wv[i] = c < per ? w[g * per + c] : 0.f;
  }
  pdl_wait(y, z, w);
  const float* yr = y + (size_t)t * width + g * per;
  const float* zr = z + (size_t)t * z_stride + g * per;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    v[i] = c < per ? yr[c] : 0.f;
    zv[i] = c < per ? zr[c] : 0.f;
  }
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    v[i] *= zv[i] / (1.0f + expf(-zv[i]));
    acc = fmaf(v[i], v[i], acc);
  }
  const float inv = 1.0f / sqrtf(block_sum(acc, scratch) / (float)per + eps);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < per) out[(size_t)t * width + g * per + c] = from_float<TO>((v[i] * inv) * wv[i]);
  }
}

// stretches of any length
template <typename TO>
__global__ void gated_group_norm_kernel(TO* __restrict__ out, const float* __restrict__ y, const float* __restrict__ z,
                                        int z_stride, const float* __restrict__ w, int width, int groups, float eps) {
  __shared__ float scratch[33];
  pdl_trigger();
  pdl_wait(y, z, w);
  const int t = blockIdx.x, g = blockIdx.y;
  const int per = width / groups;
  const float* yr = y + (size_t)t * width + g * per;
  const float* zr = z + (size_t)t * z_stride + g * per;
  float acc = 0.f;
  for (int c = threadIdx.x; c < per; c += blockDim.x) {
    const float zv = zr[c];
    const float v = yr[c] * (zv / (1.0f + expf(-zv)));
    acc = fmaf(v, v, acc);
  }
  const float inv = 1.0f / sqrtf(block_sum(acc, scratch) / (float)per + eps);
  for (int c = threadIdx.x; c < per; c += blockDim.x) {
    const float zv = zr[c];
    const float v = yr[c] * (zv / (1.0f + expf(-zv)));
    out[(size_t)t * width + g * per + c] = from_float<TO>((v * inv) * w[g * per + c]);
  }
}

}  // namespace xrt

// out [T, heads * vdim] float32.  x: rows holding heads * vdim floats; b, c: rows holding groups * n_state floats (one
// stride for both); dt: rows holding one raw step size a head.  state: [slots, heads, vdim, n_state].
XRT_EXPORT int xrt_ssd_scan(float* out, const float* x, int x_stride, const float* b, const float* c, int bc_stride,
                            const float* dt, int dt_stride, const float* dt_bias, const float* a_log, const float* d_skip,
                            float* state, const int* cu_seqlens, const int* seq_slot, int n_seqs, int n_heads,
                            int n_groups, int n_state, int vdim, int max_new, int zero_padding, cudaStream_t stream) {
  if (n_seqs < 0 || n_heads <= 0 || n_groups <= 0 || n_heads % n_groups || n_state <= 0 || vdim <= 0) return XRT_ERR_ARGUMENT;
  if (n_state > 512 || n_seqs > 65535 || n_heads > 65535) return XRT_ERR_UNSUPPORTED;
  if (n_seqs == 0) return XRT_OK;
  if (max_new < 1) max_new = 1 << 30;
  int r = 1;
  while (r < 16 && (n_state + r - 1) / r > 16) r *= 2;  // rows a lane: 16 lanes a column where the state allows
  int parts = 1;
  while (parts * r < n_state) parts *= 2;
  if (parts > 32) return XRT_ERR_UNSUPPORTED;
  xrt::SsdArgs a;
  a.out = out; a.x = x; a.b = b; a.c = c; a.dt = dt;
  a.x_stride = x_stride; a.bc_stride = bc_stride; a.dt_stride = dt_stride;
  a.dt_bias = dt_bias; a.a_log = a_log; a.d_skip = d_skip;
  a.state = state; a.cu_seqlens = cu_seqlens; a.seq_slot = seq_slot;
  a.n_heads = n_heads; a.heads_per_group = n_heads / n_groups; a.n_state = n_state; a.vdim = vdim;
  a.parts = parts;
  a.zero_padding = zero_padding != 0 && max_new == 1;
  int threads = 128;
  while (threads > 32 && threads / parts >= 2 * vdim) threads /= 2;  // no more lanes than the columns need
  a.cols = threads / parts;
  a.tile_tokens = max_new < 16 ? max_new : 16;
  auto floats = [&](int tt) { return (size_t)2 * (2 * tt * parts * r + tt * a.cols + ((tt + 3) & ~3)) + 2 * tt; };
  while (a.tile_tokens > 1 && floats(a.tile_tokens) * sizeof(float) > 44 * 1024) a.tile_tokens /= 2;
  const size_t smem = floats(a.tile_tokens) * sizeof(float);
  const bool vec = n_state % 4 == 0 && a.cols % 4 == 0 && vdim % 4 == 0 && x_stride % 4 == 0 && bc_stride % 4 == 0 &&
                   (((uintptr_t)x | (uintptr_t)b | (uintptr_t)c) & 15) == 0;
  if (max_new > 1 && vec && n_state == 128 && ((uintptr_t)state & 15) == 0) {
    // four columns a lane where their blocks still reach two thirds of the multiprocessors, two else
    if (3ll * n_seqs * n_heads * ((vdim + 31) / 32) >= 2ll * xrt::multiprocessors()) return xrt::launch_ssd_scan_wide<4>(a, n_seqs, stream);
    return xrt::launch_ssd_scan_wide<2>(a, n_seqs, stream);
  }
  dim3 grid(n_seqs, n_heads, (vdim + a.cols - 1) / a.cols);
#define XRT_SSD(R)                                                                                              \
  do {                                                                                                                 \
    if (max_new > 1 && vec) xrt::launch_kernel_alone(xrt::ssd_scan_kernel<R, true>, grid, dim3(threads), smem, stream, a); \
    else if (max_new > 1) xrt::launch_kernel_alone(xrt::ssd_scan_kernel<R, false>, grid, dim3(threads), smem, stream, a);  \
    else if (vec) xrt::launch_kernel(xrt::ssd_scan_kernel<R, true>, grid, dim3(threads), smem, stream, a);               \
    else xrt::launch_kernel(xrt::ssd_scan_kernel<R, false>, grid, dim3(threads), smem, stream, a);                       \
  } while (0)
  if (r == 1) XRT_SSD(1);
  else if (r == 2) XRT_SSD(2);
  else if (r == 4) XRT_SSD(4);
  else if (r == 8) XRT_SSD(8);
  else XRT_SSD(16);
#undef XRT_SSD
  return xrt::launch_status();
}

XRT_EXPORT int xrt_gated_group_norm(void* out, const float* y, const float* z, int z_stride, const float* weight,
                                    int n_tokens, int width, int groups, float eps, int out_dtype, cudaStream_t stream) {
  if (n_tokens < 0 || width <= 0 || groups <= 0 || width % groups || z_stride < width) return XRT_ERR_ARGUMENT;
  if (n_tokens == 0) return XRT_OK;
  if (groups > 65535) return XRT_ERR_UNSUPPORTED;
  const int per = width / groups;
  const int threads = per >= 1024 ? 256 : (per >= 256 ? 128 : 64);
  XRT_DISPATCH_DTYPE(out_dtype, TO, {
    // no more numbers a thread than a stretch has: with room for four, 64 tokens of 16 stretches of 64 took 2.8 us (the loop 2.2, one
    // number 1.8), 4,000 tokens of 4 of 256 24.4 (19.6, two numbers 17.1)
    auto kernel = per <= threads        ? xrt::gated_group_norm_rows_kernel<TO, 1>
                  : per <= 2 * threads  ? xrt::gated_group_norm_rows_kernel<TO, 2>
                  : per <= 4 * threads  ? xrt::gated_group_norm_rows_kernel<TO, 4>
                  : per <= 8 * threads  ? xrt::gated_group_norm_rows_kernel<TO, 8>
                  : per <= 16 * threads ? xrt::gated_group_norm_rows_kernel<TO, 16>
                                        : xrt::gated_group_norm_kernel<TO>;
    xrt::launch_kernel(kernel, dim3(n_tokens, groups), dim3(threads), 0, stream, (TO*)out, y, z, z_stride, weight, width, groups,
                       eps);
  });
  return xrt::launch_status();
}
