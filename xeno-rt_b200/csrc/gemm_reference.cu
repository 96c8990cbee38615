// Y[M, N] = X[M, K] . W[N, K]^T on CUDA cores with 32-bit fused multiply-adds: the matrix product
// of the true 32-bit path (no tensor cores, no reduced-precision mode), and the product that takes
// any size and any dtype mix when a tensor-core kernel refuses a shape.
//
// W is row-major [out, in] as the reference stores every matrix (crates/xrt-models/src/llama.rs:447-486),
// so both operands are contiguous along K.  The reference's own CUDA matmul_kernel
// (crates/xrt-cuda/src/lib.rs:636-772) takes B untransposed with 16x16 tiles and one fma a step;
// this one computes a 4x4 patch a thread from 64x64x16 shared-memory tiles.
// Every output element is summed over k = 0 .. K-1 in order by one thread, so a row's result does
// not depend on how many other rows the call carries.
#include "common.cuh"

namespace xrt {

constexpr int RG_BM = 64, RG_BN = 64, RG_BK = 16;

// epilogue: 0 = store, 1 = add into the 32-bit output (the residual stream)
template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_reference_kernel(TO* __restrict__ out, const TX* __restrict__ x, const TW* __restrict__ w, int M, int N,
                      int K, int ldx, int ldo, int epilogue) {
  __shared__ float xs[RG_BK][RG_BM + 4];
  __shared__ float ws[RG_BK][RG_BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * RG_BM, n0 = blockIdx.x * RG_BN;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += RG_BK) {
    // each thread loads 4 elements of each tile: row = (tid*4 + i) / 16, k = (tid*4 + i) % 16
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid * 4 + i, r = e / RG_BK, kk = e % RG_BK;
      const int gm = m0 + r, gn = n0 + r, gk = k0 + kk;
      xs[kk][r] = (gm < M && gk < K) ? to_float(x[(size_t)gm * ldx + gk]) : 0.f;
      ws[kk][r] = (gn < N && gk < K) ? to_float(w[(size_t)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < RG_BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = xs[kk][tm + i]; b[i] = ws[kk][tn + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + tm + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tn + j;
      if (gn >= N) continue;
      TO* dst = out + (size_t)gm * ldo + gn;
      if (epilogue == 1) *dst = from_float<TO>(to_float(*dst) + acc[i][j]);
      else *dst = from_float<TO>(acc[i][j]);
    }
  }
}

// The same product where 64 x 64 tiles would leave most multiprocessors empty (a step of few tokens, a small model): tiles
// of 16 x 16, one output a thread, slabs of 64 along K, the next slab's loads in flight while this one is worked on.
// What bounds such a product is the latency of its loads, one trip to memory a slab: the kernel above makes four times as
// many trips and waits for each.  The sum over k is the same chain, so results are the same bit for bit.  The first slab
// of W, which no kernel of a step writes, is asked for before the wait for the kernel before.
// Measured inside a step of 3 tokens at widths of 64 and 176: 5.7 us (64 inputs) and 13.8 (176) -> 1.8 a product.
constexpr int RS_BM = 16, RS_BN = 16, RS_BK = 64, RS_PITCH = RS_BK + 4;
template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_reference_few_kernel(TO* __restrict__ out, const TX* __restrict__ x, const TW* __restrict__ w, int M, int N,
                          int K, int ldx, int ldo, int epilogue) {
  __shared__ __align__(16) float xs[RS_BM][RS_PITCH], ws[RS_BN][RS_PITCH];
  constexpr int PER = RS_BM * RS_BK / 256, STEP = 256 / RS_BK;
  pdl_trigger();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * RS_BM, n0 = blockIdx.x * RS_BN;
  const int lk = tid % RS_BK, lr = tid / RS_BK;  // this thread's copies: column lk of rows lr, lr + 4, ...
  const int tm = tid / RS_BN, tn = tid % RS_BN;
  float nx[PER], nw[PER];
  auto ask_w = [&](int k0) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int n = n0 + lr + i * STEP;
      nw[i] = (n < N && k0 + lk < K) ? to_float(w[(size_t)n * K + k0 + lk]) : 0.f;
    }
  };
  auto ask_x = [&](int k0) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int m = m0 + lr + i * STEP;
      nx[i] = (m < M && k0 + lk < K) ? to_float(x[(size_t)m * ldx + k0 + lk]) : 0.f;
    }
  };
  ask_w(0);
  pdl_wait(x);
  ask_x(0);
  float acc = 0.f;
  for (int k0 = 0; k0 < K; k0 += RS_BK) {
    __syncthreads();  // the slab before is used up
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      xs[lr + i * STEP][lk] = nx[i];
      ws[lr + i * STEP][lk] = nw[i];
    }
    __syncthreads();
    if (k0 + RS_BK < K) {
      ask_w(k0 + RS_BK);
      ask_x(k0 + RS_BK);
    }
#pragma unroll
    for (int kk = 0; kk < RS_BK; kk += 4) {
      const float4 a = *reinterpret_cast<const float4*>(&xs[tm][kk]);
      const float4 b = *reinterpret_cast<const float4*>(&ws[tn][kk]);
      acc = fmaf(a.x, b.x, acc);
      acc = fmaf(a.y, b.y, acc);
      acc = fmaf(a.z, b.z, acc);
      acc = fmaf(a.w, b.w, acc);
    }
  }
  const int gm = m0 + tm, gn = n0 + tn;
  if (gm < M && gn < N) {
    TO* dst = out + (size_t)gm * ldo + gn;
    if (epilogue == 1) *dst = from_float<TO>(to_float(*dst) + acc);
    else *dst = from_float<TO>(acc);
  }
}

}  // namespace xrt

// x: [M, K] with row stride ldx; w: [N, K] contiguous; out: [M, N] with row stride ldo.
XRT_EXPORT int xrt_gemm_reference(void* out, const void* x, const void* w, int M, int N, int K, int ldx, int ldo,
                                  int x_dtype, int w_dtype, int out_dtype, int epilogue, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || ldx < K || ldo < N || epilogue < 0 || epilogue > 1) return XRT_ERR_ARGUMENT;
  if (epilogue == 1 && out_dtype != XRT_F32) return XRT_ERR_ARGUMENT;
  if (M == 0) return XRT_OK;
  dim3 grid((N + xrt::RG_BN - 1) / xrt::RG_BN, (M + xrt::RG_BM - 1) / xrt::RG_BM);
  if (grid.y > 65535) return XRT_ERR_UNSUPPORTED;
  // small tiles while the large ones would occupy no more than half of the multiprocessors
  const bool few = 2ll * grid.x * grid.y <= xrt::multiprocessors();
  XRT_DISPATCH_DTYPE(x_dtype, TX, {
    XRT_DISPATCH_DTYPE(w_dtype, TW, {
      XRT_DISPATCH_DTYPE(out_dtype, TO, {
        if (few)
          xrt::launch_kernel(xrt::gemm_reference_few_kernel<TX, TW, TO>,
                             dim3((N + xrt::RS_BN - 1) / xrt::RS_BN, (M + xrt::RS_BM - 1) / xrt::RS_BM), dim3(256), 0, stream,
                             (TO*)out, (const TX*)x, (const TW*)w, M, N, K, ldx, ldo, epilogue);
        else
          xrt::gemm_reference_kernel<TX, TW, TO><<<grid, 256, 0, stream>>>(
              (TO*)out, (const TX*)x, (const TW*)w, M, N, K, ldx, ldo, epilogue);
      });
    });
  });
  return xrt::launch_status();
}
