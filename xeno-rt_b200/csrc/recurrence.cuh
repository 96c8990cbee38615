// What the kernels of the recurrent mixers share: 32-bit activations and asynchronous copies to shared memory.
#pragma once

#include "common.cuh"

namespace xrt {

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplusf_(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float activate(float z, int act) {  // 0 none, 1 silu, 2 sigmoid, 3 tanh
  return act == 1 ? z * sigmoidf_(z) : (act == 2 ? sigmoidf_(z) : (act == 3 ? tanhf(z) : z));
}

template <int BYTES>
__device__ __forceinline__ void cp_async(float* smem, const float* global) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(global) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(global) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Sums of N values over the LANES neighbouring lanes, spread over them: at each level a lane gives away half of its
// values and adds what it gets to the other half, so that N values cost about N shuffles instead of N log2(LANES).
// Afterwards v[0] of lane `part` is the whole sum of value part * N / LANES (N <= LANES, powers of two).  Every sum is
// formed in the order of a butterfly over the lane bits from the highest to the lowest.
template <int N, int O, int ALL>
__device__ __forceinline__ float lane_sums_from(float (&v)[ALL], int part) {
  if constexpr (O == 0) {
    return v[0];
  } else if constexpr (N > 1) {
    const bool upper = (part & O) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const float give = upper ? v[i] : v[i + N / 2], keep = upper ? v[i + N / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, O);
    }
    return lane_sums_from<N / 2, O / 2>(v, part);
  } else {
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
    return lane_sums_from<1, O / 2>(v, part);
  }
}
template <int LANES, int N>
__device__ __forceinline__ float lane_sums(float (&v)[N], int part) {
  static_assert(N <= LANES, "one value a lane at most");
  return lane_sums_from<N, LANES / 2>(v, part);
}

// The same sums, every lane getting all N of them: sixteen at a time through lane_sums, then a broadcast each.
template <int LANES, int N>
__device__ __forceinline__ void all_lane_sums(float (&v)[N], int part) {
  static_assert(LANES >= 16, "sixteen values at a time");
#pragma unroll
  for (int first = 0; first < N; first += 16) {
    float some[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) some[i] = first + i < N ? v[first + i < N ? first + i : 0] : 0.f;
    const float sum = lane_sums<LANES>(some, part);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (first + i < N) v[first + i] = __shfl_sync(0xffffffffu, sum, i * (LANES / 16), LANES);
  }
}

}  // namespace xrt
