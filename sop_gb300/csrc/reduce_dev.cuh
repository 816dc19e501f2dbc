// Block-wide FP64 sums of several values per thread.
//
// FP64 runs at 2 lanes per clock and SM here (a warp-wide add takes 16
// cycles), so the count of adds sets the cost: reducing K values one after
// another over the lanes takes 5 K adds per lane; here every lane hands half
// of its values to its partner and keeps the sums of the other half, so the
// values spread over the lanes as they are summed (6 adds for 4 values, 9 for
// 8, instead of 20 and 40).  The order is fixed, so results repeat bit for bit.
#pragma once

namespace sop {

// The sums over the warp of v[0 .. K-1] (K a power of two up to 8); the sum
// of value k is in every lane whose top log2(K) bits spell k.
template <int K>
__device__ __forceinline__ double warp_sums(double (&v)[K]) {
  const int lane = threadIdx.x & 31;
  int off = 16;
#pragma unroll
  for (int n = K / 2; n >= 1; n >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const double keep = up ? v[k + n] : v[k], give = up ? v[k] : v[k + n];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
  double x = v[0];
#pragma unroll
  for (; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}

// The sums over the block (of up to 1,024 threads, whole warps): thread k < K
// returns the sum of value k.  red: K * 32 doubles of shared memory, free for
// other use after the caller's next barrier.
template <int K>
__device__ __forceinline__ double block_sums(double (&v)[K], double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const double x = warp_sums<K>(v);
  constexpr int kLanes = 32 / K;  // lanes that hold the same sum
  if (lane % kLanes == 0) red[(lane / kLanes) * 32 + w] = x;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < K)
    for (int k = 0; k < warps; ++k) t += red[threadIdx.x * 32 + k];
  return t;
}

}  // namespace sop
