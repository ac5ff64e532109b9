// The results a solve hands back, packed for one copy to the host.
#pragma once
#include <stdint.h>

namespace sbk {

// By a block: R energies, the index of the first least one (8 bytes; 0 when the first is NaN) and the n spins of that
// replica's x (+-1 bytes) at dst (8-byte aligned).
__device__ __forceinline__ void pack_results(const double *e, const float *x, int n, int R, int xp, uint8_t *dst) {
  __shared__ double least[32];
  __shared__ int where[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double v = 0.0;
  int k = -1;
  auto take = [&](double q, int r) {
    if (r >= 0 && (k < 0 || q < v || (q == v && r < k))) {
      v = q;
      k = r;
    }
  };
  for (int r = tid; r < R; r += (int)blockDim.x) {
    const double q = e[r];
    reinterpret_cast<double *>(dst)[r] = q;
    take(q, q == q ? r : -1);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double q = __shfl_xor_sync(0xffffffffu, v, o);
    const int r = __shfl_xor_sync(0xffffffffu, k, o);
    take(q, r);
  }
  if (lane == 0) {
    least[warp] = v;
    where[warp] = k;
  }
  __syncthreads();
  // every thread combines the warps' candidates
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) take(least[w], where[w]);
  const double first = e[0];
  const int best = first == first && k >= 0 ? k : 0;
  if (tid == 0) *reinterpret_cast<int64_t *>(dst + 8 * (size_t)R) = best;
  int8_t *s = reinterpret_cast<int8_t *>(dst) + 8 * ((size_t)R + 1);
  const float *xb = x + (size_t)best * xp;
  for (int i = tid; i < n; i += (int)blockDim.x) s[i] = xb[i] > 0.0f ? 1 : -1;
}

}  // namespace sbk
