// Plain dSB with integer couplings up to 127, the whole solve in one launch without a trip through L2 between steps
// (SignSolve). A dSB step needs only the signs of the other spins, so with J as bit planes (per 32 columns a sign
// word and P magnitude words) a field is
//   f_i = sum_j |J_ij| - 2 sum_k 2^(k-1) popc(mag_k & (sign ^ s)),
// an exact integer, as the FP32 sums of the other kernels are (n max |J| < 2^24): the same bits. A thread owns a
// row: its planes in registers, x and y too, no reduction; a warp's ballot is the sign word of its 32 rows.
//   * n <= 512 (one magnitude plane; 256 with more): one CTA holds every row; a step is a few broadcast reads, popcounts, the update, a ballot
//     and a barrier.
//   * above, a cluster of ceil(n / 128) CTAs of 128 rows: each warp sends its word to every CTA of the cluster with
//     st.async, counted in bytes on the receiver's mbarrier (one per parity of the step). A warp sends step t + 2's
//     word only after it has step t + 1's, which every warp sent after reading step t's: two buffers suffice, and
//     no CTA barrier is needed.
// Popcounts run at a quarter of the logic rate, so carry-save adders fold four masked words into two popcounts.
// us per step of 1000, against the kernels before it (signs through L2, or one launch per step where its grid is
// not co-resident): J = +-1, one replica n = 128 0.98 -> 0.18, n = 512 1.27 -> 0.40, n = 513 1.28 -> 0.58,
// n = 1000 1.38 -> 0.52, n = 2000 1.57 -> 0.71; twelve replicas n = 1000 8.2 -> 0.6, n = 2000 16.8 -> 0.81; |J| <= 7
// n = 128 0.98 -> 0.26, n = 512 1.25 -> 0.49, n = 1000 1.38 -> 0.84. 100 replicas of n = 2000 95 -> 6.0 (50 steps).
// |J| <= 127 (seven planes) n = 128 0.37, n = 256 0.64, n = 512 0.78. A cluster's step is some 0.45 us of exchange, the rest its 128 rows' logic, one warp to a scheduler.
// Replicas are independent clusters: nothing waits across them, so any number runs.
#pragma once

namespace signs {

constexpr int kMaxWords = kSignsMaxN / 32;
constexpr int kClusterRows = 128;  // rows (threads) of a clustered CTA: a warp for each scheduler

__device__ __forceinline__ void st_async_u32(uint32_t caddr, uint32_t v, uint32_t cbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(caddr), "r"(v),
               "r"(cbar)
               : "memory");
}

// W: words of a row's planes in registers (a multiple of four, at least a.words), P magnitude planes.
template <int W, int P, bool CLUSTER>
__global__ void __launch_bounds__(CLUSTER ? kClusterRows : kSignsOneCta) signs_kernel(const __grid_constant__ SignSolve a) {
  constexpr int kBlock = W <= 48 ? W : 32;  // words a branch covers (sixteen: n = 1000 0.56 us a step against 0.52)
  __shared__ __align__(16) uint32_t sg[2][kMaxWords];  // sign words (bit set: -1) of a step, by parity
  __shared__ __align__(8) uint64_t full[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = blockIdx.y;
  const int C = CLUSTER ? (int)gridDim.x : 1, rank = CLUSTER ? (int)ptx::cluster_rank() : 0;
  const int row = rank * (int)blockDim.x + tid, word = row >> 5;
  const bool have = row < a.n;
  const uint32_t bytes = (uint32_t)(C * (int)(blockDim.x >> 5) * 4);  // of a step's words
  uint32_t pl[P + 1][W];
  int row_abs = 0;
#pragma unroll
  for (int w = 0; w < W; ++w)
#pragma unroll
    for (int k = 0; k <= P; ++k) {
      pl[k][w] = have && w < a.words ? a.planes[((size_t)k * a.words + w) * a.n + row] : 0u;
      if (k > 0) row_abs += __popc(pl[k][w]) << (k - 1);
    }
  const size_t k_xy = (size_t)r * a.xp + row;
  float x = 0.0f, y = 0.0f;
  if (have && SB_BOUNDS(k_xy < (size_t)a.R * a.xp, a.status)) {
    const uint64_t e = 2 * ((uint64_t)r * a.n + row);
    x = a.init ? uniform_value(a.seed, e) : a.x_in[k_xy];
    y = a.init ? uniform_value(a.seed, e + 1) : a.y[k_xy];
  }
  const float hv = have && a.h ? a.h[row] : 0.0f;
  for (int k = tid; k < 2 * kMaxWords; k += (int)blockDim.x) (&sg[0][0])[k] = 0u;
  if (CLUSTER && tid == 0) {
    ptx::mbar_init(&full[0], 1);
    ptx::mbar_init(&full[1], 1);
    ptx::fence_mbar_init();
    ptx::mbar_arrive_expect_tx(&full[0], bytes);
    ptx::mbar_arrive_expect_tx(&full[1], bytes);
  }
  __syncthreads();
  if (CLUSTER) ptx::cluster_sync();
  // the signs of x(t), rows past n as x = 0
  uint32_t to = 0, to_bar = 0;  // lane k < C: this warp's word and the barrier in CTA k, parity 0
  if (CLUSTER) {
    to = ptx::mapa(ptx::smem_u32(&sg[0][word]), (uint32_t)min(lane, C - 1));
    to_bar = ptx::mapa(ptx::smem_u32(&full[0]), (uint32_t)min(lane, C - 1));
  }
  auto publish = [&](int t) {
    const uint32_t b = __ballot_sync(0xffffffffu, !have || !(x > 0.0f));
    const int p = t & 1;
    if (CLUSTER) {
      if (lane < C) st_async_u32(to + p * (uint32_t)sizeof(sg[0]), b, to_bar + p * 8u);
    } else if (lane == 0) {
      sg[p][word] = b;
    }
  };
  bool ok = true;
  float pump_next = a.steps > 0 ? a.pumps[0] : 0.0f;
  if (a.steps > 0) publish(0);
  for (int t = 0; t < a.steps; ++t) {
    const float pump = pump_next;
    if (t + 1 < a.steps) pump_next = a.pumps[t + 1];  // off the step's critical path
    if (CLUSTER) {
      ok = __all_sync(0xffffffffu, ptx::mbar_wait_cluster(&full[t & 1], (uint32_t)(t >> 1) & 1u, ptx::kWaitCycles));
      if (!ok) break;
      // step t + 2's words cannot arrive before this CTA has sent step t + 1's
      if (tid == 0 && t + 2 < a.steps) ptx::mbar_arrive_expect_tx(&full[t & 1], bytes);
    } else {
      __syncthreads();
    }
    const uint4 *s4 = reinterpret_cast<const uint4 *>(sg[t & 1]);
    int acc = 0;
    uint32_t ones[P];
    int twos[P];
#pragma unroll
    for (int k = 0; k < P; ++k) {
      ones[k] = 0u;
      twos[k] = 0;
    }
#pragma unroll
    for (int b = 0; b < W; b += kBlock)
      if (b < a.words) {  // a branch for every four words kept their chains apart: 1.14 us at n = 2000
#pragma unroll
        for (int q = b / 4; q < (b + kBlock) / 4; ++q) {
          const uint4 s = s4[q];
          const uint32_t z0 = pl[0][4 * q] ^ s.x, z1 = pl[0][4 * q + 1] ^ s.y, z2 = pl[0][4 * q + 2] ^ s.z,
                         z3 = pl[0][4 * q + 3] ^ s.w;
#pragma unroll
          for (int k = 0; k < P; ++k) {
            const uint32_t m0 = pl[k + 1][4 * q] & z0, m1 = pl[k + 1][4 * q + 1] & z1, m2 = pl[k + 1][4 * q + 2] & z2,
                           m3 = pl[k + 1][4 * q + 3] & z3;
            // two full adders: bits of weight one stay in `ones`, of weight two are counted
            const uint32_t u = m0 ^ m1 ^ m2, c0 = (m0 & m1) | (m2 & (m0 | m1));
            const uint32_t c1 = (u & m3) | (ones[k] & (u | m3));
            ones[k] ^= u ^ m3;
            twos[k] += __popc(c0) + __popc(c1);
          }
        }
      }
#pragma unroll
    for (int k = 0; k < P; ++k) acc += (2 * twos[k] + __popc(ones[k])) << k;
    if (have) sb_update((float)(row_abs - 2 * acc), hv, pump, a.c0, a.dt, a.dta0, x, y);
    if (t + 1 < a.steps) publish(t + 1);
  }
  // a CTA's shared memory stays until the cluster's last word has arrived
  if (CLUSTER) {
    __syncwarp();
    ptx::cluster_sync();
  }
  if (!ok) {
    if (lane == 0) atomicOr(a.status, kErrWaitTimeout);
    const long long t0 = clock64();  // words still on their way to this CTA land
    while (clock64() - t0 < 100000) __nanosleep(200);
    return;
  }
  if (have && SB_BOUNDS(k_xy < (size_t)a.R * a.xp, a.status)) {
    a.x_out[k_xy] = x;
    a.y[k_xy] = y;
  }
}

// J's planes [P + 1][words][n] (sign, then magnitudes; row fastest), a warp per row and word.
__global__ void sign_planes_kernel(const float *J, int n, int jp, int words, int P, uint32_t *planes) {
  const int lane = threadIdx.x & 31;
  const long long k = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int row = (int)(k / words), w = (int)(k % words), col = 32 * w + lane;
  if (row >= n) return;  // whole warps
  const int v = col < n ? (int)J[(size_t)row * jp + col] : 0, m = v < 0 ? -v : v;
  const uint32_t s = __ballot_sync(0xffffffffu, v < 0);
  if (lane == 0) planes[(size_t)w * n + row] = s;
  for (int q = 0; q < P; ++q) {
    const uint32_t b = __ballot_sync(0xffffffffu, (m >> q) & 1);
    if (lane == 0) planes[((size_t)(q + 1) * words + w) * n + row] = b;
  }
}

// One CTA holds the solve while a cluster's exchange costs more than its popcounts, us per step, one CTA / cluster:
// two planes n = 256 0.36 / -, n = 400 0.81 / 0.54; three planes n = 256 0.39 / -, n = 400 0.99 / 0.49; one plane
// n = 512 0.40, a cluster of five 0.58.
constexpr bool one_cta(int n, int P) { return n <= (P == 1 ? kSignsOneCta : kSignsOneCta / 2); }

template <int P>
const void *kernel_for(int n) {
  static_assert(kSignsOneCta == 16 * 32, "the forms below");
  const int words = (n + 31) / 32;
  if (words <= 4) return reinterpret_cast<const void *>(&signs_kernel<4, P, false>);
  if (words <= 8) return reinterpret_cast<const void *>(&signs_kernel<8, P, false>);
  if (words <= 16) return reinterpret_cast<const void *>(&signs_kernel<16, P, P != 1>);
  if constexpr (P <= 4)
    if (words <= 32) return reinterpret_cast<const void *>(&signs_kernel<32, P, true>);
  if constexpr (P == 1) {
    if (words <= 48) return reinterpret_cast<const void *>(&signs_kernel<48, P, true>);
    return reinterpret_cast<const void *>(&signs_kernel<64, P, true>);
  } else {
    return nullptr;
  }
}

}  // namespace signs
