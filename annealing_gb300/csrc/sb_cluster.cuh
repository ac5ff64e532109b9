// Plain FP32 solves of up to 512 spins (aSB, bSB, dSB with couplings the bit planes do not take, NMFA) in one launch of
// independent clusters: plain_persist_kernel with its exchange through distributed shared memory instead of L2.
// A warp owns two rows (the same float4 groups per lane, sums and updates, so the same bits): both take the float4 of
// x that a lane reads, the butterfly's first round leaves one row in each half of the warp, and from there on a half
// updates and sends its row. A CTA owns 32 rows and a cluster of ceil(n / 32) CTAs a replica. A half sends its row's
// x (dSB: its sign as +-1.0) to every CTA of the cluster, a lane each, with st.async, counted in bytes on the
// receiver's mbarrier, one buffer per parity of the step: a warp sends step t + 2's x only after it has all of step
// t + 1's, each of which was sent after its sender had read step t's, so no CTA barrier is needed. Nothing waits
// across clusters: any number of replicas runs.
// us per step, before (exchange through L2 where its grid is co-resident, else a launch per step) -> this: bSB one
// replica n = 128 1.13 -> 0.64, n = 300 1.32 -> 0.84, n = 512 1.33 -> 1.12; n = 128 R = 32 4.60 -> 0.96, n = 300
// R = 12 5.08 -> 1.29; aSB n = 128 4.1 -> 3.3, R = 32 10.0 -> 3.9 (20 steps, initial state and energies included);
// NMFA n = 128 1.25 -> 0.79, n = 300 R = 12 6.7 -> 1.0. (One row to a warp read x twice as often: n = 512 1.60.)
#pragma once

namespace cluster {

constexpr int kRows = 32;                       // rows of a CTA, two to a warp
constexpr int kThreads = 16 * kRows;
constexpr int kGroups = kClusterMaxN / 128;     // float4 groups per lane

template <int VARIANT>
__global__ void __launch_bounds__(kThreads) cluster_kernel(const __grid_constant__ PlainPersist a) {
  constexpr bool kSigns = VARIANT == 2;
  __shared__ __align__(16) float xs[2][kClusterMaxN];  // x(t) of every spin (dSB: its sign, +-1), by parity
  __shared__ __align__(8) uint64_t full[2];
  __shared__ float sx[kRows], sy[kRows];  // aSB: the rows' x, y for the local sub-steps
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int C = gridDim.x, rank = (int)ptx::cluster_rank(), r = blockIdx.y;
  const int own = 2 * warp + (lane >> 4);  // this half's row of the CTA
  const int row = rank * kRows + own;
  const bool have = row < a.n;
  const int ng = a.jp >> 2;  // float4 groups of a row
  const uint32_t bytes = (uint32_t)(C * kRows * 4);
  float4 jr[2][kGroups];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int k = 0; k < kGroups; ++k) {
      const int g = lane + 32 * k, i = rank * kRows + 2 * warp + q;
      jr[q][k] = (i < a.n && g < ng && SB_BOUNDS((size_t)i * a.jp + 4 * g + 4 <= (size_t)a.n * a.jp, a.status))
                     ? reinterpret_cast<const float4 *>(a.J + (size_t)i * a.jp)[g]
                     : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  const size_t k_xy = (size_t)r * a.xp + row;
  float x = 0.0f, y = 0.0f;
  if (have && SB_BOUNDS(k_xy < (size_t)a.R * a.xp, a.status)) {
    const uint64_t e = 2 * ((uint64_t)r * a.n + row);
    x = a.init ? uniform_value(a.seed, e) : a.x_in[k_xy];
    if constexpr (VARIANT != 3) y = a.init ? uniform_value(a.seed, e + 1) : a.y[k_xy];
  }
  const float hv = (have && a.h) ? a.h[row] : 0.0f;
  const size_t plane = (size_t)a.R * a.xp;
  float nv = 0.0f, z1 = 0.0f;
  uint32_t wd[5] = {0u, 0u, 0u, 0u, 0u};
  if constexpr (VARIANT == 3) {
    if (have && SB_BOUNDS(k_xy < plane, a.status)) {
      nv = a.norm[row];
#pragma unroll
      for (int q = 0; q < 5; ++q) wd[q] = a.rng[q * plane + k_xy];
    }
  }
  if (tid == 0) {
    ptx::mbar_init(&full[0], 1);
    ptx::mbar_init(&full[1], 1);
    ptx::fence_mbar_init();
    ptx::mbar_arrive_expect_tx(&full[0], bytes);
    ptx::mbar_arrive_expect_tx(&full[1], bytes);
  }
  __syncthreads();
  ptx::cluster_sync();
  // lane k < C of a half: its row's cell and the barrier in CTA k, parity 0
  const uint32_t peer = (uint32_t)min(lane & 15, C - 1);
  const uint32_t to = ptx::mapa(ptx::smem_u32(&xs[0][row]), peer), to_bar = ptx::mapa(ptx::smem_u32(&full[0]), peer);
  // rows past n send x = 0 (sign -1), as the per-step kernel reads padding spins
  auto publish = [&](int t) {
    const float v = kSigns ? (have && x > 0.0f ? 1.0f : -1.0f) : (have ? x : 0.0f);
    const int p = t & 1;
    if ((lane & 15) < C) signs::st_async_u32(to + p * (uint32_t)sizeof(xs[0]), __float_as_uint(v), to_bar + p * 8u);
  };
  bool ok = true;
  const float lost = sbasb::underflow_bound(a.mts_dt, a.kerr);  // aSB
  if (a.steps > 0) publish(0);
  float pump_next = a.steps > 0 ? a.pumps[0] : 0.0f;
  for (int t = 0; t < a.steps; ++t) {
    const float pump = pump_next;
    if (t + 1 < a.steps) pump_next = a.pumps[t + 1];  // off the step's critical path
    float z0 = z1;
    if constexpr (VARIANT == 3)
      if ((t & 1) == 0) sbm::nmfa_gauss(wd, a.noise, z0, z1);
    // (aSB meets at CTA barriers below, so its warps leave the loop together)
    ok = ptx::mbar_wait_cluster_spin(&full[t & 1], (uint32_t)(t >> 1) & 1u, ptx::kWaitCycles);
    ok = VARIANT == 0 ? __syncthreads_and(ok ? 1 : 0) != 0 : __all_sync(0xffffffffu, ok);
    if (!ok) break;
    // step t + 2's x cannot arrive before this CTA has sent step t + 1's
    if (tid == 0 && t + 2 < a.steps) ptx::mbar_arrive_expect_tx(&full[t & 1], bytes);
    const float4 *x4 = reinterpret_cast<const float4 *>(xs[t & 1]);
    float sum[2] = {0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < kGroups; ++k) {
      const int g = lane + 32 * k;
      if (g < ng) {
        const float4 xv = x4[g];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          sum[q] = __fmaf_rn(jr[q][k].x, xv.x, sum[q]);
          sum[q] = __fmaf_rn(jr[q][k].y, xv.y, sum[q]);
          sum[q] = __fmaf_rn(jr[q][k].z, xv.z, sum[q]);
          sum[q] = __fmaf_rn(jr[q][k].w, xv.w, sum[q]);
        }
      }
    }
    // the first round of both rows' butterflies: the lower half keeps the first row
    const bool upper = lane >= 16;
    float acc = __fadd_rn(upper ? sum[1] : sum[0], __shfl_xor_sync(0xffffffffu, upper ? sum[0] : sum[1], 16));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (have) {
      if constexpr (VARIANT == 0)
        y = __fmaf_rn(a.coeff, acc, y);  // aSB: the coupling kick; the next step's local sub-steps follow
      else if constexpr (VARIANT == 3)
        x = sbm::nmfa_update(acc, nv, z0, pump, a.keep, a.mix, x);
      else
        sb_update(acc, hv, pump, a.c0, a.dt, a.dta0, x, y);
    }
    if (t + 1 == a.steps) break;
    if constexpr (VARIANT == 0) {
      // the local sub-steps of the CTA's rows in the lanes of one warp
      if ((lane & 15) == 0) {
        sx[own] = x;
        sy[own] = y;
      }
      __syncthreads();
      if (warp == 0) {
        float lx = sx[lane], ly = sy[lane];
        sbasb::local(lx, ly, __fdiv_rn((float)(t + 1), (float)a.steps), a.m, a.mts_dt, a.detune, a.kerr, lost);
        sx[lane] = lx;
        sy[lane] = ly;
      }
      __syncthreads();
      x = sx[own];
      y = sy[own];
    }
    publish(t + 1);
  }
  // a CTA's shared memory stays until the cluster's last word has arrived
  __syncwarp();
  ptx::cluster_sync();
  if (!ok) {
    if (lane == 0) atomicOr(a.status, kErrWaitTimeout);
    const long long t0 = clock64();  // words still on their way to this CTA land
    while (clock64() - t0 < 100000) __nanosleep(200);
    return;
  }
  if (have && (lane & 15) == 0 && SB_BOUNDS(k_xy < (size_t)a.R * a.xp, a.status)) {
    a.x_out[k_xy] = x;
    if constexpr (VARIANT == 3) {
#pragma unroll
      for (int q = 0; q < 5; ++q) a.rng[q * plane + k_xy] = wd[q];
      if (a.samples) a.samples[(size_t)r * a.n + row] = x > 0.0f ? 1 : -1;
    } else {
      a.y[k_xy] = y;
    }
  }
}

}  // namespace cluster
