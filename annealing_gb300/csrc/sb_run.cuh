// Many dSB steps of a set of work items in one launch, the signs exchanged between SMs as tagged words.
//
// A work item is 128 spins x NR replicas of one instance. Its x, y stay in tensor memory for the whole
// launch; a step contracts the item's J rows with sign(x) of all spins of its replicas, so the items of one
// replica tile (all spin tiles of an instance) exchange their signs every step. A step's exchange is a
// dependent chain, and it is what bounds these shapes, so the chain is kept short:
//   * Signs travel as one bit each. An epilogue warp transposes its 32 spins x 32 replicas of signs into a
//     word per replica and stores (word, step tag) as one 8-byte relaxed store; a reader polls the same 8 bytes, so the data is its own
//     flag and one store and one load through L2 replace a TMA store, a fence, a release, a poll, an acquire
//     fence and a TMA load (2.5 us of a 6.2 us step at N = 2048).
//   * Four loader warps read the words (32 KB for 2048 spins x 64 replicas, against 128 KB of E2M1 operands
//     for a 128-replica tile), expand each to the operand's bytes with a shift and a LOP per 4 bytes and
//     write them to shared memory in the MMA's swizzled layout.
//   * The MMA and TMA loops run with the whole warp (ptx::elect_one).
//   * The epilogue has x and y in registers before its accumulator is complete and frees the accumulator
//     as soon as it has read it.
// A CTA owns up to kSlots items; one item's exchange overlaps another's contraction.
//   RES: J rows resident in shared memory, loaded once (all items of a CTA share them): the items of one
//        instance whose J rows fit, e.g. two 64-replica halves of a spin tile.
//   else J tiles stream through the ring from L2 each step.
// Couplings beyond E4M3's 16 (integers up to 256) come as 16 hi + lo, both exact in E4M3: a chunk of each multiplies the
// same 128 signs, so the signs are expanded once and the sums are the integers all the same.
// Word order: bit position 4 i + k of a word holds spin 8 k + i for E2M1 operands (nibble i of the k-th
// 32-bit word of the granule is then (w << (3 - k)) & 0x88888888 | 0x22222222), bit 8 j + k holds spin 4 k + j
// for the byte operands; the writer's lanes take their spins' bits in that order before they transpose.
// V(t) travels in buffer t & 1. An item overwrites the words of V(t) with V(t + 2) at the end of step t + 1,
// whose contraction needed V(t + 1) from every item of the tile, and each of them published it after its own
// contraction over V(t).
// Every wait is bounded; on expiry the kernel lets its copies and MMAs finish, frees its TMEM and returns a
// status. All CTAs wait on one another: the launch is cooperative.
#pragma once
#include "sb_grouped.h"
#include "sb_tc_fp4.cuh"
#include "sb_tc_kernel.cuh"

namespace sbk {

// An item of a launch. ll: its (instance, replica tile)'s words, [2][4 parts][NR] from this 8-byte index;
// parts: the instance's spin tiles; kchunks: 128-byte chunks of its operand rows.
struct RunItem {
  int inst, m0, r0, kchunks, parts;
  uint32_t ll;
};

struct RunArgs {
  const GInst *insts;
  const RunItem *items;
  unsigned long long *ll;  // zero before the launch
  uint32_t *status;
  int n_items, tick0, count;
  // host-side fault injection for the timeout path: item skip_item does not publish the signs of step
  // skip_step (skip_step < 0: every item publishes)
  int skip_item, skip_step;
  long long wait_cycles;
};

namespace tck {

constexpr int kLoadWarps = 4;
constexpr int kRunThreads = kTcThreads + 32 * kLoadWarps;
constexpr int kResChunks = 9;   // J chunks (16 KB each) of a resident item: leaves four 16 KB V stages at 64 replicas

// VS: V chunks of a ring stage (one for J in two parts: both multiply the same signs)
template <int NR, bool RES, int VS = 2>
struct RunCfg {
  static_assert(NR == 32 || NR == 64, "replica tile");
  static constexpr int kAcc = 2, kSlots = NR == 32 ? 6 : 2;
  // TMEM columns: accumulators, 32 block-scale columns, then x and y of each slot
  static constexpr uint32_t kSf = kAcc * NR, kState = kSf + 32;
  static_assert(kState + 2 * NR * kSlots <= 512, "TMEM columns");
  // A ring stage holds kSub J chunks (streaming), then VS V chunks. Waiting for a stage costs the MMA
  // warp ~110 clocks: 89 clocks per MMA with one chunk (4 MMAs) per stage, 63 with two, 48 without waits.
  static constexpr int kSub = 2;
  static constexpr int kATile = kBM * kChunkBytes, kBTile = NR * kChunkBytes;
  static constexpr int kVOff = RES ? 0 : kSub * kATile;  // V tiles within a stage
  static constexpr int kStage = kVOff + VS * kBTile;
  static constexpr int kRing = 212 * 1024 - (RES ? kResChunks * kATile : 0);
  static constexpr int kStages = kRing / kStage > 8 ? 8 : kRing / kStage;
  static constexpr size_t kSmem = (size_t)kStages * kStage + (RES ? kResChunks * kATile : 0) + 1024;
};

__device__ __forceinline__ void st_relaxed64(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// two adjacent words, each read whole
__device__ __forceinline__ ulonglong2 ld_relaxed64x2(const unsigned long long *p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Two FP32 operations in one instruction, each rounded as its scalar form.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// The warp's 32 x 32 bit matrix (lane = row, bit = column) transposed: lane c gets column c of all lanes.
__device__ __forceinline__ uint32_t transpose32(uint32_t w, int lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    // a block of j x j exchanges its off-diagonal halves: the upper lanes send their low bits, the lower
    // lanes their high bits
    constexpr uint32_t kLow[5] = {0x55555555u, 0x33333333u, 0x0F0F0F0Fu, 0x00FF00FFu, 0x0000FFFFu};
    const uint32_t low = kLow[j == 16 ? 4 : j == 8 ? 3 : j == 4 ? 2 : j == 2 ? 1 : 0];
    const bool up = (lane & j) != 0;
    const uint32_t got = __shfl_xor_sync(0xffffffffu, w, j);
    w = up ? ((w & ~low) | ((got >> j) & low)) : ((w & low) | ((got << j) & ~low));
  }
  return w;
}

template <int NR, int OP, bool RES>
__global__ void __launch_bounds__(kRunThreads, 1) run_kernel(const __grid_constant__ RunArgs p) {
  constexpr bool X2 = OP == kGopFp8x2;
  constexpr int kVSub = X2 ? 1 : 2;  // V chunks of a stage
  using C = RunCfg<NR, RES, kVSub>;
  constexpr int STAGES = C::kStages, kAcc = C::kAcc, kSlots = C::kSlots;
  constexpr int kATile = C::kATile, kBTile = C::kBTile, kStage = C::kStage, kSub = C::kSub;
  constexpr bool FP4 = OP == kGopE2m1, FP6 = OP == kGopE2m3;
  constexpr uint32_t kSf = C::kSf;
  constexpr uint32_t kTxJ = FP6 ? (uint32_t)kATile / 4 * 3 : (uint32_t)kATile;  // packed E2M3 counts its global bytes
  // kind::f8f6f4 formats (A bits 7-9, B bits 10-12): E4M3 = 0, E2M3 = 3. J / 4 in E2M3 meets signs of +-4 in
  // E4M3, J in E4M3 signs of +-1: the integer products either way
  constexpr uint32_t kIdesc = FP4 ? make_idesc_mxf4(kBM, NR) : (make_idesc(kTcFp8, kBM, NR) | (FP6 ? 3u << 7 : 0u));
  constexpr int kWords = FP4 ? 8 : 4;                     // 32-spin words of a chunk
  constexpr int kWordsPerLoad = NR == 64 ? 1 : 2;         // of a loader warp's 16-byte loads
  constexpr int kLoads = kWords / kWordsPerLoad;          // of them per chunk
  constexpr int kCols = NR / 2;                           // columns of an epilogue warp

  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *jres = smem + STAGES * kStage;  // RES: [kchunks][128][128] resident J
  __shared__ __align__(8) uint64_t fullj_bar[STAGES], fullv_bar[STAGES], empty_bar[STAGES], accf_bar[kAcc], acce_bar[kAcc],
      a_bar, drain_bar;
  __shared__ uint32_t tmem_base_sh;
  __shared__ RunItem mine[kSlots];
  __shared__ float hv_sh[kSlots][kBM];  // the items' fields h

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = gridDim.x;
  const long long limit = p.wait_cycles;
  bool ok = true;
  // Items of this CTA. Streaming: dealt back and forth over the longest-first list; resident: item j G + b, so
  // that the list decides which items share a CTA.
  auto item_at = [&](int j) { return (!RES && (j & 1)) ? j * G + (G - 1 - (int)blockIdx.x) : j * G + (int)blockIdx.x; };
  int nslots = 0;
  for (int j = 0; j < kSlots; ++j)
    if (item_at(j) < p.n_items) nslots = j + 1;  // only the last round may skip a CTA

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&fullj_bar[s], 1);
      ptx::mbar_init(&fullv_bar[s], kVSub);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < kAcc; ++b) {
      ptx::mbar_init(&accf_bar[b], 1);
      ptx::mbar_init(&acce_bar[b], kEpiWarps);
    }
    ptx::mbar_init(&a_bar, 1);
    ptx::mbar_init(&drain_bar, 1);
    ptx::fence_mbar_init();
    for (int j = 0; j < nslots; ++j) mine[j] = p.items[item_at(j)];
    for (int j = nslots; j < kSlots; ++j) mine[j] = mine[0];
  }
  if (warp == 1) {
    ptx::tmem_alloc(&tmem_base_sh, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_base_sh;
  for (int k = threadIdx.x; k < nslots * kBM; k += kRunThreads) {
    const GInst *in = p.insts + mine[k / kBM].inst;
    const int row = mine[k / kBM].m0 + k % kBM;
    hv_sh[k / kBM][k % kBM] = in->h && row < in->n ? in->h[row] : 0.0f;
  }
  if (FP4 && warp >= 2 && warp < 2 + kEpiWarps) {
    // every block scale = 2^0: UE8M0 0x7F in all bytes of the 32 scale columns, all 128 lanes
    uint32_t ones[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) ones[j] = 0x7F7F7F7Fu;
    ptx::tmem_st16(tmem + kSf + 16 * ((warp - 2) >> 2) + ((uint32_t)(32 * (warp & 3)) << 16), ones);
    ptx::tmem_st_wait();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();

  if (warp == 0) {
    // ---------------- J producer (the whole warp; elect_one issues) ----------------
    if constexpr (RES) {
      const RunItem w = mine[0];
      if (ptx::elect_one()) {
        ptx::mbar_arrive_expect_tx(&a_bar, (uint32_t)w.kchunks * kTxJ);
        for (int kc = 0; kc < w.kchunks; ++kc)
          ptx::tma_load_2d(jres + (size_t)kc * kATile, &p.insts[w.inst].tmA, kc * kChunkBytes, w.m0, &a_bar);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&a_bar, 0, limit));
      if (!ok) ptx::mbar_wait(&a_bar, 0);  // given up, but the copies land before this CTA exits
    } else {
      int s = 0;
      uint32_t ph = 1;      // parity of the stage's last release (a fresh barrier passes parity 1)
      uint32_t issued = 0;  // stages requested in all
      for (int ls = 0; ls < p.count && ok; ++ls)
        for (int j = 0; j < nslots && ok; ++j) {
          const RunItem w = mine[j];
          const CUtensorMap *ma = &p.insts[w.inst].tmA;
          for (int kc = 0; kc < w.kchunks; kc += kSub) {
            if (!__all_sync(0xffffffffu, ptx::mbar_wait(&empty_bar[s], ph, limit))) {
              ok = false;
              break;
            }
            const bool two = kc + 1 < w.kchunks;
            if (ptx::elect_one()) {
              ptx::mbar_arrive_expect_tx(&fullj_bar[s], two ? 2 * kTxJ : kTxJ);
              ptx::tma_load_2d(smem + s * kStage, ma, kc * kChunkBytes, w.m0, &fullj_bar[s]);
              if (two) ptx::tma_load_2d(smem + s * kStage + kATile, ma, (kc + 1) * kChunkBytes, w.m0, &fullj_bar[s]);
            }
            __syncwarp();
            ++issued;
            if (++s == STAGES) {
              s = 0;
              ph ^= 1;
            }
          }
        }
      if (!ok)  // a wait gave up: the last copy into each stage lands before this CTA exits
        for (uint32_t q = 0; q < STAGES; ++q)
          if (issued > q) ptx::mbar_wait(&fullj_bar[q], ((issued - 1 - q) / STAGES) & 1, limit);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp; elect_one issues) ----------------
    if constexpr (RES) ok = __all_sync(0xffffffffu, ptx::mbar_wait(&a_bar, 0, limit));
    int s = 0;
    uint32_t ph = 0, li = 0;
    bool have = false;  // stage s is known to be full
    // a stage's descriptors differ from stage 0's in the address field (units of 16 bytes) alone
    const uint64_t ad0 = ptx::smem_desc_sw128(ptx::smem_u32(RES ? jres : smem));
    const uint64_t bd0 = ptx::smem_desc_sw128(ptx::smem_u32(smem) + C::kVOff);
    for (int ls = 0; ls < p.count && ok; ++ls)
      for (int j = 0; j < nslots && ok; ++j, ++li) {
        const int kchunks = mine[j].kchunks;
        const uint32_t ab = li % kAcc, use = li / kAcc;
        const uint32_t t_acc = tmem + ab * NR;
        if (use > 0 && !__all_sync(0xffffffffu, ptx::mbar_wait(&acce_bar[ab], (use - 1) & 1, limit))) {
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        for (int kc = 0; kc < kchunks; kc += kSub) {
          if (!have) {
            bool got = ptx::mbar_wait(&fullv_bar[s], ph, limit);
            if constexpr (!RES) got = got && ptx::mbar_wait(&fullj_bar[s], ph, limit);
            if (!__all_sync(0xffffffffu, got)) {
              ok = false;
              break;
            }
          }
          const int cur = s;
          if (++s == STAGES) {
            s = 0;
            ph ^= 1;
          }
          bool next = ptx::mbar_test(&fullv_bar[s], ph);  // looked at while the MMAs below issue
          if constexpr (!RES) next = ptx::mbar_test(&fullj_bar[s], ph) && next;
          if (ptx::elect_one()) {
            const uint64_t ao = (uint64_t)((RES ? kc * kATile : cur * kStage) / 16), bo = (uint64_t)(cur * kStage / 16);
#pragma unroll
            for (int c = 0; c < kSub; ++c) {
              if (c > 0 && kc + c >= kchunks) continue;
#pragma unroll
              for (int k = 0; k < kChunkBytes / 32; ++k) {
                const uint64_t ad = ad0 + ao + c * (kATile / 16) + 2 * k, bd = bd0 + bo + (X2 ? 0 : c * (kBTile / 16)) + 2 * k;
                const uint32_t add = (kc > 0 || c > 0 || k > 0) ? 1u : 0u;
                if constexpr (FP4)
                  ptx::mma_mxf4(t_acc, ad, bd, kIdesc, tmem + kSf, tmem + kSf + 16, add);
                else
                  ptx::mma_f8(t_acc, ad, bd, kIdesc, add);
              }
            }
            ptx::mma_commit(&empty_bar[cur]);
            if (kc + kSub >= kchunks) ptx::mma_commit(&accf_bar[ab]);
          }
          __syncwarp();
          have = __all_sync(0xffffffffu, next);
        }
      }
    if (!ok) {
      // a wait gave up: the MMAs already issued finish before TMEM is freed
      if (ptx::elect_one()) ptx::mma_commit(&drain_bar);
      __syncwarp();
      ptx::mbar_wait(&drain_bar, 0, limit);
    }
  } else if (warp >= 2 + kEpiWarps) {
    // ---------------- loaders: tagged words -> operand bytes in shared memory ----------------
    // Warp lw takes chunk lw % kVSub of every kTurn-th stage whole, so that the four warps' polls, waits and fences
    // overlap (all four on one chunk took 0.5 us per chunk). Load i of lane l: word i and replicas 2 l, 2 l + 1
    // of the chunk (NR = 64), or word 2 i + l / 16 and replicas 2 (l % 16) + {0, 1} (NR = 32).
    const uint32_t lw = (uint32_t)(warp - (2 + kEpiWarps));
    constexpr int kTurn = kLoadWarps / kVSub;
    const int sub = (int)(lw % kVSub);
    const uint32_t ring = ptx::smem_u32(smem) + C::kVOff + sub * kBTile;
    const int wl = NR == 64 ? 0 : lane >> 4, pr = NR == 64 ? lane : lane & 15;
    // of eight lanes the first four write their even row first, the others their odd row: the eight swizzled
    // granules then fall in eight different bank groups
    const bool odd_first = (lane & 4) != 0;
    uint32_t g0 = 0;  // stages before this item's
    for (int ls = 0; ls < p.count && ok; ++ls)
      for (int j = 0; j < nslots && ok; ++j) {
        const RunItem w = mine[j];
        const uint32_t want = (uint32_t)ls + 1;
        const int words = 4 * w.parts;  // words beyond them multiply zero couplings
        const unsigned long long *src = p.ll + w.ll + (size_t)(ls & 1) * words * NR + wl * NR + 2 * pr;
        const int nst = (w.kchunks + kSub - 1) / kSub;
        ulonglong2 v[kLoads], nx[kLoads];  // this chunk's words, and the next one's on their way
        auto load = [&](int st, int i, ulonglong2 &d) {
          // a chunk past the last (an odd count's second half) has its words past `words`: nothing is read or
          // waited for, and the MMAs leave it out
          const int wd = (st * kVSub + sub) * kWords + i * kWordsPerLoad;
          if (wd + wl < words)
            d = ld_relaxed64x2(src + (size_t)wd * NR);
          else
            d.x = d.y = (unsigned long long)want << 32;
        };
        auto fresh = [&](const ulonglong2 &d) { return (uint32_t)(d.x >> 32) == want && (uint32_t)(d.y >> 32) == want; };
        int st = (int)((lw / kVSub - g0) & (uint32_t)(kTurn - 1));
        if (st < nst)
#pragma unroll
          for (int i = 0; i < kLoads; ++i) load(st, i, nx[i]);
        for (; st < nst; st += kTurn) {
#pragma unroll
          for (int i = 0; i < kLoads; ++i) v[i] = nx[i];
          if (st + kTurn < nst)
#pragma unroll
            for (int i = 0; i < kLoads; ++i) load(st + kTurn, i, nx[i]);
          bool all = true;
#pragma unroll
          for (int i = 0; i < kLoads; ++i) all = all && fresh(v[i]);
          if (!__all_sync(0xffffffffu, all)) {
            const long long t0 = clock64();
            do {
              __nanosleep(20);
              all = true;
#pragma unroll
              for (int i = 0; i < kLoads; ++i)
                if (!fresh(v[i])) load(st, i, v[i]);
#pragma unroll
              for (int i = 0; i < kLoads; ++i) all = all && fresh(v[i]);
              if (!__all_sync(0xffffffffu, clock64() - t0 <= limit)) ok = false;
            } while (ok && !__all_sync(0xffffffffu, all));
          }
          const uint32_t g = g0 + (uint32_t)st, s = g % STAGES;
          if (ok) ok = __all_sync(0xffffffffu, ptx::mbar_wait(&empty_bar[s], ((g / STAGES) & 1) ^ 1, limit));
          if (!ok) break;
          const uint32_t tile = ring + s * kStage;
#pragma unroll
          for (int i = 0; i < kLoads; ++i) {
            const uint32_t wd = i * kWordsPerLoad + wl;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const bool odd = (h == 1) != odd_first;
              const uint32_t r = 2 * pr + (odd ? 1 : 0), x = odd ? (uint32_t)v[i].y : (uint32_t)v[i].x;
              const uint32_t a = tile + r * 128 + ((r & 7) << 4);  // granule g of the row at a ^ (g << 4)
              if constexpr (FP4) {
                st_shared16(a ^ (wd << 4), ((x << 3) & 0x88888888u) | 0x22222222u,
                            ((x << 2) & 0x88888888u) | 0x22222222u, ((x << 1) & 0x88888888u) | 0x22222222u,
                            (x & 0x88888888u) | 0x22222222u);
              } else {
                constexpr uint32_t kOne = FP6 ? 0x48484848u : 0x38383838u;  // E4M3 4.0 / 1.0
                st_shared16(a ^ (wd << 5), ((x << 7) & 0x80808080u) | kOne, ((x << 6) & 0x80808080u) | kOne,
                            ((x << 5) & 0x80808080u) | kOne, ((x << 4) & 0x80808080u) | kOne);
                st_shared16(a ^ ((2 * wd + 1) << 4), ((x << 3) & 0x80808080u) | kOne, ((x << 2) & 0x80808080u) | kOne,
                            ((x << 1) & 0x80808080u) | kOne, (x & 0x80808080u) | kOne);
              }
            }
          }
          ptx::fence_proxy_async_shared();  // these stores, then the MMA's reads
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&fullv_bar[s]);
        }
        g0 += (uint32_t)nst;
      }
  } else {
    // ---------------- epilogue: 8 warps, two per TMEM lane quadrant, each half of the columns ----------------
    const int q = warp & 3;
    const int c_lo = ((warp - 2) >> 2) * kCols;
    const uint32_t lane_off = (uint32_t)(32 * q) << 16;
    auto state_at = [&](int j) { return tmem + C::kState + (uint32_t)(2 * NR * j) + lane_off; };
    // Signs of this warp's 32 spins (lanes) and its columns c_lo .. c_lo + kCols (bits, 1: spin -1): lane k
    // stores column c_lo + k's word, whose bit l is the spin of lane order[l]
    const int order = FP4 ? 8 * (lane & 3) + (lane >> 2) : 4 * (lane & 7) + (lane >> 3);
    auto publish = [&](const RunItem &w, int tag, uint32_t neg) {
      unsigned long long *dst =
          p.ll + w.ll + ((size_t)((tag - 1) & 1) * 4 * w.parts + (w.m0 / 32 + q)) * NR + c_lo + lane;
      const uint32_t word = transpose32(__shfl_sync(0xffffffffu, neg, order), lane);
      if (lane < kCols) st_relaxed64(dst, ((unsigned long long)(uint32_t)tag << 32) | word);
    };
#pragma unroll 1
    for (int j = 0; j < nslots; ++j) {
      const RunItem w = mine[j];
      const GInst *in = p.insts + w.inst;
      const int n = in->n, R = in->R, xp = in->xp, row = w.m0 + 32 * q + lane;
      uint32_t neg = 0;
#pragma unroll
      for (int g = 0; g < kCols; g += 16) {
        uint32_t vx[16], vy[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const int r = w.r0 + c_lo + g + k;
          const bool inside = row < n && r < R;
          vx[k] = __float_as_uint(inside ? in->x[(size_t)r * xp + row] : 0.0f);
          vy[k] = __float_as_uint(inside ? in->y[(size_t)r * xp + row] : 0.0f);
        }
        ptx::tmem_st16(state_at(j) + c_lo + g, vx);
        ptx::tmem_st16(state_at(j) + NR + c_lo + g, vy);
#pragma unroll
        for (int k = 0; k < 16; ++k)
          if (!(__uint_as_float(vx[k]) > 0.0f)) neg |= 1u << (g + k);
      }
      publish(w, 1, neg);
    }
    ptx::tmem_st_wait();
    uint32_t li = 0;
#pragma unroll 1
    for (int ls = 0; ls < p.count && ok; ++ls) {
#pragma unroll 1
      for (int j = 0; j < nslots && ok; ++j, ++li) {
        const uint32_t ab = li % kAcc, use = li / kAcc;
        const RunItem w = mine[j];
        const GInst *in = p.insts + w.inst;
        const float pump = in->pumps[p.tick0 + ls - in->t0];
        const float c0 = in->c0, dt = in->dt, dta0 = in->dta0;
        const float hv = hv_sh[j][32 * q + lane];
        const bool pub = ls + 1 < p.count && !(ls == p.skip_step && item_at(j) == p.skip_item);
        const uint32_t t_acc = tmem + ab * NR + lane_off + c_lo, t_x = state_at(j) + c_lo, t_y = t_x + NR;
        const uint64_t hv2 = pack2(hv, hv), np2 = pack2(-pump, -pump), c2 = pack2(c0, c0), dt2 = pack2(dt, dt),
                       da2 = pack2(dta0, dta0);
        uint32_t neg = 0;
        uint32_t vx[16], vy[16], va[16];
        ptx::tmem_ld16(t_x, vx);
        ptx::tmem_ld16(t_y, vy);
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&accf_bar[ab], use & 1, limit))) {
          ptx::tmem_ld_wait();  // the loads above, before tensor memory is freed
          ok = false;
          break;
        }
        ptx::tc_fence_after();
#pragma unroll
        for (int g = 0; g < kCols / 16; ++g) {
          if (g > 0) {
            ptx::tmem_ld16(t_x + 16 * g, vx);
            ptx::tmem_ld16(t_y + 16 * g, vy);
          }
          ptx::tmem_ld16(t_acc + 16 * g, va);
          ptx::tmem_ld_wait();
          if (16 * (g + 1) == kCols) {
            // this warp has read its part of the accumulator
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&acce_bar[ab]);
          }
          // sb_update on pairs of columns (the same operations and roundings). Padded spins hold x = y = 0
          // and see f = h = 0: they stay +0. Padded replicas run along on the field of their own signs and
          // are never stored.
#pragma unroll
          for (int k = 0; k < 16; k += 2) {
            uint64_t x2 = pack2(__uint_as_float(vx[k]), __uint_as_float(vx[k + 1]));
            uint64_t y2 = pack2(__uint_as_float(vy[k]), __uint_as_float(vy[k + 1]));
            const uint64_t f2 = add2(pack2(__uint_as_float(va[k]), __uint_as_float(va[k + 1])), hv2);
            y2 = fma2(dt2, fma2(np2, x2, mul2(c2, f2)), y2);
            x2 = fma2(da2, y2, x2);
            float x[2], y[2];
            unpack2(x2, x[0], x[1]);
            unpack2(y2, y[0], y[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              if (fabsf(x[e]) > 1.0f) {
                x[e] = copysignf(1.0f, x[e]);
                y[e] = 0.0f;
              }
              if (!(x[e] > 0.0f)) neg |= 1u << (16 * g + k + e);
              vx[k + e] = __float_as_uint(x[e]);
              vy[k + e] = __float_as_uint(y[e]);
            }
          }
          ptx::tmem_st16(t_x + 16 * g, vx);
          ptx::tmem_st16(t_y + 16 * g, vy);
        }
        if (pub) publish(w, ls + 2, neg);
        ptx::tmem_st_wait();
      }
    }
    if (ok) {
#pragma unroll 1
      for (int j = 0; j < nslots; ++j) {
        const RunItem w = mine[j];
        const GInst *in = p.insts + w.inst;
        const int n = in->n, R = in->R, xp = in->xp, row = w.m0 + 32 * q + lane;
#pragma unroll 1
        for (int c = c_lo; c < c_lo + kCols; c += 16) {
          uint32_t vx[16], vy[16];
          ptx::tmem_ld16(state_at(j) + c, vx);
          ptx::tmem_ld16(state_at(j) + NR + c, vy);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const int r = w.r0 + c + k;
            if (row < n && r < R && SB_BOUNDS(row < xp, p.status)) {
              in->x[(size_t)r * xp + row] = __uint_as_float(vx[k]);
              in->y[(size_t)r * xp + row] = __uint_as_float(vy[k]);
            }
          }
        }
      }
    }
  }
  if (!ok) atomicOr(p.status, kErrWaitTimeout);
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

}  // namespace tck
}  // namespace sbk
