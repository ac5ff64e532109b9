// Instantiations and launch of the multi-step kernel with tagged sign words.
#include "sb_run.cuh"

#include <string.h>

#include "sb_run.h"

namespace sbk {
namespace {
using namespace tck;

template <int NR, bool RES>
cudaError_t launch_as(int op, const RunArgs &a, int grid, cudaStream_t st) {
  const void *k = op == kGopE2m1   ? reinterpret_cast<const void *>(&run_kernel<NR, kGopE2m1, RES>)
                  : op == kGopE2m3 ? reinterpret_cast<const void *>(&run_kernel<NR, kGopE2m3, RES>)
                  : op == kGopFp8x2 ? reinterpret_cast<const void *>(&run_kernel<NR, kGopFp8x2, RES>)
                                   : reinterpret_cast<const void *>(&run_kernel<NR, kGopFp8, RES>);
  const size_t smem = op == kGopFp8x2 ? RunCfg<NR, RES, 1>::kSmem : RunCfg<NR, RES>::kSmem;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void *args[] = {const_cast<RunArgs *>(&a)};
  // every CTA waits for other CTAs' signs: all of them must be resident
  return cudaLaunchCooperativeKernel(k, dim3((unsigned)grid), dim3(kRunThreads), args, smem, st);
}
}  // namespace

int run_slots(int nr) {
  return nr == 32 ? RunCfg<32, false>::kSlots : (nr == 64 ? RunCfg<64, false>::kSlots : 0);
}

cudaError_t launch_run(int nr, int op, bool res, const RunArgs &a, int grid, cudaStream_t st) {
  switch (nr) {
    case 32: return res ? launch_as<32, true>(op, a, grid, st) : launch_as<32, false>(op, a, grid, st);
    case 64: return res ? launch_as<64, true>(op, a, grid, st) : launch_as<64, false>(op, a, grid, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace sbk
