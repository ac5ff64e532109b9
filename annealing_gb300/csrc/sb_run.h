// Host interface of the multi-step kernel with tagged sign words (sb_run.cuh, sb_run.cu).
#pragma once
#include <cuda_runtime.h>

namespace sbk {

struct RunArgs;  // sb_run.cuh

// Most items a CTA holds for a replica tile of nr (0: no kernel for it).
int run_slots(int nr);
// One cooperative launch of `grid` CTAs (nr 32 or 64; op: GOperand; res: J rows resident).
cudaError_t launch_run(int nr, int op, bool res, const RunArgs &a, int grid, cudaStream_t st);

}  // namespace sbk
