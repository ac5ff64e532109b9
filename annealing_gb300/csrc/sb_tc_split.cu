// Instantiations of the tcgen05 SB kernel for BF16 hi + lo operands (real couplings: dSB, and bSB with x split too;
// the dSB energy mode also ranks bSB replicas: sign operands against the split couplings).
#include "sb_tc_kernel.cuh"

namespace sbk {

bool tc_kernel_split(int variant, int nr, int emode, const void **k, size_t *smem, bool pair) {
  if (variant == 2) {
    switch (nr) {
      case 32: return tck::tc_lookup<kTcBf16Split, 2, 32, 7>(emode, k, smem);
      case 64: return tck::tc_lookup<kTcBf16Split, 2, 64, 7>(emode, k, smem);
      case 128: return tck::tc_lookup<kTcBf16Split, 2, 128, 7>(emode, k, smem);
    }
  }
  if (pair) {
    if (variant != 1 || nr != 128 || emode != tck::kEmodeStep) return false;
    tck::tc_lookup_pair<kTcBf16Split>(k, smem);
    return true;
  }
  if (variant == 1) {
    switch (nr) {
      case 32: return tck::tc_lookup<kTcBf16Split, 1, 32, 1>(emode, k, smem);
      case 64: return tck::tc_lookup<kTcBf16Split, 1, 64, 1>(emode, k, smem);
      case 128: return tck::tc_lookup<kTcBf16Split, 1, 128, 1>(emode, k, smem);
    }
  }
  return false;
}

}  // namespace sbk
