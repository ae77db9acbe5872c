// Instantiates the persistent cooperative cycle kernel (cycleKernel) for every
// (streams per word, groups per item) pair of 8 streams per word, with warp programs run by teams of warps, one block per SM.
#include "cycle_kernel.cuh"

namespace tgs {

void *cycleKernelProgramTeams(int spw, int G) { return cycleKernelPtrT<kLevelsProgramTeams>(spw, G); }

}  // namespace tgs
