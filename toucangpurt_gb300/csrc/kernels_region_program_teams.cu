// Instantiates the graph-form region kernel (regionKernel, one launch per region) for every
// (streams per word, groups per item) pair of 8 streams per word, with warp programs run by teams of warps, one block per SM.
#include "cycle_kernel.cuh"

namespace tgs {

void *regionKernelProgramTeams(int spw, int G) { return regionKernelPtrT<kLevelsProgramTeams>(spw, G); }

}  // namespace tgs
