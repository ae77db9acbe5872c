// Instantiates the persistent cooperative cycle kernel (cycleKernel) for every
// (streams per word, groups per item) pair, with warp programs kept in shared memory for the whole launch.
#include "cycle_kernel.cuh"

namespace tgs {

void *cycleKernelProgramResident(int spw, int G) { return cycleKernelPtrT<kLevelsProgramResident>(spw, G); }

}  // namespace tgs
