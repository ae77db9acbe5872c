// Instantiates the persistent cooperative cycle kernel (cycleKernel) for every
// (streams per word, groups per item) pair, with exec levels run as warp programs.
#include "cycle_kernel.cuh"

namespace tgs {

void *cycleKernelProgram(int spw, int G) { return cycleKernelPtrT<kLevelsProgram>(spw, G); }

}  // namespace tgs
