// Instantiates the graph-form region kernel (regionKernel, one launch per region) for every
// (streams per word, groups per item) pair, with exec levels run as warp programs.
#include "cycle_kernel.cuh"

namespace tgs {

void *regionKernelProgram(int spw, int G) { return regionKernelPtrT<kLevelsProgram>(spw, G); }

}  // namespace tgs
