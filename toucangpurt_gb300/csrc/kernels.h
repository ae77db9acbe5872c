// Launch wrappers of the device code (cycle_kernel.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "devimage.h"

namespace tgs {

struct LaunchCfg {
  int spw = 1, G = 1;
  int lv = kLevelsStaged;  // where blocks read the exec levels
  uint32_t blocks = 1, threads = 256;
  uint32_t teams = 1;        // teams of `threads` threads per block (kLevelsProgramTeams)
  size_t smem = 0;
  cudaStream_t stream = nullptr;
};

// A register write: nibble val[i] to register id[i].
struct RegPoke {
  uint32_t n = 0;
  uint32_t id[16];
  uint8_t val[16];
};

void *cycleKernelFor(int spw, int G, int lv);
void *regionKernelFor(int spw, int G, int lv);
// instantiated one per translation unit (kernels_*.cu)
void *cycleKernelStaged(int spw, int G);
void *cycleKernelResident(int spw, int G);
void *regionKernelStaged(int spw, int G);
void *regionKernelResident(int spw, int G);
void *cycleKernelProgram(int spw, int G);
void *cycleKernelProgramResident(int spw, int G);
void *regionKernelProgram(int spw, int G);
void *cycleKernelProgramTeams(int spw, int G);
void *regionKernelProgramTeams(int spw, int G);
// blocks that own their streams (kernels_own_streams.cu), 8 streams per word
void *ownStreamsKernelFor(int G);
cudaError_t launchOwnStreams(const LaunchCfg &c, const KParams &p, uint32_t c0, uint32_t n);
cudaError_t enqueueGraphChunk(const LaunchCfg &c, const KParams &p, uint32_t k, bool admit);
cudaError_t launchStimulus(int spw, const KParams &p, uint32_t cycle, cudaStream_t st);
cudaError_t launchCycles(const LaunchCfg &c, const KParams &p, uint32_t c0, uint32_t n);
cudaError_t launchInitState(int spw, const KParams &p, cudaStream_t st);
cudaError_t launchInitMems(const KParams &p, cudaStream_t st);
cudaError_t launchRegDigest(int spw, const uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t nStreams,
                            unsigned long long *out, cudaStream_t st);
cudaError_t launchRegDigestOne(const uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t g, uint32_t k,
                               unsigned long long *out, cudaStream_t st);
// image: the pools' initial contents (16-byte aligned, whole 16-byte pieces), or null
cudaError_t launchMemDigest(const uint8_t *mems, unsigned long long stride, uint32_t size, uint32_t nStreams,
                            const uint8_t *image, unsigned long long *out, cudaStream_t st);
cudaError_t launchGatherRegs(const uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t g, uint32_t k, uint8_t *out,
                             cudaStream_t st);
cudaError_t launchScatterRegs(uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t g, uint32_t k, const uint8_t *in,
                              cudaStream_t st);
cudaError_t launchPeekRegs(const uint32_t *regs, uint32_t gpad, uint32_t g, uint32_t k, const uint32_t *ids,
                           uint8_t *out, uint32_t n, cudaStream_t st);
cudaError_t launchPokeRegs(uint32_t *regs, uint32_t gpad, uint32_t g, uint32_t k, const RegPoke &q, cudaStream_t st);

}  // namespace tgs
