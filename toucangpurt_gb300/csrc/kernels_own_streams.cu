// Blocks that own their streams: the batched runs of designs with one
// partition per region (thousands of streams of a small design).
//
// A block evaluates both partitions of its stream groups, so no other block
// ever touches their registers, exchange words or memories.  It then needs no
// grid barrier, applies its own inputs, digests its own registers, and
// retires and admits its own slots (the queue's head is the only word shared
// with other blocks); blocks drift apart freely and a retirement holds up its
// own block alone, without the cycle that the grid-wide form spends on it.
// What is left of a cycle is the latency of its levels, its level-0 reads and
// its last levels.  1,024 queued streams of the 4K-LUT design (35 blocks, about
// 1,000 retirements in 2,000 cycles): 34.6 -> 20.8 ms a call.
#include "cycle_kernel.cuh"

namespace tgs {
namespace {

template <int G>
struct OwnStreams {
  static constexpr uint32_t N = 8u * G;
  uint32_t stream[N];  // job stream (queued) or stream, kNoStream when idle
  uint32_t start[N];   // cycle of the stream's cycle 0 (queued)
  uint32_t retire[N];  // cycle after its last one (queued)
  unsigned long long seed[N], dig[N], roll[N];
  unsigned long long red[2];  // register and memory digest of a retiring stream
  uint32_t next;              // the stream admitted in its place
};

// The next inputs of the block's streams (applyStimulus for its own groups).
template <int G>
__device__ void ownStimulus(const KParams &p, const OwnStreams<G> &o, uint32_t t, uint32_t s0) {
  const bool slots = (p.flags & kFlagSlots) != 0, stopExit = (p.flags & kFlagStopExit) != 0;
  const uint32_t k = threadIdx.x & 7u, total = p.nStim * G, lanes = (total * 8u + 31u) & ~31u;
  for (uint32_t x = threadIdx.x; x < lanes; x += blockDim.x) {
    const uint32_t i = x >> 3;
    uint32_t part = 0, *wp = nullptr;
    if (i < total) {
      const uint32_t inp = i / G, g = i % G, s = g * 8u + k;
      const uint32_t reg = __ldg(p.stimReg + inp), mask = (1u << __ldg(p.stimBits + inp)) - 1u;
      const uint32_t tog = p.stimToggle ? uint32_t(__ldg(p.stimToggle + inp)) : 0u;
      wp = p.regs + size_t(reg) * p.gpad + blockIdx.x * G + g;
      const uint32_t cur = nib(__ldcg(wp), k);
      uint32_t v = cur;
      if (o.stream[s] != kNoStream && t < o.retire[s] && !(stopExit && __ldcg(p.stopCycle + s0 + s) < t)) {
        if (!slots && p.stimTable) {
          v = __ldg(p.stimTable + (size_t(t - p.stimTableC0) * p.nStim + inp) * p.nStreams + s0 + s) & 15u;
        } else {
          const uint32_t lc = slots ? t - o.start[s] : t;
          const unsigned long long h = dmix64(o.seed[s] ^ dmix64((unsigned long long)lc << 32 | inp));
          v = tog == 0 ? uint32_t(h) & mask : (h >> 48) < tog ? cur ^ mask : cur;
        }
      }
      part = v << (4u * k);
    }
    part |= __shfl_xor_sync(kFull, part, 1);
    part |= __shfl_xor_sync(kFull, part, 2);
    part |= __shfl_xor_sync(kFull, part, 4);
    if (wp && k == 0) *wp = part;
  }
}

// Register digests of the block's streams, summed in shared memory.
template <int G>
__device__ void ownDigest(const KParams &p, OwnStreams<G> &o) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
  uint32_t chunk = 256, chunks = (p.regSlots + 255u) / 256u;
  while (chunk > 32u && chunks * G < NW) {
    chunk >>= 1;
    chunks = (p.regSlots + chunk - 1u) / chunk;
  }
  for (uint32_t u = warp; u < chunks * G; u += NW) {
    const uint32_t g = u % G, ch = u / G, end = min(p.regSlots, ch * chunk + chunk);
    unsigned long long acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0;
    for (uint32_t i = ch * chunk + lane; i < end; i += 32) {
      const uint32_t w = __ldcg(p.regs + size_t(i) * p.gpad + blockIdx.x * G + g);
      const MixIndex mix(i);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += mix(nib(w, k));
    }
    const uint32_t k = sumStreams(acc, lane);
    if ((lane & 3u) == 0u) atomicAdd(&o.dig[g * 8u + k], acc[0]);
  }
}

// Retires slot s (its stream ended before cycle t) and admits the queue's
// next stream, whose cycle 0 is cycle t.  The block reads the whole memory by
// itself, whatever its size: the others go on meanwhile, where a retirement of
// the grid-wide form holds up all of them.  1,000 streams of 50 to 500 cycles
// on 200 slots, memories of 8 KiB / 512 KiB / 2 MiB: 9.3 / 17.7 / 45.9 ms, grid-wide 15.9 /
// 25.7 / 59.2; 192 streams of 1,000 cycles beside 200 of 5: 9.6 / 12.7 / 24.1
// and 14.7 / 18.6 / 32.3.
template <int G>
__device__ void ownRetire(const KParams &p, OwnStreams<G> &o, uint32_t t, uint32_t s0, uint32_t s) {
  const uint32_t g = blockIdx.x * G + s / 8u, k = s % 8u, tid = threadIdx.x, nthr = blockDim.x;
  const uint32_t vecs = (p.memPoolSize + 15u) / 16u;
  uint8_t *mem = p.mems + (unsigned long long)(s0 + s) * p.memStride;
  if (tid < 2) o.red[tid] = 0;
  __syncthreads();
  unsigned long long a = 0, m = 0;
  for (uint32_t i = tid; i < p.regSlots; i += nthr) {
    uint32_t *w = p.regs + size_t(i) * p.gpad + g;
    const uint32_t v = __ldcg(w);
    a += MixIndex(i)(nib(v, k));
    *w = (v & ~(15u << (4u * k))) | (uint32_t(p.initRegs[i]) & 15u) << (4u * k);
  }
  for (uint32_t v = tid; v < vecs; v += nthr) {
    const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(mem) + v);  // strides are whole 16-byte pieces
    m += memTerms(q, 16u * v, min(16u, p.memPoolSize - 16u * v));
    reinterpret_cast<uint4 *>(mem)[v] = __ldg(reinterpret_cast<const uint4 *>(p.initMems) + v);
  }
  for (int w = 16; w > 0; w >>= 1) {
    a += __shfl_xor_sync(kFull, a, w);
    m += __shfl_xor_sync(kFull, m, w);
  }
  if ((tid & 31u) == 0) {
    atomicAdd(&o.red[0], a);
    atomicAdd(&o.red[1], m);
  }
  __syncthreads();
  if (tid == 0) {
    const uint32_t q = o.stream[s], sc = __ldcg(p.stopCycle + s0 + s);
    p.outReg[q] = o.red[0];
    p.outMem[q] = o.red[1];
    p.outRoll[q] = o.roll[s];
    p.outStop[q] = sc == 0xFFFFFFFFu ? sc : sc - o.start[s];
    const uint32_t at = atomicAdd(p.queueHead, 1u), qn = at < p.nJobs ? __ldg(p.queueOrder + at) : kNoStream;
    o.stream[s] = o.next = qn;
    o.start[s] = t;
    o.retire[s] = qn == kNoStream ? 0u : t + __ldg(p.jobLen + qn);
    o.seed[s] = qn == kNoStream ? 0ull : __ldg(p.jobSeed + qn);
    o.roll[s] = 0;
    o.dig[s] = 0;
    p.stop[s0 + s] = 0;
    p.stopCycle[s0 + s] = 0xFFFFFFFFu;
  }
  __syncthreads();
  // the admitted stream's first inputs, from the initial register values
  if (o.next != kNoStream && (p.flags & kFlagStimulus))
    for (uint32_t inp = tid; inp < p.nStim; inp += nthr) {
      const uint32_t reg = __ldg(p.stimReg + inp), mask = (1u << __ldg(p.stimBits + inp)) - 1u;
      const uint32_t tog = p.stimToggle ? uint32_t(__ldg(p.stimToggle + inp)) : 0u;
      const uint32_t cur = p.initRegs[reg] & 15u;
      const unsigned long long h = dmix64(o.seed[s] ^ dmix64((unsigned long long)inp));
      const uint32_t v = tog == 0 ? uint32_t(h) & mask : (h >> 48) < tog ? cur ^ mask : cur;
      uint32_t *w = p.regs + size_t(reg) * p.gpad + g;
      atomicAnd(w, ~(15u << (4u * k)));
      atomicOr(w, v << (4u * k));
    }
  __syncthreads();
}

template <int G>
__global__ void __launch_bounds__(kResidentThreads) ownStreamsKernel(const KParams p, uint32_t c0, uint32_t nCycles) {
  constexpr uint32_t N = OwnStreams<G>::N;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) unsigned long long stageMbar[2];
  __shared__ uint32_t itemLists[2 * kItemListWords];
  __shared__ OwnStreams<G> o;
  BlockSmem b;
  if (!setupBlock<G, kLevelsProgramResident>(p, smem, stageMbar, b, -1)) {
    if (threadIdx.x == 0) p.status[0] = kErrTimeout;
    return;
  }
  loadItemLists(p, b, itemLists);
  const bool slots = (p.flags & kFlagSlots) != 0, stopExit = (p.flags & kFlagStopExit) != 0;
  const bool digest = (p.flags & kFlagDigest) != 0, stim = (p.flags & kFlagStimulus) != 0;
  const uint32_t tid = threadIdx.x, s0 = blockIdx.x * N;
  for (uint32_t s = tid; s < N; s += blockDim.x) {
    const bool in = s0 + s < p.nStreams;
    const uint32_t q = !in ? kNoStream : slots ? __ldcg(p.slotStream + s0 + s) : s0 + s;
    o.stream[s] = q;
    o.start[s] = 0;
    o.retire[s] = slots ? (q == kNoStream ? 0u : __ldcg(p.slotRetire + s0 + s)) : 0xFFFFFFFFu;
    o.seed[s] = stim && q != kNoStream ? (slots ? __ldg(p.jobSeed + q) : __ldg(p.streamSeed + q)) : 0ull;
    o.dig[s] = 0;
    o.roll[s] = in && !slots ? __ldcg(p.roll + s0 + s) : 0ull;
  }
  __syncthreads();
  if (stim) ownStimulus<G>(p, o, c0, s0);
  __syncthreads();
  bool look = true;  // a slot may retire before this cycle, or none is left
  uint32_t nextRetire = 0xFFFFFFFFu;
  for (uint32_t t = c0; slots || t < c0 + nCycles; ++t) {
    if (slots && (look || t >= nextRetire)) {
      bool active = false;
      nextRetire = 0xFFFFFFFFu;
      for (uint32_t s = 0; s < N; ++s) {
        if (o.stream[s] == kNoStream) continue;
        if (t >= o.retire[s] || (stopExit && __ldcg(p.stopCycle + s0 + s) < t)) ownRetire<G>(p, o, t, s0, s);
        if (o.stream[s] == kNoStream) continue;
        active = true;
        nextRetire = min(nextRetire, o.retire[s]);
      }
      if (!active) break;
    }
    // an error that any block raised ends the run: the word is read early in
    // every sixteenth cycle and looked at behind its last barrier (0.6 % of the
    // time when every cycle did)
    const bool errCycle = (t & 15u) == 15u;
    const uint32_t err = errCycle && tid == 0 ? *static_cast<volatile uint32_t *>(p.err) : 0u;
    const uint32_t n0 = ldsU32(b.items), n1 = ldsU32(b.items + 4u * kItemListWords);
#pragma unroll 1
    for (uint32_t i = 0; i < n0 + n1; ++i) {
      if (i == n0 && digest) ownDigest<G>(p, o);  // the registers are read-only until region 1's last levels
      const uint32_t at = b.items + 4u * (i < n0 ? 1u + 2u * i : kItemListWords + 1u + 2u * (i - n0));
      evalItem<8, G, kLevelsProgramResident>(p, ldsU32(at), b.vp, b.tab, b.st, t, nullptr, ldsU32(at + 4u), b.resState);
    }
    if (stim && (slots || t + 1 < c0 + nCycles)) ownStimulus<G>(p, o, t + 1, s0);
    // (evalItem ends with a block barrier: the digests are complete)
    bool stopped = false, running = false;
    for (uint32_t s = tid; s < N; s += blockDim.x) {
      const uint32_t q = o.stream[s], sc = stopExit && q != kNoStream ? __ldcg(p.stopCycle + s0 + s) : 0xFFFFFFFFu;
      if (q == kNoStream) continue;
      stopped |= sc <= t;
      running |= sc > t;
      if (!digest || sc < t) continue;
      const unsigned long long dg = o.dig[s];
      const uint32_t lc = slots ? t - o.start[s] : t - p.cycBase;
      o.roll[s] = dmix64(o.roll[s] + dg);
      if (p.cycDig && lc < p.cycStride) p.cycDig[size_t(q) * p.cycStride + lc] = dg;
    }
    if (digest)
      for (uint32_t s = tid; s < N; s += blockDim.x) o.dig[s] = 0;
    look = false;
    if (stopExit || errCycle) {
      look = __syncthreads_or(int(stopped || err != 0u)) != 0;
      if (look && __syncthreads_or(int(err != 0u))) break;
      if (!slots && look && !__syncthreads_or(int(running))) break;  // every stream of the block is frozen
    } else {
      __syncthreads();
    }
  }
  if (!slots)
    for (uint32_t s = tid; s < N; s += blockDim.x)
      if (s0 + s < p.nStreams) p.roll[s0 + s] = o.roll[s];
  // the run's outcome for the host (zeroed before the launch): each block adds
  // what it has seen, the block that raised an error that one at least
  uint32_t any = 0;
  for (uint32_t s = tid; s < N; s += blockDim.x)
    if (s0 + s < p.nStreams) any |= __ldcg(p.stop + s0 + s);
  const int stopped = __syncthreads_or(int(any));
  if (tid == 0) {
    const uint32_t err = __ldcg(p.err);
    if (stopped) p.status[1] = 1u;
    if (err != 0u) p.status[0] = err;
  }
}

template <int G>
void *kernelPtr() {
  return reinterpret_cast<void *>(&ownStreamsKernel<G>);
}

}  // namespace

void *ownStreamsKernelFor(int G) {
  return G == 8 ? kernelPtr<8>() : G == 4 ? kernelPtr<4>() : G == 2 ? kernelPtr<2>() : kernelPtr<1>();
}

cudaError_t launchOwnStreams(const LaunchCfg &c, const KParams &p, uint32_t c0, uint32_t n) {
  KParams pp = p;
  void *args[] = {&pp, &c0, &n};
  return cudaLaunchKernel(ownStreamsKernelFor(c.G), dim3(c.blocks), dim3(c.threads), args, c.smem, c.stream);
}

}  // namespace tgs
