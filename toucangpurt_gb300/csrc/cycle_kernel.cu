// Small kernels of the cycle loop (graph-form admission, stimulus, cycle
// counter), state utilities, and the host-side launch wrappers.  The cycle
// and region kernels are instantiated in kernels_{persistent,region}_*.cu, one
// translation unit for each source of exec levels, and kernels_own_streams.cu,
// so the build compiles them in parallel.
#include "cycle_kernel.cuh"

namespace tgs {
namespace {

// Graph form, after region 1 (and the stop-exit inputs): admission (one
// block), cycle bookkeeping, the early-exit word.
template <int SPW>
__global__ void admitKernel(const KParams p, uint32_t k) {
  const uint32_t t = __ldcg(p.graphState) + k;
  // graphState[4] (exit) is written only here, after the cycle's regions
  if (t >= __ldcg(p.graphState + 2) || __ldcg(p.graphState + 4) || __ldcg(p.err)) return;
  const bool slots = (p.flags & kFlagSlots) != 0;
  const bool event = slots && __ldcg(p.retCount) != 0;
  if (event) eventAdmit<SPW>(p, t, threadIdx.x, blockDim.x);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (p.flags & kFlagCountCycles) *p.realCycles += 1;
    if (slots) {
      if (event && __ldcg(p.nDone) >= p.nJobs) p.graphState[4] = 1;
    } else if ((p.flags & kFlagStopExit) && __ldcg(p.nStopped) >= p.nStreams) {
      p.graphState[4] = 1;
    }
  }
}

// Graph form, stop exit: the next cycle's inputs, after the region-1 launch.
template <int SPW>
__global__ void graphStimulusKernel(const KParams p, uint32_t k) {
  const uint32_t t = __ldcg(p.graphState) + k;
  if (t + 1 >= __ldcg(p.graphState + 2) || __ldcg(p.graphState + 4) || __ldcg(p.err)) return;
  applyStimulus<SPW>(p, t + 1, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

__global__ void advanceKernel(uint32_t *counter, uint32_t k) { *counter += k; }

template <int SPW>
__global__ void stimulusKernel(const KParams p, uint32_t cycle) {
  applyStimulus<SPW>(p, cycle, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ---- state utilities -----------------------------------------------------------
template <int SPW>
__global__ void initStateKernel(const KParams p) {
  const size_t n = size_t(p.regSlots) * p.gpad;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    const uint32_t v = p.initRegs[i / p.gpad];
    p.regs[i] = SPW == 8 ? rep8(v) : v;
  }
  const size_t ne = size_t(p.exgSlots) * p.gpad;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < ne; i += size_t(gridDim.x) * blockDim.x) p.exg[i] = 0;
}

// Every stream's memories from the initial image: a thread reads 16 bytes
// once and writes them to each stream of its block row (image and strides are
// whole 16-byte pieces), so a reset writes each memory once and reads the
// image once per kInitStreams streams instead of copying it per stream.
// 16M-LUT design, 64 x 512 MiB: 10.4 ms -> 5.27 ms (6.5 TB/s written).
constexpr uint32_t kInitStreams = 64;

__global__ void __launch_bounds__(256) initMemsKernel(const uint8_t *__restrict__ init, uint8_t *__restrict__ mems,
                                                     unsigned long long stride, uint32_t vecs, uint32_t nStreams) {
  const uint32_t s0 = blockIdx.y * kInitStreams, s1 = min(nStreams, s0 + kInitStreams);
  for (uint32_t v = blockIdx.x * 256u + threadIdx.x; v < vecs; v += gridDim.x * 256u) {
    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(init) + v);
    for (uint32_t s = s0; s < s1; ++s) __stcs(reinterpret_cast<uint4 *>(mems + s * stride) + v, w);
  }
}

// Digest of one pool per stream: sum over i of mix64(i << 8 | v_i).
// A block takes up to kDigestStreams streams, a thread the same 16 bytes of
// each of them.  Streams' memories start equal and are written sparsely, so a
// thread computes the 16 terms of the initial image (of the first stream,
// where there is none) once and, for every stream, only what differs from it: nothing when the warp's 512 bytes are
// equal; the differing bytes when up to half of the lanes differ, gathered by
// the warp and taken 32 at a time, one a lane; all 16 terms (17 instructions a
// byte beside the index part) otherwise.
// Measured, 64 pools of 128 MiB (17.5 ms in every case when each byte took the
// whole 27-instruction mix and a thread read one byte a step): equal 1.25 ms
// (6.9 TB/s, bound by HBM), 0.5 % of a pool's bytes differing 3.25 ms (4.3 with
// each lane taking its own bytes, a few of 32 lanes at work), all random
// 12.9 ms, both bound by instructions.  Half the lanes as the line: with 8
// lanes 8.2 ms at 0.5 %, 16 and 24 lanes 4.8 ms.  64 registers (4 blocks an SM)
// over 80 and 128 (index parts kept): 4.3 / 4.8 / 5.4 ms at 0.5 %.
constexpr uint32_t kDigestThreads = 256, kDigestStreams = 64;
constexpr uint32_t kDigestQueue = 64;   // differing bytes a warp gathers
constexpr uint32_t kDigestSparse = 16;  // lanes of a warp that differ, up to which their bytes are taken one by one

__global__ void __launch_bounds__(kDigestThreads, 4)
    memDigestKernel(const uint8_t *__restrict__ mems, unsigned long long stride, uint32_t size, uint32_t nStreams,
                    const uint8_t *__restrict__ image, unsigned long long *__restrict__ out) {
  __shared__ unsigned long long sum[kDigestThreads / 32][kDigestStreams];  // per warp: stream's sum less ref's (wrapping)
  __shared__ unsigned long long sum0;
  __shared__ uint32_t piece[kDigestThreads / 32u][kDigestStreams][3], queue[kDigestThreads / 32u][kDigestQueue];
  const uint32_t s0 = blockIdx.y * kDigestStreams, ns = min(kDigestStreams, nStreams - s0);
  const uint8_t *base = mems + s0 * stride;
  // what the streams are compared with: the initial image (a byte the first
  // stream wrote would differ from every other), or the first stream
  const uint8_t *ref = image ? image : base;
  const uint32_t kFirst = image ? 0u : 1u;
  for (uint32_t i = threadIdx.x; i < kDigestThreads / 32u * kDigestStreams; i += kDigestThreads) (&sum[0][0])[i] = 0;
  for (uint32_t i = threadIdx.x; i < kDigestThreads / 32u * kDigestStreams * 3u; i += kDigestThreads) (&piece[0][0][0])[i] = 0;
  if (threadIdx.x == 0) sum0 = 0;
  __syncthreads();
  unsigned long long acc0 = 0;
  const uint32_t vecs = size / 16u, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  // whole warps iterate together (a lane past the end repeats the last vector with weight 0)
  for (uint32_t w = blockIdx.x * kDigestThreads + threadIdx.x - lane; w < vecs; w += gridDim.x * kDigestThreads) {
    const bool in = w + lane < vecs;
    const uint32_t v = in ? w + lane : vecs - 1u;
    const uint4 *src = reinterpret_cast<const uint4 *>(base) + v;
    const uint4 f = __ldg(reinterpret_cast<const uint4 *>(ref) + v);
    // the 16 indices share z >> 30 (and so its low byte) unless their low 30
    // bits wrap; values of 0x80 and above, which a pool may hold when the
    // caller wrote them, may carry out of the low byte: both take the full mix
    const unsigned long long i0 = 16ull * v, z0 = (i0 << 8) + kMixC;
    const bool flat = (uint32_t(z0) & 0x3FFFFFFFu) + 0xF00u < 0x40000000u;
    const uint32_t kk = uint32_t(z0 >> 30) & 0xFFu;
    auto sum16 = [&](const uint4 &x) {
      unsigned long long s = 0;
      if (flat && ((x.x | x.y | x.z | x.w) & 0x80808080u) == 0u) {
        const uint32_t y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 16; ++j) s += MixIndex::term(MixIndex(i0 + j).p, kk, (y[j / 4] >> (8 * (j % 4))) & 0xFFu);
      } else {
#pragma unroll 1
        for (int j = 0; j < 16; ++j) {
          const uint32_t y = j < 8 ? (j < 4 ? x.x : x.y) : (j < 12 ? x.z : x.w);
          s += dmix64((i0 + j) << 8 | ((y >> (8 * (j % 4))) & 0xFFu));
        }
      }
      return s;
    };
    const unsigned long long first = sum16(f);
    if (in) acc0 += first;
    uint32_t queued = 0;  // the same in every lane
    // the terms of up to 32 queued bytes, one a lane: added to their streams'
    // pieces (22, 21 and 21 bits: an iteration adds at most 512 times to one)
    auto flush = [&]() {
      __syncwarp();
      if (lane < queued) {
        const uint32_t e = queue[warp][lane], a = e & 0xFFu, b = (e >> 8) & 0xFFu, k = e >> 25;
        const unsigned long long i = 16ull * w + ((e >> 16) & 511u);
        unsigned long long s;
        if ((a | b) < 0x80u) {
          const MixIndex mix(i);
          s = mix(a) - mix(b);
        } else {
          s = dmix64(i << 8 | a) - dmix64(i << 8 | b);
        }
        atomicAdd(&piece[warp][k][0], uint32_t(s) & 0x3FFFFFu);
        atomicAdd(&piece[warp][k][1], uint32_t(s >> 22) & 0x1FFFFFu);
        atomicAdd(&piece[warp][k][2], uint32_t(s >> 43));
      }
      __syncwarp();
    };
    bool any = false;
    auto other = [&](uint32_t k, const uint4 &q) {
      const uint4 d = make_uint4(q.x ^ f.x, q.y ^ f.y, q.z ^ f.z, q.w ^ f.w);
      const bool differs = in && (d.x | d.y | d.z | d.w) != 0u;
      const uint32_t lanes = __ballot_sync(kFull, differs);
      if (lanes == 0u) return;
      if (__popc(lanes) > kDigestSparse) {
        // sum over the warp in three pieces that fit 32 bits
        const unsigned long long s = in ? sum16(q) - first : 0ull;
        const uint32_t x0 = __reduce_add_sync(kFull, uint32_t(s) & 0x7FFFFFFu);
        const uint32_t x1 = __reduce_add_sync(kFull, uint32_t(s >> 27) & 0x7FFFFFFu);
        const uint32_t x2 = __reduce_add_sync(kFull, uint32_t(s >> 54));
        if (lane == 0)
          sum[warp][k] += (unsigned long long)x0 + ((unsigned long long)x1 << 27) + ((unsigned long long)x2 << 54);
        return;
      }
      any = true;
      // one bit per differing byte, then a byte of each lane a round
      auto bytes = [](uint32_t x) {
        return (((((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) >> 7 & 0x01010101u) * 0x01020408u >> 24) & 15u;
      };
      uint32_t m = 0;
      if (differs) m = bytes(d.x) | bytes(d.y) << 4 | bytes(d.z) << 8 | bytes(d.w) << 12;
      for (uint32_t left = lanes; left; left = __ballot_sync(kFull, m != 0u)) {
        const uint32_t n = uint32_t(__popc(left));
        if (queued + n > kDigestQueue) {
          // full: the first 32 are taken, the rest moves down
          const uint32_t rest = queued - 32u;
          const uint32_t keep = queued;
          queued = 32u;
          flush();
          if (lane < rest) queue[warp][lane] = queue[warp][32u + lane];
          queued = keep - 32u;
          __syncwarp();
        }
        if (m) {
          const uint32_t j = uint32_t(__ffs(int(m))) - 1u, sh = 8u * (j & 3u);
          m &= m - 1u;
          const uint32_t a = ((j < 8 ? (j < 4 ? q.x : q.y) : (j < 12 ? q.z : q.w)) >> sh) & 0xFFu;
          const uint32_t b = ((j < 8 ? (j < 4 ? f.x : f.y) : (j < 12 ? f.z : f.w)) >> sh) & 0xFFu;
          queue[warp][queued + uint32_t(__popc(left & ((1u << lane) - 1u)))] = a | b << 8 | (16u * lane + j) << 16 | k << 25;
        }
        queued += n;
      }
    };
    const uint8_t *at = reinterpret_cast<const uint8_t *>(src) + kFirst * stride;
    uint32_t k = kFirst;
    for (; k + 8 <= ns; k += 8, at += 8 * stride) {
      uint4 q[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) q[u] = __ldg(reinterpret_cast<const uint4 *>(at + u * stride));
#pragma unroll
      for (int u = 0; u < 8; ++u) other(k + u, q[u]);
    }
    for (; k < ns; ++k, at += stride) other(k, __ldg(reinterpret_cast<const uint4 *>(at)));
    if (any) {
      // what is still queued, then the pieces
      if (queued > 32u) {
        const uint32_t rest = queued - 32u;
        queued = 32u;
        flush();
        if (lane < rest) queue[warp][lane] = queue[warp][32u + lane];
        queued = rest;
      }
      flush();
      for (uint32_t s = lane; s < ns; s += 32u) {
        sum[warp][s] += (unsigned long long)piece[warp][s][0] + ((unsigned long long)piece[warp][s][1] << 22) +
                        ((unsigned long long)piece[warp][s][2] << 43);
        piece[warp][s][0] = piece[warp][s][1] = piece[warp][s][2] = 0u;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  // the last size % 16 bytes
  if (blockIdx.x == 0 && threadIdx.x < size % 16u) {
    const uint32_t i = size - size % 16u + threadIdx.x;
    const unsigned long long t0 = dmix64((unsigned long long)i << 8 | ref[i]);
    acc0 += t0;
    for (uint32_t k = kFirst; k < ns; ++k)
      atomicAdd(&sum[0][k], dmix64((unsigned long long)i << 8 | base[k * stride + i]) - t0);
  }
  for (int o = 16; o > 0; o >>= 1) acc0 += __shfl_xor_sync(kFull, acc0, o);
  if (lane == 0) atomicAdd(&sum0, acc0);
  __syncthreads();
  if (threadIdx.x < ns) {
    unsigned long long s = sum0;
    for (uint32_t w = 0; w < kDigestThreads / 32u; ++w) s += sum[w][threadIdx.x];
    atomicAdd(out + s0 + threadIdx.x, s);
  }
}

// The same a byte a thread: for small pools, and for pools that are not 16-byte
// aligned (caller-owned pools).
__global__ void memDigestBytesKernel(const uint8_t *__restrict__ mems, unsigned long long stride, uint32_t size,
                                     uint32_t nStreams, unsigned long long *__restrict__ out) {
  const uint32_t s = blockIdx.y;
  if (s >= nStreams) return;
  const uint8_t *m = mems + s * stride;
  unsigned long long acc = 0;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < size; i += size_t(gridDim.x) * blockDim.x)
    acc += dmix64((unsigned long long)i << 8 | m[i]);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
  if ((threadIdx.x & 31u) == 0) atomicAdd(out + s, acc);
}

template <int SPW>
__global__ void regDigestKernel(const uint32_t *__restrict__ regs, uint32_t slots, uint32_t gpad, uint32_t nStreams,
                                unsigned long long *__restrict__ out) {
  const uint32_t g = blockIdx.y;
  unsigned long long acc[SPW];
#pragma unroll
  for (int k = 0; k < SPW; ++k) acc[k] = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += gridDim.x * blockDim.x) {
    const uint32_t w = regs[size_t(i) * gpad + g];
    const MixIndex mix(i);
#pragma unroll
    for (int k = 0; k < SPW; ++k) acc[k] += mix(nib(w, k));
  }
#pragma unroll
  for (int k = 0; k < SPW; ++k) {
    unsigned long long a = acc[k];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
    const uint32_t s = g * SPW + k;
    if ((threadIdx.x & 31u) == 0 && s < nStreams) atomicAdd(out + s, a);
  }
}

// The register digest of one stream (nibble k of group g).
__global__ void regDigestOneKernel(const uint32_t *__restrict__ regs, uint32_t slots, uint32_t gpad, uint32_t g,
                                   uint32_t k, unsigned long long *__restrict__ out) {
  unsigned long long acc = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += gridDim.x * blockDim.x)
    acc += MixIndex(i)(nib(regs[size_t(i) * gpad + g], k));
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
  if ((threadIdx.x & 31u) == 0) atomicAdd(out, acc);
}

// nibble k of every register word of group g <-> one byte per register
__global__ void gatherRegsKernel(const uint32_t *__restrict__ regs, uint32_t slots, uint32_t gpad, uint32_t g,
                                 uint32_t k, uint8_t *__restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += gridDim.x * blockDim.x)
    out[i] = uint8_t(nib(regs[size_t(i) * gpad + g], k));
}

__global__ void scatterRegsKernel(uint32_t *__restrict__ regs, uint32_t slots, uint32_t gpad, uint32_t g, uint32_t k,
                                  const uint8_t *__restrict__ in) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += gridDim.x * blockDim.x) {
    uint32_t *w = regs + size_t(i) * gpad + g;
    *w = (*w & ~(15u << (4 * k))) | ((uint32_t(in[i]) & 15u) << (4 * k));
  }
}

// Writes one register's nibbles of one stream; they come as kernel arguments,
// so that setting a register copies nothing.
__global__ void pokeRegsKernel(uint32_t *__restrict__ regs, uint32_t gpad, uint32_t g, uint32_t k, const RegPoke q) {
  const uint32_t i = threadIdx.x;
  if (i >= q.n) return;
  uint32_t *w = regs + size_t(q.id[i]) * gpad + g;
  *w = (*w & ~(15u << (4 * k))) | ((uint32_t(q.val[i]) & 15u) << (4 * k));
}

// The nibbles of the listed register ids of one stream (readRegister).
__global__ void peekRegsKernel(const uint32_t *__restrict__ regs, uint32_t gpad, uint32_t g, uint32_t k,
                               const uint32_t *__restrict__ ids, uint8_t *__restrict__ out, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = uint8_t(nib(regs[size_t(ids[i]) * gpad + g], k));
}

}  // namespace

void *cycleKernelFor(int spw, int G, int lv) {
  return lv == kLevelsProgramTeams      ? cycleKernelProgramTeams(spw, G)
         : lv == kLevelsProgramResident ? cycleKernelProgramResident(spw, G)
         : lv == kLevelsProgram         ? cycleKernelProgram(spw, G)
         : lv == kLevelsResident        ? cycleKernelResident(spw, G)
                                        : cycleKernelStaged(spw, G);
}

cudaError_t launchCycles(const LaunchCfg &c, const KParams &p, uint32_t c0, uint32_t n) {
  void *fn = cycleKernelFor(c.spw, c.G, c.lv);
  KParams pp = p;
  void *args[] = {&pp, &c0, &n};
  // one block has no other to wait for
  if (c.blocks == 1) return cudaLaunchKernel(fn, dim3(1), dim3(c.threads), args, c.smem, c.stream);
  return cudaLaunchCooperativeKernel(fn, dim3(c.blocks), dim3(c.threads, c.teams), args, c.smem, c.stream);
}

void *regionKernelFor(int spw, int G, int lv) {
  return lv == kLevelsProgramTeams ? regionKernelProgramTeams(spw, G)
         : lv == kLevelsProgram    ? regionKernelProgram(spw, G)
         : lv == kLevelsResident   ? regionKernelResident(spw, G)
                                   : regionKernelStaged(spw, G);
}

// Enqueues one chunk of k cycles in graph form on the stream (captured by
// the caller): per cycle region 0, region 1 and (admission / cycle count)
// the admit kernel; then the cycle counter advance.
cudaError_t enqueueGraphChunk(const LaunchCfg &c, const KParams &p, uint32_t k, bool admit) {
  void *fn = regionKernelFor(c.spw, c.G, c.lv);
  KParams pp = p;
  for (uint32_t i = 0; i < k; ++i) {
    for (uint32_t r = 0; r < 2; ++r) {
      uint32_t ki = i, ri = r;
      void *args[] = {&pp, &ki, &ri};
      cudaError_t e = cudaLaunchKernel(fn, dim3(c.blocks), dim3(c.threads, c.teams), args, c.smem, c.stream);
      if (e != cudaSuccess) return e;
    }
    if ((p.flags & kFlagStopExit) && (p.flags & kFlagStimulus)) {
      const uint32_t n = std::max<uint32_t>(1, p.nStim * p.gpad);
      const uint32_t blocks = std::min<uint32_t>(1024, (n + 255) / 256);
      if (c.spw == 8)
        graphStimulusKernel<8><<<blocks, 256, 0, c.stream>>>(p, i);
      else
        graphStimulusKernel<1><<<blocks, 256, 0, c.stream>>>(p, i);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    if (admit) {
      if (c.spw == 8)
        admitKernel<8><<<1, 256, 0, c.stream>>>(p, i);
      else
        admitKernel<1><<<1, 256, 0, c.stream>>>(p, i);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
  }
  advanceKernel<<<1, 1, 0, c.stream>>>(p.graphState, k);
  return cudaGetLastError();
}

cudaError_t launchStimulus(int spw, const KParams &p, uint32_t cycle, cudaStream_t st) {
  const uint32_t n = std::max<uint32_t>(1, p.nStim * p.gpad);
  const uint32_t blocks = std::min<uint32_t>(1024, (n + 255) / 256);
  if (spw == 8)
    stimulusKernel<8><<<blocks, 256, 0, st>>>(p, cycle);
  else
    stimulusKernel<1><<<blocks, 256, 0, st>>>(p, cycle);
  return cudaGetLastError();
}

cudaError_t launchInitState(int spw, const KParams &p, cudaStream_t st) {
  const size_t n = size_t(p.regSlots) * p.gpad;
  const uint32_t blocks = uint32_t(std::min<size_t>(4096, (n + 255) / 256 + 1));
  if (spw == 8)
    initStateKernel<8><<<blocks, 256, 0, st>>>(p);
  else
    initStateKernel<1><<<blocks, 256, 0, st>>>(p);
  return cudaGetLastError();
}

cudaError_t launchInitMems(const KParams &p, cudaStream_t st) {
  const uint32_t vecs = uint32_t((size_t(p.memPoolSize) + 15) / 16);
  if (!vecs) return cudaSuccess;
  const uint32_t gy = (p.nStreams + kInitStreams - 1) / kInitStreams;
  dim3 grid(std::min<uint32_t>((vecs + 255) / 256, std::max<uint32_t>(1, 4864u / gy)), gy);
  initMemsKernel<<<grid, 256, 0, st>>>(p.initMems, p.mems, p.memStride, vecs, p.nStreams);
  return cudaGetLastError();
}

cudaError_t launchRegDigest(int spw, const uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t nStreams,
                            unsigned long long *out, cudaStream_t st) {
  dim3 grid(std::max<uint32_t>(1, std::min<uint32_t>(64, (slots + 255) / 256)), gpad);
  if (spw == 8)
    regDigestKernel<8><<<grid, 256, 0, st>>>(regs, slots, gpad, nStreams, out);
  else
    regDigestKernel<1><<<grid, 256, 0, st>>>(regs, slots, gpad, nStreams, out);
  return cudaGetLastError();
}

cudaError_t launchRegDigestOne(const uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t g, uint32_t k,
                               unsigned long long *out, cudaStream_t st) {
  if (!slots) return cudaSuccess;
  regDigestOneKernel<<<std::min<uint32_t>(152, (slots + 255) / 256), 256, 0, st>>>(regs, slots, gpad, g, k, out);
  return cudaGetLastError();
}

cudaError_t launchMemDigest(const uint8_t *mems, unsigned long long stride, uint32_t size, uint32_t nStreams,
                            const uint8_t *image, unsigned long long *out, cudaStream_t st) {
  if (size == 0 || nStreams == 0) return cudaSuccess;
  // Small pools by bytes: a block that takes 64 pools one after another is
  // slower than a thread per byte while those leave the GPU room.  us, by 16
  // bytes / by bytes, 1 % of the bytes different: 1 pool of 8 KiB 4.3 / 3.6, 64
  // KiB 6.3 / 4.2, 128 KiB 6.2 / 6.3; 64 pools of 8 KiB 37 / 8, 32 KiB 45 / 35,
  // 64 KiB 45 / 76; 1,000 pools of 4 KiB 41 / 25, 8 KiB 47 / 51 (equal pools 10
  // by 16 bytes at any of these sizes; wholly different ones 70 up to 32 KiB,
  // 129 for 64 pools of 64 KiB).
  const unsigned long long total = (unsigned long long)size * nStreams;
  const bool small = total <= (128u << 10) || (size <= (32u << 10) && total <= (4u << 20));
  if (small || ((reinterpret_cast<uintptr_t>(mems) | (nStreams > 1 ? stride : 0ull)) & 15u) != 0u) {
    dim3 grid(std::max<uint32_t>(1, std::min<uint32_t>(1024, (size + 255) / 256)), nStreams);
    memDigestBytesKernel<<<grid, 256, 0, st>>>(mems, stride, size, nStreams, out);
    return cudaGetLastError();
  }
  // about 8 blocks an SM in all
  const uint32_t gy = (nStreams + kDigestStreams - 1) / kDigestStreams;
  const uint32_t full = (size / 16u + kDigestThreads - 1) / kDigestThreads;
  dim3 grid(std::max<uint32_t>(1, std::min<uint32_t>(full, std::max<uint32_t>(1, 1216u / gy))), gy);
  memDigestKernel<<<grid, kDigestThreads, 0, st>>>(mems, stride, size, nStreams, nStreams >= 8u ? image : nullptr, out);
  return cudaGetLastError();
}

cudaError_t launchGatherRegs(const uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t g, uint32_t k, uint8_t *out,
                             cudaStream_t st) {
  gatherRegsKernel<<<std::max<uint32_t>(1, std::min<uint32_t>(1024, (slots + 255) / 256)), 256, 0, st>>>(regs, slots, gpad, g, k, out);
  return cudaGetLastError();
}

cudaError_t launchScatterRegs(uint32_t *regs, uint32_t slots, uint32_t gpad, uint32_t g, uint32_t k, const uint8_t *in,
                              cudaStream_t st) {
  scatterRegsKernel<<<std::max<uint32_t>(1, std::min<uint32_t>(1024, (slots + 255) / 256)), 256, 0, st>>>(regs, slots, gpad, g, k, in);
  return cudaGetLastError();
}

cudaError_t launchPeekRegs(const uint32_t *regs, uint32_t gpad, uint32_t g, uint32_t k, const uint32_t *ids,
                           uint8_t *out, uint32_t n, cudaStream_t st) {
  if (!n) return cudaSuccess;
  peekRegsKernel<<<std::max<uint32_t>(1, std::min<uint32_t>(1024, (n + 255) / 256)), 256, 0, st>>>(regs, gpad, g, k, ids, out, n);
  return cudaGetLastError();
}

cudaError_t launchPokeRegs(uint32_t *regs, uint32_t gpad, uint32_t g, uint32_t k, const RegPoke &q, cudaStream_t st) {
  if (!q.n) return cudaSuccess;
  pokeRegsKernel<<<1, 32, 0, st>>>(regs, gpad, g, k, q);
  return cudaGetLastError();
}

}  // namespace tgs
