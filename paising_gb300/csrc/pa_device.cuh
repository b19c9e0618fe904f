// pa_device.cuh -- device-side building blocks shared by the kernels:
// Philox4x32-10, the reference-coordinate ("injected") stream, warp/block
// reductions and exact 128-bit accumulation helpers.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pa_kernels.h"
#include "pa_state.h"

namespace pa {

// ----------------------------------------------------------------- Philox
// Philox4x32-10 counter-based generator (Salmon, Moraes, Dror, Shaw,
// "Parallel random numbers: as easy as 1, 2, 3", SC'11), written from the
// paper: two 32x32->64 multiplies per round, Weyl-sequence key schedule.
constexpr uint32_t kPhiloxM0 = 0xD2511F53u;
constexpr uint32_t kPhiloxM1 = 0xCD9E8D57u;
constexpr uint32_t kPhiloxW0 = 0x9E3779B9u;
constexpr uint32_t kPhiloxW1 = 0xBB67AE85u;

struct U4 {
  uint32_t x, y, z, w;
};

__host__ __device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

__host__ __device__ __forceinline__ U4 philox10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                                 uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = mulhi32(kPhiloxM0, c0), lo0 = kPhiloxM0 * c0;
    const uint32_t hi1 = mulhi32(kPhiloxM1, c2), lo1 = kPhiloxM1 * c2;
    c0 = hi1 ^ c1 ^ k0;
    c1 = lo1;
    c2 = hi0 ^ c3 ^ k1;
    c3 = lo0;
    k0 += kPhiloxW0;
    k1 += kPhiloxW1;
  }
  return U4{c0, c1, c2, c3};
}

// Philox4x32-10 with the key schedule k + r*W precomputed (k[2r], k[2r+1] =
// round-r key); same output as philox10.  The SSC bit-plane sweep takes it as
// a __grid_constant__ kernel parameter computed on the host (0.5% faster than
// forming it in the kernel); the MSC sweeps form it from the seed (0.6%
// faster that way).
struct PhiloxKeys {
  uint32_t k[20];
  __host__ __device__ __forceinline__ explicit PhiloxKeys(unsigned long long seed) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      k[2 * r] = (uint32_t)seed + (uint32_t)r * kPhiloxW0;
      k[2 * r + 1] = (uint32_t)(seed >> 32) + (uint32_t)r * kPhiloxW1;
    }
  }
};

__device__ __forceinline__ U4 philox10k(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const PhiloxKeys& K) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned long long p0 = (unsigned long long)kPhiloxM0 * c0;
    const unsigned long long p1 = (unsigned long long)kPhiloxM1 * c2;
    const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
    const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
    c0 = hi1 ^ c1 ^ K.k[2 * r];
    c1 = lo1;
    c2 = hi0 ^ c3 ^ K.k[2 * r + 1];
    c3 = lo0;
  }
  return U4{c0, c1, c2, c3};
}

// The same generator with each round's two products written as PTX
// mul.wide.u32.  Same output; which form the compiler schedules better
// depends on the kernel around it (measured, 8 populations at L=64: the SSC
// bit-plane sweep 1.7% faster this way, the MSC sweep 1.2% slower), so a
// kernel chooses by the type of its keys.
struct PhiloxKeysWide : PhiloxKeys {
  __host__ __device__ __forceinline__ explicit PhiloxKeysWide(unsigned long long seed) : PhiloxKeys(seed) {}
};

__device__ __forceinline__ unsigned long long mul_wide_u32(uint32_t a, uint32_t b) {
  unsigned long long p;
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(p) : "r"(a), "r"(b));
  return p;
}

__device__ __forceinline__ U4 philox10k(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const PhiloxKeysWide& K) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned long long p0 = mul_wide_u32(c0, kPhiloxM0);
    const unsigned long long p1 = mul_wide_u32(c2, kPhiloxM1);
    const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
    const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
    c0 = hi1 ^ c1 ^ K.k[2 * r];
    c1 = lo1;
    c2 = hi0 ^ c3 ^ K.k[2 * r + 1];
    c3 = lo0;
  }
  return U4{c0, c1, c2, c3};
}

// Both code forms of one round's product, chosen by the key type.
__device__ __forceinline__ unsigned long long philox_mul(uint32_t m, uint32_t c, const PhiloxKeys&) {
  return (unsigned long long)m * c;
}
__device__ __forceinline__ unsigned long long philox_mul(uint32_t m, uint32_t c, const PhiloxKeysWide&) {
  return mul_wide_u32(c, m);
}

// The sweeps' counters are (c0, c1, step, tag) with step and tag fixed for a
// temperature and c1 for a half-sweep.  The first two rounds then split into
// a part of c0, step and tag alone -- the prefix, two words that hold for
// every sweep of the temperature --
//   (hi(M1 c2) ^ lo(M1 step) ^ k2, lo(M1 c2) ^ k4),  c2 = hi(M0 c0) ^ tag ^ k1,
// and a part of c1 and step alone -- the uniform, two words per half-sweep --
//   (hi(M0 u) ^ k3, lo(M0 u) ^ k5),  u = hi(M1 step) ^ c1 ^ k0;
// philox10_prefixed runs the remaining eight rounds from them (and lo(M0 c0)),
// the output of philox10k(c0, c1, step, tag).
template <class Keys>
__device__ __forceinline__ uint2 philox_prefix(uint32_t c0, uint32_t step, uint32_t tag, const Keys& K) {
  const uint32_t c2 = (uint32_t)(philox_mul(kPhiloxM0, c0, K) >> 32) ^ tag ^ K.k[1];
  const unsigned long long p = philox_mul(kPhiloxM1, c2, K);
  return make_uint2((uint32_t)(p >> 32) ^ (kPhiloxM1 * step) ^ K.k[2], (uint32_t)p ^ K.k[4]);
}

template <class Keys>
__device__ __forceinline__ uint2 philox_uniform(uint32_t c1, uint32_t step, const Keys& K) {
  const unsigned long long p = philox_mul(kPhiloxM0, mulhi32(kPhiloxM1, step) ^ c1 ^ K.k[0], K);
  return make_uint2((uint32_t)(p >> 32) ^ K.k[3], (uint32_t)p ^ K.k[5]);
}

// The prefix with its products: lo(M0 c0), the second word, and the 64-bit
// product of round 3 that the first word alone decides.  Twice the size for
// one product and one multiply less per block.
template <class Keys>
__device__ __forceinline__ uint4 philox_prefix4(uint32_t c0, uint32_t step, uint32_t tag, const Keys& K) {
  const uint2 e = philox_prefix(c0, step, tag, K);
  const unsigned long long p = philox_mul(kPhiloxM0, e.x, K);
  return make_uint4(kPhiloxM0 * c0, e.y, (uint32_t)(p >> 32), (uint32_t)p);
}

template <class Keys>
__device__ __forceinline__ U4 philox10_prefixed(uint32_t, uint4 pre, uint2 uni, const Keys& K) {
  unsigned long long p0, p1 = philox_mul(kPhiloxM1, uni.x ^ pre.x, K);
  uint32_t x = (uint32_t)(p1 >> 32) ^ pre.y, y = (uint32_t)p1, z = pre.z ^ uni.y, w = pre.w;
#pragma unroll
  for (int r = 3; r < 10; ++r) {
    p0 = philox_mul(kPhiloxM0, x, K);
    p1 = philox_mul(kPhiloxM1, z, K);
    x = (uint32_t)(p1 >> 32) ^ y ^ K.k[2 * r];
    y = (uint32_t)p1;
    z = (uint32_t)(p0 >> 32) ^ w ^ K.k[2 * r + 1];
    w = (uint32_t)p0;
  }
  return U4{x, y, z, w};
}

template <class Keys>
__device__ __forceinline__ U4 philox10_prefixed(uint32_t c0, uint2 pre, uint2 uni, const Keys& K) {
  const unsigned long long p = philox_mul(kPhiloxM0, pre.x, K);
  return philox10_prefixed(c0, make_uint4(kPhiloxM0 * c0, pre.y, (uint32_t)(p >> 32), (uint32_t)p), uni, K);
}

// The reference draws every random number from a per-thread cuRAND stream
// initialised as curand_init(seed, subsequence, 0) and consumed in order
// (PAisingSSC.cu:152,164,241; PAisingMSC.cu:171,195,355).  "Reference
// coordinates" mode evaluates, for draw number ctr of subsequence subseq,
//   H = word (ctr & 3) of Philox4x32-10(key = seed, counter = (ctr >> 2, subseq))
// so that a kernel with any thread layout can reproduce the draw a reference
// thread would have made.  A uniform double is (H + 1) * 2^-32.
__host__ __device__ __forceinline__ uint32_t ref_word(uint64_t seed, uint64_t subseq, uint64_t ctr) {
  const uint64_t blk = ctr >> 2;
  const U4 o = philox10((uint32_t)blk, (uint32_t)(blk >> 32), (uint32_t)subseq, (uint32_t)(subseq >> 32),
                        (uint32_t)seed, (uint32_t)(seed >> 32));
  const uint32_t j = (uint32_t)ctr & 3u;
  return j == 0 ? o.x : j == 1 ? o.y : j == 2 ? o.z : o.w;
}

__host__ __device__ __forceinline__ double ref_uniform(uint32_t h) {
  return ((double)h + 1.0) * (1.0 / 4294967296.0);
}

// Domain tags for the native sweep streams (counter word 3, top byte).
constexpr uint32_t kTagSscSweep = 0x53u << 24;
constexpr uint32_t kTagMscSweep = 0x4Du << 24;

// Counter word 2 of the native sweep streams: the temperature index (below
// 2^14, since schedules end at nBmax = 10000) and, above it, the population's
// run number, so that repeated runs of a handle draw fresh sweep randomness
// (runs 2^18 apart share it).
__device__ __forceinline__ uint32_t native_step_word(const PopDev* st) {
  return (uint32_t)st->step | ((uint32_t)st->run << 14);
}

// -------------------------------------------------------------- reductions
template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <class T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    T w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w < v ? w : v;
  }
  return v;
}

// Block-wide sum; every thread must call it; result valid in all threads.
// scratch: >= 32 elements of shared memory.
template <class T>
__device__ __forceinline__ T block_sum(T v, T* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  v = (lane < nw) ? scratch[lane] : T(0);
  v = warp_sum(v);
  return v;
}

// Block-wide exclusive scan of one uint32 per thread (blockDim multiple of 32,
// <= 1024).  Returns the exclusive prefix; *total receives the block total.
__device__ __forceinline__ uint32_t block_exscan(uint32_t v, uint32_t* scratch, uint32_t* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();
  if (lane == 31) scratch[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = lane < nw ? scratch[lane] : 0u, wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < nw) scratch[lane] = wi - w;
    if (lane == nw - 1) scratch[32] = wi;
  }
  __syncthreads();
  uint32_t ex = scratch[wid] + inc - v;
  *total = scratch[32];
  return ex;
}

// ------------------------------------------------ exact 128-bit accumulation
// Sums of M^4 exceed 64 bits (|M| <= N, N up to 65536).  They are kept as
// (lo, hi) pairs of uint64 and added with carry, so the total does not depend
// on the order in which replicas are accumulated.
struct U128 {
  unsigned long long lo, hi;
};

__device__ __forceinline__ void u128_add(U128& a, unsigned long long lo, unsigned long long hi) {
  const unsigned long long s = a.lo + lo;
  a.hi += hi + (s < a.lo ? 1ull : 0ull);
  a.lo = s;
}

__device__ __forceinline__ void u128_atomic_add(unsigned long long* lo_p, unsigned long long* hi_p,
                                                unsigned long long lo, unsigned long long hi) {
  const unsigned long long old = atomicAdd(lo_p, lo);
  const unsigned long long carry = (old + lo < old) ? 1ull : 0ull;
  if (hi + carry) atomicAdd(hi_p, hi + carry);
}

// m^4 for |m| <= 65536 as (lo, hi)
__device__ __forceinline__ void m4_of(int m, unsigned long long& lo, unsigned long long& hi) {
  const unsigned long long m2 = (unsigned long long)((long long)m * (long long)m);
  lo = m2 * m2;
  hi = __umul64hi(m2, m2);
}

__host__ __device__ __forceinline__ double u128_to_double(unsigned long long lo, unsigned long long hi) {
  return (double)hi * 18446744073709551616.0 + (double)lo;
}

// --------------------------------------------------------- batch work queue
// Population p and its local unit for queue entry u: prefix[p] <= u < prefix[p+1].
__device__ __forceinline__ int queue_pop(const BatchDev* b, int u, int* local) {
  int lo = 0, hi = b->npop;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (b->unit_prefix[mid] <= u) lo = mid;
    else hi = mid;
  }
  *local = u - b->unit_prefix[lo];
  return lo;
}

// First unit of a persistent CTA: its own index, and later_unit from then on.
// Blocks of low index lie on different SMs, so a launch with fewer units than
// CTAs spreads over the GPU; by the queue's counter alone the CTAs that reached
// it first took the units, about two per busy SM with half of the SMs idle
// (MSC L = 32 R = 5000, 157 units on 608 CTAs, 100 sweeps: 32.1 ms -> 20.7
// per anneal of 49 temperatures).
//
// Blocks are handed out round the GPCs, which have different numbers of SMs:
// of the first 152 blocks some SMs get two from block 112 on, three from 240
// on, four from 376 on, while others still wait for their first, second or
// third, and the fullest SM sets the time.  There a CTA's first unit is its
// place instead -- its rank among the CTAs of its SM, times the number of SMs,
// plus its SM: 0.9 us for the rank's atomic, and per half-sweep (L = 32, one
// group per unit) 1.28 us -> 0.86 at 120..152 units, 1.83 -> 1.27 at 248..304,
// 2.37 -> 1.83 at 384..456; L = 96 8.75 -> 5.47 and 12.75 -> 8.76.  At other
// counts both orders fill the SMs alike, which is why only launches of no more
// units than CTAs whose last round of the SMs is more than half full take it
// (and, in the engine, units of four warps or more: smaller ones don't fill an
// SM by fours either; the SSC bit-plane sweep, whose small populations have
// such units, goes by index).
// (Clusters are spread evenly as they are: steps at 76, 152, 228 of 2 CTAs.)
//
// nsm: SMs, gridDim.x = nsm * CTAs per SM; 0: always by index.  Every place is
// taken once: the launch has as many CTAs as places, and one that finds its
// SM's places taken (another launch delayed CTAs) takes a free one elsewhere,
// of which there is one for each CTA without: places never become free again,
// so one pass over the SMs finds it.
// Not inlined: the sweep kernels' hot loops, at the register limit, lost 1-2%
// at some sizes to the changed allocation.
static __device__ __noinline__ int first_unit(BatchDev* b, int nsm, int total) {
  if (nsm <= 0 || total > (int)gridDim.x || (total + nsm - 1) % nsm < nsm / 2) return blockIdx.x;
  const unsigned per = gridDim.x / (unsigned)nsm;
  unsigned sm, rank = per;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
  if (sm < (unsigned)nsm) rank = atomicAdd(&b->sm_taken[sm], 1u);
  for (int i = 0; rank >= per && i < nsm; ++i) {
    sm = (unsigned)i;
    if (__ldcg(&b->sm_taken[i]) < per) rank = atomicAdd(&b->sm_taken[i], 1u);
  }
  return (int)(rank * nsm + (rank & 1u ? nsm - 1 - sm : sm));  // there and back: queues begin with the longest units
}
// Unit after a CTA's (or cluster's) first, of a launch of n of them.
__device__ __forceinline__ int later_unit(BatchDev* b, int n) { return n + (int)atomicAdd(&b->work_next, 1u); }

// Allows launches of fn with `smem` bytes of dynamic shared memory.  The
// function's limit is one for all threads and handles, so it is always set to
// the device's and never to what one launch needs: a launch of another thread,
// or of a handle set up earlier, may need more.
inline cudaError_t allow_smem(const void* fn, int smem) {
  int dev, optin;
  cudaFuncAttributes a;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, fn);
  if (e != cudaSuccess) return e;
  if (smem > optin - (int)a.sharedSizeBytes) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)a.sharedSizeBytes);
}

// Persistent grid: as many CTAs of `block` threads as can be resident.
inline cudaError_t persistent_launch(const void* fn, int block, int smem, SweepLaunch* out) {
  cudaError_t e = allow_smem(fn, smem);
  if (e != cudaSuccess) return e;
  int dev, nsm, per = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, block, smem)) != cudaSuccess) return e;
  out->grid = nsm * (per > 0 ? per : 1);
  out->nsm = nsm <= kMaxSm ? nsm : 0;
  out->block = block;
  out->smem = smem;
  return cudaSuccess;
}

}  // namespace pa
