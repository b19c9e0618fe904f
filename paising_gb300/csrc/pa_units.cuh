// pa_units.cuh -- work units of the persistent gather and sweep kernels, and
// the batch's work plan: how many units each population has and their prefix
// sums, from which the kernels find a unit's population.
#pragma once

#include "pa_device.cuh"

namespace pa {

// ---------------------------------------------------------------- gathers
// SSC: up to kSscUnitVecs 16-byte vectors of one population's new buffer --
// whole replicas (floor(kSscUnitVecs / nv) of them) when a replica has at
// most kSscUnitVecs vectors, else one kSscUnitVecs part of a replica.
constexpr int kSscResThreads = 256;
constexpr int kSscVecsPerThread = 8;
constexpr int kSscUnitVecs = kSscResThreads * kSscVecsPerThread;  // 32 KB

__host__ __device__ __forceinline__ long long ssc_units(int nv, int Rn) {
  if (nv > kSscUnitVecs) return (long long)Rn * ((nv + kSscUnitVecs - 1) / kSscUnitVecs);
  const int rpu = kSscUnitVecs / nv;
  return (Rn + rpu - 1) / rpu;
}

// MSC, reference stream: 32 new groups x a strip of 32 sites, or of 8 when a
// population would otherwise have too few units to occupy the GPU (small
// lattices).
constexpr int kSub = 8;  // sites gathered per pass over the 32 source bits
__device__ __forceinline__ int res_strip(int N, int rgn) {
  const int tiles = (rgn + 31) / 32;
  return (long long)tiles * (N / 32) >= 8192 ? 32 : kSub;
}

// MSC, native stream: a few new groups x kNatSites sites (four per lane of a
// warp): 16 groups, which spread a unit's set-up and first rows thinnest, or 4
// where 16 would leave the 3648 persistent warps (152 SMs) with few units each
// (L = 64, 20000 replicas: 18.3 -> 11.0 us).
constexpr int kNatSites = 128;
__host__ __device__ __forceinline__ int nat_groups(int N, int rgn) {
  const long long strips = (N + kNatSites - 1) / kNatSites;
  return (rgn + 15) / 16 * strips >= 8192 ? 16 : 4;
}
__host__ __device__ __forceinline__ int nat_units(int N, int rgn) {
  const int g = nat_groups(N, rgn);
  return ((rgn + g - 1) / g) * ((N + kNatSites - 1) / kNatSites);
}

// ------------------------------------------------------------- work plan
// One CTA of 1024 threads (kMaxPop populations at most): units of the next
// sweep launch (energy_only: of the populations at step 0) and of the gather
// before it, their exclusive prefix sums, and fresh queues.  scratch: 33
// words of shared memory.  The populations' states are read past the L1: in a
// launch that also wrote them, another block of this SM may have read them
// before.
__device__ __forceinline__ void plan_batch(BatchDev* b, int energy_only, uint32_t* scratch) {
  const int p = threadIdx.x, np = b->npop;
  uint32_t units = 0, res = 0, groups = 0;
  if (p < np) {
    const PopDev* st = b->pops + p;
    const int step = __ldcg(&st->step), error = __ldcg(&st->error), R = __ldcg(&st->R_cur);
    const int nsteps = __ldcg(&st->nsteps), tile = st->gpt, coding = st->coding, N = st->N, mode = st->rng_mode;
    const bool stepping = step >= 1 && step <= nsteps && !error;
    const int rg = (R + kMsb - 1) / kMsb, gpt = tile > 0 ? tile : 1;
    if (energy_only ? step == 0 : stepping) units = (uint32_t)(((coding == kMSC ? rg : R) + gpt - 1) / gpt);
    if (stepping) {
      if (coding == kSSC) {
        res = (uint32_t)ssc_units(N >> 4, R);
      } else {
        const int S = res_strip(N, rg);
        groups = (uint32_t)rg;
        res = mode == kNative ? (uint32_t)nat_units(N, rg) : (uint32_t)(((rg + 31) / 32) * ((N + S - 1) / S));
      }
    }
  }
  for (int i = p; i < kMaxSm; i += blockDim.x) b->sm_taken[i] = 0;
  uint32_t total, rtotal, gtotal, ex, rex, gex;
  if (np <= 32) {  // one warp
    if (p >= 32) return;
    uint32_t a = units, r = res, g = groups;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t ta = __shfl_up_sync(0xffffffffu, a, o), tr = __shfl_up_sync(0xffffffffu, r, o),
                     tg = __shfl_up_sync(0xffffffffu, g, o);
      if (p >= o) {
        a += ta;
        r += tr;
        g += tg;
      }
    }
    total = __shfl_sync(0xffffffffu, a, 31);
    rtotal = __shfl_sync(0xffffffffu, r, 31);
    gtotal = __shfl_sync(0xffffffffu, g, 31);
    ex = a - units;
    rex = r - res;
    gex = g - groups;
  } else {
    ex = block_exscan(units, scratch, &total);
    __syncthreads();  // scratch is reused
    rex = block_exscan(res, scratch, &rtotal);
    __syncthreads();
    gex = block_exscan(groups, scratch, &gtotal);
  }
  if (p < np) {
    b->unit_prefix[p] = (int)ex;
    b->res_prefix[p] = (int)rex;
    b->grp_prefix[p] = (int)gex;
  }
  if (p == 0) {
    b->unit_prefix[np] = (int)total;
    b->res_prefix[np] = (int)rtotal;
    b->grp_prefix[np] = (int)gtotal;
    b->work_next = 0;
    b->res_next = 0;
  }
}

}  // namespace pa
