// pa_resample.cu -- resampling of the populations on the device, no host
// round trip, the per-temperature bookkeeping, and the batch launchers.
//
// Replaces, from the reference (both codings):
//   QKer        (PAisingSSC.cu:217-234, PAisingMSC.cu:319-345) + host lnQ
//               (PAisingSSC.cu:533)                  -> q_kernel
//   CalcTauKer  (PAisingSSC.cu:236-254, PAisingMSC.cu:347-360)
//   + CalcParSum block totals                        -> copy_numbers_kernel
//   CalcParSum  (PAisingSSC.cu:256-270, PAisingMSC.cu:362-395)
//                                                    -> scatter_kernel (exclusive
//               scan + map new replica -> old replica, consumed by the gathers)
//   the three in one launch where a CTA or a cluster holds the population
//                                                    -> resample_fused_kernel
//   CalcAverages + host observables (PAisingSSC.cu:282-292, 614-630)
//                                                    -> finish_step_kernel, or
//               resample_fused_kernel and finish_rows_kernel (sums are
//               accumulated exactly in integers by the sweep kernels)
//
// Population p of a batch is handled by the blocks with blockIdx.y == p.
// Every multi-block reduction ends with the last-block pattern: each block
// publishes its partial result, takes a ticket, and the block that draws the
// last ticket combines the partials in block order.  Results therefore do not
// depend on block scheduling, and no block ever waits for another.
#include <cooperative_groups.h>

#include <cfloat>
#include <climits>
#include <cmath>

#include "pa_device.cuh"
#include "pa_kernels.h"
#include "pa_thresholds.h"
#include "pa_units.cuh"

namespace pa {

namespace {

constexpr int kResThreads = 256;

__device__ __forceinline__ int pop_units(const PopDev* st, int R) {
  return st->coding == kMSC ? ((R + kMsb - 1) / kMsb) * kMsb : R;
}

// Neumaier's variant of Kahan compensated summation, FP32.
struct Comp32 {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float t = __fadd_rn(s, x);
    if (fabsf(s) >= fabsf(x))
      c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, t), x));
    else
      c = __fadd_rn(c, __fadd_rn(__fsub_rn(x, t), s));
    s = t;
  }
};

// the chain s.add(w[0]), s.add(w[1]), ... over n values >= 0 of shared
// memory: the same sums, the operands of the compensation ordered by max and
// min and the values loaded ahead, since one warp's lanes (or one thread) run
// it alone
__device__ __forceinline__ void comp_chain(Comp32& a, const float* w, int n) {
  float s = a.s, c = a.c;
  auto add = [&](float x) {
    const float t = __fadd_rn(s, x);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(fmaxf(s, x), t), fminf(s, x)));
    s = t;
  };
  int i = 0;
  for (; i + 16 <= n; i += 16) {
    float x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = w[i + j];
#pragma unroll
    for (int j = 0; j < 16; ++j) add(x[j]);
  }
  for (; i < n; ++i) add(w[i]);
  a.s = s;
  a.c = c;
}

// resampling weight of one replica in FP32: exp(-dbeta (E - Emin)) <= 1
__device__ __forceinline__ float weight32(float dBf, int E, int Emin) {
  return expf(-dBf * (float)(E - Emin));
}

// lnQ from the weight sum q relative to E_ref (PAisingSSC.cu:533)
__device__ __forceinline__ double lnq_of(double dB, double Eref, double q, double logR) {
  return -dB * Eref + log(q) - logR;
}

// copy number of one replica, mu rounded by its own uniform draw (word h)
// FP32: U = (h + 1) 2^-32 < f, the fraction of mu, as integers: f 2^32 is exact
// in FP32 and below 2^32, so h + 1 < f 2^32 iff h + 1 < g = ceil(f 2^32).  (The
// same test in FP64 took 9100 cycles of a block of 1024 at one slot each: the
// FP64 units do a warp instruction in tens of cycles.)
__device__ __forceinline__ uint32_t copies_fp32(float mu, uint32_t h) {
  const float fl = floorf(mu);
  const uint32_t g = __float2uint_ru((mu - fl) * 4294967296.0f);  // 0 for a fraction of 0 or NaN
  return (uint32_t)fl + (g != 0u && h < g - 1u ? 1u : 0u);
}
__device__ __forceinline__ uint32_t copies_fp64(double mu, uint32_t h) {
  const double fl = floor(mu);
  return (uint32_t)(ref_uniform(h) < (mu - fl) ? fl + 1 : fl);
}

// copies_fp64 as integers: x + (h < y ? 1 : 0).  U = (h + 1) 2^-32 < f iff
// h + 1 < ceil(f 2^32), f 2^32 being exact; a fraction of 0 or NaN and whole
// parts beyond 32 bits (which saturate) never get one more.
__device__ __forceinline__ uint2 copies_of(double mu) {
  const double fl = floor(mu), f = mu - fl;
  const uint32_t whole = (uint32_t)fl;
  const unsigned long long g = f > 0.0 && fl < 4294967295.0 ? (unsigned long long)ceil(f * 4294967296.0) : 0ull;
  return make_uint2(whole, g != 0ull ? (uint32_t)(g - 1ull) : 0u);
}

// last-block ticket: returns true in every thread of the block that finished
// last among the gridDim.x blocks of its population
__device__ __forceinline__ bool last_block(unsigned int* ticket) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  return s_last;
}

// contiguous chunk of [0, n) owned by this block, a whole number of tiles
__device__ __forceinline__ void block_chunk(int n, int& lo, int& hi) {
  const int per = (n + gridDim.x - 1) / gridDim.x;
  const int c = (per + blockDim.x - 1) / blockDim.x * blockDim.x;
  lo = min(n, (int)blockIdx.x * c);
  hi = min(n, lo + c);
}

}  // namespace

// -------------------------------------------------- FP64 weights by level
// The FP64 units take a warp's exponential in about 560 cycles, and q and the
// copy numbers want one each per replica, of which there are at most N + 1
// different ones (energies are -2N + 4k).  Populations well above the number of
// levels (resample_by_level) look them up: level k's weight for q, then -- once lnQ is known -- its
// mean copy number as the whole part and the draws below which it is one more.
// The same expressions, so the same values as replica by replica.  One launch
// before each pass costs about 3 us, an exponential of all replicas 1 us per
// 17000: L = 32, 10^6 replicas, q 53 -> 16 us and copy numbers 65 -> 19; L = 16,
// 100000 replicas, 5 sweeps 1.02x per anneal, 60000 would lose 3%.
constexpr int kTableUnits = 98304;  // replicas more than levels from which the tables pay
__device__ __forceinline__ int level_of(int E, int N) { return (E + 2 * N) >> 2; }

__global__ void __launch_bounds__(kResThreads) weight_table_kernel(PopDev* pops, int copies) {
  PopDev* st = pops + blockIdx.y;
  const int N = st->N, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (!st->wtab || k > N || !pop_stepping(st)) return;
  const int step = st->step, Rp = st->R_prev;
  const double dB = st->betas[step] - st->betas[step - 1];
  const int E = 4 * k - 2 * N;
  if (!copies) {
    const double Em = st->Emean;
    st->wtab[k] = exp(-dB * (E - Em));
  } else {
    const double lnQ = st->lnQ;
    reinterpret_cast<uint2*>(st->wtab)[k] = copies_of(((double)st->Rinit) / Rp * exp(-dB * (double)E - lnQ));
  }
}

// ------------------------------------------------------------------------ Q
// q = sum_j w_j over the population before resampling, then
//   lnQ = -dbeta E_ref + ln q - ln R_prev            (PAisingSSC.cu:533)
// FP64 weights: w = exp(-dbeta (E - Emean)), E_ref = Emean (the reference's
// choice, PAisingSSC.cu:222).  FP32 weights: w = exp(-dbeta (E - Emin)) <= 1,
// compensated sums, E_ref = Emin; lnQ itself is formed in FP64.
__global__ void __launch_bounds__(kResThreads) q_kernel(PopDev* pops) {
  __shared__ double s_d[33];
  __shared__ float s_f[2][kResThreads];
  PopDev* st = pops + blockIdx.y;
  if (!pop_stepping(st)) return;
  const int step = st->step, Rp = st->R_prev, n = pop_units(st, Rp);
  const double dB = st->betas[step] - st->betas[step - 1];
  const uint8_t* act = st->coding == kMSC ? st->active[st->parity] : nullptr;
  const int32_t* E = st->E;
  const int tid = threadIdx.x;
  if (st->weights == kFP64) {
    const double Em = st->Emean;
    const double* w = st->wtab;
    const int N = st->N;
    double v = 0.0;
    if (w) {
      for (int j = blockIdx.x * blockDim.x + tid; j < n; j += gridDim.x * blockDim.x)
        if (!act || act[j]) v += w[level_of(E[j], N)];
    } else {
      for (int j = blockIdx.x * blockDim.x + tid; j < n; j += gridDim.x * blockDim.x)
        if (!act || act[j]) v += exp(-dB * (E[j] - Em));
    }
    v = block_sum(v, s_d);
    if (tid == 0) st->qpart_d[blockIdx.x] = v;
    if (last_block(&st->ticket)) {
      double a = 0.0;
      for (int bb = tid; bb < (int)gridDim.x; bb += blockDim.x) a += ((volatile double*)st->qpart_d)[bb];
      a = block_sum(a, s_d);
      if (tid == 0) {
        st->q = a;
        st->lnQ = lnq_of(dB, Em, a, log((double)Rp));
        st->ticket = 0;
      }
    }
  } else {
    const int Emin = st->Emin;
    const float dBf = (float)dB;
    Comp32 acc;
    for (int j = blockIdx.x * blockDim.x + tid; j < n; j += gridDim.x * blockDim.x)
      if (!act || act[j]) acc.add(weight32(dBf, E[j], Emin));
    s_f[0][tid] = acc.s;
    s_f[1][tid] = acc.c;
    __syncthreads();
    if (tid == 0) {
      Comp32 bsum;
      float c = 0.f;
      for (int i = 0; i < (int)blockDim.x; ++i) { bsum.add(s_f[0][i]); c = __fadd_rn(c, s_f[1][i]); }
      st->qpart_f[2 * blockIdx.x] = bsum.s;
      st->qpart_f[2 * blockIdx.x + 1] = __fadd_rn(bsum.c, c);
    }
    if (last_block(&st->ticket)) {
      // thread t sums the partials of blocks t, t + 256, ... (all loads in
      // flight at once), thread 0 then the 256 thread sums in thread order:
      // a fixed order, so the result does not depend on block scheduling
      Comp32 t;
      float c = 0.f;
      const volatile float* qp = st->qpart_f;
      for (int bb = tid; bb < (int)gridDim.x; bb += blockDim.x) {
        t.add(qp[2 * bb]);
        c = __fadd_rn(c, qp[2 * bb + 1]);
      }
      __syncthreads();  // the block sums above are done with s_f
      s_f[0][tid] = t.s;
      s_f[1][tid] = __fadd_rn(t.c, c);
      __syncthreads();
      if (tid == 0) {
        Comp32 u;
        float cc = 0.f;
        for (int i = 0; i < (int)blockDim.x; ++i) { u.add(s_f[0][i]); cc = __fadd_rn(cc, s_f[1][i]); }
        const float q = __fadd_rn(u.s, __fadd_rn(u.c, cc));
        st->q = (double)q;
        st->lnQ = lnq_of(dB, (double)Emin, (double)q, log((double)Rp));
        st->ticket = 0;
      }
    }
  }
}

// ------------------------------------------------------------ copy numbers
// Nearest-integer resampling (PAisingSSC.cu:242-247):
//   mu_j = R_init / R_prev * exp(-dbeta E_j - lnQ),
//   roff_j = floor(mu_j) + [U_j < mu_j - floor(mu_j)],
// U_j the reference's draw 0 of subsequence iseq + j (j = linear replica
// index; for MSC j = 32 * group + bit, PAisingMSC.cu:355).  Block totals are
// scanned by the last block, which also publishes the new population size
// and flips the double buffer.
__global__ void __launch_bounds__(kResThreads) copy_numbers_kernel(PopDev* pops) {
  __shared__ uint32_t s_u[33];
  __shared__ uint32_t s_run;
  PopDev* st = pops + blockIdx.y;
  if (!pop_stepping(st)) return;
  const int step = st->step, Rp = st->R_prev, n = pop_units(st, Rp), Rinit = st->Rinit;
  const double dB = st->betas[step] - st->betas[step - 1], lnQ = st->lnQ;
  const uint8_t* act = st->coding == kMSC ? st->active[st->parity] : nullptr;
  const int32_t* E = st->E;
  const unsigned long long seed = st->seed, iseq = st->iseq;
  const bool fp64 = st->weights == kFP64;
  const float dBf = (float)dB, qf = (float)st->q, Rf = (float)Rinit;
  const int Emin = st->Emin, N = st->N;
  const uint2* ctab = fp64 ? reinterpret_cast<const uint2*>(st->wtab) : nullptr;
  int lo, hi;
  block_chunk(n, lo, hi);
  uint32_t tot = 0;
  for (int base = lo; base < hi; base += blockDim.x) {
    const int j = base + threadIdx.x;
    uint32_t r = 0;
    if (j < hi && (!act || act[j])) {
      const uint32_t h = ref_word(seed, iseq + (unsigned long long)j, 0);
      if (ctab) {
        const uint2 c = ctab[level_of(E[j], N)];
        r = c.x + (h < c.y ? 1u : 0u);
      } else {
        r = fp64 ? copies_fp64(((double)Rinit) / Rp * exp(-dB * (double)E[j] - lnQ), h)
                 : copies_fp32(Rf * weight32(dBf, E[j], Emin) / qf, h);
      }
    }
    if (j < hi) st->roff[j] = r;
    tot += block_sum(r, s_u);
  }
  if (threadIdx.x == 0) st->blk_tot[blockIdx.x] = tot;
  if (last_block(&st->ticket)) {
    // exclusive scan of the block totals, in block order
    if (threadIdx.x == 0) s_run = 0;
    __syncthreads();
    for (int b0 = 0; b0 < (int)gridDim.x; b0 += blockDim.x) {
      const int bb = b0 + threadIdx.x;
      const uint32_t v = bb < (int)gridDim.x ? ((volatile uint32_t*)st->blk_tot)[bb] : 0u;
      uint32_t total;
      const uint32_t ex = block_exscan(v, s_u, &total);
      if (bb < (int)gridDim.x) st->blk_off[bb] = s_run + ex;
      __syncthreads();
      if (threadIdx.x == 0) s_run += total;
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      const unsigned int Rn = s_run;
      if (Rn == 0u || Rn > (unsigned int)st->Rcap) {
        st->error = Rn == 0u ? 2 : 1;
        st->R_cur = 0;
      } else {
        st->R_cur = (int)Rn;
      }
      st->parity ^= 1;
      st->ticket = 0;
      st->heavy = 0;
    }
  }
}

// ------------------------------------------------------------------ scatter
// offs_j = exclusive prefix of roff; src[offs_j + p] = j for p < roff_j.
// The new replicas of a tile of 256 old ones are filled by the whole block,
// new index i taking the last old replica of the tile whose offset is <= i
// (a binary search over the tile's offsets in shared memory).  An old replica
// with more copies than heavy_copies -- a large dbeta against the energy spread
// makes them, up to all of the population -- would leave its block writing long
// after the others: it is listed, and scatter_heavy spreads its copies over
// many blocks (the work plan's launch, which follows anyway); a tile with one
// is filled thread by thread.  L = 32, 10^6 replicas, dbeta 0.3: 1.2 ms -> 25 us.
__device__ __forceinline__ uint32_t heavy_copies(int Rcap) {
  return (uint32_t)max(1024, Rcap / (kResBlocksMax / 2));  // no more than kResBlocksMax / 2 replicas can have more
}
// Blocks per population: 32, fewer in a batch, whose populations fill the GPU
// side by side.  32 each took 102 us per temperature of 1000 populations just
// to start and find nothing listed; with one each the plan takes 10.
static int heavy_blocks(int npop) { return npop <= 16 ? 32 : npop >= 512 ? 1 : 512 / npop; }
// The copies of a population's listed replicas, by block `block` of `blocks`.
__device__ __forceinline__ void scatter_heavy(const PopDev* st, int block, int blocks) {
  const int n = pop_stepping(st) ? min(st->heavy, kResBlocksMax) : 0;
  for (int k = 0; k < n; ++k) {
    const uint32_t j = st->blk_tot[k], off = st->offs[j], r = st->roff[j];
    for (uint32_t c = block * blockDim.x + threadIdx.x; c < r; c += blocks * blockDim.x) st->src[off + c] = j;
  }
}

__global__ void __launch_bounds__(kResThreads) scatter_kernel(PopDev* pops) {
  __shared__ uint32_t s_u[33];
  __shared__ uint32_t s_off[kResThreads + 1];
  PopDev* st = pops + blockIdx.y;
  if (!pop_stepping(st)) return;
  const int n = pop_units(st, st->R_prev);
  int lo, hi;
  block_chunk(n, lo, hi);
  uint32_t run = st->blk_off[blockIdx.x];
  const uint32_t many = heavy_copies(st->Rcap);
  const int nt = blockDim.x;
  for (int base = lo; base < hi; base += nt) {
    const int j = base + threadIdx.x;
    const uint32_t r = j < hi ? st->roff[j] : 0u;
    uint32_t total;
    const uint32_t off = run + block_exscan(r, s_u, &total);
    if (j < hi) st->offs[j] = off;
    const bool heavy = r > many;
    if (heavy) st->blk_tot[atomicAdd(&st->heavy, 1)] = (uint32_t)j;
    if (__syncthreads_or(heavy)) {  // (its barrier also ends the scan)
      if (!heavy)
        for (uint32_t c = 0; c < r; ++c) st->src[off + c] = (uint32_t)j;
      run += total;
      continue;
    }
    s_off[threadIdx.x] = off;  // non-decreasing; equal to run + total past hi
    if (threadIdx.x == 0) s_off[nt] = run + total;
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < total; t += nt) {
      const uint32_t i = run + t;
      // last k with s_off[k] <= i: s_off[0] = run <= i < s_off[nt]
      int a = 0, b = nt;
      while (b - a > 1) {
        const int m = (a + b) >> 1;
        if (s_off[m] <= i) a = m;
        else b = m;
      }
      st->src[i] = (uint32_t)(base + a);
    }
    __syncthreads();
    run += total;
  }
}

// ------------------------------------------------ Q .. scatter in one launch
// The three passes above and the work plan for populations of at most
// kFusedMaxUnits slots: a thread-block cluster of CS CTAs holds the whole
// population (a tile of 256 slots is what a block of the passes above sums),
// so q, the copy numbers, their scan and the map need two cluster barriers --
// and one split round the weights, before the first remote store -- where the
// passes need three launches, and the last cluster of the batch to
// finish makes the work plan of the gather and the sweep.  Every sum is the
// passes' own: a tile's compensated sum in slot order, the tiles' in tile
// order (FP64: the same trees), so q and all that follows are bit for bit
// theirs.
//
// What bounds it is latency: the compensated sums are serial chains (256
// slots, then the tiles), so a tile's chain is a lane's, all tiles of the CTA
// side by side, while the other warps draw the slots' uniforms.  With FP32
// weights only lnQ is left in FP64, whose logarithms take 3000 cycles each on
// one thread (the FP64 units are few): finish_step takes them (lnq_due),
// unless there is none (b null).
// At R = 1000 the passes and plans took 11.5 + 7.0 + 4.6 + 3.6 + 4.0 us and
// four launches more; one launch takes 17 us timed alone, and the L = 16
// anneal of 199 temperatures 8.0 ms instead of 10.0.
constexpr int kFusedThreads = 1024;
constexpr int kFusedTiles = 32;                                  // tiles per CTA: one chain per lane of a warp
constexpr int kFusedSlots = kFusedTiles * kResThreads / kFusedThreads;  // slots per thread
constexpr int kFusedCluster = 8;
constexpr int kFusedOneUnits = kFusedCluster * kResThreads;       // 2048: one CTA alone up to here
constexpr int kFusedMaxUnits = kFusedCluster * kFusedTiles * kResThreads;  // 65536
constexpr int kFusedPitch = kResThreads + 1;                     // words per tile: the chains' lanes hit 32 banks
constexpr uint32_t kFewCopies = 4;
constexpr int kHeavyMax = kFusedTiles * kFusedPitch / 3;

// sum of the 8 warp sums of a 256-slot tile in block_sum's order
__device__ __forceinline__ double tile_tree(const double* w) {
  return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}

// What a temperature leaves for its row, kept in the row's place until the run's
// end (graph runs without records: nothing reads a row before).  A row takes
// 4-5 us of FP64 divisions and logarithms in a launch between two temperatures;
// put off, finish_rows evaluates them a thread each.
struct RawRow {
  long long sE, sE2, sM, sM2;
  unsigned long long sM4lo, sM4hi;
  double q;
  int R, Rp, Emin, pad;
};
static_assert(sizeof(RawRow) <= kRowCols * sizeof(double), "kept in the row's place");

// The state of a population whose temperature `step` is done, without its row
// (finish_step_kernel's, other than Emean, lnQ and sumlnQ).  One thread.
__device__ __forceinline__ void finish_raw(PopDev* st, int step, bool row_due, int R, int Rp, int Emin,
                                           unsigned long long iseq) {
  if (row_due) {
    RawRow* w = reinterpret_cast<RawRow*>(st->rows + (size_t)step * kRowCols);
    const RawRow r = {st->sE, st->sE2, st->sM, st->sM2, st->sM4lo, st->sM4hi, st->q, R, Rp, st->Emin, 0};
    *w = r;
    st->raw_rows = step;
    st->R_prev = R;
  }
  st->Emin = Emin;
  st->iseq = iseq;
  st->step = step + 1;
  st->sE = st->sE2 = st->sM = st->sM2 = 0;
  st->sM4lo = st->sM4hi = 0;
  st->Emin_acc = INT_MAX;
}

// A population's state once its temperature is finished: its step, size, lowest
// energy and draws used, from the state as the sweep left it.
struct Finished {
  int step, Rp, Emin;
  unsigned long long iseq;
  bool due, row_due;
};
__device__ __forceinline__ Finished finished(const PopDev* st, bool raw) {
  const int step0 = st->step, R0 = st->R_cur, Rp0 = st->R_prev, err = st->error, nsteps = st->nsteps, Emin = st->Emin,
            Emin_acc = st->Emin_acc, coding = st->coding;
  Finished f;
  f.iseq = st->iseq;
  f.due = raw && step0 <= nsteps;
  f.row_due = f.due && step0 > 0 && !err;
  f.step = step0 + (f.due ? 1 : 0);
  f.Rp = f.row_due ? R0 : Rp0;
  f.Emin = f.row_due || (f.due && step0 == 0) ? Emin_acc : Emin;
  const unsigned long long drawn =
      (unsigned long long)(coding == kMSC ? (R0 + kMsb - 1) / kMsb : R0) * kRefThreads;  // the resampled population's
  if (f.due && step0 == 0) f.iseq += drawn;  // ReplicaInit draws
  else if (f.row_due) f.iseq += (unsigned long long)(coding == kMSC ? (Rp0 + kMsb - 1) / kMsb * kMsb : Rp0) + drawn;
  return f;
}

// RAW (FP32 weights): the temperature before is finished first, its row left raw.
template <int CS, bool RAW>
__global__ void __launch_bounds__(kFusedThreads) resample_fused_kernel(PopDev* pops, BatchDev* b) {
  extern __shared__ float s_w[];  // [kFusedTiles][kFusedPitch] weights, then the list of heavy slots
  __shared__ float s_ps[CS * kFusedTiles], s_pc[CS * kFusedTiles];  // every tile's sum and compensation
  __shared__ double s_pd[CS * kFusedTiles];                         // FP64 tile sums
  __shared__ double s_wd[kFusedTiles * 8], s_q, s_lnq, s_logr;
  __shared__ uint32_t s_tot[CS], s_u[33];
  __shared__ int s_heavy;  // slots with more than kFewCopies copies: (slot, offset, copies) in s_w
  __shared__ bool s_last;
  const int rank = CS > 1 ? (int)blockIdx.x : 0, tid = threadIdx.x, lane = tid & 31;
  // the same variable of CTA r of this cluster
  auto remote = [](auto* p, int r) { return CS > 1 ? cooperative_groups::this_cluster().map_shared_rank(p, r) : p; };
  auto cluster_sync = [] {
    if (CS > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  };
  PopDev* st = pops + blockIdx.y;
  const Finished fin = finished(st, RAW);
  const int step = fin.step, Rp = fin.Rp, Emin = fin.Emin, Rp0 = RAW ? st->R_prev : 0;
  const bool go = step >= 1 && step <= st->nsteps && !st->error;  // the same in every CTA of the cluster
  // A CTA's shared memory may be written by others only once it has started,
  // and the state only once every CTA has read it: every thread arrives when it
  // has read the state and waits before the first remote store, or before the
  // state is finished below.  The energies' loads and the weights lie between
  // the two.
  if (CS > 1) cooperative_groups::this_cluster().barrier_arrive();
  if (CS > 1 && !go) cooperative_groups::this_cluster().barrier_wait();
  if (RAW && fin.due && !go && rank == 0) {
    if (CS == 1) __syncthreads();
    if (tid == 0) finish_raw(st, step - 1, fin.row_due, Rp, Rp0, Emin, fin.iseq);
  }
  if (go) {
    const int n = pop_units(st, Rp), Rinit = st->Rinit;
    const double dB = st->betas[step] - st->betas[step - 1], Em = st->Emean;
    const bool fp64 = st->weights == kFP64;
    const uint8_t* act = st->coding == kMSC ? st->active[st->parity] : nullptr;
    const int32_t* E = st->E;
    const float dBf = (float)dB;
    const int tiles = (n + kResThreads - 1) / kResThreads, per = (tiles + CS - 1) / CS;
    const int t0 = min(tiles, rank * per), nt = min(tiles, t0 + per) - t0;  // this CTA's tiles
    const int lo = t0 * kResThreads, m = min(n, lo + nt * kResThreads) - lo;  // and slots lo .. lo + m - 1
    // slot of this thread: k * kFusedThreads + tid.  Weights (FP32) or their warp sums (FP64)
    int e[kFusedSlots];
    bool in[kFusedSlots];
#pragma unroll
    for (int k = 0; k < kFusedSlots; ++k) {
      const int i = k * kFusedThreads + tid;
      in[k] = i < m && (!act || act[lo + i]);
      e[k] = in[k] ? E[lo + i] : 0;
      if ((i & ~31) >= nt * kResThreads) continue;  // warp-uniform
      if (fp64) {
        const double v = warp_sum(in[k] ? exp(-dB * (e[k] - Em)) : 0.0);
        if (lane == 0) s_wd[i >> 5] = v;
      } else {
        s_w[(i >> 8) * kFusedPitch + (i & 255)] = in[k] ? weight32(dBf, e[k], Emin) : 0.f;
      }
    }
    __syncthreads();
    if (CS > 1) cooperative_groups::this_cluster().barrier_wait();  // every CTA has started
    if (tid < nt) {  // warp 0: a tile per lane
      if (fp64) {
        const double v = tile_tree(s_wd + 8 * tid);
        for (int r = 0; r < CS; ++r) remote(s_pd, r)[t0 + tid] = v;
      } else {
        Comp32 c;
        comp_chain(c, s_w + tid * kFusedPitch, kResThreads);
        for (int r = 0; r < CS; ++r) {
          remote(s_ps, r)[t0 + tid] = c.s;
          remote(s_pc, r)[t0 + tid] = c.c;
        }
      }
    }
    uint32_t h[kFusedSlots];  // the slots' uniforms (independent of q)
    const unsigned long long seed = st->seed, sub = fin.iseq + (unsigned long long)lo;
#pragma unroll
    for (int k = 0; k < kFusedSlots; ++k) {
      const int i = k * kFusedThreads + tid;
      h[k] = in[k] ? ref_word(seed, sub + (unsigned long long)i, 0) : 0u;
    }
    if (tid == 64) {
      if (fp64) s_logr = log((double)Rp);
      s_heavy = 0;
    }
    cluster_sync();
    if (RAW && fin.due && rank == 0 && tid == 64)  // every CTA has read the state
      finish_raw(st, step - 1, fin.row_due, Rp, Rp0, Emin, fin.iseq);
    // q from the tiles' sums, in every CTA
    if (fp64) {
      if (tid < kResThreads) {
        const double v = warp_sum(tid < tiles ? s_pd[tid < CS * kFusedTiles ? tid : 0] : 0.0);
        if (lane == 0) s_wd[tid >> 5] = v;
      }
      __syncthreads();
      if (tid == 0) {
        s_q = tile_tree(s_wd);
        s_lnq = lnq_of(dB, Em, s_q, s_logr);
      }
    } else if (tid == 0) {
      Comp32 u;
      float cc = 0.f;
      comp_chain(u, s_ps, tiles);
#pragma unroll 8
      for (int i = 0; i < tiles; ++i) cc = __fadd_rn(cc, s_pc[i]);
      s_q = (double)__fadd_rn(u.s, __fadd_rn(u.c, cc));
    }
    __syncthreads();
    const double q = s_q, lnQ = fp64 ? s_lnq : 0.0;
    const float qf = (float)q, Rf = (float)Rinit;
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < kFusedSlots; ++k) {
      if (k * kFusedThreads >= m) break;  // block-uniform
      const int i = k * kFusedThreads + tid;
      uint32_t r = 0;
      if (in[k])
        r = fp64 ? copies_fp64(((double)Rinit) / Rp * exp(-dB * (double)e[k] - lnQ), h[k])
                 : copies_fp32(Rf * s_w[(i >> 8) * kFusedPitch + (i & 255)] / qf, h[k]);
      if (i < m) st->roff[lo + i] = r;
      h[k] = r;
    }
    uint32_t off[kFusedSlots];
#pragma unroll
    for (int k = 0; k < kFusedSlots; ++k) {  // (its barriers also end the reads of the weights)
      if (k * kFusedThreads >= m) break;
      uint32_t total;
      off[k] = run + block_exscan(h[k], s_u, &total);
      run += total;
    }
    if (tid == 0)
      for (int r = 0; r < CS; ++r) remote(s_tot, r)[rank] = run;
    cluster_sync();
    uint32_t base = 0, Rn = 0;
    for (int r = 0; r < CS; ++r) {
      if (r < rank) base += s_tot[r];
      Rn += s_tot[r];
    }
    const bool bad = Rn == 0u || Rn > (uint32_t)st->Rcap;
    if (!bad) {
      // offsets and the map: a slot's few copies are written by its thread,
      // those of a slot with many (a large dbeta against the energy spread
      // makes them, up to all of the population) by a warp, or the block
      uint32_t* src = st->src + base;
      uint32_t* offs = st->offs + lo;
      uint32_t* list = reinterpret_cast<uint32_t*>(s_w);
#pragma unroll
      for (int k = 0; k < kFusedSlots; ++k) {
        if (k * kFusedThreads >= m) break;
        const int i = k * kFusedThreads + tid;
        if (i < m) offs[i] = base + off[k];
        if (h[k] <= kFewCopies) {
          for (uint32_t c = 0; c < h[k]; ++c) src[off[k] + c] = (uint32_t)(lo + i);
        } else {
          const int at = atomicAdd(&s_heavy, 1);
          if (at < kHeavyMax) {
            list[3 * at] = (uint32_t)(lo + i);
            list[3 * at + 1] = off[k];
            list[3 * at + 2] = h[k];
          } else {
            for (uint32_t c = 0; c < h[k]; ++c) src[off[k] + c] = (uint32_t)(lo + i);
          }
        }
      }
      __syncthreads();
      const int nh = min(s_heavy, kHeavyMax);
      for (int q2 = tid >> 5; q2 < nh; q2 += kFusedThreads / 32) {
        const uint32_t j = list[3 * q2], o = list[3 * q2 + 1], r = list[3 * q2 + 2];
        if (r <= kFusedThreads)
          for (uint32_t c = lane; c < r; c += 32) src[o + c] = j;
      }
      for (int q2 = 0; q2 < nh; ++q2) {
        const uint32_t j = list[3 * q2], o = list[3 * q2 + 1], r = list[3 * q2 + 2];
        if (r > kFusedThreads)
          for (uint32_t c = tid; c < r; c += kFusedThreads) src[o + c] = j;
      }
    }
    if (rank == 0 && tid == 0) {  // every CTA has read the state: publish the new one
      st->q = q;
      if (fp64) st->lnQ = lnQ;
      else if (!b) st->lnQ = lnq_of(dB, (double)Emin, q, log((double)Rp));
      st->lnq_due = !fp64 && b ? 1 : 0;
      if (bad) st->error = Rn == 0u ? kErrExtinct : kErrCapacity;
      st->R_cur = bad ? 0 : (int)Rn;
      st->parity ^= 1;
    }
  }
  if (rank != 0 || !b) return;  // no remote access follows the last cluster barrier
  if (tid == 0) {
    __threadfence();
    s_last = gridDim.y == 1 || atomicAdd(&b->plan_ticket, 1u) == gridDim.y - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  plan_batch(b, 0, s_u);
  if (tid == 0) b->plan_ticket = 0;
}

// ------------------------------------------------------------- work plan
// Block (0, 0); the others, where there are any, finish the scatter before it.
__global__ void __launch_bounds__(1024) plan_kernel(BatchDev* b, int energy_only) {
  __shared__ uint32_t s_u[33];
  if (blockIdx.x > 0) scatter_heavy(b->pops + blockIdx.y, (int)blockIdx.x - 1, (int)gridDim.x - 1);
  else if (blockIdx.y == 0) plan_batch(b, energy_only, s_u);
}

__global__ void __launch_bounds__(1024) scatter_heavy_kernel(PopDev* pops) {
  scatter_heavy(pops + blockIdx.y, (int)blockIdx.x, (int)gridDim.x);
}

// --------------------------------------------------------- run bookkeeping
__global__ void begin_run_kernel(PopDev* pops) {
  PopDev* st = pops + blockIdx.x;
  st->step = 0;
  st->run += 1;  // -1 at creation: the first run is run 0
  st->R_prev = st->R_cur = st->Rinit;
  st->parity = 0;
  st->error = 0;
  st->Emean = 0.0;  // the first resampling uses Emean = 0 (PAisingSSC.cu:483)
  st->Emin = 0;
  st->sumlnQ = 0.0;
  st->lnQ = 0.0;
  st->lnq_due = 0;
  st->raw_rows = 0;
  st->q = 0.0;
  st->sE = st->sE2 = st->sM = st->sM2 = 0;
  st->sM4lo = st->sM4hi = 0;
  st->Emin_acc = INT_MAX;
  st->ticket = 0;
  double* row = st->rows;  // beta = 0 row: only betaF and R are defined (PAisingSSC.cu:435,453)
  for (int c = 0; c < kRowCols; ++c) row[c] = 0.0;
  row[6] = st->bf0 / st->N;
  row[8] = (double)st->Rinit;
  st->last_rec = -1;
  st->last_fam = -1;
}

// ------------------------------------------------------ family statistics
// Not written by the reference: with c_f the replicas descended from initial
// replica f and R the population size, every temperature records
//   {families with c_f > 0, rho_t = sum_f c_f^2 / R,
//    S_f = -sum_f (c_f/R) ln(c_f/R) = ln R - (1/R) sum_f c_f ln c_f}.
// Ancestors are initial linear replica indices (MSC: 32 * group + bit) and
// follow every copy the resampling makes.

// c ln c, and its table for small counts (an FP64 logarithm takes a warp
// thousands of cycles; most families have few members), filled once per handle
__device__ __forceinline__ double c_ln_c(double c) { return c * log(c); }
__global__ void clnc_kernel(double* t) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < kClncTable) t[c] = c > 0 ? c_ln_c((double)c) : 0.0;
}

// After the initial population: every replica is its own family.
__global__ void family_init_kernel(PopDev* pops) {
  PopDev* st = pops + blockIdx.y;
  if (!st->family) return;
  const int n = pop_units(st, st->R_cur), R = st->R_cur;
  int32_t* a = st->anc[st->parity];
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) a[j] = j < R ? j : -1;
}

// After the spin gather of a temperature step: new replica slots take the
// ancestor of their source (SSC, and MSC with the native stream: slot s <-
// src[s]; MSC with the reference stream: slot 32 g + b holds offspring
// s = b rg_new + g, PAisingMSC.cu:413-414).
__global__ void family_resample_kernel(PopDev* pops) {
  PopDev* st = pops + blockIdx.y;
  if (!st->family || !pop_stepping(st)) return;
  const int Rn = st->R_cur, n = pop_units(st, Rn);
  const int32_t* old = st->anc[st->parity ^ 1];
  int32_t* neu = st->anc[st->parity];
  const uint32_t* src = st->src;
  const bool transposed = st->coding == kMSC && st->rng_mode == kRefCoords;
  const int rgn = (Rn + kMsb - 1) / kMsb;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int s = transposed ? (j & (kMsb - 1)) * rgn + (j >> 5) : j;
    neu[j] = s < Rn ? old[src[s]] : -1;
  }
}

// After record_kernel has counted the families of the temperature just finished:
// reduce the counts (clearing them for the next temperature); the
// last block combines the per-block partial sums in block order.
__global__ void __launch_bounds__(kResThreads) family_reduce_kernel(PopDev* pops) {
  __shared__ double s_d[33];
  __shared__ unsigned long long s_i[33];
  PopDev* st = pops + blockIdx.y;
  const int s = st->step - 1;
  if (!st->family || s <= st->last_fam || st->error) return;
  // counts and squares are whole numbers, exact in any order while R^2 stays
  // below 2^53: summed as integers; only c ln c needs FP64, in a fixed order
  const int nf_bins = st->Rinit;
  const bool exact = st->R_cur < (1 << 26);
  unsigned long long nf = 0, c2 = 0;
  double c2d = 0.0, clnc = 0.0;
  int lo, hi;
  block_chunk(nf_bins, lo, hi);
  for (int f = lo + (int)threadIdx.x; f < hi; f += blockDim.x) {
    const uint32_t c = st->fam_cnt[f];
    if (!c) continue;
    st->fam_cnt[f] = 0u;
    nf += 1;
    if (exact) c2 += (unsigned long long)c * c;
    else c2d += (double)c * (double)c;
    clnc += c < (uint32_t)kClncTable ? st->clnc[c] : c_ln_c((double)c);
  }
  nf = block_sum(nf, s_i);
  if (exact) c2 = block_sum(c2, s_i);
  else c2d = block_sum(c2d, s_d);
  clnc = block_sum(clnc, s_d);
  if (threadIdx.x == 0) {
    st->fam_part[3 * blockIdx.x] = (double)nf;
    st->fam_part[3 * blockIdx.x + 1] = exact ? (double)c2 : c2d;
    st->fam_part[3 * blockIdx.x + 2] = clnc;
  }
  if (last_block(&st->ticket)) {
    // the partials through shared memory, loaded side by side; one thread per
    // column adds them in block order
    __shared__ double s_p[3 * kResThreads], s_row[4];
    double a = 0.0;
    const int tid = threadIdx.x, col = tid >> 5;  // lane 0 of warps 0..2: the columns; of warp 3: ln R
    const double R = (double)st->R_cur;
    if (tid == 96) s_row[3] = log(R);
    for (int k0 = 0; k0 < (int)gridDim.x; k0 += kResThreads) {
      const int nk = min(kResThreads, (int)gridDim.x - k0);
      __syncthreads();
      for (int i = tid; i < 3 * nk; i += blockDim.x) s_p[i] = ((volatile double*)st->fam_part)[3 * k0 + i];
      __syncthreads();
      if ((tid & 31) == 0 && col < 3)
        for (int k = 0; k < nk; ++k) a += s_p[3 * k + col];
    }
    if ((tid & 31) == 0 && col < 3) s_row[col] = col == 0 ? a : a / R;
    __syncthreads();
    if (tid != 0) return;
    double* row = st->fam_rows + (size_t)s * 3;
    row[0] = s_row[0];
    row[1] = s_row[1];
    row[2] = s_row[3] - s_row[2];
    st->last_fam = s;
    st->ticket = 0;
  }
}

// ---------------------------------------------- per-temperature records
// (and, beside the records, the families of the temperature for
// family_reduce_kernel: a launch of its own took 5 us per temperature)
// After finish_step: the population of temperature step-1, if not recorded
// yet in this run, enters the run's energy histogram (UpdateShistE,
// PAisingSSC.cu:296-302, PAisingMSC.cu:454-460: active replicas only) and/or
// the energy ring (EnergiesPopStore, PAisingSSC.cu:563-578: energies in
// replica order; MSC group-major with the active flags).  The last block to
// finish (ticket) marks the temperature recorded, so every block has tested
// the guard before it changes.
__global__ void __launch_bounds__(kResThreads) record_kernel(PopDev* pops) {
  PopDev* st = pops + blockIdx.y;
  const int s = st->step - 1;
  const bool rec = st->rec && s > st->last_rec && !st->error, fam = st->family && s > st->last_fam && !st->error;
  if (!rec && !fam) return;
  const int R = st->R_cur, n = pop_units(st, R), N = st->N;
  const int32_t* anc = fam ? st->anc[st->parity] : nullptr;
  const bool msc = st->coding == kMSC;
  const uint8_t* act = msc ? st->active[st->parity] : nullptr;
  const int32_t* E = st->E;
  int32_t* el = nullptr;
  uint8_t* al = nullptr;
  if (rec && (st->rec & kRecEnergies)) {
    const size_t stride = msc ? (size_t)st->rgcap * kMsb : (size_t)st->Rcap;
    const size_t slot = (size_t)(s % st->ring) * stride;
    el = st->elog + slot;
    if (msc) al = st->alog + slot;
  }
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int e = E[j];
    const bool a = !act || act[j];
    if (rec && (st->rec & kRecMhr) && a) atomicAdd(&st->mhr_hist[(e + 2 * N) >> 2], 1ull);
    if (fam && a && anc[j] >= 0) atomicAdd(&st->fam_cnt[anc[j]], 1u);
    if (el) el[j] = e;
    if (al) al[j] = a ? 1 : 0;
  }
  if (rec && last_block(&st->ticket)) {
    if (threadIdx.x == 0) {
      if (el) st->nlog[s % st->ring] = n;
      st->last_rec = s;
      st->ticket = 0;
    }
  }
}

// After a sweep kernel: observables of the step (PAisingSSC.cu:620-630)
// written to the output row, state advanced to the next temperature.  The
// arithmetic uses explicitly rounded operations so that no multiply-add is
// fused and the row is identical to an unfused host evaluation.
// One block of two warps per population: FP64 divisions and logarithms are
// long serial chains, so the columns' divisions run side by side, a lane each,
// and the two logarithms of an lnQ left due on the other warp (one thread
// doing them one after the other took 8 us per temperature).
__global__ void __launch_bounds__(64) finish_step_kernel(PopDev* pops) {
  __shared__ double s_log[2];
  PopDev* st = pops + blockIdx.x;
  const int step = st->step, tid = threadIdx.x;
  if (step > st->nsteps) return;  // this population's schedule is complete
  const bool msc = st->coding == kMSC, row_due = step > 0 && !st->error;
  const int R = st->R_cur, Rp = st->R_prev, N = st->N;
  const double b = step > 0 ? st->betas[step] : 0.0, dB = step > 0 ? b - st->betas[step - 1] : 0.0;
  if (row_due && st->lnq_due && tid >= 32 && tid < 34) s_log[tid - 32] = log(tid == 32 ? st->q : (double)Rp);
  // sums over the population (lanes 0..4): E, E^2, |M|, M^2, M^4
  double v = 0.0;
  const double Rd = (double)R, Nd = (double)N;
  if (tid == 0) v = (double)st->sE;
  if (tid == 1) v = (double)st->sE2;
  if (tid == 2) v = (double)st->sM;
  if (tid == 3) v = (double)st->sM2;
  if (tid == 4) v = u128_to_double(st->sM4lo, st->sM4hi);
  if (row_due && tid < 32) v = __ddiv_rn(v, Rd);
  const double E = __shfl_sync(0xffffffffu, v, 0);
  if (tid == 1) v = __dmul_rn(__dmul_rn(__dsub_rn(v, __dmul_rn(E, E)), b), b);  // C
  if (row_due && tid < 32) {  // per site, M^2 and M^4 per site squared and to the fourth
    v = __ddiv_rn(v, Nd);
    if (tid == 3 || tid == 4) v = __ddiv_rn(v, Nd);
    if (tid == 4) v = __ddiv_rn(__ddiv_rn(v, Nd), Nd);
  }
  __syncthreads();
  double* row = st->rows + (size_t)step * kRowCols;
  if (row_due && tid < 5) row[1 + tid] = v;
  if (tid != 0) return;
  if (step == 0) {
    const int rg = (R + kMsb - 1) / kMsb;
    st->iseq += (unsigned long long)(msc ? rg : R) * kRefThreads;  // ReplicaInit draws
    st->Emin = st->Emin_acc;
  } else if (row_due) {
    const double lnQ = st->lnq_due ? -dB * (double)st->Emin + s_log[0] - s_log[1] : st->lnQ;
    const double sum = __dsub_rn(st->sumlnQ, lnQ);
    const double BF = __dadd_rn(st->bf0, sum);
    const double S = __dsub_rn(__dmul_rn(b, E), BF);
    row[0] = b;
    row[6] = __ddiv_rn(BF, Nd);
    row[7] = __ddiv_rn(S, Nd);
    row[8] = Rd;
    row[9] = lnQ;
    st->lnQ = lnQ;
    st->lnq_due = 0;
    st->sumlnQ = sum;
    st->Emean = E;
    st->Emin = st->Emin_acc;
    const int rgp = (Rp + kMsb - 1) / kMsb, rgc = (R + kMsb - 1) / kMsb;
    st->iseq += msc ? (unsigned long long)rgp * kMsb + (unsigned long long)rgc * kRefThreads
                    : (unsigned long long)Rp + (unsigned long long)R * kRefThreads;
    st->R_prev = R;
  }
  st->step = step + 1;
  st->sE = st->sE2 = st->sM = st->sM2 = 0;
  st->sM4lo = st->sM4hi = 0;
  st->Emin_acc = INT_MAX;
}

// The last temperature's state and the rows left raw: a thread per row, then the
// running sum of lnQ in order, then the columns that need it.  The arithmetic of
// finish_step_kernel, value by value.
constexpr int kRowThreads = 256;
__global__ void __launch_bounds__(kRowThreads) finish_rows_kernel(PopDev* pops) {
  __shared__ double s_lnq[kRowThreads], s_sum[kRowThreads];
  PopDev* st = pops + blockIdx.x;
  const int tid = threadIdx.x;
  const Finished fin = finished(st, true);
  const int Rp0 = st->R_prev;
  __syncthreads();
  if (tid == 0 && fin.due) finish_raw(st, fin.step - 1, fin.row_due, fin.Rp, Rp0, fin.Emin, fin.iseq);
  __syncthreads();
  const int rows = st->raw_rows;
  if (rows == 0) return;
  const double Nd = (double)st->N, bf0 = st->bf0;
  double sum0 = st->sumlnQ;  // (thread 0)
  for (int r0 = 1; r0 <= rows; r0 += kRowThreads) {
    const int step = r0 + tid;
    const bool is = step <= rows;
    double* row = st->rows + (size_t)step * kRowCols;
    double b = 0.0, E = 0.0, Rd = 0.0, lnQ = 0.0;
    if (is) {
      const RawRow w = *reinterpret_cast<const RawRow*>(row);
      b = st->betas[step];
      Rd = (double)w.R;
      E = __ddiv_rn((double)w.sE, Rd);
      const double E2 = __ddiv_rn((double)w.sE2, Rd), M = __ddiv_rn((double)w.sM, Rd), M2 = __ddiv_rn((double)w.sM2, Rd),
                   M4 = __ddiv_rn(u128_to_double(w.sM4lo, w.sM4hi), Rd);
      lnQ = -(b - st->betas[step - 1]) * (double)w.Emin + log(w.q) - log((double)w.Rp);
      row[0] = b;
      row[1] = __ddiv_rn(E, Nd);
      row[2] = __ddiv_rn(__dmul_rn(__dmul_rn(__dsub_rn(E2, __dmul_rn(E, E)), b), b), Nd);  // C
      row[3] = __ddiv_rn(M, Nd);
      row[4] = __ddiv_rn(__ddiv_rn(M2, Nd), Nd);
      row[5] = __ddiv_rn(__ddiv_rn(__ddiv_rn(__ddiv_rn(M4, Nd), Nd), Nd), Nd);
      row[8] = Rd;
      row[9] = lnQ;
    }
    s_lnq[tid] = lnQ;
    __syncthreads();
    if (tid == 0)
      for (int k = 0; k < kRowThreads && r0 + k <= rows; ++k) s_sum[k] = sum0 = __dsub_rn(sum0, s_lnq[k]);
    __syncthreads();
    if (is) {
      const double sum = s_sum[tid], BF = __dadd_rn(bf0, sum), S = __dsub_rn(__dmul_rn(b, E), BF);
      row[6] = __ddiv_rn(BF, Nd);
      row[7] = __ddiv_rn(S, Nd);
      if (step == rows) {
        st->lnQ = lnQ;
        st->lnq_due = 0;
        st->sumlnQ = sum;
        st->Emean = E;
        st->raw_rows = 0;
      }
    }
  }
}

// ------------------------------------------------- adaptive temperature step
// After temperature step-1 (>= 1) of an adaptive population: the next beta,
// as the reference's AdaptiveStep build chooses it (PAisingSSC.cu:644-660):
// starting from the previous step, grow it by 1.1x while the energy-histogram
// overlap stays >= MaxOverlap (and beta stays below beta_final), otherwise
// bisect between 0 and the step until MinOverlap <= overlap < MaxOverlap,
// and clamp the last step onto beta_final.  The overlap of step dB
// (CalcOverlap, PAisingSSC.cu:316-334) is
//   lnQ = -dB Emean + ln sum_i exp(-dB (E_i - Emean)) - ln R,
//   overlap = (1/R) sum_i min(1, Rinit/R exp(-dB E_i - lnQ)),
// evaluated here over the histogram of the population's energies (energies
// are -2N + 4k), so each evaluation costs a pass over at most N+1 bins
// instead of R replicas; one CTA per population, FP64 throughout.
//
// What bounds it: an SM's FP64 units, which take a warp's exponential in about
// 560 cycles.  The populated levels -- a few hundred of up to N+1 -- are
// therefore listed once, the exponentials taken over the list, a lane each,
// and the terms put back at their levels, where the sums run over whole
// levels in the order they always had (warps without a populated level add
// nothing).  L = 32 R = 5000: 41 -> 16 us per
// temperature, the first one (about ten evaluations) 186 -> 41.
constexpr int kAdaptThreads = 1024;
constexpr int kMaxBisect = 200;  // the reference bisects without a bound
constexpr int kAdaptLevels = 2048;      // listed levels (shared memory)
constexpr int kAdaptBins = 4096;        // histogram in shared memory up to this many levels

__global__ void __launch_bounds__(kAdaptThreads) adapt_kernel(PopDev* pops) {
  __shared__ double s_red[32];
  __shared__ double s_db, s_lnq, s_ratio;
  __shared__ bool s_done;
  __shared__ uint32_t s_hist[kAdaptBins], s_u[33];
  __shared__ int s_level[kAdaptLevels];
  __shared__ double s_term[kAdaptLevels];
  PopDev* st = pops + blockIdx.x;
  const int step = st->step;  // index of the temperature to choose (finish_step has advanced it)
  if (!st->adaptive || step < 2 || step > st->nsteps || st->error) return;
  const int N = st->N, nb = N + 1, R = st->R_cur, tid = threadIdx.x, lane = tid & 31;
  uint32_t* hist = nb <= kAdaptBins ? s_hist : st->hist;
  for (int i = tid; i < nb; i += blockDim.x) hist[i] = 0u;
  __syncthreads();
  const bool msc = st->coding == kMSC;
  const int units = pop_units(st, R);
  const uint8_t* act = msc ? st->active[st->parity] : nullptr;
  for (int i = tid; i < units; i += blockDim.x)
    if (!msc || act[i]) atomicAdd(&hist[(st->E[i] + 2 * N) >> 2], 1u);
  __syncthreads();

  // The populated levels as a list, per thread of the sums: thread t's levels
  // t, t + 1024, ... lie at s_level[first .. first + mine - 1].
  uint32_t mine = 0, nlev;
  for (int i = tid; i < nb; i += blockDim.x) mine += hist[i] != 0u;
  const uint32_t first = block_exscan(mine, s_u, &nlev);
  const bool listed = nlev <= (uint32_t)kAdaptLevels;  // else every thread evaluates its own levels
  if (listed) {
    uint32_t k = first;
    for (int i = tid; i < nb; i += blockDim.x)
      if (hist[i]) s_level[k++] = i;
  }
  __syncthreads();

  // Scalars are thread 0's alone: an FP64 logarithm or division that every
  // thread of the block makes takes 32 warps' time on the FP64 units.
  const double Em = st->Emean;
  double logR = 0.0, Rd = 0.0;
  if (tid == 0) {
    Rd = (double)R;
    logR = log(Rd);
    s_ratio = (double)st->Rinit / Rd;
  }
  // sum over the levels of term(level, count), in block_sum's order; thread 0
  // has it
  auto level_sum = [&](auto term) {
    double v = 0.0;
    if (listed) {
      for (uint32_t k = tid; k < nlev; k += blockDim.x) s_term[k] = term(s_level[k], (double)hist[s_level[k]]);
      __syncthreads();
      for (uint32_t k = 0; k < mine; ++k) v += s_term[first + k];
    } else {
      for (int i = tid; i < nb; i += blockDim.x)
        if (hist[i]) v += term(i, (double)hist[i]);
    }
    if (__any_sync(0xffffffffu, mine != 0u)) v = warp_sum(v);
    if (lane == 0) s_red[tid >> 5] = v;
    __syncthreads();
    return tid < 32 ? warp_sum(s_red[lane]) : 0.0;
  };

  const double Bp = st->betas[step - 1], Bfin = st->beta_fin, lo = st->min_ov, hi = st->max_ov;
  double dBmin = 0.0, dBmax = st->dbeta_cur, dBmean = 0.0;
  bool grow = true;
  int it = 0;
  if (tid == 0) {
    s_db = dBmax;
    s_done = false;
  }
  __syncthreads();
  for (;;) {
    const double dB = s_db;
    const double q = level_sum([&](int i, double c) { return c * exp(-dB * ((double)(4 * i - 2 * N) - Em)); });
    if (tid == 0) s_lnq = -dB * Em + log(q) - logR;
    __syncthreads();
    const double lnQ = s_lnq, ratio = s_ratio;
    double ov = level_sum([&](int i, double c) {
      return c * fmin(1.0, ratio * exp(-dB * (double)(4 * i - 2 * N) - lnQ));
    });
    if (tid == 0) {
      ov /= Rd;
      bool done = false;
      if (grow) {
        if (ov >= hi && Bp + dBmax < Bfin) {
          dBmax *= 1.1;
          s_db = dBmax;
        } else if (ov >= lo) {
          dBmean = dBmax;
          done = true;
        } else {
          grow = false;
        }
      } else if (it + 1 >= kMaxBisect) {
        done = true;
      } else {
        if (ov < lo) dBmax = dBmean;
        else if (ov >= hi) dBmin = dBmean;
        else done = true;
        ++it;
      }
      if (!grow && !done) {
        dBmean = 0.5 * (dBmin + dBmax);
        s_db = dBmean;
      }
      s_done = done;
    }
    __syncthreads();
    if (s_done) break;
  }
  if (tid >= 32) return;
  int more = 0;
  double next = 0.0;
  if (tid == 0) {
    const double dB = (Bp < Bfin && Bp + dBmean > Bfin) ? Bfin - Bp : dBmean;
    const double Bn = Bp + dB;
    st->dbeta_cur = dB;
    if (!(Bn <= Bfin)) {
      st->nsteps = step - 1;  // the schedule ends with the temperature just computed
    } else if (step >= kNBmax - 1) {
      st->error = kErrTooManySteps;  // PAisingSSC.cu:634-641
    } else {
      st->betas[step] = Bn;
      next = Bn;
      more = 1;
    }
  }
  // a lane per threshold word: twelve FP64 exponentials side by side.  The new
  // temperature comes by the shuffle itself, which orders no memory between lanes
  more = __shfl_sync(0xffffffffu, more, 0);
  next = __shfl_sync(0xffffffffu, next, 0);
  if (more && tid < kThrPerStep) st->thr[(size_t)step * kThrPerStep + tid] = threshold_word(next, tid);
}

// ------------------------------------------------------------ launchers
int res_blocks(long long units) {
  long long b = (units + kResThreads - 1) / kResThreads;
  if (b > kResBlocksMax) b = kResBlocksMax;
  return (int)(b < 1 ? 1 : b);
}

void geom_to_pop(const SweepGeom& g, PopDev* h) {
  h->Wr = g.Wr;
  h->rpp = g.rpp;
  h->T = g.T;
  h->npass = g.npass;
  h->kconst = g.kconst;
  h->gpt = g.G;
  h->seg = g.seg;
  h->invL = recip32(g.L);
  h->invWr = recip32(g.Wr);
}

cudaError_t sweep_setup(int coding, int rng_mode, int smem, SweepLaunch* out, int kind) {
  out->kind = kGeneral;
  return coding == kMSC ? msc_sweep_setup(rng_mode, smem, out, kind) : ssc_sweep_setup(rng_mode, smem, out);
}

template <int CS, bool RAW>
static cudaError_t fused_launch(PopDev* pops, BatchDev* b, int npop, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(CS, npop);
  cfg.blockDim = dim3(kFusedThreads);
  cfg.dynamicSmemBytes = kFusedTiles * kFusedPitch * sizeof(float);
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, resample_fused_kernel<CS, RAW>, pops, b);
}

// FP64 weights: an SM's FP64 units take an exponential of 1024 slots in about
// 18000 cycles, so one launch pays only while a CTA has one tile (2048 slots;
// at 20000 a cluster took 53 us where the passes spread over 79 SMs take 40);
// a cluster from the first slot on for the same reason.  FP32: one CTA up to
// 2048 slots, where a cluster's barriers cost more than its CTAs save.
//
// A cluster of eight CTAs of 1024 threads, one per SM, serves one population:
// fifteen run side by side, and in a larger batch the rest wait, where the
// passes pack a tile of 256 slots into a block and eight blocks into an SM.
// Whole temperatures, L = 8, one sweep, us by the passes and by one launch:
// 1300 replicas (2336 slots) 24 populations 60 and 56, 38 69 and 73, 1000 764
// and 1295; 2500 (4256) 24 63 and 56, 38 76 and 78, 1000 944 and 1410; 6000
// (9856) 57 123 and 120, 76 148 and 154, 1000 1523 and 1798; from 20000 (32256)
// on one launch is the faster at any number (1000: 3920 and 3455).  FP64, 300
// replicas: 8 populations 49 and 45, 16 54 and 62, 1000 632 and 1433.  (One CTA
// per population, FP32: at any number, 1000 populations of 300 678 and 595.)
constexpr int kFusedPops64 = 15;          // FP64
constexpr int kFusedPops = 16;            // FP32 clusters: one more with every 256 slots,
constexpr int kFusedManyUnits = 16384;    // and from here on any number
bool resample_fused(long long max_units, int weights, int npop) {
  if (weights == kFP64) return max_units <= kFusedOneUnits && npop <= kFusedPops64;
  if (max_units <= kFusedOneUnits || max_units > kFusedMaxUnits) return max_units <= kFusedOneUnits;
  return max_units >= kFusedManyUnits || npop <= kFusedPops + max_units / kResThreads;
}

cudaError_t launch_resample_fused(PopDev* pops, BatchDev* b, int npop, long long max_units, int weights, bool raw,
                                  cudaStream_t s) {
  if (weights == kFP64) return fused_launch<kFusedCluster, false>(pops, b, npop, s);
  if (max_units <= kFusedOneUnits)
    return raw ? fused_launch<1, true>(pops, b, npop, s) : fused_launch<1, false>(pops, b, npop, s);
  return raw ? fused_launch<kFusedCluster, true>(pops, b, npop, s) : fused_launch<kFusedCluster, false>(pops, b, npop, s);
}

cudaError_t launch_plan(BatchDev* b, int npop, int energy_only, bool scattered, cudaStream_t s) {
  plan_kernel<<<scattered ? dim3(1 + heavy_blocks(npop), npop) : dim3(1), 1024, 0, s>>>(b, energy_only);
  return cudaGetLastError();
}

cudaError_t launch_sweep(BatchDev* b, int coding, int rng_mode, int energy_only, unsigned long long seed,
                         const SweepLaunch& sl, cudaStream_t s) {
  return coding == kMSC ? launch_msc_sweep(b, rng_mode, energy_only, seed, sl, s)
                        : launch_ssc_sweep(b, rng_mode, energy_only, seed, sl, s);
}

cudaError_t launch_init(PopDev* pops, int npop, int coding, cudaStream_t s) {
  return coding == kMSC ? launch_msc_init(pops, npop, s) : launch_ssc_init(pops, npop, s);
}

cudaError_t launch_resample(BatchDev* b, int coding, int rng_mode, cudaStream_t s) {
  return coding == kMSC ? launch_msc_resample(b, rng_mode, s) : launch_ssc_resample(b, s);
}

cudaError_t launch_q(PopDev* pops, int npop, int blocks, cudaStream_t s) {
  q_kernel<<<dim3(blocks, npop), kResThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

bool resample_by_level(int R, int N, int weights) { return weights == kFP64 && R >= N + kTableUnits; }

cudaError_t launch_weight_table(PopDev* pops, int npop, int maxN, int copies, cudaStream_t s) {
  weight_table_kernel<<<dim3(maxN / kResThreads + 1, npop), kResThreads, 0, s>>>(pops, copies);
  return cudaGetLastError();
}

cudaError_t launch_copy_numbers(PopDev* pops, int npop, int blocks, cudaStream_t s) {
  copy_numbers_kernel<<<dim3(blocks, npop), kResThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_scatter(PopDev* pops, int npop, int blocks, cudaStream_t s) {
  scatter_kernel<<<dim3(blocks, npop), kResThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_scatter_heavy(PopDev* pops, int npop, cudaStream_t s) {
  scatter_heavy_kernel<<<dim3(heavy_blocks(npop), npop), 1024, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_begin_run(PopDev* pops, int npop, cudaStream_t s) {
  begin_run_kernel<<<npop, 1, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_finish_step(PopDev* pops, int npop, cudaStream_t s) {
  finish_step_kernel<<<npop, 64, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_finish_rows(PopDev* pops, int npop, cudaStream_t s) {
  finish_rows_kernel<<<npop, kRowThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_clnc(double* table, cudaStream_t s) {
  clnc_kernel<<<kClncTable / 256, 256, 0, s>>>(table);
  return cudaGetLastError();
}

cudaError_t launch_family_init(PopDev* pops, int npop, int blocks, cudaStream_t s) {
  family_init_kernel<<<dim3(blocks, npop), kResThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_family_resample(PopDev* pops, int npop, int blocks, cudaStream_t s) {
  family_resample_kernel<<<dim3(blocks, npop), kResThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_family_stats(PopDev* pops, int npop, int blocks, cudaStream_t s) {
  family_reduce_kernel<<<dim3(blocks, npop), kResThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_record(PopDev* pops, int npop, int blocks, cudaStream_t s) {
  record_kernel<<<dim3(blocks, npop), kResThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_adapt(PopDev* pops, int npop, cudaStream_t s) {
  adapt_kernel<<<npop, kAdaptThreads, 0, s>>>(pops);
  return cudaGetLastError();
}

}  // namespace pa
