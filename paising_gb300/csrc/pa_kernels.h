// pa_kernels.h -- host-side launchers of the engine's CUDA kernels.
//
// All launchers work on a batch of populations: per-population kernels take
// the population from blockIdx.y (resampling) or blockIdx.x (bookkeeping);
// the sweep kernels are persistent and take work units of all populations
// from one queue (BatchDev::work_next).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "pa_state.h"

namespace pa {

// Thread layout of a sweep over one lattice size (chosen on the host and
// stored per population in PopDev).
struct SweepGeom {
  int L, N, half;
  int Wr;      // 32-bit words per sublattice row (SSC: 4 sites/word -> L/8; MSC: 1 site/word -> L/2)
  int rpp;     // sublattice rows handled per pass
  int T;       // threads doing site work = Wr * rpp (<= kSweepThreads)
  int npass;   // ceil(L / rpp)
  int kconst;  // (N/2)/128 when 128 divides N/2 (draws per reference thread per half sweep), else 0
  int smem;    // dynamic shared memory bytes for one work unit
  int G = 1;   // MSC groups per work unit: G lattices stacked as G*L rows of one sweep
              // (SSC bit planes: replicas per work unit)
  int seg = 0; // SSC bit planes: sites of a sublattice row per word segment
};

// ceil(2^32 / d) for 2 <= d < 2^16: then __umulhi(n, recip32(d)) == n / d
// for every n < 2^16 (the rounding error n * (ceil - 2^32/d) / 2^32 < 2^-16 is
// smaller than the distance 1/d from n/d to the next integer).
inline unsigned int recip32(int d) {
  return (unsigned int)((0x100000000ull + (unsigned long long)d - 1) / (unsigned long long)d);
}

bool ssc_geom(int L, SweepGeom* g);
// tile: groups per work unit (0 automatic); groups: how many groups the
// sweep launches will hold and slots: resident CTAs of the persistent grid,
// which together drive the automatic choice (single-group tiles when either
// is 0)
bool msc_geom(int L, SweepGeom* g, int tile = 0, long long groups = 0, int slots = 0);
void geom_to_pop(const SweepGeom& g, PopDev* h);

// Kernel of an MSC native-stream launch, by the forms its populations need:
constexpr int kGeneral = 0;   // units of several batches per thread, other sizes
constexpr int kOneBatch = 1;  // units of one batch of two to four sites per thread
constexpr int kCommon = 2;    // L = 64 and 128, one site per thread, or several kinds without 96
constexpr int kMixed = 3;     // L = 96 (one group per unit), alone or among others
struct SweepLaunch {
  int grid, block, smem;
  int nsm;      // one-CTA sweeps: SMs that first units are spread over (first_unit), 0: by block index
  int kind;     // MSC, native stream: which kernel (msc_kind)
};
// Persistent grid for a sweep kernel with `smem` bytes of dynamic shared memory.
cudaError_t sweep_setup(int coding, int rng_mode, int smem, SweepLaunch* out, int kind = kGeneral);
// The kind of an MSC population's work units, and of a launch that holds kinds a and b.
int msc_kind(const SweepGeom& g);
int msc_kinds(int a, int b);

// Work plan of the next gather and sweep launches: unit counts of the
// populations that take part (energy_only: populations at step 0), prefix
// sums, queue resets.
// scattered: it follows launch_scatter and does launch_scatter_heavy's work as well.
cudaError_t launch_plan(BatchDev* b, int npop, int energy_only, bool scattered, cudaStream_t s);
// `seed` keys the native sweep stream of the whole batch.
cudaError_t launch_sweep(BatchDev* b, int coding, int rng_mode, int energy_only, unsigned long long seed,
                         const SweepLaunch& sl, cudaStream_t s);

// Random (or caller-supplied) initial populations.
cudaError_t launch_init(PopDev* pops, int npop, int coding, cudaStream_t s);

// Resampling (both codings); `blocks` from res_blocks().
int res_blocks(long long max_units);
cudaError_t launch_q(PopDev* pops, int npop, int blocks, cudaStream_t s);
// FP64 weights by energy level, before q (copies 0) and before the copy numbers
// (1), for populations with a table: those of resample_by_level's sizes.
bool resample_by_level(int R, int N, int weights);
cudaError_t launch_weight_table(PopDev* pops, int npop, int maxN, int copies, cudaStream_t s);
cudaError_t launch_copy_numbers(PopDev* pops, int npop, int blocks, cudaStream_t s);
cudaError_t launch_scatter(PopDev* pops, int npop, int blocks, cudaStream_t s);
// The copies of replicas with very many, which launch_scatter leaves out.
cudaError_t launch_scatter_heavy(PopDev* pops, int npop, cudaStream_t s);
// The three and the work plan (b; may be null: no plan) as one launch, for
// batches whose populations and slots (max_units, the largest's) pass
// resample_fused.
bool resample_fused(long long max_units, int weights, int npop);
cudaError_t launch_resample_fused(PopDev* pops, BatchDev* b, int npop, long long max_units, int weights, bool raw,
                                  cudaStream_t s);
// Gather of the resampled populations of the batch, planned by launch_plan or
// launch_resample_fused: persistent, units of every population from one queue.
cudaError_t launch_resample(BatchDev* b, int coding, int rng_mode, cudaStream_t s);

// Coding-specific launchers behind the generic ones above.
cudaError_t ssc_sweep_setup(int rng_mode, int smem, SweepLaunch* out);
cudaError_t msc_sweep_setup(int rng_mode, int smem, SweepLaunch* out, int kind);
cudaError_t launch_ssc_sweep(BatchDev* b, int rng_mode, int energy_only, unsigned long long seed,
                             const SweepLaunch& sl, cudaStream_t s);
cudaError_t launch_msc_sweep(BatchDev* b, int rng_mode, int energy_only, unsigned long long seed,
                             const SweepLaunch& sl, cudaStream_t s);
cudaError_t launch_ssc_init(PopDev* pops, int npop, cudaStream_t s);
cudaError_t launch_msc_init(PopDev* pops, int npop, cudaStream_t s);
cudaError_t launch_ssc_resample(BatchDev* b, cudaStream_t s);
cudaError_t launch_msc_resample(BatchDev* b, int rng_mode, cudaStream_t s);

// SSC populations swept on bit planes (native stream): tiles of G replicas
// packed to one bit per site in shared memory, a sublattice row as Wr words
// of `seg` sites (several replicas' rows per word when a row is at most 16
// sites).  False where L has no such layout.  Replicas per tile: `tile` if
// given (the largest tile for L halved k times, else false), else the
// largest such tile that still leaves a tile for each of `slots` resident
// CTAs given the batch's replicas, else the largest tile (about 1024 words
// per plane).
bool ssc_bits_geom(int L, SweepGeom* g, int tile = 0, long long replicas = 0, int slots = 0);
// Fraction of the bits of the packed words that hold sites (1 at L = 16, 32,
// 64, 128, 256; 0.75 at L = 24, 48, 96; 0 where no bit-plane layout exists).
double ssc_bits_fill(int L);
cudaError_t ssc_bits_setup(int smem, SweepLaunch* out);
cudaError_t launch_ssc_bits_sweep(BatchDev* b, int energy_only, unsigned long long seed, const SweepLaunch& sl,
                                  cudaStream_t s);

// MSC sweep by thread-block clusters of cs = 2 or 4 CTAs (one horizontal
// stripe of the group per CTA), for lattices too large for one CTA.
bool msc_cluster_geom(int L, int cs, int threads, SweepGeom* g);
int msc_cluster_threads(int cs, int maxL);
cudaError_t msc_cluster_setup(int cs, int threads, int rng_mode, int smem, SweepLaunch* out);
cudaError_t launch_msc_cluster_sweep(int cs, int threads, BatchDev* b, int rng_mode, int energy_only, unsigned long long seed,
                                     const SweepLaunch& sl, cudaStream_t s);

// Per-run / per-step bookkeeping.
cudaError_t launch_begin_run(PopDev* pops, int npop, cudaStream_t s);
cudaError_t launch_finish_step(PopDev* pops, int npop, cudaStream_t s);
// After a graph run's last sweep, where the fused resampling left the rows raw.
cudaError_t launch_finish_rows(PopDev* pops, int npop, cudaStream_t s);
// Populations with records or family statistics: histogram, energy ring and
// family counts of the temperature just finished (after launch_finish_step);
// `blocks` from res_blocks().
cudaError_t launch_record(PopDev* pops, int npop, int blocks, cudaStream_t s);
// Family statistics: ancestors set at the initial population, carried by
// each resampling (MSC, native stream: in launch_resample; else after it),
// counted by launch_record and summed by launch_family_stats.
cudaError_t launch_clnc(double* table, cudaStream_t s);  // c ln c of family sizes (kClncTable), once per handle
cudaError_t launch_family_init(PopDev* pops, int npop, int blocks, cudaStream_t s);
cudaError_t launch_family_resample(PopDev* pops, int npop, int blocks, cudaStream_t s);
cudaError_t launch_family_stats(PopDev* pops, int npop, int blocks, cudaStream_t s);
// Adaptive populations: choose the next temperature (after launch_finish_step).
cudaError_t launch_adapt(PopDev* pops, int npop, cudaStream_t s);

}  // namespace pa
