// pa_stages.cu -- stage entry points of the C ABI: one reference kernel (or
// kernel group) each, on caller-owned device buffers.  They run the same
// kernels as the engine on a batch of one population whose PopDev describes
// the caller's buffers; that descriptor, the reductions' partial sums and the
// MSC gather's pair lists live in scratch device memory held for the duration
// of the call (Scratch).
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/paising.h"
#include "pa_device.cuh"
#include "pa_error.h"
#include "pa_kernels.h"
#include "pa_thresholds.h"
#include "pa_units.cuh"

using namespace pa;

namespace {

int stage_fail(cudaError_t e, const char* what) {
  pa::g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
  return PA_ERR_CUDA;
}

// Device scratch of one stage call: one of kSlots slots of the library's own
// device memory, so that a call makes no cudaMalloc, no cudaFree (which waits
// for the whole device) and no copy from pageable memory; these took 190 us of
// every call.  A slot belongs to one call at a time, from any thread and for
// any stream: the call takes it, enqueues its work and gives it back after its
// stream has been waited for.  Calls beyond the slots allocate their own.  The
// array's address is looked up on the current device each time, so it stays
// right when a context is made anew.
constexpr int kPairGroups = 4096;  // new groups whose pair lists a slot holds: larger gathers go chunk by chunk
// Chunks of a gather at most: the launches of one take about 16 us more than its
// share of one gather of all groups, an allocation for them all 190.
constexpr int kChunksMax = 12;
constexpr size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kOffSt = up256(sizeof(BatchDev)), kOffBetas = kOffSt + up256(sizeof(PopDev)), kOffThr = kOffBetas + 256,
                 kOffBlk = kOffThr + up256(2 * kThrPerStep * 4), kOffQd = kOffBlk + up256(2 * kResBlocksMax * 4),
                 kOffQf = kOffQd + up256(kResBlocksMax * 8), kOffCnt = kOffQf + up256(2 * kResBlocksMax * 4),
                 kOffPairs = kOffCnt + up256(kPairGroups * 4), kSlotBytes = kOffPairs + kPairGroups * kMsb * sizeof(uint2);
constexpr int kSlots = 4, kMaxDevices = 64;

__device__ __align__(256) unsigned char g_stage_slots[kSlots][kSlotBytes];  // 4.4 MB

struct SlotPool {
  std::mutex m;
  bool busy[kMaxDevices][kSlots] = {};
};
SlotPool g_slots;

struct Scratch {
  BatchDev* b = nullptr;
  PopDev* st = nullptr;
  double* betas = nullptr;
  uint32_t* thr = nullptr;
  uint32_t* blk = nullptr;  // blk_tot | blk_off
  double* qd = nullptr;
  float* qf = nullptr;
  uint32_t* cnt = nullptr;
  uint2* pairs = nullptr;
  cudaStream_t stream;
  void* base = nullptr;  // allocated for this call
  void* lists = nullptr;  // and the pair lists of a gather of many chunks
  int dev = -1, slot = -1;
  bool waited = false;  // the stream has been waited for since the last launch

  explicit Scratch(cudaStream_t s) : stream(s) {}
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  cudaError_t alloc() {
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < kMaxDevices) {
      std::lock_guard<std::mutex> g(g_slots.m);
      for (int i = 0; i < kSlots && slot < 0; ++i)
        if (!g_slots.busy[dev][i]) {
          g_slots.busy[dev][i] = true;
          slot = i;
        }
    }
    void* at = nullptr;
    if (slot >= 0) {
      if ((e = cudaGetSymbolAddress(&at, g_stage_slots)) != cudaSuccess) return e;
      at = (char*)at + (size_t)slot * kSlotBytes;
    } else {
      if ((e = cudaMalloc(&base, kSlotBytes)) != cudaSuccess) return e;
      at = base;
    }
    char* p = (char*)at;
    b = (BatchDev*)p;
    st = (PopDev*)(p + kOffSt);
    betas = (double*)(p + kOffBetas);
    thr = (uint32_t*)(p + kOffThr);
    blk = (uint32_t*)(p + kOffBlk);
    qd = (double*)(p + kOffQd);
    qf = (float*)(p + kOffQf);
    cnt = (uint32_t*)(p + kOffCnt);
    pairs = (uint2*)(p + kOffPairs);
    waited = true;  // nothing enqueued yet
    return cudaSuccess;
  }
  // Counts and pair lists of `groups` groups in memory of the call's own; false
  // where there is none (the slot's then serve, chunk by chunk).
  bool own_lists(size_t groups) {
    const size_t cnt_bytes = up256(groups * 4);
    if (cudaMalloc(&lists, cnt_bytes + groups * kMsb * sizeof(uint2)) != cudaSuccess) {
      cudaGetLastError();
      lists = nullptr;
      return false;
    }
    cnt = (uint32_t*)lists;
    pairs = (uint2*)((char*)lists + cnt_bytes);
    return true;
  }
  ~Scratch() {
    if (!waited) cudaStreamSynchronize(stream);  // a call that failed half way
    if (lists) cudaFree(lists);
    if (base) cudaFree(base);
    if (slot >= 0) {
      std::lock_guard<std::mutex> g(g_slots.m);
      g_slots.busy[dev][slot] = false;
    }
  }
};

// What a call sets up, passed as a kernel parameter: no copy from the host.
struct StageSetup {
  PopDev h;
  double betas[2];
  uint32_t thr[2 * kThrPerStep];
};
static_assert(sizeof(StageSetup) < 4000 && sizeof(PopDev) % 8 == 0, "kernel parameter");

// The call's descriptor, its schedule of one step and its work plan (one warp).
__global__ void __launch_bounds__(32) stage_setup_kernel(BatchDev* b, PopDev* st, double* betas, uint32_t* thr,
                                                         const __grid_constant__ StageSetup a) {
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&a.h);
  for (int i = threadIdx.x; i < (int)(sizeof(PopDev) / 8); i += 32)
    reinterpret_cast<unsigned long long*>(st)[i] = src[i];
  if (threadIdx.x < 2) betas[threadIdx.x] = a.betas[threadIdx.x];
  if (threadIdx.x < 2 * kThrPerStep) thr[threadIdx.x] = a.thr[threadIdx.x];
  if (threadIdx.x == 0) {
    b->npop = 1;
    b->pops = st;
    b->plan_ticket = 0;
  }
  __threadfence();
  __syncwarp();
  plan_batch(b, 0, nullptr);
}

void fill_thr(double beta, uint32_t* t) { thresholds(beta, t); }

// A one-population state at temperature step 1 of a one-step schedule.
PopDev base_state(int coding, int L) {
  PopDev h;
  std::memset(&h, 0, sizeof(h));
  h.coding = coding;
  h.L = L;
  h.N = L * L;
  h.step = 1;
  h.nsteps = 1;
  h.Emin_acc = 0x7fffffff;
  SweepGeom g;
  if (coding == kMSC ? msc_geom(L, &g) : ssc_geom(L, &g)) geom_to_pop(g, &h);
  return h;
}

int upload(Scratch& S, const PopDev& h, const double* betas, const uint32_t* thr) {
  StageSetup a;
  a.h = h;
  for (int i = 0; i < 2; ++i) a.betas[i] = betas ? betas[i] : 0.0;
  for (int i = 0; i < 2 * kThrPerStep; ++i) a.thr[i] = thr ? thr[i] : 0u;
  S.waited = false;
  stage_setup_kernel<<<1, 32, 0, S.stream>>>(S.b, S.st, S.betas, S.thr, a);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PA_OK : stage_fail(e, "upload");
}

int finish(Scratch& S, cudaError_t e, const char* what) {
  if (e == cudaSuccess) e = cudaStreamSynchronize(S.stream);
  S.waited = e == cudaSuccess;
  return e == cudaSuccess ? PA_OK : stage_fail(e, what);
}

// bits: the SSC bit-plane sweep (native stream only)
int sweep_stage(int coding, void* spins, uint8_t* active, int L, int units, int sweeps, double beta, int rng_mode,
                uint64_t seed, uint64_t iseq, int step, int32_t* E, int32_t* M, void* stream, bool bits = false) {
  cudaStream_t s = (cudaStream_t)stream;
  SweepGeom g;
  if (bits ? !ssc_bits_geom(L, &g) : coding == kMSC ? !msc_geom(L, &g) : !ssc_geom(L, &g)) return PA_ERR_ARG;
  SweepLaunch sl;
  cudaError_t e = bits ? ssc_bits_setup(g.smem, &sl)
                       : sweep_setup(coding, rng_mode, g.smem, &sl,
                                     coding == kMSC && rng_mode == PA_RNG_NATIVE ? msc_kind(g) : kGeneral);
  if (e != cudaSuccess) return stage_fail(e, "sweep setup");
  Scratch S(s);
  if ((e = S.alloc()) != cudaSuccess) return stage_fail(e, "scratch");
  PopDev h = base_state(coding, L);
  h.spins[0] = spins;
  h.active[0] = active;
  h.R_cur = h.Rinit = coding == kMSC ? units * kMsb : units;
  h.sweeps = sweeps;
  h.rng_mode = rng_mode;
  h.seed = seed;
  h.iseq = iseq;
  h.pop_id = step;  // native stream key: the stage call folds (step, population) into pop_id
  h.E = E;
  h.M = M;
  h.betas = S.betas;
  h.thr = S.thr;
  double b[2] = {0.0, beta};
  uint32_t t[2 * kThrPerStep];
  fill_thr(0.0, t);
  fill_thr(beta, t + kThrPerStep);
  if (bits) geom_to_pop(g, &h);
  int rc = upload(S, h, b, t);
  if (rc) return rc;
  e = bits ? launch_ssc_bits_sweep(S.b, 0, seed, sl, s) : launch_sweep(S.b, coding, rng_mode, 0, seed, sl, s);
  return finish(S, e, "sweep");
}

}  // namespace

extern "C" {

int pa_ssc_init(int8_t* spins, int L, int R, uint64_t seed, uint64_t iseq, void* stream) {
  SweepGeom g;
  if (!spins || R < 1 || !ssc_geom(L, &g)) return PA_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Scratch S(s);
  cudaError_t e = S.alloc();
  if (e != cudaSuccess) return stage_fail(e, "scratch");
  PopDev h = base_state(kSSC, L);
  h.spins[0] = spins;
  h.R_cur = h.Rinit = R;
  h.seed = seed;
  h.iseq = iseq;
  int rc = upload(S, h, nullptr, nullptr);
  if (rc) return rc;
  return finish(S, launch_init(S.st, 1, kSSC, s), "ssc_init");
}

int pa_ssc_sweep(int8_t* spins, int L, int R, int sweeps, double beta, int rng_mode, uint64_t seed,
                 uint64_t iseq, int step, int32_t* E, int32_t* M, void* stream) {
  SweepGeom g;
  if (!spins || !E || !M || R < 1 || sweeps < 0 || step < 0 || !ssc_geom(L, &g)) return PA_ERR_ARG;
  if (rng_mode != PA_RNG_NATIVE && rng_mode != PA_RNG_REFERENCE) return PA_ERR_ARG;
  return sweep_stage(kSSC, spins, nullptr, L, R, sweeps, beta, rng_mode, seed, iseq, step, E, M, stream);
}

int pa_ssc_sweep_bits(int8_t* spins, int L, int R, int sweeps, double beta, uint64_t seed, int step, int32_t* E,
                      int32_t* M, void* stream) {
  SweepGeom g;
  if (!spins || !E || !M || R < 1 || sweeps < 0 || step < 0 || !ssc_bits_geom(L, &g)) return PA_ERR_ARG;
  return sweep_stage(kSSC, spins, nullptr, L, R, sweeps, beta, PA_RNG_NATIVE, seed, 0, step, E, M, stream, true);
}

int pa_msc_init(uint32_t* words, uint8_t* active, int L, int R, uint64_t seed, uint64_t iseq, void* stream) {
  SweepGeom g;
  if (!words || !active || R < 1 || !msc_geom(L, &g)) return PA_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Scratch S(s);
  cudaError_t e = S.alloc();
  if (e != cudaSuccess) return stage_fail(e, "scratch");
  PopDev h = base_state(kMSC, L);
  h.spins[0] = words;
  h.active[0] = active;
  h.R_cur = h.Rinit = R;
  h.seed = seed;
  h.iseq = iseq;
  int rc = upload(S, h, nullptr, nullptr);
  if (rc) return rc;
  return finish(S, launch_init(S.st, 1, kMSC, s), "msc_init");
}

int pa_msc_sweep(uint32_t* words, const uint8_t* active, int L, int rg, int sweeps, double beta, int rng_mode,
                 uint64_t seed, uint64_t iseq, int step, int32_t* E, int32_t* M, void* stream) {
  SweepGeom g;
  if (!words || !active || !E || !M || rg < 1 || sweeps < 0 || step < 0 || !msc_geom(L, &g)) return PA_ERR_ARG;
  if (rng_mode != PA_RNG_NATIVE && rng_mode != PA_RNG_REFERENCE) return PA_ERR_ARG;
  return sweep_stage(kMSC, words, const_cast<uint8_t*>(active), L, rg, sweeps, beta, rng_mode, seed, iseq, step, E,
                     M, stream);
}

int pa_resample_plan(const int32_t* E, const uint8_t* active, int coding, int R_prev, int Rinit, int Rcap,
                     double beta_prev, double beta, double e_ref, int weights, uint64_t seed, uint64_t iseq,
                     uint32_t* roff, uint32_t* offs, uint32_t* src, double* out, void* stream) {
  if (!E || !roff || !offs || !src || !out || R_prev < 1 || Rinit < 1 || Rcap < 1) return PA_ERR_ARG;
  if (coding != PA_CODING_SSC && coding != PA_CODING_MSC) return PA_ERR_ARG;
  if (coding == PA_CODING_MSC && !active) return PA_ERR_ARG;
  if (weights != PA_WEIGHTS_FP32 && weights != PA_WEIGHTS_FP64) return PA_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Scratch S(s);
  cudaError_t e = S.alloc();
  if (e != cudaSuccess) return stage_fail(e, "scratch");
  PopDev h = base_state(coding, 8);
  h.Rinit = Rinit;
  h.Rcap = Rcap;
  h.rgcap = (Rcap + kMsb - 1) / kMsb;
  h.R_prev = R_prev;
  h.R_cur = R_prev;
  h.weights = weights;
  h.seed = seed;
  h.iseq = iseq;
  h.Emean = e_ref;
  h.Emin = (int)e_ref;
  h.E = const_cast<int32_t*>(E);
  h.active[0] = h.active[1] = const_cast<uint8_t*>(active);
  h.roff = roff;
  h.offs = offs;
  h.src = src;
  h.blk_tot = S.blk;
  h.blk_off = S.blk + kResBlocksMax;
  h.qpart_d = S.qd;
  h.qpart_f = S.qf;
  h.betas = S.betas;
  const long long units = coding == PA_CODING_MSC ? (long long)((R_prev + kMsb - 1) / kMsb) * kMsb : R_prev;
  const int blocks = res_blocks(units);
  double b[2] = {beta_prev, beta};
  int rc = upload(S, h, b, nullptr);
  if (rc) return rc;
  if (resample_fused(units, weights, 1)) {
    if ((e = launch_resample_fused(S.st, nullptr, 1, units, weights, false, s)) != cudaSuccess) return stage_fail(e, "resample plan");
  } else {
    if ((e = launch_q(S.st, 1, blocks, s)) != cudaSuccess) return stage_fail(e, "q");
    if ((e = launch_copy_numbers(S.st, 1, blocks, s)) != cudaSuccess) return stage_fail(e, "copy numbers");
    if ((e = launch_scatter(S.st, 1, blocks, s)) != cudaSuccess) return stage_fail(e, "scatter");
    if ((e = launch_scatter_heavy(S.st, 1, s)) != cudaSuccess) return stage_fail(e, "scatter");
  }
  PopDev back;
  if ((e = cudaMemcpyAsync(&back, S.st, sizeof(PopDev), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return stage_fail(e, "readback");
  const int rc2 = finish(S, cudaSuccess, "resample plan");
  if (rc2) return rc2;
  out[0] = back.lnQ;
  out[1] = back.q;
  out[2] = back.error ? 0.0 : (double)back.R_cur;
  if (back.error == 1) return PA_ERR_CAPACITY;
  if (back.error == 2) return PA_ERR_EXTINCT;
  return PA_OK;
}

int pa_ssc_resample(const int8_t* old_spins, int L, const uint32_t* src, int R_new, int8_t* new_spins, void* stream) {
  SweepGeom g;
  if (!old_spins || !src || !new_spins || R_new < 1 || !ssc_geom(L, &g)) return PA_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Scratch S(s);
  cudaError_t e = S.alloc();
  if (e != cudaSuccess) return stage_fail(e, "scratch");
  PopDev h = base_state(kSSC, L);
  h.spins[0] = new_spins;
  h.spins[1] = const_cast<int8_t*>(old_spins);
  h.R_cur = R_new;
  h.src = const_cast<uint32_t*>(src);
  int rc = upload(S, h, nullptr, nullptr);
  if (rc) return rc;
  return finish(S, launch_resample(S.b, kSSC, kRefCoords, s), "ssc_resample");
}

int pa_msc_resample(const uint32_t* old_words, int L, const uint32_t* src, int R_new, uint32_t* new_words,
                    uint8_t* new_active, void* stream) {
  SweepGeom g;
  if (!old_words || !src || !new_words || !new_active || R_new < 1 || !msc_geom(L, &g)) return PA_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Scratch S(s);
  cudaError_t e = S.alloc();
  if (e != cudaSuccess) return stage_fail(e, "scratch");
  PopDev h = base_state(kMSC, L);
  h.rng_mode = kRefCoords;
  h.spins[0] = new_words;
  h.spins[1] = const_cast<uint32_t*>(old_words);
  h.active[0] = new_active;
  h.R_cur = R_new;
  h.src = const_cast<uint32_t*>(src);
  int rc = upload(S, h, nullptr, nullptr);
  if (rc) return rc;
  return finish(S, launch_resample(S.b, kMSC, kRefCoords, s), "msc_resample");
}

int pa_msc_resample_native(const uint32_t* old_words, int L, int R_old, const uint32_t* src, int R_new,
                           uint32_t* new_words, uint8_t* new_active, void* stream) {
  SweepGeom g;
  (void)g;
  if (!old_words || !src || !new_words || !new_active || R_old < 1 || R_new < 1 || L < 4 || L % 2 || L > 256)
    return PA_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Scratch S(s);
  cudaError_t e = S.alloc();
  if (e != cudaSuccess) return stage_fail(e, "scratch");
  // chunks of kPairGroups new groups, whose pair lists the scratch holds, or all at once
  const int rg_new = (R_new + kMsb - 1) / kMsb;
  const int chunk = rg_new > kChunksMax * kPairGroups && S.own_lists((size_t)rg_new) ? rg_new : kPairGroups;
  for (int g0 = 0; g0 < rg_new; g0 += chunk) {
    PopDev h = base_state(kMSC, L);
    h.rng_mode = kNative;
    h.spins[0] = new_words + (size_t)g0 * h.N;
    h.spins[1] = const_cast<uint32_t*>(old_words);
    h.active[0] = new_active + (size_t)g0 * kMsb;
    h.rgcap = (R_old + kMsb - 1) / kMsb;  // groups the old buffer holds
    h.R_cur = R_new - g0 * kMsb;
    if (h.R_cur > (long long)chunk * kMsb) h.R_cur = chunk * kMsb;
    h.src = const_cast<uint32_t*>(src) + (size_t)g0 * kMsb;
    h.res_pairs = S.pairs;
    h.res_cnt = S.cnt;
    const int rc = upload(S, h, nullptr, nullptr);
    if (rc) return rc;
    if ((e = launch_resample(S.b, kMSC, kNative, s)) != cudaSuccess) break;
  }
  return finish(S, e, "msc_resample_native");
}

}  // extern "C"
