// pa_ssc.cu -- single-spin coding (one int8 +-1 per site).
//
// Replaces, from the reference PAisingSSC.cu:
//   ReplicaInit   (PAisingSSC.cu:150-157)  -> ssc_init_kernel
//   checkKerALL   (PAisingSSC.cu:159-193)  -> ssc_sweep_kernel (all sweeps of a
//   energyKer     (PAisingSSC.cu:195-215)     replica in shared memory, energy
//                                             and magnetisation fused at the end)
//   resampleKer   (PAisingSSC.cu:272-280)  -> ssc_resample_kernel (gather into
//                                             the other half of a double buffer)
//
// Layout in HBM: replica r occupies N bytes at spins + r*N, sublattice A
// (sites with x+y even) first, then B; inside a sublattice, site (x, y) is at
// idx = y*L/2 + x/2, the reference's checkerboard index (PAisingSSC.cu:169).
#include <climits>

#include <type_traits>

#include "pa_device.cuh"
#include "pa_kernels.h"
#include "pa_units.cuh"

namespace pa {

namespace {

constexpr uint32_t kLsb = 0x01010101u;

__device__ __forceinline__ uint32_t minus_bits(uint32_t w) { return (w >> 1) & kLsb; }  // 1 per byte == -1

// per-replica statistics kept by thread 0 of a sweep CTA until the CTA moves
// to another population or finishes
struct StatAcc {
  long long sE, sE2, sM, sM2;
  U128 m4;
  int emin;
  __device__ void reset() {
    sE = sE2 = sM = sM2 = 0;
    m4 = U128{0, 0};
    emin = INT_MAX;
  }
  __device__ void add(int e, int m) {
    const long long am = m < 0 ? -(long long)m : (long long)m;
    sE += e;
    sE2 += (long long)e * e;
    sM += am;
    sM2 += am * am;
    unsigned long long lo, hi;
    m4_of(m, lo, hi);
    u128_add(m4, lo, hi);
    emin = e < emin ? e : emin;
  }
  __device__ void flush(PopDev* st) const {
    if (emin == INT_MAX) return;
    atomicAdd((unsigned long long*)&st->sE, (unsigned long long)sE);
    atomicAdd((unsigned long long*)&st->sE2, (unsigned long long)sE2);
    atomicAdd((unsigned long long*)&st->sM, (unsigned long long)sM);
    atomicAdd((unsigned long long*)&st->sM2, (unsigned long long)sM2);
    u128_atomic_add(&st->sM4lo, &st->sM4hi, m4.lo, m4.hi);
    atomicMin(&st->Emin_acc, emin);
  }
};

}  // namespace

// ------------------------------------------------------------------ init
// ReplicaInit (PAisingSSC.cu:150-157): reference thread t of block B draws,
// for its k-th site idx = t + 128k, uniform number 2k for gA[idx] and 2k+1
// for gB[idx] from subsequence iseq + t + 128 B; spin = +1 iff U >= 0.5.
__global__ void ssc_init_kernel(PopDev* pops) {
  PopDev* st = pops + blockIdx.y;
  const int N = st->N, h = N >> 1, R = st->R_cur;
  const unsigned long long seed = st->seed, iseq = st->iseq;
  int8_t* sp = (int8_t*)st->spins[st->parity];
  if (st->init_src) {  // caller-supplied population: copy, 16 bytes per thread
    const uint4* src = (const uint4*)st->init_src;
    uint4* dst = (uint4*)sp;
    const long long nv = (long long)R * N / 16;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x)
      dst[v] = src[v];
    return;
  }
  const long long total = (long long)R * h;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e / h), idx = (int)(e - (long long)r * h);
    const int t = idx & (kRefThreads - 1), k = idx >> 7;
    const unsigned long long sub = iseq + (unsigned long long)t + (unsigned long long)kRefThreads * r;
    sp[(size_t)r * N + idx] = ref_uniform(ref_word(seed, sub, 2ull * k)) >= 0.5 ? 1 : -1;
    sp[(size_t)r * N + h + idx] = ref_uniform(ref_word(seed, sub, 2ull * k + 1)) >= 0.5 ? 1 : -1;
  }
}

// ----------------------------------------------------------------- sweep
// Persistent: every CTA takes replicas of any population from the batch's
// work queue and anneals one replica at a time, the whole lattice resident in
// shared memory as 32-bit words of 4 int8 spins.  Thread (rsub, cw) owns word
// column cw of sublattice rows rsub, rsub+rpp, ...
//
// MODE kRefCoords reproduces checkKerALL's decisions exactly: site idx of
// replica r, sweep sw, half-sweep hf uses draw
//     ctr = sw*2K + hf*K + k   of subsequence  iseq + t + 128 r,
// t = idx mod 128, k = idx div 128, K = draws per reference thread per half
// sweep, and flips iff (H+1)/2^32 < boltz[idxT0 + 2 idxT1], evaluated as the
// integer test H < thr10[...] with thr10 = ceil(2^32 p) - 1 (exact).
// MODE kNative flips iff dE <= 0 or U < T = ceil(2^32 exp(-beta dE)) for a
// uniform 32-bit U, decided one byte at a time: U's top byte b against T's
// top byte t settles the test unless b == t (probability 1/256), and only
// then are U's low 24 bits drawn and compared with T's.  One Philox4x32-10
// block serves two words (8 sites): words x, y give the top bytes, z, w the
// low bits of up to two undecided sites; more than two take another block.
// Each site's acceptance probability is exactly T / 2^32.
template <int MODE>
__global__ void __launch_bounds__(kSweepThreads, 4)
    ssc_sweep_kernel(BatchDev* b, int energy_only, unsigned long long stream_seed, int nsm) {
  extern __shared__ __align__(16) uint32_t lat[];  // N/4 words: A then B
  __shared__ uint32_t s_thr[16];
  __shared__ int s_unit, s_pop;
  __shared__ int s_red[2][33];

  const int tid = threadIdx.x;
  const int total = b->unit_prefix[b->npop];
  int cur = -1;
  PopDev* st = nullptr;
  int L = 0, N = 0, h = 0, Wr = 1, hw = 0, rpp = 1, kconst = 0, step = 0, sweeps = 0;
  uint32_t nstep = 0;  // counter word 2 of the native stream
  unsigned long long seed = 0, iseq = 0;
  // native stream key: one seed for the whole batch; populations differ in counter word 3
  const PhiloxKeys keys(stream_seed);
  uint32_t tag = 0;
  int8_t* spins = nullptr;
  bool worker = false;
  int cw = 0, rsub = 0, cwl = 0, cwr = 0;
  StatAcc acc;
  acc.reset();

  for (;;) {
    __syncthreads();
    if (tid == 0) {
      const int u = cur < 0 ? first_unit(b, nsm, total) : later_unit(b, gridDim.x);
      int loc = 0;
      s_pop = u < total ? queue_pop(b, u, &loc) : -1;
      s_unit = loc;
    }
    __syncthreads();
    const int p = s_pop, r = s_unit;
    if (p < 0) break;
    if (p != cur) {  // block-uniform: load the population's parameters
      if (tid == 0 && st) {
        acc.flush(st);
        acc.reset();
      }
      cur = p;
      st = b->pops + p;
      L = st->L; N = st->N; h = N >> 1; hw = h >> 2; Wr = st->Wr; rpp = st->rpp; kconst = st->kconst;
      step = st->step;
      nstep = native_step_word(st);
      sweeps = energy_only ? 0 : st->sweeps;
      seed = st->seed;
      tag = kTagSscSweep | (uint32_t)st->pop_id;
      // draws consumed by the resampling of this step come before the sweep's
      iseq = st->iseq + (step > 0 ? (unsigned long long)st->R_prev : 0ull);
      spins = (int8_t*)st->spins[st->parity];
      worker = tid < st->T;
      cw = worker ? tid % Wr : 0;
      rsub = worker ? tid / Wr : 0;
      cwl = (cw == 0 ? Wr - 1 : cw - 1);
      cwr = (cw + 1 == Wr ? 0 : cw + 1);
      if (tid < kThrPerStep) s_thr[tid] = st->thr[(size_t)step * kThrPerStep + tid];
    }
    const uint4* gsrc = (const uint4*)(spins + (size_t)r * N);
    uint4* lat4 = (uint4*)lat;
    for (int v = tid; v < (N >> 4); v += blockDim.x) lat4[v] = gsrc[v];
    __syncthreads();

    // native stream, one Philox block (one or two words of 4 sites, rpp rows
    // apart): the site's number is the first word's in the population
    struct HalfKeys {
      uint32_t c1;
      uint2 uni;
    };
    auto half_keys = [&](int sw, int hf) {
      const uint32_t c1 = (uint32_t)(sw * 2 + hf) * 2u;
      return HalfKeys{c1, philox_uniform(c1, nstep, keys)};
    };
    // twice the anti-parallel neighbour count (0..4) of each of the 4 sites of
    // a word: +-1 bytes that differ do so in bit 1
    auto count2 = [](uint32_t s, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
      constexpr uint32_t m = 0x02020202u;
      return (((s ^ a) & m) + ((s ^ b) & m)) + (((s ^ c) & m) + ((s ^ d) & m));
    };
    // of word (ty, cw); the horizontal neighbour that is not at the same idx is
    // x-1 for A on even rows and B on odd rows, x+1 otherwise (PAisingSSC.cu:170,182)
    auto anti2 = [&](int ty, const uint32_t* oth, uint32_t s, int hf_) {
      const int row = ty * Wr, rowu = (ty == 0 ? L - 1 : ty - 1) * Wr, rowd = (ty + 1 == L ? 0 : ty + 1) * Wr;
      const uint32_t o = oth[row + cw];
      const bool left = (hf_ == 0) == ((ty & 1) == 0);
      const uint32_t oside = __byte_perm(o, oth[row + (left ? cwl : cwr)], left ? 0x2107 : 0x4321);
      return count2(s, o, oside, oth[rowu + cw], oth[rowd + cw]);
    };
    const uint32_t T4 = s_thr[10], T8 = s_thr[11], t4b = (T4 >> 24) * kLsb, t8b = (T8 >> 24) * kLsb;
    // flip[q] = 0xFE in the bytes of word q's sites that flip
    auto decide = [&](auto nw_c, const uint32_t (&na)[2], uint32_t site, uint2 pre, const HalfKeys& hk,
                      uint32_t (&flip)[2]) {
      constexpr int NW = decltype(nw_c)::value;
      constexpr uint32_t kMsbs = 0x80808080u;
      const U4 rn = philox10_prefixed(site, pre, hk.uni, keys);
      uint32_t strag[2] = {0u, 0u}, fl[2] = {0u, 0u};
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        const uint32_t x = q ? rn.y : rn.x;
        const uint32_t sure = (na[q] >> 2 | na[q] >> 3) & kLsb;    // two or more: flips
        const uint32_t one = (na[q] >> 1 & ~sure & kLsb) * 0xFFu;  // exactly one: T4, else T8
        const uint32_t tb = (t4b & one) | (t8b & ~one);            // T's top byte per site
        const uint32_t d = (x | kMsbs) - (tb & ~kMsbs), z = x ^ tb;
        const uint32_t lt = (~x & tb) | (~z & ~d);                // bytes x < tb (bit 7)
        const uint32_t ne = ((z & ~kMsbs) + ~kMsbs) | z;          // bytes x != tb (bit 7)
        fl[q] = (lt >> 7 & kLsb) | sure;
        strag[q] = ~(ne >> 7) & ~sure & kLsb;                     // top bytes equal: undecided
      }
      if (strag[0] | strag[1]) {  // probability ~ 2/256 per site needing a decision
        // the undecided sites in order; their low 24 bits come from rn.z, rn.w,
        // then from further blocks, four words each
        uint32_t a0 = rn.z, a1 = rn.w, a2 = 0u, a3 = 0u;
        int used = 0;
#pragma unroll 1
        while (strag[0] | strag[1]) {
          const bool q = NW > 1 && strag[0] == 0u;
          const uint32_t m = q ? strag[1] : strag[0], bit = m & (0u - m);
          strag[0] = q ? 0u : m ^ bit;
          if (q) strag[1] = m ^ bit;
          if (used == 2 || used == 6) {
            const U4 x = philox10k(site, hk.c1 + 1u, nstep, tag | ((uint32_t)(used >> 2) << 12), keys);
            a0 = x.x; a1 = x.y; a2 = x.z; a3 = x.w;
          }
          const uint32_t T = ((q ? na[1] : na[0]) >> 1 & bit) ? T4 : T8;  // undecided: no or one anti-parallel
          const uint32_t take = (a0 & 0xFFFFFFu) < (T & 0xFFFFFFu) ? bit : 0u;
          fl[0] |= q ? 0u : take;
          if (NW > 1) fl[1] |= q ? take : 0u;
          a0 = a1; a1 = a2; a2 = a3;
          ++used;
        }
      }
#pragma unroll
      for (int q = 0; q < NW; ++q) flip[q] = fl[q] * 0xFEu;
    };
    // One block per thread and half-sweep (one word up to L = 40, two up to 64):
    // addresses, sides and the block's first rounds stay in registers, a single
    // word pays for one, and warps without words leave the others' barriers.
    // Instruction issue bounds the sweep (a block's ten rounds are about half of
    // it): L = 40, 10000 replicas, 20 sweeps 347 -> 519 attempts/ns (with the
    // byte tests of decide in place of the SIMD intrinsics, which alone gave the
    // general form below 1.17-1.2x: L = 128 688 -> 827), L = 16 155 -> 258,
    // L = 64 656 -> 813.
    auto one_block = [&](auto nw_c) {
      constexpr int NW = decltype(nw_c)::value;
      const int threads = (Wr * rpp + 31) & ~31;  // whole warps that hold words
      if (tid >= threads) return;
      int at[2], up[2], dn[2], sideA[2], sideB[2];
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        const int ty = rsub + q * rpp, row = ty * Wr;
        at[q] = row + cw;
        up[q] = (ty == 0 ? L - 1 : ty - 1) * Wr + cw;
        dn[q] = (ty + 1 == L ? 0 : ty + 1) * Wr + cw;
        sideA[q] = row + (ty & 1 ? cwr : cwl);
        sideB[q] = row + (ty & 1 ? cwl : cwr);
      }
      const uint32_t site = (uint32_t)(r * hw + at[0]);
      const uint2 pre = philox_prefix(site, nstep, tag, keys);
      const bool odd = rsub & 1, odd1 = (rsub + rpp) & 1;
      for (int sw = 0; sw < sweeps; ++sw) {
#pragma unroll 1
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t* self = lat + (hf ? hw : 0);
          const uint32_t* oth = lat + (hf ? 0 : hw);
          const HalfKeys hk = half_keys(sw, hf);
          uint32_t sp[2], na[2] = {0u, 0u}, flip[2];
#pragma unroll
          for (int q = 0; q < NW; ++q) {
            const bool left = (hf == 0) != (q ? odd1 : odd);
            const uint32_t o = oth[at[q]];
            sp[q] = self[at[q]];
            na[q] = count2(sp[q], o, __byte_perm(o, oth[hf ? sideB[q] : sideA[q]], left ? 0x2107 : 0x4321), oth[up[q]], oth[dn[q]]);
          }
          decide(nw_c, na, site, pre, hk, flip);
          if (worker)
#pragma unroll
            for (int q = 0; q < NW; ++q) self[at[q]] = sp[q] ^ flip[q];
          asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
        }
      }
    };
    const int npass = L / rpp;  // rpp divides L
    const bool single = MODE == kNative && npass <= 2;
    if constexpr (MODE == kNative) {
      if (single) {
        if (npass == 1) one_block(std::integral_constant<int, 1>());
        else one_block(std::integral_constant<int, 2>());
        __syncthreads();
      }
    }
    for (int sw = 0; !single && sw < sweeps; ++sw) {
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t* self = lat + (hf ? hw : 0);
        const uint32_t* oth = lat + (hf ? 0 : hw);
        if (worker && MODE == kNative) {
          const HalfKeys hk = half_keys(sw, hf);
          for (int ty0 = rsub; ty0 < L; ty0 += 2 * rpp) {
            const int ty1 = ty0 + rpp;
            const bool two = ty1 < L;
            const int w0 = ty0 * Wr + cw, w1 = two ? ty1 * Wr + cw : w0;
            const uint32_t sp[2] = {self[w0], self[w1]};
            const uint32_t na[2] = {anti2(ty0, oth, sp[0], hf), two ? anti2(ty1, oth, sp[1], hf) : 0x04040404u};
            uint32_t flip[2];
            const uint32_t site = (uint32_t)(r * hw + w0);
            decide(std::integral_constant<int, 2>(), na, site, philox_prefix(site, nstep, tag, keys), hk, flip);
            self[w0] = sp[0] ^ flip[0];
            if (two) self[w1] = sp[1] ^ flip[1];
          }
        }
        if (worker && MODE == kRefCoords) {
          for (int ty = rsub; ty < L; ty += rpp) {
            const int row = ty * Wr, rowu = (ty == 0 ? L - 1 : ty - 1) * Wr, rowd = (ty + 1 == L ? 0 : ty + 1) * Wr;
            const int w = row + cw;
            const uint32_t s = self[w];
            const uint32_t o = oth[w];
            const bool left = (hf == 0) == ((ty & 1) == 0);
            const uint32_t oside = left ? __byte_perm(oth[row + cwl], o, 0x6543) : __byte_perm(o, oth[row + cwr], 0x4321);
            const uint32_t ou = oth[rowu + cw], od = oth[rowd + cw];
            uint32_t flip = 0;
            {
              const uint32_t nminus = minus_bits(o) + minus_bits(oside) + minus_bits(ou) + minus_bits(od);
              // idxT0 + 2 idxT1 = (1 - s_minus) + 2 (4 - n_minus) per byte
              const uint32_t tix = 0x09090909u - minus_bits(s) - (nminus << 1);
              const int idx0 = ty * (h / L) + cw * 4;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int idx = idx0 + j, t = idx & (kRefThreads - 1), k = idx >> 7;
                const int K = kconst ? kconst : (t < h ? (h - t + kRefThreads - 1) / kRefThreads : 0);
                const unsigned long long sub = iseq + (unsigned long long)t + (unsigned long long)kRefThreads * r;
                const unsigned long long ctr = (unsigned long long)sw * 2 * K + (unsigned long long)hf * K + k;
                const uint32_t u = ref_word(seed, sub, ctr);
                if (u < s_thr[(tix >> (8 * j)) & 0xFFu]) flip |= 0xFEu << (8 * j);
              }
            }
            self[w] = s ^ flip;
          }
        }
        __syncthreads();
      }
    }

    // energy: every bond joins one A and one B site, so E = -sum_A s_A sum_nn s_B
    // = -2N + 2 * (number of anti-parallel bonds seen from A); M = N - 2 #minus.
    int anti = 0, nminus = 0;
    if (worker) {
      for (int ty = rsub; ty < L; ty += rpp) {
        const int row = ty * Wr, rowu = (ty == 0 ? L - 1 : ty - 1) * Wr, rowd = (ty + 1 == L ? 0 : ty + 1) * Wr;
        const int w = row + cw;
        const uint32_t s = lat[w], o = lat[hw + w];
        const bool left = (ty & 1) == 0;
        const uint32_t oside = left ? __byte_perm(lat[hw + row + cwl], o, 0x6543) : __byte_perm(o, lat[hw + row + cwr], 0x4321);
        const uint32_t na = ((s ^ o) >> 1 & kLsb) + ((s ^ oside) >> 1 & kLsb) + ((s ^ lat[hw + rowu + cw]) >> 1 & kLsb) +
                            ((s ^ lat[hw + rowd + cw]) >> 1 & kLsb);
        anti += (int)((na * kLsb) >> 24);
        nminus += __popc(minus_bits(s)) + __popc(minus_bits(o));
      }
    }
    anti = warp_sum(anti);
    nminus = warp_sum(nminus);
    if ((tid & 31) == 0) { s_red[0][tid >> 5] = anti; s_red[1][tid >> 5] = nminus; }
    // write the lattice back while the reduction completes
    uint4* gdst = (uint4*)(spins + (size_t)r * N);
    __syncthreads();
    for (int v = tid; v < (N >> 4); v += blockDim.x) gdst[v] = lat4[v];
    if (tid == 0) {
      int a = 0, m = 0;
      for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { a += s_red[0][i]; m += s_red[1][i]; }
      const int E = -2 * N + 2 * a, Mg = N - 2 * m;
      st->E[r] = E;
      st->M[r] = Mg;
      acc.add(E, Mg);
    }
  }
  if (tid == 0 && st) acc.flush(st);
}

// -------------------------------------------------------------- resample
// Gather form of resampleKer: new replica s copies old replica src[s].
//
// Units (ssc_units) of all populations of the batch come from one queue and
// are taken by persistent CTAs, so a batch of
// uneven populations keeps every SM copying until the last unit; each thread
// issues all its loads of a unit before its stores.
constexpr int kSscResBlocksPerSM = 4;  // 64 registers

__global__ void __launch_bounds__(kSscResThreads, kSscResBlocksPerSM) ssc_resample_kernel(BatchDev* b) {
  __shared__ int s_u[2];  // this unit and the next one (taken ahead by thread 0)
  const int tid = threadIdx.x, total = b->res_prefix[b->npop];
  if (tid == 0) s_u[0] = (int)atomicAdd(&b->res_next, 1u);
  __syncthreads();
  for (int it = 0;; ++it) {
    const int u = s_u[it & 1];
    if (u >= total) break;  // block-uniform
    if (tid == 0) s_u[(it + 1) & 1] = (int)atomicAdd(&b->res_next, 1u);
    int lo = 0, hi = b->npop;  // population of unit u
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (b->res_prefix[mid] <= u) lo = mid;
      else hi = mid;
    }
    const PopDev* st = b->pops + lo;
    const int nv = st->N >> 4, Rn = st->R_cur, loc = u - b->res_prefix[lo];
    const uint4* old = (const uint4*)st->spins[st->parity ^ 1];
    uint4* neu = (uint4*)st->spins[st->parity];
    const uint32_t* src = st->src;
    // the unit as replicas [s0, s0 + ns) x vectors [j0, j0 + nj) of each
    int s0, ns, j0, nj;
    if (nv > kSscUnitVecs) {
      const int upr = (nv + kSscUnitVecs - 1) / kSscUnitVecs, part = loc % upr;
      s0 = loc / upr;
      ns = 1;
      j0 = part * kSscUnitVecs;
      nj = min(kSscUnitVecs, nv - j0);
    } else {
      const int rpu = kSscUnitVecs / nv;
      s0 = loc * rpu;
      ns = min(rpu, Rn - s0);
      j0 = 0;
      nj = nv;
    }
    const int n = ns * nj;                     // vectors in the unit (<= kSscUnitVecs)
    const uint32_t inv = 0xffffffffu / (uint32_t)nj + 1u;  // n / nj by __umulhi: n * nj < 2^32
    // vector i of the unit is vector j0 + i % nj of new replica s0 + i / nj
    auto at = [&](int i, int& s) {
      const int q = ns == 1 ? 0 : (int)__umulhi((uint32_t)i, inv);
      s = s0 + q;
      return j0 + i - q * nj;
    };
    uint4 r[kSscVecsPerThread];
#pragma unroll
    for (int k = 0; k < kSscVecsPerThread; ++k) {
      const int i = tid + k * kSscResThreads;
      if (i < n) {
        int s;
        const int j = at(i, s);
        r[k] = __ldg(old + (size_t)src[s] * nv + j);
      }
    }
#pragma unroll
    for (int k = 0; k < kSscVecsPerThread; ++k) {
      const int i = tid + k * kSscResThreads;
      if (i < n) {
        int s;
        const int j = at(i, s);
        neu[(size_t)s * nv + j] = r[k];
      }
    }
    __syncthreads();  // s_u[(it + 1) & 1] is visible; s_u[it & 1] may be overwritten
  }
}

// -------------------------------------------------------------- geometry
static int pick_rpp(int L, int Wr) {
  int best = 1;
  for (int r = 1; r <= L; ++r)
    if (L % r == 0 && Wr * r <= kSweepThreads) best = r;
  return best;
}

bool ssc_geom(int L, SweepGeom* g) {
  if (L < 8 || L % 8 != 0 || L > 256) return false;
  g->L = L;
  g->N = L * L;
  g->half = g->N / 2;
  g->Wr = L / 8;
  g->rpp = pick_rpp(L, g->Wr);
  g->T = g->Wr * g->rpp;
  g->npass = (L + g->rpp - 1) / g->rpp;
  g->kconst = (g->half % kRefThreads == 0) ? g->half / kRefThreads : 0;
  g->smem = g->N;
  return true;
}

// -------------------------------------------------------------- launchers
static const void* ssc_sweep_fn(int rng_mode) {
  return rng_mode == kRefCoords ? (const void*)ssc_sweep_kernel<kRefCoords> : (const void*)ssc_sweep_kernel<kNative>;
}

cudaError_t ssc_sweep_setup(int rng_mode, int smem, SweepLaunch* out) {
  return persistent_launch(ssc_sweep_fn(rng_mode), kSweepThreads, smem, out);
}

cudaError_t launch_ssc_sweep(BatchDev* b, int rng_mode, int energy_only, unsigned long long seed,
                             const SweepLaunch& sl, cudaStream_t s) {
  if (rng_mode == kRefCoords)
    ssc_sweep_kernel<kRefCoords><<<sl.grid, sl.block, sl.smem, s>>>(b, energy_only, seed, sl.nsm);
  else
    ssc_sweep_kernel<kNative><<<sl.grid, sl.block, sl.smem, s>>>(b, energy_only, seed, sl.nsm);
  return cudaGetLastError();
}

cudaError_t launch_ssc_init(PopDev* pops, int npop, cudaStream_t s) {
  ssc_init_kernel<<<dim3(512, npop), 256, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_ssc_resample(BatchDev* b, cudaStream_t s) {
  int dev, nsm;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  ssc_resample_kernel<<<nsm * kSscResBlocksPerSM, kSscResThreads, 0, s>>>(b);  // persistent CTAs
  return cudaGetLastError();
}

}  // namespace pa
