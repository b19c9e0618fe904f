// pa_msc.cu -- multi-spin coding: 32 replicas bit-packed per uint32 word.
//
// Replaces, from the reference PAisingMSC.cu (MSbits = 32):
//   ReplicaInit  (PAisingMSC.cu:169-188)  -> msc_init_kernel
//   checkKerALL  (PAisingMSC.cu:191-266)  -> msc_sweep_kernel (group resident in
//   energyKer    (PAisingMSC.cu:268-317)     shared memory for all sweeps; per
//                                            replica energy and magnetisation by
//                                            bitsliced counters in the epilogue)
//   resampleKer  (PAisingMSC.cu:397-435)  -> msc_resample_kernel (gather: each new
//                                            word assembles its 32 source bits,
//                                            no atomics, no memset)
//
// Layout in HBM: group g occupies N words at spins + g*N (sublattice A words,
// then B); bit k of a word is replica k of the group, 1 == spin +1.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "pa_kernels.h"
#include "pa_msc_core.cuh"
#include "pa_units.cuh"

namespace pa {

using namespace msc;

// ------------------------------------------------------------------ init
__global__ void msc_init_kernel(PopDev* pops) {
  PopDev* st = pops + blockIdx.y;
  const int N = st->N, h = N >> 1, R = st->R_cur, rg = (R + kMsb - 1) / kMsb;
  const unsigned long long seed = st->seed, iseq = st->iseq;
  uint32_t* wd = (uint32_t*)st->spins[st->parity];
  uint8_t* act = st->active[st->parity];
  if (st->init_src) {  // caller-supplied population (replica 32g+k at group g, bit k)
    const uint4* src = (const uint4*)st->init_src;
    uint4* dst = (uint4*)wd;
    const long long nv = (long long)rg * N / 4;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x)
      dst[v] = src[v];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)rg * kMsb;
         i += (long long)gridDim.x * blockDim.x)
      act[i] = i < R;
    return;
  }
  // ReplicaInit (PAisingMSC.cu:169-188): reference thread t of block B draws
  // words 2k (gA) and 2k+1 (gB) of subsequence iseq + t + 128 B for idx = t + 128 k
  const long long total = (long long)rg * h;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int g = (int)(e / h), idx = (int)(e - (long long)g * h);
    const int t = idx & (kRefThreads - 1), k = idx >> 7;
    const unsigned long long sub = iseq + (unsigned long long)t + (unsigned long long)kRefThreads * g;
    wd[(size_t)g * N + idx] = ref_word(seed, sub, 2ull * k);
    wd[(size_t)g * N + h + idx] = ref_word(seed, sub, 2ull * k + 1);
    if (idx < kMsb) act[g * kMsb + idx] = (g * kMsb + idx) < R;
  }
}

// ----------------------------------------------------------------- sweep
// Persistent: every CTA takes tiles of G groups of 32 replicas of any
// population from the batch's work queue and anneals one tile at a time,
// resident in shared memory as all G sublattices A, then all G sublattices B
// (so the tile is one stack of G*L sublattice rows of Wr words; a row's
// vertical neighbours wrap inside its own group).  Thread (rsub, tx) owns
// word column tx of stacked rows rsub, rsub+rpp, ...; with one group per
// tile (G = 1) in the native stream it owns the consecutive rows
// rsub*npass .. rsub*npass + npass - 1 instead, and each sublattice carries
// periodic copies of rows -1 and L (msc_move_tile), so that a batch of four
// rows shares its six rows of the other sublattice and nothing wraps.
//
// MODE kRefCoords: decisions of checkKerALL exactly -- one draw per word-site
//   (ctr = sw*2K + hf*K + k of subsequence iseq + t + 128 g) expanded to 32
//   numbers by the LCG and compared with T4 = ceil(2^32 e^-4b), T8.
// MODE kNative: U_i < T/2^32 for the 32 replica bits is decided digit by
//   digit, most significant first, each digit a fresh Philox4x32-10 bit
//   (accept_native); each replica's acceptance probability is exactly
//   T/2^32, as in the reference.  The stream is keyed by stream_seed (one
//   per batch; populations differ in counter word 3).
// Tile gi0 (gc groups present) <-> HBM.  G > 1 (implies h % 4 == 0): group
// gi0+g's sublattice X goes to lat + X*G*h + g*h.  G = 1: sublattice X is a
// block of L + 2 rows at lat + X*sb -- row -1 (a copy of row L-1), rows
// 0..L-1, row L (a copy of row 0) -- so that the native sweep reads its
// vertical neighbours without wrapping; the sweep keeps the copies current.
// Out of line: keeps the sweep loop's registers free.
__device__ __noinline__ void msc_move_tile(const UnitParams& P, uint32_t* lat, int gi0, int gc, bool to_smem) {
  const int N = P.N, h = P.h, G = P.G;
  uint4* lat4 = (uint4*)lat;
  uint4* g4 = (uint4*)(P.words + (size_t)gi0 * N);
  if (G == 1) {
    const int Wr = P.Wr, L = P.L;
    uint32_t* gw = P.words + (size_t)gi0 * N;
    if ((Wr & 3) == 0) {  // rows start on 16-byte boundaries in both places
      const int h4 = h >> 2;
      for (int v = threadIdx.x; v < 2 * h4; v += blockDim.x) {
        const int X = v >= h4 ? 1 : 0, i = v - X * h4;
        uint4* s = (uint4*)(lat + X * P.sb + Wr) + i;
        uint4* d = (uint4*)(gw + X * h) + i;
        if (to_smem) *s = *d;
        else *d = *s;
      }
    } else {
      for (int v = threadIdx.x; v < N; v += blockDim.x) {
        const int X = v >= h ? 1 : 0, i = v - X * h;
        uint32_t* s = lat + X * P.sb + Wr + i;
        if (to_smem) *s = gw[v];
        else gw[v] = *s;
      }
    }
    if (to_smem)  // periodic copies: row -1 = row L-1, row L = row 0
      for (int v = threadIdx.x; v < 4 * Wr; v += blockDim.x) {
        const int X = v >= 2 * Wr ? 1 : 0, r = v - X * 2 * Wr, top = r < Wr ? 1 : 0, i = top ? r : r - Wr;
        lat[X * P.sb + (top ? 0 : (L + 1) * Wr) + i] = gw[X * h + (top ? (L - 1) * Wr : 0) + i];
      }
    return;
  }
  const int h4 = h >> 2, n4 = N >> 2;
  for (int v = threadIdx.x; v < 2 * gc * h4; v += blockDim.x) {
    const int X = v >= gc * h4 ? 1 : 0, r = v - X * gc * h4;
    const int g = (int)__umulhi((uint32_t)r, P.invH4), i = r - g * h4;
    uint4* s = lat4 + X * G * h4 + g * h4 + i;
    uint4* d = g4 + (size_t)g * n4 + X * h4 + i;
    if (to_smem) *s = *d;
    else *d = *s;
  }
}

// Prefix tables of tile ti (groups gi0, ...): one entry per word of the
// sublattice stack, and one per chain (thread, batch).
__device__ __noinline__ void msc_tables(const UnitParams& P, uint32_t* lat, int gi0, int ti,
                                        unsigned long long stream_seed) {
  const PhiloxKeys keys(stream_seed);
  uint2* tab = reinterpret_cast<uint2*>(lat + P.tab);
  uint2* ctab = reinterpret_cast<uint2*>(lat + P.ctab);
  const uint32_t step = (uint32_t)P.step, base = (uint32_t)gi0 * (uint32_t)P.h;
  const int n = P.tab ? P.G * P.h : 0;
  for (int v = threadIdx.x; v < n; v += blockDim.x) tab[v] = philox_prefix(base + (uint32_t)v, step, P.tag, keys);
  for (int q = 0; q < 2 * P.nbatch; ++q)
    ctab[q * kSweepThreads + threadIdx.x] =
        philox_prefix(((uint32_t)ti * blockDim.x + threadIdx.x) * (uint32_t)P.nbatch + (uint32_t)(q >> 1), step,
                      q & 1 ? P.tag ^ kFinishTagFlip : P.tag, keys);
}

// Energy and magnetisation per replica bit of the tile: the left and up
// bond of every A and B site (PAisingMSC.cu:272-294), counted per bit in
// bitsliced counters (BitCounters) and added into cntE / cntM [group of the
// tile][bit].  Each warp works inside one group (kSweepThreads/32/G warps per
// group, at most h / (32 wpg) <= 32 words per lane), so its counts never mix
// groups.
__device__ __noinline__ void msc_count(const UnitParams& P, const uint32_t* lat, int gc, int* cntE, int* cntM) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int L = P.L, Wr = P.Wr, h = P.h, G = P.G, wpg = (kSweepThreads / 32) / G;
  const int w = tid >> 5, g = w / wpg, ws = w - g * wpg;
  if (g >= gc) return;  // warp-uniform
  BitCounters bc;
  bc.reset();
  const uint32_t* A = G == 1 ? lat + Wr : lat + g * h;
  const uint32_t* B = G == 1 ? lat + P.sb + Wr : lat + G * h + g * h;
  for (int j0 = ws * 32 + lane; j0 - lane < h; j0 += 4 * wpg * 32) {
    BondWord w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int j = j0 + k * wpg * 32;
      w[k] = BondWord{};
      if (j < h) {
        const int y = (int)__umulhi((uint32_t)j, P.invWr), x = j - y * Wr;
        const int iL = y * Wr + (x == 0 ? Wr - 1 : x - 1), iU = (y + 1 == L ? 0 : y + 1) * Wr + x;
        const uint32_t sA = A[j], sB = B[j];
        // the left bond that is not between the two words: B's on odd rows, A's on even
        w[k] = BondWord{{sA ^ sB, (y & 1 ? A : B)[iL] ^ (y & 1 ? sB : sA), sA ^ B[iU], sB ^ A[iU]}, sA, sB};
      }
    }
    bc.add(w);
  }
  bc.totals(lane, (h + wpg * 32 - 1) / (wpg * 32), cntE + g * kMsb, cntM + g * kMsb);
}

static_assert(kMaxTile * kMsb == kSweepThreads, "one thread per (group of the tile, bit) in the epilogue");
// KIND: which forms of the native sweep the kernel holds (msc_kind).  One kernel
// with all of them gives each form a register allocation that the others
// decide; a kernel of its own is worth, in attempts per second, 4% to
// units of one batch with two sites per thread (L = 32) and 1-3% with four
// (stacked tiles), and 7-9% to the general form of one group (L = 56, 72, 80;
// 4% at 100; 15% at 48), whose remainder batches have code of their own there
// only.  L = 64, 96, 128 and units of one site per thread gained nothing from
// kernels of their own (0.96-1.01): kMixed holds all forms, for L = 96 alone or
// beside others; kCommon all but L = 96's, which costs L = 64 2.4%.
// Spills at 64 registers (four CTAs per SM): kGeneral none, the others 280 to
// 300 bytes of stores and 456 to 548 of loads.  They lie outside the hot loops of
// L = 64 and 96 (0.1% and 0.3% of the instructions executed are loads of
// spilled words) but inside those of one-batch units (L = 32, 200000 replicas:
// 4.2%), which are the faster for all that.
template <int MODE, int KIND>
__global__ void __launch_bounds__(kSweepThreads, 4)
    msc_sweep_kernel(BatchDev* b, int energy_only, unsigned long long stream_seed, int nsm) {
  const PhiloxKeys keys(stream_seed);
  extern __shared__ __align__(16) uint32_t lat[];  // G sublattices A, then G sublattices B; prefix tables
  __shared__ int s_unit, s_pop;
  __shared__ int s_cntE[kMaxTile * kMsb], s_cntM[kMaxTile * kMsb];  // [group of the tile][bit]
  __shared__ __align__(16) uint2 s_dig[kDigits];  // per digit j: digit_table(T4, T8, j)
  __shared__ UnitParams P;
  __shared__ BitStats stats;

  const int tid = threadIdx.x, lane = tid & 31;
  const int total = b->unit_prefix[b->npop];
  int cur = -1;
  int tx = 0, rsub = 0, txl = 0, txr = 0;
  bool worker = false;
  if (tid < kMsb) stats.reset(tid);

  for (;;) {
    __syncthreads();
    if (tid == 0) {
      const int u = cur < 0 ? first_unit(b, nsm, total) : later_unit(b, gridDim.x);
      int loc = 0;
      const int p = u < total ? queue_pop(b, u, &loc) : -1;
      s_pop = p;
      s_unit = loc;
      if (p >= 0 && p != cur) {  // parameters of a new population
        const PopDev* st = b->pops + p;
        // every field is loaded before the first store: the compiler cannot
        // move a load past a store to shared memory, and one by one the loads
        // took 3 us
        const int L = st->L, N = st->N, Wr = st->Wr, rpp = st->rpp, npass = st->npass, kconst = st->kconst,
                  step = st->step, sweeps = st->sweeps, gpt = st->gpt, R = st->R_cur, Rp = st->R_prev,
                  parity = st->parity, pop_id = st->pop_id;
        const uint32_t nstep = native_step_word(st);
        const unsigned long long seed = st->seed, iseq = st->iseq;
        const uint32_t invL = st->invL, invWr = st->invWr;
        void* const sp0 = st->spins[0];
        void* const sp1 = st->spins[1];
        const uint8_t *act0 = st->active[0], *act1 = st->active[1];
        int32_t *E = st->E, *M = st->M;
        const uint32_t* thr = st->thr + (size_t)step * kThrPerStep;
        const uint32_t T4 = thr[10], T8 = thr[11];
        P.L = L; P.N = N; P.h = N >> 1; P.Wr = Wr; P.rpp = rpp; P.npass = npass;
        P.kconst = kconst;
        P.step = (int)nstep;
        P.sweeps = energy_only ? 0 : sweeps;
        P.nbatch = (npass + kKB - 1) / kKB;
        P.G = gpt > 0 ? gpt : 1;
        P.rg = (R + kMsb - 1) / kMsb;
        P.sb = msc_halo_block(L, Wr);
        P.invL = invL;
        P.invWr = invWr;
        P.invH4 = 0xFFFFFFFFu / (uint32_t)(N >> 3) + 1u;  // ceil(2^32 / (h / 4))
        const TableLayout tl = msc_unit_layout(L, Wr, P.G, P.nbatch);
        P.tab = tl.tab;
        P.ctab = tl.ctab;
        P.tag = kTagMscSweep | (uint32_t)pop_id;
        P.T4 = T4;
        P.T8 = T8;
        P.seed = seed;
        const int rg_prev = (Rp + kMsb - 1) / kMsb;
        P.iseq = iseq + (step > 0 ? (unsigned long long)rg_prev * kMsb : 0ull);
        P.words = (uint32_t*)(parity ? sp1 : sp0);
        P.act = parity ? act1 : act0;
        P.E = E;
        P.M = M;
      }
    }
    s_cntE[tid] = 0;  // kMaxTile * kMsb == kSweepThreads
    s_cntM[tid] = 0;
    __syncthreads();
    const int p = s_pop, ti = s_unit;  // population, tile
    if (p < 0) break;
    if (p != cur) {  // block-uniform
      if (tid < kMsb && cur >= 0) stats.flush(b->pops + cur, tid);
      cur = p;
      const int Wr = P.Wr;
      worker = tid < Wr * P.rpp;
      tx = worker ? tid % Wr : 0;
      rsub = worker ? tid / Wr : 0;
      txl = (tx == 0 ? Wr - 1 : tx - 1);
      txr = (tx + 1 == Wr ? 0 : tx + 1);
      if (tid < kDigits) s_dig[tid] = digit_table(P.T4, P.T8, tid);
    }
    const int N = P.N, h = P.h, G = P.G, gi0 = ti * G;
    const int gc = min(G, P.rg - gi0);  // groups present in this tile
    msc_move_tile(P, lat, gi0, gc, true);
    if (MODE == kNative && P.ctab && P.sweeps > 0) msc_tables(P, lat, gi0, ti, stream_seed);
    __syncthreads();

    // stacked row v of the tile -> group g, row y in the group, smem offsets
    // of the row and its vertical neighbours (periodic inside the group)
    struct RowPos {
      int g, y, row, rowu, rowd;
    };
    auto row_pos = [&](int v) {
      RowPos q;
      const int L = P.L, Wr = P.Wr;
      q.g = (int)__umulhi((uint32_t)v, P.invL);
      q.y = v - q.g * L;
      q.row = v * Wr;
      q.rowu = (q.y == 0 ? v + L - 1 : v - 1) * Wr;
      q.rowd = (q.y + 1 == L ? v + 1 - L : v + 1) * Wr;
      return q;
    };
    const int vrows = gc * P.L;  // stacked rows present
    const int sweeps = P.sweeps;
    // Units of one batch per thread and half-sweep (small lattices: up to
    // L = 45 alone, stacked tiles of up to 1024 words): the batch's addresses,
    // wraps and prefixes stay in registers for the whole temperature.  One or
    // two sites per thread leave few warps' worth of work per SM, which waits
    // for chains of rounds: their blocks are drawn side by side.  Same slots,
    // chains and draws as the general forms below.  One population, L = 32
    // R = 5000 (two sites per thread, one unit per SM), 100 sweeps: 19.8 ->
    // 14.6 ms per anneal of 49 temperatures; full GPU, L = 16 R = 200000 (tiles
    // of 8 groups, four sites per thread): 3125 -> 3275 attempts/ns.
    auto one_batch = [&](auto nv_c, auto stack_c) {
      constexpr int NV = decltype(nv_c)::value;
      constexpr bool kStack = decltype(stack_c)::value;
      const int threads = (P.Wr * P.rpp + 31) & ~31;  // whole warps that hold words
      if (tid >= threads) return;
      const int Wr = P.Wr, L = P.L, npass = P.npass;
      // rows of the slots; a thread without sites stands at row 0, a slot
      // without one at its thread's slot 0, and both decide nothing
      const int first = kStack ? rsub : rsub * npass, step_r = kStack ? P.rpp : 1, step_w = step_r * Wr;
      const bool any = worker && first < vrows;
      const int row0 = any ? first : 0;
      const int at = row0 * Wr + tx;  // slot 0's word of its sublattice
      // per slot a bit: holds a site (0..3), wraps up (4..7), wraps down (8..11), odd row (12..15)
      uint32_t flags = 0;
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        const bool is = any && k < npass && row0 + k * step_r < vrows;
        const int v = is ? row0 + k * step_r : row0;
        const int y = kStack ? v - (int)__umulhi((uint32_t)v, P.invL) * L : v;
        flags |= ((is ? 1u : 0u) | (y == 0 ? 16u : 0u) | (y + 1 == L ? 256u : 0u) | (uint32_t)(y & 1) << 12) << k;
      }
      auto valid = [&](int k) { return (flags >> k & 1u) != 0u; };
      auto up0 = [&](int k) { return (flags >> (4 + k) & 1u) != 0u; };
      auto dn0 = [&](int k) { return (flags >> (8 + k) & 1u) != 0u; };
      constexpr bool kHold = NV <= 2;  // prefixes in registers (four sites' would spill)
      uint2 pre[NV], pd, pf;
      auto site_tab = [&](int k) { return reinterpret_cast<const uint2*>(lat + P.tab)[at + (valid(k) ? k * step_w : 0)]; };
      auto chain_tab = [&](int f) { return reinterpret_cast<const uint2*>(lat + P.ctab)[tid + f * kSweepThreads]; };
      if constexpr (kHold) {
#pragma unroll
        for (int k = 0; k < NV; ++k) pre[k] = site_tab(k);
        pd = chain_tab(0);
        pf = chain_tab(1);
      }
      const uint32_t base = (uint32_t)gi0 * (uint32_t)h + (uint32_t)at;
      const uint32_t chain = (uint32_t)ti * blockDim.x + (uint32_t)tid;  // one batch per thread
      const uint32_t step = (uint32_t)P.step, tag = P.tag;
      const int dl = txl - tx, dr = txr - tx;
      const uint4* dig = reinterpret_cast<const uint4*>(s_dig);
      for (int sw = 0; sw < sweeps; ++sw) {
#pragma unroll 1
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t* self = (kStack ? lat + (hf ? G * h : 0) : lat + (hf ? P.sb : 0) + Wr) + at;
          const uint32_t* oth = (kStack ? lat + (hf ? 0 : G * h) : lat + (hf ? 0 : P.sb) + Wr) + at;
          const HalfSweep hs((uint32_t)((sw * 2 + hf) << 4), step, tag, P.T4, P.T8, keys);
          uint32_t av[kKB], un[kKB], ac[kKB], site[kKB];
#pragma unroll
          for (int k = 0; k < NV; ++k) {
            const bool v = valid(k);
            const int w = v ? k * step_w : 0;
            const bool left = (hf == 0) == ((flags >> (12 + k) & 1u) == 0u);
            int wu = w - Wr, wd = w + Wr;
            if (kStack) {
              if (up0(k)) wu += h;
              if (dn0(k)) wd -= h;
            }
            count_masks(self[w], oth[w + (left ? dl : dr)], oth[w], oth[wu], oth[wd], av[k], ac[k]);
            un[k] = v ? 0xFFFFFFFFu - ac[k] : 0u;
            site[k] = base + (uint32_t)w;
          }
          accept_native<NV, (NV <= 2)>(
              av, un, ac, site, chain, hs, keys, dig, NV,
              [&](int k) {
                if constexpr (kHold) return pre[k];
                else return site_tab(k);
              },
              [&](int f) {
                if constexpr (kHold) return f ? pf : pd;
                else return chain_tab(f);
              });
#pragma unroll
          for (int k = 0; k < NV; ++k)
            if (valid(k)) {
              const uint32_t nw = self[k * step_w] ^ ac[k];
              self[k * step_w] = nw;
              if (!kStack) {
                if (up0(k)) self[k * step_w + h] = nw;  // copy below row L-1
                if (dn0(k)) self[k * step_w - h] = nw;  // copy above row 0
              }
            }
          asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
        }
      }
    };
    constexpr bool kSingles = MODE == kNative && (KIND == kOneBatch || KIND == kMixed || KIND == kCommon);
    const bool single = kSingles && P.nbatch == 1 && P.tab;
    if constexpr (kSingles) {
      if (single) {
        if (G == 1) {
          if (KIND != kOneBatch && P.npass == 1) one_batch(std::integral_constant<int, 1>(), std::false_type());
          else if (P.npass == 2) one_batch(std::integral_constant<int, 2>(), std::false_type());
          else one_batch(std::integral_constant<int, 4>(), std::false_type());
        } else {
          if (KIND != kOneBatch && P.npass == 1) one_batch(std::integral_constant<int, 1>(), std::true_type());
          else if (P.npass == 2) one_batch(std::integral_constant<int, 2>(), std::true_type());
          else one_batch(std::integral_constant<int, 4>(), std::true_type());
        }
        __syncthreads();
      } else if (KIND == kOneBatch && tid == 0 && sweeps > 0) {
        b->pops[p].error = kErrSweepForm;
      }
    }
    for (int sw = 0; KIND != kOneBatch && !single && sw < sweeps; ++sw) {
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {
        // row 0 of the swept and of the other sublattice
        uint32_t* self = G == 1 ? lat + (hf ? P.sb : 0) + P.Wr : lat + (hf ? G * h : 0);
        const uint32_t* oth = G == 1 ? lat + (hf ? 0 : P.sb) + P.Wr : lat + (hf ? 0 : G * h);
        const int Wr = P.Wr, rpp = P.rpp, npass = P.npass;
        if (MODE == kRefCoords) {
#pragma unroll 1
          for (int pass = 0; pass < npass; ++pass) {
            const int v = rsub + pass * rpp;
            const bool valid = worker && v < vrows;
            const RowPos q = row_pos(valid ? v : 0);
            const int sidx = q.row + tx;       // word in the tile's sublattice array
            const int idx = q.y * Wr + tx;     // word in the group's sublattice
            const int gi = gi0 + q.g;
            // horizontal neighbour not at the same idx (PAisingMSC.cu:203, 238)
            const bool left = (hf == 0) == ((q.y & 1) == 0);
            const uint32_t s = self[sidx];
            const uint32_t n1 = oth[q.row + (left ? txl : txr)], n2 = oth[sidx], n3 = oth[q.rowu + tx],
                           n4 = oth[q.rowd + tx];
            uint32_t s0, s1, s2;
            adder4(s ^ n1, s ^ n2, s ^ n3, s ^ n4, s0, s1, s2);
            const int t = idx & (kRefThreads - 1), k = idx >> 7;
            const int K = P.kconst ? P.kconst : (t < h ? (h - t + kRefThreads - 1) / kRefThreads : 0);
            const unsigned long long sub = P.iseq + (unsigned long long)t + (unsigned long long)kRefThreads * gi;
            uint32_t ran = ref_word(P.seed, sub, (unsigned long long)sw * 2 * K + (unsigned long long)hf * K + k);
            const uint32_t T4 = P.T4, T8 = P.T8;
            uint32_t c4 = 0, c8 = 0;
#pragma unroll 8
            for (int i = 0; i < kMsb; ++i) {
              c4 |= (ran < T4 ? 1u : 0u) << i;
              c8 |= (ran < T8 ? 1u : 0u) << i;
              ran = kLcgA * ran + kLcgC;
            }
            const uint32_t hi = s1 | s2;
            const uint32_t acc = hi | (~hi & ((s0 & c4) | (~s0 & c8)));
            if (valid) self[sidx] = s ^ acc;
          }
        } else {
          const HalfSweep hs((uint32_t)((sw * 2 + hf) << 4), (uint32_t)P.step, P.tag, P.T4, P.T8, keys);
          const uint4* dig = reinterpret_cast<const uint4*>(s_dig);
          // prefix tables (null: none): entry i of the first is site base + i
          const uint2* tab = P.tab ? reinterpret_cast<const uint2*>(lat + P.tab) : nullptr;
          const uint2* ctab = reinterpret_cast<const uint2*>(lat + P.ctab) + tid;
          auto chain_formed = [&](uint32_t chain, int f) {
            return philox_prefix(chain, hs.step, f ? hs.tag ^ kFinishTagFlip : hs.tag, keys);
          };
          const uint32_t base = (uint32_t)gi0 * (uint32_t)h;  // site number of the tile's first word
          // the general forms' prefixes: one branch for the batch, so that its four heads interleave
          auto site_prefixes = [&](const uint32_t (&site)[kKB], auto& pre) {
            constexpr int n = (int)(sizeof(pre) / sizeof(pre[0]));
            if (tab) {
#pragma unroll
              for (int k = 0; k < n; ++k) pre[k] = tab[site[k] - base];
            } else {
#pragma unroll
              for (int k = 0; k < n; ++k) pre[k] = philox_prefix(site[k], hs.step, hs.tag, keys);
            }
          };
          // L = 64, 96 and 128 with every size fixed at compile time: kW = L/2
          // words per row, kR = kSweepThreads/kW thread rows of kRows =
          // ceil(kL/kR) consecutive rows each (64: a warp per row, 8 rows per
          // thread; 96: 5 x 20 rows, the last batch of the fifth thread row
          // past the lattice; 128: two warps per row, 32 rows per thread);
          // every offset an immediate.  Same batches as the general form.
          auto native_fixed = [&](auto l_c) {
            constexpr int kL = decltype(l_c)::value, kW = kL / 2, kR = kSweepThreads / kW;
            constexpr int kRows = (kL + kR - 1) / kR;
            constexpr TableLayout kLay = msc_unit_layout(kL, kW, 1, kRows / kKB);
            constexpr bool kTab = kLay.tab != 0, kChainTab = kLay.ctab != 0;
            static_assert(kRows % kKB == 0 && (kR * kRows - kL) % kKB == 0, "whole batches, each in or past the lattice");
            const int vb0 = rsub * kRows;
            const uint32_t* txs = oth + (hf == 0 ? txl : txr);  // side neighbour on even rows
            const uint32_t* txo = oth + (hf == 0 ? txr : txl);  // and on odd rows
#pragma unroll 1
            for (int p0 = 0; p0 < kRows; p0 += kKB) {
              // a batch past the lattice (or of a thread without a column)
              // reads rows 0..3 and decides nothing, but takes part in the
              // warp's acceptance
              constexpr bool kAll = kR * kW == kSweepThreads && kR * kRows == kL;  // every batch of every thread
              const bool bvalid = kAll || (worker && vb0 + p0 < kL);
              const int vb = bvalid ? vb0 + p0 : 0;
              const uint32_t* po = oth + (vb - 1) * kW + tx;  // rows vb-1 .. vb+4 (rows -1 and kL: copies)
              uint32_t* ps = self + vb * kW + tx;
              uint32_t av[kKB], un[kKB], ac[kKB], site[kKB];
#pragma unroll
              for (int k = 0; k < kKB; ++k) {
                const uint32_t s = ps[k * kW];
                const uint32_t side = ((k & 1) ? txo : txs)[(vb + k) * kW];
                count_masks(s, side, po[(k + 1) * kW], po[k * kW], po[(k + 2) * kW], av[k], ac[k]);
                un[k] = bvalid ? 0xFFFFFFFFu - ac[k] : 0u;  // = ~ac, on the FMA pipe
                site[k] = base + (uint32_t)((vb + k) * kW + tx);
              }
              const uint32_t chain =
                  ((uint32_t)ti * blockDim.x + (uint32_t)tid) * (uint32_t)(kRows / kKB) + (uint32_t)(p0 / kKB);
              // L = 64 has both tables, 96 the chains', 128 none
              accept_native(
                  av, un, ac, site, chain, hs, keys, dig, kKB,
                  [&](int k) {
                    if constexpr (kTab) return tab[(vb + k) * kW + tx];
                    else return philox_prefix(site[k], hs.step, hs.tag, keys);
                  },
                  [&](int f) {
                    if constexpr (kChainTab) return ctab[(2 * (p0 / kKB) + f) * kSweepThreads];
                    else return chain_formed(chain, f);
                  });
              if (bvalid) {
#pragma unroll
                for (int k = 0; k < kKB; ++k) {
                  const uint32_t nw = ps[k * kW] ^ ac[k];
                  ps[k * kW] = nw;
                  if (vb + k == 0) self[kL * kW + tx] = nw;         // copy below row kL-1
                  if (vb + k == kL - 1) self[-kW + tx] = nw;        // copy above row 0
                }
              }
            }
          };
          if ((KIND == kMixed || KIND == kCommon) && G == 1 && P.L == 64) {
            native_fixed(std::integral_constant<int, 64>());
          } else if ((KIND == kMixed || KIND == kCommon) && G == 1 && P.L == 128) {
            native_fixed(std::integral_constant<int, 128>());
          } else if (KIND == kMixed && G == 1 && P.L == 96) {
            native_fixed(std::integral_constant<int, 96>());
          } else if (G == 1) {
            // one group, any other L: thread rsub owns the
            // consecutive rows rsub*npass .. rsub*npass + npass - 1 of column
            // tx, so a batch of kKB rows shares the other sublattice's rows
            // around them, and the periodic copies of rows -1 and L spare the
            // vertical wrap
            // (kGeneral: where a thread's rows are not whole batches, the last
            // one runs in code of its own for its number of rows: L = 48, five
            // rows, 3050 -> 3400 attempts/ns; L = 80, fourteen, 4090 -> 4290.)
            const int L = P.L;
            auto rows = [&](auto nv_c, int p0) {
              constexpr int NV = decltype(nv_c)::value;
              const int vb = rsub * npass + p0;  // first row of the batch
              uint32_t o[NV + 2];  // other sublattice, rows vb-1 .. vb+NV (clamped to the copy of row 0)
#pragma unroll
              for (int j = 0; j < NV + 2; ++j) o[j] = oth[min(vb - 1 + j, L) * Wr + tx];
              // horizontal neighbour not at the same index: left for A on even
              // rows and B on odd rows (PAisingMSC.cu:203, 238); alternates by row
              const bool left0 = (hf == 0) == ((vb & 1) == 0);
              uint32_t av[kKB], un[kKB], ac[kKB], site[kKB];
              uint32_t vm = 0;  // slots holding a site
#pragma unroll
              for (int k = 0; k < NV; ++k) {
                const int y = vb + k;
                const bool valid = worker && (KIND == kGeneral || p0 + k < npass) && y < L;
                const int row = min(y, L) * Wr;
                const uint32_t s = self[row + tx];
                const uint32_t side = oth[row + ((left0 != ((k & 1) != 0)) ? txl : txr)];
                count_masks(s, side, o[k + 1], o[k], o[k + 2], av[k], ac[k]);
                un[k] = valid ? 0xFFFFFFFFu - ac[k] : 0u;  // = ~ac, on the FMA pipe
                vm |= valid ? 1u << k : 0u;
                site[k] = base + (uint32_t)(row + tx);  // = group * h + word in the group
              }
              const uint32_t chain = ((uint32_t)ti * blockDim.x + (uint32_t)tid) * (uint32_t)P.nbatch + (uint32_t)(p0 / kKB);
              uint2 pre[NV];
              site_prefixes(site, pre);
              accept_native<NV>(
                  av, un, ac, site, chain, hs, keys, dig, KIND == kGeneral ? NV : npass - p0, [&](int k) { return pre[k]; },
                  [&](int f) {
                    return P.ctab ? ctab[(2 * (p0 / kKB) + f) * kSweepThreads] : chain_formed(chain, f);
                  });
#pragma unroll
              for (int k = 0; k < NV; ++k)
                if (vm >> k & 1u) {
                  const int y = vb + k;
                  const uint32_t nw = self[y * Wr + tx] ^ ac[k];
                  self[y * Wr + tx] = nw;
                  if (y == 0) self[L * Wr + tx] = nw;         // copy below row L-1
                  if (y == L - 1) self[-Wr + tx] = nw;        // copy above row 0
                }
            };
            const int whole = KIND != kGeneral ? npass : npass & ~(kKB - 1);
#pragma unroll 1
            for (int p0 = 0; p0 < whole; p0 += kKB) rows(std::integral_constant<int, kKB>(), p0);
            const int rest = npass - whole;
            if constexpr (KIND == kGeneral) {
              if (rest == 1) rows(std::integral_constant<int, 1>(), whole);
              else if (rest == 2) rows(std::integral_constant<int, 2>(), whole);
              else if (rest == 3) rows(std::integral_constant<int, 3>(), whole);
            }
          } else {
            // stacked tiles: thread (rsub, tx) takes stacked rows rsub + pass*rpp
#pragma unroll 1
            for (int p0 = 0; p0 < npass; p0 += kKB) {
              uint32_t av[kKB], un[kKB], ac[kKB], site[kKB];
              uint32_t vm = 0;  // slots holding a site
#pragma unroll
              for (int k = 0; k < kKB; ++k) {
                const int pass = p0 + k;
                const int v = rsub + pass * rpp;
                const bool valid = worker && pass < npass && v < vrows;
                const int vc = valid ? v : 0;
                const RowPos q = row_pos(vc);
                const int sidx = q.row + tx;
                // row parity: stacked groups have even L, so v and y agree
                const bool left = (hf == 0) == ((vc & 1) == 0);
                const uint32_t s = self[sidx];
                const uint32_t n1 = oth[q.row + (left ? txl : txr)], n2 = oth[sidx], n3 = oth[q.rowu + tx],
                               n4 = oth[q.rowd + tx];
                count_masks(s, n1, n2, n3, n4, av[k], ac[k]);
                un[k] = valid ? 0xFFFFFFFFu - ac[k] : 0u;  // = ~ac, on the FMA pipe
                vm |= valid ? 1u << k : 0u;
                site[k] = base + (uint32_t)sidx;  // = group * h + word in the group
              }
              const uint32_t chain = ((uint32_t)ti * blockDim.x + (uint32_t)tid) * (uint32_t)P.nbatch + (uint32_t)(p0 / kKB);
              uint2 pre[kKB];
              site_prefixes(site, pre);
              accept_native(
                  av, un, ac, site, chain, hs, keys, dig, npass - p0, [&](int k) { return pre[k]; },
                  [&](int f) {
                    return P.ctab ? ctab[(2 * (p0 / kKB) + f) * kSweepThreads] : chain_formed(chain, f);
                  });
#pragma unroll
              for (int k = 0; k < kKB; ++k)
                if (vm >> k & 1u) self[site[k] - base] ^= ac[k];
            }
          }
        }
        __syncthreads();
      }
    }

    msc_count(P, lat, gc, s_cntE, s_cntM);
    msc_move_tile(P, lat, gi0, gc, false);
    __syncthreads();
    if (tid < gc * kMsb) {
      const int gi = gi0 + (tid >> 5);
      const int E = 2 * s_cntE[tid] - 2 * N, Mg = 2 * s_cntM[tid] - N;
      P.E[gi * kMsb + lane] = E;
      P.M[gi * kMsb + lane] = Mg;
    }
    if (tid < kMsb) {  // lane k of warp 0 owns the statistics of bit k
      for (int g = 0; g < gc; ++g) {
        const int gi = gi0 + g, E = 2 * s_cntE[g * kMsb + tid] - 2 * N, Mg = 2 * s_cntM[g * kMsb + tid] - N;
        if (P.act[gi * kMsb + tid]) stats.add(tid, E, Mg);
      }
    }
  }
  if (tid < kMsb && cur >= 0) stats.flush(b->pops + cur, tid);
}

// -------------------------------------------------------------- resample
// Reference stream: resampleKer places offspring number s (in the scan order
// of (old group, bit)) at new group s % rg_new, bit s / rg_new
// (PAisingMSC.cu:413-414), which the reference-stream parity needs.  Here every new word gathers its 32 bits:
// bit k of new group j comes from old replica src[k*rg_new + j].
//
// Work unit of one warp: 32 consecutive new groups (lane g builds group
// j0 + g) x a strip of 32 sites.  Lane g resolves the sources of its 32 bits
// into row pointers and rotations held in registers, four bits at a time,
// and gathers its 32 output words with loads at immediate offsets.  The 32
// lanes' sources are 32 consecutive new replicas, i.e. neighbouring old
// replicas in one or two old groups, so a load instruction touches one or two
// old words: the gather costs about one warp load per output word, and no L2
// traffic beyond the old rows themselves.  Units of all populations of the
// batch come from one queue (plan_batch) and are taken by
// persistent warps, so uneven populations finish together.
constexpr int kResampleThreads = 256;

// Native stream gather (msc_resample_native_kernel)
constexpr int kNatThreads = 256;
constexpr int kNatBlocksPerSM = 3;
constexpr int kNatRing = 8;    // old rows in flight or in use per warp (a power of two)
constexpr int kNatAhead = 4;   // groups whose loads run ahead of the one being built
constexpr int kNatLists = 8;   // pair lists per warp (a power of two above kNatAhead)

template <bool kFull>
__device__ __forceinline__ void gather_sub(const uint32_t* const (&p)[4], const uint32_t (&rot)[4],
                                           const uint32_t (&msk)[4], int nv, uint32_t (&w)[kSub]) {
#pragma unroll
  for (int t = 0; t < kSub; ++t) {
    const int tc = kFull ? t : min(t, nv - 1);  // partial: repeat the last site (not stored)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t v = __ldg(p[q] + tc);
      w[t] |= __funnelshift_l(v, v, rot[q]) & msk[q];  // source bit rotated into bit k
    }
  }
}

constexpr int kResampleBlocksPerSM = 3;  // 80 registers, no spills

__global__ void __launch_bounds__(kResampleThreads, kResampleBlocksPerSM) msc_resample_kernel(BatchDev* b) {
  const int lane = threadIdx.x & 31;
  const int total = b->res_prefix[b->npop];
  for (;;) {
    int u = 0;
    if (lane == 0) u = (int)atomicAdd(&b->res_next, 1u);
    u = __shfl_sync(kFull, u, 0);
    if (u >= total) break;
    int lo = 0, hi = b->npop;  // population of unit u
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (b->res_prefix[mid] <= u) lo = mid;
      else hi = mid;
    }
    const PopDev* st = b->pops + lo;
    const int N = st->N, Rn = st->R_cur, rgn = (Rn + kMsb - 1) / kMsb, S = res_strip(N, rgn);
    const int nstrip = (N + S - 1) / S;
    const int loc = u - b->res_prefix[lo], tile = loc / nstrip, strip = loc - tile * nstrip;
    const int j = tile * 32 + lane, t0 = strip * S, nt = min(S, N - t0);
    const bool jv = j < rgn;
    const uint32_t* old = (const uint32_t*)st->spins[st->parity ^ 1];
    const uint32_t* src = st->src;
    if (strip == 0 && jv) {
      uint8_t* act = st->active[st->parity];
#pragma unroll 4
      for (int k = 0; k < kMsb; ++k) act[j * kMsb + k] = (k * rgn + j) < Rn ? 1 : 0;
    }
    uint32_t* dst = (uint32_t*)st->spins[st->parity] + (size_t)j * N + t0;
#pragma unroll 1
    for (int tc = 0; tc < nt; tc += kSub) {
      const int nv = min(kSub, nt - tc);  // a multiple of 4: N and t0 are
      uint32_t w[kSub];
#pragma unroll
      for (int t = 0; t < kSub; ++t) w[t] = 0u;
#pragma unroll 1
      for (int k0 = 0; k0 < kMsb; k0 += 4) {
        const uint32_t* p[4];
        uint32_t rot[4], msk[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int k = k0 + q, s = k * rgn + j;
          const bool v = jv && s < Rn;
          const uint32_t lin = v ? src[s] : 0u;  // an invalid bit reads old word 0 and is masked off
          p[q] = old + (size_t)(lin >> 5) * N + t0 + tc;
          rot[q] = ((uint32_t)k - (lin & 31u)) & 31u;
          msk[q] = v ? 1u << k : 0u;
        }
        if (nv == kSub) gather_sub<true>(p, rot, msk, nv, w);
        else gather_sub<false>(p, rot, msk, nv, w);
      }
      if (jv) {
        uint4* d4 = reinterpret_cast<uint4*>(dst + tc);
        d4[0] = make_uint4(w[0], w[1], w[2], w[3]);
        if (nv > 4) d4[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
  }
}

// --------------------------------------------- resample, native stream
// With the engine's own stream the placement of offspring is free (replicas
// are exchangeable), so offspring s goes to slot s: group s / 32, bit s % 32.
// The sources of a new group's 32 bits are then 32 consecutive entries of the
// monotone gather map, i.e. a window of old replicas that are mostly
// consecutive themselves: with offsets o_b = src[32j + b] - 32 (first - 1),
// first = src[32j] / 32, bit b of the new word is bit o_b of the bit string
// W = old words first-1, first, first+1, first+2 at that site (W's word 0 is
// never selected: o_b >= 32).  Bits sharing the shift d = o_b - b form one
// mask M_d, and the new word is OR_d ((W >> d) & M_d), one funnel shift and
// one logic operation per distinct shift instead of per bit.  Copy numbers
// of 1 keep the shift; a duplicate lowers it by one, a replica without
// offspring raises it, so a word has a handful of distinct shifts.
//
// Copies of one parent are the exception: a run of k new bits with the same
// source has k distinct shifts, so a parent with many copies (a large dbeta
// against the energy spread) would turn a word into 32 single-bit pairs.
// A run of four or more is one broadcast pair instead: the run's mask M and
// the source's bit B in its window word, new |= M where that word has B.
//
// msc_pairs_kernel (one warp per new group of every population, lane b for
// bit b) lists a group's distinct shifts of the other bits as (M_d, d mod 32)
// pairs ordered by the window word d / 32 they start in (counts n0, n1, n2),
// then its runs of four or more bits of one source as (M, B) pairs ordered by the window word p / 32 holding the source (counts k1, k2,
// k3): the lanes sharing a shift or a source find each other with one match
// each, and the lowest of them writes the pair.  A group whose sources span more than the
// four-word window (more than 64 replicas without offspring among ~96
// consecutive ones), or whose counts do not fit the 5-bit fields of its count
// word, is flagged and gathered bit by bit.
__global__ void __launch_bounds__(256) msc_pairs_kernel(BatchDev* b) {
  const int lane = threadIdx.x & 31, np = b->npop, total = b->grp_prefix[np];
  const uint32_t lt = (1u << lane) - 1u;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total; i += (gridDim.x * blockDim.x) >> 5) {
    int lo = 0, hi = np;  // population of new group i (warp-uniform)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (b->grp_prefix[mid] <= i) lo = mid;
      else hi = mid;
    }
    PopDev* st = b->pops + lo;
    const int j = i - b->grp_prefix[lo], nb = min(kMsb, st->R_cur - j * kMsb);
    const uint32_t* src = st->src + (size_t)j * kMsb;
    const bool v = lane < nb;
    // source of bit b relative to the window, o = src[b] - 32 (first - 1) >= 32
    // (src nondecreasing, src[0] >= 32 first), and its shift d = o - b >= 1
    const uint32_t base = ((src[0] >> 5) - 1u) * 32u;  // may wrap; only differences matter
    const uint32_t s = v ? src[lane] : 0xFFFFFFFFu;    // the invalid bits share 0xFFFFFFFF
    if (st->family) st->anc[st->parity][(size_t)j * kMsb + lane] = v ? st->anc[st->parity ^ 1][s] : -1;  // family_resample
    const uint32_t o = s - base, d = o - (uint32_t)lane;
    bool fallback = __any_sync(kFull, v && d >= 96u);  // then o < 128 for every bit
    // bits with this bit's source; a run of k >= 4 of them is one broadcast
    // pair (as shifts its first and last bits join their neighbours' pairs,
    // the k - 2 between take a pair each)
    const uint32_t ms = __match_any_sync(kFull, s);
    const bool run = v && __popc(ms) >= 4;
    const uint32_t m = __match_any_sync(kFull, v && !run ? d : 0xFFFFFFFFu);  // bits outside runs with this shift
    const bool lead_d = v && !run && (m & lt) == 0u, lead_r = run && (ms & lt) == 0u;
    const uint32_t wd = d >> 5, wr = o >> 5;
    const uint32_t l0 = __ballot_sync(kFull, lead_d && wd == 0u), l1 = __ballot_sync(kFull, lead_d && wd == 1u),
                   l2 = __ballot_sync(kFull, lead_d && wd == 2u), r1 = __ballot_sync(kFull, lead_r && wr == 1u),
                   r2 = __ballot_sync(kFull, lead_r && wr == 2u), r3 = __ballot_sync(kFull, lead_r && wr == 3u);
    const uint32_t n0 = __popc(l0), n1 = __popc(l1), n2 = __popc(l2), k1 = __popc(r1), k2 = __popc(r2),
                   k3 = __popc(r3);
    fallback = fallback || n0 > 31u || n1 > 31u || n2 > 31u;  // a run has four bits: k <= 8
    if (!fallback && lead_d && wd < 3u) {
      const uint32_t at = wd == 0u ? __popc(l0 & lt) : wd == 1u ? n0 + __popc(l1 & lt) : n0 + n1 + __popc(l2 & lt);
      st->res_pairs[(size_t)j * kMsb + at] = make_uint2(m, d & 31u);
    }
    if (!fallback && lead_r) {
      const uint32_t c = n0 + n1 + n2;
      const uint32_t at = wr == 1u ? c + __popc(r1 & lt) : wr == 2u ? c + k1 + __popc(r2 & lt)
                                                                  : c + k1 + k2 + __popc(r3 & lt);
      st->res_pairs[(size_t)j * kMsb + at] = make_uint2(ms, 1u << (o & 31u));
    }
    if (lane == 0)
      st->res_cnt[j] = fallback ? 1u << 31 : n0 | n1 << 5 | n2 << 10 | k1 << 15 | k2 << 20 | k3 << 25;
  }
}

// The gather.  A warp takes a unit of nat_groups consecutive new groups x 128
// consecutive sites, lane = four consecutive sites, so that loads and stores
// are coalesced 512-byte row segments of 16-byte vectors and a group's pair
// list is the same for all lanes.  Of a window's four rows the first is never
// selected (0 stands in); the other three are first .. first + 2, and as first
// does not decrease from group to group, most of them are the previous group's:
// the warp keeps a ring of old rows in shared memory, each loaded once per unit
// (asynchronously, up to kNatAhead groups ahead of the one being built; every
// lane reads back only what it loaded itself), beside a ring of pair lists.
// Units are spread over the persistent warps by a grid stride (the batch-wide
// unit prefix gives each population its range).
//
// What bounds it: a pair costs two ALU operations per site (shift and mask),
// so at ten pairs per group the ALU pipe needs about as long as HBM; the rest
// of a pair -- its broadcast read and the loop -- is shared by a lane's four
// sites.  One GB300, read + write of the population: L = 128, 131072 replicas,
// copies spread by 0.3: 234 us (2.29 TB/s, two sites per lane, four rows per
// group through the L1) -> 133 us (4.05 TB/s); spread 0.05: 207 -> 117 us
// (4.6 TB/s); L = 32, 10^6: 119 -> 67 us.
struct Sites4 {
  uint32_t w[4];
};
__device__ __forceinline__ Sites4 sites(uint4 q) { return Sites4{{q.x, q.y, q.z, q.w}}; }

__device__ __forceinline__ void nat_apply(Sites4& out, const Sites4& lo, const Sites4& hi, const uint2* pg, int i0,
                                          int i1) {
#pragma unroll 2
  for (int i = i0; i < i1; ++i) {
    const uint2 a = pg[i];
#pragma unroll
    for (int k = 0; k < 4; ++k) out.w[k] |= __funnelshift_r(lo.w[k], hi.w[k], a.y) & a.x;
  }
}

// broadcast pairs (M, B): every bit of M where the window word has bit B
__device__ __forceinline__ void nat_bcast(Sites4& out, const Sites4& w, const uint2* pg, int i0, int i1) {
#pragma unroll 2
  for (int i = i0; i < i1; ++i) {
    const uint2 a = pg[i];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (w.w[k] & a.y) out.w[k] |= a.x;
  }
}

// a group's words at four sites from its window rows and pair list
__device__ __forceinline__ Sites4 nat_words(const Sites4& w1, const Sites4& w2, const Sites4& w3, const uint2* pg,
                                            uint32_t cnt) {
  const int c1 = cnt & 31u, c2 = c1 + ((cnt >> 5) & 31u), c3 = c2 + ((cnt >> 10) & 31u);
  const int c4 = c3 + ((cnt >> 15) & 31u), c5 = c4 + ((cnt >> 20) & 31u), c6 = c5 + ((cnt >> 25) & 31u);
  Sites4 out = {{0u, 0u, 0u, 0u}};
  const Sites4 zero = {{0u, 0u, 0u, 0u}};
  nat_apply(out, zero, w1, pg, 0, c1);
  nat_apply(out, w1, w2, pg, c1, c2);
  nat_apply(out, w2, w3, pg, c2, c3);
  nat_bcast(out, w1, pg, c3, c4);
  nat_bcast(out, w2, pg, c4, c5);
  nat_bcast(out, w3, pg, c5, c6);
  return out;
}

// The same words bit by bit, at one site: groups whose sources span more than
// the window, and buffers that are not aligned to 16-byte vectors.
__device__ __forceinline__ uint32_t nat_bits(const uint32_t* old, const uint32_t* src, int N, int nb) {
  uint32_t w = 0u;
#pragma unroll 4
  for (int bb = 0; bb < nb; ++bb) {
    const uint32_t lin = src[bb];
    w |= ((__ldg(old + (size_t)(lin >> 5) * N) >> (lin & 31u)) & 1u) << bb;
  }
  return w;
}

__device__ __forceinline__ void async_copy16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
               : "memory");
}
__device__ __forceinline__ void async_copy8(void* smem, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
               : "memory");
}
// all but the youngest `ahead` (< kNatAhead) commits have landed
__device__ __forceinline__ void async_wait(int ahead) {
  static_assert(kNatAhead == 4, "one case per count");
  if (ahead >= 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
  else if (ahead == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
  else if (ahead == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else asm volatile("cp.async.wait_group 0;" ::: "memory");
}

__global__ void __launch_bounds__(kNatThreads, kNatBlocksPerSM) msc_resample_native_kernel(BatchDev* b) {
  __shared__ __align__(16) uint4 s_rows[kNatThreads / 32][kNatRing][32];
  __shared__ __align__(16) uint2 s_lists[kNatThreads / 32][kNatLists][kMsb];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int total = b->res_prefix[b->npop];
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < total; u += nwarps) {
    int lo = 0, hi = b->npop;  // population of unit u (warp-uniform)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (b->res_prefix[mid] <= u) lo = mid;
      else hi = mid;
    }
    const PopDev* st = b->pops + lo;
    const int N = st->N, Rn = st->R_cur, rgn = (Rn + kMsb - 1) / kMsb, nstrip = (N + kNatSites - 1) / kNatSites;
    const int per = nat_groups(N, rgn);
    const int loc = u - b->res_prefix[lo], tile = loc / nstrip, strip = loc - tile * nstrip;
    const int j0 = tile * per, ng = min(per, rgn - j0);
    const int t = strip * kNatSites + 4 * lane;  // N is a multiple of 4: all four sites exist, or none
    const bool tv = t < N;
    const uint32_t* old = (const uint32_t*)st->spins[st->parity ^ 1] + t;  // this lane's first site in old group 0
    uint32_t* neu = (uint32_t*)st->spins[st->parity] + (size_t)j0 * N + t;
    const uint32_t* src = st->src + (size_t)j0 * kMsb;
    const uint2* pairs = st->res_pairs + (size_t)j0 * kMsb;
    const int gmax = st->rgcap - 1;
    if (strip == 0) {  // active flags: lane = bit
      uint8_t* act = st->active[st->parity];
      for (int g = 0; g < ng; ++g) act[(j0 + g) * kMsb + lane] = ((j0 + g) * kMsb + lane) < Rn ? 1 : 0;
    }
    if ((((uintptr_t)old | (uintptr_t)neu) & 15) != 0) {  // warp-uniform: t and N are multiples of 4
      for (int g = 0; g < ng && tv; ++g)
        for (int k = 0; k < 4; ++k)
          neu[(size_t)g * N + k] = nat_bits(old + k, src + g * kMsb, N, min(kMsb, Rn - (j0 + g) * kMsb));
      continue;
    }
    // lane g < ng: count word, first row and its place in the ring's sequence
    // of group j0 + g (a group adds the rows past the previous group's last)
    uint32_t cnt_l = 0u;
    int first_l = 0;
    if (lane < ng) {
      cnt_l = st->res_cnt[j0 + lane];
      first_l = (int)(src[lane * kMsb] >> 5);
    }
    const int before = __shfl_up_sync(kFull, first_l, 1);
    int seq_l = lane > 0 && lane < ng ? min(first_l - before, 3) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFull, seq_l, o);
      if (lane >= o) seq_l += v;
    }
    __syncwarp();  // the previous unit is done with the lists
    int issued = 0;
#pragma unroll 1
    for (int g = 0; g < ng; ++g) {
      const int sg = __shfl_sync(kFull, seq_l, g);
      // loads of the groups ahead while the ring has room behind this window
      for (; issued < ng && issued - g < kNatAhead; ++issued) {
        const int si = __shfl_sync(kFull, seq_l, issued), fi = __shfl_sync(kFull, first_l, issued);
        if (si + 2 - sg >= kNatRing) break;
        const int have = issued > 0 ? __shfl_sync(kFull, seq_l, issued > 0 ? issued - 1 : 0) + 3 : 0;
#pragma unroll
        for (int r = 0; r < 3; ++r)  // (rows past the buffer are never selected by a mask)
          if (si + r >= have && tv)
            async_copy16(&s_rows[wid][(si + r) & (kNatRing - 1)][lane], old + (size_t)min(fi + r, gmax) * N);
        async_copy8(&s_lists[wid][issued & (kNatLists - 1)][lane], pairs + issued * kMsb + lane);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      async_wait(issued - g - 1);
      __syncwarp();  // the whole list has landed
      const uint32_t cnt = __shfl_sync(kFull, cnt_l, g);
      Sites4 out;
      if (cnt >> 31) {  // sources beyond the window (warp-uniform)
        for (int k = 0; k < 4; ++k)
          out.w[k] = tv ? nat_bits(old + k, src + g * kMsb, N, min(kMsb, Rn - (j0 + g) * kMsb)) : 0u;
      } else {
        out = nat_words(sites(s_rows[wid][sg & (kNatRing - 1)][lane]), sites(s_rows[wid][(sg + 1) & (kNatRing - 1)][lane]),
                        sites(s_rows[wid][(sg + 2) & (kNatRing - 1)][lane]), s_lists[wid][g & (kNatLists - 1)], cnt);
      }
      if (tv) *reinterpret_cast<uint4*>(neu + (size_t)g * N) = make_uint4(out.w[0], out.w[1], out.w[2], out.w[3]);
    }
  }
}

// -------------------------------------------------------------- geometry
// A work unit is a tile of G groups whose lattices are stacked into G*L
// sublattice rows; every pass of a half-sweep updates rpp of those rows with
// Wr threads each.  G is chosen to fill the thread slots of whole kKB-site
// batches: small lattices (L=16: 128 words per half-sweep) would otherwise
// leave most of a 256-thread CTA idle.
static double msc_fill(int L, int G, int* rpp, int* npass) {
  const int Wr = L / 2, VR = G * L;
  int r = kSweepThreads / Wr;
  if (r > VR) r = VR;
  const int np = (VR + r - 1) / r, padded = (np + kKB - 1) / kKB * kKB;
  *rpp = r;
  *npass = np;
  return (double)VR * Wr / ((double)padded * kSweepThreads);
}

bool msc_geom(int L, SweepGeom* g, int tile, long long groups, int slots) {
  if (L < 8 || L % 2 != 0 || L > 128) return false;
  g->L = L;
  g->N = L * L;
  g->half = g->N / 2;
  g->Wr = L / 2;
  // G > 1 moves each sublattice with 16-byte vectors (h % 4 == 0) and keeps
  // the tile's lattices, without their prefix tables, small enough for four
  // resident CTAs per SM
  auto allowed = [&](int G) {
    return G == 1 || (G == 2 || G == 4 || G == kMaxTile) && g->half % 4 == 0 && G * g->N * 4 <= kTileSmemMax;
  };
  int best_G = 1, rpp = 0, npass = 0;
  if (tile > 0) {
    if (!allowed(tile)) return false;
    best_G = tile;
  } else if (groups > 0 && slots > 0) {
    // automatic, by a cost model: waves of work units over the resident
    // CTAs times the thread slots one unit occupies per half-sweep (whole
    // kKB-site batches), with the stacking arithmetic of G > 1 counted as
    // 7% more work (the measured gap at equal fill)
    auto cost = [&](int G) {
      int r, np;
      msc_fill(L, G, &r, &np);
      const double waves = std::max(1.0, (double)((groups + G - 1) / G) / slots);
      return waves * ((np + kKB - 1) / kKB * kKB) * (G > 1 ? 1.07 : 1.0);
    };
    double best = cost(1);
    for (int G = 2; G <= kMaxTile; G *= 2) {
      if (!allowed(G)) continue;
      const double c = cost(G);
      if (c < best - 1e-9) {
        best = c;
        best_G = G;
      }
    }
  }
  g->G = best_G;
  msc_fill(L, best_G, &rpp, &npass);
  g->rpp = rpp;
  g->T = g->Wr * rpp;
  g->npass = npass;
  g->kconst = (g->half % kRefThreads == 0) ? g->half / kRefThreads : 0;
  g->smem = msc_unit_layout(L, g->Wr, best_G, (npass + kKB - 1) / kKB).bytes;
  return true;
}

// -------------------------------------------------------------- launchers
int msc_kind(const SweepGeom& g) {
  if (g.G == 1 && g.L == 96) return kMixed;
  if (g.npass == 1 || (g.G == 1 && (g.L == 64 || g.L == 128))) return kCommon;
  return g.npass <= kKB ? kOneBatch : kGeneral;
}

int msc_kinds(int a, int b) { return a == b ? a : a == kMixed || b == kMixed ? kMixed : kCommon; }

using MscSweepFn = void (*)(BatchDev*, int, unsigned long long, int);
static MscSweepFn msc_sweep_fn(int rng_mode, int kind) {
  if (rng_mode == kRefCoords) return msc_sweep_kernel<kRefCoords, kGeneral>;
  switch (kind) {
    case kOneBatch: return msc_sweep_kernel<kNative, kOneBatch>;
    case kCommon: return msc_sweep_kernel<kNative, kCommon>;
    case kMixed: return msc_sweep_kernel<kNative, kMixed>;
    default: return msc_sweep_kernel<kNative, kGeneral>;
  }
}

cudaError_t msc_sweep_setup(int rng_mode, int smem, SweepLaunch* out, int kind) {
  out->kind = kind;
  return persistent_launch((const void*)msc_sweep_fn(rng_mode, kind), kSweepThreads, smem, out);
}

cudaError_t launch_msc_sweep(BatchDev* b, int rng_mode, int energy_only, unsigned long long seed,
                             const SweepLaunch& sl, cudaStream_t s) {
  msc_sweep_fn(rng_mode, sl.kind)<<<sl.grid, sl.block, sl.smem, s>>>(b, energy_only, seed, sl.nsm);
  return cudaGetLastError();
}

cudaError_t launch_msc_init(PopDev* pops, int npop, cudaStream_t s) {
  msc_init_kernel<<<dim3(256, npop), 256, 0, s>>>(pops);
  return cudaGetLastError();
}

cudaError_t launch_msc_resample(BatchDev* b, int rng_mode, cudaStream_t s) {
  int dev, nsm;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e;
  if (rng_mode == kRefCoords) {
    msc_resample_kernel<<<nsm * kResampleBlocksPerSM, kResampleThreads, 0, s>>>(b);  // persistent warps
    return cudaGetLastError();
  }
  msc_pairs_kernel<<<nsm * 8, 256, 0, s>>>(b);  // a warp per new group, grid-stride
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  msc_resample_native_kernel<<<nsm * kNatBlocksPerSM, kNatThreads, 0, s>>>(b);
  return cudaGetLastError();
}

}  // namespace pa
