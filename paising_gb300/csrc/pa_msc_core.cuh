// pa_msc_core.cuh -- device building blocks of the multi-spin-coded sweeps
// (single-CTA and cluster variants): the bitsliced neighbour adder, the
// digit-serial acceptance for 32 replicas per word, per-population parameters
// and per-bit statistics.
#pragma once

#include <climits>

#include "pa_device.cuh"

namespace pa {
namespace msc {

constexpr uint32_t kLcgA = 1664525u;     // PAisingMSC.cu:53
constexpr uint32_t kLcgC = 1013904223u;  // PAisingMSC.cu:54
constexpr uint32_t kFull = 0xffffffffu;
constexpr int kKB = 4;  // word-sites per thread decided together (native stream)
constexpr int kMaxTile = 8;                // groups per work unit of the one-CTA sweep (one warp each at least)
constexpr int kDigits = 8;  // digits of a comparison decided by digit_step (finish_bit takes the rest)
constexpr int kTileSmemMax = 44 * 1024;    // shared memory of a tile of more than one group

// Bitsliced count of anti-parallel neighbours (4 inputs -> 3 bit planes),
// the adder of PAisingMSC.cu:212-218.
__device__ __forceinline__ void adder4(uint32_t I1, uint32_t I2, uint32_t I3, uint32_t I4, uint32_t& s0,
                                       uint32_t& s1, uint32_t& s2) {
  const uint32_t x12 = I1 ^ I2, x34 = I3 ^ I4, a12 = I1 & I2, a34 = I3 & I4;
  s0 = x12 ^ x34;
  s1 = (x12 & x34) ^ a12 ^ a34;
  s2 = a12 & a34;
}

// Per-replica-bit sums over the words of a warp, for the energy epilogue.
// Each lane adds its words' four bonds and two spins into bitsliced counters
// (bit k of plane l holds bit l of the lane's running count for replica bit k)
// through full adders, four words at a time: two logic operations per bit
// added, and one carry to ripple through the upper planes per four words.  The
// warp's sum is a butterfly of bitsliced additions, energies on the lower half
// warp and spins on the upper, with as many planes as the counts need.
// What bounds it is the number of logic operations: a word added alone rippled
// through every plane (95 instructions) and fifteen 32 x 32 transpositions made
// the warp's sums (460); now about 40 and 140-200.  A launch of energies alone,
// L = 32, 10^6 replicas: 240 -> 184 us, L = 64, 160000: 106 -> 78.  Eight planes hold the counts of up to
// 63 words per lane.
struct BondWord {
  uint32_t b[4], sA, sB;  // anti-parallel bonds, spins; all zero: no word
};
struct BitCounters {
  uint32_t e[8], m[8];
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int l = 0; l < 8; ++l) e[l] = m[l] = 0u;
  }
  // s += a + b, bit by bit: the sum stays, the carry is returned
  __device__ __forceinline__ static uint32_t full_add(uint32_t& s, uint32_t a, uint32_t b) {
    const uint32_t c = (s & a) | (b & (s | a));
    s = s ^ a ^ b;
    return c;
  }
  // c += x << at, bit by bit (ripple of half adders)
  __device__ __forceinline__ static void ripple(uint32_t (&c)[8], int at, uint32_t x) {
#pragma unroll
    for (int l = 0; l < 8; ++l)
      if (l >= at) {
        const uint32_t t = c[l] & x;
        c[l] ^= x;
        x = t;
      }
  }
  __device__ __forceinline__ void add(const BondWord (&w)[4]) {
    uint32_t g[2], o[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      uint32_t f[2], n[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const BondWord& x = w[2 * p + i];
        const uint32_t t = full_add(e[0], x.b[0], x.b[1]), u = full_add(e[0], x.b[2], x.b[3]);
        f[i] = full_add(e[1], t, u);
        n[i] = full_add(m[0], x.sA, x.sB);
      }
      g[p] = full_add(e[2], f[0], f[1]);
      o[p] = full_add(m[1], n[0], n[1]);
    }
    ripple(e, 4, full_add(e[3], g[0], g[1]));
    ripple(m, 3, full_add(m[2], o[0], o[1]));
  }
  // the planes' sums over the warp, of counts below 2^K: in the low half word
  // that of replica bit lane & 15, in the high one that of 16 more; of the
  // bonds in the lower half warp, of the spins in the upper
  template <int K>
  __device__ __forceinline__ uint32_t warp_sums(int lane) const {
    uint32_t p[K + 5], c = 0;
    const bool upper = (lane & 16) != 0;
#pragma unroll
    for (int l = 0; l < K; ++l) {
      p[l] = upper ? m[l] : e[l];
      c = full_add(p[l], __shfl_xor_sync(kFull, upper ? e[l] : m[l], 16), c);
    }
    p[K] = c;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      c = 0;
#pragma unroll
      for (int l = 0; l < K + 1 + s; ++l) c = full_add(p[l], __shfl_xor_sync(kFull, p[l], 8 >> s), c);
      p[K + 1 + s] = c;
    }
    uint32_t sum = 0;
#pragma unroll
    for (int l = 0; l < K + 5; ++l) sum += (p[l] >> (lane & 15) & 0x00010001u) << l;
    return sum;
  }
  // whole warp, at most `words` words per lane: adds the sums to cntE and cntM [replica bit]
  __device__ __forceinline__ void totals(int lane, int words, int* cntE, int* cntM) const {
    const uint32_t s = words <= 3 ? warp_sums<4>(lane) : words <= 7 ? warp_sums<5>(lane)
                       : words <= 15 ? warp_sums<6>(lane) : warp_sums<8>(lane);
    int* to = (lane & 16 ? cntM : cntE) + (lane & 15);
    atomicAdd(to, (int)(s & 0xFFFFu));
    atomicAdd(to + 16, (int)(s >> 16));
  }
};

// The two masks the acceptance needs from a word's four neighbour words:
// odd = an odd number of anti-parallel neighbours (among undecided bits: one,
// threshold T4), ge2 = two or more (dE <= 0: flipped outright) -- adder4's s0
// and s1 | s2.  Three neighbours through a full adder (sum x, carry m), then
// the fourth: flipping all inputs of a full adder flips its outputs, so the
// spin itself enters as m ^ s and x ^ s; five logic operations in all.
__device__ __forceinline__ void count_masks(uint32_t s, uint32_t n1, uint32_t n2, uint32_t n3, uint32_t n4,
                                            uint32_t& odd, uint32_t& ge2) {
  const uint32_t x = n1 ^ n2 ^ n3, m = (n1 & n2) | (n3 & (n1 | n2));
  odd = x ^ n4;
  ge2 = ((x ^ s) & (n4 ^ s)) | (m ^ s);
}

// One binary digit of the comparison U < T/2^32 done for 32 bits at once:
// U's digit j is bit i of the random word u for replica bit i, T's digit j
// is selected per bit from T4 (bits in s0: one anti-parallel neighbour,
// dE = 4) or T8 (no anti-parallel neighbour, dE = 8).  dg = digit_table(j)
// gives that selection as one multiply-add, p = s0 * dg.x + dg.y (see
// digit_table), on the FMA pipe.  Bits decided at this digit leave `und`;
// those decided "less" enter `lt`.  Both updates read und directly, so that
// consecutive digits are one logic operation apart in the chain of und: with
// the decided bits formed first and subtracted from und they were two, and
// L = 64 (8 populations of 20000, 100 sweeps) ran at 5405 instead of 5523
// attempts/ns.
__device__ __forceinline__ void digit_step(uint32_t u, uint32_t s0, uint32_t dx, uint32_t dy, uint32_t& und,
                                           uint32_t& lt) {
  const uint32_t p = s0 * dx + dy;
  lt += und & p & ~u;  // disjoint from the bits decided before
  und &= ~(p ^ u);
}

// Digit j of the thresholds T4, T8 as (m, c) with s0 * m + c = the bits'
// threshold digits: T4's digit where s0 is set, T8's elsewhere.  With D = all
// ones iff the digit is 1: both digits equal -> (0, D8); T4's 1, T8's 0 ->
// (1, 0) = s0; T4's 0, T8's 1 -> (-1, ~0) = ~s0.
__host__ __device__ inline uint2 digit_table(uint32_t T4, uint32_t T8, int j) {
  const uint32_t b4 = (T4 >> (31 - j)) & 1u, b8 = (T8 >> (31 - j)) & 1u;
  return make_uint2(b4 == b8 ? 0u : b4 ? 1u : 0xFFFFFFFFu, 0u - b8);
}

// The last undecided bits of a comparison word: their first 8 digits equal
// T's, so U < T/2^32 is decided by the remaining 24 digits at once,
// U mod 2^24 < T mod 2^24, with one fresh 32-bit word w per bit (its top 24
// bits are U's remaining digits): w < (T mod 2^24) * 2^8, compared against
// t4 = T4 << 8 and t8 = T8 << 8.  Takes the lowest undecided bit; a no-op
// when none is left.
__device__ __forceinline__ void finish_bit(uint32_t w, uint32_t am, uint32_t t4, uint32_t t8, uint32_t& und,
                                           uint32_t& lt) {
  const uint32_t b = und & (0u - und);
  const uint32_t t = (am & b) ? t4 : t8;
  // b is a bit of und and not yet of lt: the updates are additions, which
  // the FMA pipe can take (the sweep's logic operations keep the ALU pipe
  // the busier one)
  lt += w < t ? b : 0u;
  und -= b;
}

// Tag of the words that finish single bits (finish_bit): the sweep's tag with
// bit 29 flipped ('M' -> 'm', 'S' -> 's'), a stream of its own.
constexpr uint32_t kFinishTagFlip = 0x20u << 24;

// The uniform inputs of a half-sweep's draws: every block's counter is
// (site or chain, c1 | sub-draw, step, tag).
struct HalfSweep {
  uint32_t c1, step, tag, T4, T8;
  uint2 u0, u1;  // philox_uniform of c1 (heads, first finishing block) and of c1 | 1 (the tail's digits)
  template <class Keys>
  __device__ __forceinline__ HalfSweep(uint32_t c1_, uint32_t step_, uint32_t tag_, uint32_t T4_, uint32_t T8_,
                                       const Keys& K)
      : c1(c1_), step(step_), tag(tag_), T4(T4_), T8(T8_), u0(philox_uniform(c1_, step_, K)),
        u1(philox_uniform(c1_ | 1u, step_, K)) {}
};

// Remaining digits (from digit 4 on) of one 32-bit comparison word: digits
// 4..7 of every bit from one Philox block, digits() (counter (c0, c1 | sub,
// step, tag)); the few bits still undecided after them (1/16 of those
// entering) are finished one at a time by finish_bit, four per Philox block,
// first() and then more(k) (counter (c0, c1 | (fsub + k), step, tag ^
// kFinishTagFlip), k = 0..7, enough for all 32 bits).  Returns the bits
// decided "less".
template <class Digits, class First, class More>
__device__ __forceinline__ uint32_t finish_digits(uint32_t und, uint32_t am, const uint4* dig, uint32_t T4, uint32_t T8,
                                                  const Digits& digits, const First& first, const More& more) {
  // no vote first: some lane of the warp nearly always has undecided bits
  // here (and the overflow path only calls when one has); a lane without
  // them is left unchanged by every step below
  uint32_t lt = 0;
  {
    const uint4 d45 = dig[2], d67 = dig[3];
    const U4 r = digits();
    digit_step(r.x, am, d45.x, d45.y, und, lt);
    digit_step(r.y, am, d45.z, d45.w, und, lt);
    digit_step(r.z, am, d67.x, d67.y, und, lt);
    digit_step(r.w, am, d67.z, d67.w, und, lt);
  }
  const uint32_t t4 = T4 << 8, t8 = T8 << 8;
  // the first block and two of its words without a vote either: nearly every
  // warp has a lane with a bit left after digit 7 and most have one with two;
  // a third in some lane is rarer (a third of the warps at half a bit per
  // lane), so the other two words are behind a vote (1-2% of the sweep)
  U4 r = first();
#pragma unroll 1
  for (uint32_t k = 1;; ++k) {
    finish_bit(r.x, am, t4, t8, und, lt);
    finish_bit(r.y, am, t4, t8, und, lt);
    if (!__any_sync(kFull, und != 0u)) break;
    finish_bit(r.z, am, t4, t8, und, lt);
    finish_bit(r.w, am, t4, t8, und, lt);
    if (k == 8u || !__any_sync(kFull, und != 0u)) break;
    r = more(k);
  }
  return lt;
}

// Exact Metropolis decisions U < T/2^32 for kKB word-sites of one thread.
// Head: digits 0..3 of every site come from the site's own Philox block;
// after them only ~1/16 of the bits are undecided.  Tail: those sparse bits
// of the kKB sites are merged into one word, site k's masks rotated by rot_k
// so that every (site, replica) pair gets its own bit position -- hence its
// own fresh digits -- and the remaining digits are drawn once for all sites.
// A site whose bits find no free rotation is finished on its own.
//   a[k]   : bits with one anti-parallel neighbour (threshold T4), else T8
//   und[k] : bits needing a random decision (consumed)
//   acc[k] : accepted bits (in: outright accepts; out: all accepts)
//   nvalid : block-uniform count of the leading slots that hold sites; the
//            other slots have und = 0 and draw nothing
//   K      : PhiloxKeys or PhiloxKeysWide (the same stream, two code forms)
//   site_pre(k), chain_pre(f): the prefixes (philox_prefix or _prefix4) of
//            site k's block and of the chain's digit block (f = 0) and first
//            finishing block (f = 1) -- read from a table made for the
//            temperature where the shared memory allows one, else formed on
//            the spot
// What bounds it: instruction issue on two pipes.  A Philox round is two
// 64-bit products (4 cycles each of an SM sub-partition's FMA pipe, and with
// two or more logic operations beside it 2 of the ALU pipe's) and two logic
// operations (2 cycles each of the ALU pipe); a batch draws six blocks of ten
// rounds, and its digits, merging and neighbour counts fill the ALU pipe
// about as much.  The prefixes take two of the ten rounds out of every block
// where a table holds them, the uniforms the c1 halves of the next two.  One
// GB300, 100 sweeps, attempts/ns before (no prefixes, uniforms per batch, the
// earlier digit step and finish) -> now: L = 64, 8 x 20000 5403 -> 5975 (6115
// with the later epilogue and tables), one population on clusters of 2 4281 ->
// 4726; L = 128 (no table) 5181 -> 5570; L = 256 (chain table) 4764 -> 5075; SSC
// bit planes L = 64 4434 -> 4874.
// Tables of L = 96 and 128 kept in global memory gained nothing (L2 reads in
// place of the products: 96 +2%, 128 -1%).
//   NV     : slots in use (a batch of fewer than kKB sites)
//   SIDE   : all blocks are drawn first, side by side: for launches whose few
//            warps wait for a chain of rounds, not for the pipes
template <int NV = kKB, bool SIDE = false, class Keys, class SitePre, class ChainPre>
__device__ __forceinline__ void accept_native(const uint32_t (&a)[kKB], uint32_t (&und)[kKB], uint32_t (&acc)[kKB],
                                              const uint32_t (&site)[kKB], uint32_t chain, const HalfSweep& hs,
                                              const Keys& K, const uint4* dig, int nvalid, const SitePre& site_pre,
                                              const ChainPre& chain_pre) {
  const uint4 d01 = dig[0], d23 = dig[1];
  auto digits = [&](int k, const U4& r) {
    digit_step(r.x, a[k], d01.x, d01.y, und[k], acc[k]);
    digit_step(r.y, a[k], d01.z, d01.w, und[k], acc[k]);
    digit_step(r.z, a[k], d23.x, d23.y, und[k], acc[k]);
    digit_step(r.w, a[k], d23.z, d23.w, und[k], acc[k]);
  };
  auto head = [&](int k) { return philox10_prefixed(site[k], site_pre(k), hs.u0, K); };
  auto tail = [&]() { return philox10_prefixed(chain, chain_pre(0), hs.u1, K); };
  auto first = [&]() { return philox10_prefixed(chain, chain_pre(1), hs.u0, K); };
  U4 rd, rf;
  if constexpr (SIDE) {
    U4 r[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) r[k] = head(k);
    rd = tail();
    rf = first();
#pragma unroll
    for (int k = 0; k < NV; ++k) digits(k, r[k]);
  } else if (nvalid >= NV) {
    // independent Philox chains of the sites, interleaved by the compiler
#pragma unroll
    for (int k = 0; k < NV; ++k) digits(k, head(k));
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (k < nvalid) digits(k, head(k));
  }
  uint32_t m = und[0], am = a[0] & und[0];
  uint32_t rot[NV];
  rot[0] = 0;
  uint32_t ovf = 0;
#pragma unroll
  for (int k = 1; k < NV; ++k) {
    uint32_t r = 0;
    while (r < 32u && (m & __funnelshift_l(und[k], und[k], r))) ++r;
    rot[k] = r;
    if (r < 32u) {  // disjoint from the bits merged so far: additions, on the FMA pipe
      m += __funnelshift_l(und[k], und[k], r);
      am += __funnelshift_l(a[k] & und[k], a[k] & und[k], r);
    } else {
      ovf |= 1u << k;
    }
  }
  const uint32_t ftag = hs.tag ^ kFinishTagFlip;
  auto more = [&](uint32_t k) { return philox10k(chain, hs.c1 | k, hs.step, ftag, K); };
  uint32_t lt;
  if constexpr (SIDE) {
    lt = finish_digits(m, am, dig, hs.T4, hs.T8, [&]() { return rd; }, [&]() { return rf; }, more);
  } else {
    lt = finish_digits(m, am, dig, hs.T4, hs.T8, tail, first, more);
  }
  acc[0] |= lt & und[0];
#pragma unroll
  for (int k = 1; k < NV; ++k)
    if (!(ovf >> k & 1u)) acc[k] |= __funnelshift_r(lt, lt, rot[k]) & und[k];
  if (NV > 1 && __any_sync(kFull, ovf != 0u)) {  // rare: one vote for the other sites
#pragma unroll
    for (int k = 1; k < NV; ++k)
      if (__any_sync(kFull, ovf >> k & 1u))
        acc[k] |= finish_digits(
            (ovf >> k & 1u) ? und[k] : 0u, a[k] & und[k], dig, hs.T4, hs.T8,
            [&]() { return philox10k(site[k], hs.c1 | 8u, hs.step, hs.tag, K); },
            [&]() { return philox10k(site[k], hs.c1 | 8u, hs.step, ftag, K); },
            [&](uint32_t j) { return philox10k(site[k], hs.c1 | (8u + j), hs.step, ftag, K); });
  }
}

// One-group work units keep each sublattice in shared memory as L + 2 rows of
// Wr words (row -1 and row L are periodic copies); sublattice B's block
// starts at this word offset (A's block rounded up to 16 bytes).
__host__ __device__ constexpr int msc_halo_block(int L, int Wr) { return ((L + 2) * Wr + 3) & ~3; }

// Prefix tables of a work unit (native stream), in shared memory behind its
// lattice: 8 bytes per word of a sublattice (both sublattices number their
// sites alike; only c1 tells their draws apart) and 16 per chain, formed when
// the unit is loaded and read in every half-sweep.
struct TableLayout {
  int tab, ctab, bytes;  // word offsets of the two tables (0: none), shared memory of lattice and tables
};
// lat_words: the lattice's words; sites, chains: entries; max_bytes: what the
// unit may take without fewer resident CTAs.  Both tables where they fit, the
// chains' alone (two of a batch's six blocks for a third of the bytes) where
// only that does, else none.
__host__ __device__ constexpr TableLayout table_layout(int lat_words, int sites, int chains, int max_bytes) {
  const int at = (lat_words + 3) & ~3, site_words = (2 * sites + 3) & ~3;
  if ((at + site_words + 4 * chains) * 4 <= max_bytes)
    return TableLayout{at, at + site_words, (at + site_words + 4 * chains) * 4};
  if ((at + 4 * chains) * 4 <= max_bytes) return TableLayout{0, at, (at + 4 * chains) * 4};
  return TableLayout{0, 0, lat_words * 4};
}

// Per-population parameters of the group a CTA is annealing.  They live in
// shared memory and are read where used, which keeps the hot loops' register
// footprint independent of how many populations the batch holds.
struct UnitParams {
  int L, N, h, Wr, rpp, npass, kconst, step, sweeps, nbatch;
  int G, rg;                    // groups per tile, groups in the population
  int sb;                       // one-group units: word offset of sublattice B's block in shared memory
  int tab, ctab;                // word offsets of the prefix tables of sites and chains in shared memory, 0: none
  uint32_t invL, invWr, invH4;  // reciprocals (recip32) of L, Wr and h/4
  uint32_t tag, T4, T8;
  unsigned long long seed, iseq;
  uint32_t* words;
  const uint8_t* act;
  int32_t* E;
  int32_t* M;
};

// Shared memory of a one-CTA work unit of G groups: the lattice, and the
// prefix tables where three CTAs per SM still fit beside each other (76 KB
// each of an SM's 228 KB, 1 KB of it the system's and up to 5 KB this kernel's
// static arrays).  Three CTAs with tables beat four without: the pipes are the
// limit, and three keep them nearly as busy.  Against tables for four CTAs
// (51 KB): L = 48 1.045x, 72 and 80 1.023x, 96 (the chains' table) 1.026x, 128
// (none either way) 1.000x, 16 populations of L = 8..64 1.029x; tables for two
// CTAs (108 KB) lose 2-6% at all of them.
constexpr int kUnitSmemMax = 70 * 1024;
__host__ __device__ constexpr TableLayout msc_unit_layout(int L, int Wr, int G, int nbatch) {
  // one group: row L (the copy below row L-1) has entries of its own, read by slots past the lattice
  return G == 1 ? table_layout(msc_halo_block(L, Wr) + (L + 2) * Wr, (L + 1) * Wr, nbatch * kSweepThreads, kUnitSmemMax)
                : table_layout(2 * G * L * Wr, G * L * Wr, nbatch * kSweepThreads, kUnitSmemMax);
}

// Statistics of the groups a CTA annealed for one population, accumulated in
// shared memory by lane k of warp 0 for replica bit k (registers stay free
// for the sweep); flushed to the population when the CTA moves on.
struct BitStats {
  long long sE[kMsb], sE2[kMsb], sM[kMsb], sM2[kMsb];
  unsigned long long m4lo[kMsb], m4hi[kMsb];
  int emin[kMsb];
  __device__ void reset(int k) {
    sE[k] = sE2[k] = sM[k] = sM2[k] = 0;
    m4lo[k] = m4hi[k] = 0;
    emin[k] = INT_MAX;
  }
  __device__ void add(int k, int E, int Mg) {
    const long long am = Mg < 0 ? -(long long)Mg : (long long)Mg;
    sE[k] += E;
    sE2[k] += (long long)E * E;
    sM[k] += am;
    sM2[k] += am * am;
    unsigned long long lo, hi;
    m4_of(Mg, lo, hi);
    U128 m{m4lo[k], m4hi[k]};
    u128_add(m, lo, hi);
    m4lo[k] = m.lo;
    m4hi[k] = m.hi;
    emin[k] = E < emin[k] ? E : emin[k];
  }
  // warp 0 only, lane k = bit k
  __device__ void flush(PopDev* st, int k) {
    const long long e = warp_sum(sE[k]), e2 = warp_sum(sE2[k]), m = warp_sum(sM[k]), m2 = warp_sum(sM2[k]);
    const int mn = warp_min(emin[k]);
    U128 q{m4lo[k], m4hi[k]};
    for (int o = 16; o > 0; o >>= 1) {  // 128-bit sum across the warp, carries into hi
      const unsigned long long lo = __shfl_xor_sync(kFull, q.lo, o);
      const unsigned long long hi = __shfl_xor_sync(kFull, q.hi, o);
      u128_add(q, lo, hi);
    }
    if (k == 0 && mn != INT_MAX) {
      atomicAdd((unsigned long long*)&st->sE, (unsigned long long)e);
      atomicAdd((unsigned long long*)&st->sE2, (unsigned long long)e2);
      atomicAdd((unsigned long long*)&st->sM, (unsigned long long)m);
      atomicAdd((unsigned long long*)&st->sM2, (unsigned long long)m2);
      u128_atomic_add(&st->sM4lo, &st->sM4hi, q.lo, q.hi);
      atomicMin(&st->Emin_acc, mn);
    }
    reset(k);
  }
};

}  // namespace msc
}  // namespace pa
