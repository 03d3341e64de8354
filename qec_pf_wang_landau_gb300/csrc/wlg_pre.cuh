// The pre-run's histogram-biased walk (wl.cu:473-560), shared by the batched
// pre-run and the pre-run operator: one CTA per sample, one thread per walker.
//
// Rounds are synchronous: every walker decides on the histogram as the round
// before left it, then all increments land, and each still-empty coarse bin
// takes the lattice of the lowest-index walker that entered it.
//
//   * one barrier a round: the histogram is kept twice.  In round r walkers
//     read copy r & 1 and add their visits of rounds r - 1 and r to the other,
//     which nobody reads before the barrier;
//   * a claim on a coarse bin is the key (round + 1) << 10 | walker under
//     atomicMin, so no later round undercuts it; the winner's lattice is
//     stored after the next barrier;
//   * the histogram has an entry per energy the lattice can have (every 2nd or
//     4th), or its loads and atomics would share 8 of the 32 banks;
//   * lattices are kept as unsatisfied bonds, a row of right bonds and of down
//     bonds in one word (up to 16 columns) or two (up to 32), [word][walker],
//     plus the spin of site 0: a proposal reads two or three words and no
//     couplings, and is prepared before the barrier;
//   * acceptance u < exp(H[old] - H[new]) needs no exp: the draw alone gives
//     the largest count difference it accepts (accept_limit).
//
// What bounds it is one round's latency with one warp on an SM partition:
// barrier, histogram loads, decision, lattice words, energy change (about 110
// warp instructions; the Philox block, the next site and its tables run beside
// them, and rare cases sit in one warp-uniform block so that nothing else
// branches).  GB300, 128 walkers a sample, time per round, against int8 lattices
// with 64-bit counts, an acceptance table read after the histogram and two
// barriers: 24x24 1.09 -> 0.18 us, 16x16 1.12 -> 0.16 us; 120 uneven lattices of
// 4-16 a side 27.3 -> 4.4 ms; the operator, 64 samples of 9x9, 1000 rounds, with
// set-up 2.05 -> 0.28 ms.  On the way: branches around site fallback and claims
// 0.40 us a round; a branch in the barrier, around the lattice stores and a load
// of the claim each round 0.26; a histogram entry per energy value 0.21.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "wlg_accept.cuh"
#include "wlg_engine.h"
#include "wlg_rng.cuh"

namespace wlg {
namespace {

// Site of a draw: trunc(double(u) * ((N-1) + 0.999999)) (wl.cu:63-65).  With
// f = x / 2^32 the reference's product lies within N*2^-23 + 1e-6 of f*N, so
// floor(f*N) = umulhi(x, N) is exact unless the fraction x*N mod 2^32 lies
// within site_thr (= 2^32 (N 2^-21 + 2^-18), >= 4x that bound) of an
// integer; there the reference's own float/double expression below decides.
// Out of line: inlined, its FP64 multiply and conversions would be scheduled
// into every step.
__device__ __noinline__ int site_exact(uint32_t x, double scale)
{
  return static_cast<int>(trunc(static_cast<double>(unit_float(x)) * scale));
}

// acc_thr[t], t <= 24: the least 32-bit draw whose uniform reaches the device's
// exp(-t) (uniforms are monotone in the draw); 0 beyond, where exp(-t) < 2^-33
// <= u.  The draw x accepts a count difference H[new] - H[old] = t exactly when
// x < acc_thr[t] (wl.cu:536-537); a negative one always (exp(1) > 1 >= u).
__device__ __forceinline__ void fill_accept(uint32_t* acc_thr, int tid)
{
  if (tid >= kAcceptEntries) return;
  if (tid > 24) {
    acc_thr[tid] = 0;
    return;
  }
  const double e = exp(static_cast<double>(-tid));
  unsigned long long lo = 0, hi = 1ull << 32;
  while (lo < hi) {
    const unsigned long long mid = (lo + hi) >> 1;
    if (static_cast<double>(unit_float(static_cast<uint32_t>(mid))) >= e) hi = mid;
    else lo = mid + 1;
  }
  acc_thr[tid] = static_cast<uint32_t>(lo);  // <= 2^32 - 128: u reaches 1 there
}

// The largest t >= 0 with x < acc_thr[t], or -1.  -log u names it up to one.
__device__ __noinline__ int accept_limit(uint32_t x, const uint32_t* acc_thr)
{
  const int k = max(static_cast<int>(-log_uniform(x)), 0);
  return k - 1 + (x < acc_thr[k] ? 1 : 0) + (x < acc_thr[k + 1] ? 1 : 0);
}

struct PreSync {
  int threads;
  __device__ __forceinline__ void operator()() const { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }
};

// A store under a predicate; without it the compiler branches around a pair.
__device__ __forceinline__ void store_if(bool p, uint32_t* a, uint32_t v)
{
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.u32 [%1], %2;\n\t}" ::"r"(
                 static_cast<uint32_t>(p)),
               "r"(static_cast<uint32_t>(__cvta_generic_to_shared(a))), "r"(v)
               : "memory");
}

// A sample's walk: where its pieces lie and its parameters.
struct PreWalk {
  int X, Y, boundary;
  int e_min, lg;       // lowest energy a walker can have in the range; energies lie 2^lg apart
  int len;             // such energies in the range
  int stride;          // words from one copy of the histogram to the other, more than len
  int bin0;            // e_min above the first coarse bin's edge
  int n_int, len_int, n_iter;
  int threads;         // walkers, rounded up to a warp
  uint32_t* hist;      // [2][stride], both copies the same
  uint32_t* claim;     // [n_int]: kPreEmpty, the winner's key, or 0 (stored before the walk)
  int* found_E;        // [n_int] energy of the stored lattice
  const uint32_t* acc_thr;
  const uint2* col;    // [Y] {bits of the column's bonds, its missing bonds}
  const uint4* row;    // [X] {masks of the bonds in its word(s) and in the row above, missing bonds}
  const uint32_t *Jr, *Jd;  // [X] coupling bits
  uint32_t* words;     // [X][1 or 2][threads]
  int8_t* found_lat;   // global [n_int][N]
};

constexpr uint32_t kPreEmpty = 0xFFFFFFFFu;

// Tables of the bonds of each column and row.  One word: right bonds in bits
// 0-15, down bonds in bits 16-31; two words: col.x holds the right bonds.
template <bool kTwo>
__device__ __forceinline__ void fill_bonds(uint2* col, uint4* row, int X, int Y, int boundary, int tid, int threads)
{
  const bool open = boundary != 0;
  for (int j = tid; j < Y; j += threads) {
    uint32_t h = (1u << j) | (1u << (j == 0 ? Y - 1 : j - 1));
    if (open) h &= ~(1u << (Y - 1));
    const uint32_t miss = open ? (j == 0 ? 1u : 0u) + (j == Y - 1 ? 1u : 0u) : 0u;
    col[j] = make_uint2(kTwo ? h : h | 0x10000u << j, miss);
  }
  for (int i = tid; i < X; i += threads) {
    const bool up = !open || i > 0, dn = !open || i < X - 1;
    row[i] = make_uint4(dn ? 0xFFFFFFFFu : (kTwo ? 0u : 0x0000FFFFu), up ? (kTwo ? 0xFFFFFFFFu : 0xFFFF0000u) : 0u,
                        (up ? 0u : 1u) + (dn ? 0u : 1u), 0u);
  }
}

// Word(s) of row i from its spin bits and those of the row below.
template <bool kTwo>
__device__ __forceinline__ void bond_words(uint32_t r, uint32_t dn, uint32_t Jr, uint32_t Jd, int Y, bool open, bool last,
                                           uint32_t& h, uint32_t& v)
{
  const uint32_t all = Y == 32 ? 0xFFFFFFFFu : (1u << Y) - 1u;
  h = (r ^ ((r >> 1) | ((r & 1u) << (Y - 1))) ^ Jr) & all;
  v = (r ^ dn ^ Jd) & all;
  if (open) {
    h &= ~(1u << (Y - 1));
    if (last) v = 0;
  }
  if constexpr (!kTwo) h |= v << 16;
}

// Spins of walker `w` (of this warp) as +-1 bytes, written by the warp's lanes
// row by row: along column 0 and then along the row, a bond flips the spin when
// coupling bit and unsatisfied bit differ.  s0: site 0's spin bit.
template <bool kTwo>
__device__ __noinline__ void store_spins(const PreWalk& p, int w, uint32_t s0, int8_t* dst)
{
  constexpr int kW = kTwo ? 2 : 1;
  for (int i = static_cast<int>(threadIdx.x & 31u); i < p.X; i += 32) {
    uint32_t s = s0;
    for (int k = 0; k < i; ++k) {
      const uint32_t v = kTwo ? p.words[(k * kW + 1) * p.threads + w] : p.words[k * p.threads + w] >> 16;
      s ^= (v ^ p.Jd[k]) & 1u;
    }
    const uint32_t turn = p.words[i * kW * p.threads + w] ^ p.Jr[i];
    for (int j = 0; j < p.Y; ++j) {
      dst[i * p.Y + j] = s != 0 ? -1 : 1;
      s ^= (turn >> j) & 1u;
    }
  }
}

template <int kC>
struct Copy {
  static constexpr int value = kC;
};

// The walk of this thread's walker `w` (live: it exists).  E, s0 and pos (draws
// consumed, even) are updated; kRange: a proposal outside the range
// stops the walker (wl.cu:522-529) and leaves its energy in E.  Every thread of
// the CTA's first p.threads calls it.  On return both copies of the histogram
// hold all visits.
template <bool kTwo, bool kRange, bool kKeys>
__device__ __forceinline__ void pre_walk(const PreWalk& p, const PreSync& sync, int w, bool live, uint64_t key,
                                         uint64_t subseq, uint64_t& pos, int& E, uint32_t& s0)
{
  constexpr int kW = kTwo ? 2 : 1;
  const int T = p.threads, X = p.X, Y = p.Y, N = X * Y;
  const int Lh = p.stride, lg = p.lg;
  const int spare = Lh - 1;  // takes the visits of threads without a walker
  const uint32_t site_thr = static_cast<uint32_t>(N) * 2048u + 16384u;
  const double site_scale = (N - 1 + 0.999999);
  // n / len_int = umulhi(n, magic) for n < 2^15; len_int = 1 divides by itself
  const uint32_t len_magic = static_cast<uint32_t>((0xFFFFFFFFull + p.len_int) / p.len_int);
  const bool len_one = p.len_int == 1;
  const uint32_t k0 = static_cast<uint32_t>(key), k1 = static_cast<uint32_t>(key >> 32);
  const uint32_t s_lo = static_cast<uint32_t>(subseq), s_hi = static_cast<uint32_t>(subseq >> 32);
  uint32_t* lat = p.words + w;
  bool ok = live;
  if (kRange) ok = ok && E >= p.e_min && (E - p.e_min) >> lg < p.len;
  int io = ok ? (E - p.e_min) >> lg : spare;
  int hit_before = spare;
  int e_start = io;     // batched walk: the one bin visited without a move into it
  int want = -1;        // coarse bin claimed in the round before
  bool claims = false;  // a lane of this warp has one
  uint32_t claim_key = 1u << 10;  // of this round

  // The proposal under way: where it leads, the words it would write, the
  // largest count difference its draw accepts.
  int in = 0, wa = 0, wb = 0, wc = 0, limit = 0;
  uint32_t na = 0, nb = 0, nc = 0, first_site = 0;
  auto propose = [&](uint32_t i, uint32_t j) {
    const uint2 c = p.col[j];
    const uint4 m = p.row[i];
    const uint32_t iu = min(i - 1u, static_cast<uint32_t>(X) - 1u);
    first_site = (i | j) == 0 ? 1u : 0u;
    uint32_t unsat;
    wa = static_cast<int>(i) * kW * T;
    if constexpr (kTwo) {
      wb = static_cast<int>(iu) * kW * T + T;
      wc = wa + T;
      na = lat[wa];
      nb = lat[wb];
      nc = lat[wc];
      const uint32_t b = 1u << j, mb = b & m.y, mc = b & m.x;
      unsat = __popc(na & c.x) + __popc(nb & mb) + __popc(nc & mc);
      na ^= c.x;
      nb ^= mb;
      nc ^= mc;
    } else {
      wb = static_cast<int>(iu) * T;
      na = lat[wa];
      nb = lat[wb];
      const uint32_t ma = c.x & m.x, mb = c.x & m.y;
      unsat = __popc(na & ma) + __popc(nb & mb);
      na ^= ma;
      nb ^= mb;
    }
    in = io + (2 * (4 - static_cast<int>(c.y + m.z) - 2 * static_cast<int>(unsat)) >> lg);
  };
  // Prepares the next round from its two draws, and claims the coarse bin of
  // this round's move when it is still empty (`key`: this round's).  What is
  // rare (a site next to a cell edge, a draw next to a threshold, an empty
  // bin) is settled in one warp-uniform block: the rest has no branch.
  // fresh: the bin moved into had no visit before this round.  In a batched walk
  // only such bins, and the one all walkers start in, can lie in an empty
  // coarse bin; the operator's histogram may hold earlier visits.
  auto prepare = [&](uint32_t x_site, uint32_t x_acc, bool moved, bool fresh, uint32_t key_now) {
    const uint64_t xi = static_cast<uint64_t>(x_site) * static_cast<uint32_t>(X);
    const uint64_t xj = static_cast<uint64_t>(static_cast<uint32_t>(xi)) * static_cast<uint32_t>(Y);
    const bool edge = static_cast<uint32_t>(xj) + site_thr < 2u * site_thr;
    propose(static_cast<uint32_t>(xi >> 32), static_cast<uint32_t>(xj >> 32));
    // the largest t with u < exp(-t), i.e. t < -log u, from the nearest integer
    const float v = -log_uniform(x_acc);
    const float big = v + 0x1.8p23f, away = v - (big - 0x1.8p23f);
    limit = __float_as_int(big) - 0x4B400000 - (away < 0.0f ? 1 : 0);
    const bool close = fabsf(away) < 2.0f * kLogAbsErr;
    auto coarse = [&]() {
      const int n = p.bin0 + (io << lg);
      return min(len_one ? n : static_cast<int>(__umulhi(static_cast<uint32_t>(n), len_magic)), p.n_int - 1);
    };
    bool empty = kRange ? moved & (p.claim[coarse()] >= key_now) : moved & (fresh | (io == e_start));
    claims = false;
    want = -1;
    if (__any_sync(0xFFFFFFFFu, edge | close | empty)) [[unlikely]] {
      if (edge) {
        const uint32_t site = static_cast<uint32_t>(site_exact(x_site, site_scale)), i = site / static_cast<uint32_t>(Y);
        propose(i, site - i * static_cast<uint32_t>(Y));
      }
      if (close) limit = accept_limit(x_acc, p.acc_thr);
      if (empty) {
        const int q = coarse();
        empty = p.claim[q] >= key_now;  // empty, or claimed in this round
        if (empty) {
          atomicMin(&p.claim[q], key_now | static_cast<uint32_t>(w));
          want = q;
        } else if (io == e_start) {
          e_start = -1;
        }
      }
      claims = __any_sync(0xFFFFFFFFu, empty);
    }
  };
  // last round's claims, after its barrier: the winner's lattice is still as
  // it was then
  auto settle = [&]() {
    const uint32_t mine = (claim_key - (1u << 10)) | static_cast<uint32_t>(w);
    unsigned won = __ballot_sync(0xFFFFFFFFu, want >= 0 && p.claim[max(want, 0)] == mine);
    while (won != 0) {
      const int lane = __ffs(won) - 1;
      won &= won - 1;
      const int bin = __shfl_sync(0xFFFFFFFFu, want, lane);
      const int e = __shfl_sync(0xFFFFFFFFu, io, lane);
      const uint32_t s = __shfl_sync(0xFFFFFFFFu, s0, lane);
      if (static_cast<int>(threadIdx.x & 31u) == lane) p.found_E[bin] = (e << lg) + p.e_min;
      store_spins<kTwo>(p, (w & ~31) + lane, s, p.found_lat + static_cast<long long>(bin) * N);
      __syncwarp();
    }
  };
  // One round, reading histogram copy kCopy, and the next one's preparation.
  // beside(): work that waits for nothing here.
  auto round = [&](auto copy, uint32_t x_site, uint32_t x_acc, auto beside) {
    constexpr int kCopy = decltype(copy)::value;
    sync();
    if (claims) [[unlikely]] settle();
    const uint32_t* now = p.hist + kCopy * Lh;
    uint32_t* other = p.hist + (1 - kCopy) * Lh;
    bool can = ok;
    if (kRange) {
      if (ok && (in < 0 || in >= p.len)) {  // the walker stops and keeps the offending energy
        ok = can = false;
        E = in * (1 << lg) + p.e_min;
        pos += 1;  // it consumed the site's draw alone
      }
    }
    const uint32_t h_old = now[io], h_new = now[can ? in : spare];
    beside();
    const bool acc = can & (static_cast<int>(h_new - h_old) <= limit);
    store_if(acc, lat + wa, na);
    store_if(acc, lat + wb, nb);
    if constexpr (kTwo) store_if(acc, lat + wc, nc);
    io = acc ? in : io;
    s0 ^= acc ? first_site : 0u;
    const int hit = ok ? io : spare;
    atomicAdd(&other[hit_before], 1u);
    atomicAdd(&other[hit], 1u);
    hit_before = hit;
    if (kRange && ok) pos += 2;
    const uint32_t key_now = claim_key;
    claim_key += 1u << 10;
    prepare(x_site, x_acc, acc, h_new == 0u, key_now);
  };

  // four draws at a time from an even position (a fresh walk's is 0)
  uint64_t blk = pos >> 2;
  // kKeys: round keys in registers, 18 additions fewer per block
  uint32_t ka[10], kb[10];
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    ka[r] = k0 + static_cast<uint32_t>(r) * kPhiloxWeylA;
    kb[r] = k1 + static_cast<uint32_t>(r) * kPhiloxWeylB;
    if constexpr (kKeys) asm volatile("" : "+r"(ka[r]), "+r"(kb[r]));
  }
  auto block = [&]() {
    uint4 c = make_uint4(static_cast<uint32_t>(blk), static_cast<uint32_t>(blk >> 32), s_lo, s_hi);
#pragma unroll
    for (int r = 0; r < 10; ++r) c = philox_round(c, ka[r], kb[r]);
    ++blk;
    return c;
  };
  const uint64_t pos_in = pos;
  const bool half = kRange && (pos & 2u) != 0;  // starts in the middle of a block
  uint4 ahead = half ? block() : make_uint4(0u, 0u, 0u, 0u);
  auto four = [&]() {
    const uint4 c = block();
    if (!kRange) return c;
    const uint4 o = half ? make_uint4(ahead.z, ahead.w, c.x, c.y) : c;
    ahead = c;
    return o;
  };
  uint4 a = four();
  prepare(a.x, a.y, false, false, claim_key);
  int left = p.n_iter;
  // not unrolled, rare cases out of line: the loop then stays in the instruction
  // cache (16x16 0.181 -> 0.161 us a round)
#pragma unroll 1
  for (; left >= 2; left -= 2) {
    uint4 b;
    round(Copy<0>{}, a.z, a.w, [&] { b = four(); });
    round(Copy<1>{}, b.x, b.y, [] {});
    a = b;
  }
  if (left > 0) round(Copy<0>{}, a.z, a.w, [] {});
  if (!kRange) pos = pos_in + 2 * static_cast<uint64_t>(p.n_iter);
  if (ok) E = (io << lg) + p.e_min;
  // the last round's claims and visits
  sync();
  if (claims) settle();
  atomicAdd(&p.hist[((p.n_iter & 1) ^ 1) * Lh + hit_before], 1u);
  sync();
}

}  // namespace
}  // namespace wlg
