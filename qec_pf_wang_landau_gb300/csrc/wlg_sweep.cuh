// One Wang-Landau sweep of a team's walkers (wl.cu:1077-1175), shared by the
// persistent main run and the sweep operator: the step, the exact decisions,
// the draw ring, and the additions of ln f at its end.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "wlg_accept.cuh"
#include "wlg_engine.h"
#include "wlg_rng.cuh"
#include "wlg_shadow.cuh"

namespace wlg {
namespace {

// steps of one part of a sweep: counts stay exact floats, and the rounding of
// a bin's additions stays small against the decision's error bound
constexpr int kPart = 1 << 16;
// Steps between two looks for walkers that need an exact decision; even.
constexpr int kChunk = 16;

// Shared-memory accesses of the step by 32-bit address.  Volatile keeps them in
// program order among themselves; plain C++ accesses to the same memory are
// separated from them by compiler barriers around the sweep.
__device__ __forceinline__ uint32_t lds_u32(uint32_t a)
{
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
template <int kOff>
__device__ __forceinline__ uint32_t lds_u32_at(uint32_t a)
{
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kOff));
  return v;
}
__device__ __forceinline__ uint2 lds_u64(uint32_t a)
{
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds_u128(uint32_t a)
{
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 lds_pair(uint32_t a)
{
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts_count(uint32_t a, float v)  // the pair's second float
{
  asm volatile("st.shared.f32 [%0+4], %1;" ::"r"(a), "f"(v));
}
__device__ __forceinline__ void sts_if(bool p, uint32_t a, uint32_t v)
{
  asm volatile(
    "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.u32 [%1], %2;\n\t}" ::"r"(static_cast<uint32_t>(p)),
    "r"(a), "r"(v));
}
template <int kOff>
__device__ __forceinline__ void sts_if_at(bool p, uint32_t a, uint32_t v)
{
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.u32 [%1+%3], %2;\n\t}" ::"r"(
                 static_cast<uint32_t>(p)),
               "r"(a), "r"(v), "n"(kOff));
}

// Site of a draw: trunc(double(u) * ((N-1) + 0.999999)) (wl.cu:63-65).  With
// f = x / 2^32 the reference's product lies within N*2^-23 + 1e-6 of f*N, so
// floor(f*N) = umulhi(x, N) is exact unless the fraction x*N mod 2^32 lies
// within site_thr (= 2^32 (N 2^-21 + 2^-18), >= 4x that bound) of an
// integer; there the reference's own float/double expression below decides.
__device__ __noinline__ int main_site_exact(uint32_t x, double scale)
{
  return static_cast<int>(trunc(static_cast<double>(unit_float(x)) * scale));
}

// The reference's acceptance u < min(1, exp(g - g_new)) (wl.cu:1113-1116).
__device__ __noinline__ bool accept_exact(uint32_t x2, double g, double g_new)
{
  return static_cast<double>(unit_float(x2)) < fmin(1.0, exp(g - g_new));
}

// g after n more additions of c, each rounded to double (wl.cu:1124 n times),
// for c >= 0 (and g >= 0 unless kSigned), mostly without the FP64 pipe (1/64 of
// the FP32 rate).  While the sum keeps g's exponent, each addition moves g by c
// rounded to g's grid: a fixed number of units in the last place, unless c ends
// exactly half-way between two of them.  Additions that leave the binade, ties
// and |g| < c take the FP64 addition; they are few (a tie needs the last
// log2(|g| / c) bits of c to be 10..0).
// Where no addition rounds at all (ln f = 1 on whole numbers, until the first
// average: bins cross binades all the time then) one fused multiply-add is the sum.
template <bool kSigned>
__device__ __forceinline__ double add_times(double g, double c, uint32_t n)
{
  const unsigned long long bc = __double_as_longlong(c);
  const unsigned long long m = (bc & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int ec = static_cast<int>(bc >> 52);
  {
    // exact: c and g are multiples of the largest partial sum's unit
    const double sum = fma(static_cast<double>(n), c, g);
    const int eg = (__double2hiint(g) >> 20) & 0x7FF, es = (__double2hiint(sum) >> 20) & 0x7FF, top = max(eg, es);
    const unsigned long long below = (1ull << (min(top - eg, 52))) - 1;
    if (top - ec <= __ffsll(static_cast<long long>(m)) - 1 && (__double_as_longlong(g) & below) == 0 &&
        (eg > 0 || g == 0.0) && top - (eg > 0 ? eg : top) <= 52)
      return sum;
  }
  while (n > 0) {
    unsigned long long bg = __double_as_longlong(g);
    const bool neg = kSigned && (bg >> 63) != 0;
    const int sh = (static_cast<int>(bg >> 52) & 0x7FF) - ec;
    if (sh >= 1 && sh <= 52 && ec > 0) {
      const unsigned long long r = m & ((1ull << sh) - 1), half = 1ull << (sh - 1);
      const unsigned long long step = (m >> sh) + (r > half ? 1u : 0u);
      const unsigned long long frac = bg & 0xFFFFFFFFFFFFFull;
      // units left in the binade: upwards, or (negative g) towards 0, where the
      // binade's lowest value may already stand for a sum rounded below it
      const unsigned long long room = neg ? (frac > 0 ? frac - 1 : 0) : 0xFFFFFFFFFFFFFull - frac;
      if (r != half && step != 0) {
        if (__umul64hi(step, n) == 0 && step * n <= room)
          return __longlong_as_double(static_cast<long long>(neg ? bg - step * n : bg + step * n));
        // the steps that surely stay in the binade
        const uint32_t k = static_cast<uint32_t>(
          fminf(__ull2float_rz(room) / __ull2float_rz(step) * (1.0f - 0x1p-20f), static_cast<float>(n - 1)));
        bg = neg ? bg - step * k : bg + step * k;
        n -= k;
        g = __longlong_as_double(static_cast<long long>(bg));
      }
    }
    const double g1 = g + c;
    if (g1 == g) return g;  // c below half a unit of g
    g = g1;
    --n;
  }
  return g;
}

// add_times without a loop, for n < 2^31 and g >= 0: the sum when it keeps g's
// exponent and no tie or g < c comes up, else ok = false.  m, ec: significand and
// exponent field of c (split_addend); integer operations only, about 25.
struct Addend {
  unsigned long long m;
  int ec;
};
__device__ __forceinline__ Addend split_addend(double c)
{
  const unsigned long long b = __double_as_longlong(c);
  return Addend{(b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull, static_cast<int>(b >> 52)};
}
__device__ __forceinline__ double add_times_in_binade(double g, const Addend& c, uint32_t n, bool& ok)
{
  const unsigned long long bg = __double_as_longlong(g);
  const int sh = static_cast<int>(bg >> 52) - c.ec;
  const unsigned long long cut = c.m << ((64 - sh) & 63);  // the bits of c below g's grid, from the top
  const unsigned long long step = (c.m >> (sh & 63)) + (cut > 0x8000000000000000ull ? 1u : 0u);
  // n steps: step < 2^52 and n < 2^31 as two 32-bit products; up must stay
  // below what is left of the binade, so its high word below 2^20
  const unsigned long long low = static_cast<unsigned long long>(static_cast<uint32_t>(step)) * n;
  const unsigned long long high = (step >> 32) * n + (low >> 32);
  const unsigned long long up = high << 32 | static_cast<uint32_t>(low);
  ok = (sh >= 1) & (sh <= 52) & (c.ec > 0) & (cut != 0x8000000000000000ull) & (high < (1u << 20)) &
       (up <= 0xFFFFFFFFFFFFFull - (bg & 0xFFFFFFFFFFFFFull));
  return __longlong_as_double(static_cast<long long>(bg + up));
}

// Split and shadow of a log g of either sign (kSigned), else of g >= 0.
template <bool kSigned>
__device__ __forceinline__ Split split_of(double g)
{
  if constexpr (!kSigned) return split_float(g);
  const Split a = split_float(fabs(g));
  const bool neg = __double2hiint(g) < 0;
  return Split{neg ? -a.hi : a.hi, neg ? -a.lo : a.lo};
}
template <bool kSigned>
__device__ __forceinline__ float shadow_of(double g, const Split& base)
{
  if constexpr (!kSigned) return shadow_split(g, base);
  const Split a = split_of<true>(g);
  return (a.hi - base.hi) + (a.lo - base.lo);
}

template <int kR>
struct Rounds {
  static constexpr int value = kR;
};

struct Lat {
  uint64_t r;       // spins in a register (N <= 64)
  uint32_t a;       // or the shared address of the walker's first word
  uint32_t stride;  // and the bytes between its words
};

template <bool kReg>
__device__ __forceinline__ uint32_t spin_bit(const Lat& l, int q)
{
  if constexpr (kReg) {
    return static_cast<uint32_t>(l.r >> q) & 1u;
  } else {
    return (lds_u32(l.a + static_cast<uint32_t>(q >> 5) * l.stride) >> (q & 31)) & 1u;
  }
}

template <bool kReg>
__device__ __forceinline__ uint32_t bond_bit(uint64_t reg, const uint32_t* sm, int q)
{
  if constexpr (kReg) {
    return static_cast<uint32_t>(reg >> q) & 1u;
  } else {
    return (sm[q >> 5] >> (q & 31)) & 1u;
  }
}

struct Nbr {
  int up, dn, lf, rt, i, j;
};

__device__ __forceinline__ Nbr neighbours(int site, const MainDesc& d)
{
  Nbr n;
  n.i = static_cast<int>((static_cast<uint32_t>(site) * d.site_magic) >> 20);
  n.j = site - n.i * d.Y;
  n.up = (n.i == 0 ? d.X - 1 : n.i - 1) * d.Y + n.j;
  n.dn = (n.i == d.X - 1 ? 0 : n.i + 1) * d.Y + n.j;
  n.lf = n.i * d.Y + (n.j == 0 ? d.Y - 1 : n.j - 1);
  n.rt = n.i * d.Y + (n.j == d.Y - 1 ? 0 : n.j + 1);
  return n;
}

// Energy change of flipping `site` (wl.cu:52-156 on bits: a neighbour term
// s_nb * J is -1 exactly when its spin bit and bond bit differ).
template <bool kReg>
__device__ __forceinline__ int flip_energy(const Lat& l, uint64_t JR, uint64_t JD, const uint32_t* Jr_s,
                                           const uint32_t* Jd_s, int site, const MainDesc& d)
{
  const Nbr n = neighbours(site, d);
  const int t_up = static_cast<int>(spin_bit<kReg>(l, n.up) ^ bond_bit<kReg>(JD, Jd_s, n.up));
  const int t_lf = static_cast<int>(spin_bit<kReg>(l, n.lf) ^ bond_bit<kReg>(JR, Jr_s, n.lf));
  const int t_dn = static_cast<int>(spin_bit<kReg>(l, n.dn) ^ bond_bit<kReg>(JD, Jd_s, site));
  const int t_rt = static_cast<int>(spin_bit<kReg>(l, n.rt) ^ bond_bit<kReg>(JR, Jr_s, site));
  int sigma;
  if (d.boundary == 0) {
    sigma = 4 - 2 * (t_up + t_lf + t_dn + t_rt);
  } else {
    sigma = (n.i > 0 ? 1 - 2 * t_up : 0) + (n.j > 0 ? 1 - 2 * t_lf : 0) + (n.i < d.X - 1 ? 1 - 2 * t_dn : 0) +
            (n.j < d.Y - 1 ? 1 - 2 * t_rt : 0);
  }
  return 2 * (1 - 2 * static_cast<int>(spin_bit<kReg>(l, site))) * sigma;
}

// Energy change of flipping site (i, j) on the row layout (lattice_rows), the
// same arithmetic as wl.cu:52-156: with r, ru, rd the rows of the site and of
// the rows above and below, a bond is unsatisfied (s_a s_b J = -1) exactly when
// the two spin bits and the coupling bit have odd parity, and flipping the
// site changes the energy by 2 (deg - 2 unsat) over its deg bonds.  Without
// a branch on the boundary: a horizontal bond belongs to the column on its
// left and is missing on an open lattice exactly when that is the last
// column (hedge clears its bit), a vertical bond is missing at the first or
// last row (wl.cu:134-137).  Also returns the address of the site's row word
// and that word with the site flipped.
__device__ __forceinline__ int flip_energy_rows(const Lat& l, const uint32_t* Jr_s, const uint32_t* Jd_s, int i, int j,
                                                const MainDesc& d, uint32_t hedge, bool open, uint32_t& row_a,
                                                uint32_t& row_new)
{
  const int iu = i == 0 ? d.X - 1 : i - 1;
  const int id = i == d.X - 1 ? 0 : i + 1;
  row_a = l.a + i * l.stride;
  const uint32_t r = lds_u32(row_a), ru = lds_u32(l.a + iu * l.stride), rd = lds_u32(l.a + id * l.stride);
  const uint32_t mj = 1u << j;
  const uint32_t mjl = j == 0 ? 1u << (d.Y - 1) : mj >> 1;
  const uint32_t rr = (r >> 1) | ((r & 1u) << (d.Y - 1));  // bit c: spin (i, c + 1 mod Y)
  const uint32_t h = r ^ rr ^ Jr_s[i];                     // bit c: bond (i, c)-(i, c + 1) unsatisfied
  const bool up = !open || i != 0, dn = !open || i != d.X - 1;
  const uint32_t vu = up ? (r ^ ru ^ Jd_s[iu]) & mj : 0u;  // bond (i - 1, j)-(i, j) unsatisfied
  const uint32_t vd = dn ? (r ^ rd ^ Jd_s[i]) & mj : 0u;   // bond (i, j)-(i + 1, j) unsatisfied
  const uint32_t hm = (mj | mjl) & hedge;
  row_new = r ^ mj;
  const int unsat = __popc(h & hm) + __popc(vu) + __popc(vd);
  const int deg = __popc(hm) + (up ? 1 : 0) + (dn ? 1 : 0);
  return 2 * (deg - 2 * unsat);
}

__device__ __forceinline__ uint32_t shared_addr(const void* p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Bond tables: per column the bits of its two horizontal bonds (low half) and
// its down bond (high half), and its missing bonds in bin bytes; per row the
// masks of what exists in its own word and in the word above, and its missing
// bonds.  kTwo: horizontal bonds alone per column, masks of all or nothing for
// the down bonds of the row and of the one above.
template <bool kTwo>
__device__ __forceinline__ void fill_bond_tables(uint2* col, uint4* row, int X, int Y, bool open, int dlt_bytes, int t,
                                                 int P)
{
  for (int j = t; j < Y; j += P) {
    uint32_t h = (1u << j) | (1u << (j == 0 ? Y - 1 : j - 1));
    if (open) h &= ~(1u << (Y - 1));
    const int miss = open ? (j == 0 ? 1 : 0) + (j == Y - 1 ? 1 : 0) : 0;
    col[j] = make_uint2(kTwo ? h : h | 0x10000u << j, static_cast<uint32_t>(-miss * dlt_bytes));
  }
  for (int i = t; i < X; i += P) {
    const bool up = !open || i > 0, dn = !open || i < X - 1;
    const int miss = (up ? 0 : 1) + (dn ? 0 : 1);
    row[i] = make_uint4(dn ? 0xFFFFFFFFu : (kTwo ? 0u : 0x0000FFFFu), up ? (kTwo ? 0xFFFFFFFFu : 0xFFFF0000u) : 0u,
                        static_cast<uint32_t>(-miss * dlt_bytes), 0u);
  }
}

// The bonds of a row from its spin bits r, those of the row below and the
// coupling bits: bit j of h is bond (i, j)-(i, j + 1), bit j of v bond
// (i, j)-(i + 1, j); set when unsatisfied, 0 when missing.
__device__ __forceinline__ void bond_bits(uint32_t r, uint32_t below, uint32_t Jr, uint32_t Jd, int Y, bool open, bool last,
                                          uint32_t& h, uint32_t& v)
{
  const uint32_t all = Y == 32 ? 0xFFFFFFFFu : (1u << Y) - 1u;
  h = (r ^ ((r >> 1) | ((r & 1u) << (Y - 1))) ^ Jr) & all;
  v = (r ^ below ^ Jd) & all;
  if (open) {
    h &= ~(1u << (Y - 1));
    if (last) v = 0;
  }
}

// Both in one word, rows of up to 16 sites.
__device__ __forceinline__ uint32_t bond_word(uint32_t r, uint32_t below, uint32_t Jr, uint32_t Jd, int Y, bool open,
                                              bool last)
{
  uint32_t h, v;
  bond_bits(r, below, Jr, Jd, Y, open, last, h, v);
  return h | v << 16;
}

constexpr int kRingAhead = kRingSlots - 4 + 1;  // a block is added while it fits

// What the team's walkers have in common.
struct SweepTeam {
  const MainDesc& d;  // lattice, draws and energy step
  int P;              // walkers side by side in shared memory
  uint32_t jt_a;      // table: neighbours and degrees per site; bonds: masks per column
  uint32_t rt_a;      // table: degrees; bonds: masks per row
  const uint32_t *Jr_s, *Jd_s;  // coupling words (spins in shared memory)
  uint64_t JR, JD;              // couplings (spins in a register)
};

// A walker, kept between sweeps.
template <bool kTight>
struct Walker {
  Lat lt;
  int E;                // energy
  int lo, hi, bb, len;  // window; its first energy on the walker's grid, and bins
  float2* pair;         // its bin 0: {float shadow of log g, visits}, P apart
  uint32_t ring_a;      // its draw ring
  Stream rng;           // keys and position
  // The draw ring and the shadows stay between sweeps.  blk, fill: the next
  // Philox block and its ring position; fresh: the shadows (relative to gs,
  // |shadow| <= amax, high words of log g <= ghi) match log g.
  uint64_t blk;
  uint32_t fill;
  bool fresh;
  Split gs;
  float amax;
  int ghi;
  uint32_t s0;                                   // spin of site 0 (kSign)
  uint32_t tight_ring[kTight ? kRingSlots : 1];  // the ring in local memory where shared memory has no room
  __device__ __forceinline__ void start()
  {
    blk = rng.pos >> 2;
    fill = static_cast<uint32_t>(blk) * 512u;
    fresh = false;
    gs = Split{0.0f, 0.0f};
    amax = 0.0f;
    ghi = 0;
  }
};

// n_iter steps of the lane's walker; the lanes of wmask call it together.
// ahead: draws to be left in the ring (at most kRingAhead).
// kSign (the caller's arrays): keep the spin of site 0, which bond words alone
// do not tell, and take log g of either sign.
// log_g(c): FP64 log g of bin c; is_bad(E): the pre-run never saw E
// (wl.cu:1091-1104); new_energy(E, step): such a proposal stopped the walker;
// fold(visits of the current bin, its index, last): adds the visits kept in the
// walker's bins to histogram and log g and clears them.
template <int kStore, bool kTight, bool kSign, class LogG, class IsBad, class NewEnergy, class Fold>
__device__ __forceinline__ void wl_sweep(const SweepTeam& team, Walker<kTight>& wk, unsigned wmask, int n_iter, bool frozen,
                                         double lnf, int ahead, LogG log_g, IsBad is_bad, NewEnergy new_energy, Fold fold)
{
  constexpr bool kTable = kStore == kStoreTable;
  constexpr bool kReg = kStore == kStoreReg || kTable;
  constexpr bool kRows = kStore == kStoreRows;
  constexpr bool kTwo = store_two_words(kStore);
  constexpr bool kBonds = store_bonds(kStore);
  // bonds of periodic lattices: every row and column alike, no masks for rows
  constexpr bool kMissing = kStore == kStoreBondsOpen || kStore == kStoreBonds2Open;
  // Pairs of steps unrolled in the persistent run, so that ptxas schedules
  // across them: 16x16 on every SM 0.368 -> 0.339 us a step, 12x12 0.157 ->
  // 0.148, 6x6 0.129 -> 0.122.  Not for the longer steps of rows and linear
  // words (24x24 0.666 -> 0.691) nor for the operator, whose launches find the
  // instruction cache cold (a run on the operators 5.4 -> 6.5 ms).
  constexpr int kUnroll = !kSign && (kTable || kBonds) ? 4 : 1;
  const float kInf = __int_as_float(0x7F800000);
  const MainDesc& d = team.d;
  const int P = team.P;
  const uint32_t jt_a = team.jt_a;
  [[maybe_unused]] const uint32_t rt_a = team.rt_a, degs_a = team.rt_a;
  [[maybe_unused]] const uint32_t *Jr_s = team.Jr_s, *Jd_s = team.Jd_s;
  [[maybe_unused]] const uint64_t JR = team.JR, JD = team.JD;
  Lat& lt = wk.lt;
  int& E = wk.E;
  const int lo = wk.lo, hi = wk.hi, bb = wk.bb, len = wk.len;
  float2* const pair = wk.pair;
  const uint32_t ring_a = wk.ring_a;
  Stream& rng = wk.rng;
  uint64_t& blk = wk.blk;
  uint32_t& fill = wk.fill;
  bool& fresh = wk.fresh;
  Split& gs = wk.gs;
  float& amax = wk.amax;
  int& ghi = wk.ghi;
  uint32_t(&tight_ring)[kTight ? kRingSlots : 1] = wk.tight_ring;
  const float lnf_f = static_cast<float>(lnf);
  const float inc = frozen ? 0.0f : 1.0f;
  const uint32_t bin0 = shared_addr(pair);
  // bytes between a walker's neighbouring bins, and bin-address change per
  // bond satisfied minus unsatisfied (dE = 2 (deg - 2 unsat))
  const int bin_bytes = 8 * P, dlt_bytes = 2 * (bin_bytes >> d.lg);
  const uint32_t uN = static_cast<uint32_t>(d.N), uX = static_cast<uint32_t>(d.X), uY = static_cast<uint32_t>(d.Y);
  const uint32_t d_thr = d.site_thr;
  const bool open_bc = d.boundary != 0;
  // row layout: open lattices have no bond right of the last column
  [[maybe_unused]] const uint32_t hedge = open_bc ? ~(1u << (d.Y - 1)) : 0xFFFFFFFFu;
  bool stopped = false;
  for (int left = n_iter; left > 0 && __any_sync(wmask, !stopped);) {
    const int part = min(left, kPart);
    left -= part;
    const int c_first = min(max((E - bb) >> d.lg, 0), max(len - 1, 0));
    const int e_off = E - (bb + c_first * (1 << d.lg));  // 0 unless every proposal is bad
    // shadows of this walker's log g relative to a base near it:
    // differences inside a window stay small while values reach 1e4
    if (!fresh) {
      const double gbase = log_g(c_first);
      gs = split_of<kSign>(gbase);
      ghi = __double2hiint(gbase) & 0x7FFFFFFF;
      amax = 0.0f;
#pragma unroll 2
      for (int c = 0; c < len; ++c) {
        const double g = log_g(c);
        const float a = shadow_of<kSign>(g, gs);
        if (kTight || pair[c * P].x == pair[c * P].x) {
          pair[c * P].x = a;
          amax = fmaxf(amax, fabsf(a));
          ghi = max(ghi, __double2hiint(g) & 0x7FFFFFFF);
        }
      }
      fresh = true;
    }
    // |df - d| for the reference's difference d of log g values and the
    // step's df = (a_c - a_n) + (n_c - n_n) ln f: shadows 2^-23 |a| +
    // 2^-43 g each; the float roundings of a_c - a_n, of ln f (its
    // product is at most |df| + 2 amax) and of the sum, 2^-24 each; a
    // rounding of each of the sums' part additions at most.  The terms in
    // |df| count up to |df| = 32: beyond it the decision has |df| / 4 to
    // spare, and its rounding is below the last factor.
    const float gmax = static_cast<float>(__hiloint2double(ghi + 1, 0));
    const float eps = 0x1p-21f * amax + 0x1p-18f + 0x1p-42f * gmax +
                      static_cast<float>(part) * 0x1p-51f * (gmax + static_cast<float>(part) * lnf_f);
    const float thr0 = (eps + kLogAbsErr) * (1.0f + 0x1p-18f);
    float thr = e_off == 0 && !stopped ? thr0 : kInf;  // +inf: the walker waits for an exact step, or is done
    float a_c = pair[c_first * P].x;
    if (a_c != a_c) a_c = shadow_of<kSign>(log_g(c_first), gs);  // a start energy the pre-run did not report
    float n_c = 0.0f;
    uint32_t cur = bin0 + static_cast<uint32_t>(c_first * bin_bytes);
    if constexpr (kTight) cur = static_cast<uint32_t>(c_first);  // bin index
    // Draws: ring slot s holds the draw whose position is s mod 16 (slot
    // 16 repeats slot 0, so two neighbouring draws lie 128 bytes apart).
    // Positions count in bytes of a slot, 128 per draw, modulo 2^32.  At
    // least 8 draws lie ahead before every pair of steps: each pair
    // takes 4 at most and a block is added whenever there is room.
    const uint64_t pos0 = rng.pos;
    uint32_t pos = static_cast<uint32_t>(pos0) * 128u;
    const uint32_t pos_start = pos;
    if (static_cast<int>(fill - pos) < 0) {  // the exchange drew more than the ring holds
      blk = pos0 >> 2;
      fill = static_cast<uint32_t>(blk) * 512u;
    }
    auto ring_get = [&](uint32_t at) {  // draw at byte position `at`
      if constexpr (kTight) return tight_ring[(at >> 7) & 15u];
      else return lds_u32(ring_a + (at & 2047u));
    };
    uint4 ph;               // the next block, advanced in pieces beside the steps
    uint32_t ka = 0, kb = 0;  // its round keys
    auto philox_begin = [&]() {
      ph = make_uint4(static_cast<uint32_t>(blk), static_cast<uint32_t>(blk >> 32), rng.s0, rng.s1);
      ka = rng.k0;
      kb = rng.k1;
    };
    auto philox_some = [&](auto rounds) {
      constexpr int kR = decltype(rounds)::value;
      ph = philox_rounds<kR>(ph, ka, kb);
      ka += kR * kPhiloxWeylA;
      kb += kR * kPhiloxWeylB;
    };
    auto philox_store = [&]() {
      const uint4 c = ph;
      const bool room = static_cast<int>(fill - pos) <= 12 * 128;
      if constexpr (kTight) {
        if (room) {
          const uint32_t s = (fill >> 7) & 15u;
          tight_ring[s] = c.x;
          tight_ring[s + 1] = c.y;
          tight_ring[s + 2] = c.z;
          tight_ring[s + 3] = c.w;
        }
      } else {
        const uint32_t off = fill & 2047u, a = ring_a + off;
        sts_if(room, a, c.x);
        sts_if_at<128>(room, a, c.y);
        sts_if_at<256>(room, a, c.z);
        sts_if_at<384>(room, a, c.w);
        sts_if_at<2048>(room && off == 0, ring_a, c.x);
      }
      blk += room ? 1u : 0u;
      fill += room ? 512u : 0u;
    };
    auto produce = [&]() {
      philox_begin();
      philox_some(Rounds<10>{});
      philox_store();
    };
    asm volatile("" ::: "memory");
    while (__any_sync(wmask, static_cast<int>(fill - pos) < 8 * 128)) produce();
    uint32_t xa, xb, xc, xd;  // the draws at pos .. pos + 3
    auto reload = [&]() {
      xa = ring_get(pos);
      xb = ring_get(pos + 128);
      xc = ring_get(pos + 256);
      xd = ring_get(pos + 384);
    };
    reload();
    int rem = part;
    // What a draw proposes, fetched one step ahead: the site is
    // trunc(u (N - 1 + 0.999999)) (wl.cu:60-66) as floor(x N / 2^32), its
    // row floor(x X / 2^32) and its column the rest, unless x N lies
    // within site_thr of a multiple of 2^32 (ok false).
    struct Site {
      bool ok;
      uint32_t i, j;  // table: i is the site
      uint4 row;      // table: neighbours; bonds: row masks
      uint2 col;      // table: degree; bonds: column masks
    };
    auto fetch = [&](uint32_t x) {
      Site f;
      uint32_t lo_s;
      if constexpr (kTable) {
        const uint64_t xn = static_cast<uint64_t>(x) * uN;
        f.i = static_cast<uint32_t>(xn >> 32);
        lo_s = static_cast<uint32_t>(xn);
        f.row = lds_u128(jt_a + 16 * f.i);
        f.col.x = lds_u32(degs_a + 4 * f.i);
      } else {
        const uint64_t xi = static_cast<uint64_t>(x) * uX;
        f.i = static_cast<uint32_t>(xi >> 32);
        const uint32_t rest = static_cast<uint32_t>(xi);
        if constexpr (kBonds && !kMissing) {  // two products: 16x16 on every SM 3 % faster
          f.j = __umulhi(rest, uY);
          lo_s = rest * uY;
        } else {
          const uint64_t xj = static_cast<uint64_t>(rest) * uY;
          f.j = static_cast<uint32_t>(xj >> 32);
          lo_s = static_cast<uint32_t>(xj);
        }
        if constexpr (kBonds) {
          if constexpr (kMissing) {
            f.col = lds_u64(jt_a + 8 * f.j);
            f.row = lds_u128(rt_a + 16 * f.i);
          } else {
            f.col = make_uint2(lds_u32(jt_a + 8 * f.j), 0u);
            f.row = make_uint4(0xFFFFFFFFu, kTwo ? 0xFFFFFFFFu : 0xFFFF0000u, 0u, 0u);
          }
        }
      }
      f.ok = lo_s + d_thr >= 2u * d_thr;
      return f;
    };
    Site cs = fetch(xa);
    // One step.  Loads come before the decision's stores in program order,
    // or they would wait for it; beside1() and beside2() are independent
    // work for the two waits on shared memory.
    auto step = [&](auto beside1, auto beside2) {
      uint32_t next;           // address (tight: index) of the proposal's bin
      [[maybe_unused]] uint64_t flip_mask = 0;  // register spins
      [[maybe_unused]] uint32_t wa = 0, wb = 0, wc = 0, na = 0, nb = 0, nc = 0;  // shared words to rewrite on acceptance
      [[maybe_unused]] int dE = 0;
      if constexpr (kTable) {
        const int deg = static_cast<int>(cs.col.x);
        const int sgn = 1 - 2 * static_cast<int>((lt.r >> cs.i) & 1ull);
        const int unsat = __popc((static_cast<uint32_t>(lt.r) ^ cs.row.z) & cs.row.x) +
                          __popc((static_cast<uint32_t>(lt.r >> 32) ^ cs.row.w) & cs.row.y);
        flip_mask = 1ull << cs.i;
        if constexpr (kTight) dE = sgn * 2 * (deg / dlt_bytes - 2 * unsat);
        else next = (cur + sgn * deg) + unsat * (-2 * dlt_bytes * sgn);
      } else if constexpr (kBonds) {
        int unsat;
        if constexpr (kTwo) {
          wa = lt.a + 2u * cs.i * lt.stride;
          wc = wa + lt.stride;
          wb = lt.a + (2u * min(cs.i - 1u, uX - 1u) + 1u) * lt.stride;
          na = lds_u32(wa);
          nb = lds_u32(wb);
          nc = lds_u32(wc);
          const uint32_t m = 1u << cs.j, m2 = m & cs.row.y, m3 = m & cs.row.x;
          unsat = __popc(na & cs.col.x) + __popc(nb & m2) + __popc(nc & m3);
          na ^= cs.col.x;
          nb ^= m2;
          nc ^= m3;
        } else {
          wa = lt.a + cs.i * lt.stride;
          wb = lt.a + min(cs.i - 1u, uX - 1u) * lt.stride;
          na = lds_u32(wa);
          nb = lds_u32(wb);
          const uint32_t m1 = cs.col.x & cs.row.x, m2 = cs.col.x & cs.row.y;
          unsat = __popc(na & m1) + __popc(nb & m2);
          na ^= m1;
          nb ^= m2;
        }
        next = (cur + 4 * dlt_bytes + cs.col.y + cs.row.z) + unsat * (-2 * dlt_bytes);
      } else {
        if constexpr (kRows) {
          dE = flip_energy_rows(lt, Jr_s, Jd_s, static_cast<int>(cs.i), static_cast<int>(cs.j), d, hedge, open_bc, wa,
                                na);
        } else {
          const int site = static_cast<int>(cs.i * uY + cs.j);
          dE = flip_energy<kReg>(lt, JR, JD, Jr_s, Jd_s, site, d);
          if constexpr (kReg) {
            flip_mask = 1ull << site;
          } else {
            wa = lt.a + static_cast<uint32_t>(site >> 5) * lt.stride;
            na = lds_u32(wa) ^ (1u << (site & 31));
          }
        }
        if constexpr (!kTight) next = cur + dE * (bin_bytes >> d.lg);
      }
      beside1();
      float2 v;
      bool inside, in_doubt = false;
      if constexpr (kTight) {
        // no guard bins: classify the proposal explicitly
        const int En = bb + (static_cast<int>(cur) << d.lg) + dE;
        inside = En >= lo && En <= hi;
        in_doubt = is_bad(En);
        next = static_cast<uint32_t>(min(max(static_cast<int>(cur) + (dE >> d.lg), 0), d.L - 1));
        v = lds_pair(bin0 + next * bin_bytes);
        if (!inside) v.x = kInf;
      } else {
        v = lds_pair(next);
      }
      const float lu = log_uniform(xb);
      beside2();
      if constexpr (!kTight) inside = v.x < kInf;
      // the next step's draws and site, as if this step needs no exact
      // decision; a walker that does reloads them after it
      const uint32_t pos_next = pos + (inside ? 256u : 128u);
      xa = inside ? xc : xb;
      xb = inside ? xd : xc;
      const Site ns = fetch(xa);
      if constexpr (kTight) {
        xc = ring_get(pos_next + 256);
        xd = ring_get(pos_next + 384);
      } else {
        const uint32_t a = ring_a + ((pos_next + 256u) & 2047u);
        xc = lds_u32(a);
        xd = lds_u32_at<128>(a);
      }
      // u < min(1, exp(g_cur - g_new)) (wl.cu:1113-1116) as log u < df; a
      // NaN shadow leaves `known` false, an infinite one known and
      // rejected; u = 1 (log 0) is left to the exact step
      const float df = fmaf(n_c - v.y, lnf_f, a_c - v.x);
      const float diff = lu - df;
      const bool known = fabsf(diff) > thr && lu < 0.0f && cs.ok && !in_doubt;
      const bool acc = known && diff < 0.0f;
      if constexpr (kReg) {
        lt.r ^= acc ? flip_mask : 0ull;
      } else {
        sts_if(acc, wa, na);
        if constexpr (kBonds) sts_if(acc, wb, nb);
        if constexpr (kTwo) sts_if(acc, wc, nc);
      }
      if constexpr (kSign) wk.s0 ^= acc & ((cs.i | cs.j) == 0) ? 1u : 0u;
      cur = acc ? next : cur;
      a_c = acc ? v.x : a_c;
      n_c = acc ? v.y : n_c;
      n_c += known ? inc : 0.0f;
      sts_count(kTight ? bin0 + cur * bin_bytes : cur, n_c);
      pos = known ? pos_next : pos;
      rem -= known ? 1 : 0;
      thr = known ? thr : kInf;
      cs = ns;
    };
    // The one step of a walker that waits, by the reference's expressions.
    auto exact_step = [&]() {
      if (thr == kInf && rem > 0 && !stopped) {
        const uint32_t x1 = ring_get(pos), x2 = ring_get(pos + 128);
        const int site = main_site_exact(x1, d.site_scale);
        const int i = static_cast<int>((static_cast<uint32_t>(site) * d.site_magic) >> 20), j = site - i * d.Y;
        const int c_cur = kTight ? static_cast<int>(cur) : static_cast<int>((cur - bin0) / bin_bytes);
        uint32_t w1 = 0, w2 = 0, n1 = 0, n2 = 0;
        [[maybe_unused]] uint32_t w3 = 0, n3 = 0;
        int dE;
        if constexpr (kBonds) {
          const uint32_t iu = static_cast<uint32_t>(i == 0 ? d.X - 1 : i - 1);
          const uint2 cm = lds_u64(jt_a + 8 * j);
          const uint4 rm = lds_u128(rt_a + 16 * i);
          uint32_t m1, m2, m3 = 0;
          if constexpr (kTwo) {
            w1 = lt.a + 2u * static_cast<uint32_t>(i) * lt.stride;
            w3 = w1 + lt.stride;
            w2 = lt.a + (2u * iu + 1u) * lt.stride;
            m1 = cm.x;
            m2 = (1u << j) & rm.y;
            m3 = (1u << j) & rm.x;
            n3 = lds_u32(w3);
          } else {
            w1 = lt.a + static_cast<uint32_t>(i) * lt.stride;
            w2 = lt.a + iu * lt.stride;
            m1 = cm.x & rm.x;
            m2 = cm.x & rm.y;
          }
          n1 = lds_u32(w1);
          n2 = lds_u32(w2);
          dE = 2 * (__popc(m1) + __popc(m2) + __popc(m3) - 2 * (__popc(n1 & m1) + __popc(n2 & m2) + __popc(n3 & m3)));
          n1 ^= m1;
          n2 ^= m2;
          n3 ^= m3;
        } else if constexpr (kRows) {
          dE = flip_energy_rows(lt, Jr_s, Jd_s, i, j, d, hedge, open_bc, w1, n1);
        } else {
          dE = flip_energy<kReg>(lt, JR, JD, Jr_s, Jd_s, site, d);
          if constexpr (!kReg) {
            w1 = lt.a + static_cast<uint32_t>(site >> 5) * lt.stride;
            n1 = lds_u32(w1) ^ (1u << (site & 31));
          }
        }
        const int En = bb + c_cur * (1 << d.lg) + e_off + dE;
        pos += 128u;
        if (is_bad(En)) {  // wl.cu:1091-1104: a new energy stops the problem
          stopped = true;
          new_energy(En, n_iter - left - rem);
        } else {
          thr = thr0;
          --rem;
          if (En >= lo && En <= hi) {
            pos += 128u;
            const int c_new = (En - bb) >> d.lg;
            const float n_new = c_new == c_cur ? n_c : lds_pair(bin0 + c_new * bin_bytes).y;
            const double g_cur = frozen ? log_g(c_cur) : add_times<kSign>(log_g(c_cur), lnf, static_cast<uint32_t>(n_c));
            const double g_new =
              frozen ? log_g(c_new) : add_times<kSign>(log_g(c_new), lnf, static_cast<uint32_t>(n_new));
            if (accept_exact(x2, g_cur, g_new)) {
              if constexpr (kSign) wk.s0 ^= site == 0 ? 1u : 0u;
              if constexpr (kReg) {
                lt.r ^= 1ull << site;
              } else {
                sts_if(true, w1, n1);
                if constexpr (kBonds) sts_if(true, w2, n2);
                if constexpr (kTwo) sts_if(true, w3, n3);
              }
              if (c_new != c_cur) {
                a_c = lds_pair(bin0 + c_new * bin_bytes).x;
                n_c = n_new;
              }
              cur = kTight ? static_cast<uint32_t>(c_new) : bin0 + c_new * bin_bytes;
            }
          }
          n_c += inc;
          sts_count(kTight ? bin0 + cur * bin_bytes : cur, n_c);
        }
      }
      produce();  // a waiting walker may have used draws since its last block
      reload();
      cs = fetch(xa);
    };
    __syncwarp(wmask);
    const int chunks = part / kChunk;
    auto none = [] {};
    auto two = [&] { philox_some(Rounds<2>{}); };
    for (int k = 0; k < chunks; ++k) {
#pragma unroll kUnroll
      for (int h = 0; h < kChunk / 2; ++h) {
        philox_begin();
        step(two, [&] { philox_some(Rounds<3>{}); });
        step(two, [&] { philox_some(Rounds<3>{}); });
        philox_store();
      }
      if (__any_sync(wmask, thr == kInf)) exact_step();
    }
    // walkers that waited catch up, and the rest of the part
    for (;;) {
      if (rem <= 0) thr = kInf;
      if (!__any_sync(wmask, rem > 0 && !stopped)) break;
      if (__any_sync(wmask, static_cast<int>(fill - pos) < 8 * 128)) produce();
      step(none, none);
      if (__any_sync(wmask, thr == kInf && rem > 0 && !stopped)) exact_step();
    }
    asm volatile("" ::: "memory");
    const int c_last = kTight ? static_cast<int>(cur) : static_cast<int>((cur - bin0) / bin_bytes);
    E = bb + c_last * (1 << d.lg) + e_off;
    rng.pos = pos0 + ((pos - pos_start) >> 7);
    if (left == 0)
      while (__any_sync(wmask, static_cast<int>(fill - pos) < ahead * 128)) produce();
    fold(n_c, c_last, left == 0);
  }
}

}  // namespace
}  // namespace wlg
