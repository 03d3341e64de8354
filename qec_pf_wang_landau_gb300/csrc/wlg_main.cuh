// The persistent main run of the batched engine, k_main_batch.
//
// A team of threads (one per walker, a multiple of 32) takes a problem from a
// global work counter and runs the reference's whole main-run loop
// (mainrun.cu:243-383) for it without leaving the GPU: WL sweeps, flatness
// vote, window averaging, reset, convergence and replica exchange, then takes
// the next problem.
//
// A step touches as little as the walk allows:
//   * every walker has a column of {shadow, count} pairs, one per energy bin:
//     the float shadow of its log g at the start of the sweep and its visits
//     since.  log g and the histogram themselves wait for the end of the
//     sweep, when the counts are folded into them (fold_bins): a bin visited n
//     times gets n additions of ln f, rounded one by one as the reference
//     rounds them, but in a few integer operations (add_times);
//   * the column has guard bins below and above the window.  A shadow of +inf
//     marks an energy outside the window, NaN one that the pre-run never saw,
//     so the one load that fetches the proposal's log g also classifies it;
//   * random draws come from a ring of 16 per walker, refilled by one Philox
//     block per two steps, independent of the steps it runs beside; the next
//     step's site and table entries are fetched before this step is decided;
//   * spins: one u64 register for N <= 64 (with a neighbour table); for larger
//     lattices with rows of up to 16 sites the unsatisfied bonds instead of the
//     spins, so that a proposal reads two words and no couplings; one row per
//     word up to 32 sites a row; else linear words.
//
// Acceptance u < min(1, exp(dlogg)) is decided as log u < dlogg with FP32
// values and a proven error bound.  What FP32 cannot settle (an acceptance
// inside the bound, a site pick next to a cell edge, a draw of u = 1, an energy
// the pre-run missed) stops the walker where it stands; every eight steps the
// warp looks for such walkers and makes their one step with the reference's
// FP64 expressions (exact_step).  Every decision equals the reference's.
//
// What bounds it: with few walkers (one warp an SM partition) the step's serial
// chain, two dependent shared-memory loads and about 15 dependent operations;
// with four warps a partition instruction issue.  Against the step that kept
// log g itself up to date (FP64 addition, shadow and count written back on every
// change of energy, bins classified by a mask load, Philox in registers), time
// per step of the longest problem, GB300: 6x6 0.29 -> 0.12 us (247 -> 97 warp
// instructions), up to 12x12 mixed 0.35 -> 0.15 us, 16x16 with 512 walkers on
// every SM 0.94 -> 0.36 us, 24x24 1.12 -> 0.63 us; between the sweeps, open
// lattices of 7-11 with sweeps of 100 steps, 20.4 -> 15.1 ms per 400 iterations.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "../../include/wlg.h"
#include "wlg_accept.cuh"
#include "wlg_engine.h"
#include "wlg_main_fn.h"
#include "wlg_rng.cuh"
#include "wlg_shadow.cuh"

namespace wlg {
namespace {

constexpr double kE = 2.718281828459045;  // std::numbers::e, mainrun.cu:56

// steps of one part of a sweep: counts stay exact floats, and the rounding of
// a bin's additions stays small against the decision's error bound
constexpr int kPart = 1 << 16;
// steps between two looks for walkers that need an exact decision; even
constexpr int kChunk = 8;

struct Team {
  int size;  // threads
  int id;    // barrier id (1..15) or 0 for a single warp
  __device__ __forceinline__ void sync() const
  {
    if (size == 32) {
      __syncwarp();
    } else {
      asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(size) : "memory");
    }
  }
};

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
// for g >= 0, c >= 0, mostly without the FP64 pipe (1/64 of the FP32 rate).
// While the sum keeps g's exponent, each addition moves g by c rounded to g's
// grid: a fixed number of units in the last place, unless c ends exactly
// half-way between two of them.  Additions that leave the binade, ties and
// g < c take the FP64 addition; they are few (a tie needs the last
// log2(g / c) bits of c to be 10..0).
__device__ __forceinline__ double add_times(double g, double c, uint32_t n)
{
  const unsigned long long bc = __double_as_longlong(c);
  const unsigned long long m = (bc & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int ec = static_cast<int>(bc >> 52);
  while (n > 0) {
    unsigned long long bg = __double_as_longlong(g);
    const int sh = static_cast<int>(bg >> 52) - ec;
    if (sh >= 1 && sh <= 52 && ec > 0) {
      const unsigned long long r = m & ((1ull << sh) - 1), half = 1ull << (sh - 1);
      const unsigned long long step = (m >> sh) + (r > half ? 1u : 0u);
      const unsigned long long room = 0xFFFFFFFFFFFFFull - (bg & 0xFFFFFFFFFFFFFull);
      if (r != half && step != 0) {
        if (__umul64hi(step, n) == 0 && step * n <= room) return __longlong_as_double(static_cast<long long>(bg + step * n));
        // the steps that surely stay in the binade
        const uint32_t k = static_cast<uint32_t>(
          fminf(__ull2float_rz(room) / __ull2float_rz(step) * (1.0f - 0x1p-20f), static_cast<float>(n - 1)));
        bg += step * k;
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

// u < min(1, exp(a) exp(b)) (wl.cu:871-878).  With neither factor out of
// double's range the product is exp(a + b) to 2^-50, so log u against a + b
// decides as in the sweep (two FP64 exps took most of an exchange pass).
__device__ __forceinline__ bool exchange_accepts(uint32_t x, double a, double b)
{
  const float s = static_cast<float>(a + b);
  const bool range = (__double2hiint(a) & 0x7FFFFFFF) < 0x4085E000 && (__double2hiint(b) & 0x7FFFFFFF) < 0x4085E000;
  const Decision r = decide(x, log_uniform(x), s, 0x1p-22f * fabsf(s) + 1e-9f, false);
  if (range && r.known) return r.acc;
  return static_cast<double>(unit_float(x)) < fmin(1.0, exp(a) * exp(b));
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

__device__ __forceinline__ bool mask_has(const uint32_t* mask, int c) { return (mask[c >> 5] >> (c & 31)) & 1u; }

__device__ __forceinline__ long long device_clock_ns()
{
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t shared_addr(const void* p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

template <int kStore, bool kTight>
__device__ void run_problem(const TeamHead& head, int p, const Team& team, int t, unsigned char* base, double* gslot,
                            bool global_g, const uint32_t* __restrict__ Jpool, const uint32_t* __restrict__ latpool,
                            const int* __restrict__ winpool, const uint32_t* __restrict__ maskpool,
                            double* __restrict__ outpool, MainResult* __restrict__ results,
                            unsigned char* __restrict__ statepool)
{
  constexpr bool kTable = kStore == kStoreTable;
  constexpr bool kReg = kStore == kStoreReg || kTable;
  constexpr bool kRows = kStore == kStoreRows;
  constexpr bool kBonds = kStore == kStoreBonds;
  const MainDesc& d = head.d;
  const int P = team.size;
  // start time straight into the result slot: a value kept live through the
  // sweep costs the step registers
  if (t == 0) results[p].t_start = device_clock_ns();
  // resumable run: state saved at the end of a launch, restored at the start
  unsigned char* const st = d.off_state >= 0 ? statepool + d.off_state : nullptr;
  const StateLayout& sl = head.state;
  const TeamLayout& lay = head.lay;
  // FP64 log g and the histogram change once per sweep: in the team's shared
  // memory where that costs no resident team, else in global memory (this
  // resident team's slice of a pool, or the saved state itself), L2-resident
  const bool in_state = global_g && st != nullptr;
  double* G = global_g ? (in_state ? reinterpret_cast<double*>(st + sl.off_G) : gslot)
                       : reinterpret_cast<double*>(base + lay.off_G);
  uint32_t* H = global_g ? (in_state ? reinterpret_cast<uint32_t*>(st + sl.off_H)
                                     : reinterpret_cast<uint32_t*>(gslot + static_cast<long long>(d.L) * P))
                         : reinterpret_cast<uint32_t*>(base + lay.off_H);
  const int guard = kTight ? 0 : guard_bins(d.lg);
  float2* pair = reinterpret_cast<float2*>(base + lay.off_pair) + guard * P;  // [bin -guard .. L + guard)[P]
  uint32_t* lat_s = reinterpret_cast<uint32_t*>(base + lay.off_lat);
  int* E_s = reinterpret_cast<int*>(base + lay.off_E);
  int* perm = reinterpret_cast<int*>(base + lay.off_perm);
  uint32_t* mask = reinterpret_cast<uint32_t*>(base + lay.off_mask);
  uint32_t* Js = reinterpret_cast<uint32_t*>(base + lay.off_J);
  double* fwin = reinterpret_cast<double*>(base + lay.off_f);
  double* lnfw = fwin + d.I;  // log(f) of each window, recomputed only when f changes
  int* cond = reinterpret_cast<int*>(base + lay.off_cond);
  int* flat = reinterpret_cast<int*>(base + lay.off_flat);
  // A finished window (cond stays 1) is frozen: its walkers no longer change
  // log g, so once an averaging pass leaves every value as it was, every
  // later pass would too; such windows are skipped (stab).  Not saved with a
  // suspended run: a resumed one recomputes one pass, with the same result.
  int* stab = reinterpret_cast<int*>(base + lay.off_stab);
  int* chg = stab + d.I;
  int* win = reinterpret_cast<int*>(base + lay.off_win);  // start, end, base, Lb, E0
  int* misc = reinterpret_cast<int*>(base + lay.off_misc);
  unsigned long long* new_key = reinterpret_cast<unsigned long long*>(misc + 4);
  const int I = d.I, W = d.W;
  int* w_start = win;
  int* w_end = win + I;
  int* w_base = win + 2 * I;
  int* w_len = win + 3 * I;

  // ---- load the problem
  for (int q = t; q < d.nwM; q += P) mask[q] = maskpool[d.off_mask + q];
  for (int q = t; q < 2 * d.nwL; q += P) Js[q] = Jpool[d.off_J + q];
  for (int q = t; q < 5 * I; q += P) win[q] = winpool[d.off_win + q];
  for (int q = t; q < I; q += P) {
    fwin[q] = kE;
    lnfw[q] = log(kE);
    cond[q] = 0;
    flat[q] = 0;
    stab[q] = 0;
    chg[q] = 0;
  }
  const bool resumed = st != nullptr && reinterpret_cast<const int*>(st)[4] != 0;
  if (!resumed)
    for (int c = 0; c < d.L; ++c) {
      G[c * P + t] = 0.0;
      H[c * P + t] = 0u;
    }
  if (t < 8) misc[t] = 0;
  const bool live = t < d.nwalk;
  const int b = live ? t / W : 0;
  const int w = t - b * W;
  perm[t] = w;
  team.sync();
  const int lo = live ? w_start[b] : 0, hi = live ? w_end[b] : 0, bb = live ? w_base[b] : 0;
  const int len = live ? w_len[b] : 0;
  const int step_mask = (1 << d.lg) - 1;
  const int span = d.e_max - d.e_min;
  // what a proposal of energy En is: bad (the pre-run never saw it,
  // wl.cu:1091-1104), else inside or outside the window
  auto is_bad = [&](int En) {
    const int rel = En - d.e_min;
    return rel < 0 || rel > span || (rel & step_mask) != 0 || !mask_has(mask, rel >> d.lg);
  };
  for (int c = -guard; c < d.L + guard; ++c) {
    const int En = bb + c * (1 << d.lg);
    const float x = is_bad(En) ? __int_as_float(0x7FC00000)
                               : (En >= lo && En <= hi ? 0.0f : __int_as_float(0x7F800000));
    pair[c * P + t] = make_float2(kTight ? 0.0f : x, 0.0f);
  }

  uint64_t JR = 0, JD = 0;
  if constexpr (kReg) {
    JR = Js[0] | (d.nwL > 1 ? static_cast<uint64_t>(Js[1]) << 32 : 0ull);
    JD = Js[d.nwL] | (d.nwL > 1 ? static_cast<uint64_t>(Js[d.nwL + 1]) << 32 : 0ull);
  }
  const uint32_t* Jr_s = Js;
  const uint32_t* Jd_s = Js + d.nwL;
  const bool open_bc = d.boundary != 0;
  // bytes between a walker's neighbouring bins, and bin-address change per
  // bond satisfied minus unsatisfied (dE = 2 (deg - 2 unsat))
  const int bin_bytes = 8 * P;
  const int dlt_bytes = 2 * (bin_bytes >> d.lg);
  if constexpr (kTable) {
    // neighbour table: bits of the neighbours of each site, and of those
    // whose connecting bond is -1 (X, Y >= 3, so the 4 neighbours differ);
    // then each site's degree in bin bytes
    ulonglong2* nbt = reinterpret_cast<ulonglong2*>(base + lay.off_tab);
    int* degs = reinterpret_cast<int*>(nbt + d.N);
    for (int site = t; site < d.N; site += P) {
      const Nbr n = neighbours(site, d);
      uint64_t m = 0, bnd = 0;
      auto put = [&](bool has, int q, uint64_t J, int bond) {
        if (!has) return;
        m |= 1ull << q;
        bnd |= static_cast<uint64_t>((J >> bond) & 1ull) << q;
      };
      put(!open_bc || n.i > 0, n.up, JD, n.up);
      put(!open_bc || n.j > 0, n.lf, JR, n.lf);
      put(!open_bc || n.i < d.X - 1, n.dn, JD, site);
      put(!open_bc || n.j < d.Y - 1, n.rt, JR, site);
      nbt[site] = make_ulonglong2(m, bnd);
      degs[site] = __popcll(m) * dlt_bytes;
    }
  }
  if constexpr (kBonds) {
    // per column the bits of its two horizontal bonds (h, low half) and its
    // down bond (v, high half), and its missing bonds in bin bytes; per row
    // the masks of what exists in its own word and in the word above
    uint2* jt = reinterpret_cast<uint2*>(base + lay.off_tab);
    uint4* rt = reinterpret_cast<uint4*>(base + lay.off_tab + align16(8 * d.Y));
    for (int j = t; j < d.Y; j += P) {
      uint32_t h = (1u << j) | (1u << (j == 0 ? d.Y - 1 : j - 1));
      if (open_bc) h &= ~(1u << (d.Y - 1));
      const int miss = open_bc ? (j == 0 ? 1 : 0) + (j == d.Y - 1 ? 1 : 0) : 0;
      jt[j] = make_uint2(h | 0x10000u << j, static_cast<uint32_t>(-miss * dlt_bytes));
    }
    for (int i = t; i < d.X; i += P) {
      const bool up = !open_bc || i > 0, dn = !open_bc || i < d.X - 1;
      const int miss = (up ? 0 : 1) + (dn ? 0 : 1);
      rt[i] = make_uint4(dn ? 0xFFFFFFFFu : 0x0000FFFFu, up ? 0xFFFF0000u : 0u, static_cast<uint32_t>(-miss * dlt_bytes),
                         0u);
    }
  }
  Lat lt;
  lt.a = shared_addr(lat_s + t);
  lt.stride = static_cast<uint32_t>(4 * P);
  lt.r = 0;
  if (live && !resumed) {
    const uint32_t* src = latpool + d.off_lat + static_cast<long long>(b) * d.nwL;
    if constexpr (kReg) {
      lt.r = src[0] | (d.nwL > 1 ? static_cast<uint64_t>(src[1]) << 32 : 0ull);
    } else if constexpr (kBonds) {
      // unsatisfied bonds of the start lattice: bit j of h is bond (i, j)-(i, j + 1),
      // bit j of v is bond (i, j)-(i + 1, j); missing bonds stay 0
      for (int i = 0; i < d.X; ++i) {
        const uint32_t r = src[i], dn = src[i + 1 < d.X ? i + 1 : 0];
        uint32_t h = r ^ ((r >> 1) | ((r & 1u) << (d.Y - 1))) ^ Jr_s[i], v = r ^ dn ^ Jd_s[i];
        if (open_bc) {
          h &= ~(1u << (d.Y - 1));
          if (i + 1 == d.X) v = 0;
        }
        const uint32_t row = (1u << d.Y) - 1u;
        lat_s[i * P + t] = (h & row) | (v & row) << 16;
      }
    } else {
      for (int q = 0; q < d.nwL; ++q) lat_s[q * P + t] = src[q];
    }
  }
  int E = live ? win[4 * I + b] : 0;
  Stream rng;
  rng.init(d.key_wl, static_cast<uint64_t>(t), 0);
  const bool keys_differ = d.key_ex != static_cast<uint64_t>(d.key_wl);
  const double reset_lim = exp(d.beta);  // wl.cu:609
  // row layout: open lattices have no bond right of the last column
  const uint32_t hedge = open_bc ? ~(1u << (d.Y - 1)) : 0xFFFFFFFFu;

  long long outer = 0;
  long long counter = 1;
  int status = WLG_OK;
  if (resumed) {
    const long long* hdr = reinterpret_cast<const long long*>(st);
    outer = hdr[0];
    counter = hdr[1];
    if (t < I) {
      fwin[t] = reinterpret_cast<const double*>(st + sl.off_f)[t];
      lnfw[t] = log(fwin[t]);
      cond[t] = reinterpret_cast<const int*>(st + sl.off_cond)[t];
    }
    perm[t] = reinterpret_cast<const int*>(st + sl.off_perm)[t];
    if (live) {
      E = reinterpret_cast<const int*>(st + sl.off_E)[t];
      rng.init(d.key_wl, static_cast<uint64_t>(t), reinterpret_cast<const unsigned long long*>(st + sl.off_pos)[t]);
      const uint32_t* ls = reinterpret_cast<const uint32_t*>(st + sl.off_lat);
      if constexpr (kReg) {
        lt.r = ls[t] | (d.nwL > 1 ? static_cast<uint64_t>(ls[P + t]) << 32 : 0ull);
      } else {
        for (int q = 0; q < d.nwL; ++q) lat_s[q * P + t] = ls[q * P + t];
      }
    }
    if (!global_g) {
      const uint32_t* hs = reinterpret_cast<const uint32_t*>(st + sl.off_H);
      const double* gs = reinterpret_cast<const double*>(st + sl.off_G);
      for (int c = 0; c < d.L; ++c) {
        H[c * P + t] = hs[c * P + t];
        G[c * P + t] = gs[c * P + t];
      }
    }
  }
  // The walker's draw ring and shadows stay between sweeps.  blk, fill: the
  // next Philox block and its ring position; fresh: the shadows (relative to
  // gs, |shadow| <= amax, high words of log g <= ghi) match log g.
  uint64_t blk = rng.pos >> 2;
  uint32_t fill = static_cast<uint32_t>(blk) * 512u;
  bool fresh = false;
  uint32_t tight_ring[kTight ? kRingSlots : 1];  // the ring in local memory where shared memory has no room
  Split gs{0.0f, 0.0f};
  float amax = 0.0f;
  int ghi = 0;
  const bool w_pow2 = (W & (W - 1)) == 0;
  if (resumed && t == 0) misc[7] = static_cast<int>(outer + 1);  // finished windows get one averaging pass
  int launch_outer = 0;  // outer iterations of this launch
  bool suspended = false;
  team.sync();

  for (;;) {
    if (d.max_outer > 0 && outer >= d.max_outer) {
      status = WLG_ERR_TIMEOUT;
      break;
    }
    // ---- WL sweep (wl.cu:1077-1175)
    const unsigned wmask = __ballot_sync(0xFFFFFFFFu, live);
    if (live) {
      const bool frozen = cond[b] != 0;
      const double lnf = lnfw[b];  // log(f) (wl.cu:1124)
      const float lnf_f = static_cast<float>(lnf);
      const float inc = frozen ? 0.0f : 1.0f;
      const uint32_t bin0 = shared_addr(pair + t);
      const uint32_t jt_a = shared_addr(base + lay.off_tab), rt_a = jt_a + align16(8 * d.Y);
      const uint32_t degs_a = jt_a + 16 * d.N;
      const uint32_t uN = static_cast<uint32_t>(d.N), uX = static_cast<uint32_t>(d.X), uY = static_cast<uint32_t>(d.Y);
      const uint32_t d_thr = d.site_thr;
      const float kInf = __int_as_float(0x7F800000);
      const uint32_t ring_a = kTight ? 0u : shared_addr(base + lay.off_ring) + (t >> 5) * kRingWarpBytes + 4 * (t & 31);
      bool stopped = false;
      for (int left = d.n_iter; left > 0 && __any_sync(wmask, !stopped);) {
        const int part = min(left, kPart);
        left -= part;
        const int c_first = min(max((E - bb) >> d.lg, 0), max(len - 1, 0));
        const int e_off = E - (bb + c_first * (1 << d.lg));  // 0 unless every proposal is bad
        // shadows of this walker's log g relative to a base near it:
        // differences inside a window stay small while values reach 1e4
        if (!fresh) {
          const double gbase = G[c_first * P + t];
          gs = split_float(gbase);
          ghi = __double2hiint(gbase);
          amax = 0.0f;
#pragma unroll 2
          for (int c = 0; c < len; ++c) {
            const double g = G[c * P + t];
            const float a = shadow_split(g, gs);
            if (kTight || pair[c * P + t].x == pair[c * P + t].x) {
              pair[c * P + t].x = a;
              amax = fmaxf(amax, fabsf(a));
              ghi = max(ghi, __double2hiint(g));
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
        float a_c = pair[c_first * P + t].x;
        if (a_c != a_c) a_c = shadow_split(G[c_first * P + t], gs);  // a start energy the pre-run did not report
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
        while (__any_sync(wmask, static_cast<int>(fill - pos) <= 12 * 128)) produce();
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
            const uint64_t xj = static_cast<uint64_t>(static_cast<uint32_t>(xi)) * uY;
            f.j = static_cast<uint32_t>(xj >> 32);
            lo_s = static_cast<uint32_t>(xj);
            if constexpr (kBonds) {
              f.col = lds_u64(jt_a + 8 * f.j);
              f.row = lds_u128(rt_a + 16 * f.i);
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
          [[maybe_unused]] uint32_t wa = 0, wb = 0, na = 0, nb = 0;  // shared words to rewrite on acceptance
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
            wa = lt.a + cs.i * lt.stride;
            wb = lt.a + min(cs.i - 1u, uX - 1u) * lt.stride;
            na = lds_u32(wa);
            nb = lds_u32(wb);
            const uint32_t m1 = cs.col.x & cs.row.x, m2 = cs.col.x & cs.row.y;
            const int unsat = __popc(na & m1) + __popc(nb & m2);
            na ^= m1;
            nb ^= m2;
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
          }
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
            int dE;
            if constexpr (kBonds) {
              w1 = lt.a + static_cast<uint32_t>(i) * lt.stride;
              w2 = lt.a + static_cast<uint32_t>(i == 0 ? d.X - 1 : i - 1) * lt.stride;
              const uint2 cm = lds_u64(jt_a + 8 * j);
              const uint4 rm = lds_u128(rt_a + 16 * i);
              const uint32_t m1 = cm.x & rm.x, m2 = cm.x & rm.y;
              n1 = lds_u32(w1);
              n2 = lds_u32(w2);
              dE = 2 * (__popc(m1) + __popc(m2) - 2 * (__popc(n1 & m1) + __popc(n2 & m2)));
              n1 ^= m1;
              n2 ^= m2;
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
              misc[1] = 1;
              // reported: the last one found, by step, then by walker
              atomicMax(new_key, static_cast<unsigned long long>(d.n_iter - left - rem) << 32 |
                                   static_cast<unsigned long long>(t) << 16 | static_cast<unsigned>(En + 32768));
            } else {
              thr = thr0;
              --rem;
              if (En >= lo && En <= hi) {
                pos += 128u;
                const int c_new = (En - bb) >> d.lg;
                const float n_new = c_new == c_cur ? n_c : lds_pair(bin0 + c_new * bin_bytes).y;
                const double g_cur = frozen ? G[c_cur * P + t] : add_times(G[c_cur * P + t], lnf, static_cast<uint32_t>(n_c));
                const double g_new =
                  frozen ? G[c_new * P + t] : add_times(G[c_new * P + t], lnf, static_cast<uint32_t>(n_new));
                if (accept_exact(x2, g_cur, g_new)) {
                  if constexpr (kReg) {
                    lt.r ^= 1ull << site;
                  } else {
                    sts_if(true, w1, n1);
                    if constexpr (kBonds) sts_if(true, w2, n2);
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
#pragma unroll 1
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
          produce();
          step(none, none);
          if (__any_sync(wmask, thr == kInf && rem > 0 && !stopped)) exact_step();
        }
        asm volatile("" ::: "memory");
        const int c_last = kTight ? static_cast<int>(cur) : static_cast<int>((cur - bin0) / bin_bytes);
        E = bb + c_last * (1 << d.lg) + e_off;
        rng.pos = pos0 + ((pos - pos_start) >> 7);
        // Fold the part's visits into histogram and log g, and with both at
        // hand refresh the shadows and take the flatness counts of
        // wl.cu:892-967 (the last part's stand).
        if (!frozen) {
          gs = split_float(fma(static_cast<double>(n_c), lnf, G[c_last * P + t]));
          amax = 0.0f;
          ghi = 0;
          uint32_t mn = 2147483647u;
          unsigned long long sum = 0;
          int cnt = 0;
          const int cb = (bb - d.e_min) >> d.lg;
#pragma unroll 2
          for (int c = 0; c < len; ++c) {
            const float2 v = pair[c * P + t];
            const uint32_t k = static_cast<uint32_t>(v.y);
            const uint32_t h = H[c * P + t] + k;
            double g = G[c * P + t];
            const bool on = kTight ? mask_has(mask, cb + c) : v.x == v.x;
            if (k != 0) {
              g = add_times(g, lnf, k);
              G[c * P + t] = g;
              H[c * P + t] = h;
            }
            const float a = shadow_split(g, gs);
            pair[c * P + t] = make_float2(kTight || on ? a : v.x, 0.0f);
            if (on) {
              mn = min(mn, h);
              sum += h;
              ++cnt;
              amax = fmaxf(amax, fabsf(a));
              ghi = max(ghi, __double2hiint(g));
            } else if (kTight) {
              amax = fmaxf(amax, fabsf(a));
              ghi = max(ghi, __double2hiint(g));
            }
          }
          if (left == 0 && cnt > 0) {
            // min >= alpha * (sum / cnt): in FP32 unless the sides are close
            const float have = static_cast<float>(mn) * static_cast<float>(cnt);
            const float want = static_cast<float>(d.alpha) * static_cast<float>(sum);
            bool is_flat = have > want;
            if (!(fabsf(have - want) > 1e-5f * fabsf(want)))
              is_flat = static_cast<double>(mn) >= d.alpha * (static_cast<double>(sum) / cnt);
            if (is_flat && atomicAdd(&flat[b], 1) == W - 1) misc[3] = static_cast<int>(outer + 1);
          }
        }
      }
    }
    team.sync();
    ++outer;
    if (misc[1] != 0) {
      status = WLG_ERR_NEW_ENERGY;
      break;
    }
    // misc stamped with the iteration: [3] a window became flat, [7] a
    // finished window still needs averaging, [6] not all windows are finished,
    // [2] a factor is above the loop's limit
    const int stamp = static_cast<int>(outer);
    // a window all of whose walkers are flat counts as finished from here on
    // (wl.cu:892-967); its state follows below
    auto finished = [&](int wb) { return cond[wb] == 1 || flat[wb] == W; };
    if (live && cond[b] == 0 && flat[b] == W)
      for (int c = 0; c < len; ++c) H[c * P + t] = 0u;
    if (live && finished(b) && stab[b] == 0) fresh = false;
    // ---- window averages (wl.cu:710-783 + :969-1031)
    const int n_avg = misc[3] == stamp || misc[7] == stamp ? I * d.L : 0;
    for (int q = t; q < n_avg; q += P) {
      const int wb = q / d.L;
      const int c = q - wb * d.L;
      if (!finished(wb) || stab[wb] != 0 || c >= w_len[wb]) continue;
      double avg = 0.0;
      if (mask_has(mask, ((w_base[wb] - d.e_min) >> d.lg) + c)) {
        // a division by a power of two is exact as a product
        if (w_pow2) {
          const double inv = 1.0 / W;
          for (int v = 0; v < W; ++v) avg += G[c * P + wb * W + v] * inv;
        } else {
          for (int v = 0; v < W; ++v) avg += G[c * P + wb * W + v] / W;
        }
      }
      bool same = true;
      for (int v = 0; v < W; ++v) {
        same = same && __double_as_longlong(G[c * P + wb * W + v]) == __double_as_longlong(avg);
        G[c * P + wb * W + v] = avg;
      }
      if (!same) chg[wb] = 1;
    }
    team.sync();
    // ---- reset and convergence (wl.cu:596-613, :662-708, mainrun.cu:243, :342-344)
    if (t < I) {
      if (cond[t] == 0 && flat[t] == W) {
        fwin[t] = sqrt(fwin[t]);
        lnfw[t] = log(fwin[t]);
        cond[t] = 1;
      }
      const double f = fwin[t];
      if (cond[t] == 1 && f > reset_lim) cond[t] = 0;
      stab[t] = cond[t] == 1 && (stab[t] != 0 || chg[t] == 0) ? 1 : 0;
      chg[t] = 0;
      flat[t] = 0;
      if (cond[t] == 1 && stab[t] == 0) misc[7] = stamp + 1;
      if (cond[t] != 1) misc[6] = stamp;
      if (f - d.loop_lim > 1e-10) misc[2] = stamp;
    }
    team.sync();
    const bool done = misc[6] != stamp;
    const bool stop = misc[2] != stamp;  // the largest factor is at the limit
    // ---- replica exchange (wl.cu:785-890)
    if (!done && counter % d.exch_every == 0) {
      if (live) {
        E_s[t] = E;
        if constexpr (kReg) {
          lat_s[t] = static_cast<uint32_t>(lt.r);
          lat_s[P + t] = static_cast<uint32_t>(lt.r >> 32);
        }
        if (keys_differ) {
          rng.init(d.key_ex, static_cast<uint64_t>(t), rng.pos);
        } else {
          rng.refill();
        }
      }
      const int nw = kReg ? 2 : d.nwL;
      for (int pass = 0; pass < 2; ++pass) {
        const int even = pass == 0;
        team.sync();
        const int par = (b + d.parity_base) & 1;
        const bool active = live && b < I - 1 && ((even && par == 0) || (!even && par == 1));
        if (active && w == 0) {  // Fisher-Yates by the window's first walker
          for (int i = W - 1; i > 0; --i) {
            // trunc(u (i + 0.999999)), as the sweep's site among i + 1
            const uint32_t x = rng.raw(), n1 = static_cast<uint32_t>(i) + 1u, thr = n1 * 2048u + 16384u;
            int r = static_cast<int>(__umulhi(x, n1));
            if (x * n1 + thr < 2u * thr) r = main_site_exact(x, i + 0.999999);
            const int tmp = perm[t + i];
            perm[t + i] = perm[t + r];
            perm[t + r] = tmp;
          }
        }
        team.sync();
        if (active) {
          const int o = (b + 1) * W + perm[t];
          const int et = E_s[t], eo = E_s[o];
          if (et >= w_start[b + 1] && et <= w_end[b + 1] && eo >= w_start[b] && eo <= w_end[b]) {
            const int nb = w_base[b + 1];
            const double gi_x = G[((et - bb) >> d.lg) * P + t];
            const double gi_y = G[((eo - bb) >> d.lg) * P + t];
            const double gj_y = G[((eo - nb) >> d.lg) * P + o];
            const double gj_x = G[((et - nb) >> d.lg) * P + o];
            if (exchange_accepts(rng.raw(), gi_x - gi_y, gj_y - gj_x)) {
              E_s[t] = eo;
              E_s[o] = et;
              for (int q = 0; q < nw; ++q) {
                const uint32_t a = lat_s[q * P + t];
                lat_s[q * P + t] = lat_s[q * P + o];
                lat_s[q * P + o] = a;
              }
            }
          }
        }
      }
      team.sync();
      if (live) {
        E = E_s[t];
        if constexpr (kReg) lt.r = lat_s[t] | static_cast<uint64_t>(lat_s[P + t]) << 32;
        if (keys_differ) rng.init(d.key_wl, static_cast<uint64_t>(t), rng.pos);
      }
    }
    if (d.exch_mode == 1) ++counter;
    team.sync();
    if (stop) break;
    if (st != nullptr && d.epoch_outer > 0 && ++launch_outer >= d.epoch_outer) {
      suspended = true;
      break;
    }
  }

  if (suspended) {  // save the state; the next launch resumes from it
    if (t == 0) {
      long long* hdr = reinterpret_cast<long long*>(st);
      hdr[0] = outer;
      hdr[1] = counter;
      reinterpret_cast<int*>(st)[4] = 1;
    }
    if (t < I) {
      reinterpret_cast<double*>(st + sl.off_f)[t] = fwin[t];
      reinterpret_cast<int*>(st + sl.off_cond)[t] = cond[t];
    }
    reinterpret_cast<int*>(st + sl.off_perm)[t] = perm[t];
    if (live) {
      reinterpret_cast<int*>(st + sl.off_E)[t] = E;
      reinterpret_cast<unsigned long long*>(st + sl.off_pos)[t] = rng.pos;
      uint32_t* ls = reinterpret_cast<uint32_t*>(st + sl.off_lat);
      for (int q = 0; q < d.nwL; ++q) {
        if constexpr (kReg) {
          ls[q * P + t] = static_cast<uint32_t>(lt.r >> (32 * q));
        } else {
          ls[q * P + t] = lat_s[q * P + t];
        }
      }
    }
    if (!global_g) {
      uint32_t* hs = reinterpret_cast<uint32_t*>(st + sl.off_H);
      double* gs = reinterpret_cast<double*>(st + sl.off_G);
      for (int c = 0; c < d.L; ++c) {
        hs[c * P + t] = H[c * P + t];
        gs[c * P + t] = G[c * P + t];
      }
    }
    if (t == 0) {
      MainResult r{};
      r.status = WLG_OK;
      r.outer = outer;
      r.flips = outer * static_cast<long long>(d.nwalk) * d.n_iter;
      r.done = 0;
      r.t_start = results[p].t_start;
      r.t_end = device_clock_ns();
      results[p] = r;
    }
    team.sync();
    return;
  }

  // ---- results
  if (live && w == 0) {
    for (int c = 0; c < d.L; ++c) outpool[d.off_out + static_cast<long long>(b) * d.L + c] = G[c * P + t];
  }
  if (t == 0) {
    MainResult r{};
    r.status = status;
    r.new_energy = misc[1] != 0 ? static_cast<int>(*new_key & 0xFFFFu) - 32768 : 0;
    r.outer = outer;
    r.flips = outer * static_cast<long long>(d.nwalk) * d.n_iter;
    r.done = 1;
    r.t_start = results[p].t_start;
    r.t_end = device_clock_ns();
    results[p] = r;
  }
  team.sync();
}

template <int kStore, bool kTight, int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads)
  k_main_batch(const MainDesc* __restrict__ descs, const int* __restrict__ order, int n, int team_size, int team_bytes,
               int global_g, int* __restrict__ next, double* __restrict__ gpool, long long gslot_doubles,
               const uint32_t* __restrict__ Jpool, const uint32_t* __restrict__ latpool,
               const int* __restrict__ winpool, const uint32_t* __restrict__ maskpool, double* __restrict__ outpool,
               MainResult* __restrict__ results, unsigned char* __restrict__ statepool)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int tix = threadIdx.x / team_size;
  Team team{team_size, team_size == 32 ? 0 : 1 + tix};
  const int t = threadIdx.x - tix * team_size;
  unsigned char* base = smem + static_cast<size_t>(tix) * team_bytes;
  int* slot = reinterpret_cast<int*>(base + team_bytes - 16);
  // tight states have no shared memory to spare for the head
  TeamHead own;
  TeamHead* head = kTight ? &own : reinterpret_cast<TeamHead*>(base);
  for (;;) {
    if (t == 0) *slot = atomicAdd(next, 1);
    team.sync();
    const int q = *slot;
    team.sync();
    if (q >= n) return;
    const int p = order[q];
    if (descs[p].off_state >= 0 && results[p].done != 0) continue;  // resumable run that finished in an earlier launch
    for (int w = kTight ? 0 : t; w < static_cast<int>(sizeof(MainDesc) / 4); w += kTight ? 1 : team_size)
      reinterpret_cast<uint32_t*>(&head->d)[w] = reinterpret_cast<const uint32_t*>(descs + p)[w];
    team.sync();
    if (kTight || t == 0) {
      head->lay = team_layout(head->d, team_size, kStore, global_g != 0, kTight);
      head->state = state_layout(team_size, head->d.I, head->d.nwL, head->d.L);
    }
    team.sync();
    double* gslot = global_g != 0 && gpool != nullptr
                      ? gpool + (static_cast<long long>(blockIdx.x) * (blockDim.x / team_size) + tix) * gslot_doubles
                      : nullptr;
    run_problem<kStore, kTight>(*head, p, team, t, base, gslot, global_g != 0, Jpool, latpool, winpool, maskpool, outpool,
                                results, statepool);
  }
}

// The kernel for a storage; tight states never keep bonds (lattice_store).
template <int kMaxThreads>
MainFn main_fn_of(int store, bool tight)
{
  switch (store) {
    case kStoreReg: return tight ? &k_main_batch<kStoreReg, true, kMaxThreads> : &k_main_batch<kStoreReg, false, kMaxThreads>;
    case kStoreTable:
      return tight ? &k_main_batch<kStoreTable, true, kMaxThreads> : &k_main_batch<kStoreTable, false, kMaxThreads>;
    case kStoreRows:
      return tight ? &k_main_batch<kStoreRows, true, kMaxThreads> : &k_main_batch<kStoreRows, false, kMaxThreads>;
    case kStoreBonds: return &k_main_batch<kStoreBonds, false, kMaxThreads>;
    default:
      return tight ? &k_main_batch<kStoreLinear, true, kMaxThreads> : &k_main_batch<kStoreLinear, false, kMaxThreads>;
  }
}

}  // namespace
}  // namespace wlg
