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
//     word (or its bonds in two) up to 32 sites a row; else linear words.
//
// Acceptance u < min(1, exp(dlogg)) is decided as log u < dlogg with FP32
// values and a proven error bound.  What FP32 cannot settle (an acceptance
// inside the bound, a site pick next to a cell edge, a draw of u = 1, an energy
// the pre-run missed) stops the walker where it stands; every sixteen steps the
// warp looks for such walkers and makes their one step with the reference's
// FP64 expressions (exact_step).  Every decision equals the reference's.
//
// What bounds it: with few walkers (one warp an SM partition) the step's serial
// chain, two dependent shared-memory loads and about 15 dependent operations;
// with four warps a partition instruction issue.  Against the step that kept
// log g itself up to date (FP64 addition, shadow and count written back on every
// change of energy, bins classified by a mask load, Philox in registers), time
// per step of the longest problem, GB300: 6x6 0.29 -> 0.12 us (247 -> 97 warp
// instructions), 12x12 0.35 -> 0.14 us, 16x16 with 512 walkers on every SM 0.94 ->
// 0.30 us, 24x24 1.12 -> 0.62 us, four such problems over clusters 0.17 us; open
// lattices of 7-11 with sweeps of 100 steps, 20.4 -> 10.9 ms per 400 iterations.
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
#include "wlg_sweep.cuh"

namespace wlg {
namespace {

constexpr double kE = 2.718281828459045;  // std::numbers::e, mainrun.cu:56

template <int kC>
struct Count {
  static constexpr int value = kC;
};

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

__device__ __forceinline__ bool mask_has(const uint32_t* mask, int c) { return (mask[c >> 5] >> (c & 31)) & 1u; }

__device__ __forceinline__ long long device_clock_ns()
{
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A problem whose windows are spread over the CTAs of a thread-block cluster
// (kCluster): every CTA runs its share as a team of its own.  Exchange between
// its last window and the next CTA's first, a new energy and the convergence
// votes go through distributed shared memory.
__device__ __forceinline__ uint32_t cluster_rank()
{
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_ranks()
{
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync()
{
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The address of p's counterpart in the shared memory of CTA `rank`.
template <typename T>
__device__ __forceinline__ T* at_rank(T* p, uint32_t rank)
{
  T* q;
  asm volatile("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
  return q;
}

// One word or one double from global to shared memory, waited for by cp.async.wait_all.
template <int kBytes>
__device__ __forceinline__ void copy_async(void* shared, const void* global)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(shared_addr(shared)), "l"(global), "n"(kBytes) : "memory");
}

template <int kStore, bool kTight, bool kCluster>
__device__ void run_problem(const TeamHead& head, int p, const Team& team, int t, unsigned char* base, double* gslot, long long gslot_doubles,
                            bool global_g, const uint32_t* __restrict__ Jpool, const uint32_t* __restrict__ latpool,
                            const int* __restrict__ winpool, const uint32_t* __restrict__ maskpool,
                            double* __restrict__ outpool, MainResult* __restrict__ results,
                            unsigned char* __restrict__ statepool)
{
  constexpr bool kTable = kStore == kStoreTable;
  constexpr bool kReg = kStore == kStoreReg || kTable;
  constexpr bool kTwo = store_two_words(kStore);
  constexpr bool kBonds = store_bonds(kStore);
  const MainDesc& d = head.d;
  const int P = team.size;
  // start time straight into the result slot: a value kept live through the
  // sweep costs the step registers
  if (t == 0 && (!kCluster || cluster_rank() == 0)) results[p].t_start = device_clock_ns();
  // resumable run: state saved at the end of a launch, restored at the start
  unsigned char* const st = !kCluster && d.off_state >= 0 ? statepool + d.off_state : nullptr;
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
  [[maybe_unused]] int* above = stab + 2 * d.I;
  int* win = reinterpret_cast<int*>(base + lay.off_win);  // start, end, base, Lb, E0
  int* misc = reinterpret_cast<int*>(base + lay.off_misc);
  // this team's windows: b0 .. b0 + I - 1 of the problem's I_all
  const int ranks = kCluster ? static_cast<int>(cluster_ranks()) : 1, rank = kCluster ? static_cast<int>(cluster_rank()) : 0;
  const int I_all = d.I, W = d.W, b0 = kCluster ? I_all * rank / ranks : 0;
  const int I = kCluster ? I_all * (rank + 1) / ranks - b0 : I_all;
  const int t0 = b0 * W;  // the problem's index of this team's first walker
  // where the team's CTAs meet, and the flags they share
  auto sync_all = [&]() {
    if constexpr (kCluster) cluster_sync();
    else team.sync();
  };
  int* misc_all = kCluster ? at_rank(misc, 0) : misc;
  unsigned long long* new_key = reinterpret_cast<unsigned long long*>(misc + 4);
  int* w_start = win;
  int* w_end = win + I;
  int* w_base = win + 2 * I;
  int* w_len = win + 3 * I;

  // ---- load the problem
  for (int q = t; q < d.nwM; q += P) mask[q] = maskpool[d.off_mask + q];
  for (int q = t; q < 2 * d.nwL; q += P) Js[q] = Jpool[d.off_J + q];
  for (int q = t; q < 5 * I; q += P) {
    const int k = q / I;
    win[q] = winpool[d.off_win + k * I_all + b0 + q - k * I];
  }
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
  const bool live = t < I * W;
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
    fill_bond_tables<kTwo>(reinterpret_cast<uint2*>(base + lay.off_tab),
                     reinterpret_cast<uint4*>(base + lay.off_tab + align16(8 * d.Y)), d.X, d.Y, open_bc, dlt_bytes, t, P);
  }
  Walker<kTight> wk;
  Lat& lt = wk.lt;
  lt.a = shared_addr(lat_s + t);
  lt.stride = static_cast<uint32_t>(4 * P);
  lt.r = 0;
  if (live && !resumed) {
    const uint32_t* src = latpool + d.off_lat + static_cast<long long>(b0 + b) * d.nwL;
    if constexpr (kReg) {
      lt.r = src[0] | (d.nwL > 1 ? static_cast<uint64_t>(src[1]) << 32 : 0ull);
    } else if constexpr (kBonds) {
      // unsatisfied bonds of the start lattice
      for (int i = 0; i < d.X; ++i) {
        uint32_t h, v;
        bond_bits(src[i], src[i + 1 < d.X ? i + 1 : 0], Jr_s[i], Jd_s[i], d.Y, open_bc, i + 1 == d.X, h, v);
        if constexpr (kTwo) {
          lat_s[2 * i * P + t] = h;
          lat_s[(2 * i + 1) * P + t] = v;
        } else {
          lat_s[i * P + t] = h | v << 16;
        }
      }
    } else {
      for (int q = 0; q < d.nwL; ++q) lat_s[q * P + t] = src[q];
    }
  }
  int& E = wk.E;
  E = live ? win[4 * I + b] : 0;
  Stream& rng = wk.rng;
  rng.init(d.key_wl, static_cast<uint64_t>(t0 + t), 0);
  const bool keys_differ = d.key_ex != static_cast<uint64_t>(d.key_wl);
  // what a factor exceeds: 2 the limit that resets a window (wl.cu:609), 1 the
  // loop's (mainrun.cu:243); kept per window, as factors rarely change (the
  // tight layout has no room for it)
  const double reset_lim = exp(d.beta);
  auto limits = [&](double f) { return (f > reset_lim ? 2 : 0) + (f - d.loop_lim > 1e-10 ? 1 : 0); };
  if constexpr (!kTight)
    for (int q = t; q < I; q += P) above[q] = limits(kE);
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
      if constexpr (!kTight) above[t] = limits(fwin[t]);
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
        for (int q = 0; q < d.nwL; ++q) copy_async<4>(lat_s + q * P + t, ls + q * P + t);
      }
    }
    // Copies that do not wait for each other, one wait for all of them: a launch's
    // prologue 39 000 -> 21 000 cycles for 25 bins a walker.  Lattices in registers,
    // with few bins, keep plain loads: ptxas schedules the step behind them 1 % better.
    if (!global_g) {
      const uint32_t* hs = reinterpret_cast<const uint32_t*>(st + sl.off_H);
      const double* gs = reinterpret_cast<const double*>(st + sl.off_G);
      for (int c = 0; c < d.L; ++c) {
        if constexpr (kReg) {
          H[c * P + t] = hs[c * P + t];
          G[c * P + t] = gs[c * P + t];
        } else {
          copy_async<4>(H + c * P + t, hs + c * P + t);
          copy_async<8>(G + c * P + t, gs + c * P + t);
        }
      }
    }
    if constexpr (!kReg) asm volatile("cp.async.wait_all;" ::: "memory");
  }
  wk.lo = lo;
  wk.hi = hi;
  wk.bb = bb;
  wk.len = len;
  wk.pair = pair + t;
  wk.ring_a = kTight ? 0u : shared_addr(base + lay.off_ring) + (t >> 5) * kRingWarpBytes + 4 * (t & 31);
  wk.start();
  const uint32_t tab_a = shared_addr(base + lay.off_tab);
  const SweepTeam common{d, P, tab_a, tab_a + (kTable ? 16 * d.N : align16(8 * d.Y)), Jr_s, Jd_s, JR, JD};
  const bool w_pow2 = (W & (W - 1)) == 0;
  // the exchange takes at most W draws of a walker, from its ring where that
  // holds them and the keys agree
  const bool ring_draws = !kTight && !keys_differ && W <= kRingAhead;
  auto draw = [&]() {
    if constexpr (!kTight) {
      if (ring_draws) return lds_u32(wk.ring_a + (static_cast<uint32_t>(rng.pos++) * 128u & 2047u));
    }
    return rng.raw();
  };
  if (resumed && t == 0) misc[7] = static_cast<int>(outer + 1);  // finished windows get one averaging pass
  int launch_outer = 0;  // outer iterations of this launch
  bool suspended = false;
  sync_all();

  for (;;) {
    if (d.max_outer > 0 && outer >= d.max_outer) {
      status = WLG_ERR_TIMEOUT;
      break;
    }
    const bool exchange_next = counter % d.exch_every == 0;
    // ---- WL sweep (wl.cu:1077-1175)
    const unsigned wmask = __ballot_sync(0xFFFFFFFFu, live);
    if (live) {
      const bool frozen = cond[b] != 0;
      const double lnf = lnfw[b];  // log(f) (wl.cu:1124)
      auto log_g = [&](int c) { return G[c * P + t]; };
      auto new_energy = [&](int En, int step) {
        misc_all[1] = 1;
        // reported: the last one found, by step, and of several the lowest walker's
        atomicMax(new_key, static_cast<unsigned long long>(step) << 32 |
                             static_cast<unsigned long long>(0xFFFF - (t0 + t)) << 16 | static_cast<unsigned>(En + 32768));
      };
      // Fold the part's visits into histogram and log g, and with both at
      // hand refresh the shadows and take the flatness counts of
      // wl.cu:892-967 (the last part's stand).
      auto fold = [&](float n_c, int c_last, bool last) {
        if (frozen) return;
        wk.gs = split_float(fma(static_cast<double>(n_c), lnf, G[c_last * P + t]));
        wk.amax = 0.0f;
        wk.ghi = 0;
        uint32_t mn = 2147483647u;
        unsigned long long sum = 0;
        int cnt = 0;
        const int cb = (bb - d.e_min) >> d.lg;
        // four bins at a time, so that their loads and integer chains overlap
        // (200 -> 70 cycles a bin); what add_times_in_binade leaves goes one by one
        const Addend add = split_addend(lnf);
        auto fold_bins = [&](int c, auto count) {
          constexpr int kN = decltype(count)::value;
          float2 v[kN];
          double g[kN];
          uint32_t h[kN], k[kN];
          unsigned slow = 0;
#pragma unroll
          for (int u = 0; u < kN; ++u) {
            v[u] = pair[(c + u) * P + t];
            g[u] = G[(c + u) * P + t];
            h[u] = H[(c + u) * P + t];
          }
#pragma unroll
          for (int u = 0; u < kN; ++u) {
            k[u] = static_cast<uint32_t>(v[u].y);
            h[u] += k[u];
            bool ok = true;
            const double sum = add_times_in_binade(g[u], add, k[u], ok);
            slow |= k[u] != 0 && !ok ? 1u << u : 0u;
            g[u] = k[u] != 0 && ok ? sum : g[u];
          }
          if (slow != 0) {
#pragma unroll
            for (int u = 0; u < kN; ++u)
              if ((slow >> u) & 1u) g[u] = add_times<false>(g[u], lnf, k[u]);
          }
#pragma unroll
          for (int u = 0; u < kN; ++u) {
            const int q = (c + u) * P + t;
            const bool on = kTight ? mask_has(mask, cb + c + u) : v[u].x == v[u].x;
            const float a = shadow_split(g[u], wk.gs);
            pair[q] = make_float2(kTight || on ? a : v[u].x, 0.0f);
            G[q] = g[u];
            H[q] = h[u];
            mn = on ? min(mn, h[u]) : mn;
            sum += on ? h[u] : 0u;
            cnt += on ? 1 : 0;
            wk.amax = kTight || on ? fmaxf(wk.amax, fabsf(a)) : wk.amax;
            wk.ghi = kTight || on ? max(wk.ghi, __double2hiint(g[u]) & 0x7FFFFFFF) : wk.ghi;
          }
        };
        int c = 0;
        for (; c + 4 <= len; c += 4) fold_bins(c, Count<4>{});
        for (; c < len; ++c) fold_bins(c, Count<1>{});
        if (last && cnt > 0) {
          // min >= alpha * (sum / cnt): in FP32 unless the sides are close
          const float have = static_cast<float>(mn) * static_cast<float>(cnt);
          const float want = static_cast<float>(d.alpha) * static_cast<float>(sum);
          bool is_flat = have > want;
          if (!(fabsf(have - want) > 1e-5f * fabsf(want)))
            is_flat = static_cast<double>(mn) >= d.alpha * (static_cast<double>(sum) / cnt);
          if (is_flat && atomicAdd(&flat[b], 1) == W - 1) misc[3] = static_cast<int>(outer + 1);
        }
      };
      wl_sweep<kStore, kTight, false>(common, wk, wmask, d.n_iter, frozen, lnf, exchange_next && ring_draws ? W : 0, log_g, is_bad, new_energy, fold);
    }
    sync_all();
    ++outer;
    if (misc_all[1] != 0) {
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
    if (live && finished(b) && stab[b] == 0) wk.fresh = false;
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
        if constexpr (!kTight) above[t] = limits(fwin[t]);
        cond[t] = 1;
      }
      const int over = kTight ? limits(fwin[t]) : above[t];
      if (cond[t] == 1 && over >= 2) cond[t] = 0;
      stab[t] = cond[t] == 1 && (stab[t] != 0 || chg[t] == 0) ? 1 : 0;
      chg[t] = 0;
      flat[t] = 0;
      if (cond[t] == 1 && stab[t] == 0) misc[7] = stamp + 1;
      if (cond[t] != 1) misc_all[6] = stamp;
      if ((over & 1) != 0) misc_all[2] = stamp;
    }
    sync_all();
    const bool done = misc_all[6] != stamp;
    const bool stop = misc_all[2] != stamp;  // the largest factor is at the limit
    // ---- replica exchange (wl.cu:785-890)
    if (!done && exchange_next) {
      if (live) {
        E_s[t] = E;
        if constexpr (kReg) {
          lat_s[t] = static_cast<uint32_t>(lt.r);
          lat_s[P + t] = static_cast<uint32_t>(lt.r >> 32);
        }
        if (keys_differ) {
          rng.init(d.key_ex, static_cast<uint64_t>(t0 + t), rng.pos);
        } else if (!ring_draws) {
          rng.refill();
        }
      }
      const int nw = kReg ? 2 : (kTwo ? 2 * d.nwL : d.nwL);
      for (int pass = 0; pass < 2; ++pass) {
        const int even = pass == 0;
        sync_all();
        const int par = (b0 + b + d.parity_base) & 1;
        const bool active = live && b0 + b < I_all - 1 && ((even && par == 0) || (!even && par == 1));
        if (active && w == 0) {  // Fisher-Yates by the window's first walker
          for (int i = W - 1; i > 0; --i) {
            // trunc(u (i + 0.999999)), as the sweep's site among i + 1
            const uint32_t x = draw(), n1 = static_cast<uint32_t>(i) + 1u, thr = n1 * 2048u + 16384u;
            int r = static_cast<int>(__umulhi(x, n1));
            if (x * n1 + thr < 2u * thr) r = main_site_exact(x, i + 0.999999);
            const int tmp = perm[t + i];
            perm[t + i] = perm[t + r];
            perm[t + r] = tmp;
          }
        }
        team.sync();
        if (active) {
          // the partner's window: the next one, or the next CTA's first
          int o = (b + 1) * W + perm[t], next = b + 1, I_next = I;
          int *E_o = E_s, *win_o = win;
          uint32_t* lat_o = lat_s;
          const double* G_o = G;
          if (kCluster && next == I) {
            o = perm[t];
            next = 0;
            I_next = I_all * (rank + 2) / ranks - I_all * (rank + 1) / ranks;
            E_o = at_rank(E_s, rank + 1);
            win_o = at_rank(win, rank + 1);
            lat_o = at_rank(lat_s, rank + 1);
            G_o = global_g ? G + gslot_doubles : at_rank(G, rank + 1);
          }
          const int et = E_s[t], eo = E_o[o];
          if (et >= win_o[next] && et <= win_o[I_next + next] && eo >= lo && eo <= hi) {
            const int nb = win_o[2 * I_next + next];
            const double gi_x = G[((et - bb) >> d.lg) * P + t];
            const double gi_y = G[((eo - bb) >> d.lg) * P + t];
            // another CTA's log g in global memory: past this SM's L1
            const auto g_o = [&](int e) {
              const double* a = G_o + ((e - nb) >> d.lg) * P + o;
              return kCluster && global_g ? __ldcg(a) : *a;
            };
            const double gj_y = g_o(eo);
            const double gj_x = g_o(et);
            if (exchange_accepts(draw(), gi_x - gi_y, gj_y - gj_x)) {
              E_s[t] = eo;
              E_o[o] = et;
              // four words at a time: their loads overlap
              for (int q = 0; q < nw; q += 4) {
                uint32_t a[4], c[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const int r = min(q + u, nw - 1) * P;
                  a[u] = lat_s[r + t];
                  c[u] = lat_o[r + o];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const int r = min(q + u, nw - 1) * P;
                  lat_s[r + t] = c[u];
                  lat_o[r + o] = a[u];
                }
              }
            }
          }
        }
      }
      sync_all();
      if (live) {
        E = E_s[t];
        if constexpr (kReg) lt.r = lat_s[t] | static_cast<uint64_t>(lat_s[P + t]) << 32;
        if (keys_differ) rng.init(d.key_wl, static_cast<uint64_t>(t0 + t), rng.pos);
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
    for (int c = 0; c < d.L; ++c) outpool[d.off_out + static_cast<long long>(b0 + b) * d.L + c] = G[c * P + t];
  }
  if (rank == 0 && t == 0) {
    MainResult r{};
    r.status = status;
    if (status == WLG_ERR_NEW_ENERGY) {
      unsigned long long key = *new_key;
      if constexpr (kCluster)
        for (int q = 1; q < ranks; ++q) key = max(key, *at_rank(new_key, q));
      r.new_energy = static_cast<int>(key & 0xFFFFu) - 32768;
    }
    r.outer = outer;
    r.flips = outer * static_cast<long long>(d.nwalk) * d.n_iter;
    r.done = 1;
    r.t_start = results[p].t_start;
    r.t_end = device_clock_ns();
    results[p] = r;
  }
  sync_all();  // no CTA leaves or starts anew while another may still reach into it
}

template <int kStore, bool kTight, bool kCluster, int kMaxThreads>
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
    int q;
    if constexpr (kCluster) {  // one problem per cluster, taken by its first CTA
      if (t == 0 && cluster_rank() == 0) *slot = atomicAdd(next, 1);
      cluster_sync();
      q = *at_rank(slot, 0);
      cluster_sync();
    } else {
      if (t == 0) *slot = atomicAdd(next, 1);
      team.sync();
      q = *slot;
      team.sync();
    }
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
    run_problem<kStore, kTight, kCluster>(*head, p, team, t, base, gslot, gslot_doubles, global_g != 0, Jpool, latpool, winpool, maskpool, outpool,
                                results, statepool);
  }
}

// The kernel for a storage; tight states never keep bonds (lattice_store).
template <int kMaxThreads>
MainFn main_fn_of(int store, bool tight)
{
#define WLG_MAIN_FN(S) \
  (tight ? &k_main_batch<S, true, false, kMaxThreads> : &k_main_batch<S, false, false, kMaxThreads>)
  switch (store) {
    case kStoreReg: return WLG_MAIN_FN(kStoreReg);
    case kStoreTable: return WLG_MAIN_FN(kStoreTable);
    case kStoreRows: return WLG_MAIN_FN(kStoreRows);
    case kStoreBonds: return &k_main_batch<kStoreBonds, false, false, kMaxThreads>;
    case kStoreBonds2: return &k_main_batch<kStoreBonds2, false, false, kMaxThreads>;
    case kStoreBondsOpen: return &k_main_batch<kStoreBondsOpen, false, false, kMaxThreads>;
    case kStoreBonds2Open: return &k_main_batch<kStoreBonds2Open, false, false, kMaxThreads>;
    default: return WLG_MAIN_FN(kStoreLinear);
  }
#undef WLG_MAIN_FN
}

// The kernel for problems spread over a cluster.
template <int kMaxThreads>
MainFn main_fn_cluster_of(int store)
{
  switch (store) {
    case kStoreReg: return &k_main_batch<kStoreReg, false, true, kMaxThreads>;
    case kStoreTable: return &k_main_batch<kStoreTable, false, true, kMaxThreads>;
    case kStoreRows: return &k_main_batch<kStoreRows, false, true, kMaxThreads>;
    case kStoreBonds: return &k_main_batch<kStoreBonds, false, true, kMaxThreads>;
    case kStoreBonds2: return &k_main_batch<kStoreBonds2, false, true, kMaxThreads>;
    case kStoreBondsOpen: return &k_main_batch<kStoreBondsOpen, false, true, kMaxThreads>;
    case kStoreBonds2Open: return &k_main_batch<kStoreBonds2Open, false, true, kMaxThreads>;
    default: return &k_main_batch<kStoreLinear, false, true, kMaxThreads>;
  }
}

}  // namespace
}  // namespace wlg
