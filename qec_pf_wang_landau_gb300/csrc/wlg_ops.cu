// Operator layer: one sm_103a kernel per device operation of the reference's
// kernel library (src/wl.cu of dfki-ric-quantum/qec_pf_wang_landau), on the
// reference's data layout, behind the extern "C" entry points of wlg.h.
//
// Layout (shared with the reference): spins int8 +-1, lattice t at
// d_offset_lattice[t]; couplings int8 [sample][2N] with the right bond of
// site (i,j) at i*Y+j and its down bond at N+i*Y+j; per-walker dense
// histogram / log g slices starting at d_offset_histogram[t], indexed by
// E - start[window]; walker t belongs to window t / W and sample t / (I*W).

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <algorithm>
#include <cstdio>

#include "../../include/wlg.h"
#include "wlg_internal.h"
#include "wlg_lattice.cuh"
#include "wlg_pre.cuh"
#include "wlg_sweep.cuh"
#include "wlg_rng.cuh"

namespace wlg {
namespace {

constexpr int kThreads = 128;

// -------------------------------------------------------------- disorder ----

// t / n, mostly as 32-bit numbers (a 64-bit division is some 100 instructions).
__device__ __forceinline__ size_t divide(size_t t, size_t n)
{
  return ((t | n) >> 32) == 0 ? static_cast<uint32_t>(t) / static_cast<uint32_t>(n) : t / n;
}

// SMs of the current device.
inline int sm_count()
{
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return 1;
  return std::max(sms, 1);
}

// Element t of a sample takes the stream's draw t: a thread takes the four of a
// Philox block.
__global__ void k_init_interactions(int8_t* __restrict__ J, size_t N, int R, int seed, float prob)
{
  const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t blocks = (2 * N + 3) / 4;
  if (t >= blocks * static_cast<size_t>(R)) return;
  const size_t k = divide(t, blocks), first = 4 * (t - k * blocks);
  Stream st;
  st.init(key_size(seed, k), 0, first);
  const uint32_t x[4] = {st.blk.x, st.blk.y, st.blk.z, st.blk.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double u = unit_float(x[q]);
    if (first + q < 2 * N) J[k * 2 * N + first + q] = (u < prob) ? -1 : 1;
  }
}

// which: 0 = horizontal chain (down bonds of row 0), 1 = vertical chain
// (right bonds of column 0).
__global__ void k_apply_chain(int8_t* __restrict__ J, int X, int Y, int R, int which)
{
  const int len = which == 0 ? Y : X;
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<long long>(len) * R) return;
  const size_t N = static_cast<size_t>(X) * Y;
  const size_t k = static_cast<size_t>(t / len);
  const int q = static_cast<int>(t % len);
  const size_t idx = k * 2 * N + (which == 0 ? N + q : static_cast<size_t>(q) * Y);
  J[idx] = static_cast<int8_t>(-J[idx]);
}

// Draw 0 of a sample is its share of -1 spins, site s takes draw s + 1: a thread
// takes the sites of a Philox block.  8192 lattices of 9x9 8.2 -> 4.2 us, 2^20 of 4x4 123 -> 45.
__global__ void k_init_lattice(int8_t* __restrict__ lat, int X, int Y, size_t num_lattices, int seed, int wpi)
{
  const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t N = static_cast<size_t>(X) * Y, blocks = N / 4 + 1;
  if (t >= blocks * num_lattices) return;
  const size_t l = divide(t, blocks), first = 4 * (t - l * blocks);
  const uint64_t key = key_u32(seed, divide(l, static_cast<size_t>(wpi)));
  Stream st;
  st.init(key, 1, 0);
  const float p0 = st.uniform();
  st.init(key, 1, first);
  const uint32_t x[4] = {st.blk.x, st.blk.y, st.blk.z, st.blk.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double u = unit_float(x[q]);
    if (first + q >= 1 && first + q <= N) lat[l * N + first + q - 1] = (u < p0) ? -1 : 1;
  }
}

// ---------------------------------------------------------------- energy ----

// wl.cu:261-340, a thread or a warp per lattice: a warp's loads lie side by side
// and do not wait for each other, at a division a site.
// us with 1 / 32 lanes: 8192 lattices of 9x9 8.3 / 6.3, 32 768 10.3 / 14.4; 12x12,
// 4096 12.4 / 6.2, 131 072 63 / 55; 24x24, 8192 71 / 14; 5x5, 16 384 4.2 / 6.3.
inline int energy_lanes(long long N, size_t num_lattices)
{
  return N >= 128 || (N >= 48 && num_lattices <= 8192) ? 32 : 1;
}
__global__ void k_calc_energy(int boundary, int* __restrict__ E, const int8_t* __restrict__ lat,
                              const int8_t* __restrict__ J, const int* __restrict__ off_lat, int X, int Y,
                              size_t num_lattices, int wpi, int lanes)
{
  const size_t t = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) / lanes;
  const int lane = threadIdx.x & (lanes - 1), N = X * Y;
  int acc = 0;
  if (lanes == 1) {
    if (t < num_lattices) E[t] = energy_i8(lat + off_lat[t], J + divide(t, static_cast<size_t>(wpi)) * 2 * N, X, Y, boundary);
    return;
  }
  if (t < num_lattices) {
    const int8_t* s = lat + off_lat[t];
    const int8_t* Jk = J + divide(t, static_cast<size_t>(wpi)) * 2 * N;
#pragma unroll 4
    for (int site = lane; site < N; site += lanes) {
      const int i = static_cast<int>(static_cast<unsigned>(site) / static_cast<unsigned>(Y)), j = site - i * Y;
      const int above = i > 0 ? site - Y : site + N - Y, before = j > 0 ? site - 1 : site + Y - 1;
      int up = s[above] * Jk[N + above];
      int left = s[before] * Jk[before];
      if (boundary == 1) {
        up = i == 0 ? 0 : up;
        left = j == 0 ? 0 : left;
      }
      acc += s[site] * (up + left);
    }
  }
  for (int d = lanes / 2; d > 0; d >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, d);
  if (lane == 0 && t < num_lattices) E[t] = -acc;
}

// --------------------------------------------------------------- pre-run ----
// One CTA per sample, one thread per walker (round-synchronous, see
// wlg_pre.cuh).
struct PrerunArgs {
  int* E;
  int* flag_found;
  int8_t* lat;
  int8_t* found_lat;
  unsigned long long* H;
  uint64_t* seed_off;
  const int8_t* J;
  const int* off_lat;
  int E_min, E_max, n_iter, X, Y, seed, n_int, len_int, wpi, boundary;
  int bonds;  // the walk on bond words fits
};

// The walk on bond words, on the caller's lattices, histogram and draws.
template <bool kTwo, bool kKeys>
__device__ __forceinline__ void prerun_bonds(const PrerunArgs& a, unsigned char* smem)
{
  constexpr int kW = kTwo ? 2 : 1;
  const int k = blockIdx.x, w = threadIdx.x, X = a.X, Y = a.Y, N = X * Y;
  const int lg = energy_step_log2(a.boundary), all = a.E_max - a.E_min + 1, len = ((all - 1) >> lg) + 1;
  const int threads = blockDim.x, Lh = pre_hist_words(len);
  const bool live = w < a.wpi;
  const size_t t = static_cast<size_t>(k) * a.wpi + w;
  const PreLayout l = pre_layout(X, Y, len, a.n_int, threads);
  uint32_t* hist = reinterpret_cast<uint32_t*>(smem + l.off_hist);
  uint32_t* thr = reinterpret_cast<uint32_t*>(smem + l.off_thr);
  uint32_t* Jr = reinterpret_cast<uint32_t*>(smem + l.off_J);
  uint2* col = reinterpret_cast<uint2*>(smem + l.off_col);
  uint4* row = reinterpret_cast<uint4*>(smem + l.off_row);
  PreWalk p{X, Y, a.boundary, a.E_min, lg, len, Lh, 0, a.n_int, min(a.len_int, 1 << 15), a.n_iter, threads, hist,
                  reinterpret_cast<uint32_t*>(smem + l.off_claim), reinterpret_cast<int*>(smem + l.off_foundE), thr, col,
                  row, Jr, Jr + X, reinterpret_cast<uint32_t*>(smem + l.off_words),
                  a.found_lat + static_cast<long long>(k) * a.n_int * N};
  const PreSync sync{threads};
  // all walkers of a sample have energies a step apart (k_prerun)
  p.bin0 = (a.E[static_cast<size_t>(k) * a.wpi] - a.E_min) & ((1 << lg) - 1);
  p.e_min += p.bin0;
  p.len = (all - 1 - p.bin0 >> lg) + 1;
  for (int q = w; q < Lh; q += threads) {
    const int e = p.bin0 + (q << lg);
    const uint32_t h = e < all ? static_cast<uint32_t>(a.H[static_cast<size_t>(k) * all + e]) : 0u;
    hist[q] = hist[Lh + q] = h;
  }
  for (int q = w; q < a.n_int; q += threads)
    p.claim[q] = a.flag_found[static_cast<size_t>(k) * a.n_int + q] == 0 ? kPreEmpty : 0u;
  for (int q = w; q < X; q += threads) {
    const int8_t* Jk = a.J + static_cast<size_t>(k) * 2 * N + q * Y;
    uint32_t r = 0, dn = 0;
#pragma unroll 8
    for (int j = 0; j < Y; ++j) {
      r |= Jk[j] < 0 ? 1u << j : 0u;
      dn |= Jk[N + j] < 0 ? 1u << j : 0u;
    }
    Jr[q] = r;
    Jr[X + q] = dn;
  }
  fill_accept(thr, w);
  fill_bonds<kTwo>(col, row, X, Y, a.boundary, w, threads);
  sync();
  int8_t* s = live ? a.lat + a.off_lat[t] : nullptr;
  auto row_bits = [&](int i) {
    uint32_t r = 0;
#pragma unroll 8
    for (int j = 0; j < Y; ++j) r |= s[i * Y + j] < 0 ? 1u << j : 0u;
    return r;
  };
  uint32_t s0 = 0;
  int E = 0;
  uint64_t pos = 0;
  if (live) {
    const uint32_t first = row_bits(0);
    uint32_t r = first;
    for (int i = 0; i < X; ++i) {
      const uint32_t dn = i + 1 < X ? row_bits(i + 1) : first;
      uint32_t h, v = 0;
      bond_words<kTwo>(r, dn, Jr[i], Jr[X + i], Y, a.boundary != 0, i + 1 == X, h, v);
      p.words[i * kW * threads + w] = h;
      if constexpr (kTwo) p.words[(i * kW + 1) * threads + w] = v;
      r = dn;
    }
    s0 = first & 1u;
    E = a.E[t];
    pos = a.seed_off[t];
  } else {
    for (int q = 0; q < X * kW; ++q) p.words[q * threads + w] = 0;
  }
  pre_walk<kTwo, true, kKeys>(p, sync, w, live, key_u32(a.seed, static_cast<uint64_t>(k)), 2 + static_cast<uint64_t>(w), pos, E,
                       s0);
  for (int q = w; q < p.len; q += threads) a.H[static_cast<size_t>(k) * all + p.bin0 + (q << lg)] = hist[q];
  for (int q = w; q < a.n_int; q += threads)
    if (p.claim[q] != kPreEmpty && p.claim[q] != 0u) a.flag_found[static_cast<size_t>(k) * a.n_int + q] = 1;
  if (live) {
    // spins from the bonds: down column 0, then along each row
    uint32_t edge = s0;
    for (int i = 0; i < X; ++i) {
      const uint32_t word = p.words[i * kW * threads + w];
      const uint32_t turn = word ^ Jr[i];
      uint32_t sp = edge;
      for (int j = 0; j < Y; ++j) {
        s[i * Y + j] = sp != 0 ? -1 : 1;
        sp ^= (turn >> j) & 1u;
      }
      edge ^= ((kTwo ? p.words[(i * kW + 1) * threads + w] : word >> 16) ^ Jr[X + i]) & 1u;
    }
    a.E[t] = E;
    a.seed_off[t] = pos;
  }
}

// The walk on the caller's int8 lattices with 64-bit counts, for everything
// else: values other than +-1, odd draw offsets, counts of 2^31 and more, rows of
// more than 32 sites.
__device__ __forceinline__ void prerun_i8(const PrerunArgs& a, unsigned char* smem)
{
  int* const E = a.E;
  int* const flag_found = a.flag_found;
  unsigned long long* const H = a.H;
  const int E_min = a.E_min, E_max = a.E_max, X = a.X, Y = a.Y, n_int = a.n_int, wpi = a.wpi, boundary = a.boundary;
  const int len_hist = E_max - E_min + 1;
  unsigned long long* hist = reinterpret_cast<unsigned long long*>(smem);
  int* claim = reinterpret_cast<int*>(hist + len_hist);
  int* found = claim + n_int;

  const int k = blockIdx.x;
  const int w = threadIdx.x;
  const int N = X * Y;
  const bool live = w < wpi;
  const size_t t = static_cast<size_t>(k) * wpi + w;

  for (int q = threadIdx.x; q < len_hist; q += blockDim.x) hist[q] = H[static_cast<size_t>(k) * len_hist + q];
  for (int q = threadIdx.x; q < n_int; q += blockDim.x) {
    claim[q] = INT_MAX;
    found[q] = flag_found[static_cast<size_t>(k) * n_int + q];
  }

  Stream rng;
  int energy = 0;
  int8_t* s = nullptr;
  bool ok = true;
  if (live) {
    rng.init(key_u32(a.seed, static_cast<uint64_t>(k)), 2 + static_cast<uint64_t>(w), a.seed_off[t]);
    energy = E[t];
    s = a.lat + a.off_lat[t];
    ok = energy >= E_min && energy <= E_max;  // a walker outside the range never indexes the histogram
  }
  const int8_t* Jk = a.J + static_cast<size_t>(k) * 2 * N;
  const double site_scale = (N - 1 + 0.999999);
  __syncthreads();

  for (int it = 0; it < a.n_iter; ++it) {
    int hit = -1;
    bool acc = false;
    if (live && ok) {
      const Move m = propose_i8(rng, s, Jk, energy, X, Y, site_scale, boundary);
      if (m.new_energy > E_max || m.new_energy < E_min) {  // wl.cu:522-529: the walker stops
        energy = m.new_energy;                               // and keeps the offending energy
        ok = false;
      } else {
        const int io = energy - E_min;
        const int in = m.new_energy - E_min;
        const double prob = exp(static_cast<double>(hist[io]) - static_cast<double>(hist[in]));
        const double u = rng.uniform();
        if (u < prob) {
          s[m.site] = static_cast<int8_t>(-s[m.site]);
          energy = m.new_energy;
          acc = true;
          hit = in;
        } else {
          hit = io;
        }
      }
    }
    __syncthreads();
    int bin = -1;
    if (hit >= 0) atomicAdd(&hist[hit], 1ull);
    if (acc) {
      const int q = (energy - E_min) / a.len_int;
      bin = (q < n_int) ? q : n_int - 1;
      if (found[bin] == 0) atomicMin(&claim[bin], w);
      else bin = -1;
    }
    __syncthreads();
    if (bin >= 0 && claim[bin] == w && found[bin] == 0) {
      found[bin] = 1;
      int8_t* dst = a.found_lat + (static_cast<size_t>(k) * n_int + bin) * N;
      for (int q = 0; q < N; ++q) dst[q] = s[q];
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < len_hist; q += blockDim.x) H[static_cast<size_t>(k) * len_hist + q] = hist[q];
  for (int q = threadIdx.x; q < n_int; q += blockDim.x)
    flag_found[static_cast<size_t>(k) * n_int + q] = found[q];
  if (live) {
    E[t] = energy;
    a.seed_off[t] = rng.pos;
  }
}

template <int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads, 1) k_prerun(const PrerunArgs a)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int k = blockIdx.x, N = a.X * a.Y, len = a.E_max - a.E_min + 1;
  bool fast = a.bonds != 0;
  if (fast) {
    // every load is made whatever came before it, so that they overlap: a call
    // of 10 rounds on 64 samples of 9x9 33 -> 25 us
    auto spin = [](int v) { return (v == 1) | (v == -1); };
    for (int q = threadIdx.x; q < 2 * N; q += blockDim.x) fast &= spin(a.J[static_cast<size_t>(k) * 2 * N + q]);
    const unsigned long long most = (1ull << 31) - 1 - static_cast<unsigned long long>(a.n_iter) * a.wpi;
    for (int q = threadIdx.x; q < len; q += blockDim.x) fast &= a.H[static_cast<size_t>(k) * len + q] <= most;
    const int w = threadIdx.x;
    const size_t t = static_cast<size_t>(k) * a.wpi + w;
    if constexpr (kMaxThreads > 256) {
      // More lattices than the L1 cache holds lines for: a warp reads one after
      // another, 32 sites in one piece (1024 walkers of 24x24 640 -> 78 us; 128
      // walkers 44 -> 58).
      const int lane = w & 31, mine = min(32, a.wpi - (w - lane));
      const long long at = w < a.wpi ? a.off_lat[t] : 0;
#pragma unroll 4
      for (int j = 0; j < mine; ++j) {
        const int8_t* s = a.lat + __shfl_sync(0xFFFFFFFFu, at, j);
#pragma unroll 4
        for (int q = lane; q < N; q += 32) fast &= spin(s[q]);
      }
    } else if (w < a.wpi) {
      const int8_t* s = a.lat + a.off_lat[t];
#pragma unroll 16
      for (int q = 0; q < N; ++q) fast &= spin(s[q]);
    }
    if (w < a.wpi) {
      fast = fast && (a.seed_off[t] & 1u) == 0;
      // energies on one grid, as the lattices of one sample have them
      fast = fast && ((a.E[t] - a.E[static_cast<size_t>(k) * a.wpi]) & ((1 << energy_step_log2(a.boundary)) - 1)) == 0;
    }
  }
  if (__syncthreads_and(fast ? 1 : 0) == 0) {
    prerun_i8(a, smem);
  } else if (a.Y <= 16) {
    prerun_bonds<false, kMaxThreads <= 256>(a, smem);
  } else {
    prerun_bonds<true, kMaxThreads <= 256>(a, smem);
  }
}

// Whether n_iter rounds make up for packing a sample's walkers into bond words.
// Packing and unpacking cost about 6 us and, per site, 60 ns and what the walkers'
// strided lattices cost; an int8 round is 1.6 us longer than one on bond words, and
// 10 ns per walker where there are many.  Samples beyond one an SM wait for each
// other.  us of a call, bond words / int8: 64 samples of 9x9, 128 walkers, 5 rounds
// 29 / 27, 20 rounds 32 / 60; 64 of 16x16, 20 rounds 94 / 74, 80 rounds 107 / 194; 2 of
// 24x24, 1024 walkers, 80 rounds 1446 / 1051, 160 rounds 1615 / 1917; 400 of 16x16, 40
// rounds 233 / 162, 80 rounds 246 / 287.
inline bool bonds_pay(long long N, long long walkers, long long n_iter, long long samples)
{
  const long long sms = sm_count();
  const long long pack_ns = (6000 + N * (60 + walkers + walkers * walkers / 1024)) * std::max(samples, sms) / sms;
  const long long round_ns = std::max(1600ll, 10 * walkers) * std::max(samples, 2 * sms) / (2 * sms);
  return n_iter * round_ns >= pack_ns;
}

// ------------------------------------------------------- main WL sweep -----
// wl.cu:1033-1175 on the caller's arrays.
struct SweepArgs {
  int8_t* lat;
  const int8_t* J;
  unsigned long long* H;
  double* logG;
  const double* factor;
  int* E;
  int* newE;
  uint64_t* off_iter;
  int* found;
  const int *start, *end, *off_hist, *off_lat;
  const int8_t *cond, *spectrum;
  const int *off_spec, *cond_inter;
  int X, Y, n_iter, num_lattices, n_int, wpi, seed, boundary;
  int L;           // bins a walker's column holds (k_wl_sweep)
  uint32_t magic;  // site / Y = site * magic >> 20
};

// One walker by one thread, straight on global memory.  The parameters' __restrict__
// lets couplings, windows and spectrum be read past the stores: 64x32, 64 steps 154
// -> 126 us against the same body on a struct of pointers.
__device__ __forceinline__ void sweep_global(
    int t, int8_t* __restrict__ lat, const int8_t* __restrict__ J, unsigned long long* __restrict__ H, double* __restrict__ logG,
    const double* __restrict__ factor, int* __restrict__ E, int* __restrict__ newE, uint64_t* __restrict__ off_iter,
    int* __restrict__ found, const int* __restrict__ start, const int* __restrict__ end,
    const int* __restrict__ off_hist, const int* __restrict__ off_lat, const int8_t* __restrict__ cond,
    const int8_t* __restrict__ spectrum, const int* __restrict__ off_spec, const int* __restrict__ cond_inter, int X, int Y,
    int n_iter, int num_lattices, int n_int, int wpi, int seed, int boundary)
{
  const int W = wpi / n_int;
  const int k = t / wpi;
  const int b = t / W;
  const int N = X * Y;
  Stream rng;
  rng.init(key_u32(seed, static_cast<uint64_t>(k)), static_cast<uint64_t>(t % wpi), off_iter[t]);
  int8_t* s = lat + off_lat[t];
  const int8_t* Jk = J + static_cast<size_t>(k) * 2 * N;
  const int8_t* mask = spectrum + off_spec[k] - start[k * n_int];
  const int e_first = start[k * n_int], e_last = end[k * n_int + n_int - 1];
  const int lo = start[b], hi = end[b];
  unsigned long long* Hw = H + off_hist[t] - lo;
  double* Gw = logG + off_hist[t] - lo;
  const double lnf = log(factor[t]);
  const double site_scale = (N - 1 + 0.999999);
  const bool frozen = cond[b] != 0;
  int energy = E[t];
  int flag = 0;
  for (int it = 0; it < n_iter; ++it) {
    const Move m = propose_i8(rng, s, Jk, energy, X, Y, site_scale, boundary);
    // wl.cu:1091-1104; an energy outside the sample's spectrum range counts
    // as new too (the reference reads the mask out of bounds there).
    if (m.new_energy < e_first || m.new_energy > e_last || mask[m.new_energy] != 1) {
      flag = t + 1;
      newE[t] = m.new_energy;
      break;
    }
    const bool inside = m.new_energy <= hi && m.new_energy >= lo;
    if (!frozen) {
      if (!inside) {
        Hw[energy] += 1;
        Gw[energy] += lnf;
        continue;
      }
      const double prob = fmin(1.0, exp(Gw[energy] - Gw[m.new_energy]));
      const double u = rng.uniform();
      if (u < prob) {
        s[m.site] = static_cast<int8_t>(-s[m.site]);
        energy = m.new_energy;
      }
      Hw[energy] += 1;
      Gw[energy] += lnf;
    } else if (inside) {
      const double prob = fmin(1.0, exp(Gw[energy] - Gw[m.new_energy]));
      const double u = rng.uniform();
      if (u < prob) {
        s[m.site] = static_cast<int8_t>(-s[m.site]);
        energy = m.new_energy;
      }
    }
  }
  if (n_iter > 0) found[t] = flag;
  E[t] = energy;
  off_iter[t] = rng.pos;
}

__global__ void k_wang_landau(
    int8_t* __restrict__ lat, const int8_t* __restrict__ J, unsigned long long* __restrict__ H, double* __restrict__ logG,
    const double* __restrict__ factor, int* __restrict__ E, int* __restrict__ newE, uint64_t* __restrict__ off_iter,
    int* __restrict__ found, const int* __restrict__ start, const int* __restrict__ end,
    const int* __restrict__ off_hist, const int* __restrict__ off_lat, const int8_t* __restrict__ cond,
    const int8_t* __restrict__ spectrum, const int* __restrict__ off_spec, const int* __restrict__ cond_inter, int X, int Y,
    int n_iter, int num_lattices, int n_int, int wpi, int seed, int boundary)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= num_lattices || cond_inter[t / wpi] == -1) return;
  sweep_global(t, lat, J, H, logG, factor, E, newE, off_iter, found, start, end, off_hist, off_lat, cond, spectrum, off_spec,
               cond_inter, X, Y, n_iter, num_lattices, n_int, wpi, seed, boundary);
}

// Shared memory of k_wl_sweep: 32 walkers (bytes).
constexpr int kSweepWarps = 8;  // at most
static_assert(8 * 32 * kSweepWarps <= kRingWarpBytes);
struct SweepLayout {
  int off_desc, off_J, off_tab, off_ring, off_lat, off_pair, bytes;
};
WLG_HD inline SweepLayout sweep_layout(int X, int Y, int L, int lg)
{
  SweepLayout l{};
  int o = 0;
  l.off_desc = o;
  o = align16(o + static_cast<int>(sizeof(MainDesc)));
  l.off_J = o;
  o = align16(o + 8 * X);
  l.off_tab = o;
  o = align16(o + align16(8 * Y) + 16 * X);
  l.off_ring = o;
  o = align16(o + kRingWarpBytes);
  l.off_lat = o;
  o = align16(o + 4 * X * 32);
  l.off_pair = o;
  o = align16(o + 8 * (L + 2 * guard_bins(lg)) * 32);
  l.bytes = o;
  return l;
}

// How a call makes its sweep.
struct SweepPlan {
  int warps;  // of a block
  bool pays;  // packed walkers, or the walk on global memory
};
// Warps a block: helpers while all blocks fit beside each other (by their registers
// two blocks of 8 warps on an SM, or four of 4), or where shared memory leaves room
// for no more; else one warp, each lane packing its own walker.  1 / 4 / 8 warps, us
// for 1 and 1000 steps: 10x10, 32 blocks 27 199 / 21 180 / 17 173; 10x10, 512 blocks
// 40 212 / 25 187 / 33 343 (two waves); 6x6, 1024 blocks 21 211 / 31 324 / 47 619.
// Packing costs a block with 8 warps about 3 us, 36 ns a site and 30 ns a bin of
// the columns, twice that for each of several waves, and single warps 0.65 ns a site
// of all blocks together; a step on global memory takes 1 us and more, 1 us per
// 20 000 walkers.  A sweep whose steps do not make up for the packing stays on
// global memory.  us of a call, packed / global: 6x6, 15 blocks, 4 steps 14 / 13, 16 steps 17 / 31; 16x16, 256
// blocks, 8 steps 28 / 22, 32 steps 35 / 58; 32x32, 8 blocks, 8 steps 67 / 21, 64 steps
// 90 / 112; 10x10, 3200 blocks, 16 steps 222 / 96, 64 steps 241 / 345.
inline SweepPlan sweep_plan(const SweepArgs& a, int blocks, int bytes)
{
  const int sms = sm_count();
  const int room = std::max(kSharedBytes / (bytes + 1024), 1);  // blocks an SM's shared memory holds
  SweepPlan p{1, false};
  if (blocks <= 2 * sms || room <= 2) p.warps = kSweepWarps;
  else if (blocks <= 4 * sms || room <= 4) p.warps = kSweepWarps / 2;
  const long long beside = static_cast<long long>(sms) * std::min(room, p.warps > 1 ? 16 / p.warps : 16);
  const long long waves = (blocks + beside - 1) / beside, N = static_cast<long long>(a.X) * a.Y;
  const long long block_ns = kSweepWarps / p.warps * (3000 + 36 * N + 30ll * a.L);
  const long long pack_ns = p.warps > 1 ? (waves > 1 ? 2 * waves : 1) * block_ns
                                        : std::max(13 * N * blocks * 152 / (20ll * sms), (waves - 1) * block_ns);
  const long long step_ns = std::max(std::max(1000, a.num_lattices / 20) - 200 * (waves - 1), 100ll);
  p.pays = a.n_iter * step_ns >= pack_ns;
  return p;
}

// The sweep of the persistent main run (wlg_sweep.cuh) on the caller's arrays:
// the first warp of a block walks 32 walkers of a sample.  All its warps pack
// the lattices (bonds or rows) and the bins of the windows into shared memory,
// and write lattices, visits and log g back at the end: a warp reads and writes
// a lattice 32 sites at a time, and the bins of the walkers are dealt out over
// the warps, because these short chains of dependent global loads, not bytes,
// are what a short sweep spends its time on.
// The step on global memory is one chain of dependent loads and an FP64 exp,
// 1.2 to 2 us with few walkers; here 0.13 us.  With helpers, loads that do not wait
// for each other and the shadows made while packing, a call of 200 steps took, us:
// 1024 walkers of 10x10 84 -> 52, 8192 of 6x6 61 -> 50; 81 920 walkers, 1000 steps:
// 10x10 599 -> 562, 6x6 411 -> 440.  A run of 16 samples of 6x6 on the operators 5.4
// -> 5.0 ms (45 with the step on global memory).
// Blocks with arrays the sweep does not take (couplings or spins other than
// +-1, log g of 2^100 and more, factors below 1, an energy outside its window,
// windows wider than the columns) walk on global memory.
template <int kStore>
__global__ void __launch_bounds__(32 * kSweepWarps) k_wl_sweep(const SweepArgs a)
{
  constexpr bool kBonds = store_bonds(kStore);
  constexpr unsigned kAll = 0xFFFFFFFFu;
  extern __shared__ __align__(16) unsigned char smem[];
  const int groups = (a.wpi + 31) / 32, tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, warps = nt >> 5;
  // every warp: a lane per walker
  const int k = blockIdx.x / groups, w = (blockIdx.x - k * groups) * 32 + lane, t = k * a.wpi + w;
  const bool live = w < a.wpi && t < a.num_lattices;
  if (a.cond_inter[k] == -1) return;
  const unsigned wmask = __ballot_sync(kAll, live);
  const int X = a.X, Y = a.Y, N = X * Y, lg = a.boundary == 0 ? 2 : 1, guard = guard_bins(lg);
  const bool open = a.boundary != 0;
  const uint32_t row_mask = Y == 32 ? kAll : (1u << Y) - 1u;
  const SweepLayout l = sweep_layout(X, Y, a.L, lg);
  MainDesc& d = *reinterpret_cast<MainDesc*>(smem + l.off_desc);
  uint32_t* Jr = reinterpret_cast<uint32_t*>(smem + l.off_J);
  uint32_t* words = reinterpret_cast<uint32_t*>(smem + l.off_lat);  // word r of walker q: [r * 32 + q]
  float2* top = reinterpret_cast<float2*>(smem + l.off_ring);  // until the walk begins
  float2* pair = reinterpret_cast<float2*>(smem + l.off_pair) + guard * 32 + lane;
  const long long at = live ? a.off_lat[t] : 0;
  bool ok = true;
  // sites to words of 32
  const int nw = (N + 31) / 32;
  if (warps == 1) {  // a lane a walker
    for (int c = 0; c < nw && live; ++c) {
      const int8_t* s = a.lat + at + c * 32;
      const int n = min(32, N - c * 32);
      uint32_t bits = 0;
#pragma unroll 8
      for (int j = 0; j < n; ++j) {
        const int v = s[j];
        ok = ok && (v == 1 || v == -1);
        bits |= v < 0 ? 1u << j : 0u;
      }
      words[c * 32 + lane] = bits;
    }
  } else {
#pragma unroll 8
    for (int x = warp; x < 32 * nw; x += warps) {
      const int q = x & 31, site = (x >> 5) * 32 + lane;
      const int8_t* s = a.lat + __shfl_sync(kAll, at, q);
      const int v = ((wmask >> q) & 1u) != 0 && site < N ? s[site] : 1;
      ok = ok && (v == 1 || v == -1);
      const uint32_t bits = __ballot_sync(kAll, v < 0);
      if (lane == 0) words[x] = bits;
    }
  }
  if (tid == 0) {
    d.X = X;
    d.Y = Y;
    d.N = N;
    d.boundary = a.boundary;
    d.lg = lg;
    d.site_thr = static_cast<uint32_t>(N) * 2048u + 16384u;
    d.site_scale = (N - 1 + 0.999999);
    d.site_magic = a.magic;
  }
  const int8_t* Jk = a.J + static_cast<size_t>(k) * 2 * N;
  for (int q = nt - 1 - tid; q < 2 * X; q += nt) {  // coupling bits: right, then down
    const int8_t* src = Jk + q * Y;
    uint32_t bits = 0;
#pragma unroll 8
    for (int j = 0; j < Y; ++j) {
      const int v = src[j];
      ok = ok && (v == 1 || v == -1);
      bits |= v < 0 ? 1u << j : 0u;
    }
    Jr[q] = bits;
  }
  uint2* col = reinterpret_cast<uint2*>(smem + l.off_tab);
  fill_bond_tables<false>(col, reinterpret_cast<uint4*>(smem + l.off_tab + align16(8 * Y)), X, Y, open, 2 * (256 >> lg),
                          tid, nt);
  const int b = t / (a.wpi / a.n_int);
  const int e_first = a.start[k * a.n_int], e_last = a.end[k * a.n_int + a.n_int - 1];
  const int8_t* mask = a.spectrum + a.off_spec[k] - e_first;
  auto is_bad = [&](int En) { return En < e_first || En > e_last || mask[En] != 1; };
  Walker<false> wk;
  wk.lo = wk.hi = wk.bb = wk.len = wk.E = 0;
  double lnf = 0.0;
  unsigned long long* H = nullptr;
  double* G = nullptr;
  bool frozen = true;
  Split gs{0.0f, 0.0f};
  float amax = 0.0f;
  int ghi = 0;
  if (live) {
    wk.E = a.E[t];
    wk.lo = a.start[b];
    wk.hi = a.end[b];
    frozen = a.cond[b] != 0;
    bool own = wk.E >= wk.lo && wk.E <= wk.hi;
    wk.bb = wk.lo + ((wk.E - wk.lo) & ((1 << lg) - 1));  // the walker's energies, a step apart
    wk.len = ((wk.hi - wk.bb) >> lg) + 1;
    own = own && wk.len <= a.L;
    lnf = log(a.factor[t]);
    own = own && lnf >= 0.0 && lnf < 1e6;
    H = a.H + a.off_hist[t] + (wk.bb - wk.lo);
    G = a.logG + a.off_hist[t] + (wk.bb - wk.lo);
    if (own) {  // bins with their shadows (wl_sweep)
      const double gbase = G[wk.E - wk.bb];
      gs = split_of<true>(gbase);
      ghi = __double2hiint(gbase) & 0x7FFFFFFF;
#pragma unroll 4
      for (int c = warp - guard; c < wk.len + guard; c += warps) {
        const int En = wk.bb + c * (1 << lg);
        const bool bad = is_bad(En), in = En >= wk.lo && En <= wk.hi;
        const double g = in ? G[c * (1 << lg)] : 0.0;
        const int g_hi = __double2hiint(g) & 0x7FFFFFFF;
        own = own && g_hi < 0x46300000;  // |g| < 2^100
        const float shadow = shadow_of<true>(g, gs);
        if (in && !bad) {
          amax = fmaxf(amax, fabsf(shadow));
          ghi = max(ghi, g_hi);
        }
        pair[c * 32] = make_float2(bad ? __int_as_float(0x7FC00000) : (in ? shadow : __int_as_float(0x7F800000)), 0.0f);
      }
    }
    ok = ok && own;
  }
  top[warp * 32 + lane] = make_float2(amax, __int_as_float(ghi));
  if (__syncthreads_or(!ok)) {
    if (live && warp == 0)
      sweep_global(t, a.lat, a.J, a.H, a.logG, a.factor, a.E, a.newE, a.off_iter, a.found, a.start, a.end, a.off_hist,
                   a.off_lat, a.cond, a.spectrum, a.off_spec, a.cond_inter, X, Y, a.n_iter, a.num_lattices, a.n_int, a.wpi,
                   a.seed, a.boundary);
    return;
  }
  if (warp == 0) {
    if (live) {
      // words of 32 sites to rows, from the last: row i lies in words up to i
      uint32_t* mine = words + lane;
      auto row_at = [&](int i) {
        const int bit = i * Y, f = bit >> 5, e = (bit + Y - 1) >> 5;
        return __funnelshift_r(mine[f * 32], mine[e * 32], bit & 31) & row_mask;
      };
      const uint32_t first = mine[0] & row_mask;
      for (uint32_t i = X, below = first; i-- > 0;) {
        const uint32_t r = row_at(i);
        mine[i * 32] = kBonds ? bond_word(r, below, Jr[i], Jr[X + i], Y, open, i + 1 == X) : r;
        below = r;
      }
      wk.s0 = first & 1u;
      wk.lt.r = 0;
      wk.lt.a = shared_addr(words + lane);
      wk.lt.stride = 128u;
      wk.pair = pair;
      wk.ring_a = shared_addr(smem + l.off_ring) + 4 * lane;
      wk.rng.init(key_u32(a.seed, static_cast<uint64_t>(k)), static_cast<uint64_t>(w), a.off_iter[t]);
      wk.start();
      for (int v = 0; v < warps; ++v) {
        amax = fmaxf(amax, top[v * 32 + lane].x);
        ghi = max(ghi, __float_as_int(top[v * 32 + lane].y));
      }
      __syncwarp(wmask);
      wk.gs = gs;
      wk.amax = amax;
      wk.ghi = ghi;
      wk.fresh = true;
      const uint32_t tab_a = shared_addr(col);
      const SweepTeam team{d, 32, tab_a, tab_a + align16(8 * Y), Jr, Jr + X, 0, 0};
      int flag = 0;
      auto log_g = [&](int c) { return G[c << lg]; };
      auto new_energy = [&](int En, int) {
        flag = t + 1;
        a.newE[t] = En;
      };
      auto fold = [&](float, int, bool last) {
        if (last) return;  // by all warps, below
        wk.fresh = false;
        if (frozen) return;
        for (int c = 0; c < wk.len; ++c) {
          const uint32_t n = static_cast<uint32_t>(pair[c * 32].y);
          if (n == 0) continue;
          pair[c * 32].y = 0.0f;
          H[c << lg] += n;
          G[c << lg] = add_times<true>(G[c << lg], lnf, n);
        }
      };
      wl_sweep<kStore, false, true>(team, wk, wmask, a.n_iter, frozen, lnf, 0, log_g, is_bad, new_energy, fold);
      if constexpr (kBonds) {  // to rows: down column 0, then along each row
        uint32_t edge = wk.s0;
        for (int i = 0; i < X; ++i) {
          const uint32_t word = mine[i * 32];
          uint32_t r = (word ^ Jr[i]) << 1;
          r ^= r << 1;
          r ^= r << 2;
          r ^= r << 4;
          r ^= r << 8;
          mine[i * 32] = r ^ (0u - edge);
          edge ^= ((word >> 16) ^ Jr[X + i]) & 1u;
        }
      }
      a.found[t] = flag;
      a.E[t] = wk.E;
      a.off_iter[t] = wk.rng.pos;
    }
    __syncwarp();
  }
  __syncthreads();
  if (!frozen)
    for (int c = warp; c < wk.len; c += warps) {
      const uint32_t n = static_cast<uint32_t>(pair[c * 32].y);
      if (n == 0) continue;
      H[c << lg] += n;
      G[c << lg] = add_times<true>(G[c << lg], lnf, n);
    }
  if (warps == 1) {
    for (int i = 0; i < X && live; ++i) {
      const uint32_t r = words[i * 32 + lane];
      int8_t* s = a.lat + at + i * Y;
#pragma unroll 4
      for (int j = 0; j < Y; ++j) s[j] = (r >> j) & 1u ? -1 : 1;
    }
    return;
  }
#pragma unroll 4
  for (int x = warp; x < 32 * nw; x += warps) {
    const int q = x & 31, site = (x >> 5) * 32 + lane;
    int8_t* s = a.lat + __shfl_sync(kAll, at, q);
    if (((wmask >> q) & 1u) == 0 || site >= N) continue;
    const int i = static_cast<int>((static_cast<uint32_t>(site) * a.magic) >> 20);
    s[site] = (words[i * 32 + q] >> (site - i * Y)) & 1u ? -1 : 1;
  }
}

// -------------------------------------------------------------- flatness ----
// wl.cu:892-967, one block per window, 1 to 32 lanes per walker: the loads of a
// histogram do not wait for each other.
constexpr int kFlatThreads = 512;  // of a block, at most
// Lanes a walker: as many as a block has threads for, while all windows' threads
// are few (a warp's fill whatever they are): beyond, short histograms leave most
// lanes of a walker idle and the blocks queue.  us for 1 / 32 lanes, 8 bins: 640
// windows of 16 walkers 5.5 / 13.5, 2560 of 8 8.1 / 21, one of 1024, flat 22 / 144;
// 120 bins: 16 windows of 8 walkers 24.9 / 5.2.
inline int flat_lanes(long long windows, int W)
{
  int lanes = 32;
  while (lanes > 1 && (W * lanes > kFlatThreads || (W * lanes > 32 && windows * W * lanes > 65536))) lanes /= 2;
  return lanes;
}
__global__ void k_check_histogram(unsigned long long* __restrict__ H, double* __restrict__ factor,
                                  int8_t* __restrict__ cond, const int* __restrict__ off_hist,
                                  const int* __restrict__ end, const int* __restrict__ start,
                                  const int8_t* __restrict__ spectrum, const int* __restrict__ off_spec,
                                  const int* __restrict__ cond_inter, double alpha, int W, int wpi, int n_int, int lanes)
{
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const int b = blockIdx.x;
  const int first = threadIdx.x / lanes, lane = threadIdx.x & (lanes - 1), side = blockDim.x / lanes;
  const int k = (b * W) / wpi;
  if (cond[b] == 1 || cond_inter[k] == -1) return;
  const int len = end[b] - start[b] + 1;
  const int8_t* mask = spectrum + off_spec[k] + start[b] - start[k * n_int];
  bool flat = true;
  for (int w = first; w - first < W && __all_sync(kAll, flat); w += side) {
    unsigned long long mn = 2147483647ull;
    unsigned long long sum = 0;  // exact: the reference's double sum of integers is exact below 2^53
    int cnt = 0;
    if (w < W) {
      const unsigned long long* h = H + off_hist[b * W + w];
#pragma unroll 4
      for (int i = lane; i < len; i += lanes) {
        const unsigned long long v = h[i];
        const bool on = mask[i] == 1;
        mn = on && v < mn ? v : mn;
        sum += on ? v : 0ull;
        cnt += on ? 1 : 0;
      }
    }
    for (int d = lanes / 2; d > 0; d >>= 1) {
      const unsigned long long o = __shfl_xor_sync(kAll, mn, d);
      mn = o < mn ? o : mn;
      sum += __shfl_xor_sync(kAll, sum, d);
      cnt += __shfl_xor_sync(kAll, cnt, d);
    }
    const double avg = static_cast<double>(sum) / max(cnt, 1);
    flat = w >= W || (cnt > 0 && static_cast<double>(mn) >= alpha * avg);
  }
  if (!__syncthreads_and(flat)) return;
  for (int w = first; w < W; w += side) {
    unsigned long long* h = H + off_hist[b * W + w];
    for (int i = lane; i < len; i += lanes) h[i] = 0;
    if (lane == 0) factor[b * W + w] = sqrt(factor[b * W + w]);
  }
  if (threadIdx.x == 0) cond[b] = 1;
}

// ------------------------------------------------------- log g averaging ----
// wl.cu:710-783 + :969-1031 fused; one block per window, threads over bins.
__global__ void k_average_log_g(double* __restrict__ logG, const int* __restrict__ start,
                                const int* __restrict__ end, const int8_t* __restrict__ spectrum,
                                const int* __restrict__ off_spec, const int8_t* __restrict__ cond,
                                const int* __restrict__ off_hist, const int* __restrict__ cond_inter, int R, int W,
                                int n_int)
{
  const int total = R * n_int;
  for (int b = blockIdx.x; b < total; b += gridDim.x) {
    const int k = b / n_int;
    if (cond[b] != 1 || cond_inter[k] == -1) continue;
    const int len = end[b] - start[b] + 1;
    const int8_t* mask = spectrum + off_spec[k] + start[b] - start[k * n_int];
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
      double avg = 0.0;
      if (mask[i] == 1) {
        for (int w = 0; w < W; ++w) avg += logG[off_hist[b * W + w] + i] / W;
      }
      for (int w = 0; w < W; ++w) logG[off_hist[b * W + w] + i] = avg;
    }
  }
}

__global__ void k_reset_cond(int8_t* __restrict__ cond, const double* __restrict__ factor, int total, double beta,
                             int W)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  if (cond[t] == 1 && factor[static_cast<size_t>(t) * W] > exp(beta)) cond[t] = 0;
}

__global__ void k_check_finished(int* __restrict__ cond_inter, const int8_t* __restrict__ cond, int n_int, int R)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= R) return;
  int s = 0;
  for (int b = 0; b < n_int; ++b) s += cond[k * n_int + b];
  cond_inter[k] = (s == n_int) ? -1 : s;
}

// ------------------------------------------------------ replica exchange ----
// wl.cu:785-890, one block per window, one thread per walker.
__global__ void k_replica_exchange(int* __restrict__ off_lat, int* __restrict__ E, int* __restrict__ perm,
                                   uint64_t* __restrict__ off_iter, const int* __restrict__ start,
                                   const int* __restrict__ end, const int* __restrict__ off_hist,
                                   const int* __restrict__ cond_inter, const double* __restrict__ logG, int even,
                                   int seed, int n_int, int W, int wpi, int global_parity)
{
  const int b = blockIdx.x;
  if (b % n_int == n_int - 1) return;
  const int par = global_parity ? b : (b % n_int);
  if ((even && par % 2 != 0) || (!even && par % 2 == 0)) return;
  const int k = (b * W) / wpi;
  if (cond_inter[k] == -1) return;
  const int w = threadIdx.x;
  const int t0 = b * W;
  const int t = t0 + w;
  // the permutation's draws by a thread each, its swaps by one in shared memory
  __shared__ int swap[1024], order[1024];
  Stream st;
  uint64_t pos = 0;
  int et = 0;
  if (w < W) {
    const uint64_t first = off_iter[t0];
    if (w > 0) {
      st.init(key_i32(seed, static_cast<uint64_t>(k)), static_cast<uint64_t>(t0 % wpi), first + (W - 1 - w));
      double u = st.uniform();
      u *= (w + 0.999999);
      swap[w] = static_cast<int>(trunc(u));
    }
    order[w] = perm[t];
    pos = w == 0 ? first + (W - 1) : off_iter[t];
    et = E[t];
  }
  __syncthreads();
  if (w == 0) {
    for (int i = W - 1; i > 0; --i) {
      const int r = swap[i], tmp = order[i];
      order[i] = order[r];
      order[r] = tmp;
    }
  }
  __syncthreads();
  if (w >= W) return;
  perm[t] = order[w];
  if (w == 0) off_iter[t] = pos;
  const int o = W * (b + 1) + order[w];
  const int eo = E[o];
  if (et > end[b + 1] || et < start[b + 1]) return;
  if (eo > end[b] || eo < start[b]) return;
  const double gi_x = logG[off_hist[t] + et - start[b]];
  const double gi_y = logG[off_hist[t] + eo - start[b]];
  const double gj_y = logG[off_hist[o] + eo - start[b + 1]];
  const double gj_x = logG[off_hist[o] + et - start[b + 1]];
  const double prob = fmin(1.0, exp(gi_x - gi_y) * exp(gj_y - gj_x));
  st.init(key_i32(seed, static_cast<uint64_t>(k)), static_cast<uint64_t>(t % wpi), pos);
  if (st.uniform() < prob) {
    const int tmp = off_lat[t];
    off_lat[t] = off_lat[o];
    off_lat[o] = tmp;
    E[t] = eo;
    E[o] = et;
  }
  off_iter[t] = st.pos;
}

// ------------------------------------------------------------ reductions ----

__global__ void k_max_int(const int* __restrict__ in, size_t n, int* __restrict__ out)
{
  int m = INT_MIN;
  for (size_t q = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < n;
       q += static_cast<size_t>(gridDim.x) * blockDim.x)
    m = max(m, in[q]);
  for (int d = 16; d > 0; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Maximum of non-negative doubles through their bit patterns, which order
// like the values.
__global__ void k_max_f64_nonneg(const double* __restrict__ in, size_t n, unsigned long long* __restrict__ out)
{
  unsigned long long m = 0;
  for (size_t q = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < n;
       q += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const unsigned long long v = static_cast<unsigned long long>(__double_as_longlong(in[q]));
    m = v > m ? v : m;
  }
  for (int d = 16; d > 0; d >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, m, d);
    m = o > m ? o : m;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void k_fill_int(int* out, int v) { *out = v; }

inline int blocks_for(size_t n) { return static_cast<int>((n + kThreads - 1) / kThreads); }

}  // namespace
}  // namespace wlg

using namespace wlg;

// ------------------------------------------------------------ C ABI -------

extern "C" {

wlg_status wlg_init_interactions(int8_t* d_J, size_t lattice_size, int num_samples, int seed, float prob,
                                 wlg_stream stream)
{
  if (d_J == nullptr || lattice_size == 0 || num_samples <= 0) return WLG_ERR_INVALID;
  const size_t n = (2 * lattice_size + 3) / 4 * static_cast<size_t>(num_samples);
  k_init_interactions<<<blocks_for(n), kThreads, 0, as_stream(stream)>>>(d_J, lattice_size, num_samples, seed, prob);
  return launch_status();
}

wlg_status wlg_apply_error_class(int8_t* d_J, int X, int Y, int num_samples, char error_class, wlg_stream stream)
{
  if (d_J == nullptr || X <= 0 || Y <= 0 || num_samples <= 0) return WLG_ERR_INVALID;
  cudaStream_t s = as_stream(stream);
  if (error_class == 'h' || error_class == 'c')
    k_apply_chain<<<blocks_for(static_cast<size_t>(Y) * num_samples), kThreads, 0, s>>>(d_J, X, Y, num_samples, 0);
  if (error_class == 'v' || error_class == 'c')
    k_apply_chain<<<blocks_for(static_cast<size_t>(X) * num_samples), kThreads, 0, s>>>(d_J, X, Y, num_samples, 1);
  return launch_status();
}

wlg_status wlg_init_lattice(int8_t* d_lattice, int X, int Y, size_t num_lattices, int seed, int walker_per_sample,
                            wlg_stream stream)
{
  if (d_lattice == nullptr || X <= 0 || Y <= 0 || walker_per_sample <= 0) return WLG_ERR_INVALID;
  if (num_lattices == 0) return WLG_OK;
  const size_t n = (static_cast<size_t>(X) * Y / 4 + 1) * num_lattices;
  k_init_lattice<<<blocks_for(n), kThreads, 0, as_stream(stream)>>>(d_lattice, X, Y, num_lattices, seed,
                                                                     walker_per_sample);
  return launch_status();
}

wlg_status wlg_calc_energy(int boundary, int* d_energy, const int8_t* d_lattice, const int8_t* d_J,
                           const int* d_offset_lattice, int X, int Y, size_t num_lattices, int walker_per_sample,
                           wlg_stream stream)
{
  if ((boundary != 0 && boundary != 1) || X <= 0 || Y <= 0 || walker_per_sample <= 0) return WLG_ERR_INVALID;
  if (num_lattices == 0) return WLG_OK;
  const long long N = static_cast<long long>(X) * Y;
  const int lanes = energy_lanes(N, num_lattices);
  k_calc_energy<<<blocks_for(num_lattices * lanes), kThreads, 0, as_stream(stream)>>>(
    boundary, d_energy, d_lattice, d_J, d_offset_lattice, X, Y, num_lattices, walker_per_sample, lanes);
  return launch_status();
}

wlg_status wlg_wang_landau_pre_run(int* d_energy, int* d_flag_found_interval, int8_t* d_lattice,
                                   int8_t* d_found_interval_lattice, unsigned long long* d_histogram,
                                   uint64_t* d_seed_offset, const int8_t* d_J, const int* d_offset_lattice, int E_min,
                                   int E_max, int num_iterations, int X, int Y, int seed, unsigned num_intervals,
                                   int len_interval, size_t num_total_walker, int walker_per_sample, int boundary,
                                   wlg_stream stream)
{
  if ((boundary != 0 && boundary != 1) || X <= 0 || Y <= 0 || walker_per_sample <= 0 || walker_per_sample > 1024 ||
      num_intervals == 0 || len_interval <= 0 || E_max < E_min || num_total_walker % walker_per_sample != 0)
    return WLG_ERR_INVALID;
  const int R = static_cast<int>(num_total_walker / walker_per_sample);
  if (R == 0 || num_iterations <= 0) return WLG_OK;
  const int len_hist = E_max - E_min + 1;
  size_t smem = static_cast<size_t>(len_hist) * sizeof(unsigned long long) + 2 * sizeof(int) * num_intervals;
  if (smem > 200 * 1024) return WLG_ERR_INVALID;
  const int threads = (walker_per_sample + 31) / 32 * 32;
  PrerunArgs a{d_energy, d_flag_found_interval, d_lattice, d_found_interval_lattice, d_histogram, d_seed_offset, d_J,
               d_offset_lattice, E_min, E_max, num_iterations, X, Y, seed, static_cast<int>(num_intervals), len_interval,
               walker_per_sample, boundary, 0};
  if (static_cast<long long>(X) * Y <= 4096 && pre_walk_fits(X, Y, walker_per_sample, num_iterations) &&
      bonds_pay(static_cast<long long>(X) * Y, walker_per_sample, num_iterations, R)) {
    const size_t bytes = static_cast<size_t>(
      pre_layout(X, Y, ((len_hist - 1) >> energy_step_log2(boundary)) + 1, a.n_int, threads).bytes);
    if (bytes <= 227 * 1024) {
      a.bonds = 1;
      smem = std::max(smem, bytes);
    }
  }
  cudaStream_t s = as_stream(stream);
  const auto kernel = threads <= 256 ? &k_prerun<256> : &k_prerun<1024>;
  if (smem > 48 * 1024 && !allow_shared(kernel)) return WLG_ERR_CUDA;
  kernel<<<R, threads, smem, s>>>(a);
  return launch_status();
}

wlg_status wlg_wang_landau(int8_t* d_lattice, const int8_t* d_J, unsigned long long* d_H, double* d_logG,
                           const double* d_factor, int* d_energy, int* d_new_energy, uint64_t* d_offset_iter,
                           int* d_found, const int* d_start, const int* d_end, const int* d_offset_histogram,
                           const int* d_offset_lattice, const int8_t* d_cond, const int8_t* d_spectrum,
                           const int* d_offset_spectrum, const int* d_cond_sample, int X, int Y, int num_iterations,
                           int num_lattices, int num_intervals, int walker_per_sample, int seed, int boundary,
                           wlg_stream stream)
{
  if ((boundary != 0 && boundary != 1) || X <= 0 || Y <= 0 || num_intervals <= 0 || walker_per_sample <= 0 ||
      walker_per_sample % num_intervals != 0 || num_lattices < 0)
    return WLG_ERR_INVALID;
  if (num_lattices == 0) return WLG_OK;
  SweepArgs a{d_lattice, d_J, d_H, d_logG, d_factor, d_energy, d_new_energy, d_offset_iter, d_found, d_start, d_end,
              d_offset_histogram, d_offset_lattice, d_cond, d_spectrum, d_offset_spectrum, d_cond_sample, X, Y,
              num_iterations, num_lattices, num_intervals, walker_per_sample, seed, boundary, 0, 0};
  cudaStream_t s = as_stream(stream);
  const int N = X * Y, lg = boundary == 0 ? 2 : 1;
  bool packed = X >= 2 && Y >= 2 && Y <= 32 && static_cast<long long>(X) * Y <= 4096 && num_iterations > 0;
  if (packed) {
    // Columns for windows of up to 8 / num_intervals of the energy range: the
    // last window is up to twice as long as the others, which take
    // 1 / (1 + overlap (num_intervals - 1)) of it.
    const int full = (4 * N >> lg) + 1;
    a.L = std::min(full, 8 * full / num_intervals + 8);
    // 2^20 / Y rounded up: e < 32 too large, so that site * e < 4096 * 32 < 2^20
    // never carries site * magic >> 20 past site / Y
    a.magic = static_cast<uint32_t>(((1u << 20) + Y - 1) / Y);
    packed = sweep_layout(X, Y, a.L, lg).bytes <= kSharedBytes;
  }
  const int samples = (num_lattices + walker_per_sample - 1) / walker_per_sample;
  const int blocks = samples * ((walker_per_sample + 31) / 32);
  const int smem = packed ? sweep_layout(X, Y, a.L, lg).bytes : 0;
  const SweepPlan plan = packed ? sweep_plan(a, blocks, smem) : SweepPlan{1, false};
  if (!plan.pays) {
    k_wang_landau<<<blocks_for(static_cast<size_t>(num_lattices)), kThreads, 0, s>>>(
      d_lattice, d_J, d_H, d_logG, d_factor, d_energy, d_new_energy, d_offset_iter, d_found, d_start, d_end,
      d_offset_histogram, d_offset_lattice, d_cond, d_spectrum, d_offset_spectrum, d_cond_sample, X, Y, num_iterations,
      num_lattices, num_intervals, walker_per_sample, seed, boundary);
    return launch_status();
  }
  const auto kernel =
    Y > 16 ? &k_wl_sweep<kStoreRows> : (boundary == 0 ? &k_wl_sweep<kStoreBonds> : &k_wl_sweep<kStoreBondsOpen>);
  if (smem > 48 * 1024 && !allow_shared(kernel)) return WLG_ERR_CUDA;
  kernel<<<blocks, 32 * plan.warps, smem, s>>>(a);
  return launch_status();
}

wlg_status wlg_check_histogram(unsigned long long* d_H, double* d_factor, int8_t* d_cond,
                               const int* d_offset_histogram, const int* d_end, const int* d_start,
                               const int8_t* d_spectrum, const int* d_offset_spectrum, const int* d_cond_sample,
                               double alpha, int num_walker_total, int walker_per_sample, int num_intervals,
                               wlg_stream stream)
{
  if (num_intervals <= 0 || walker_per_sample <= 0 || walker_per_sample % num_intervals != 0) return WLG_ERR_INVALID;
  const int W = walker_per_sample / num_intervals;
  if (W > 1024 || num_walker_total % W != 0) return WLG_ERR_INVALID;
  const int windows = num_walker_total / W;
  if (windows == 0) return WLG_OK;
  const int lanes = flat_lanes(windows, W);
  const int threads = std::min((W * lanes + 31) / 32 * 32, kFlatThreads);
  k_check_histogram<<<windows, threads, 0, as_stream(stream)>>>(
    d_H, d_factor, d_cond, d_offset_histogram, d_end, d_start, d_spectrum, d_offset_spectrum, d_cond_sample, alpha, W,
    walker_per_sample, num_intervals, lanes);
  return launch_status();
}

wlg_status wlg_average_log_g(double* d_logG, const int* d_start, const int* d_end, const int8_t* d_spectrum,
                             const int* d_offset_spectrum, const int8_t* d_cond, const int* d_offset_histogram,
                             const int* d_cond_sample, int num_samples, int walker_per_interval, int num_intervals,
                             wlg_stream stream)
{
  if (num_samples < 0 || walker_per_interval <= 0 || num_intervals <= 0) return WLG_ERR_INVALID;
  const int total = num_samples * num_intervals;
  if (total == 0) return WLG_OK;
  const int grid = total < 65535 ? total : 65535;
  k_average_log_g<<<grid, kThreads, 0, as_stream(stream)>>>(d_logG, d_start, d_end, d_spectrum, d_offset_spectrum,
                                                             d_cond, d_offset_histogram, d_cond_sample, num_samples,
                                                             walker_per_interval, num_intervals);
  return launch_status();
}

wlg_status wlg_reset_cond(int8_t* d_cond, const double* d_factor, int total_intervals, double beta,
                          int walker_per_interval, wlg_stream stream)
{
  if (total_intervals < 0 || walker_per_interval <= 0) return WLG_ERR_INVALID;
  if (total_intervals == 0) return WLG_OK;
  k_reset_cond<<<blocks_for(static_cast<size_t>(total_intervals)), kThreads, 0, as_stream(stream)>>>(
    d_cond, d_factor, total_intervals, beta, walker_per_interval);
  return launch_status();
}

wlg_status wlg_check_finished(int* d_cond_sample, const int8_t* d_cond, int num_intervals, int num_samples,
                              wlg_stream stream)
{
  if (num_intervals <= 0 || num_samples < 0) return WLG_ERR_INVALID;
  if (num_samples == 0) return WLG_OK;
  k_check_finished<<<blocks_for(static_cast<size_t>(num_samples)), kThreads, 0, as_stream(stream)>>>(
    d_cond_sample, d_cond, num_intervals, num_samples);
  return launch_status();
}

wlg_status wlg_replica_exchange(int* d_offset_lattice, int* d_energy, int* d_replica_indices,
                                uint64_t* d_offset_iter, const int* d_start, const int* d_end,
                                const int* d_offset_histogram, const int* d_cond_sample, const double* d_logG,
                                int even, int seed, int num_intervals, int walker_per_sample, int total_intervals,
                                int global_parity, wlg_stream stream)
{
  if (num_intervals <= 0 || walker_per_sample <= 0 || walker_per_sample % num_intervals != 0 || total_intervals < 0)
    return WLG_ERR_INVALID;
  const int W = walker_per_sample / num_intervals;
  if (W > 1024) return WLG_ERR_INVALID;
  if (total_intervals == 0) return WLG_OK;
  k_replica_exchange<<<total_intervals, (W + 31) / 32 * 32, 0, as_stream(stream)>>>(
    d_offset_lattice, d_energy, d_replica_indices, d_offset_iter, d_start, d_end, d_offset_histogram, d_cond_sample,
    d_logG, even, seed, num_intervals, W, walker_per_sample, global_parity);
  return launch_status();
}

wlg_status wlg_max_int(const int* d_in, size_t n, int* d_out, wlg_stream stream)
{
  if (d_in == nullptr || d_out == nullptr) return WLG_ERR_INVALID;
  cudaStream_t s = as_stream(stream);
  k_fill_int<<<1, 1, 0, s>>>(d_out, INT_MIN);
  if (n > 0) {
    const int blocks = static_cast<int>(std::min<size_t>((n + kThreads - 1) / kThreads, 1024));
    k_max_int<<<blocks, kThreads, 0, s>>>(d_in, n, d_out);
  }
  return launch_status();
}

wlg_status wlg_max_f64_nonneg(const double* d_in, size_t n, double* d_out, wlg_stream stream)
{
  if (d_in == nullptr || d_out == nullptr) return WLG_ERR_INVALID;
  cudaStream_t s = as_stream(stream);
  if (cudaMemsetAsync(d_out, 0, sizeof(double), s) != cudaSuccess) return WLG_ERR_CUDA;
  if (n > 0) {
    const int blocks = static_cast<int>(std::min<size_t>((n + kThreads - 1) / kThreads, 1024));
    k_max_f64_nonneg<<<blocks, kThreads, 0, s>>>(d_in, n, reinterpret_cast<unsigned long long*>(d_out));
  }
  return launch_status();
}

}  // extern "C"

// ------------------------------------------------------------ diagnostics ---

namespace wlg {
namespace {
__global__ void k_uniforms(uint64_t key, uint64_t subseq, uint64_t offset, int n, float* out)
{
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  Stream st;
  st.init(key, subseq, offset);
  for (int q = 0; q < n; ++q) out[q] = st.uniform();
}
}  // namespace
}  // namespace wlg

extern "C" wlg_status wlg_uniforms(uint64_t key, uint64_t subseq, uint64_t offset, int n, float* d_out,
                                   wlg_stream stream)
{
  if (n < 0 || (n > 0 && d_out == nullptr)) return WLG_ERR_INVALID;
  if (n == 0) return WLG_OK;
  wlg::k_uniforms<<<1, 32, 0, wlg::as_stream(stream)>>>(key, subseq, offset, n, d_out);
  return wlg::launch_status();
}
