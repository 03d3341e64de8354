// Batched Wang-Landau engine for sm_103a: the pre-run kernel and the launchers.
//
// k_pre_batch:  one CTA per problem runs the whole pre-run of the reference
//               (prerun.cu:52-133) — disorder, error chain, lattice init,
//               energy, histogram-biased walk, stored lattices — with the
//               sample's histogram in shared memory.
// k_main_batch: the persistent main run (wlg_main.cuh), compiled per CTA size
//               in wlg_main_*.cu.

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "../../include/wlg.h"
#include "wlg_batch.h"
#include "wlg_engine.h"
#include "wlg_internal.h"
#include "wlg_lattice.cuh"
#include "wlg_main_fn.h"
#include "wlg_rng.cuh"

namespace wlg {
namespace {

// ------------------------------------------------------------ pre-run -----

// Site of a draw: trunc(double(u) * ((N-1) + 0.999999)) (wl.cu:63-65).  With
// f = x / 2^32 the reference's product lies within N*2^-23 + 1e-6 of f*N, so
// floor(f*N) = umulhi(x, N) is exact unless the fraction x*N mod 2^32 lies
// within site_thr (= 2^32 (N 2^-21 + 2^-18), >= 4x that bound) of an
// integer; there the reference's own float/double expression below decides.
// No int<->float conversion on the common path (they share GB300's slow
// FP64 pipe).  Out of line: inlined, its FP64 multiply and conversions would
// be scheduled into every step.
__device__ __noinline__ int site_exact(uint32_t x, double scale)
{
  return static_cast<int>(trunc(static_cast<double>(unit_float(x)) * scale));
}

__global__ void __launch_bounds__(1024) k_pre_batch(const PreDesc* __restrict__ descs, int n,
                                                    int8_t* __restrict__ Jpool, uint8_t* __restrict__ seen_pool,
                                                    int8_t* __restrict__ found_pool, int* __restrict__ fflag_pool)
{
  const int p = blockIdx.x;
  if (p >= n) return;
  const PreDesc d = descs[p];
  const int N = d.N, X = d.X, Y = d.Y;
  const int L = 4 * N + 1;
  const int e_min = -2 * N;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long* hist = reinterpret_cast<unsigned long long*>(smem);
  int* claim = reinterpret_cast<int*>(hist + L);
  int* found = claim + d.n_int;
  int* misc = found + d.n_int;  // [0] start energy
  int8_t* J = reinterpret_cast<int8_t*>(misc + 4);
  int8_t* lat = J + 2 * N;  // [walkers][N]

  const int tid = threadIdx.x;
  // disorder (wl.cu:364-386), or the caller's pattern, and the error chain
  // (wl.cu:388-428, prerun.cu:56-75)
  for (int q = tid; q < 2 * N; q += blockDim.x) {
    if (d.given_J) {
      J[q] = Jpool[d.off_J + q];
      continue;
    }
    Stream st;
    st.init(key_size(d.seed, static_cast<uint64_t>(d.sample)), 0, static_cast<uint64_t>(q));
    const double u = st.uniform();
    J[q] = (u < d.prob) ? -1 : 1;
  }
  for (int q = tid; q < L; q += blockDim.x) hist[q] = 0;
  for (int q = tid; q < d.n_int; q += blockDim.x) {
    claim[q] = INT_MAX;
    found[q] = 0;
  }
  __syncthreads();
  if (d.error_class == 'h' || d.error_class == 'c')
    for (int q = tid; q < Y; q += blockDim.x) J[N + q] = static_cast<int8_t>(-J[N + q]);
  if (d.error_class == 'v' || d.error_class == 'c')
    for (int q = tid; q < X; q += blockDim.x) J[q * Y] = static_cast<int8_t>(-J[q * Y]);
  // lattice (wl.cu:430-457, CAS winner fixed to site 0)
  const uint64_t key_l = key_u32(d.seed, static_cast<uint64_t>(d.sample));
  for (int q = tid; q < N; q += blockDim.x) {
    Stream st;
    st.init(key_l, 1, 0);
    const float p0 = st.uniform();
    st.init(key_l, 1, static_cast<uint64_t>(q) + 1);
    const double u = st.uniform();
    lat[q] = (u < p0) ? -1 : 1;
  }
  __syncthreads();
  for (int q = tid; q < 2 * N; q += blockDim.x) Jpool[d.off_J + q] = J[q];
  const int w = tid;
  const bool live = w < d.walkers;
  int8_t* s = lat + static_cast<size_t>(w) * N;
  if (live && w > 0)
    for (int q = 0; q < N; ++q) s[q] = lat[q];
  if (tid == 0) misc[0] = energy_i8(lat, J, X, Y, d.boundary);
  __syncthreads();

  // histogram-biased walk (wl.cu:473-560), round-synchronous
  Stream rng;
  int energy = misc[0];
  if (live) rng.init(key_u32(d.seed, static_cast<uint64_t>(d.sample)), 2 + static_cast<uint64_t>(w), 0);
  const double site_scale = (N - 1 + 0.999999);
  const uint32_t site_thr = static_cast<uint32_t>(N) * 2048u + 16384u;  // as MainDesc::site_thr
  // u < exp(H[old] - H[new]) (wl.cu:536-537) for an integer count difference
  // dd: always for dd >= 1 (exp(dd) > 1 >= u); never for dd <= -25
  // (exp(dd) < 2^-33 <= u); else x < acc_thr[-dd], the least draw whose
  // uniform reaches the device's exp(dd) (uniforms are monotone in the draw)
  __shared__ uint32_t acc_thr[25];
  if (tid < 25) {
    const double e = exp(static_cast<double>(-tid));
    unsigned long long lo = 0, hi = 1ull << 32;
    while (lo < hi) {
      const unsigned long long mid = (lo + hi) >> 1;
      if (static_cast<double>(unit_float(static_cast<uint32_t>(mid))) >= e) hi = mid;
      else lo = mid + 1;
    }
    acc_thr[tid] = static_cast<uint32_t>(lo);  // <= 2^32 - 128: u reaches 1 there
  }
  __syncthreads();
  bool ok = live;
  for (int it = 0; it < d.n_iter; ++it) {
    int hit = -1;
    bool acc = false;
    if (ok) {
      // site trunc(u (N - 1 + 0.999999)) (wl.cu:60-66): floor(x N / 2^32)
      // unless x N lies next to a multiple of 2^32 (see the main run)
      const uint32_t xs = rng.raw();
      const uint32_t lo_s = xs * static_cast<uint32_t>(N);
      int site = static_cast<int>(__umulhi(xs, static_cast<uint32_t>(N)));
      if (lo_s < site_thr || lo_s > ~site_thr) site = site_exact(xs, site_scale);  // out of line: FP64
      const Move m = move_i8(s, J, energy, X, Y, site, d.boundary, d.site_magic);
      const int io = energy - e_min;
      const int in = m.new_energy - e_min;
      const long long dd = static_cast<long long>(hist[io]) - static_cast<long long>(hist[in]);
      const uint32_t xa = rng.raw();
      const int ti = static_cast<int>(min(max(-dd, 0ll), 24ll));
      acc = dd >= 1 || (dd >= -24 && xa < acc_thr[ti]);
      if (acc) s[m.site] = static_cast<int8_t>(-s[m.site]);
      energy = acc ? m.new_energy : energy;
      hit = acc ? in : io;
    }
    __syncthreads();
    int bin = -1;
    {
      // warp-aggregated histogram update: walkers sit on few energies (all
      // start on one), so lanes with the same bin add their count once
      const unsigned on = __ballot_sync(0xFFFFFFFFu, hit >= 0);
      if (hit >= 0) {
        const unsigned same = __match_any_sync(on, hit);
        if (static_cast<int>(threadIdx.x & 31u) == __ffs(same) - 1)
          atomicAdd(&hist[hit], static_cast<unsigned long long>(__popc(same)));
      }
    }
    if (acc) {
      const int q = (energy - e_min) / d.len_int;
      bin = (q < d.n_int) ? q : d.n_int - 1;
      if (found[bin] == 0) atomicMin(&claim[bin], w);
      else bin = -1;
    }
    __syncthreads();
    if (bin >= 0 && claim[bin] == w && found[bin] == 0) {
      found[bin] = 1;
      int8_t* dst = found_pool + d.off_found + static_cast<long long>(bin) * N;
      for (int q = 0; q < N; ++q) dst[q] = s[q];
    }
  }
  __syncthreads();
  for (int q = tid; q < L; q += blockDim.x) seen_pool[d.off_seen + q] = hist[q] != 0 ? 1 : 0;
  // energies of the stored lattices (prerun.cu:123-133)
  for (int q = tid; q < d.n_int; q += blockDim.x) {
    fflag_pool[d.off_fflag + q] = found[q];
    int e = 0;
    if (found[q]) e = energy_i8(found_pool + d.off_found + static_cast<long long>(q) * N, J, X, Y, d.boundary);
    fflag_pool[d.off_fflag + d.n_int + q] = e;
  }
}

}  // namespace

// ------------------------------------------------------------ launchers ----

wlg_status launch_pre_batch(const PreDesc* d_descs, int n, int threads, int smem, int8_t* Jpool, uint8_t* seen_pool,
                            int8_t* found_pool, int* fflag_pool, cudaStream_t s)
{
  if (n == 0) return WLG_OK;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_pre_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return WLG_ERR_CUDA;
  }
  k_pre_batch<<<n, threads, smem, s>>>(d_descs, n, Jpool, seen_pool, found_pool, fflag_pool);
  return launch_status();
}

MainFn main_fn(int variant, int cta_threads)
{
  const bool tight = (variant & kVariantTight) != 0;
  if (cta_threads <= 256) return main_fn_256(variant_store(variant), tight);
  if (cta_threads <= 512) return main_fn_512(variant_store(variant), tight);
  return main_fn_1024(variant_store(variant), tight);
}

// Returns the number of resident CTAs the launch may use (0 if the
// configuration does not fit).
int main_batch_capacity(int variant, int cta_threads, int smem)
{
  MainFn fn = main_fn(variant, cta_threads);
  int per_sm = 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, cta_threads, smem) != cudaSuccess) return 0;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return per_sm * sms;
}

wlg_status launch_main_batch(int variant, const MainDesc* d_descs, const int* d_order, int n, int team_size,
                             int team_bytes, int teams_per_cta, int grid, int* d_next, double* gpool,
                             long long gslot_doubles, const uint32_t* Jpool,
                             const uint32_t* latpool, const int* winpool, const uint32_t* maskpool, double* outpool,
                             MainResult* results, unsigned char* statepool, cudaStream_t s)
{
  if (n == 0) return WLG_OK;
  const int threads = team_size * teams_per_cta;
  const int smem = team_bytes * teams_per_cta;
  MainFn fn = main_fn(variant, threads);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return WLG_ERR_CUDA;
  fn<<<grid, threads, smem, s>>>(d_descs, d_order, n, team_size, team_bytes, (variant & kVariantGlobal) != 0 ? 1 : 0,
                                 d_next, gpool, gslot_doubles, Jpool, latpool, winpool, maskpool, outpool, results,
                                 statepool);
  return launch_status();
}

}  // namespace wlg
