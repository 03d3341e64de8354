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
#include "wlg_pre.cuh"
#include "wlg_rng.cuh"

namespace wlg {
namespace {

// ------------------------------------------------------------ pre-run -----

// Draws, in {-1, 1}: the couplings of a sample with its error chain
// (wl.cu:364-428, prerun.cu:56-75) and the lattice every walker starts from
// (wl.cu:430-457, CAS winner fixed to site 0).
__device__ __forceinline__ int8_t draw_coupling(const PreDesc& d, const int8_t* __restrict__ Jpool, int q)
{
  int8_t v;
  if (d.given_J) {
    v = Jpool[d.off_J + q];
  } else {
    Stream st;
    st.init(key_size(d.seed, static_cast<uint64_t>(d.sample)), 0, static_cast<uint64_t>(q));
    const double u = st.uniform();
    v = (u < d.prob) ? -1 : 1;
  }
  const bool h = d.error_class == 'h' || d.error_class == 'c', vert = d.error_class == 'v' || d.error_class == 'c';
  if (h && q >= d.N && q < d.N + d.Y) v = static_cast<int8_t>(-v);
  if (vert && q < d.N && q % d.Y == 0) v = static_cast<int8_t>(-v);
  return v;
}

__device__ __forceinline__ int8_t draw_spin(const PreDesc& d, int q)
{
  const uint64_t key = key_u32(d.seed, static_cast<uint64_t>(d.sample));
  Stream st;
  st.init(key, 1, 0);
  const float p0 = st.uniform();
  st.init(key, 1, static_cast<uint64_t>(q) + 1);
  const double u = st.uniform();
  return (u < p0) ? -1 : 1;
}

// The whole pre-run of one problem on bond words.
template <bool kTwo, bool kKeys>
__device__ __forceinline__ void pre_problem(const PreDesc& d, unsigned char* smem, int8_t* __restrict__ Jpool,
                                            uint8_t* __restrict__ seen_pool, int8_t* __restrict__ found_pool,
                                            int* __restrict__ fflag_pool)
{
  constexpr int kW = kTwo ? 2 : 1;
  const int N = d.N, X = d.X, Y = d.Y, L = 4 * N + 1, tid = threadIdx.x;
  const int lg = energy_step_log2(d.boundary), len = (4 * N >> lg) + 1;
  const int threads = (d.walkers + 31) / 32 * 32, Lh = pre_hist_words(len);
  if (tid >= threads) return;  // warps beyond this problem's walkers
  const PreLayout l = pre_layout(X, Y, len, d.n_int, threads);
  uint32_t* hist = reinterpret_cast<uint32_t*>(smem + l.off_hist);
  uint32_t* thr = reinterpret_cast<uint32_t*>(smem + l.off_thr);
  uint32_t* Jr = reinterpret_cast<uint32_t*>(smem + l.off_J);
  uint32_t* base = reinterpret_cast<uint32_t*>(smem + l.off_base);
  uint2* col = reinterpret_cast<uint2*>(smem + l.off_col);
  uint4* row = reinterpret_cast<uint4*>(smem + l.off_row);
  PreWalk p{X, Y, d.boundary, -2 * N, lg, len, Lh, 0, d.n_int, d.len_int, d.n_iter, threads, hist,
            reinterpret_cast<uint32_t*>(smem + l.off_claim), reinterpret_cast<int*>(smem + l.off_foundE), thr,
            col, row, Jr, Jr + X, reinterpret_cast<uint32_t*>(smem + l.off_words), found_pool + d.off_found};
  const PreSync sync{threads};
  for (int q = tid; q < 2 * Lh; q += threads) hist[q] = 0;
  for (int q = tid; q < d.n_int; q += threads) {
    p.claim[q] = kPreEmpty;
    p.found_E[q] = 0;
  }
  for (int q = tid; q < X; q += threads) Jr[q] = Jr[X + q] = base[q] = 0;
  fill_accept(thr, tid);
  fill_bonds<kTwo>(col, row, X, Y, d.boundary, tid, threads);
  sync();
  for (int q = tid; q < 2 * N; q += threads) {
    const int8_t v = draw_coupling(d, Jpool, q);
    const int s = q < N ? q : q - N, i = s / Y;
    if (v < 0) atomicOr(&Jr[(q < N ? 0 : X) + i], 1u << (s - i * Y));
    Jpool[d.off_J + q] = v;
  }
  for (int q = tid; q < N; q += threads) {
    const int i = q / Y;
    if (draw_spin(d, q) < 0) atomicOr(&base[i], 1u << (q - i * Y));
  }
  sync();
  const int w = tid;
  uint32_t unsat = 0;
  for (int i = 0; i < X; ++i) {
    uint32_t h, v = 0;
    bond_words<kTwo>(base[i], base[i + 1 < X ? i + 1 : 0], Jr[i], Jr[X + i], Y, d.boundary != 0, i + 1 == X, h, v);
    p.words[i * kW * threads + w] = h;
    unsat += __popc(h);
    if constexpr (kTwo) {
      p.words[(i * kW + 1) * threads + w] = v;
      unsat += __popc(v);
    }
  }
  // wl.cu:261-340: minus the sum over bonds of s s J
  const int bonds = d.boundary == 0 ? 2 * N : 2 * N - X - Y;
  int E = 2 * static_cast<int>(unsat) - bonds;
  p.bin0 = (E + 2 * N) & ((1 << lg) - 1);  // the lattice's energies start there
  p.e_min += p.bin0;
  uint32_t s0 = base[0] & 1u;
  uint64_t pos = 0;
  pre_walk<kTwo, false, kKeys>(p, sync, w, w < d.walkers, key_u32(d.seed, static_cast<uint64_t>(d.sample)),
                        2 + static_cast<uint64_t>(w), pos, E, s0);
  for (int q = tid; q < L; q += threads)
    seen_pool[d.off_seen + q] = ((q - p.bin0) & ((1 << lg) - 1)) == 0 && hist[(q - p.bin0) >> lg] != 0 ? 1 : 0;
  for (int q = tid; q < d.n_int; q += threads) {
    const bool found = p.claim[q] != kPreEmpty;
    fflag_pool[d.off_fflag + q] = found ? 1 : 0;
    fflag_pool[d.off_fflag + d.n_int + q] = found ? p.found_E[q] : 0;
  }
}

// The whole pre-run on int8 lattices, 64-bit counts and two barriers a round:
// rows of more than 32 sites, 2^31 visits and more, and bond words too large
// for shared memory.
__device__ __forceinline__ void pre_problem_i8(const PreDesc& d, unsigned char* smem, int8_t* __restrict__ Jpool,
                                               uint8_t* __restrict__ seen_pool, int8_t* __restrict__ found_pool,
                                               int* __restrict__ fflag_pool)
{
  const int N = d.N, X = d.X, Y = d.Y;
  const int L = 4 * N + 1;
  const int e_min = -2 * N;
  unsigned long long* hist = reinterpret_cast<unsigned long long*>(smem);
  int* claim = reinterpret_cast<int*>(hist + L);
  int* found = claim + d.n_int;
  int* misc = found + d.n_int;  // [0] start energy
  int8_t* J = reinterpret_cast<int8_t*>(misc + 4);
  int8_t* lat = J + 2 * N;  // [walkers][N]

  const int tid = threadIdx.x;
  for (int q = tid; q < 2 * N; q += blockDim.x) {
    J[q] = draw_coupling(d, Jpool, q);
    Jpool[d.off_J + q] = J[q];
  }
  for (int q = tid; q < L; q += blockDim.x) hist[q] = 0;
  for (int q = tid; q < d.n_int; q += blockDim.x) {
    claim[q] = INT_MAX;
    found[q] = 0;
  }
  for (int q = tid; q < N; q += blockDim.x) lat[q] = draw_spin(d, q);
  __shared__ uint32_t acc_thr[kAcceptEntries];
  static_assert(sizeof(acc_thr) <= kPreTableBytes);
  fill_accept(acc_thr, tid);
  __syncthreads();
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
      acc = dd >= 1 || (dd >= -24 && xa < acc_thr[ti]);  // see fill_accept
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

// One CTA per problem.  CTAs of up to 256 threads may take 255 registers each:
// the walk is latency-bound, and its loads are then issued further ahead.
template <int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads, 1)
  k_pre_batch(const PreDesc* __restrict__ descs, int n, int8_t* __restrict__ Jpool, uint8_t* __restrict__ seen_pool,
              int8_t* __restrict__ found_pool, int* __restrict__ fflag_pool)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int p = blockIdx.x;
  if (p >= n) return;
  const PreDesc d = descs[p];
  if (d.bonds == 0) {
    pre_problem_i8(d, smem, Jpool, seen_pool, found_pool, fflag_pool);
  } else if (d.Y <= 16) {
    pre_problem<false, kMaxThreads <= 256>(d, smem, Jpool, seen_pool, found_pool, fflag_pool);
  } else {
    pre_problem<true, kMaxThreads <= 256>(d, smem, Jpool, seen_pool, found_pool, fflag_pool);
  }
}

}  // namespace

// ------------------------------------------------------------ launchers ----

wlg_status launch_pre_batch(const PreDesc* d_descs, int n, int threads, int smem, int8_t* Jpool, uint8_t* seen_pool,
                            int8_t* found_pool, int* fflag_pool, cudaStream_t s)
{
  if (n == 0) return WLG_OK;
  const auto kernel = threads <= 256 ? &k_pre_batch<256> : &k_pre_batch<1024>;
  if (smem > 48 * 1024 && !allow_shared(kernel, kPreTableBytes)) return WLG_ERR_CUDA;
  kernel<<<n, threads, smem, s>>>(d_descs, n, Jpool, seen_pool, found_pool, fflag_pool);
  return launch_status();
}

MainFn main_fn(int variant, int cta_threads)
{
  if (variant_ranks(variant) > 1) return main_fn_cluster(variant_store(variant));
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
  if (smem > kSharedBytes || !allow_shared(fn)) return 0;
  const int ranks = variant_ranks(variant);
  if (ranks > 1) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(ranks);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(ranks));
    cfg.blockDim = dim3(static_cast<unsigned>(cta_threads));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) return 0;
    return clusters * ranks;
  }
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
  if (!allow_shared(fn)) return WLG_ERR_CUDA;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = s;
  if (variant_ranks(variant) > 1) {
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(variant_ranks(variant));
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
  }
  const cudaError_t e =
    cudaLaunchKernelEx(&cfg, fn, d_descs, d_order, n, team_size, team_bytes, (variant & kVariantGlobal) != 0 ? 1 : 0,
                       d_next, gpool, gslot_doubles, Jpool, latpool, winpool, maskpool, outpool, results, statepool);
  return e == cudaSuccess ? launch_status() : WLG_ERR_CUDA;
}

}  // namespace wlg
