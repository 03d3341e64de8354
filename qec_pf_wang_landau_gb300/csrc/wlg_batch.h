// Batch pipeline internals shared by the batch entry points
// (wlg_engine_host.cpp) and the serving loop (wlg_server.cpp): where a batch
// runs, the pre-run -> main-run hand-off, the kernel launchers and result
// stitching.  Not part of the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <string>
#include <utility>
#include <vector>

#include "../../include/wlg.h"
#include "wlg_engine.h"
#include "wlg_pool.h"

namespace wlg {

// ---- kernels (wlg_engine.cu)
wlg_status launch_pre_batch(const PreDesc* d_descs, int n, int threads, int smem, int8_t* Jpool, uint8_t* seen_pool,
                            int8_t* found_pool, int* fflag_pool, cudaStream_t s);
// variant: kernel_variant
int main_batch_capacity(int variant, int cta_threads, int smem);
wlg_status launch_main_batch(int variant, const MainDesc* d_descs, const int* d_order, int n, int team_size,
                             int team_bytes, int teams_per_cta, int grid, int* d_next, double* gpool,
                             long long gslot_doubles, const uint32_t* Jpool, const uint32_t* latpool,
                             const int* winpool, const uint32_t* maskpool, double* outpool, MainResult* results,
                             unsigned char* statepool, cudaStream_t s);

// ---- windows and stitching (interval.cpp, result_handling.cpp)
wlg_status make_windows(int e_min, int e_max, int n, float overlap, std::vector<int>& start, std::vector<int>& end);
using Curve = std::map<int, double>;
// mode: WLG_STITCH_REFERENCE or WLG_STITCH_DEFINED (wlg_context_set_stitching).
wlg_status stitch_windows(std::vector<Curve> windows, int X, int Y, std::vector<std::pair<int, double>>& out,
                          int mode = WLG_STITCH_REFERENCE);

// Stitched, normalised (E, log g) of one finished problem from its compact
// walker-0 output out[I][L] and its windows win[5 I] (start, end, base, Lb, E0).
wlg_status stitched_curve(const MainDesc& d, const double* out, const int* win,
                          std::vector<std::pair<int, double>>& res, int mode = WLG_STITCH_REFERENCE);

// ---- where a batch runs
// Device buffers of one batch, by role.
enum Slot {
  kPreDesc,
  kJ8,
  kSeen,
  kFound,
  kFflag,
  kMainDesc,
  kOrder,
  kNext,
  kJw,
  kLatw,
  kWin,
  kMask,
  kOut,
  kRes,
  kGpool,
  kState,
  kSlots
};

// A stream, a provider of device buffers, optional timing events, and what
// the batch did.
struct Exec {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t* ev = nullptr;  // 4 events, or nullptr for no timing
  float t_pre = 0, t_main = 0;
  double t_handoff = 0;
  long long h2d = 0, d2h = 0;
  int launches = 0;
  int main_forms = 0;  // bit v: a main-run launch of form v
  // per problem of the batch: when its main run started and ended (ms from
  // the first start, device clock); -1 for problems without a main run
  std::vector<double> p_start_ms, p_end_ms;
  std::string err;
  // teams per CTA chosen by an autotuner, by (form, team size); nullptr or
  // no entry: the built-in rule
  const std::map<std::pair<int, int>, int>* per_cta = nullptr;
  bool may_spread = true;  // problems over clusters, where SMs are idle
  WorkerPool* pool = nullptr;  // host threads for the per-problem phases; nullptr: the calling thread
  // streams on which the main-run launches of different groups run side by
  // side (fork/join through aux_ev: [0] fork, [1 + a] join of aux[a])
  cudaStream_t* aux = nullptr;
  cudaEvent_t* aux_ev = nullptr;
  // how many of `wanted` such streams there are; 0: all on `stream`, one after another
  virtual int side_streams(int wanted)
  {
    (void)wanted;
    return 0;
  }
  virtual ~Exec() = default;
  // device buffer for `slot` of at least `bytes` bytes
  virtual wlg_status buffer(Slot slot, size_t bytes, void** out) = 0;
  // bytes that buffer(slot) could be given now, when that is limited
  virtual size_t available(Slot slot)
  {
    (void)slot;
    return ~size_t{0} >> 1;
  }
};

inline wlg_status fail(Exec& ex, wlg_status st, const std::string& msg)
{
  ex.err = msg;
  return st;
}

template <typename T>
wlg_status upload(Exec& ex, Slot slot, const std::vector<T>& h, void** dptr)
{
  const size_t bytes = h.size() * sizeof(T);
  wlg_status st = ex.buffer(slot, bytes, dptr);
  if (st != WLG_OK || bytes == 0) return st;
  const cudaError_t e = cudaMemcpyAsync(*dptr, h.data(), bytes, cudaMemcpyHostToDevice, ex.stream);
  ex.h2d += static_cast<long long>(bytes);
  return e == cudaSuccess ? WLG_OK : fail(ex, WLG_ERR_CUDA, cudaGetErrorString(e));
}

template <typename T>
wlg_status download(Exec& ex, const void* dptr, std::vector<T>& h)
{
  if (h.empty()) return WLG_OK;
  const cudaError_t e = cudaMemcpyAsync(h.data(), dptr, h.size() * sizeof(T), cudaMemcpyDeviceToHost, ex.stream);
  ex.d2h += static_cast<long long>(h.size() * sizeof(T));
  return e == cudaSuccess ? WLG_OK : fail(ex, WLG_ERR_CUDA, cudaGetErrorString(e));
}

inline int round32(int x) { return (x + 31) / 32 * 32; }

wlg_status check_problem(const wlg_problem& q);

struct Prepared {
  std::vector<MainDesc> main;                  // problems that reach the main run
  std::vector<int> main_problem;               // index into the batch
  std::vector<std::vector<int>> starts, ends;  // per batch problem
  std::vector<int> lg;                         // per main entry: log2 of the energy step
};

// Main-run inputs of a prepared batch, on the host: packed couplings, start
// lattices, spectrum masks (32-bit words), windows, and the size of the
// walker-0 output; MainDesc offsets index these arrays.
struct Handoff {
  std::vector<uint32_t> Jw, latw, maskw;
  std::vector<int> win;
  long long n_out = 0;
};

// Pre-run outputs on the host, concatenated in problem order with the
// offsets of each PreDesc: couplings J8 [2N], visited energies seen [4N+1]
// (0/1), stored lattices found [n_int][N] (+-1, 0 where none), and fflag
// [n_int] found flags followed by [n_int] their energies.
struct PreOut {
  std::vector<PreDesc> pd;
  std::vector<int8_t> J8, found;
  std::vector<uint8_t> seen;
  std::vector<int> fflag;
};

// Validation and pre-run descriptors (sizes the PreOut arrays).
wlg_status prerun_descs(const wlg_problem* probs, int n, wlg_result* results, PreOut& po, int& threads, int& smem,
                        std::string& err);
// Validation and the pre-run of every problem (one launch).
// couplings (int8 [sum 2N], problem order): the class-'i' bond patterns of the
// problems whose given[p] != 0 (all of them when given is null); the others
// draw theirs.  Null couplings: every problem draws.
wlg_status run_prerun(Exec& ex, const wlg_problem* probs, int n, wlg_result* results, PreOut& po,
                      const int8_t* couplings = nullptr, const unsigned char* given = nullptr);
// The hand-off to the main run on the host.  Problems that cannot start the
// main run get their status in `results` and no MainDesc.
wlg_status handoff(Exec& ex, const wlg_problem* probs, int n, wlg_result* results, const PreOut& po, Prepared& prep,
                   Handoff& ho);
// run_prerun + handoff.
wlg_status prepare_batch(Exec& ex, const wlg_problem* probs, int n, wlg_result* results, Prepared& prep, Handoff& ho,
                         const int8_t* couplings = nullptr, const unsigned char* given = nullptr);

// A main-run kernel: how it keeps the lattice (Store), plus where FP64 log g
// and the histogram live and whether the team does without guard bins and ring.
constexpr int kVariantGlobal = 8;  // log g and histogram in global memory
constexpr int kVariantTight = 16;  // see team_layout; always with kVariantGlobal
constexpr int kSmemBytes = 227 * 1024;

// in bits 8 and up: CTAs of the cluster a problem is spread over, 0 or 1 none
constexpr int kVariantRanks = 256;

inline int variant_store(int variant) { return variant & 7; }
inline int variant_ranks(int variant) { return variant >= kVariantRanks ? variant / kVariantRanks : 1; }

// The form wlg.h reports: 0 lattice and log g in shared memory, 1 lattice in a
// register, 2 the register with a neighbour table, 3 log g in global memory.
inline int variant_form(int variant)
{
  if ((variant & kVariantGlobal) != 0) return 3;
  const int s = variant_store(variant);
  return s == kStoreReg || s == kStoreTable ? s : 0;
}

// Shared-memory bytes of a team running d in `variant`.
inline int team_bytes(const MainDesc& d, int variant, int team)
{
  return align16(
    team_layout(d, team, variant_store(variant), (variant & kVariantGlobal) != 0, (variant & kVariantTight) != 0).bytes +
    16);
}

// The lattice storage of d: registers up to 64 sites, else bonds where a row's
// right and down bonds fit one word (Y <= 16: two words read per proposal
// instead of three rows and three couplings; periodic lattices, with no bond
// missing, do without masks per row: 16x16 on every SM 0.322 -> 0.303 us a step),
// else rows, else linear words.
// Tight states keep rows, whose tables take no room.
inline int lattice_store(const MainDesc& d, bool tight)
{
  if (d.N <= 64) return d.X >= 3 && d.Y >= 3 ? kStoreTable : kStoreReg;
  if (d.rows == 0) return kStoreLinear;
  if (d.Y > 16 || tight) return kStoreRows;
  return d.boundary == 0 ? kStoreBonds : kStoreBondsOpen;
}

inline int tight_variant(const MainDesc& d) { return lattice_store(d, true) | kVariantGlobal | kVariantTight; }

// Bytes that decide whether a problem is taken at all: 8 per bin and walker
// (16 for lattices in registers) plus the lattice must fit one SM.
inline int admission_bytes(const MainDesc& d, int team)
{
  const int store = lattice_store(d, true);
  const bool reg = store == kStoreReg || store == kStoreTable;
  return team_bytes(d, tight_variant(d), team) +
         (reg ? 8 * d.L * team - (store == kStoreTable ? align16(4 * d.N) : 0) : 0);
}

// The kernel of d: everything in shared memory where it fits, else log g and
// the histogram in global memory (read and written once per sweep), else the
// tight layout.  Rows of 17 to 32 sites keep their bonds in two words where that
// fits (24x24, 128 walkers on an SM: 0.25 -> 0.19 us a step against rows), not in
// resumable runs, whose saved lattices have a word a row.  Problems of one launch
// share it.
inline int kernel_variant(const MainDesc& d, int team, bool resumable)
{
  const int store = lattice_store(d, false);
  if (store == kStoreRows && !resumable) {
    const int two = d.boundary == 0 ? kStoreBonds2 : kStoreBonds2Open;
    if (team_bytes(d, two, team) <= kSmemBytes) return two;
    if (team_bytes(d, two | kVariantGlobal, team) <= kSmemBytes) return two | kVariantGlobal;
  }
  if (team_bytes(d, store, team) <= kSmemBytes) return store;
  if (team_bytes(d, store | kVariantGlobal, team) <= kSmemBytes) return store | kVariantGlobal;
  return tight_variant(d);
}

// Threads of one of the teams a problem is spread over.
inline int rank_team(const MainDesc& d, int ranks) { return round32((d.I + ranks - 1) / ranks * d.W); }

// CTAs a problem is spread over when each may take `spread`: no team smaller than
// four warps, one per partition of an SM, and a window at least in each.  A team
// the cluster kernel has no threads for (kClusterThreads; windows of many walkers,
// or a small spread) leaves the problem on one CTA.
inline int problem_ranks(const MainDesc& d, int spread)
{
  int r = 1;
  while (r < spread && d.team / (2 * r) >= 128 && d.I >= 2 * r) r *= 2;
  return rank_team(d, r) <= kClusterThreads ? r : 1;
}

// The largest spread (up to 8) that leaves every team an SM of its own.  A
// problem of 512 walkers on one SM has four warps on each partition, which share
// its issue slots; on four SMs each warp has its own.
inline int spread_ranks(const Prepared& prep, int sms)
{
  int spread = 1;
  for (int s = 2; s <= 8; s *= 2) {
    int teams = 0;
    for (const MainDesc& d : prep.main) teams += problem_ranks(d, s);
    if (teams <= sms) spread = s;
  }
  return spread;
}

// How run_main launches d: its kernel (a cluster's ranks included) and the
// threads of a team.  Tight states are not spread.
struct MainLaunch {
  int variant, team;
};
inline MainLaunch main_launch(const MainDesc& d, int spread, bool resumable)
{
  const int ranks = problem_ranks(d, spread);
  if (ranks > 1) {
    const int team = rank_team(d, ranks), variant = kernel_variant(d, team, resumable);
    if ((variant & kVariantTight) == 0) return {variant | ranks * kVariantRanks, team};
  }
  return {kernel_variant(d, d.team, resumable), d.team};
}

}  // namespace wlg
