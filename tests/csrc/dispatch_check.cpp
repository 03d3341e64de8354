// The main run's dispatch (qec_pf_wang_landau_gb300/csrc/wlg_batch.h) on the CPU.
//
// Without arguments: over all window counts and walkers of a window, batches of
// every size and several devices, no problem gets a team that its kernel has no
// threads for, no rank is without a window, and the spread teams fit the SMs.
// Prints "ok".
//
// X Y boundary lg intervals walkers L problems sms resumable: prints "store global
// tight ranks team" for a batch of that many such problems whose longest window
// has L bins.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "wlg_batch.h"

namespace {

wlg::MainDesc desc(int X, int Y, int boundary, int lg, int I, int W, int L)
{
  wlg::MainDesc d{};
  d.X = X;
  d.Y = Y;
  d.N = X * Y;
  d.boundary = boundary;
  d.lg = lg;
  d.I = I;
  d.W = W;
  d.nwalk = I * W;
  d.team = wlg::round32(d.nwalk);
  d.L = L;
  d.nwL = wlg::lattice_words(X, Y);
  d.nwM = (((4 * d.N) >> lg) + 32) / 32;
  d.rows = wlg::lattice_rows(X, Y) ? 1 : 0;
  return d;
}

bool holds(const wlg::MainDesc& d, const wlg::MainLaunch& l, int spread, int n, int sms)
{
  const int ranks = wlg::variant_ranks(l.variant);
  if (ranks == 1) return l.team == d.team;
  for (int r = 0; r < ranks; ++r) {
    const int windows = d.I * (r + 1) / ranks - d.I * r / ranks;
    if (windows < 1 || windows * d.W > l.team) return false;
  }
  return l.team <= wlg::kClusterThreads && ranks <= spread && ranks <= 8 && static_cast<long long>(n) * ranks <= sms;
}

}  // namespace

int main(int argc, char** argv)
{
  if (argc == 11) {
    int v[10];
    for (int q = 0; q < 10; ++q) v[q] = std::atoi(argv[q + 1]);
    const wlg::MainDesc d = desc(v[0], v[1], v[2], v[3], v[4], v[5], v[6]);
    wlg::Prepared prep;
    prep.main.assign(static_cast<size_t>(v[7]), d);
    const int spread = v[9] != 0 ? 1 : wlg::spread_ranks(prep, v[8]);
    const wlg::MainLaunch l = wlg::main_launch(d, spread, v[9] != 0);
    std::printf("%d %d %d %d %d\n", wlg::variant_store(l.variant), (l.variant & wlg::kVariantGlobal) != 0 ? 1 : 0,
                (l.variant & wlg::kVariantTight) != 0 ? 1 : 0, wlg::variant_ranks(l.variant), l.team);
    return 0;
  }
  for (int I = 1; I <= 1024; ++I)
    for (int W = 1; I * W <= 1024; ++W)
      for (const int n : {1, 2, 4, 19, 39, 76, 77, 152, 153}) {
        const wlg::MainDesc d = desc(16, 16, 0, 2, I, W, std::max(2, 300 / I));
        wlg::Prepared prep;
        prep.main.assign(static_cast<size_t>(n), d);
        for (const int sms : {8, 132, 152}) {
          const int spread = wlg::spread_ranks(prep, sms);
          if (!holds(d, wlg::main_launch(d, spread, false), spread, n, sms)) {
            std::printf("%d windows of %d walkers, %d problems on %d SMs\n", I, W, n, sms);
            return 1;
          }
        }
      }
  std::printf("ok\n");
  return 0;
}
