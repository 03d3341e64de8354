// The main-run kernel for problems spread over a thread-block cluster, CTAs of up
// to kClusterThreads threads.
#include "wlg_main.cuh"
#include "wlg_main_fn.h"

namespace wlg {

MainFn main_fn_cluster(int store) { return main_fn_cluster_of<kClusterThreads>(store); }

}  // namespace wlg
