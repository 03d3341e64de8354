// The main-run kernel for CTAs of up to 1024 threads.
#include "wlg_main.cuh"
#include "wlg_main_fn.h"

namespace wlg {

MainFn main_fn_1024(int store, bool tight) { return main_fn_of<1024>(store, tight); }

}  // namespace wlg
