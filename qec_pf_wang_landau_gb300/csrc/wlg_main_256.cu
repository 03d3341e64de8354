// The main-run kernel for CTAs of up to 256 threads.
#include "wlg_main.cuh"
#include "wlg_main_fn.h"

namespace wlg {

MainFn main_fn_256(int store, bool tight) { return main_fn_of<256>(store, tight); }

}  // namespace wlg
