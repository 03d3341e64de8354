// The main-run kernel for CTAs of up to 512 threads.
#include "wlg_main.cuh"
#include "wlg_main_fn.h"

namespace wlg {

MainFn main_fn_512(int store, bool tight) { return main_fn_of<512>(store, tight); }

}  // namespace wlg
