// Entry points of the persistent main-run kernel, one translation unit per
// largest CTA size (wlg_main_256.cu, wlg_main_512.cu, wlg_main_1024.cu), and one
// for clusters (wlg_main_cluster.cu).
#pragma once

#include <cstdint>

#include "wlg_engine.h"

namespace wlg {

using MainFn = void (*)(const MainDesc*, const int*, int, int, int, int, int*, double*, long long, const uint32_t*,
                        const uint32_t*, const int*, const uint32_t*, double*, MainResult*, unsigned char*);

// The kernel for a lattice storage (Store), with or without the tight layout.
MainFn main_fn_256(int store, bool tight);
MainFn main_fn_512(int store, bool tight);
MainFn main_fn_1024(int store, bool tight);
MainFn main_fn_cluster(int store);  // a problem's windows spread over a cluster

}  // namespace wlg
