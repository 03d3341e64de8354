// Shared helpers of the engine's translation units (not part of the ABI).
#pragma once

#include <cuda_runtime.h>

#include <new>

#include "../../include/wlg.h"

namespace wlg {

inline cudaStream_t as_stream(wlg_stream s) { return static_cast<cudaStream_t>(s); }

// Status of the launches just issued (configuration errors surface here;
// faults inside a kernel surface at the next synchronising call).
inline wlg_status launch_status()
{
  return cudaGetLastError() == cudaSuccess ? WLG_OK : WLG_ERR_CUDA;
}

inline wlg_status cuda_status(cudaError_t e)
{
  if (e == cudaSuccess) return WLG_OK;
  if (e == cudaErrorMemoryAllocation) return WLG_ERR_OOM;
  return WLG_ERR_CUDA;
}

// Shared memory a CTA can have on sm_103.
constexpr int kSharedBytes = 227 * 1024;

// Lets `kernel`, which has static_bytes of static shared memory, be launched with
// as much dynamic shared memory as a CTA can have.  The limit is a property of the
// function that all threads share: always the same value, so that no thread lowers
// it between another's call and launch.
template <typename Kernel>
bool allow_shared(Kernel kernel, int static_bytes = 0)
{
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedBytes - static_bytes) ==
         cudaSuccess;
}

// Runs an entry point's body so that no C++ exception crosses the C ABI:
// allocation failures become WLG_ERR_OOM, anything else WLG_ERR_INVALID.
template <typename F>
wlg_status guarded(F&& body) noexcept
{
  try {
    return body();
  } catch (const std::bad_alloc&) {
    return WLG_ERR_OOM;
  } catch (...) {
    return WLG_ERR_INVALID;
  }
}

}  // namespace wlg
