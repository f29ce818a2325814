// Host-side helpers shared by the .cu files: error reporting and launch checks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/dsa_b200.h"

namespace dsa {

// Records a message for dsa_last_error_string() and returns `code`.
int set_error(int code, const char* fmt, ...);
// cudaGetLastError() after a launch; no synchronisation.
int check_launch(const char* what);
// A launch that, with `overlapped`, may start under the end of the kernel before it on the stream (griddepcontrol in both).
template <typename... Params, typename... Args>
inline void launch_after(int overlapped, void (*kern)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = overlapped ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);          // its error is the launch check's
}
// Multiprocessor count of the current device (cached per device).
int sm_count();

}  // namespace dsa
