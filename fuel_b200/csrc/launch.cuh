#pragma once
#include <cuda_runtime.h>

namespace fq {

// Every kernel goes out with the programmatic-dependent-launch attribute: all of them call griddepcontrol.wait before they
// touch memory an earlier kernel of the stream may have written, so the attribute changes when a kernel's blocks are put on
// the SMs, never what they see. What FUELQ_OPT_PDL adds is the caller's promise that WEIGHTS are not written by the stream's
// preceding work, which lets a call's first kernel stream them before that wait (`early_w` of the mat-vec kernels; the later
// kernels of a call always may: its first kernel lets them start only after its own wait, see quantize_q8k_kernel's
// `late_trigger`).
template <typename... KArgs, typename... Args>
cudaError_t launch_if(bool dependent, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  return launch_if(true, kernel, grid, block, smem, stream, args...);
}

}  // namespace fq
