// The integer batch kernels, in a translation unit of their own: the library's two large sets of kernels compile side by side
// (53 s with --threads, 105 one after the other).
#include "ibatch.cuh"

#include "launch.cuh"

namespace fq {
namespace {
template <class F, int MT, bool kGrouped>
cudaError_t launch_kernel(const IbParams& p, unsigned grid, int warps, size_t smem, int max_smem, cudaStream_t stream) {
  // the plan deals the groups out over two thread blocks of eight warps an SM: registers for sixteen
  static_assert(!kGrouped || MT <= kIbGroupRows / 8, "wider forms have registers for eight warps only");
  static bool attr_set[64] = {};
  auto kern = ibatch_kernel<F, MT, kGrouped>;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  return launch(kern, dim3(grid), dim3(32 * warps), smem, stream, p);
}

template <class F>
cudaError_t launch_tiles(int mt, const IbParams& p, unsigned grid, int warps, size_t smem, int max_smem, cudaStream_t stream) {
  switch (mt) {
    case 1: return launch_kernel<F, 1, false>(p, grid, warps, smem, max_smem, stream);
    case 2: return launch_kernel<F, 2, false>(p, grid, warps, smem, max_smem, stream);
    case 3: return launch_kernel<F, 3, false>(p, grid, warps, smem, max_smem, stream);
    case 4: return launch_kernel<F, 4, false>(p, grid, warps, smem, max_smem, stream);
    case 6: return launch_kernel<F, 6, false>(p, grid, warps, smem, max_smem, stream);
    case 8: return launch_kernel<F, 8, false>(p, grid, warps, smem, max_smem, stream);
    default: return cudaErrorInvalidValue;
  }
}
template <class F>
cudaError_t launch_groups(int mt, const IbParams& p, unsigned grid, int warps, size_t smem, int max_smem, cudaStream_t stream) {
  switch (mt) {
    case 1: return launch_kernel<F, 1, true>(p, grid, warps, smem, max_smem, stream);
    case 2: return launch_kernel<F, 2, true>(p, grid, warps, smem, max_smem, stream);
    case 4: return launch_kernel<F, 4, true>(p, grid, warps, smem, max_smem, stream);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace

cudaError_t ibatch_launch(int type, int mt, bool grouped, const IbParams& p, unsigned grid, int warps, size_t smem, int max_smem, cudaStream_t stream) {
  if (grouped) {
    if (type == kQ4K) return launch_groups<IbQ4K>(mt, p, grid, warps, smem, max_smem, stream);
    if (type == kQ6K) return launch_groups<IbQ6K>(mt, p, grid, warps, smem, max_smem, stream);
    return cudaErrorInvalidValue;
  }
  switch (type) {
    case kQ4K: return launch_tiles<IbQ4K>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ5K: return launch_tiles<IbQ5K>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ6K: return launch_tiles<IbQ6K>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ8_0: return launch_tiles<IbQ8_0>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ2K: return launch_tiles<IbQ2K>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ3K: return launch_tiles<IbQ3K>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ4_0: return launch_tiles<IbQ4_0>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ4_1: return launch_tiles<IbQ4_1>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ5_0: return launch_tiles<IbQ5_0>(mt, p, grid, warps, smem, max_smem, stream);
    case kQ5_1: return launch_tiles<IbQ5_1>(mt, p, grid, warps, smem, max_smem, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t ibatch_device_error(int* code, bool clear) {
  cudaError_t e = cudaMemcpyFromSymbol(code, g_fq_dev_error, sizeof(int));
  if (e == cudaSuccess && clear && *code) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_fq_dev_error, &zero, sizeof(int));
  }
  return e;
}

}  // namespace fq
