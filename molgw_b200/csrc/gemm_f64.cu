// Instantiations and launchers of the FP64 DMMA tile engine.
#include <utility>

#include "kernels.cuh"

namespace rigw {

template <int BM, int BN>
static void launch_dgemm(const GemmItem* items, int n, int ny, cudaStream_t s) {
  if (n <= 0 || ny <= 0) return;
  using Cfg = DgemmCfg<BM, BN>;
  dgemm_mn_kernel<BM, BN><<<dim3(n, ny), Cfg::kThreads, Cfg::kSmemBytes, s>>>(items);
}

void launch_dgemm_128x128(const GemmItem* items, int n, int ny, cudaStream_t s) {
  launch_dgemm<128, 128>(items, n, ny, s);
}
void launch_dgemm_64x128(const GemmItem* items, int n, int ny, cudaStream_t s) {
  launch_dgemm<64, 128>(items, n, ny, s);
}

void launch_dgemm_256x32(const GemmItem* items, int n, int ny, cudaStream_t s) {
  launch_dgemm<256, 32>(items, n, ny, s);
}
void launch_dgemm_128x64(const GemmItem* items, int n, int ny, cudaStream_t s) {
  launch_dgemm<128, 64>(items, n, ny, s);
}

// Tiles of 32 columns and 32-row warps: an SM does 64 FP64 multiply-adds per clock, so a 128 x
// 128 x 128 product takes 17 us on one of them however it is written.  Launches that leave SMs
// idle (the panel solve and the diagonal update on the factorization's critical path, small
// problems) are cut into these.
void launch_dgemm_128x32(const GemmItem* items, int n, int ny, cudaStream_t s) {
  if (n > 0 && ny > 0)
    dgemm_mn_kernel<128, 32, 3, 32>
        <<<dim3(n, ny), DgemmCfg<128, 32, 3, 32>::kThreads, DgemmCfg<128, 32, 3, 32>::kSmemBytes, s>>>(items);
}
void launch_dgemm_64x32(const GemmItem* items, int n, int ny, cudaStream_t s) {
  if (n > 0 && ny > 0)
    dgemm_mn_kernel<64, 32, 3, 32>
        <<<dim3(n, ny), DgemmCfg<64, 32, 3, 32>::kThreads, DgemmCfg<64, 32, 3, 32>::kSmemBytes, s>>>(items);
}

cudaError_t prepare_dgemm_kernels() {
  for (auto set : {std::make_pair(&dgemm_mn_kernel<128, 32, 3, 32>, DgemmCfg<128, 32, 3, 32>::kSmemBytes),
                   std::make_pair(&dgemm_mn_kernel<64, 32, 3, 32>, DgemmCfg<64, 32, 3, 32>::kSmemBytes)}) {
    cudaError_t es = cudaFuncSetAttribute(*set.first, cudaFuncAttributeMaxDynamicSharedMemorySize, int(set.second));
    if (es != cudaSuccess) return es;
  }
  cudaError_t e = cudaFuncSetAttribute(dgemm_mn_kernel<256, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(DgemmCfg<256, 32>::kSmemBytes));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(dgemm_mn_kernel<128, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           int(DgemmCfg<128, 64>::kSmemBytes));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(dgemm_mn_kernel<128, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(DgemmCfg<128, 128>::kSmemBytes));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(dgemm_mn_kernel<64, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              int(DgemmCfg<64, 128>::kSmemBytes));
}

}  // namespace rigw
