// kernels_f32.cu -- FP32 instantiation of the hot-path kernels (multiply-add
// contraction enabled).
#include "fused2d.cuh"
#include "grad.cuh"
#include "kernels.cuh"

namespace mmc {
MMC_INSTANTIATE_LAUNCHERS(float)
MMC_INSTANTIATE_FUSED(float)
MMC_INSTANTIATE_GRAD(float)
bool mc_split_eligible(const Geom& g, const FftPlan& px) { return mc_split_ok<float>(g, px) && g.nx <= 12288; }
bool col_pipe_eligible(const FftPlan& py) { return col_pipe_ok(py); }
cudaError_t launch_split_rows(const Geom& g, float* a, int count, bool to_split, cudaStream_t st) {
  const long long rows = (long long)g.ny * g.nz, all = 3 * rows * count;
  if (all > INT_MAX) return cudaErrorInvalidValue;
  k_split_rows<<<(unsigned)all, std::min(256, (g.nx + 31) / 32 * 32), g.nx * sizeof(float), st>>>(
      a, g.nx, FastDiv((uint32_t)rows), FastDiv((uint32_t)g.ny), to_split ? 1 : 0);
  return cudaGetLastError();
}
}  // namespace mmc
