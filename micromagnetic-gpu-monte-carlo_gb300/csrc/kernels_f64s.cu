// kernels_f64s.cu -- FP64 transforms whose products and sums round one by one
// (f64s), where kernels_f64.cu's passes use multiply-adds: the transform of the
// demag tensor, whose spectrum every precision's kernels read, and the demag
// convolution of the relaxation.
#include "kernels.cuh"

namespace mmc {

cudaError_t launch_demag_sym_relax(const Geom& g, const FftPlan& px, const FftPlan& py, const FftPlan& pz,
                                   const DemagTuning& tun, const double* m, double* h, void* spec, const void* khat,
                                   cudaStream_t st) {
  return demag_impl<f64s>(g, px, py, pz, tun, reinterpret_cast<const f64s*>(m), reinterpret_cast<f64s*>(h), spec,
                          khat, st, 1, nullptr, PASS_SYM);
}

// Forward transform of the six real tensor blocks k6[c][z][y][x] (padded
// grid) into spec64[c][kz][ky][kx] (src/main.cu:593-642 ran cuFFT D2Z here).
cudaError_t launch_tensor_fft(const Geom& g, const FftPlan& px, const FftPlan& py, const FftPlan& pz,
                              const DemagTuning& tun, const double* k6, double2* spec64, cudaStream_t st) {
  const long long ns = g.nspec;
  f64s2* spec = reinterpret_cast<f64s2*>(spec64);
  MMC_TRY(cudaMemsetAsync(spec64, 0, 6 * (size_t)ns * sizeof(double2), st));
  MMC_TRY(run_x_forward<f64s>(px, 6, g.nxp, g.nyp, g.nyp * g.nzp, reinterpret_cast<const f64s*>(k6), g.np, spec, ns, g.nyp, g.hx, g.hxp, 1,
                                tun.x_threads, st, 1, 0, 0));
  const long long ystride = g.hxp, yplane = (long long)g.nyp * g.hxp;
  for (int half = 0; half < 2; ++half) {
    f64s2* S = spec + 3 * half * ns;
    if (g.nyp > 1)
      MMC_TRY(run_col_pass<f64s>(py, 3, S, ns, nullptr, g.hx, g.nzp, yplane, ystride, g.nyp, g.nyp, PASS_FWD, 1.0,
                                   tun.col_tx, tun.col_threads, st));
    if (g.nzp > 1)
      MMC_TRY(run_col_pass<f64s>(pz, 3, S, ns, nullptr, g.hx, g.nyp, ystride, yplane, g.nzp, g.nzp, PASS_FWD, 1.0,
                                   tun.col_tx, tun.col_threads, st));
  }
  return cudaSuccess;
}

cudaError_t launch_prepare_f64s(int max_dyn_smem) { return prepare_passes<f64s>(max_dyn_smem); }

}  // namespace mmc
