// Choice of the kernel that evaluates a Green-function launch:
//   * a tridiagonalisation per k (tg_tridiag.cu) or an eigendecomposition per k
//     (tg_spectral.cu) where the launch carries one;
//   * else an inversion per (k, z) point, replacing invers = zgetrf + zgetri
//     (mod_tools.F90:796-829): blocked Gauss-Jordan on the FP64 tensor cores
//     (tg_green_mma.cu) for the dimensions it is instantiated for; the one-warp kernel
//     (tg_green_warp.cu) for dimensions of at most 20, whose panels would be mostly padding;
//     the thread-block-cluster kernel (tg_green_cluster.cu) for every other one up to 288.
#include "tg_internal.cuh"

namespace tg {

// dimensions with a single-SM inversion kernel and its fused output stages
int green_supported(int n) { return green_mma_supported(n, MODE_RAW) || green_warp_supported(n, MODE_RAW); }

bool green_is_spectral(const GreenArgs& a) {
  return a.eigU && a.eigL && a.n_e > 0 && spectral_supported(a.mode, a.mode2, a.out2 != nullptr);
}

cudaError_t launch_green(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used) {
  if (a.triQ) {
    if (grid_used) *grid_used = 0;
    return launch_green_tri(a, num_sms, s);
  }
  if (green_is_spectral(a)) {
    if (grid_used) *grid_used = 0;
    return launch_green_spectral(a, a.eigU, a.eigL, a.outinv, num_sms, s);
  }
  if (a.eout || a.eout2) return cudaErrorInvalidValue;   // only the spectral kernel writes sidecars
  // eigendecompositions without an H(k) table: the pass is k-major, which only the spectral
  // kernel walks without a table
  if (a.eigU && !a.htab) return cudaErrorInvalidValue;
  if (green_mma_supported(a.n, a.mode)) return launch_green_mma(a, num_sms, s, grid_used);
  if (green_warp_supported(a.n, a.mode)) return launch_green_warp(a, num_sms, s, grid_used);
  if (grid_used) *grid_used = 0;
  if (green_cluster_supported(a.n, a.mode)) return launch_green_cluster(a, num_sms, s);
  return cudaErrorInvalidValue;
}

}  // namespace tg
