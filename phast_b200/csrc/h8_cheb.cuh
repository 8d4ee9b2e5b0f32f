// One-launch Chebyshev solve of the coarsest multigrid level (h8_cheb.cu).
#pragma once
#include "h8_kernels.cuh"
#include "reduce.cuh"

namespace phastb {

constexpr int kChebMaxSteps = 15;

// Exchange words of a level; zero them once (coarse_cheb_reset) before the first solve.
size_t coarse_cheb_bytes(const VoxGeom& g);
int coarse_cheb_reset(const VoxGeom& g, void* exchange, cudaStream_t s);

// From x = 0 with right-hand side b (less bsums / n_red per component when given): d = invd b inv_theta, x = d, then
// `steps` times r -= A d, d = c1 d + c2 invd r, x += d.  With sums, x's component sums go to sums->out.  lam, mu: (E,
// 8) moduli.  PHASTB_UNSUPPORTED when the level does not fit or the device cannot run it.
int coarse_cheb_launch(const VoxGeom& g, const float* lam, const float* mu, const float* b, const float* invd, float* x,
                       const double* bsums, double inv_theta, const double* c1, const double* c2, int steps,
                       const RedWs* sums, void* exchange, const int* guard, cudaStream_t s);

}  // namespace phastb
