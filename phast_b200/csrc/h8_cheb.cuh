// One-launch Chebyshev solve of the coarsest multigrid level (h8_cheb.cu).
#pragma once
#include "h8_tile.cuh"

namespace phastb {

constexpr int kChebMaxSteps = 15;
constexpr int kChebBlocks = kMaxBlocks;  // blocks of one launch at most

// Exchange words of a level of so many nodes; zero them once (coarse_cheb_reset) before the first solve.
size_t coarse_cheb_bytes(long long nodes);
int coarse_cheb_reset(long long nodes, void* exchange, cudaStream_t s);

// From x = 0 with right-hand side b (less bsums / n_red per component when given): d = invd b inv_theta, x = d, then
// `steps` times r -= A d, d = c1 d + c2 invd r, x += d.  With sums, x's component sums go to sums->out.  lam, mu: (E,
// 8) moduli.  PHASTB_UNSUPPORTED when the level does not fit or the device cannot run it.
int coarse_cheb_launch(const VoxGeom& g, const float* lam, const float* mu, const float* b, const float* invd, float* x,
                       const double* bsums, double inv_theta, const double* c1, const double* c2, int steps,
                       const RedWs* sums, void* exchange, const int* guard, cudaStream_t s);

// The same for every live cell of a packed batch (cells: the host's copy of the table): per-cell theta and delta (c2
// in units of inv_delta), bsums and sums as per-cell workspaces, guard words guard_stride apart.
int coarse_cheb_batch_launch(const BatchCell* d_cells, const BatchCell* cells, int n_cells, long long nodes,
                             const float* lam, const float* mu, const float* b, const float* invd, float* x,
                             const char* bsums, const double* inv_theta, const double* inv_delta, const double* c1,
                             const double* c2, int steps, char* sums, void* exchange, const int* guard,
                             int guard_stride, cudaStream_t s);

}  // namespace phastb
