// The coarsest multigrid level's Chebyshev solve in one cooperative launch (FP32).
//
// A block owns a brick of nodes for all steps: direction with a one-node halo, iterate, residual, inverse diagonal
// and the moduli of its elements stay in shared memory, and a step sends only the new direction on the brick's rim
// to the neighbouring bricks, one tagged 16-byte word per node (grid_sync.cuh's idea; there is no grid-wide sum).
// What bounds it: latency, a march of two element layers and one exchange through L2 per step.  On 16^3 (the
// coarsest level of a 64^3 cell) five steps took 25.3 us as launches of their own, with the gaps 28; here 19.8.  The
// cells' mixed solves, before and after: 24^3 5.6 / 5.2 ms, 64^3 14.2 / 13.7, 96^3 37.3 / 35.2, 160^3 214 / 210.
// A batch's coarsest levels share one launch, several bricks per SM: 8^3 to 16^3 together 24 us instead of 50.
#include <algorithm>
#include <cstring>

#include "grid_sync.cuh"
#include "h8_elastic.cuh"
#include "h8_cheb.cuh"

namespace phastb {

bool persistent_pcg_enabled();

namespace {

using T = float;
constexpr int OX = 8, OY = 8, EX = OX + 1, EXY = EX * (OY + 1), NTX = OX + 2, PL = NTX * (OY + 2), OXY = OX * OY;
constexpr int TPS = (EXY + 31) / 32 * 32;  // threads of a sub-brick
constexpr int kMaxDepth = 2;               // node layers per sub-brick

struct ChebArgs {
  VoxGeom g;
  int tiles_x, tiles_xy, kz, steps;
  TileK<T> k;
  T inv_theta, c1[kChebMaxSteps], c2[kChebMaxSteps];
  const T *lam, *mu, *b, *invd;
  T* x;
  const double* bsums;
  RedWs ws;       // component sums of x at ws.out (counter null: none)
  Tagged* words;  // one per node, and again word_stride further on
  long long word_stride;
  unsigned *epoch, *err;  // epoch: one word per brick
  const int* guard;
};

// Several cells of a packed batch (BatchCell): the arrays hold the cells' vectors one after another, factors and
// reductions are per cell.
struct ChebBatchArgs {
  const BatchCell* cells;
  int first, n_cells;  // the cells of this launch
  int kz, steps, guard_stride, pad_;
  double c1[kChebMaxSteps], c2[kChebMaxSteps];  // c2: in units of inv_delta
  const double *inv_theta, *inv_delta;
  const T *lam, *mu, *b, *invd;
  T* x;
  const char* bsums;  // per-cell workspaces (sums of b in, sums of x out)
  char* sums;
  Tagged* words;
  long long word_stride;
  unsigned *epoch, *err;
  const int* guard;
};

template <int NS>
struct ChebLayout {
  size_t p, own, fc, q, hn, hb, total;
  __host__ __device__ explicit ChebLayout(int kz) {
    const size_t planes = (size_t)NS * kz + 2, halo = planes * PL - (size_t)NS * kz * OXY;
    size_t o = 0;
    p = o;
    o += 3 * planes * PL * sizeof(T);
    own = o;
    o += 12 * (size_t)NS * kz * OXY * sizeof(T);  // x, res, 1 / diag, new direction
    fc = o;
    o += (size_t)NS * 24 * EXY * sizeof(T);
    q = o;
    o += (size_t)NS * (kz + 1) * 16 * EXY * sizeof(T);
    hn = o;
    o += halo * sizeof(int);
    hb = o;
    o += halo * sizeof(int);
    total = o;
  }
};

// Brick vb of the vgrid bricks of one grid.
template <int NS, bool LAYERS>
__device__ __forceinline__ void cheb_body(const ChebArgs& a, int vb, int vgrid) {
  if (a.guard && *a.guard == 0) return;
  constexpr int kT = NS * TPS;
  extern __shared__ __align__(16) unsigned char smem[];
  const VoxGeom& g = a.g;
  const int kz = a.kz, tid = threadIdx.x, sub = tid / TPS, t = tid - sub * TPS;
  const ChebLayout<NS> lay(kz);
  const int PP = (NS * kz + 2) * PL, own_n = NS * kz * OXY;
  T* P = reinterpret_cast<T*>(smem + lay.p);  // [3][planes][PL]
  T* XS = reinterpret_cast<T*>(smem + lay.own);
  T *RS = XS + 3 * own_n, *DS = RS + 3 * own_n, *DN = DS + 3 * own_n;  // [3][own_n] each
  T* FC = reinterpret_cast<T*>(smem + lay.fc) + (size_t)sub * 24 * EXY;
  T* Q = reinterpret_cast<T*>(smem + lay.q) + (size_t)sub * (kz + 1) * 16 * EXY;
  int *HN = reinterpret_cast<int*>(smem + lay.hn), *HB = reinterpret_cast<int*>(smem + lay.hb);
  __shared__ int s_halo, s_lost;
  const int txy = vb % a.tiles_xy, bz = vb / a.tiles_xy;
  const int i0 = (txy % a.tiles_x) * OX, j0 = (txy / a.tiles_x) * OY, k0 = bz * NS * kz;
  const int nk = min(NS * kz, g.rz - k0);                      // node layers of the block
  const int wx = min(OX, g.rx - i0), wy = min(OY, g.ry - j0);  // owned nodes per axis
  const size_t plane_n = (size_t)g.rx * g.ry, plane_e = (size_t)g.nx * g.ny;
  const unsigned epoch = a.epoch[vb];  // the same in every brick of the grid: each launch moves all of them on
  if (tid == 0) s_halo = s_lost = 0;
  __syncthreads();
  T mean[3] = {T(0), T(0), T(0)};
  if (a.bsums) {
#pragma unroll
    for (int c = 0; c < 3; ++c) mean[c] = T(a.bsums[c] / g.n_red);
  }
  // first step from x = 0: the direction everywhere in the box
  for (int b = tid; b < PP; b += kT) {
    const int plane = b / PL, r = b - plane * PL, row = r / NTX, col = r - row * NTX;
    const bool owned = plane >= 1 && plane <= nk && row >= 1 && row <= wy && col >= 1 && col <= wx;
    int n = -1;
    if (plane <= nk + 1 && row <= wy + 1 && col <= wx + 1) {
      const int i = wrap_node(i0 - 1 + col, g.nx, g.rx, g.px), j = wrap_node(j0 - 1 + row, g.ny, g.ry, g.py);
      const int k = wrap_node(k0 - 1 + plane, g.nz, g.rz, g.pz);
      if (i >= 0 && j >= 0 && k >= 0) n = i + g.rx * (j + g.ry * k);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      T d = T(0);
      if (n >= 0) {
        T bi = a.b[3 * (size_t)n + c];
        if (a.bsums) bi -= mean[c];
        const T iv = a.invd[3 * (size_t)n + c];
        d = iv * bi * a.inv_theta;
        if (owned) {
          const int o = c * own_n + (plane - 1) * OXY + (row - 1) * OX + col - 1;
          RS[o] = bi;
          DS[o] = iv;
          XS[o] = d;
        }
      }
      P[c * PP + b] = d;
    }
    if (n >= 0 && !owned) {
      const int e = atomicAdd(&s_halo, 1);  // (any order: every entry is a node of its own)
      HN[e] = n;
      HB[e] = b;
    }
  }
  // this thread's owned column and element column (see h8_dpcg_kernel)
  const int ni = t % OX, nj = t / OX, K = max(0, min(kz, nk - sub * kz)), kb = k0 + sub * kz;
  const bool owner = t < OXY && ni < wx && nj < wy;
  const int no = (i0 + ni) + g.rx * (j0 + nj);
  const bool rim_xy = ni == 0 || nj == 0 || ni == wx - 1 || nj == wy - 1;
  const int o0 = sub * kz * OXY + t, p0 = (sub * kz + 1) * PL + (nj + 1) * NTX + ni + 1;
  const int ea = t % EX, eb = t / EX, pe = sub * kz * PL + eb * NTX + ea;
  int eo = -1;
  if (t < EXY && ea <= wx && eb <= wy) {
    const int gi = wrap_elem(i0 - 1 + ea, g.nx, g.px), gj = wrap_elem(j0 - 1 + eb, g.ny, g.py);
    if (gi >= 0 && gj >= 0) eo = gi + g.nx * gj;
  }
  unsigned live = 0;  // bit kk: element layer kb - 1 + kk of the column exists
  for (int kk = 0; kk <= K; ++kk) {
    const int gk = wrap_elem(kb - 1 + kk, g.nz, g.pz);
    if (K > 0 && eo >= 0 && gk >= 0) {
      live |= 1u << kk;
      const size_t e8 = 8 * (plane_e * gk + eo);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        Q[(kk * 16 + q) * EXY + t] = __ldg(a.lam + e8 + q);
        Q[(kk * 16 + 8 + q) * EXY + t] = __ldg(a.mu + e8 + q);
      }
    }
  }
  const int e11 = (ni + 1) + EX * (nj + 1), e01 = ni + EX * (nj + 1), e10 = (ni + 1) + EX * nj, e00 = ni + EX * nj;
  const T w = T(g.w);
  auto load_face = [&](int b, Face<T>& f) {
    T v[4][3];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < 3; ++c) v[q][c] = P[c * PP + b + (q >> 1) * NTX + (q & 1)];
    elastic_face(v, f);
  };
  __syncthreads();
  for (int it = 0; it < a.steps; ++it) {
    const bool last = it + 1 == a.steps;
    const unsigned tag = epoch + 1u + (unsigned)it;
    // a word is written again two steps later, when its readers have sent what they formed from it
    Tagged* words = a.words + (it & 1 ? a.word_stride : 0);
    const T c1 = a.c1[it], c2 = a.c2[it];
    if (K > 0) {
      Face<T> fl;
      if (t < EXY) load_face(pe, fl);
      FaceForce<T> pend;
#pragma unroll
      for (int c = 0; c < 3; ++c) pend.M[c] = pend.X[c] = pend.Y[c] = pend.XY[c] = T(0);
      for (int kk = 0; kk <= K; ++kk) {
        T* fc = FC + (kk & 1) * 12 * EXY;
        if (t < EXY) {
          Face<T> fu;
          load_face(pe + (kk + 1) * PL, fu);
          FaceForce<T> lo = pend;
#pragma unroll
          for (int c = 0; c < 3; ++c) pend.M[c] = pend.X[c] = pend.Y[c] = pend.XY[c] = T(0);
          if (live >> kk & 1u) {
            T lm[8];
            auto half = [&](int qz) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                lm[q] = Q[(kk * 16 + 4 * qz + q) * EXY + t];
                lm[4 + q] = Q[(kk * 16 + 8 + 4 * qz + q) * EXY + t];
              }
            };
            auto stress = [&](int q, const T(&ep)[6], T(&sg)[6]) { iso_stress(lm[q] * w, lm[4 + q] * w, ep, sg); };
            elastic_element<false>(fl, fu, a.k, (const T*)nullptr, half, stress, [](int, T, T, T) {}, lo, pend);
          }
          fl = fu;
          if (kk >= 1) corner_forces(lo, fc, EXY, t);
        }
        if (kk >= 1) {  // (the first element layer only fills pend)
          sub_barrier(1 + sub, TPS);
          if (owner) {
            const int l = kk - 1, o = o0 + l * OXY, q = p0 + l * PL;
            T dn[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const T r = RS[c * own_n + o] - node_force(fc, EXY, c, e11, e01, e10, e00);
              RS[c * own_n + o] = r;
              dn[c] = c1 * P[c * PP + q] + c2 * DS[c * own_n + o] * r;
              DN[c * own_n + o] = dn[c];
              XS[c * own_n + o] = XS[c * own_n + o] + dn[c];
            }
            if (!last && (rim_xy || (sub == 0 && l == 0) || sub * kz + l == nk - 1))
              st_node(words + plane_n * (kb + l) + no, dn[0], dn[1], dn[2], tag);
          }
        }
      }
    }
    if (last) break;
    __syncthreads();  // every element has read the direction
    if (owner) {
      for (int l = 0; l < K; ++l) {
#pragma unroll
        for (int c = 0; c < 3; ++c) P[c * PP + p0 + l * PL] = DN[c * own_n + o0 + l * OXY];
      }
    }
    for (int e = tid; e < s_halo; e += kT) {
      T v[3];
      if (!wait_node(words + HN[e], tag, v, a.err)) {
        s_lost = 1;
        break;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) P[c * PP + HB[e]] = v[c];
    }
    __syncthreads();
    if (s_lost) break;
  }
  // The sums of x per block, or in a batch (LAYERS) per node layer of an OX x OY tile whatever the bricks' depth: a
  // batched cell's bits must not depend on the cells that share its launch.  (Per layer also for a single cell: 64^3
  // solves 0.6 to 1.1 % slower.)
  const bool sums = a.ws.counter != nullptr;
  double acc[3] = {0.0, 0.0, 0.0};
  __shared__ double sh[LAYERS ? NS * kMaxDepth * 3 * (OXY / 32) : 32 * 3];
  for (int l = 0; l < K; ++l) {
    const size_t n3 = 3 * (plane_n * (kb + l) + no);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      T v = T(0);
      if (owner) {
        // a lost wait: make the result unusable (every solver reports a non-finite value)
        v = s_lost ? T(NAN) : XS[c * own_n + o0 + l * OXY];
        a.x[n3 + c] = v;
      }
      if constexpr (LAYERS) {
        if (sums && t < OXY) {
          const double w = warp_sum(double(v));
          if ((t & 31) == 0) sh[(3 * (sub * kz + l) + c) * (OXY / 32) + (t >> 5)] = w;
        }
      } else {
        acc[c] += double(v);
      }
    }
  }
  if (tid == 0) a.epoch[vb] = epoch + (unsigned)a.steps;
  if (!sums) return;
  int parts = vgrid;
  if constexpr (LAYERS) {
    parts = a.tiles_xy * g.rz;
    __syncthreads();
    if (tid < 3 * nk) {
      const int l = tid / 3, c = tid - 3 * l;
      double w = 0.0;
#pragma unroll
      for (int i = 0; i < OXY / 32; ++i) w += sh[tid * (OXY / 32) + i];
      a.ws.part[c * kMaxPartials + (size_t)(k0 + l) * a.tiles_xy + txy] = w;
    }
  } else {
    block_sum_multi<3>(acc, sh);
    if (tid == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) a.ws.part[c * kMaxPartials + vb] = acc[c];
    }
  }
  if (arrive_last_n(a.ws.counter, vgrid)) {
    if constexpr (LAYERS) {
      if (tid < 96) {  // a warp per component
        double w = 0.0;
        for (int i = tid & 31; i < parts; i += 32) w += __ldcg(a.ws.part + (tid >> 5) * kMaxPartials + i);
        w = warp_sum(w);
        if ((tid & 31) == 0) a.ws.out[tid >> 5] = w;
      }
    } else {
      double f[3];
      fold_sum_multi<3>(a.ws.part, kMaxPartials, parts, f, sh);
      if (tid == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a.ws.out[c] = f[c];
      }
    }
    if (tid == 0) *a.ws.counter = 0u;
  }
}

template <int NS>
__global__ void __launch_bounds__(NS* TPS, 1) h8_cheb_kernel(ChebArgs a) {
  cheb_body<NS, false>(a, blockIdx.x, gridDim.x);
}

template <int NS>
__host__ __device__ __forceinline__ int cheb_blocks(const VoxGeom& g, int kz) {
  return ((g.rx + OX - 1) / OX) * ((g.ry + OY - 1) / OY) * ((g.rz + NS * kz - 1) / (NS * kz));
}

template <int NS>
__global__ void __launch_bounds__(NS* TPS, 1) h8_cheb_batch_kernel(ChebBatchArgs b) {
  __shared__ ChebArgs sa;
  __shared__ int s_vb, s_vgrid;
  if (threadIdx.x == 0) {
    int c = b.first, vb = blockIdx.x, n = cheb_blocks<NS>(b.cells[c].g, b.kz);
    while (vb >= n) {  // (the grid is the sum over the launch's cells)
      vb -= n;
      n = cheb_blocks<NS>(b.cells[++c].g, b.kz);
    }
    const BatchCell& cl = b.cells[c];
    sa.g = cl.g;
    sa.tiles_x = (cl.g.rx + OX - 1) / OX;
    sa.tiles_xy = sa.tiles_x * ((cl.g.ry + OY - 1) / OY);
    sa.kz = b.kz;
    sa.steps = b.steps;
    sa.k = cl.kf;
    sa.inv_theta = T(b.inv_theta[c]);
    for (int i = 0; i < b.steps; ++i) {
      sa.c1[i] = T(b.c1[i]);
      sa.c2[i] = T(b.c2[i] * b.inv_delta[c]);
    }
    sa.lam = b.lam + 8 * cl.elem_off;
    sa.mu = b.mu + 8 * cl.elem_off;
    sa.b = b.b + cl.mech_off;
    sa.invd = b.invd + cl.mech_off;
    sa.x = b.x + cl.mech_off;
    sa.bsums = b.bsums ? red_ws(const_cast<char*>(b.bsums) + (size_t)c * red_ws_bytes()).out : nullptr;
    sa.ws = red_ws(b.sums + (size_t)c * red_ws_bytes());
    sa.words = b.words + cl.node_off;
    sa.word_stride = b.word_stride;
    sa.epoch = b.epoch + cl.node_off;  // (a brick holds a node at least)
    sa.err = b.err;
    sa.guard = b.guard ? b.guard + (size_t)c * b.guard_stride : nullptr;
    s_vb = vb;
    s_vgrid = n;
  }
  __syncthreads();
  cheb_body<NS, true>(sa, s_vb, s_vgrid);
}

// Opt-in to the shared memory of every depth, and how many blocks of depth kz the device holds at once (0: none).
template <int NS, class Kernel>
int resident_blocks(Kernel kern, int kz) {
  int dev = 0, sms = 0, coop = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ChebLayout<NS>(kMaxDepth).total) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, NS * TPS, ChebLayout<NS>(kz).total) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return std::min(sms * per, kChebBlocks);
}

template <int NS, class Kernel, class Args>
int launch(Kernel kern, Args a, int grid, cudaStream_t s) {
  void* args[] = {&a};
  if (cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(NS * TPS), args, ChebLayout<NS>(a.kz).total, s) !=
      cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  note_launch();
  return PHASTB_OK;
}

// One grid with a block per SM at most: more SMs than that only lengthen the rim.
template <int NS>
int try_cell(ChebArgs& a, int kz, cudaStream_t s) {
  const int grid = cheb_blocks<NS>(a.g, kz);
  a.kz = kz;
  if (grid > kGridBlocks || grid > resident_blocks<NS>(h8_cheb_kernel<NS>, kz)) return PHASTB_UNSUPPORTED;
  return launch<NS>(h8_cheb_kernel<NS>, a, grid, s);
}

// All cells of a launch at once, several blocks per SM where they fit.
template <int NS>
int try_batch(ChebBatchArgs& a, const BatchCell* cells, int kz, cudaStream_t s) {
  long long grid = 0;
  for (int c = 0; c < a.n_cells; ++c) grid += cheb_blocks<NS>(cells[a.first + c].g, kz);
  a.kz = kz;
  if (grid > resident_blocks<NS>(h8_cheb_batch_kernel<NS>, kz)) return PHASTB_UNSUPPORTED;
  return launch<NS>(h8_cheb_batch_kernel<NS>, a, (int)grid, s);
}

}  // namespace

size_t coarse_cheb_bytes(long long nodes) {
  return align_up(2 * sizeof(Tagged) * (size_t)nodes) + align_up(sizeof(unsigned) * ((size_t)nodes + 1));
}

int coarse_cheb_reset(long long nodes, void* exchange, cudaStream_t s) {
  return cuda_status(cudaMemsetAsync(exchange, 0, coarse_cheb_bytes(nodes), s));
}

int coarse_cheb_launch(const VoxGeom& g, const float* lam, const float* mu, const float* b, const float* invd, float* x,
                       const double* bsums, double inv_theta, const double* c1, const double* c2, int steps,
                       const RedWs* sums, void* exchange, const int* guard, cudaStream_t s) {
  if (steps < 1 || steps > kChebMaxSteps || !aligned16(exchange) || !persistent_pcg_enabled()) return PHASTB_UNSUPPORTED;
  ChebArgs a;
  std::memset(&a, 0, sizeof(a));
  a.tiles_x = (g.rx + OX - 1) / OX;
  a.tiles_xy = a.tiles_x * ((g.ry + OY - 1) / OY);
  a.g = g;
  a.steps = steps;
  a.k = tile_args<T>(g, 1).k;
  a.inv_theta = T(inv_theta);
  for (int i = 0; i < steps; ++i) {
    a.c1[i] = T(c1[i]);
    a.c2[i] = T(c2[i]);
  }
  a.lam = lam;
  a.mu = mu;
  a.b = b;
  a.invd = invd;
  a.x = x;
  a.bsums = bsums;
  if (sums) a.ws = *sums;
  a.words = static_cast<Tagged*>(exchange);
  a.word_stride = g.n_red;
  a.epoch = reinterpret_cast<unsigned*>(static_cast<char*>(exchange) + align_up(2 * sizeof(Tagged) * (size_t)g.n_red));
  a.err = a.epoch + g.n_red;
  a.guard = guard;
  // the shallowest brick that needs no second block on an SM
  int st = try_cell<1>(a, 1, s);
  if (st == PHASTB_UNSUPPORTED) st = try_cell<2>(a, 1, s);
  if (st == PHASTB_UNSUPPORTED) st = try_cell<4>(a, 1, s);
  if (st == PHASTB_UNSUPPORTED) st = try_cell<4>(a, 2, s);
  return st;
}

int coarse_cheb_batch_launch(const BatchCell* d_cells, const BatchCell* cells, int n_cells, long long nodes,
                             const float* lam, const float* mu, const float* b, const float* invd, float* x,
                             const char* bsums, const double* inv_theta, const double* inv_delta, const double* c1,
                             const double* c2, int steps, char* sums, void* exchange, const int* guard,
                             int guard_stride, cudaStream_t s) {
  if (steps < 1 || steps > kChebMaxSteps || !aligned16(exchange) || !persistent_pcg_enabled())
    return PHASTB_UNSUPPORTED;
  ChebBatchArgs a;
  std::memset(&a, 0, sizeof(a));
  a.cells = d_cells;
  a.steps = steps;
  a.guard_stride = guard_stride;
  for (int i = 0; i < steps; ++i) {
    a.c1[i] = c1[i];
    a.c2[i] = c2[i];
  }
  a.inv_theta = inv_theta;
  a.inv_delta = inv_delta;
  a.lam = lam;
  a.mu = mu;
  a.b = b;
  a.invd = invd;
  a.x = x;
  a.bsums = bsums;
  a.sums = sums;
  a.words = static_cast<Tagged*>(exchange);
  a.word_stride = nodes;
  a.epoch = reinterpret_cast<unsigned*>(static_cast<char*>(exchange) + align_up(2 * sizeof(Tagged) * (size_t)nodes));
  a.err = a.epoch + nodes;
  a.guard = guard;
  // Every cell takes this form or none does, so that a cell's result does not depend on the others: as many cells per
  // launch as the deepest bricks allow, and 64 at most (a block finds its cell by counting), the rest in further
  // launches.  A plan's coarsest cells are small enough to fit alone.
  const int most = resident_blocks<4>(h8_cheb_batch_kernel<4>, kMaxDepth);
  for (int c = 0; c < n_cells; ++c)
    if (cheb_blocks<4>(cells[c].g, kMaxDepth) > most || cheb_blocks<1>(cells[c].g, 1) > kMaxPartials)
      return PHASTB_UNSUPPORTED;
  while (a.first < n_cells) {
    int blocks = 0;
    for (a.n_cells = 0; a.n_cells < 64 && a.first + a.n_cells < n_cells; ++a.n_cells) {
      blocks += cheb_blocks<4>(cells[a.first + a.n_cells].g, kMaxDepth);
      if (blocks > most) break;
    }
    int st = try_batch<1>(a, cells, 1, s);
    if (st == PHASTB_UNSUPPORTED) st = try_batch<2>(a, cells, 1, s);
    if (st == PHASTB_UNSUPPORTED) st = try_batch<4>(a, cells, 1, s);
    if (st == PHASTB_UNSUPPORTED) st = try_batch<4>(a, cells, 2, s);
    if (st) return st;
    a.first += a.n_cells;
  }
  return PHASTB_OK;
}

}  // namespace phastb
