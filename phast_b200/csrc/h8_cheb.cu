// The coarsest multigrid level's Chebyshev solve in one cooperative launch (FP32).
//
// A block owns a brick of nodes for all steps: direction with a one-node halo, iterate, residual, inverse diagonal
// and the moduli of its elements stay in shared memory, and a step sends only the new direction on the brick's rim
// to the neighbouring bricks, one tagged 16-byte word per node (grid_sync.cuh's idea; there is no grid-wide sum).
// What bounds it: latency, a march of two element layers and one exchange through L2 per step.  On 16^3 (the
// coarsest level of a 64^3 cell) five steps took 25.3 us as launches of their own, with the gaps 28; here 19.8.  The
// cells' mixed solves, before and after: 24^3 5.6 / 5.2 ms, 64^3 14.2 / 13.7, 96^3 37.3 / 35.2, 160^3 214 / 210.
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
  Tagged* words;  // [2][n_red]
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

// A node's three values and the step they belong to in one 16-byte word.
__device__ __forceinline__ void st_node(Tagged* p, T x, T y, T z, unsigned tag) {
  st_tagged(p, __hiloint2double(__float_as_int(y), __float_as_int(x)),
            ((unsigned long long)tag << 32) | (unsigned)__float_as_int(z));
}
// Waits (bounded) for the word of step `tag`; false: gave up, or another wait of the grid has.
__device__ __forceinline__ bool wait_node(const Tagged* p, unsigned tag, T (&v)[3], unsigned* err) {
  Tagged t = ld_tagged(p);
  if ((unsigned)(t.tag >> 32) != tag) {
    const unsigned long long t0 = grid_clock_ns();
    for (unsigned i = 1;; ++i) {
      t = ld_tagged(p);
      if ((unsigned)(t.tag >> 32) == tag) break;
      if ((i & 255u) == 0u && (*reinterpret_cast<volatile unsigned*>(err) != 0u || i >= kGridPolls ||
                               grid_clock_ns() - t0 > kGridLimitNs)) {
        atomicExch(err, 1u);
        return false;
      }
    }
  }
  v[0] = __int_as_float(__double2loint(t.v));
  v[1] = __int_as_float(__double2hiint(t.v));
  v[2] = __int_as_float((int)(unsigned)t.tag);
  return true;
}

template <int NS>
__global__ void __launch_bounds__(NS* TPS, 1) h8_cheb_kernel(ChebArgs a) {
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
  const int txy = blockIdx.x % a.tiles_xy, bz = blockIdx.x / a.tiles_xy;
  const int i0 = (txy % a.tiles_x) * OX, j0 = (txy / a.tiles_x) * OY, k0 = bz * NS * kz;
  const int nk = min(NS * kz, g.rz - k0);                      // node layers of the block
  const int wx = min(OX, g.rx - i0), wy = min(OY, g.ry - j0);  // owned nodes per axis
  const size_t plane_n = (size_t)g.rx * g.ry, plane_e = (size_t)g.nx * g.ny;
  const unsigned epoch = a.epoch[blockIdx.x];  // the same in every block: each launch moves all of them on
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
    Tagged* words = a.words + (size_t)(it & 1) * g.n_red;
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
  double acc[3] = {0.0, 0.0, 0.0};
  if (owner) {
    for (int l = 0; l < K; ++l) {
      const size_t n3 = 3 * (plane_n * (kb + l) + no);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        // a lost wait: make the result unusable (every solver reports a non-finite value)
        const T v = s_lost ? T(NAN) : XS[c * own_n + o0 + l * OXY];
        a.x[n3 + c] = v;
        acc[c] += double(v);
      }
    }
  }
  if (tid == 0) a.epoch[blockIdx.x] = epoch + (unsigned)a.steps;
  if (a.ws.counter) reduce_multi<3>(acc, a.ws);
}

template <int NS>
int launch(const ChebArgs& a0, int grid, cudaStream_t s) {
  ChebArgs a = a0;
  void* args[] = {&a};
  const size_t bytes = ChebLayout<NS>(a.kz).total;
  if (cudaFuncSetAttribute(h8_cheb_kernel<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)ChebLayout<NS>(kMaxDepth).total) != cudaSuccess ||
      cudaLaunchCooperativeKernel((const void*)h8_cheb_kernel<NS>, dim3(grid), dim3(NS * TPS), args, bytes, s) !=
          cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  note_launch();
  return PHASTB_OK;
}

}  // namespace

size_t coarse_cheb_bytes(const VoxGeom& g) {
  return align_up(2 * sizeof(Tagged) * (size_t)g.n_red) + align_up(sizeof(unsigned) * (kGridBlocks + 1));
}

int coarse_cheb_reset(const VoxGeom& g, void* exchange, cudaStream_t s) {
  return cuda_status(cudaMemsetAsync(exchange, 0, coarse_cheb_bytes(g), s));
}

int coarse_cheb_launch(const VoxGeom& g, const float* lam, const float* mu, const float* b, const float* invd, float* x,
                       const double* bsums, double inv_theta, const double* c1, const double* c2, int steps,
                       const RedWs* sums, void* exchange, const int* guard, cudaStream_t s) {
  int dev = 0, sms = 0, coop = 0;
  if (steps < 1 || steps > kChebMaxSteps || !persistent_pcg_enabled()) return PHASTB_UNSUPPORTED;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  ChebArgs a;
  std::memset(&a, 0, sizeof(a));
  a.tiles_x = (g.rx + OX - 1) / OX;
  a.tiles_xy = a.tiles_x * ((g.ry + OY - 1) / OY);
  const int blocks = std::min(sms, kGridBlocks);
  if (!coop || a.tiles_xy > blocks) return PHASTB_UNSUPPORTED;
  // as many slabs as there are SMs for; a slab's layers go to sub-bricks first, then to their depth
  const int slabs = std::min(blocks / a.tiles_xy, g.rz), layers = (g.rz + slabs - 1) / slabs;
  const int ns = layers <= 1 ? 1 : (layers <= 2 ? 2 : 4);
  a.kz = (layers + ns - 1) / ns;
  if (a.kz > kMaxDepth) return PHASTB_UNSUPPORTED;
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
  a.epoch = reinterpret_cast<unsigned*>(static_cast<char*>(exchange) + align_up(2 * sizeof(Tagged) * (size_t)g.n_red));
  a.err = a.epoch + kGridBlocks;
  a.guard = guard;
  const int grid = a.tiles_xy * ((g.rz + ns * a.kz - 1) / (ns * a.kz));
  return ns == 1 ? launch<1>(a, grid, s) : (ns == 2 ? launch<2>(a, grid, s) : launch<4>(a, grid, s));
}

}  // namespace phastb
