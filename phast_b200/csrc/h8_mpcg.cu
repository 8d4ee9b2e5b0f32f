// The FP64 mechanics CG of a small voxel cell with its state on the SMs (one cooperative launch per solve).
//
// As in the damage CG (h8_dpcg.cu), a block owns a brick of nodes for the whole solve: the direction p with a
// one-node halo, the damage field that g(d) is formed from, the iterate, residual, inverse diagonal and A p of the
// owned nodes live in shared memory, and per iteration only the neighbours' z on the brick's rim (tagged words) and
// the two reductions cross the chip (grid_sync.cuh).  What bounds it: the latency of the march, with eight warps of
// up to 255 registers per SM, and the two waits on the grid.  As separate launches (action 10 us, update 7, direction
// 2, and the gaps) a 32^3 iteration took 21 us; here it takes 11.5.  Whole solves, separate launches and this: 12^3 3.9 / 2.0
// ms, 24^3 8.7 / 4.6, 32^3 12.8 / 7.6, 40^3 20.2 / 12.8, 48^3 28.0 / 20.9 (about the largest that fits).  Four
// sub-bricks of 96 threads at 168 registers: 8.0 ms at 32^3 and 35 at 48^3, from the spills and the repeated layers.
#include <algorithm>
#include <cstring>

#include "engine.cuh"
#include "grid_sync.cuh"
#include "h8_elastic.cuh"

namespace phastb {

bool persistent_pcg_enabled();

namespace {

using T = double;
constexpr int kT = 256, NS = 2, TPS = kT / NS;  // NS stacked sub-bricks of TPS threads each
constexpr int kMaxDepth = 10;                   // node layers per sub-brick: three mask bits each in one word
constexpr size_t kSmemMax = 220 * 1024;

struct MBrickArgs {
  VoxGeom g;
  int tiles_x, tiles_xy, kz, maxiter;  // kz: node layers per sub-brick
  int mode, pad_;
  const uint8_t* slot;
  TileK<T> k;
  const T *gq, *d;
  const uint8_t* mask;
  T *r, *x;
  const T *p, *inv_diag;
  Tagged* z;  // rim values by degree of freedom
  Tagged* slots;
  unsigned* err;
  PcgState* st;
};

template <int OX, int OY>
struct MBrickLayout {
  static constexpr int EX = OX + 1, EXY = EX * (OY + 1), NTX = OX + 2, PL = NTX * (OY + 2), OXY = OX * OY;
  static_assert(EXY <= TPS, "one element per thread of a sub-brick");
  size_t p, d, hv, own, fc, hn, hb, sl, total;  // offsets in bytes
  __host__ __device__ explicit MBrickLayout(int kz) {
    const size_t planes = (size_t)NS * kz + 2, w = sizeof(T);
    const size_t halo = planes * PL - (size_t)NS * kz * OXY;  // the most halo nodes a block has
    size_t o = 0;
    p = o;
    o += 3 * planes * PL * w;
    d = o;
    o += planes * PL * w;
    hv = o;
    o += 3 * halo * w;
    own = o;
    o += 12 * (size_t)NS * kz * OXY * w;  // x, r, 1 / diag, A p
    fc = o;
    o += (size_t)NS * 2 * 12 * EXY * w;
    hn = o;
    o += halo * sizeof(int);
    hb = o;
    o += halo * sizeof(int);
    sl = o;
    o += (size_t)NS * (kz + 1) * EXY;
    total = (o + 15) / 16 * 16;
  }
};

template <int COEF, int OX, int OY>
__global__ void __launch_bounds__(kT, 1) h8_mpcg_kernel(MBrickArgs a, VoxMat<T> m) {
  using L = MBrickLayout<OX, OY>;
  constexpr int EX = L::EX, EXY = L::EXY, NTX = L::NTX, PL = L::PL, OXY = L::OXY;
  extern __shared__ __align__(16) unsigned char smem[];
  const VoxGeom& g = a.g;
  const int tid = threadIdx.x;
  const int kz = a.kz;
  const L lay(kz);
  const int PP = (NS * kz + 2) * PL;  // one component of P
  T* P = reinterpret_cast<T*>(smem + lay.p);
  T* D = reinterpret_cast<T*>(smem + lay.d);
  // the block's halo nodes: position in P, node, and the z they sent
  T* HV = reinterpret_cast<T*>(smem + lay.hv);
  int *HN = reinterpret_cast<int*>(smem + lay.hn), *HB = reinterpret_cast<int*>(smem + lay.hb);
  __shared__ int s_halo;
  const int own_n = NS * kz * OXY;
  T* XS = reinterpret_cast<T*>(smem + lay.own);  // [3][own_n], and so on
  T *RS = XS + 3 * own_n, *DS = RS + 3 * own_n, *AS = DS + 3 * own_n;
  const int sub = tid / TPS, t = tid - sub * TPS;
  T* FC = reinterpret_cast<T*>(smem + lay.fc) + (size_t)sub * 24 * EXY;
  uint8_t* SL = smem + lay.sl + (size_t)sub * (kz + 1) * EXY;
  const int txy = blockIdx.x % a.tiles_xy, bz = blockIdx.x / a.tiles_xy;
  const int i0 = (txy % a.tiles_x) * OX, j0 = (txy / a.tiles_x) * OY, k0 = bz * NS * kz;
  const int nk = min(NS * kz, g.rz - k0);                      // node layers of the block
  const int wx = min(OX, g.rx - i0), wy = min(OY, g.ry - j0);  // owned nodes per axis
  const size_t plane_n = (size_t)g.rx * g.ry, plane_e = (size_t)g.nx * g.ny;
  const bool use_d = a.d != nullptr && a.gq == nullptr;
  PcgState S = *a.st;
  GridSync gs{a.slots, a.err, 0ull};
  __shared__ int s_lost;  // a halo wait of this block ran out
  if (tid == 0) s_lost = s_halo = 0;
  auto fail = [&] {  // a wait ran out
    if (tid == 0) atomicExch(&a.st->grid_error, 1);
  };
  // box position b (plane, row, column): its node, or -1 (outside the grid or beyond the layer next to the
  // owned nodes); owned: a node of this block
  auto box_node = [&](int b, bool& owned) -> int {
    const int plane = b / PL, r = b - plane * PL, row = r / NTX, col = r - row * NTX;
    owned = plane >= 1 && plane <= nk && row >= 1 && row <= wy && col >= 1 && col <= wx;
    if (plane > nk + 1 || row > wy + 1 || col > wx + 1) return -1;
    const int i = wrap_node(i0 - 1 + col, g.nx, g.rx, g.px), j = wrap_node(j0 - 1 + row, g.ny, g.ry, g.py);
    const int k = wrap_node(k0 - 1 + plane, g.nz, g.rz, g.pz);
    return i >= 0 && j >= 0 && k >= 0 ? i + g.rx * (j + g.ry * k) : -1;
  };
  // this thread's owned column: nodes (ni, nj, kb + kk), kk < K
  const int ni = t % OX, nj = t / OX;
  const int K = max(0, min(kz, nk - sub * kz));
  const bool owner = t < OXY && ni < wx && nj < wy;
  const int no = (i0 + ni) + g.rx * (j0 + nj);
  const int kb = k0 + sub * kz;  // first node layer of the sub-brick
  const bool rim_xy = ni == 0 || nj == 0 || ni == wx - 1 || nj == wy - 1;
  auto rim = [&](int kk) { return rim_xy || (sub == 0 && kk == 0) || sub * kz + kk == nk - 1; };
  // the column in the owned arrays (stride OXY per layer) and in P (stride PL)
  const int o0 = sub * kz * OXY + t, p0 = (sub * kz + 1) * PL + (nj + 1) * NTX + ni + 1;
  __syncthreads();
  for (int b = tid; b < PP; b += kT) {
    bool owned;
    const int n = box_node(b, owned);
    D[b] = n >= 0 && use_d ? a.d[n] : T(0);
#pragma unroll
    for (int c = 0; c < 3; ++c) P[c * PP + b] = n >= 0 ? a.p[3 * (size_t)n + c] : T(0);
    if (n >= 0 && !owned) {
      const int e = atomicAdd(&s_halo, 1);  // (any order: every entry is a node of its own)
      HN[e] = n;
      HB[e] = b;
    }
  }
  unsigned masked = 0;  // masked components of the column, three bits per layer
  if (owner) {
    for (int kk = 0; kk < K; ++kk) {
      const size_t n3 = 3 * (plane_n * (kb + kk) + no);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int o = c * own_n + o0 + kk * OXY;
        XS[o] = a.x[n3 + c];
        RS[o] = a.r[n3 + c];
        DS[o] = a.inv_diag ? a.inv_diag[n3 + c] : T(1);
        if (a.mask && a.mask[n3 + c]) masked |= 1u << (3 * kk + c);
      }
    }
  }
  // this thread's element column: element layers kb - 1 .. kb - 1 + K
  const int ea = t % EX, eb = t / EX;
  int eo = -1;
  if (t < EXY && ea <= wx && eb <= wy) {
    const int gi = wrap_elem(i0 - 1 + ea, g.nx, g.px), gj = wrap_elem(j0 - 1 + eb, g.ny, g.py);
    if (gi >= 0 && gj >= 0) eo = gi + g.nx * gj;
  }
  for (int kk = 0; kk <= kz; ++kk) {
    const int gk = kk <= K ? wrap_elem(kb - 1 + kk, g.nz, g.pz) : -1;
    if (t < EXY) SL[kk * EXY + t] = eo >= 0 && gk >= 0 ? a.slot[plane_e * gk + eo] : 0;
  }
  // elements whose corner forces meet at the owned node
  const int e11 = (ni + 1) + EX * (nj + 1), e01 = ni + EX * (nj + 1), e10 = (ni + 1) + EX * nj, e00 = ni + EX * nj;
  const int pe = sub * kz * PL + eb * NTX + ea;
  const int gk0 = wrap_elem(kb - 1, g.nz, g.pz);
  const T w = T(g.w), kap = T(m.kappa), okap = T(1) - kap;
  auto load_face = [&](int b, Face<T>& f) {
    T v[4][3];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < 3; ++c) v[q][c] = P[c * PP + b + (q >> 1) * NTX + (q & 1)];
    elastic_face(v, f);
    if (use_d) damage_face(D[b], D[b + 1], D[b + NTX], D[b + NTX + 1], a.k, f);
  };
  __syncthreads();
  for (int it = 0; it < a.maxiter && S.active; ++it) {
    double v1[1] = {0.0};
    if (K > 0) {
      // ---- A p over the sub-brick
      Face<T> fl;
      if (t < EXY) load_face(pe, fl);
      FaceForce<T> pend;
#pragma unroll
      for (int c = 0; c < 3; ++c) pend.M[c] = pend.X[c] = pend.Y[c] = pend.XY[c] = T(0);
      int gk = gk0;
      T dot = T(0);
      for (int kk = 0; kk <= K; ++kk) {
        T* fc = FC + (kk & 1) * 12 * EXY;
        if (t < EXY) {
          Face<T> fu;
          load_face(pe + (kk + 1) * PL, fu);
          FaceForce<T> lo = pend;
#pragma unroll
          for (int c = 0; c < 3; ++c) pend.M[c] = pend.X[c] = pend.Y[c] = pend.XY[c] = T(0);
          if (eo >= 0 && gk >= 0) {
            const int sl = SL[kk * EXY + t];
            const T lw = COEF == kCoefIso ? m.lam[sl] * w : T(0), mw = COEF == kCoefIso ? m.mu[sl] * w : T(0);
            const T* ge = a.gq ? a.gq + 8 * (plane_e * gk + eo) : nullptr;
            T gv[4];
            auto half = [&](int qz) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                if (ge) {
                  gv[q] = __ldg(ge + 4 * qz + q);
                } else if (use_d) {
                  const T o = intact_at(fl, fu, a.k, qz, q);
                  gv[q] = okap * (o * o) + kap;
                } else {
                  gv[q] = T(1);
                }
              }
            };
            auto stress = [&](int q, const T(&ep)[6], T(&sg)[6]) {
              if constexpr (COEF == kCoefAniso) {
                voigt_stress(m, sl, ep, sg);
                const T gw = gv[q] * w;
#pragma unroll
                for (int i = 0; i < 6; ++i) sg[i] *= gw;
              } else {
                iso_stress(lw * gv[q], mw * gv[q], ep, sg);
              }
            };
            elastic_element<false>(fl, fu, a.k, (const T*)nullptr, half, stress, [](int, T, T, T) {}, lo, pend);
          }
          fl = fu;
          if (kk >= 1) corner_forces(lo, fc, EXY, t);
        }
        gk = gk + 1 < g.nz ? gk + 1 : (g.pz ? 0 : -1);
        if (kk >= 1) {  // (the first element layer only fills pend)
          // two corner buffers in turn: a buffer is written again after the next layer's barrier
          sub_barrier(1 + sub, TPS);
          if (owner) {
            const int o = o0 + (kk - 1) * OXY, q = p0 + (kk - 1) * PL;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              T v = node_force(fc, EXY, c, e11, e01, e10, e00);
              if (masked >> (3 * (kk - 1) + c) & 1u) v = T(0);
              AS[c * own_n + o] = v;
              dot += P[c * PP + q] * v;
            }
          }
        }
      }
      v1[0] = dot;
    }
    if (!grid_reduce<1, 0, kT>(v1, gs)) return fail();
    const double PAP = v1[0];
    // the state rules of pcg_update_dot_kernel (Jacobi / identity, not PCG_PERIODIC)
    S.iter += 1;
    if (!(isfinite(PAP) && PAP > 0.0)) {
      if (!isfinite(PAP)) S.nonfinite = 1;
      if (!(PAP > 0.0)) S.breakdown = 1;
      S.active = 0;
      break;
    }
    S.alpha = S.rz / PAP;
    S.steps += 1;
    const T al = T(S.alpha);
    double v2[2] = {0.0, 0.0};  // r . z, r . r
    if (owner) {
      for (int kk = 0; kk < K; ++kk) {
        const size_t n3 = 3 * (plane_n * (kb + kk) + no);
        const bool edge = rim(kk);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int o = c * own_n + o0 + kk * OXY;
          XS[o] = XS[o] + al * P[c * PP + p0 + kk * PL];
          const T r = RS[o] - al * AS[o];
          RS[o] = r;
          v2[1] += r * r;
          const T z = r * DS[o];
          v2[0] += r * z;
          if (edge) st_tagged(a.z + n3 + c, z, it + 1);
        }
      }
    }
    // the halo's z arrives beside the sums
    const int halo = 3 * s_halo;
    auto take_halo = [&](int i, int step) {
      constexpr int B = 4;  // polls in flight
      auto word = [&](int e) { return a.z + 3 * (size_t)HN[e / 3] + e % 3; };
      for (int e = i; e < halo; e += B * step) {
        Tagged q[B];
#pragma unroll
        for (int j = 0; j < B; ++j)
          if (e + j * step < halo) q[j] = ld_tagged(word(e + j * step));
#pragma unroll
        for (int j = 0; j < B; ++j) {
          const int f = e + j * step;
          if (f < halo) {
            if (q[j].tag != (unsigned long long)(it + 1) && !wait_tagged(word(f), it + 1, &q[j].v, a.err)) s_lost = 1;
            HV[f] = q[j].v;
          }
        }
      }
    };
    if (!grid_reduce<2, 0, kT>(v2, gs, take_halo) || s_lost) return fail();
    const double RZ = v2[0], RR = v2[1];
    if (!isfinite(RR) || !isfinite(RZ)) S.nonfinite = 1;
    S.rr = RR;
    if (!(RR > S.thr_sq)) {
      S.converged = 1;
      S.active = 0;
    } else {
      if (a.mode == PCG_STRICT && !(RZ > 0.0)) S.breakdown = 1;
      S.beta = (a.mode == PCG_STRICT) ? RZ / S.rz : ((S.rz > 0.0) ? RZ / S.rz : 0.0);
      S.rz = RZ;
    }
    if (S.breakdown || S.nonfinite) S.active = 0;
    if (!S.active) break;
    const T be = T(S.beta);
    for (int e = tid; e < halo; e += kT) {
      T& p = P[(e % 3) * PP + HB[e / 3]];
      p = HV[e] + be * p;
    }
    if (owner) {
      for (int kk = 0; kk < K; ++kk) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int o = c * own_n + o0 + kk * OXY, q = c * PP + p0 + kk * PL;
          P[q] = RS[o] * DS[o] + be * P[q];
        }
      }
    }
    __syncthreads();
  }
  if (owner) {
    for (int kk = 0; kk < K; ++kk) {
      const size_t n3 = 3 * (plane_n * (kb + kk) + no);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        a.x[n3 + c] = XS[c * own_n + o0 + kk * OXY];
        a.r[n3 + c] = RS[c * own_n + o0 + kk * OXY];
      }
    }
  }
  if (blockIdx.x == 0 && tid == 0) store_pcg_state(a.st, S);
}

// Bricks of one shape: the least depth that covers the grid with at most `blocks` blocks; 0 when none fits.
template <int OX, int OY>
int brick_depth(const VoxGeom& g, int blocks) {
  const int txy = ((g.rx + OX - 1) / OX) * ((g.ry + OY - 1) / OY);
  if (txy > blocks) return 0;
  const int slabs = std::min(blocks / txy, g.rz);
  const int layers = (g.rz + slabs - 1) / slabs, kz = (layers + NS - 1) / NS;
  return kz <= kMaxDepth && MBrickLayout<OX, OY>(kz).total <= kSmemMax ? kz : 0;
}

template <int COEF, int OX, int OY>
int launch_bricks(MBrickArgs a, const VoxMat<T>& m, int kz, cudaStream_t s) {
  const VoxGeom& g = a.g;
  a.tiles_x = (g.rx + OX - 1) / OX;
  a.tiles_xy = a.tiles_x * ((g.ry + OY - 1) / OY);
  a.kz = kz;
  const int grid = a.tiles_xy * ((g.rz + NS * kz - 1) / (NS * kz));
  auto kern = h8_mpcg_kernel<COEF, OX, OY>;
  VoxMat<T> mm = m;
  void* args[] = {&a, &mm};
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) != cudaSuccess ||
      cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kT), args, MBrickLayout<OX, OY>(kz).total, s) !=
          cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  note_launch();
  return PHASTB_OK;
}

}  // namespace

int h8_mech_brick_pcg(const VoxGeom& g, const VoxMat<double>& m, const uint8_t* slot, const double* gq,
                      const double* d, const uint8_t* mask, const PcgWs<double>& w, void* tagged,
                      size_t tagged_bytes, double* x, const double* inv_diag, int maxiter, int mode, cudaStream_t s) {
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  const size_t words = 3 * (size_t)g.n_red;
  if (!coop || mode == PCG_PERIODIC || !mask || tagged_bytes < words * sizeof(Tagged) ||
      !aligned16(tagged) || !aligned16(w.part) || !persistent_pcg_enabled())
    return PHASTB_UNSUPPORTED;
  const int blocks = std::min(sms, kGridBlocks);
  // the march is kz + 1 layers whatever the shape, so the least depth wins
  const int depth[2] = {brick_depth<14, 7>(g, blocks), brick_depth<8, 8>(g, blocks)};
  const int best = depth[0] && (!depth[1] || depth[0] < depth[1]) ? 0 : 1;
  if (!depth[best]) return PHASTB_UNSUPPORTED;
  MBrickArgs a;
  std::memset(&a, 0, sizeof(a));
  a.g = g;
  a.maxiter = maxiter;
  a.mode = mode;
  a.slot = slot;
  a.k = tile_args<T>(g, 0).k;
  a.gq = gq;
  a.d = d;
  a.mask = mask;
  a.r = w.r;
  a.x = x;
  a.p = w.p;
  a.inv_diag = inv_diag;
  a.z = static_cast<Tagged*>(tagged);
  a.slots = reinterpret_cast<Tagged*>(w.part);
  a.err = w.counter;
  a.st = w.st;
  int st = cuda_status(cudaMemsetAsync(w.part, 0, grid_slot_bytes(), s));
  if (!st) st = cuda_status(cudaMemsetAsync(w.counter, 0, 4 * sizeof(unsigned), s));
  if (!st) st = cuda_status(cudaMemsetAsync(tagged, 0, words * sizeof(Tagged), s));
  if (st) return st;
  if (m.iso)
    return best == 0 ? launch_bricks<kCoefIso, 14, 7>(a, m, depth[0], s)
                     : launch_bricks<kCoefIso, 8, 8>(a, m, depth[1], s);
  return best == 0 ? launch_bricks<kCoefAniso, 14, 7>(a, m, depth[0], s)
                   : launch_bricks<kCoefAniso, 8, 8>(a, m, depth[1], s);
}

}  // namespace phastb
