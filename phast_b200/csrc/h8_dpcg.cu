// The damage CG of a voxel cell with its whole state on the SMs (one
// cooperative launch per solve; the larger cells run h8_damage_pcg_kernel).
//
// A block owns a brick of nodes and keeps it for the whole solve: the direction
// p with a one-node halo, the iterate, residual, inverse diagonal and A p of the
// owned nodes live in shared memory, and an iteration reads only the history H
// (streamed from L2 one element layer ahead) and the neighbours' z on the brick's
// rim, which travels as tagged words beside the dot products (grid_sync.cuh).
// NS groups of threads march NS stacked sub-bricks, so a block's march is kz + 1
// element layers long.  What bounds it: shared-memory bandwidth (60 wavefronts
// per warp and element layer, half of them H on its way through) with sixteen
// warps to hide the march's latency, and the two waits on the grid (1.6 us each).
// On the 64^3 cell an iteration takes 20 us; staging every layer and vector
// through L2 with a counter barrier took 31.
#include <algorithm>
#include <cstring>

#include "engine.cuh"
#include "grid_sync.cuh"
#include "h8_march.cuh"

namespace phastb {

bool persistent_pcg_enabled();

namespace {

constexpr int kT = 512;
constexpr size_t kSmemMax = 220 * 1024;

template <typename T>
struct BrickArgs {
  VoxGeom g;
  int tiles_x, tiles_xy, kz, maxiter;  // kz: node layers per sub-brick
  int mode, pad_;
  const uint8_t* slot;
  T gcw[PHASTB_MAX_SLOTS], k2[PHASTB_MAX_SLOTS];
  T chw;
  DElemK<T> ek;
  const T* H;
  const uint8_t* mask;
  T *r, *x;
  const T *p, *inv_diag;
  Tagged* z;  // rim values by node
  Tagged* slots;
  unsigned* err;
  PcgState* st;
};

template <typename T, int OX, int OY, int NS>
struct BrickLayout {
  static constexpr int TPS = kT / NS, EX = OX + 1, EXY = EX * (OY + 1), NTX = OX + 2, PL = NTX * (OY + 2),
                       OXY = OX * OY;
  static_assert(EXY <= TPS, "one element per thread of a sub-brick");
  static constexpr int kHChunks = kStageH * (int)sizeof(T) / 16;
  // offsets in bytes; the H staging first (16-byte aligned)
  size_t hs, p, hv, own, fc, hn, hb, sl, total;
  __host__ __device__ explicit BrickLayout(int kz) {
    const size_t planes = (size_t)NS * kz + 2, w = sizeof(T);
    size_t o = 0;
    hs = o;
    o += (size_t)NS * 2 * kHChunks * EXY * 16;
    p = o;
    o += planes * PL * w;
    const size_t halo = planes * PL - (size_t)NS * kz * OXY;  // the most halo nodes a block has
    hv = o;
    o += halo * w;
    own = o;
    o += 4 * (size_t)NS * kz * OXY * w;  // x, r, 1 / diag, A p
    fc = o;
    o += (size_t)NS * 2 * 4 * EXY * w;
    hn = o;
    o += halo * sizeof(int);
    hb = o;
    o += halo * sizeof(int);
    sl = o;
    o += (size_t)NS * (kz + 1) * EXY;
    total = (o + 15) / 16 * 16;
  }
};

template <typename T, int OX, int OY, int NS>
__global__ void __launch_bounds__(kT, 1) h8_dpcg_kernel(BrickArgs<T> a) {
  using L = BrickLayout<T, OX, OY, NS>;
  constexpr int TPS = L::TPS, EX = L::EX, EXY = L::EXY, NTX = L::NTX, PL = L::PL, OXY = L::OXY;
  extern __shared__ __align__(16) unsigned char smem[];
  const L lay(a.kz);
  const VoxGeom& g = a.g;
  const int kz = a.kz;
  T* P = reinterpret_cast<T*>(smem + lay.p);
  // the block's halo nodes: position in P, node, and the z they sent
  T* HV = reinterpret_cast<T*>(smem + lay.hv);
  int *HN = reinterpret_cast<int*>(smem + lay.hn), *HB = reinterpret_cast<int*>(smem + lay.hb);
  __shared__ int s_halo;
  const int own_n = NS * kz * OXY;
  T* XS = reinterpret_cast<T*>(smem + lay.own);
  T *RS = XS + own_n, *DS = RS + own_n, *AS = DS + own_n;
  const int tid = threadIdx.x, sub = tid / TPS, t = tid - sub * TPS;
  T* FC = reinterpret_cast<T*>(smem + lay.fc) + (size_t)sub * 8 * EXY;
  unsigned char* HS = smem + lay.hs + (size_t)sub * 2 * L::kHChunks * EXY * 16;
  uint8_t* SL = smem + lay.sl + (size_t)sub * (kz + 1) * EXY;
  const int txy = blockIdx.x % a.tiles_xy, bz = blockIdx.x / a.tiles_xy;
  const int i0 = (txy % a.tiles_x) * OX, j0 = (txy / a.tiles_x) * OY, k0 = bz * NS * kz;
  const int nk = min(NS * kz, g.rz - k0);                 // node layers of the block
  const int wx = min(OX, g.rx - i0), wy = min(OY, g.ry - j0);  // owned nodes per axis
  const size_t plane_n = (size_t)g.rx * g.ry, plane_e = (size_t)g.nx * g.ny;
  PcgState S = *a.st;
  GridSync gs{a.slots, a.err, 0ull};
  __shared__ int s_lost;  // a halo wait of this block ran out
  if (tid == 0) s_lost = s_halo = 0;
  auto fail = [&] {  // a wait ran out
    if (tid == 0) atomicExch(&a.st->grid_error, 1);
  };
  // box position b (plane, row, column) of the halo: its node, or -1 (owned here, outside the grid, or beyond
  // the layer next to the owned nodes)
  const int box_n = (nk + 2) * PL;
  auto halo_node = [&](int b) -> int {
    const int plane = b / PL, r = b - plane * PL, row = r / NTX, col = r - row * NTX;
    if (plane >= 1 && plane <= nk && row >= 1 && row <= wy && col >= 1 && col <= wx) return -1;
    if (row > wy + 1 || col > wx + 1) return -1;
    const int i = wrap_node(i0 - 1 + col, g.nx, g.rx, g.px), j = wrap_node(j0 - 1 + row, g.ny, g.ry, g.py);
    const int k = wrap_node(k0 - 1 + plane, g.nz, g.rz, g.pz);
    return i >= 0 && j >= 0 && k >= 0 ? i + g.rx * (j + g.ry * k) : -1;
  };
  // this thread's owned column: nodes (ni, nj, k0 + sub kz + kk), kk < K
  const int ni = t % OX, nj = t / OX;
  const int K = max(0, min(kz, nk - sub * kz));
  const bool owner = t < OXY && ni < wx && nj < wy;
  const int no = (i0 + ni) + g.rx * (j0 + nj);
  const int kb = k0 + sub * kz;  // first node layer of the sub-brick
  const bool rim_xy = ni == 0 || nj == 0 || ni == wx - 1 || nj == wy - 1;
  auto rim = [&](int kk) { return rim_xy || (sub == 0 && kk == 0) || sub * kz + kk == nk - 1; };
  // the column in the owned arrays (stride OXY per layer) and in P (stride PL)
  const int o0 = sub * kz * OXY + t, p0 = (sub * kz + 1) * PL + (nj + 1) * NTX + ni + 1;
  // masked nodes of the column (the depth is at most 32, brick_depth)
  unsigned masked = 0;
  for (int b = tid; b < (NS * kz + 2) * PL; b += kT) P[b] = T(0);
  __syncthreads();
  if (owner) {
    for (int kk = 0; kk < K; ++kk) {
      const size_t n = plane_n * (kb + kk) + no;
      const int o = o0 + kk * OXY;
      XS[o] = a.x[n];
      RS[o] = a.r[n];
      DS[o] = a.inv_diag ? a.inv_diag[n] : T(1);
      P[p0 + kk * PL] = a.p[n];
      if (a.mask && a.mask[n]) masked |= 1u << kk;
    }
  }
  for (int b = tid; b < box_n; b += kT) {
    const int n = halo_node(b);
    if (n >= 0) {
      P[b] = a.p[n];
      const int e = atomicAdd(&s_halo, 1);  // (any order: every entry is a node of its own)
      HN[e] = n;
      HB[e] = b;
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
  const bool h_async = a.H != nullptr && aligned16(a.H);
  // corner results of the four columns that meet at the owned node
  const int f0 = (ni + 1) + EX * (nj + 1), f1 = EXY + ni + EX * (nj + 1), f2 = 2 * EXY + (ni + 1) + EX * nj,
            f3 = 3 * EXY + ni + EX * nj;
  const T* pe = P + (size_t)sub * kz * PL + eb * NTX + ea;
  const int gk0 = wrap_elem(kb - 1, g.nz, g.pz);
  auto next_layer = [&](int gk) { return gk + 1 < g.nz ? gk + 1 : (g.pz ? 0 : -2); };
  __syncthreads();
  for (int it = 0; it < a.maxiter && S.active; ++it) {
    double v1[1] = {0.0};
    if (K > 0) {
      // ---- A p over the sub-brick
      DFace<T> fl{};
      if (t < EXY) fl = dface(pe[0], pe[1], pe[NTX], pe[NTX + 1]);
      DForce<T> pend{T(0), T(0), T(0), T(0)};
      auto stage_h = [&](int kk, int gk) {
        if (h_async && eo >= 0 && gk >= 0)
          stage_chunks(HS + (size_t)(kk & 1) * L::kHChunks * EXY * 16, EXY, t, 0,
                       a.H + kStageH * (plane_e * gk + eo), L::kHChunks);
        cp_async_commit();
      };
      int gk = gk0;
      stage_h(0, gk);
      T dot = T(0);
      const T* pu = pe;
      const T* pn = P + p0 - PL;
      T* ao = AS + o0 - OXY;
      const uint8_t* sp = SL + t;
      for (int kk = 0; kk <= K; ++kk) {
        const int gn = kk < K ? next_layer(gk) : -1;
        stage_h(kk + 1, gn);
        cp_async_wait<1>();  // this thread's H of element layer kk
        T* fc = FC + (kk & 1) * 4 * EXY;
        pu += PL;
        if (t < EXY) {
          const DFace<T> fu = dface(pu[0], pu[1], pu[NTX], pu[NTX + 1]);
          DForce<T> lo = pend;
          pend = DForce<T>{T(0), T(0), T(0), T(0)};
          if (eo >= 0 && gk >= 0) {
            T hq[kStageH];
            if (h_async) {
              load_chunks<T, kStageH>(HS + (size_t)(kk & 1) * L::kHChunks * EXY * 16, EXY, t, hq);
            } else {
              const size_t e = plane_e * gk + eo;
#pragma unroll
              for (int q = 0; q < 8; ++q) hq[q] = a.H ? __ldg(a.H + 8 * e + q) : T(0);
            }
            const int sl = *sp;
            damage_element(fl, fu, hq, a.gcw[sl], a.chw, a.k2[sl], a.ek, lo, pend);
          }
          fl = fu;
          if (kk >= 1) {
            T c[4];
            dcorners(lo, c);
#pragma unroll
            for (int q = 0; q < 4; ++q) fc[q * EXY + t] = c[q];
          }
        }
        sp += EXY;
        gk = gn;
        if (kk >= 1) {  // (the first element layer only fills pend)
          // two corner buffers in turn: a buffer is written again after the next layer's barrier
          sub_barrier(1 + sub, TPS);
          if (owner) {
            // (diagonal pairs first; h8_dtile_kernel adds the four in rows.  Either rounds alike, but the last
            // places move iteration counts of several hundred by a few, which the fixtures' tests compare exactly.)
            T v = (fc[f0] + fc[f3]) + (fc[f1] + fc[f2]);
            if (masked >> (kk - 1) & 1u) v = T(0);
            *ao = v;
            dot += *pn * v;
          }
        }
        ao += OXY;
        pn += PL;
      }
      cp_async_wait<0>();
      v1[0] = double(dot);
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
        const int o = o0 + kk * OXY;
        XS[o] = XS[o] + al * P[p0 + kk * PL];
        const T r = RS[o] - al * AS[o];
        RS[o] = r;
        v2[1] += double(r) * double(r);
        const T z = r * DS[o];
        v2[0] += double(r) * double(z);
        if (rim(kk)) st_tagged(a.z + plane_n * (kb + kk) + no, double(z), it + 1);
      }
    }
    // the halo's z arrives beside the sums
    auto take_halo = [&](int i, int step) {
      constexpr int B = 4;  // polls in flight
      for (int e = i; e < s_halo; e += B * step) {
        Tagged q[B];
#pragma unroll
        for (int j = 0; j < B; ++j)
          if (e + j * step < s_halo) q[j] = ld_tagged(a.z + HN[e + j * step]);
#pragma unroll
        for (int j = 0; j < B; ++j) {
          const int f = e + j * step;
          if (f < s_halo) {
            if (q[j].tag != (unsigned long long)(it + 1) && !wait_tagged(a.z + HN[f], it + 1, &q[j].v, a.err))
              s_lost = 1;
            HV[f] = T(q[j].v);
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
    for (int e = tid; e < s_halo; e += kT) {
      T& p = P[HB[e]];
      p = HV[e] + be * p;
    }
    if (owner) {
      for (int kk = 0; kk < K; ++kk) {
        const int o = o0 + kk * OXY, q = p0 + kk * PL;
        P[q] = RS[o] * DS[o] + be * P[q];
      }
    }
    __syncthreads();
  }
  if (owner) {
    for (int kk = 0; kk < K; ++kk) {
      const size_t n = plane_n * (kb + kk) + no;
      a.x[n] = XS[o0 + kk * OXY];
      a.r[n] = RS[o0 + kk * OXY];
    }
  }
  if (blockIdx.x == 0 && tid == 0) store_pcg_state(a.st, S);
}

// Bricks of one shape: the least depth that covers the grid with at most `blocks` blocks; 0 when none fits.
template <typename T, int OX, int OY, int NS>
int brick_depth(const VoxGeom& g, int blocks) {
  const int txy = ((g.rx + OX - 1) / OX) * ((g.ry + OY - 1) / OY);
  if (txy > blocks) return 0;
  const int slabs = std::min(blocks / txy, g.rz);
  const int layers = (g.rz + slabs - 1) / slabs, kz = (layers + NS - 1) / NS;
  return kz <= 32 && BrickLayout<T, OX, OY, NS>(kz).total <= kSmemMax ? kz : 0;
}

template <typename T, int OX, int OY, int NS>
int launch_bricks(BrickArgs<T> a, int kz, cudaStream_t s) {
  const VoxGeom& g = a.g;
  a.tiles_x = (g.rx + OX - 1) / OX;
  a.tiles_xy = a.tiles_x * ((g.ry + OY - 1) / OY);
  a.kz = kz;
  const int grid = a.tiles_xy * ((g.rz + NS * kz - 1) / (NS * kz));
  auto kern = h8_dpcg_kernel<T, OX, OY, NS>;
  void* args[] = {&a};
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) != cudaSuccess ||
      cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kT), args, BrickLayout<T, OX, OY, NS>(kz).total,
                                  s) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  note_launch();
  return PHASTB_OK;
}

}  // namespace

template <typename T>
int h8_damage_brick_pcg(const DTileArgs<T>& d, const PcgWs<T>& w, void* tagged, T* x, const T* inv_diag, int maxiter,
                        int mode, cudaStream_t s) {
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  if (!coop || !tagged || !aligned16(tagged) || !aligned16(w.part) || mode == PCG_PERIODIC || !persistent_pcg_enabled())
    return PHASTB_UNSUPPORTED;
  const int blocks = std::min(sms, kGridBlocks);
  // 16 x 14 bricks recompute the least halo; 14 x 7 and 8 x 8 follow ragged grids more closely.  The march is
  // kz + 1 layers whatever the shape, so the least depth wins.
  const VoxGeom& g = d.g;
  const int depth[3] = {brick_depth<T, 16, 14, 2>(g, blocks), brick_depth<T, 14, 7, 4>(g, blocks),
                        brick_depth<T, 8, 8, 4>(g, blocks)};
  int best = -1;
  for (int i = 0; i < 3; ++i)
    if (depth[i] && (best < 0 || depth[i] < depth[best])) best = i;
  if (best < 0) return PHASTB_UNSUPPORTED;
  BrickArgs<T> a;
  std::memset(&a, 0, sizeof(a));
  a.g = g;
  a.maxiter = maxiter;
  a.mode = mode;
  a.slot = d.slot;
  const double wsc = g.w * d.scale / 64.0;
  for (int i = 0; i < PHASTB_MAX_SLOTS; ++i) {
    a.gcw[i] = T(wsc) * d.gc_ell[i];
    a.k2[i] = d.gc_k2[i];
  }
  a.chw = T(wsc) * T(2.0 * (1.0 - d.kappa));
  a.ek = damage_elem_k<T>(g, d.scale);
  a.H = d.H;
  a.mask = d.mask;
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
  if (!st) st = cuda_status(cudaMemsetAsync(tagged, 0, sizeof(Tagged) * (size_t)g.n_red, s));
  if (st) return st;
  if (best == 0) return launch_bricks<T, 16, 14, 2>(a, depth[0], s);
  if (best == 1) return launch_bricks<T, 14, 7, 4>(a, depth[1], s);
  return launch_bricks<T, 8, 8, 4>(a, depth[2], s);
}

template int h8_damage_brick_pcg<double>(const DTileArgs<double>&, const PcgWs<double>&, void*, double*,
                                         const double*, int, int, cudaStream_t);
template int h8_damage_brick_pcg<float>(const DTileArgs<float>&, const PcgWs<float>&, void*, float*, const float*, int,
                                        int, cudaStream_t);

}  // namespace phastb
