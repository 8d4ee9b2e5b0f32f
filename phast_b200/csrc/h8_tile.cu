// Tiled z-marching voxel H8 elastic action (see h8_tile.cuh).
#include "h8_tile.cuh"
#include "h8_elastic.cuh"
#include <cuda.h>
#include <cudaTypedefs.h>
#include "engine.cuh"

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

namespace phastb {

namespace {

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---- TMA staging of node layers (cp.async.bulk.tensor, completion on an mbarrier)
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Orders this thread's earlier generic-proxy accesses of shared memory (reads of
// a buffer, stores of patched halo values) before async-proxy (TMA) writes.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// 3D tiled copy global -> this CTA's shared memory (no multicast); the innermost
// coordinate c0 times the element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
// A TMA completion wait gives up after kTmaLimitNs of global time (a normal wait
// is well under a microsecond); the caller then marks its output non-finite.
constexpr unsigned long long kTmaLimitNs = 1000000000ull;
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
  if (mbar_try_wait(bar, parity)) return true;  // the usual case: the copy landed during the last layer
  const unsigned long long t0 = global_ns();
  for (unsigned i = 0; i < (1u << 26); ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 63u && global_ns() - t0 > kTmaLimitNs) return false;
  }
  return false;
}
__device__ __forceinline__ int floor_mult(int v, int m) { return (v >= 0 ? v / m : -((-v + m - 1) / m)) * m; }

// A thread's (at most two) nodes of a layer, in registers (the wrapped halo nodes
// that TMA staging patches).
template <typename T>
struct Staged {
  T v[2][4];
};

__device__ __forceinline__ void get4(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x;
  v[1] = q.y;
  v[2] = q.z;
  v[3] = q.w;
}
__device__ __forceinline__ void get4(const double* p, double (&v)[4]) {
  const double2 q = reinterpret_cast<const double2*>(p)[0], r = reinterpret_cast<const double2*>(p)[1];
  v[0] = q.x;
  v[1] = q.y;
  v[2] = r.x;
  v[3] = r.y;
}

}  // namespace

// What bounds it: instruction issue.  An element costs about 490 FP instructions: its strains and forces are
// evaluated in the Haar (modal) basis of its eight corners, where a gradient component at the Gauss points is two
// butterflies of scaled modes, and each face's modes and force modes are formed once and shared by the two
// elements that meet there, through registers, since a thread marches up its element column.  The nodal form
// before it (interpolating every face difference per element, lower and upper corner forces through shared
// memory) issued 1 250.  Node layers are copied global -> shared with cp.async two layers ahead (no staging
// registers), and in-plane offsets are formed once per brick.  Measured per action, this and the nodal form:
// 64^3 FP32 24.7 / 29.3 us, FP64 32.9 / 51.8; 192^3 FP32 284 / 450, FP64 511 / 804; 97 x 83 x 110 FP64 84 / 144.
//
// One launch = every brick of the grid (persistent blocks).  COEF selects the
// element coefficients (material slot + g(d), isotropic or general Voigt, or
// per-Gauss-point moduli of a multigrid coarse level); MODE selects the node
// epilogue: y = A x, y plus x . y, y plus the energy, or one Chebyshev
// smoothing step on (res, d, x) driven by A d.
// TMA: the node layers are staged by tensor-map copies (tmx: u~ as a (3 rx,
// ry, rz) array, tmd: d as (rx, ry, rz)) issued by one thread and completed on an
// mbarrier per layer buffer; halo nodes that wrap around a periodic edge read
// the zero fill and are patched by per-thread loads.  Otherwise every thread
// copies its (at most two) halo-tile nodes into shared memory with cp.async.
// The action over the bricks vb, vb + vgrid, ... of one grid: a plain launch runs it with
// its block index and grid size, a batched launch with the block's virtual index inside its cell.
template <typename T, int COEF, int MODE, int OX, int OY, bool TMA>
__device__ __forceinline__ void tile_body(const TileArgs<T>& a, const VoxMat<T>& m, const CUtensorMap* tmx,
                                          const CUtensorMap* tmd, const int vb, const int vgrid) {
  if (a.guard && *a.guard == 0) return;
  constexpr bool SLOT = COEF != kCoefQP;
  constexpr bool DOT = MODE == kModeDot, ENERGY = MODE == kModeEnergy, CHEB = MODE == kModeCheb;
  // E rows (macro strain) exist on the fine operator; a Chebyshev step and a
  // nodal-block action leave them alone (masked)
  constexpr bool NODAL = MODE == kModeNodal, RES = MODE == kModeRes, SMOOTH = MODE == kModeSmooth;
  constexpr bool EROWS = SLOT && !CHEB && !NODAL && !RES && !SMOOTH;
  constexpr bool RED = EROWS || DOT || ENERGY || SMOOTH;
  constexpr bool EPI = CHEB || RES || SMOOTH;  // the epilogue reads vectors of the owned nodes
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const VoxGeom& g = a.g;
  if (NODAL && vb == 0 && threadIdx.x < 6 && a.y) a.y[3 * (size_t)g.n_red + threadIdx.x] = T(0);
  const T* __restrict__ x = a.x;
  const T* __restrict__ d = SLOT ? a.d : nullptr;
  // OX, OY > 0: a compiled tile shape (constant shared-memory offsets)
  const int ox = OX ? OX : a.ts.ox, oy = OY ? OY : a.ts.oy, kz = a.ts.kz;
  const int ex = ox + 1, exy = ex * (oy + 1);
  const int ntx = ox + 2, nt = ntx * (oy + 2);
  // TMA: shared memory from a 128-byte boundary; u~ layer buffers of W words per
  // halo row, d layer buffers of Wd words, each started from a 16-byte aligned column
  unsigned char* sbase =
      TMA ? reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127))
          : smem_raw;
  const int W = tma_wx<T>(ox), Wd = tma_wd<T>(ox);
  const size_t xbb = tma_xbytes<T>(ox, oy), dbb = tma_dbytes<T>(ox, oy);
  T* nb = reinterpret_cast<T*>(sbase);  // [3 buffers][nt][4 fields] (without TMA)
  size_t off_face = 0, off_qp = 0, off_cheb = 0;
  if (TMA) {
    tile_layout_tma<T>(ox, oy, COEF == kCoefQP, EPI, &off_face, &off_qp, &off_cheb);
  } else {
    tile_layout<T>(ox, oy, COEF == kCoefQP, EPI, &off_qp, &off_cheb);
    off_face = sizeof(T) * 12 * (size_t)nt;
  }
  T* FC = reinterpret_cast<T*>(sbase + off_face);  // corner forces of one node layer, [4 corners][3 comps][exy]
  // staged by cp.async, two buffers each: kCoefQP (lam_q, mu_q) of this thread's
  // element one element layer ahead, chunk-major [2][chunks][exy]; kModeCheb
  // (res, invd, xs) of this thread's owned node, [2][9][ox*oy], copied while the
  // layer's elements are computed
  constexpr int kQChunks = kStageQP * (int)sizeof(T) / 16;
  unsigned char* QS = sbase + off_qp;
  T* CS = reinterpret_cast<T*>(sbase + off_cheb);
  __shared__ __align__(8) unsigned long long s_mbar[3];
  unsigned mphase = 0;  // bit b: parity of the next completion of buffer b's barrier
  bool tma_fault = false;
  const bool use_d = SLOT && d != nullptr && a.gq == nullptr;
  const unsigned tma_tx = (unsigned)(sizeof(T) * (size_t)W * (oy + 2) + (use_d ? sizeof(T) * (size_t)Wd * (oy + 2) : 0));
  if (TMA) {
    if (threadIdx.x == 0) {
      for (int b = 0; b < 3; ++b) mbar_init(&s_mbar[b], 1);
      mbar_init_fence();
    }
    __syncthreads();
  }
  const int oxy = ox * oy;
  const bool q_async = COEF == kCoefQP && aligned16(a.lam_q) && aligned16(a.mu_q);
  const int tid = threadIdx.x;
  const T w = T(g.w);
  const T c1 = T(a.c1), c2 = T(a.c2);
  // macro strain, read from shared memory where it is used (six registers fewer per thread); a Chebyshev
  // step smooths the nodal block only (E rows masked).  The first barrier of the march orders the store.
  // All six E rows masked (a cell under full macro-strain control): CG's action does not form their sums, and
  // its reduction shrinks from eight values to the dot product.
  bool e_live = EROWS;
  if constexpr (EROWS && DOT) {
    if (a.mask) {
      const uint8_t* em = a.mask + 3 * (size_t)g.n_red;
      e_live = !(__ldg(em) && __ldg(em + 1) && __ldg(em + 2) && __ldg(em + 3) && __ldg(em + 4) && __ldg(em + 5));
      if (!e_live && vb == 0 && threadIdx.x < 6 && a.y) a.y[3 * (size_t)g.n_red + threadIdx.x] = T(0);
    }
  }
  __shared__ T E6[6];
  if (EROWS && tid < 6) E6[tid] = __ldg(x + 3 * (size_t)g.n_red + tid);
  const int tiles_x = (g.rx + ox - 1) / ox, tiles_y = (g.ry + oy - 1) / oy;
  const int tiles_xy = tiles_x * tiles_y;
  const int n_tiles = tiles_xy * ((g.rz + kz - 1) / kz);
  // element / owned-node coordinates of this thread inside the tile
  const int ea = tid % ex, eb = tid / ex;
  const int ni = tid % ox, nj = tid / ox;
  const bool is_elem = tid < exy, is_node = tid < ox * oy;
  constexpr int kA = 16 / (int)sizeof(T);  // words per 16 bytes
  int xr = 0, dr = 0, xs0 = 0, ds0 = 0;    // TMA: row start columns and remainders of the current tile
  // node value of component c (3: d) at halo-tile position (row, col) of layer buffer `buf`
  auto nval = [&](int buf, int c, int row, int col) -> T {
    if constexpr (TMA) {
      if (c < 3) return reinterpret_cast<const T*>(sbase + (size_t)buf * xbb)[row * W + xr + 3 * col + c];
      return reinterpret_cast<const T*>(sbase + 3 * xbb + (size_t)buf * dbb)[row * Wd + dr + col];
    } else {
      return nb[4 * (nt * buf + row * ntx + col) + c];
    }
  };
  // the upper or lower face of this thread's element from layer buffer `buf`
  auto load_face = [&](int buf, Face<T>& f) {
    T v[4][4];  // [corner][ux, uy, uz, d]
#pragma unroll
    for (int L = 0; L < 4; ++L) {
      const int row = eb + (L >> 1), col = ea + (L & 1);
      if constexpr (TMA) {
#pragma unroll
        for (int c = 0; c < 3; ++c) v[L][c] = nval(buf, c, row, col);
        v[L][3] = use_d ? nval(buf, 3, row, col) : T(0);
      } else {
        get4(nb + 4 * (nt * buf + row * ntx + col), v[L]);
      }
    }
    elastic_face(v, f);
    if (use_d) damage_face(v[0][3], v[1][3], v[2][3], v[3][3], a.k, f);
  };
  // TMA: thread 0 issues the copies of node layer kn into buffer b
  auto tma_issue = [&](int i0, int j0, int kn, int b) {
    if constexpr (TMA) {
      if (threadIdx.x == 0) {
        const int gz = g.pz ? wrap_node(kn, g.nz, g.rz, 1) : kn;  // out of range: the zero fill
        fence_proxy_async();
        mbar_expect_tx(&s_mbar[b], tma_tx);
        tma_load_3d(sbase + (size_t)b * xbb, tmx, xs0, j0 - 1, gz, &s_mbar[b]);
        if (use_d) tma_load_3d(sbase + 3 * xbb + (size_t)b * dbb, tmd, ds0, j0 - 1, gz, &s_mbar[b]);
      }
    }
  };
  // TMA: halo nodes of layer kn that wrap around a periodic edge (the copy read the zero fill there)
  auto wrap_load = [&](int i0, int j0, int kn, Staged<T>& r, unsigned& on) {
    on = 0;
    if constexpr (TMA) {
      const int gk = wrap_node(kn, g.nz, g.rz, g.pz);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = threadIdx.x + h * blockDim.x;
        if (t < nt && gk >= 0) {
          const int ri = i0 - 1 + t % ntx, rj = j0 - 1 + t / ntx;
          const bool wx = g.px && (ri < 0 || ri >= g.rx), wy = g.py && (rj < 0 || rj >= g.ry);
          if (wx || wy) {
            const int gi = wrap_node(ri, g.nx, g.rx, g.px), gj = wrap_node(rj, g.ny, g.ry, g.py);
            if (gi >= 0 && gj >= 0) {
              const size_t n = (size_t)gi + (size_t)g.rx * ((size_t)gj + (size_t)g.ry * gk);
              r.v[h][0] = __ldg(x + 3 * n);
              r.v[h][1] = __ldg(x + 3 * n + 1);
              r.v[h][2] = __ldg(x + 3 * n + 2);
              r.v[h][3] = use_d ? __ldg(d + n) : T(0);
              on |= 1u << h;
            }
          }
        }
      }
    }
  };
  auto wrap_store = [&](const Staged<T>& r, unsigned on, int b) {
    if constexpr (TMA) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (on & (1u << h)) {
          const int t = threadIdx.x + h * blockDim.x, col = t % ntx, row = t / ntx;
          T* xbuf = reinterpret_cast<T*>(sbase + (size_t)b * xbb);
#pragma unroll
          for (int c = 0; c < 3; ++c) xbuf[row * W + xr + 3 * col + c] = r.v[h][c];
          if (use_d) reinterpret_cast<T*>(sbase + 3 * xbb + (size_t)b * dbb)[row * Wd + dr + col] = r.v[h][3];
        }
      }
      // these generic-proxy writes must be ordered before the tensor copy that later refills the buffer
      if (on) fence_proxy_async();
    }
  };
  // TMA: waits (bounded) for buffer b's copies of its current fill
  auto tma_wait = [&](int b) {
    if constexpr (TMA) {
      if (!mbar_wait(&s_mbar[b], (mphase >> b) & 1u)) tma_fault = true;
      mphase ^= 1u << b;
    }
  };
  double accd[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  // a coarse level's last Chebyshev step also sums x's components (a reduction workspace is given then)
  const bool sum_x = CHEB && !SLOT && a.ws.counter != nullptr;
  const size_t plane_n = (size_t)g.rx * g.ry, plane_e = (size_t)g.nx * g.ny;

  for (int tile = vb; tile < n_tiles; tile += vgrid) {
    const int tz = tile / tiles_xy, txy = tile - tz * tiles_xy;
    const int i0 = (txy % tiles_x) * ox, j0 = (txy / tiles_x) * oy;
    const int k0 = tz * kz, k1 = min(k0 + kz, g.rz);
    // In-plane offsets of this thread's staged nodes, element and owned node, once per brick (-1: outside
    // the grid or not this thread's); a layer then adds one uniform plane offset.
    int so[2], eo = -1, no = -1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = tid + h * blockDim.x;
      so[h] = -1;
      if (t < nt) {
        const int gi = wrap_node(i0 - 1 + t % ntx, g.nx, g.rx, g.px);
        const int gj = wrap_node(j0 - 1 + t / ntx, g.ny, g.ry, g.py);
        if (gi >= 0 && gj >= 0) so[h] = gi + g.rx * gj;
      }
    }
    if (is_elem) {
      const int gi = wrap_elem(i0 - 1 + ea, g.nx, g.px);
      const int gj = wrap_elem(j0 - 1 + eb, g.ny, g.py);
      if (gi >= 0 && gj >= 0) eo = gi + g.nx * gj;
    }
    if (is_node && i0 + ni < g.rx && j0 + nj < g.ry) no = (i0 + ni) + g.rx * (j0 + nj);
    const bool own_xy = ea >= 1 && eb >= 1 && i0 - 1 + ea < g.rx && j0 - 1 + eb < g.ry;
    // cp.async of node layer kn into buffer b (zeros outside the grid)
    auto stage_nodes = [&](int kn, int b) {
      const int gk = wrap_node(kn, g.nz, g.rz, g.pz);
      const T* xk = x + 3 * (plane_n * (size_t)(gk < 0 ? 0 : gk));
      const T* dk = use_d ? d + plane_n * (size_t)(gk < 0 ? 0 : gk) : nullptr;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = tid + h * blockDim.x;
        if (t < nt) {
          const bool live = so[h] >= 0 && gk >= 0;
          const int o = so[h] >= 0 ? so[h] : 0;
          T* dst = nb + 4 * (nt * b + t);
#pragma unroll
          for (int c = 0; c < 3; ++c) cp_async_word_or_zero(dst + c, xk + 3 * (size_t)o + c, live);
          if (use_d) cp_async_word_or_zero(dst + 3, dk + o, live);
        }
      }
    };
    // material slot of this thread's element in layer ke (0 outside the grid)
    auto elem_slot = [&](int ke) -> int {
      const int gk = wrap_elem(ke, g.nz, g.pz);
      return SLOT && eo >= 0 && gk >= 0 ? __ldg(a.slot + plane_e * gk + eo) : 0;
    };
    // fixed-dof bits (one per component) of this thread's owned node in layer kn
    auto node_mask = [&](int kn) -> int {
      if (!a.mask || no < 0 || kn >= g.rz) return 0;
      const uint8_t* mp = a.mask + 3 * (plane_n * kn + no);
      return (__ldg(mp) ? 1 : 0) | (__ldg(mp + 1) ? 2 : 0) | (__ldg(mp + 2) ? 4 : 0);
    };
    // kCoefQP: cp.async of element layer ke's (lam_q, mu_q) into buffer `buf`
    auto stage_qp = [&](int ke, int buf) {
      if constexpr (COEF == kCoefQP) {
        const int gk = wrap_elem(ke, g.nz, g.pz);
        if (q_async && eo >= 0 && gk >= 0) {
          const size_t e = plane_e * gk + eo;
          unsigned char* dst = QS + (size_t)buf * kQChunks * exy * 16;
          stage_chunks(dst, exy, tid, 0, a.lam_q + 8 * e, kQChunks / 2);
          stage_chunks(dst, exy, tid, kQChunks / 2, a.mu_q + 8 * e, kQChunks / 2);
        }
      }
    };
    // kModeCheb: cp.async of (res, invd, xs) of the owned node in node layer kn into buffer `buf` (kModeSmooth:
    // res and invd, kModeRes: res)
    auto stage_cheb = [&](int kn, int buf) {
      if constexpr (EPI) {
        if (no >= 0) {
          const size_t n3 = 3 * (plane_n * kn + no);
          T* dst = CS + (size_t)buf * 9 * oxy + tid;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            cp_async_word(dst + c * oxy, a.res + n3 + c);
            if (!RES) cp_async_word(dst + (3 + c) * oxy, a.invd + n3 + c);
            if (CHEB) cp_async_word(dst + (6 + c) * oxy, a.xs + n3 + c);
          }
        }
      }
    };
    T tacc[8] = {T(0), T(0), T(0), T(0), T(0), T(0), T(0), T(0)};
    Face<T> fl;         // lower face of this thread's element
    FaceForce<T> pend;  // force of the element below on that face
#pragma unroll
    for (int c = 0; c < 3; ++c) pend.M[c] = pend.X[c] = pend.Y[c] = pend.XY[c] = T(0);
    Staged<T> pf;
    unsigned pf_on = 0;
    __syncthreads();  // the previous tile's last node phase is done with the buffers
    if constexpr (TMA) {
      xs0 = floor_mult(3 * (i0 - 1), kA);
      xr = 3 * (i0 - 1) - xs0;
      ds0 = floor_mult(i0 - 1, kA);
      dr = (i0 - 1) - ds0;
      tma_issue(i0, j0, k0 - 1, 0);
      tma_issue(i0, j0, k0, 1);
      wrap_load(i0, j0, k0 - 1, pf, pf_on);
      tma_wait(0);
      wrap_store(pf, pf_on, 0);
      wrap_load(i0, j0, k0, pf, pf_on);
    } else {
      stage_nodes(k0 - 1, 0);
      stage_nodes(k0, 1);
    }
    int sl_next = elem_slot(k0 - 1);
    stage_qp(k0 - 1, 0);
    cp_async_commit();
    int mk_next = node_mask(k0), mk_cur = 0;
    const int K = k1 - k0;
    // Commit groups of a step: the Chebyshev data of node layer ke, then the moduli of element layer ke + 1
    // with node layer ke + 2.
    for (int kk = 0; kk <= K; ++kk) {
      const int ke = k0 - 1 + kk;  // element layer of this step
      const int ib0 = kk % 3, ib1 = (kk + 1) % 3;
      if constexpr (TMA) {
        tma_wait(ib1);  // node layer ke + 1
        wrap_store(pf, pf_on, ib1);
      }
      cp_async_wait<0>();  // node layer ke + 1 and the moduli of element layer ke have landed
      const int sl = sl_next;
      if (kk >= 1) {
        mk_cur = mk_next;
        if (kk < K) mk_next = node_mask(ke + 1);
      }
      __syncthreads();
      // every thread is done with buffer (kk + 2) % 3 (node layer ke - 1): refill it with layer ke + 2
      if constexpr (EPI) {
        if (kk >= 1) stage_cheb(ke, kk & 1);
        cp_async_commit();
      }
      if (kk < K) {
        if constexpr (TMA) {
          tma_issue(i0, j0, ke + 2, (kk + 2) % 3);
          wrap_load(i0, j0, ke + 2, pf, pf_on);
        } else {
          stage_nodes(ke + 2, (kk + 2) % 3);
        }
        stage_qp(ke + 1, (kk + 1) & 1);
        sl_next = elem_slot(ke + 1);
      }
      cp_async_commit();
      // ---- element phase: one element of the (ox+1) x (oy+1) tile per thread
      if (is_elem) {
        if (kk == 0) load_face(ib0, fl);
        Face<T> fu;
        load_face(ib1, fu);
        const int gk = wrap_elem(ke, g.nz, g.pz);
        // lo: the column's whole force on node layer ke, the upper face of the element below (pend) plus
        // the lower face of this one
        FaceForce<T> lo = pend;
#pragma unroll
        for (int c = 0; c < 3; ++c) pend.M[c] = pend.X[c] = pend.Y[c] = pend.XY[c] = T(0);
        if (eo >= 0 && gk >= 0) {
          const size_t e = plane_e * gk + eo;
          const bool own = own_xy && kk >= 1;
          // coefficients of the material: lam and mu times the quadrature weight
          const T lw = COEF == kCoefIso ? m.lam[sl] * w : T(0), mw = COEF == kCoefIso ? m.mu[sl] * w : T(0);
          const T kap = T(m.kappa), okap = T(1) - kap;
          // degradation (and, on coarse levels, the moduli) of a half's four Gauss points
          T gv[4], lm[8];
          auto half = [&](int qz) {
            if (SLOT) {
              if (a.gq) {
#pragma unroll
                for (int q = 0; q < 4; ++q) gv[q] = __ldg(a.gq + 8 * e + 4 * qz + q);
              } else if (d) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  const T o = intact_at(fl, fu, a.k, qz, q);
                  gv[q] = okap * (o * o) + kap;
                }
              } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) gv[q] = T(1);
              }
            } else if (q_async) {
              // chunks of the half: lam_q at qz * n, mu_q after all of lam_q
              constexpr int nc = kQChunks / 4;
              const unsigned char* qs = QS + (size_t)(kk & 1) * kQChunks * exy * 16;
              T l4[4], m4[4];
              load_chunks<T, 4>(qs + (size_t)qz * nc * exy * 16, exy, tid, l4);
              load_chunks<T, 4>(qs + (size_t)(2 + qz) * nc * exy * 16, exy, tid, m4);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                lm[q] = l4[q];
                lm[4 + q] = m4[q];
              }
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                lm[q] = __ldg(a.lam_q + 8 * e + 4 * qz + q);
                lm[4 + q] = __ldg(a.mu_q + 8 * e + 4 * qz + q);
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
              iso_stress(COEF == kCoefIso ? lw * gv[q] : lm[q] * w, COEF == kCoefIso ? mw * gv[q] : lm[4 + q] * w, ep,
                         sg);
            }
            if (ENERGY && own) {
#pragma unroll
              for (int i = 0; i < 6; ++i) tacc[kOutEnergy] += T(0.5) * sg[i] * ep[i];
            }
          };
          auto rows = [&](int c, T sx, T sy, T sz) {
            if (EROWS && own && e_live) {
              if (c == 0) {
                tacc[0] += sx;
                tacc[5] += sy;
                tacc[4] += sz;
              } else if (c == 1) {
                tacc[1] += sy;
                tacc[3] += sz;
              } else {
                tacc[2] += sz;
              }
            }
          };
          elastic_element<EROWS>(fl, fu, a.k, E6, half, stress, rows, lo, pend);
        }
        fl = fu;
        if (kk >= 1) {
          corner_forces(lo, FC, exy, tid);  // of node layer ke
        }
      }
      if (kk == 0) continue;  // the first element layer only fills pend
      __syncthreads();
      if constexpr (EPI) cp_async_wait<1>();  // this thread's (res, invd, xs) of node layer ke
      // ---- node phase: node layer ke, the four columns that meet at the node
      if (no >= 0) {
        const int e11 = (ni + 1) + ex * (nj + 1), e01 = ni + ex * (nj + 1);
        const int e10 = (ni + 1) + ex * nj, e00 = ni + ex * nj;
        {
          const size_t n = plane_n * ke + no;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            T v = node_force(FC, exy, c, e11, e01, e10, e00);
            if (mk_cur & (1 << c)) v = T(0);
            const size_t i = 3 * n + c;
            const T xin = nval(ib0, c, nj + 1, ni + 1);
            if (CHEB) {
              const T* cs = CS + (size_t)(kk & 1) * 9 * oxy + tid;
              const T r = cs[c * oxy] - v;
              a.res[i] = r;
              const T dn = c1 * xin + c2 * cs[(3 + c) * oxy] * r;
              a.d_out[i] = dn;
              const T xn = cs[(6 + c) * oxy] + dn;
              a.xs[i] = xn;
              if (!SLOT && sum_x) accd[c] += double(xn);
            } else if (RES || SMOOTH) {
              const T b = CS[(size_t)(kk & 1) * 9 * oxy + tid + c * oxy];
              T r = b - v;
              if (RES) {
                if (mk_cur & (1 << c)) r = T(0);
                a.y[i] = r;
              } else {
                const T z = xin + c2 * CS[(size_t)(kk & 1) * 9 * oxy + tid + (3 + c) * oxy] * r;
                a.y[i] = z;
                if (SLOT)
                  accd[0] += double(b) * double(z);
                else
                  accd[c] += double(z);
              }
            } else {
              if (a.y) a.y[i] = v;
              if (DOT) tacc[kOutDot] += xin * v;
            }
          }
        }
      }
    }
    if (RED && !SMOOTH) {
#pragma unroll
      for (int k = 0; k < 8; ++k) accd[k] += double(tacc[k]);
    }
  }
  if (TMA && tma_fault) {
    // a layer copy did not complete in time: the result is unusable, so make it non-finite
    // (every solver reports PHASTB_NONFINITE for it) instead of returning wrong numbers
    const T bad = T(NAN);
    if (a.y) a.y[0] = bad;
    if (CHEB && a.res) a.res[0] = bad;
#pragma unroll
    for (int k = 0; k < 8; ++k) accd[k] = NAN;
  }

  // Sums of v[0..NK) over the grid's (or cell's) blocks: the last block to arrive folds the partials.
  auto grid_sum = [&](auto nk, double* v, auto finish) {
    constexpr int NK = decltype(nk)::value;
    __shared__ double sh[32 * NK];
    double b[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) b[k] = v[k];
    block_sum_multi<NK>(b, sh);
    if (tid == 0) {
#pragma unroll
      for (int k = 0; k < NK; ++k) a.ws.part[k * kMaxPartials + vb] = b[k];
    }
    if (arrive_last_n(a.ws.counter, vgrid)) {
      double f[NK];
      fold_sum_multi<NK>(a.ws.part, kMaxPartials, vgrid, f, sh);
      if (tid == 0) {
        finish(f);
        *a.ws.counter = 0u;
      }
    }
  };
  if constexpr (CHEB && !SLOT) {
    if (sum_x)
      grid_sum(std::integral_constant<int, 3>{}, accd, [&](const double* f) {
        for (int k = 0; k < 3; ++k) a.ws.out[k] = f[k];
      });
  } else if constexpr (SMOOTH) {
    if constexpr (SLOT) {
      if (vb == 0 && tid == 0) {  // the E rows' Jacobi step and their share of res . y
        const size_t e = 3 * (size_t)g.n_red;
        for (int k = 0; k < 6; ++k) {
          const T z = a.e_fixed[k] ? T(0) : a.res[e + k] / a.e_diag[k];
          a.y[e + k] = z;
          accd[0] += double(a.res[e + k]) * double(z);
        }
      }
      grid_sum(std::integral_constant<int, 1>{}, accd, [&](const double* f) { a.ws.out[0] = f[0]; });
    } else {
      grid_sum(std::integral_constant<int, 3>{}, accd, [&](const double* f) {
        for (int k = 0; k < 3; ++k) a.ws.out[k] = f[k];
      });
    }
  } else if constexpr (RED) {
    constexpr int NK = DOT ? 8 : (ENERGY ? 7 : 6);
    if (e_live || !EROWS) {
      grid_sum(std::integral_constant<int, NK>{}, accd, [&](const double* f) {
        double dot_e = 0.0;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          const double t = f[k];
          if (k < 6) {
            a.ws.out[k] = t;
            const size_t idx = 3 * (size_t)g.n_red + k;
            const T yv = (a.mask && a.mask[idx]) ? T(0) : T(t);
            if (a.y) a.y[idx] = yv;
            dot_e += double(x[idx]) * double(yv);
          } else if (k == kOutEnergy) {
            a.ws.out[k] = t;
          } else {
            a.ws.out[k] = t + dot_e;
          }
        }
      });
    } else if constexpr (DOT) {
      grid_sum(std::integral_constant<int, 1>{}, accd + kOutDot, [&](const double* f) { a.ws.out[kOutDot] = f[0]; });
    }
  }
}

// Threads and resident blocks per SM the kernel is compiled for: 128 registers per thread in FP32 (about 16
// warps per SM), 255 in FP64 (8 warps).  Fewer registers and more warps measured slower: FP32 at 96 registers
// 30.4 against 25.9 us on 64^3, FP64 at two blocks of 160 threads 45.4 against 43.5 us (the spills).
template <typename T, int OX, int OY>
struct TileBounds {
  static constexpr int threads = OX ? ((OX + 1) * (OY + 1) + 31) / 32 * 32 : kTileMaxThreads;
  static constexpr int blocks = sizeof(T) == 4 ? 512 / threads : (threads > 128 ? 1 : 256 / threads);
};

template <typename T, int COEF, int MODE, int OX, int OY, bool TMA>
__global__ void __launch_bounds__(TileBounds<T, OX, OY>::threads, TileBounds<T, OX, OY>::blocks)
    h8_tile_kernel(TileArgs<T> a, VoxMat<T> m, const __grid_constant__ CUtensorMap tmx,
                   const __grid_constant__ CUtensorMap tmd) {
  tile_body<T, COEF, MODE, OX, OY, TMA>(a, m, &tmx, &tmd, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------ damage action

// Scalar AT2 damage action on the same brick schedule:
//   y = scale * [Gc_e (M / ell + ell L) d + 2 (1 - kappa) sum_q w H_q N_q N_q^T d]
// (damage_element), masked rows zero.  One pass covers every brick of this
// (persistent) block: node values come from node_val(n), each owned node's
// result goes to on_owned(n, x_n, y_n), and the return value is this thread's
// share of sum_n x_n y_n (with DOT).  A thread keeps its column's upper face and
// force in registers, as the elastic march does.
template <typename T, int OX, int OY, bool DOT, class NodeVal, class OnOwned>
__device__ __forceinline__ double dtile_pass(const DTileArgs<T>& a, unsigned char* smem_raw, NodeVal node_val,
                                             OnOwned on_owned, const int vb, const int vgrid) {
  const VoxGeom& g = a.g;
  const int ox = OX ? OX : a.ts.ox, oy = OY ? OY : a.ts.oy, kz = a.ts.kz;
  const int ex = ox + 1, exy = ex * (oy + 1);
  const int ntx = ox + 2, nt = ntx * (oy + 2);
  T* nb = reinterpret_cast<T*>(smem_raw);  // [3 buffers][nt]
  T* FC = nb + 3 * nt;                     // corner results of one node layer, [4 corners][exy]
  // H of this thread's element, staged one element layer ahead, chunk-major [2][chunks][exy]
  constexpr int kHChunks = kStageH * (int)sizeof(T) / 16;
  unsigned char* HS = smem_raw + tile_stage_offset<T>(nt, exy, 3, 4);
  const int tid = threadIdx.x;
  const T wsc = T(g.w * a.scale / 64.0), chw = wsc * T(2.0 * (1.0 - a.kappa));
  const DElemK<T> ek = damage_elem_k<T>(g, a.scale);
  const int tiles_x = (g.rx + ox - 1) / ox, tiles_y = (g.ry + oy - 1) / oy;
  const int tiles_xy = tiles_x * tiles_y;
  const int n_tiles = tiles_xy * ((g.rz + kz - 1) / kz);
  const int ea = tid % ex, eb = tid / ex;
  const int ni = tid % ox, nj = tid / ox;
  const bool is_elem = tid < exy, is_node = tid < ox * oy;
  const bool h_async = a.H != nullptr && aligned16(a.H);
  const size_t plane_n = (size_t)g.rx * g.ry, plane_e = (size_t)g.nx * g.ny;
  double accd = 0.0;
  for (int tile = vb; tile < n_tiles; tile += vgrid) {
    const int tz = tile / tiles_xy, txy = tile - tz * tiles_xy;
    const int i0 = (txy % tiles_x) * ox, j0 = (txy / tiles_x) * oy;
    const int k0 = tz * kz, k1 = min(k0 + kz, g.rz);
    // in-plane offsets, once per brick (-1: outside the grid or not this thread's)
    int so[2], eo = -1, no = -1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = tid + h * blockDim.x;
      so[h] = -1;
      if (t < nt) {
        const int gi = wrap_node(i0 - 1 + t % ntx, g.nx, g.rx, g.px);
        const int gj = wrap_node(j0 - 1 + t / ntx, g.ny, g.ry, g.py);
        if (gi >= 0 && gj >= 0) so[h] = gi + g.rx * gj;
      }
    }
    if (is_elem) {
      const int gi = wrap_elem(i0 - 1 + ea, g.nx, g.px);
      const int gj = wrap_elem(j0 - 1 + eb, g.ny, g.py);
      if (gi >= 0 && gj >= 0) eo = gi + g.nx * gj;
    }
    if (is_node && i0 + ni < g.rx && j0 + nj < g.ry) no = (i0 + ni) + g.rx * (j0 + nj);
    // issues the copy of element layer ke's H into buffer `buf` (one commit group
    // per call, empty when there is nothing to copy) and returns its material slot
    auto stage_elem = [&](int ke, int buf) -> int {
      const int gk = wrap_elem(ke, g.nz, g.pz);
      int sl = 0;
      if (eo >= 0 && gk >= 0) {
        const size_t e = plane_e * gk + eo;
        sl = __ldg(a.slot + e);
        if (h_async) stage_chunks(HS + (size_t)buf * kHChunks * exy * 16, exy, tid, 0, a.H + kStageH * e, kHChunks);
      }
      cp_async_commit();
      return sl;
    };
    auto stage1 = [&](int kn, T (&r)[2]) {
      const int gk = wrap_node(kn, g.nz, g.rz, g.pz);
#pragma unroll
      for (int h = 0; h < 2; ++h) r[h] = so[h] >= 0 && gk >= 0 ? node_val(plane_n * gk + so[h]) : T(0);
    };
    auto store1 = [&](const T (&r)[2], T* buf) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = tid + h * blockDim.x;
        if (t < nt) buf[t] = r[h];
      }
    };
    auto load_face = [&](const T* buf) {
      const T* c = buf + eb * ntx + ea;
      return dface(c[0], c[1], c[ntx], c[ntx + 1]);
    };
    T tdot = T(0);
    T pf[2];
    DFace<T> fl;
    DForce<T> pend{T(0), T(0), T(0), T(0)};
    stage1(k0 - 1, pf);
    __syncthreads();
    store1(pf, nb);
    stage1(k0, pf);
    int sl_next = stage_elem(k0 - 1, 0);
    const int K = k1 - k0;
    for (int kk = 0; kk <= K; ++kk) {
      const int ke = k0 - 1 + kk;
      T* b0 = nb + nt * (kk % 3);
      T* b1 = nb + nt * ((kk + 1) % 3);
      store1(pf, b1);
      const int sl = sl_next;
      if (kk < K) {
        stage1(ke + 2, pf);
        sl_next = stage_elem(ke + 1, (kk + 1) & 1);
        cp_async_wait<1>();  // this thread's copy of layer ke has landed
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      if (is_elem) {
        if (kk == 0) fl = load_face(b0);
        const DFace<T> fu = load_face(b1);
        const int gk = wrap_elem(ke, g.nz, g.pz);
        DForce<T> lo = pend;
        pend = DForce<T>{T(0), T(0), T(0), T(0)};
        if (eo >= 0 && gk >= 0) {
          T hq[kStageH];
          if (h_async) {
            load_chunks<T, kStageH>(HS + (size_t)(kk & 1) * kHChunks * exy * 16, exy, tid, hq);
          } else {
            const size_t e = plane_e * gk + eo;
#pragma unroll
            for (int q = 0; q < 8; ++q) hq[q] = a.H ? __ldg(a.H + 8 * e + q) : T(0);
          }
          damage_element(fl, fu, hq, wsc * a.gc_ell[sl], chw, a.gc_k2[sl], ek, lo, pend);
        }
        fl = fu;
        if (kk >= 1) {
          T c[4];
          dcorners(lo, c);
#pragma unroll
          for (int L = 0; L < 4; ++L) FC[L * exy + tid] = c[L];
        }
      }
      if (kk == 0) continue;  // the first element layer only fills pend
      __syncthreads();
      if (no >= 0) {
        const int e11 = (ni + 1) + ex * (nj + 1), e01 = ni + ex * (nj + 1);
        const int e10 = (ni + 1) + ex * nj, e00 = ni + ex * nj;
        const size_t n = plane_n * ke + no;
        T v = (FC[e11] + FC[exy + e01]) + (FC[2 * exy + e10] + FC[3 * exy + e00]);
        if (a.mask && __ldg(a.mask + n)) v = T(0);
        const T xn = b0[(nj + 1) * ntx + ni + 1];
        on_owned(n, xn, v);
        if (DOT) tdot += xn * v;
      }
    }
    if (DOT) accd += double(tdot);
  }
  return accd;
}

// Per-slot factors of the damage element, Gc / ell and 2 w Gc ell, formed once on
// the host in the order the element arithmetic would form them (same bits).
template <typename T>
void damage_slot_coefs(DTileArgs<T>& a, const VoxMat<T>& m) {
  const T w = T(a.g.w), ell = T(a.ell);
  // PF-CZM tangent: no mass term of its own, Gc (2 ell / pi) L
  const T lt = T(2.0 * a.ell / 3.14159265358979323846);
  for (int i = 0; i < PHASTB_MAX_SLOTS; ++i) {
    const T gc = m.Gc[i];
    a.gc_ell[i] = m.dform == 1 ? T(0) : gc / ell;
    a.gc_k2[i] = m.dform == 1 ? T(2) * w * gc * lt : T(2) * w * gc * ell;
  }
}

// The damage action as its own launch (MODE == kModeDot also x . y into ws.out[kOutDot]).
template <typename T, int MODE, int OX, int OY>
__device__ __forceinline__ void dtile_body(const DTileArgs<T>& a, const int vb, const int vgrid) {
  if (a.guard && *a.guard == 0) return;
  constexpr bool DOT = MODE == kModeDot;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const T* __restrict__ x = a.x;
  T* __restrict__ y = a.y;
  const double accd = dtile_pass<T, OX, OY, DOT>(
      a, smem_raw, [&](size_t n) { return __ldg(x + n); }, [&](size_t n, T, T v) { y[n] = v; }, vb, vgrid);
  if constexpr (DOT) {
    __shared__ double sh[32];
    const double sm = block_sum(accd, sh);
    if (threadIdx.x == 0) a.ws.part[kOutDot * kMaxPartials + vb] = sm;
    if (arrive_last_n(a.ws.counter, vgrid)) {
      const double t = fold_sum(a.ws.part + kOutDot * kMaxPartials, vgrid, sh);
      if (threadIdx.x == 0) {
        a.ws.out[kOutDot] = t;
        *a.ws.counter = 0u;
      }
    }
  }
}

template <typename T, int MODE, int OX, int OY>
__global__ void __launch_bounds__(kTileMaxThreads, 2) h8_dtile_kernel(DTileArgs<T> a) {
  dtile_body<T, MODE, OX, OY>(a, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------- persistent damage PCG

// A grid-barrier wait gives up after kBarLimitNs of the GPU's global timer (a
// normal wait is a few microseconds); kBarSpins polls of ~64 ns sleep bound it
// a second time, should the timer not advance.
constexpr unsigned long long kBarLimitNs = 2000000000ull;
constexpr unsigned kBarSpins = 1u << 26;

// Grid-wide barrier of a cooperative launch (every block resident).  The last
// block to arrive resets the count and advances the generation; the others
// poll the generation.  A wait that runs out (limit_ns of global time) sets
// st->grid_error, and every block that sees the error leaves the barrier with
// false, so the kernel ends instead of hanging.  gen: this block's copy of the
// generation (thread 0).
__device__ __forceinline__ bool grid_barrier(PcgState* st, unsigned& gen,
                                             unsigned long long limit_ns = kBarLimitNs) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned g0 = gen;
    __threadfence();
    if (atomicAdd(&st->bar_count, 1u) == gridDim.x - 1) {
      atomicExch(&st->bar_count, 0u);
      __threadfence();
      atomicAdd(&st->bar_gen, 1u);
    } else {
      const unsigned long long t0 = global_ns();
      unsigned spins = 0;
      while (*reinterpret_cast<volatile unsigned*>(&st->bar_gen) == g0) {
        if (++spins > kBarSpins || global_ns() - t0 > limit_ns ||
            *reinterpret_cast<volatile int*>(&st->grid_error)) {
          atomicExch(&st->grid_error, 1);
          ok = 0;
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
    gen = g0 + 1;
    s_ok = ok && !*reinterpret_cast<volatile int*>(&st->grid_error);
  }
  __syncthreads();
  return s_ok != 0;
}

// Self-test of the barrier's bounded wait: every block but `skip` arrives twice;
// with skip >= 0 the first wait of the others runs out after limit_ns and the
// kernel ends with st->grid_error set.
__global__ void grid_barrier_test_kernel(PcgState* st, int skip, unsigned long long limit_ns, int* passed) {
  if ((int)blockIdx.x == skip) return;
  unsigned gen = 0;
  if (!grid_barrier(st, gen, limit_ns)) return;
  if (!grid_barrier(st, gen, limit_ns)) return;
  if (threadIdx.x == 0) atomicAdd(passed, 1);
}

template <typename T>
struct DamagePcgArgs {
  int n, maxiter, mode, pad_;
  T *r, *z, *p, *p_alt, *Ap, *x;
  const T* inv_diag;
  double* part;  // 3 * kMaxPartials
  PcgState* st;
};

// Every iteration of a Jacobi-preconditioned CG on the damage operator in one
// cooperative launch, continuing from the state left by pcg_start_kernel:
//   A: p = z + beta p (formed while the bricks are staged; two direction
//      buffers, so a neighbour's halo never sees a new value), Ap, p . Ap
//   -- grid barrier --  alpha = rz / p.Ap  (every block folds the partials)
//   B: x += alpha p, r -= alpha Ap, z = r / diag, r . z, r . r
//   -- grid barrier --  beta, convergence: the state rules of
//      pcg_update_dot_kernel, evaluated identically in every block.
// Data written inside the launch is read through L2 (__ldcg).
template <typename T, int OX, int OY>
__global__ void __launch_bounds__(kTileMaxThreads, 2) h8_damage_pcg_kernel(DTileArgs<T> a, DamagePcgArgs<T> c) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[64];
  const int tid = threadIdx.x;
  PcgState S = *c.st;
  unsigned gen = S.bar_gen;
  const T* p_src = c.p;
  T* p_dst = c.p_alt;
  const int n = c.n;
  for (int it = 0; it < c.maxiter && S.active; ++it) {
    const T beta = T(S.beta);
    double pap = dtile_pass<T, OX, OY, true>(
        a, smem_raw, [&](size_t i) { return __ldcg(c.z + i) + beta * __ldcg(p_src + i); },
        [&](size_t i, T pn, T v) {
          c.Ap[i] = v;
          p_dst[i] = pn;
        },
        blockIdx.x, gridDim.x);
    pap = block_sum(pap, sh);
    if (tid == 0) c.part[blockIdx.x] = pap;
    if (!grid_barrier(c.st, gen)) return;
    const double PAP = fold_sum(c.part, gridDim.x, sh);
    const bool ok = isfinite(PAP) && PAP > 0.0;
    const double alpha = S.rz / PAP;
    const T al = T(alpha);
    double v2[2] = {0.0, 0.0};  // r . z, r . r
    if (ok) {
      for (int i = blockIdx.x * blockDim.x + tid; i < n; i += gridDim.x * blockDim.x) {
        c.x[i] = c.x[i] + al * __ldcg(p_dst + i);
        const T r = c.r[i] - al * __ldcg(c.Ap + i);
        c.r[i] = r;
        v2[1] += double(r) * double(r);
        const T z = c.inv_diag ? r * __ldg(c.inv_diag + i) : r;
        c.z[i] = z;
        v2[0] += double(r) * double(z);
      }
    }
    block_sum_multi<2>(v2, sh);
    if (tid == 0) {
      c.part[kMaxPartials + blockIdx.x] = v2[0];
      c.part[2 * kMaxPartials + blockIdx.x] = v2[1];
    }
    if (!grid_barrier(c.st, gen)) return;
    double f2[2];
    fold_sum_multi<2>(c.part + kMaxPartials, kMaxPartials, gridDim.x, f2, sh);
    const double RZ = f2[0], RR = f2[1];
    // the state rules of pcg_update_dot_kernel (Jacobi / identity, not PCG_PERIODIC)
    S.iter += 1;
    if (!ok) {
      if (!isfinite(PAP)) S.nonfinite = 1;
      if (!(PAP > 0.0)) S.breakdown = 1;
      S.active = 0;
    } else {
      S.alpha = alpha;
      S.steps += 1;
      if (!isfinite(RR) || !isfinite(RZ)) S.nonfinite = 1;
      S.rr = RR;
      if (!(RR > S.thr_sq)) {
        S.converged = 1;
        S.active = 0;
      } else {
        if (c.mode == PCG_STRICT && !(RZ > 0.0)) S.breakdown = 1;
        S.beta = (c.mode == PCG_STRICT) ? RZ / S.rz : ((S.rz > 0.0) ? RZ / S.rz : 0.0);
        S.rz = RZ;
      }
      if (S.breakdown || S.nonfinite) S.active = 0;
    }
    if (blockIdx.x == 0 && tid == 0) store_pcg_state(c.st, S);
    const T* t = p_src;
    p_src = p_dst;
    p_dst = const_cast<T*>(t);
  }
}

// ------------------------------------------------------------------ host side

namespace {

// Modes whose epilogue stages vectors of the owned nodes (see tile_layout's cheb).
constexpr bool mode_epi(int mode) { return mode == kModeCheb || mode == kModeRes || mode == kModeSmooth; }

std::mutex g_shape_mu;
std::map<std::tuple<int, int, int, int, int, int, int, int>, TileShape> g_shapes;

auto shape_key(const VoxGeom& g, int word, int cls) {
  return std::make_tuple(g.rx, g.ry, g.rz, g.px, g.py, g.pz, word, cls);
}

// Shape of the damage kernels' bricks (class 2): among owned-node tiles of <= kTileMaxThreads element
// threads, prefer shapes whose sides divide the grid (no ragged tiles) and the least recomputed halo; the z
// depth is left to the launch (kz = 0, launch_kz).
TileShape heuristic_shape(const VoxGeom& g) {
  static const int cand[][2] = {{16, 12}, {12, 16}, {14, 14}, {24, 8}, {16, 8}, {8, 16}, {20, 8}, {32, 4},
                                {12, 12}, {10, 10}, {8, 8},   {6, 6},   {4, 4},  {2, 2},  {1, 1}};
  TileShape best{1, 1, 1};
  double best_cost = 1e300;
  for (const auto& c : cand) {
    TileShape t{std::min(c[0], g.rx), std::min(c[1], g.ry), 1};
    if (!tile_ok(t)) continue;
    const int tx = (g.rx + t.ox - 1) / t.ox, ty = (g.ry + t.oy - 1) / t.oy;
    // element-thread slots launched per node layer / useful nodes per layer
    const double cost = double(tx) * ty * tile_threads(t) / (double(g.rx) * g.ry);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = t;
    }
  }
  best.kz = 0;
  return best;
}

// Z depth of a damage tile whose shape leaves it to the launch (kz = 0), from the
// number of blocks that can be resident at once (`capacity`): the fewest
// rounds of resident blocks, each round costing one tile's kz + 1 element
// layers plus its two-layer prologue.  A power-of-two depth leaves a second,
// mostly idle round on e.g. 64^3 (512 tiles of kz = 4 for 444 resident blocks);
// kz = 5 runs 416 tiles in one round.
int launch_kz(long long tiles_xy, int rz, long long capacity) {
  int best = 1;
  double best_cost = 1e300;
  for (int kz = 1; kz <= rz; ++kz) {
    const long long tiles = tiles_xy * ((rz + kz - 1) / kz);
    const double cost = double((tiles + capacity - 1) / capacity) * (kz + 2);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = kz;
    }
  }
  return best;
}

// Modelled time of an elastic march: `tiles` bricks of kz node layers and `warps` warps, per_sm of them resident
// on each of `sms` SMs.  A round of resident bricks runs kz + 1 element layers plus a prologue of about one;
// a layer costs a fixed latency (two barriers and the element's dependent chain) and issue time in proportion
// to the warps that share a scheduler.  The coefficients (microseconds) come from sweeps of shape and depth and are
// there to rank them: on 64^3 the model gives 20.8 us for FP32 16 x 8 x 5 (measured 24.6), 23.8 for 16 x 8 x 6 (26.7),
// 29.0 for 16 x 8 x 4 (28.9), and in FP64 29.0 for 16 x 14 x 10 (32.9), 43.0 for 16 x 8 x 16 (43.1).
double march_cost(int word, int warps, long long tiles, int per_sm, int sms, int kz) {
  const double a = word == 4 ? 0.82 : 1.5, b = word == 4 ? 0.5 : 0.42;
  const long long cap = std::min<long long>((long long)per_sm * sms, kMaxPartials);
  const long long full = tiles / cap, rem = tiles % cap;
  // (the last term prefers fewer warps between equals)
  auto layer = [&](long long blocks) {
    return a + b * double((blocks * warps + 3) / 4) + 0.01 * double(blocks * warps);
  };
  double c = double(full) * layer((cap + sms - 1) / sms);
  if (rem) c += layer((rem + sms - 1) / sms);
  return c * (kz + 2);
}

// The depth with the least modelled time; its cost through *cost.  Only depths that lower the number of
// z slabs differ in their bricks, so one depth per slab count is looked at.
int mech_kz(int word, int threads, long long tiles_xy, int rz, int per_sm, int sms, double* cost = nullptr) {
  int best = 1;
  double best_cost = 1e300;
  for (int slabs = 1; slabs <= rz; ++slabs) {
    const int kz = (rz + slabs - 1) / slabs;
    const int used = (rz + kz - 1) / kz;
    if (used < slabs) continue;  // the same depth as fewer slabs
    const double c = march_cost(word, threads / 32, tiles_xy * used, per_sm, sms, kz);
    if (c < best_cost - 1e-9) {
      best_cost = c;
      best = kz;
    }
  }
  if (cost) *cost = best_cost;
  return best;
}

// Shape of the elastic action's bricks (classes 0 and 1): the least modelled time.  In FP64 one block of up to
// 256 threads fits an SM, so a shape that fills its eight warps wins (192^3: 16 x 14 508 us, 16 x 8 with five
// warps 805 us); in FP32 about sixteen warps fit either way (285 against 302 us) and the ragged rest of the
// grid decides.  Shapes without a kernel of their own run the one with run-time offsets, about a tenth slower.
TileShape mech_shape(const VoxGeom& g, int word) {
  static const int cand[][2] = {{16, 14}, {16, 8}, {14, 7}, {8, 8}, {16, 12}, {15, 15}, {14, 14}, {12, 12}, {10, 10}};
  constexpr int kSms = 148;
  TileShape best{1, 1, 0};
  double best_cost = 1e300;
  for (const auto& c : cand) {
    const TileShape t{std::min(c[0], g.rx), std::min(c[1], g.ry), 0};
    if (!tile_ok(t)) continue;
    const int threads = tile_threads(t);
    const int per_sm = word == 4 ? 512 / threads : (threads > 128 ? 1 : 256 / threads);
    const long long tiles = (long long)((g.rx + t.ox - 1) / t.ox) * ((g.ry + t.oy - 1) / t.oy);
    double cost;
    mech_kz(word, threads, tiles, g.rz, per_sm, kSms, &cost);
    const bool own = (t.ox == 16 && (t.oy == 14 || t.oy == 8)) || (t.ox == 14 && t.oy == 7) || (t.ox == 8 && t.oy == 8);
    if (!own) cost *= 1.1;
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = t;
    }
  }
  return best;
}

// TMA staging of the elastic action's node layers (PHASTB_TMA=1 turns it on).
bool tma_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("PHASTB_TMA");
    return e && e[0] == '1';
  }();
  return on;
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// Tensor maps of u~ (a (3 rx, ry, rz) array) and d ((rx, ry, rz)) for the TMA
// staging of a launch; false (cp.async instead) when TMA is off,
// the row strides are not multiples of 16 bytes (rx a multiple of 16 / sizeof(T)),
// a buffer is not 16-byte aligned, or the driver refuses a map.
template <typename T>
bool tile_tensor_maps(const TileArgs<T>& a, CUtensorMap* mx, CUtensorMap* md) {
  std::memset(mx, 0, sizeof(*mx));
  std::memset(md, 0, sizeof(*md));
  if (!tma_enabled()) return false;
  const VoxGeom& v = a.g;
  const int A = 16 / (int)sizeof(T);
  if (v.rx % A != 0) return false;
  if ((reinterpret_cast<uintptr_t>(a.x) & 15u) || (a.d && (reinterpret_cast<uintptr_t>(a.d) & 15u))) return false;
  const int W = tma_wx<T>(a.ts.ox), Wd = tma_wd<T>(a.ts.ox), rows = a.ts.oy + 2;
  if (W > 256 || Wd > 256 || rows > 256) return false;
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const CUtensorMapDataType dt = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  const cuuint32_t es[3] = {1, 1, 1};
  {
    const cuuint64_t dims[3] = {3ull * (cuuint64_t)v.rx, (cuuint64_t)v.ry, (cuuint64_t)v.rz};
    const cuuint64_t strides[2] = {3ull * v.rx * sizeof(T), 3ull * v.rx * v.ry * sizeof(T)};
    const cuuint32_t box[3] = {(cuuint32_t)W, (cuuint32_t)rows, 1};
    if (enc(mx, dt, 3, const_cast<T*>(a.x), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  if (a.d) {
    const cuuint64_t dims[3] = {(cuuint64_t)v.rx, (cuuint64_t)v.ry, (cuuint64_t)v.rz};
    const cuuint64_t strides[2] = {(cuuint64_t)v.rx * sizeof(T), (cuuint64_t)v.rx * v.ry * sizeof(T)};
    const cuuint32_t box[3] = {(cuuint32_t)Wd, (cuuint32_t)rows, 1};
    if (enc(md, dt, 3, const_cast<T*>(a.d), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  return true;
}

template <typename T, int COEF, int MODE, int OX, int OY, bool TMA>
int launch_variant_t(const TileArgs<T>& a, const VoxMat<T>& m, cudaStream_t s, const CUtensorMap& mx,
                     const CUtensorMap& md) {
  auto kern = h8_tile_kernel<T, COEF, MODE, OX, OY, TMA>;
  size_t off_face = 0, off_qp = 0, off_cheb = 0;
  const size_t smem = TMA ? tile_layout_tma<T>(a.ts.ox, a.ts.oy, COEF == kCoefQP, mode_epi(MODE), &off_face,
                                               &off_qp, &off_cheb)
                          : tile_layout<T>(a.ts.ox, a.ts.oy, COEF == kCoefQP, mode_epi(MODE), &off_qp, &off_cheb);
  const int threads = tile_threads(a.ts);
  static std::mutex mu;
  static size_t smem_set = 0;
  static std::map<std::pair<int, size_t>, int> occ;  // (threads, smem) -> resident blocks per SM
  int per_sm = 1;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (smem > smem_set) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return PHASTB_ERR_CUDA;
      }
      smem_set = smem;
    }
    auto it = occ.find({threads, smem});
    if (it == occ.end()) {
      int b = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        b = 1;
      }
      it = occ.emplace(std::make_pair(threads, smem), b < 1 ? 1 : b).first;
    }
    per_sm = it->second;
  }
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const VoxGeom& v = a.g;
  const long long tiles_xy = (long long)((v.rx + a.ts.ox - 1) / a.ts.ox) * ((v.ry + a.ts.oy - 1) / a.ts.oy);
  const long long cap = std::min<long long>((long long)per_sm * sms, kMaxPartials);
  TileArgs<T> b = a;
  if (b.ts.kz <= 0) b.ts.kz = mech_kz((int)sizeof(T), threads, tiles_xy, v.rz, per_sm, sms);
  const long long n_tiles = tiles_xy * ((v.rz + b.ts.kz - 1) / b.ts.kz);
  const long long grid = std::min<long long>(n_tiles, cap);
  { note_launch(); kern<<<(int)grid, threads, smem, s>>>(b, m, mx, md); }
  return last_launch_status();
}

template <typename T, int COEF, int MODE, int OX, int OY>
int launch_variant(const TileArgs<T>& a, const VoxMat<T>& m, cudaStream_t s) {
  CUtensorMap mx, md;
  const bool tma = tile_tensor_maps<T>(a, &mx, &md);
  if (tma) {  // opt-in: compiled for 16 x 8 bricks and for any shape
    constexpr bool own = OX == 16 && OY == 8;
    return launch_variant_t<T, COEF, MODE, own ? OX : 0, own ? OY : 0, true>(a, m, s, mx, md);
  }
  return launch_variant_t<T, COEF, MODE, OX, OY, false>(a, m, s, mx, md);
}

}  // namespace

bool tile_shape_lookup(const VoxGeom& g, int word, int cls, TileShape* t) {
  std::lock_guard<std::mutex> lk(g_shape_mu);
  auto it = g_shapes.find(shape_key(g, word, cls));
  if (it == g_shapes.end()) return false;
  *t = it->second;
  return true;
}

TileShape tile_shape_for(const VoxGeom& g, int word, int cls) {
  TileShape t;
  if (tile_shape_lookup(g, word, cls, &t)) return t;
  if (cls == 2) return heuristic_shape(g);
  // the model's choice, remembered per host thread: it depends on the grid alone
  using Key = decltype(shape_key(g, word, cls));
  static thread_local std::vector<std::pair<Key, TileShape>> seen;
  const Key key = shape_key(g, word, 0);
  for (const auto& s : seen)
    if (s.first == key) return s.second;
  if (seen.size() >= 64) seen.clear();
  t = mech_shape(g, word);
  seen.emplace_back(key, t);
  return t;
}

void tile_shape_record(const VoxGeom& g, int word, int cls, const TileShape& t) {
  std::lock_guard<std::mutex> lk(g_shape_mu);
  g_shapes[shape_key(g, word, cls)] = t;
}

namespace {

// Lazy tuning is opt-in (PHASTB_AUTOTUNE=1): shapes picked by timing can differ
// between processes, and the tile shape sets the grouping of the fused dot
// products, so only the deterministic heuristic keeps runs bit-reproducible.
// On the 64^3 cell the heuristic's shapes are also faster inside the solver
// than the ones timed in isolation.
bool autotune_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("PHASTB_AUTOTUNE");
    return e && e[0] == '1';
  }();
  return on;
}

TileShape clamp_shape(TileShape t, const VoxGeom& v) {
  t.ox = std::min(t.ox, v.rx);
  t.oy = std::min(t.oy, v.ry);
  t.kz = std::min(t.kz, v.rz);
  return t;
}

// The hot variants are also compiled for a few fixed tile shapes (every
// shared-memory offset then becomes a constant); other shapes run the generic
// kernel.
template <typename T, int COEF, int MODE>
int by_shape(const TileArgs<T>& a, const VoxMat<T>& m, cudaStream_t s) {
  const int ox = a.ts.ox, oy = a.ts.oy;
  if (ox == 16 && oy == 14) return launch_variant<T, COEF, MODE, 16, 14>(a, m, s);
  if (ox == 16 && oy == 8) return launch_variant<T, COEF, MODE, 16, 8>(a, m, s);
  if (ox == 14 && oy == 7) return launch_variant<T, COEF, MODE, 14, 7>(a, m, s);
  if (ox == 8 && oy == 8) return launch_variant<T, COEF, MODE, 8, 8>(a, m, s);
  return launch_variant<T, COEF, MODE, 0, 0>(a, m, s);
}

template <typename T>
int dispatch(const TileArgs<T>& a, const VoxMat<T>& m, int coef, int mode, cudaStream_t s) {
  switch (coef * 8 + mode) {
    case kCoefIso * 8 + kModeApply: return by_shape<T, kCoefIso, kModeApply>(a, m, s);
    case kCoefIso * 8 + kModeDot: return by_shape<T, kCoefIso, kModeDot>(a, m, s);
    case kCoefIso * 8 + kModeEnergy: return launch_variant<T, kCoefIso, kModeEnergy, 0, 0>(a, m, s);
    case kCoefIso * 8 + kModeCheb: return by_shape<T, kCoefIso, kModeCheb>(a, m, s);
    case kCoefIso * 8 + kModeNodal: return by_shape<T, kCoefIso, kModeNodal>(a, m, s);
    case kCoefIso * 8 + kModeRes: return by_shape<T, kCoefIso, kModeRes>(a, m, s);
    case kCoefIso * 8 + kModeSmooth: return by_shape<T, kCoefIso, kModeSmooth>(a, m, s);
    case kCoefAniso * 8 + kModeRes: return launch_variant<T, kCoefAniso, kModeRes, 0, 0>(a, m, s);
    case kCoefAniso * 8 + kModeSmooth: return launch_variant<T, kCoefAniso, kModeSmooth, 0, 0>(a, m, s);
    case kCoefQP * 8 + kModeRes: return by_shape<T, kCoefQP, kModeRes>(a, m, s);
    case kCoefQP * 8 + kModeSmooth: return by_shape<T, kCoefQP, kModeSmooth>(a, m, s);
    case kCoefAniso * 8 + kModeApply: return launch_variant<T, kCoefAniso, kModeApply, 0, 0>(a, m, s);
    case kCoefAniso * 8 + kModeDot: return launch_variant<T, kCoefAniso, kModeDot, 0, 0>(a, m, s);
    case kCoefAniso * 8 + kModeEnergy: return launch_variant<T, kCoefAniso, kModeEnergy, 0, 0>(a, m, s);
    case kCoefAniso * 8 + kModeCheb: return launch_variant<T, kCoefAniso, kModeCheb, 0, 0>(a, m, s);
    case kCoefAniso * 8 + kModeNodal: return launch_variant<T, kCoefAniso, kModeNodal, 0, 0>(a, m, s);
    case kCoefQP * 8 + kModeApply: return by_shape<T, kCoefQP, kModeApply>(a, m, s);
    case kCoefQP * 8 + kModeCheb: return by_shape<T, kCoefQP, kModeCheb>(a, m, s);
    default: return PHASTB_ERR_ARG;
  }
}

// Times the (coef, mode) launch of `a` over the candidate shapes (a's outputs
// are overwritten; modes that update their inputs in place are not timed).
template <typename T>
int tune_shape(TileArgs<T> a, const VoxMat<T>& m, int coef, int mode, cudaStream_t s, TileShape* best_out,
               float* best_ms) {
  static const int cand[][2] = {{16, 8}, {32, 4},  {8, 8},   {8, 4},   {4, 4},   {16, 12}, {12, 16},
                                {14, 14}, {24, 8}, {20, 8}, {12, 12}, {10, 10}, {6, 6},   {2, 4}};
  static const int kzs[] = {0, 1, 2, 4, 8, 16};  // 0: chosen at launch
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return PHASTB_ERR_CUDA;
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return PHASTB_ERR_CUDA;
  }
  int st = PHASTB_OK;
  float best = 1e30f;
  TileShape bs = clamp_shape(mech_shape(a.g, (int)sizeof(T)), a.g);
  std::vector<TileShape> seen;
  for (const auto& c : cand) {
    for (int kz : kzs) {
      const TileShape t = clamp_shape(TileShape{c[0], c[1], kz}, a.g);
      if (!tile_ok(t)) continue;
      bool dup = false;
      for (const auto& q : seen) dup |= (q.ox == t.ox && q.oy == t.oy && q.kz == t.kz);
      if (dup) continue;
      seen.push_back(t);
      a.ts = t;
      if ((st = dispatch<T>(a, m, coef, mode, s))) break;
      const int reps = 3;
      cudaEventRecord(e0, s);
      for (int r = 0; r < reps && !st; ++r) st = dispatch<T>(a, m, coef, mode, s);
      cudaEventRecord(e1, s);
      if (st || (st = cuda_status(cudaEventSynchronize(e1)))) break;
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      ms /= reps;
      if (ms < best) {
        best = ms;
        bs = t;
      }
    }
    if (st) break;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (st) return st;
  *best_out = bs;
  if (best_ms) *best_ms = best;
  return PHASTB_OK;
}

}  // namespace

template <typename T>
TileArgs<T> tile_args(const VoxGeom& v, int cls) {
  TileArgs<T> a;
  std::memset(&a, 0, sizeof(a));
  a.g = v;
  a.ts = clamp_shape(tile_shape_for(v, (int)sizeof(T), cls), v);
  a.k.c1 = T(kC1);
  a.k.c2 = T(kC2);
  set_modal_k(a.k, v);
  return a;
}

template <typename T>
int h8_tile_launch(const TileArgs<T>& a, const VoxMat<T>& m, int coef, int mode, cudaStream_t s, bool tune) {
  if (!tile_ok(a.ts) || a.ts.ox > a.g.rx || a.ts.oy > a.g.ry || a.ts.kz > a.g.rz) return PHASTB_ERR_ARG;
  const int cls = coef == kCoefQP ? 1 : 0;
  TileShape known;
  if (tune && autotune_enabled() && (mode == kModeApply || mode == kModeDot) && a.guard == nullptr &&
      !tile_shape_lookup(a.g, (int)sizeof(T), cls, &known)) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone) {
      TileShape best;
      int st = tune_shape<T>(a, m, coef, mode, s, &best, nullptr);
      if (st) return st;
      tile_shape_record(a.g, (int)sizeof(T), cls, best);
      TileArgs<T> b = a;
      b.ts = best;
      return dispatch<T>(b, m, coef, mode, s);
    }
    cudaGetLastError();
  }
  return dispatch<T>(a, m, coef, mode, s);
}

template <typename T>
int h8_mech_tile_launch(const VoxGeom& v, const VoxMat<T>& m, const uint8_t* slot, const T* x, const T* gq,
                        const T* d, const uint8_t* mask, T* y, RedWs ws, const int* guard, bool dot, bool energy,
                        cudaStream_t s, const TileShape* force_shape) {
  TileArgs<T> a = tile_args<T>(v, 0);
  if (force_shape) a.ts = clamp_shape(*force_shape, v);
  a.slot = slot;
  a.gq = gq;
  a.d = d;
  a.x = x;
  a.y = y;
  a.mask = mask;
  a.ws = ws;
  a.guard = guard;
  const int coef = m.iso ? kCoefIso : kCoefAniso;
  return h8_tile_launch<T>(a, m, coef, dot ? kModeDot : (energy ? kModeEnergy : kModeApply), s, !force_shape);
}

template <typename T, int MODE, int OX, int OY>
int dlaunch_variant(const DTileArgs<T>& a, cudaStream_t s) {
  auto kern = h8_dtile_kernel<T, MODE, OX, OY>;
  const int nt = (a.ts.ox + 2) * (a.ts.oy + 2), exy = (a.ts.ox + 1) * (a.ts.oy + 1);
  const size_t smem = tile_stage_offset<T>(nt, exy, 3, 4) + sizeof(T) * 2 * kStageH * (size_t)exy;
  const int threads = tile_threads(a.ts);
  static std::mutex mu;
  static size_t smem_set = 0;
  static std::map<std::pair<int, size_t>, int> occ;
  int per_sm = 1;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (smem > smem_set) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return PHASTB_ERR_CUDA;
      }
      smem_set = smem;
    }
    auto it = occ.find({threads, smem});
    if (it == occ.end()) {
      int b = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        b = 1;
      }
      it = occ.emplace(std::make_pair(threads, smem), b < 1 ? 1 : b).first;
    }
    per_sm = it->second;
  }
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const VoxGeom& v = a.g;
  const long long tiles_xy = (long long)((v.rx + a.ts.ox - 1) / a.ts.ox) * ((v.ry + a.ts.oy - 1) / a.ts.oy);
  const long long cap = std::min<long long>((long long)per_sm * sms, kMaxPartials);
  DTileArgs<T> b = a;
  if (b.ts.kz <= 0) b.ts.kz = launch_kz(tiles_xy, v.rz, cap);
  const long long n_tiles = tiles_xy * ((v.rz + b.ts.kz - 1) / b.ts.kz);
  const long long grid = std::min<long long>(n_tiles, cap);
  { note_launch(); kern<<<(int)grid, threads, smem, s>>>(b); }
  return last_launch_status();
}

template <typename T, int MODE>
int dby_shape(const DTileArgs<T>& a, cudaStream_t s) {
  const int ox = a.ts.ox, oy = a.ts.oy;
  if (ox == 16 && oy == 8) return dlaunch_variant<T, MODE, 16, 8>(a, s);
  if (ox == 32 && oy == 4) return dlaunch_variant<T, MODE, 32, 4>(a, s);
  if (ox == 8 && oy == 8) return dlaunch_variant<T, MODE, 8, 8>(a, s);
  return dlaunch_variant<T, MODE, 0, 0>(a, s);
}

template <typename T, int OX, int OY>
int dpcg_variant(const DTileArgs<T>& a0, const DamagePcgArgs<T>& c0, cudaStream_t s) {
  auto kern = h8_damage_pcg_kernel<T, OX, OY>;
  const int nt = (a0.ts.ox + 2) * (a0.ts.oy + 2), exy = (a0.ts.ox + 1) * (a0.ts.oy + 1);
  const size_t smem = tile_stage_offset<T>(nt, exy, 3, 4) + sizeof(T) * 2 * kStageH * (size_t)exy;
  const int threads = tile_threads(a0.ts);
  static std::mutex mu;
  static size_t smem_set = 0;
  static std::map<std::pair<int, size_t>, int> occ;
  int per_sm = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (smem > smem_set) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return PHASTB_UNSUPPORTED;
      }
      smem_set = smem;
    }
    auto it = occ.find({threads, smem});
    if (it == occ.end()) {
      int b = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        b = 0;
      }
      it = occ.emplace(std::make_pair(threads, smem), b).first;
    }
    per_sm = it->second;
  }
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  if (!coop || per_sm < 1 || sms < 1) return PHASTB_UNSUPPORTED;
  const VoxGeom& v = a0.g;
  const long long tiles_xy = (long long)((v.rx + a0.ts.ox - 1) / a0.ts.ox) * ((v.ry + a0.ts.oy - 1) / a0.ts.oy);
  // every block must be resident at once (the grid barriers wait for all of them)
  const long long cap = std::min<long long>((long long)per_sm * sms, kMaxPartials);
  DTileArgs<T> a = a0;
  if (a.ts.kz <= 0) a.ts.kz = launch_kz(tiles_xy, v.rz, cap);
  const long long n_tiles = tiles_xy * ((v.rz + a.ts.kz - 1) / a.ts.kz);
  const int grid = (int)std::min<long long>(n_tiles, cap);
  DamagePcgArgs<T> c = c0;
  void* args[] = {&a, &c};
  if (cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(threads), args, smem, s) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  note_launch();
  return PHASTB_OK;
}

// PHASTB_PERSISTENT_PCG=0 runs the damage CG as separate launches per iteration.
bool persistent_pcg_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("PHASTB_PERSISTENT_PCG");
    return !(e && e[0] == '0');
  }();
  return on;
}

template <typename T>
int h8_damage_tile_launch(const VoxGeom& v, const VoxMat<T>& m, const uint8_t* slot, const T* x, const T* H,
                          double scale, const uint8_t* mask, T* y, RedWs ws, const int* guard, bool dot,
                          cudaStream_t s) {
  DTileArgs<T> a;
  std::memset(&a, 0, sizeof(a));
  const TileArgs<T> base = tile_args<T>(v, 2);
  a.g = v;
  a.ts = base.ts;
  a.slot = slot;
  a.kappa = double(m.kappa);
  a.ell = double(m.ell);
  damage_slot_coefs(a, m);
  a.scale = scale;
  a.H = H;
  a.x = x;
  a.y = y;
  a.mask = mask;
  a.ws = ws;
  a.guard = guard;
  if (!tile_ok(a.ts)) return PHASTB_ERR_ARG;
  auto run = [&](const DTileArgs<T>& b) { return dot ? dby_shape<T, kModeDot>(b, s) : dby_shape<T, kModeApply>(b, s); };
  TileShape known;
  if (autotune_enabled() && guard == nullptr && !tile_shape_lookup(v, (int)sizeof(T), 2, &known)) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone) {
      // time the candidate shapes on this call's buffers (y is recomputed below)
      static const int cand[][2] = {{16, 8}, {32, 4}, {8, 8}, {16, 12}, {14, 14}, {10, 10}, {8, 4}, {4, 4}};
      static const int kzs[] = {0, 2, 4, 8, 16};  // 0: chosen at launch
      cudaEvent_t e0, e1;
      if (cudaEventCreate(&e0) != cudaSuccess) return PHASTB_ERR_CUDA;
      if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return PHASTB_ERR_CUDA;
      }
      int st = PHASTB_OK;
      float best = 1e30f;
      TileShape bs = a.ts;
      DTileArgs<T> b = a;
      for (const auto& c : cand) {
        for (int kz : kzs) {
          b.ts = clamp_shape(TileShape{c[0], c[1], kz}, v);
          if (!tile_ok(b.ts)) continue;
          if ((st = run(b))) break;
          cudaEventRecord(e0, s);
          for (int r = 0; r < 3 && !st; ++r) st = run(b);
          cudaEventRecord(e1, s);
          if (st || (st = cuda_status(cudaEventSynchronize(e1)))) break;
          float ms = 0.f;
          cudaEventElapsedTime(&ms, e0, e1);
          if (ms < best) {
            best = ms;
            bs = b.ts;
          }
        }
        if (st) break;
      }
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      if (st) return st;
      tile_shape_record(v, (int)sizeof(T), 2, bs);
      a.ts = bs;
    } else {
      cudaGetLastError();
    }
  }
  return run(a);
}

template int h8_damage_tile_launch<double>(const VoxGeom&, const VoxMat<double>&, const uint8_t*, const double*,
                                           const double*, double, const uint8_t*, double*, RedWs, const int*, bool,
                                           cudaStream_t);
template int h8_damage_tile_launch<float>(const VoxGeom&, const VoxMat<float>&, const uint8_t*, const float*,
                                          const float*, double, const uint8_t*, float*, RedWs, const int*, bool,
                                          cudaStream_t);

template <typename T>
int h8_damage_pcg_launch(const VoxGeom& v, const VoxMat<T>& m, const uint8_t* slot, const T* H, double scale,
                         const uint8_t* mask, const PcgWs<T>& w, T* p_alt, T* x, const T* inv_diag, int maxiter,
                         int mode, cudaStream_t s, void* tagged) {
  if (mode == PCG_PERIODIC || !persistent_pcg_enabled()) return PHASTB_UNSUPPORTED;
  DTileArgs<T> a;
  std::memset(&a, 0, sizeof(a));
  const TileArgs<T> base = tile_args<T>(v, 2);
  a.g = v;
  a.ts = base.ts;
  a.slot = slot;
  a.kappa = double(m.kappa);
  a.ell = double(m.ell);
  damage_slot_coefs(a, m);
  a.scale = scale;
  a.H = H;
  a.mask = mask;
  if (!tile_ok(a.ts)) return PHASTB_ERR_ARG;
  if (tagged) {
    const int st = h8_damage_brick_pcg<T>(a, w, tagged, x, inv_diag, maxiter, mode, s);
    if (st != PHASTB_UNSUPPORTED) return st;
  }
  DamagePcgArgs<T> c;
  std::memset(&c, 0, sizeof(c));
  c.n = v.n_red;
  c.maxiter = maxiter;
  c.mode = mode;
  c.r = w.r;
  c.z = w.z;
  c.p = w.p;
  c.p_alt = p_alt;
  c.Ap = w.Ap;
  c.x = x;
  c.inv_diag = inv_diag;
  c.part = w.part;
  c.st = w.st;
  const int ox = a.ts.ox, oy = a.ts.oy;
  if (ox == 16 && oy == 8) return dpcg_variant<T, 16, 8>(a, c, s);
  if (ox == 32 && oy == 4) return dpcg_variant<T, 32, 4>(a, c, s);
  if (ox == 8 && oy == 8) return dpcg_variant<T, 8, 8>(a, c, s);
  return dpcg_variant<T, 0, 0>(a, c, s);
}

template int h8_damage_pcg_launch<double>(const VoxGeom&, const VoxMat<double>&, const uint8_t*, const double*,
                                          double, const uint8_t*, const PcgWs<double>&, double*, double*,
                                          const double*, int, int, cudaStream_t, void*);
template int h8_damage_pcg_launch<float>(const VoxGeom&, const VoxMat<float>&, const uint8_t*, const float*,
                                         double, const uint8_t*, const PcgWs<float>&, float*, float*, const float*,
                                         int, int, cudaStream_t, void*);
// ------------------------------------------------------------ packed cell batches

template <typename T>
__device__ __forceinline__ TileK<T> batch_k(const BatchCell& c) {
  if constexpr (sizeof(T) == 4)
    return c.kf;
  else
    return c.kd;
}

// One brick of one cell per block: the block builds its cell's arguments in shared
// memory and runs the single-grid tile body with its brick index inside the cell.
template <typename T, int MODE, int OX, int OY, int COEF = kCoefIso>
__global__ void __launch_bounds__(TileBounds<T, OX, OY>::threads, TileBounds<T, OX, OY>::blocks)
    h8_tile_batch_kernel(TileBatchArgs<T> b, VoxMat<T> m) {
  __shared__ TileArgs<T> sa;
  const int2 wk = b.work[blockIdx.x];
  const BatchCell& c = b.cells[wk.x];
  if (threadIdx.x == 0) {
    TileArgs<T> a;
    a.g = c.g;
    a.ts = c.ts;
    a.pad_ = 0;
    a.slot = b.slot ? b.slot + c.elem_off : nullptr;
    a.gq = nullptr;
    a.d = b.d ? b.d + c.node_off : nullptr;
    a.lam_q = b.lam_q ? b.lam_q + 8 * c.elem_off : nullptr;
    a.mu_q = b.mu_q ? b.mu_q + 8 * c.elem_off : nullptr;
    a.x = b.x + c.mech_off;
    a.y = b.y ? b.y + c.mech_off : nullptr;
    a.mask = b.mask ? b.mask + c.mech_off : nullptr;
    a.res = b.res ? b.res + c.mech_off : nullptr;
    a.invd = b.invd ? b.invd + c.mech_off : nullptr;
    a.xs = b.xs ? b.xs + c.mech_off : nullptr;
    a.d_out = b.d_out ? b.d_out + c.mech_off : nullptr;
    a.c1 = b.c1;
    a.c2 = b.c2 * (b.c2_scale ? b.c2_scale[wk.x] : 1.0);
    const long long e6 = c.mech_off + 3LL * c.g.n_red;
    a.e_diag = b.e_diag ? b.e_diag + e6 : nullptr;
    a.e_fixed = b.e_fixed ? b.e_fixed + e6 : nullptr;
    a.ws = b.ws ? red_ws(b.ws + (size_t)wk.x * red_ws_bytes()) : RedWs{nullptr, nullptr, nullptr};
    a.guard = b.guard ? b.guard + (size_t)wk.x * b.guard_stride : nullptr;
    a.k = batch_k<T>(c);
    sa = a;
  }
  __syncthreads();
  tile_body<T, COEF, MODE, OX, OY, false>(sa, m, nullptr, nullptr, wk.y, c.nvb);
}

template <typename T, int MODE, int OX, int OY>
__global__ void __launch_bounds__(kTileMaxThreads, 2) h8_dtile_batch_kernel(TileBatchArgs<T> b, VoxMat<T> m) {
  __shared__ DTileArgs<T> sa;
  const int2 wk = b.work[blockIdx.x];
  const BatchCell& c = b.cells[wk.x];
  if (threadIdx.x == 0) {
    DTileArgs<T> a;
    a.g = c.g;
    a.ts = c.ts;
    a.pad_ = 0;
    a.slot = b.slot + c.elem_off;
    // per-slot factors in the order of damage_slot_coefs (same bits as a single-cell launch)
    const T w = T(c.g.w), ell = T(c.ell);
    for (int i = 0; i < PHASTB_MAX_SLOTS; ++i) {
      const T gc = m.Gc[i];
      a.gc_ell[i] = gc / ell;
      a.gc_k2[i] = T(2) * w * gc * ell;
    }
    a.kappa = b.kappa;
    a.ell = c.ell;
    a.scale = b.dscale ? c.dscale : 1.0;
    a.H = b.H ? b.H + 8 * c.elem_off : nullptr;
    a.x = b.x + c.node_off;
    a.y = b.y + c.node_off;
    a.mask = b.mask ? b.mask + c.node_off : nullptr;
    a.ws = red_ws(b.ws + (size_t)wk.x * red_ws_bytes());
    a.guard = b.guard ? b.guard + (size_t)wk.x * b.guard_stride : nullptr;
    sa = a;
  }
  __syncthreads();
  dtile_body<T, MODE, OX, OY>(sa, wk.y, c.nvb);
}

namespace {

template <class K>
int batch_smem_attr(K kern, size_t smem) {
  static std::mutex mu;
  static std::map<const void*, size_t> set;
  std::lock_guard<std::mutex> lk(mu);
  auto it = set.find((const void*)kern);
  if (it != set.end() && it->second >= smem) return PHASTB_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_ERR_CUDA;
  }
  set[(const void*)kern] = smem;
  return PHASTB_OK;
}

template <typename T, int MODE, int OX, int OY>
int tile_batch_variant(const TileBatchArgs<T>& b, const VoxMat<T>& m, cudaStream_t s) {
  auto kern = h8_tile_batch_kernel<T, MODE, OX, OY>;
  size_t oq = 0, oc = 0;
  const size_t smem = tile_layout<T>(OX, OY, false, false, &oq, &oc);
  int st = batch_smem_attr(kern, smem);
  if (st) return st;
  const int threads = ((OX + 1) * (OY + 1) + 31) / 32 * 32;
  { note_launch(); kern<<<b.n_blocks, threads, smem, s>>>(b, m); }
  return last_launch_status();
}

template <int COEF, int MODE, int OX, int OY>
int tile_batch_level_variant(const TileBatchArgs<float>& b, const VoxMat<float>& m, cudaStream_t s) {
  auto kern = h8_tile_batch_kernel<float, MODE, OX, OY, COEF>;
  size_t oq = 0, oc = 0;
  const size_t smem = tile_layout<float>(OX, OY, COEF == kCoefQP, mode_epi(MODE), &oq, &oc);
  int st = batch_smem_attr(kern, smem);
  if (st) return st;
  const int threads = ((OX + 1) * (OY + 1) + 31) / 32 * 32;
  { note_launch(); kern<<<b.n_blocks, threads, smem, s>>>(b, m); }
  return last_launch_status();
}

template <typename T, int MODE, int OX, int OY>
int dtile_batch_variant(const TileBatchArgs<T>& b, const VoxMat<T>& m, cudaStream_t s) {
  auto kern = h8_dtile_batch_kernel<T, MODE, OX, OY>;
  const int nt = (OX + 2) * (OY + 2), exy = (OX + 1) * (OY + 1);
  const size_t smem = tile_stage_offset<T>(nt, exy, 3, 4) + sizeof(T) * 2 * kStageH * (size_t)exy;
  int st = batch_smem_attr(kern, smem);
  if (st) return st;
  const int threads = ((OX + 1) * (OY + 1) + 31) / 32 * 32;
  { note_launch(); kern<<<b.n_blocks, threads, smem, s>>>(b, m); }
  return last_launch_status();
}

}  // namespace

template <typename T>
int h8_tile_batch_launch(const TileBatchArgs<T>& b, const VoxMat<T>& m, int mode, int ox, int oy, cudaStream_t s) {
  if (!m.iso) return PHASTB_UNSUPPORTED;
  if (b.n_blocks < 1) return PHASTB_OK;
  const bool dot = mode == kModeDot;
  if (mode != kModeApply && !dot) return PHASTB_ERR_ARG;
  if (ox == 16 && oy == 8)
    return dot ? tile_batch_variant<T, kModeDot, 16, 8>(b, m, s) : tile_batch_variant<T, kModeApply, 16, 8>(b, m, s);
  if (ox == 8 && oy == 8)
    return dot ? tile_batch_variant<T, kModeDot, 8, 8>(b, m, s) : tile_batch_variant<T, kModeApply, 8, 8>(b, m, s);
  return PHASTB_ERR_ARG;
}

int h8_tile_batch_level_launch(const TileBatchArgs<float>& b, const VoxMat<float>& m, int coef, int mode, int ox,
                               int oy, cudaStream_t s) {
  if (b.n_blocks < 1) return PHASTB_OK;
  if (coef == kCoefIso && !m.iso) return PHASTB_UNSUPPORTED;
  if (coef == kCoefIso && ox == 16 && oy == 8) {
    if (mode == kModeCheb) return tile_batch_level_variant<kCoefIso, kModeCheb, 16, 8>(b, m, s);
    if (mode == kModeRes) return tile_batch_level_variant<kCoefIso, kModeRes, 16, 8>(b, m, s);
    if (mode == kModeSmooth) return tile_batch_level_variant<kCoefIso, kModeSmooth, 16, 8>(b, m, s);
    if (mode == kModeNodal) return tile_batch_level_variant<kCoefIso, kModeNodal, 16, 8>(b, m, s);
  }
  if (coef == kCoefIso && ox == 8 && oy == 8) {
    if (mode == kModeCheb) return tile_batch_level_variant<kCoefIso, kModeCheb, 8, 8>(b, m, s);
    if (mode == kModeRes) return tile_batch_level_variant<kCoefIso, kModeRes, 8, 8>(b, m, s);
    if (mode == kModeSmooth) return tile_batch_level_variant<kCoefIso, kModeSmooth, 8, 8>(b, m, s);
    if (mode == kModeNodal) return tile_batch_level_variant<kCoefIso, kModeNodal, 8, 8>(b, m, s);
  }
  if (coef == kCoefQP && ox == 8 && oy == 8) {
    if (mode == kModeCheb) return tile_batch_level_variant<kCoefQP, kModeCheb, 8, 8>(b, m, s);
    if (mode == kModeRes) return tile_batch_level_variant<kCoefQP, kModeRes, 8, 8>(b, m, s);
    if (mode == kModeSmooth) return tile_batch_level_variant<kCoefQP, kModeSmooth, 8, 8>(b, m, s);
    if (mode == kModeApply) return tile_batch_level_variant<kCoefQP, kModeApply, 8, 8>(b, m, s);
  }
  return PHASTB_ERR_ARG;
}

template <typename T>
int h8_dtile_batch_launch(const TileBatchArgs<T>& b, const VoxMat<T>& m, bool dot, int ox, int oy, cudaStream_t s) {
  if (b.n_blocks < 1) return PHASTB_OK;
  if (ox == 16 && oy == 8)
    return dot ? dtile_batch_variant<T, kModeDot, 16, 8>(b, m, s) : dtile_batch_variant<T, kModeApply, 16, 8>(b, m, s);
  if (ox == 8 && oy == 8)
    return dot ? dtile_batch_variant<T, kModeDot, 8, 8>(b, m, s) : dtile_batch_variant<T, kModeApply, 8, 8>(b, m, s);
  return PHASTB_ERR_ARG;
}

template int h8_tile_batch_launch<double>(const TileBatchArgs<double>&, const VoxMat<double>&, int, int, int,
                                          cudaStream_t);
template int h8_tile_batch_launch<float>(const TileBatchArgs<float>&, const VoxMat<float>&, int, int, int,
                                         cudaStream_t);
template int h8_dtile_batch_launch<double>(const TileBatchArgs<double>&, const VoxMat<double>&, bool, int, int,
                                           cudaStream_t);

template TileArgs<double> tile_args<double>(const VoxGeom&, int);
template TileArgs<float> tile_args<float>(const VoxGeom&, int);
template int h8_tile_launch<double>(const TileArgs<double>&, const VoxMat<double>&, int, int, cudaStream_t, bool);
template int h8_tile_launch<float>(const TileArgs<float>&, const VoxMat<float>&, int, int, cudaStream_t, bool);
template int h8_mech_tile_launch<double>(const VoxGeom&, const VoxMat<double>&, const uint8_t*, const double*,
                                         const double*, const double*, const uint8_t*, double*, RedWs, const int*,
                                         bool, bool, cudaStream_t, const TileShape*);
template int h8_mech_tile_launch<float>(const VoxGeom&, const VoxMat<float>&, const uint8_t*, const float*,
                                        const float*, const float*, const uint8_t*, float*, RedWs, const int*, bool,
                                        bool, cudaStream_t, const TileShape*);

}  // namespace phastb

// ------------------------------------------------------------------ autotuner

namespace phastb {
bool valid_vox(const phastb_voxel_grid* g);
bool valid_mat(const phastb_voxel_material* m);

namespace {

template <typename T>
int tune_t(const VoxGeom& v, const VoxMat<T>& m, const uint8_t* slot, const T* x, const T* d, T* y, RedWs ws,
           cudaStream_t s, TileShape* best_out, float* best_ms) {
  TileArgs<T> a = tile_args<T>(v, 0);
  a.slot = slot;
  a.d = d;
  a.x = x;
  a.y = y;
  a.ws = ws;
  int st = tune_shape<T>(a, m, m.iso ? kCoefIso : kCoefAniso, kModeApply, s, best_out, best_ms);
  if (st) return st;
  tile_shape_record(v, (int)sizeof(T), 0, *best_out);
  return PHASTB_OK;
}

}  // namespace
}  // namespace phastb

using namespace phastb;

extern "C" {

int phastb_h8_tile_shape(const phastb_voxel_grid* g, int dtype, int set, int* shape) {
  if (!valid_vox(g) || !shape || (dtype != PHASTB_F32 && dtype != PHASTB_F64)) return PHASTB_ERR_ARG;
  const VoxGeom v = make_vox_geom(*g);
  const int word = dtype == PHASTB_F32 ? 4 : 8;
  if (set) {
    TileShape t{shape[0], shape[1], shape[2]};
    if (!tile_ok(t)) return PHASTB_ERR_ARG;
    tile_shape_record(v, word, 0, t);
    return PHASTB_OK;
  }
  const TileShape t = tile_shape_for(v, word, 0);
  shape[0] = std::min(t.ox, v.rx);
  shape[1] = std::min(t.oy, v.ry);
  shape[2] = std::min(t.kz, v.rz);
  return PHASTB_OK;
}

int phastb_h8_autotune(const phastb_voxel_grid* g, const phastb_voxel_material* m, int dtype, const uint8_t* slot,
                       const void* x, const void* d, void* y, void* scratch, size_t scratch_bytes, int* shape,
                       float* ms, void* stream) {
  if (!valid_vox(g) || !valid_mat(m) || !slot || !x || !y || !shape || !ms) return PHASTB_ERR_ARG;
  if (dtype != PHASTB_F32 && dtype != PHASTB_F64) return PHASTB_ERR_ARG;
  if (!scratch || scratch_bytes < red_ws_bytes()) return PHASTB_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return PHASTB_ERR_ARG;
  const VoxGeom v = make_vox_geom(*g);
  RedWs ws = red_ws(scratch);
  int st;
  if ((st = red_ws_reset(ws, s))) return st;
  TileShape t{};
  if (dtype == PHASTB_F64)
    st = tune_t<double>(v, make_vox_mat<double>(*m), slot, (const double*)x, (const double*)d, (double*)y, ws, s,
                        &t, ms);
  else
    st = tune_t<float>(v, make_vox_mat<float>(*m), slot, (const float*)x, (const float*)d, (float*)y, ws, s, &t, ms);
  if (st) return st;
  shape[0] = t.ox;
  shape[1] = t.oy;
  shape[2] = t.kz;
  return PHASTB_OK;
}

}  // extern "C"

extern "C" int phastb_test_grid_barrier(int blocks, int skip_block, double limit_s, int* grid_error_host,
                                        int* passed_host) {
  using namespace phastb;
  if (blocks < 1 || blocks > 64 || skip_block >= blocks || !(limit_s > 0) || limit_s > 10.0 || !grid_error_host ||
      !passed_host)
    return PHASTB_ERR_ARG;
  int dev = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return PHASTB_UNSUPPORTED;
  PcgState* st = nullptr;
  int* passed = nullptr;
  if (cudaMalloc(&st, sizeof(PcgState)) != cudaSuccess) return PHASTB_ERR_CUDA;
  if (cudaMalloc(&passed, sizeof(int)) != cudaSuccess) {
    cudaFree(st);
    return PHASTB_ERR_CUDA;
  }
  int status = cuda_status(cudaMemset(st, 0, sizeof(PcgState)));
  if (!status) status = cuda_status(cudaMemset(passed, 0, sizeof(int)));
  unsigned long long limit_ns = (unsigned long long)(limit_s * 1e9);
  void* args[] = {&st, &skip_block, &limit_ns, &passed};
  if (!status) {
    note_launch();
    status = cuda_status(cudaLaunchCooperativeKernel((const void*)grid_barrier_test_kernel, dim3(blocks), dim3(32),
                                                     args, 0, nullptr));
  }
  if (!status) status = cuda_status(cudaDeviceSynchronize());
  PcgState hs{};
  if (!status) status = cuda_status(cudaMemcpy(&hs, st, sizeof(PcgState), cudaMemcpyDeviceToHost));
  if (!status) status = cuda_status(cudaMemcpy(passed_host, passed, sizeof(int), cudaMemcpyDeviceToHost));
  cudaFree(st);
  cudaFree(passed);
  if (status) return status;
  *grid_error_host = hs.grid_error;
  return hs.grid_error ? PHASTB_ERR_CUDA : PHASTB_OK;
}

extern "C" int phastb_h8_tma_staging(const phastb_voxel_grid* g, int dtype) {
  using namespace phastb;
  if (!valid_vox(g) || (dtype != PHASTB_F64 && dtype != PHASTB_F32)) return -1;
  const VoxGeom v = make_vox_geom(*g);
  const int A = dtype == PHASTB_F32 ? 4 : 2;
  return (tma_enabled() && v.rx % A == 0 && tensor_map_encoder() != nullptr) ? 1 : 0;
}
