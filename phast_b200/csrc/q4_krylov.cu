// Persistent Krylov solves on a structured Q4 grid (see q4_krylov.cuh).
//
// The 2D grids hold 1e3 to 3e5 nodes: a solve's whole state fits the SMs, and
// an iteration as separate launches (operator, reductions, updates) is six or
// four kernels of a few microseconds each that mostly wait for their launch.
// Here one cooperative launch runs the solve.  A block owns a tx x ty tile of
// nodes (one block per SM): the rows of the operator, formed once, and the
// direction p of the tile with a one-node halo live in shared memory, the
// iterate and residual in registers.  Only z of a tile's rim goes to the
// neighbours, as tagged words beside the dot products (grid_sync.cuh), and every
// thread updates p of its share of the halo with the same beta.  An iteration
// waits on the grid twice (1.6 us each on 148 blocks, of about 5 to 7).
//
// Measured per solve, separate launches and this: bound-projected PCG on 401 x
// 161 nodes 4.2 and 1.1 ms, CG on 201 x 201 nodes (2 700 iterations) 50.8 and
// 14.3 ms, on 257 x 257 nodes 1.7 and 0.7 ms (damage), 0.9 and 0.3 ms (adjoint).
#include "q4_krylov.cuh"

#include <algorithm>
#include <cstddef>
#include <cstring>

#include "grid_sync.cuh"
#include "q4_kernels.cuh"

namespace phastb {

namespace {

constexpr int kT = 512;  // threads per block
constexpr size_t kSmemMax = 220 * 1024;

struct Tiling {
  int NX, NY;  // nodes per axis
  int tx, ty, tiles_x, tiles_y;
};

// Rows of the scalar damage operator: 9 coefficients per node, neighbour (di, dj) at 3 (dj + 1) + di + 1.
struct DamageRows {
  static constexpr int NC = 1, W = 9;
  Q4Tab<double> t;
  const double* Hq;
  double rsh;
  const double* rsh_e;
  double gcl0;
  const double* gcl0_e;
  const uint8_t* mask;

  // b and 1 / diag of q4_damage_prepare_kernel in its order, through b_out, minv_out (may be null)
  __device__ void row(int i, int j, double (&c)[W], double* b_out, double* minv_out) const {
#pragma unroll
    for (int k = 0; k < W; ++k) c[k] = 0.0;
    double bb = 0, dg = 0;
#pragma unroll
    for (int dj = 0; dj < 2; ++dj)
#pragma unroll
      for (int di = 0; di < 2; ++di) {
        const int ei = i - 1 + di, ej = j - 1 + dj;
        if (ei < 0 || ei >= t.nx || ej < 0 || ej >= t.ny) continue;
        const int e = ej * t.nx + ei;
        const int a = q4_local(1 - di, 1 - dj);
        const double2 h01 = __ldg(reinterpret_cast<const double2*>(Hq) + 2 * e);
        const double2 h23 = __ldg(reinterpret_cast<const double2*>(Hq) + 2 * e + 1);
        const double H[4] = {h01.x, h01.y, h23.x, h23.y};
        const double sh = rsh_e ? __ldg(rsh_e + e) : rsh, gl = gcl0_e ? __ldg(gcl0_e + e) : gcl0;
        double lapd = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          bb += t.N[q][a] * (2.0 * H[q] * t.w);
          lapd += t.w * (t.gx[q][a] * t.gx[q][a] + t.gy[q][a] * t.gy[q][a]);
          dg += (t.N[q][a] * t.N[q][a]) * ((2.0 * H[q] + sh) * t.w);
        }
        dg += gl * lapd;
#pragma unroll
        for (int ly = 0; ly < 2; ++ly)
#pragma unroll
          for (int lx = 0; lx < 2; ++lx) {
            const int b = q4_local(lx, ly);
            double lap = 0, mass = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              lap += t.w * (t.gx[q][a] * t.gx[q][b] + t.gy[q][a] * t.gy[q][b]);
              mass += t.N[q][a] * ((2.0 * H[q] + sh) * t.N[q][b] * t.w);
            }
            c[3 * (dj + ly) + di + lx] += gl * lap + mass;
          }
      }
    if (mask && mask[j * (t.nx + 1) + i]) {
#pragma unroll
      for (int k = 0; k < W; ++k) c[k] = 0.0;
    }
    if (b_out) *b_out = bb;
    if (minv_out) *minv_out = 1.0 / (dg + 1e-30);
  }

  // y = row . p; rows at r[k * rs], p at its own node with row pitch pw
  __device__ __forceinline__ static void apply(const double* r, int rs, const double* p, int pw, int, double (&y)[1]) {
    double a = 0, b = 0, c = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      a += r[k * rs] * p[-pw + k - 1];
      b += r[(3 + k) * rs] * p[k - 1];
      c += r[(6 + k) * rs] * p[pw + k - 1];
    }
    y[0] = (a + c) + b;
  }
};

// Rows of the elastic operator: for the eight neighbours (in the order of DamageRows, without the node itself)
// a 2 x 2 block.  A rigid translation gives no force, so y_i = sum_j K_ij (p_j - p_i): differences of nodal
// values, as the strain of an element takes them, without the cancellation of the diagonal block.
struct MechRows {
  static constexpr int NC = 2, W = 32;
  Q4Tab<double> t;
  Mat2<double> m;
  const double* d;
  const double* u;
  const uint8_t* mask;

  __device__ void row(int i, int j, double (&c)[W], double*, double*) const {
#pragma unroll
    for (int k = 0; k < W; ++k) c[k] = 0.0;
#pragma unroll
    for (int dj = 0; dj < 2; ++dj)
#pragma unroll
      for (int di = 0; di < 2; ++di) {
        const int ei = i - 1 + di, ej = j - 1 + dj;
        if (ei < 0 || ei >= t.nx || ej < 0 || ej >= t.ny) continue;
        const int a = q4_local(1 - di, 1 - dj);
        int n[4];
        q4_corners(ei, ej, t.nx, n);
        double ux[4], uy[4], dd[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          ux[b] = uy[b] = 0.0;
          if (u) load2(u, n[b], ux[b], uy[b]);
          dd[b] = d ? __ldg(d + n[b]) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double exx = 0, eyy = 0, gxy = 0, dq = 0;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            exx += t.gx[q][b] * ux[b];
            eyy += t.gy[q][b] * uy[b];
            gxy += t.gy[q][b] * ux[b] + t.gx[q][b] * uy[b];
            dq += t.N[q][b] * dd[b];
          }
          const double g = d ? degr(m, dq) : 1.0;
          // the stress of unit strains: columns of the (tangent) moduli
          double sx[3], sy[3], sz[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const double e0 = k == 0 ? 1.0 : 0.0, e1 = k == 1 ? 1.0 : 0.0, e2 = k == 2 ? 1.0 : 0.0;
            if (u)
              dstress2(m, m.ssplit, exx, eyy, gxy, e0, e1, e2, g, sx[k], sy[k], sz[k]);
            else
              stress2(m, m.ssplit, e0, e1, e2, g, sx[k], sy[k], sz[k]);
          }
          const double ax = t.gx[q][a] * t.w, ay = t.gy[q][a] * t.w;
          // rows (f_x, f_y) of the node against unit strains
          double fx[3], fy[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            fx[k] = ax * sx[k] + ay * sz[k];
            fy[k] = ay * sy[k] + ax * sz[k];
          }
#pragma unroll
          for (int ly = 0; ly < 2; ++ly)
#pragma unroll
            for (int lx = 0; lx < 2; ++lx) {
              const int k9 = 3 * (dj + ly) + di + lx;
              if (k9 == 4) continue;
              const int b = q4_local(lx, ly), k8 = 4 * (k9 - (k9 > 4 ? 1 : 0));
              const double bx = t.gx[q][b], by = t.gy[q][b];
              c[k8] += fx[0] * bx + fx[2] * by;
              c[k8 + 1] += fx[1] * by + fx[2] * bx;
              c[k8 + 2] += fy[0] * bx + fy[2] * by;
              c[k8 + 3] += fy[1] * by + fy[2] * bx;
            }
        }
      }
    if (mask) {
      const int node = j * (t.nx + 1) + i;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (mask[2 * node]) c[4 * k] = c[4 * k + 1] = 0.0;
        if (mask[2 * node + 1]) c[4 * k + 2] = c[4 * k + 3] = 0.0;
      }
    }
  }

  // p: x components at p, y components ps doubles later
  __device__ __forceinline__ static void apply(const double* r, int rs, const double* p, int pw, int ps,
                                               double (&y)[2]) {
    const double x0 = p[0], y0 = p[ps];
    double a0 = 0, a1 = 0, b0 = 0, b1 = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int k9 = k + (k >= 4 ? 1 : 0), o = (k9 / 3 - 1) * pw + k9 % 3 - 1;
      const double dx = p[o] - x0, dy = p[ps + o] - y0;
      a0 += r[(4 * k) * rs] * dx;
      a1 += r[(4 * k + 1) * rs] * dy;
      b0 += r[(4 * k + 2) * rs] * dx;
      b1 += r[(4 * k + 3) * rs] * dy;
    }
    y[0] = a0 + a1;
    y[1] = b0 + b1;
  }
};

// The tile of a block and one thread's share of it: NPT nodes and the halo nodes h, h + kT, ...
template <class ROWS, int NPT>
struct Tile {
  static constexpr int NC = ROWS::NC;
  Tiling g;
  int i0, j0, nt, pw, ps;  // nt: nodes of a tile (row pitch of the coefficient arrays); ps: one component of p
  double* rows;            // [W][nt]
  double* p;               // [NC][(ty + 2) (tx + 2)]
  int node[NPT], at[NPT];  // global node (-1: none) and index in p
  bool rim[NPT];           // a neighbour's halo node

  __device__ Tile(const Tiling& g_, double* smem) : g(g_) {
    i0 = (blockIdx.x % g.tiles_x) * g.tx;
    j0 = (blockIdx.x / g.tiles_x) * g.ty;
    nt = g.tx * g.ty;
    pw = g.tx + 2;
    ps = pw * (g.ty + 2);
    rows = smem;
    p = smem + (size_t)ROWS::W * nt;
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      const int l = threadIdx.x + k * kT, li = l % g.tx, lj = l / g.tx;
      const bool in = l < nt && i0 + li < g.NX && j0 + lj < g.NY;
      node[k] = in ? (j0 + lj) * g.NX + i0 + li : -1;
      at[k] = (lj + 1) * pw + li + 1;
      rim[k] = in && (li == 0 || li == g.tx - 1 || lj == 0 || lj == g.ty - 1);
    }
  }
  __device__ __forceinline__ int halo_count() const { return 2 * pw + 2 * g.ty; }
  // halo node h: its index in p; returns its global node, -1 outside the grid
  __device__ __forceinline__ int halo(int h, int& where) const {
    int li, lj;
    if (h < pw) {
      li = h, lj = 0;
    } else if (h < 2 * pw) {
      li = h - pw, lj = g.ty + 1;
    } else {
      const int r = h - 2 * pw;
      li = (r & 1) ? g.tx + 1 : 0, lj = 1 + (r >> 1);
    }
    where = lj * pw + li;
    const int gi = i0 + li - 1, gj = j0 + lj - 1;
    return gi >= 0 && gi < g.NX && gj >= 0 && gj < g.NY ? gj * g.NX + gi : -1;
  }
  __device__ __forceinline__ void apply(int k, double (&y)[NC]) const {
    ROWS::apply(rows + threadIdx.x + k * kT, nt, p + at[k], pw, ps, y);
  }
};

// p of the tile's own nodes outside the grid is zero (they are never read with a nonzero coefficient, but are read)
template <class ROWS, int NPT>
__device__ __forceinline__ void clear_p(const Tile<ROWS, NPT>& t) {
  for (int i = threadIdx.x; i < ROWS::NC * t.ps; i += kT) t.p[i] = 0.0;
}

// ------------------------------------------------------------------ PCG

struct PcgArgs {
  Tiling g;
  int maxiter, check_every, mode, pad_;
  double *r, *x;
  const double* p;
  const double* inv_diag;  // null: identity
  Tagged* z;               // rim values, by unknown
  Tagged* slots;
  unsigned* err;
  PcgState* st;
};

template <class ROWS, int NPT>
__global__ void __launch_bounds__(kT, 1) q4_pcg_kernel(ROWS rows, PcgArgs a) {
  constexpr int NC = ROWS::NC, W = ROWS::W;
  extern __shared__ __align__(16) double smem[];
  Tile<ROWS, NPT> t(a.g, smem);
  PcgState S = *a.st;
  GridSync gs{a.slots, a.err, 0ull};
  double* hz = t.p + NC * t.ps;  // z of the halo
  __shared__ int s_lost;  // a halo wait of this block ran out
  if (threadIdx.x == 0) s_lost = 0;
  auto fail = [&] {  // a wait ran out
    if (threadIdx.x == 0) atomicExch(&a.st->grid_error, 1);
  };
  clear_p(t);
  __syncthreads();
  double x[NPT][NC], r[NPT][NC], mi[NPT][NC];
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const int n = t.node[k];
#pragma unroll
    for (int c = 0; c < NC; ++c) x[k][c] = r[k][c] = mi[k][c] = 0.0;
    if (n >= 0) {
      double c[W];
      rows.row(n % a.g.NX, n / a.g.NX, c, nullptr, nullptr);
#pragma unroll
      for (int w = 0; w < W; ++w) t.rows[(size_t)w * t.nt + threadIdx.x + k * kT] = c[w];
#pragma unroll
      for (int c2 = 0; c2 < NC; ++c2) {
        x[k][c2] = a.x[NC * n + c2];
        r[k][c2] = a.r[NC * n + c2];
        mi[k][c2] = a.inv_diag ? a.inv_diag[NC * n + c2] : 1.0;
        t.p[c2 * t.ps + t.at[k]] = a.p[NC * n + c2];
      }
    }
  }
  for (int h = threadIdx.x; h < t.halo_count(); h += kT) {
    int at;
    const int n = t.halo(h, at);
    if (n >= 0) {
#pragma unroll
      for (int c = 0; c < NC; ++c) t.p[c * t.ps + at] = a.p[NC * n + c];
    }
  }
  __syncthreads();
  for (int it = 0; it < a.maxiter && S.active; ++it) {
    double ap[NPT][NC], v1[1] = {0.0};
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
#pragma unroll
      for (int c = 0; c < NC; ++c) ap[k][c] = 0.0;
      if (t.node[k] >= 0) {
        t.apply(k, ap[k]);
#pragma unroll
        for (int c = 0; c < NC; ++c) v1[0] += t.p[c * t.ps + t.at[k]] * ap[k][c];
      }
    }
    if (!grid_reduce<1, 0, kT>(v1, gs)) return fail();
    const double PAP = v1[0];
    // the state rules of pcg_alpha_kernel
    S.iter += 1;
    if (a.mode == PCG_PERIODIC) {
      if (!isfinite(PAP) || PAP <= 1e-30) {
        S.breakdown = 1;
        S.active = 0;
        break;
      }
      S.alpha = S.rr / (PAP + 1e-30);
    } else {
      if (!isfinite(PAP)) S.nonfinite = 1;
      if (!(PAP > 0.0)) S.breakdown = 1;
      if (S.breakdown || S.nonfinite) {
        S.active = 0;
        break;
      }
      S.alpha = S.rz / PAP;
      S.steps += 1;
    }
    double v2[2] = {0.0, 0.0}, z[NPT][NC];  // r . z, r . r
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      const int n = t.node[k];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        z[k][c] = 0.0;
        if (n >= 0) {
          x[k][c] += S.alpha * t.p[c * t.ps + t.at[k]];
          r[k][c] -= S.alpha * ap[k][c];
          z[k][c] = r[k][c] * mi[k][c];
          if (t.rim[k]) st_tagged(a.z + NC * n + c, z[k][c], it + 1);
          v2[0] += r[k][c] * z[k][c];
          v2[1] += r[k][c] * r[k][c];
        }
      }
    }
    // the halo's z arrives beside the sums
    auto take_halo = [&](int i, int step) {
      for (int h = i; h < t.halo_count(); h += step) {
        int at;
        const int n = t.halo(h, at);
        if (n >= 0) {
#pragma unroll
          for (int c = 0; c < NC; ++c)
            if (!wait_tagged(a.z + NC * n + c, it + 1, &hz[NC * h + c], a.err)) s_lost = 1;
        }
      }
    };
    if (!grid_reduce<2, 0, kT>(v2, gs, take_halo) || s_lost) return fail();
    const double RZ = v2[0], RR = v2[1];
    // the state rules of pcg_update_kernel
    if (!isfinite(RR) || !isfinite(RZ)) S.nonfinite = 1;
    if (a.mode == PCG_PERIODIC) {
      S.beta = RR / (S.rr + 1e-30);
      S.rr = RR;
      S.rz = RR;
      if (S.iter % a.check_every == 0) {
        if (RR < S.thr_sq) {
          S.converged = 1;
          S.active = 0;
        } else if (RR > 1e12 * S.rr0) {
          S.active = 0;
        }
      }
    } else {
      S.rr = RR;
      if (!(RR > S.thr_sq)) {
        S.converged = 1;
        S.active = 0;
      } else {
        if (a.mode == PCG_STRICT && !(RZ > 0.0)) S.breakdown = 1;
        S.beta = (a.mode == PCG_STRICT) ? RZ / S.rz : ((S.rz > 0.0) ? RZ / S.rz : 0.0);
        S.rz = RZ;
      }
    }
    if (S.breakdown || S.nonfinite) S.active = 0;
    if (!S.active) break;
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      if (t.node[k] >= 0) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          double& p = t.p[c * t.ps + t.at[k]];
          p = z[k][c] + S.beta * p;
        }
      }
    }
    for (int h = threadIdx.x; h < t.halo_count(); h += kT) {
      int at;
      const int n = t.halo(h, at);
      if (n >= 0) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          double& p = t.p[c * t.ps + at];
          p = hz[NC * h + c] + S.beta * p;
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const int n = t.node[k];
    if (n >= 0) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        a.x[NC * n + c] = x[k][c];
        a.r[NC * n + c] = r[k][c];
      }
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) store_pcg_state(a.st, S);
}

// ------------------------------------------------------------------ PPCG

struct PpcgArgs {
  Tiling g;
  int max_iter, check_every;
  double tol;
  const double *d_prev, *d_init;
  const uint8_t* fixed;
  const double* vals;
  double* d;
  Tagged *pub_z, *pub_d;  // rim values of z, and of d when a residual is recomputed, by node
  Tagged* slots;
  unsigned* err;
  PpcgState* st;
};

__device__ __forceinline__ bool bound_active(double d, double lb, double r, bool fixed) {
  const double atol = 1e-14;  // bound_atol (damage_solver.py:3559)
  return ((d <= lb + atol) && (r < 0.0)) || ((d >= 1.0 - atol) && (r > 0.0)) || fixed;
}

// The iterations of ppcg_solve: its kernels' rules with the state in registers, evaluated alike in every block.
template <int NPT>
__global__ void __launch_bounds__(kT, 1) q4_ppcg_kernel(DamageRows rows, PpcgArgs a) {
  constexpr int W = DamageRows::W;
  extern __shared__ __align__(16) double smem[];
  Tile<DamageRows, NPT> t(a.g, smem);
  GridSync gs{a.slots, a.err, 0ull};
  __shared__ int s_lost;  // a halo wait of this block ran out
  if (threadIdx.x == 0) s_lost = 0;
  double* ds = t.p + t.ps;   // d with its halo, where a residual is recomputed
  double* hz = ds + t.ps;    // z of the halo
  clear_p(t);
  for (int i = threadIdx.x; i < t.ps; i += kT) ds[i] = 0.0;
  __syncthreads();
  auto start = [&](int n) {  // the start value of a node
    if (a.fixed && a.fixed[n]) return a.vals[n];
    return a.d_init ? a.d_init[n] : a.d_prev[n];
  };
  double d[NPT], lb[NPT], b[NPT], mi[NPT], r[NPT], z[NPT];
  bool act[NPT], fx[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const int n = t.node[k];
    d[k] = lb[k] = b[k] = mi[k] = r[k] = z[k] = 0.0;
    act[k] = fx[k] = false;
    if (n >= 0) {
      double c[W];
      rows.row(n % a.g.NX, n / a.g.NX, c, &b[k], &mi[k]);
#pragma unroll
      for (int w = 0; w < W; ++w) t.rows[(size_t)w * t.nt + threadIdx.x + k * kT] = c[w];
      fx[k] = a.fixed && a.fixed[n];
      d[k] = start(n);
      lb[k] = fx[k] ? a.vals[n] : a.d_prev[n];
      if (fx[k]) mi[k] = 0.0;
      t.p[t.at[k]] = d[k];
    }
  }
  for (int h = threadIdx.x; h < t.halo_count(); h += kT) {
    int at;
    const int n = t.halo(h, at);
    if (n >= 0) t.p[at] = start(n);
  }
  __syncthreads();
  double v3[3] = {0.0, 0.0, 0.0};  // r . r, b . b, r . z
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const int n = t.node[k];
    if (n >= 0) {
      double y[1];
      t.apply(k, y);
      r[k] = fx[k] ? 0.0 : b[k] - y[0];
      act[k] = bound_active(d[k], lb[k], r[k], fx[k]);
      z[k] = act[k] ? 0.0 : r[k] * mi[k];
      if (t.rim[k]) st_tagged(a.pub_z + n, z[k], 1);
      v3[0] += r[k] * r[k];
      v3[1] += b[k] * b[k];
      v3[2] += act[k] ? 0.0 : r[k] * z[k];
    }
  }
  int it = 0;
  // the halo's z arrives beside the sums
  auto take_halo = [&](int i, int step) {
    for (int h = i; h < t.halo_count(); h += step) {
      int at;
      const int n = t.halo(h, at);
      if (n >= 0 && !wait_tagged(a.pub_z + n, it + 1, &hz[h], a.err)) s_lost = 1;
    }
  };
  if (!grid_reduce<3, 0, kT>(v3, gs, take_halo) || s_lost) return;
  const double r0sq = v3[0];
  const double ref = fmax(fmax(sqrt(v3[1]), sqrt(v3[0])), 1e-30);
  const double tol_sq = (a.tol * ref) * (a.tol * ref);
  double rz = v3[2], beta = 0.0;
  bool reset = true;
  int reason = 1, last = a.max_iter;
  while (it < a.max_iter) {
    // p = z, or z + beta p; zero on the active set (there z is zero, and so is p unless reset)
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      if (t.node[k] >= 0) {
        double& p = t.p[t.at[k]];
        p = act[k] ? 0.0 : (reset ? z[k] : beta * p + z[k]);
      }
    }
    for (int h = threadIdx.x; h < t.halo_count(); h += kT) {
      int at;
      const int n = t.halo(h, at);
      if (n >= 0) {
        t.p[at] = reset ? hz[h] : beta * t.p[at] + hz[h];
      }
    }
    __syncthreads();
    double ap[NPT], v1[3] = {0.0, INFINITY, INFINITY};  // p . Ap, the largest steps up and down
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      ap[k] = 0.0;
      if (t.node[k] >= 0) {
        double y[1];
        t.apply(k, y);
        ap[k] = y[0];
        const double p = t.p[t.at[k]];
        v1[0] += p * y[0];
        if (p > 0.0) v1[1] = fmin(v1[1], (1.0 - d[k]) / p);
        if (p < 0.0) v1[2] = fmin(v1[2], (lb[k] - d[k]) / p);
      }
    }
    if (!grid_reduce<1, 2, kT>(v1, gs)) return;
    ++it;
    if (v1[0] <= 0.0) {  // degenerate direction: the reference breaks out
      reason = 2;
      last = it;
      break;
    }
    const double acg = rz / (v1[0] + 1e-30);
    double alpha = acg;
    if (v1[1] < alpha) alpha = v1[1];
    if (v1[2] < alpha) alpha = v1[2];
    const bool capped = alpha < acg && alpha >= 0.0;
    if (!capped) alpha = acg;
    const bool need = capped || it % a.check_every == 0;
    double v2[3] = {0.0, 0.0, 0.0};  // r_free . r_free, r_free . z, active-set changes
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      if (t.node[k] >= 0) {
        double dn = d[k] + alpha * t.p[t.at[k]];
        if (capped)
          dn = fmin(fmax(dn, lb[k]), 1.0);
        else
          r[k] = r[k] - alpha * ap[k];
        d[k] = dn;
        if (need) {
          ds[t.at[k]] = dn;
          if (t.rim[k]) st_tagged(a.pub_d + t.node[k], dn, it);
        }
      }
    }
    if (need) {  // the true residual b - A d, and the active set at it
      for (int h = threadIdx.x; h < t.halo_count(); h += kT) {
        int at;
        const int n = t.halo(h, at);
        if (n >= 0 && !wait_tagged(a.pub_d + n, it, &ds[at], a.err)) s_lost = 1;
      }
      __syncthreads();
      if (s_lost) return;
#pragma unroll
      for (int k = 0; k < NPT; ++k) {
        if (t.node[k] >= 0) {
          double y[1];
          DamageRows::apply(t.rows + threadIdx.x + k * kT, t.nt, ds + t.at[k], t.pw, t.ps, y);
          r[k] = fx[k] ? 0.0 : b[k] - y[0];
          const bool an = bound_active(d[k], lb[k], r[k], fx[k]);
          if (an != act[k]) v2[2] += 1.0;
          act[k] = an;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      if (t.node[k] >= 0) {
        const double rf = act[k] ? 0.0 : r[k];
        z[k] = act[k] ? 0.0 : rf * mi[k];
        if (t.rim[k]) st_tagged(a.pub_z + t.node[k], z[k], it + 1);
        v2[0] += rf * rf;
        v2[1] += rf * z[k];
      }
    }
    if (!grid_reduce<3, 0, kT>(v2, gs, take_halo) || s_lost) return;
    if (need) {
      if (v2[0] < tol_sq) {
        reason = 0;
        last = it;
        break;
      }
      if (v2[0] > 1e12 * fmax(r0sq, 1e-30)) {
        reason = 3;
        last = it;
        break;
      }
    }
    reset = capped || v2[2] != 0.0;
    if (!reset) beta = v2[1] / (rz + 1e-30);
    rz = v2[1];
  }
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    if (t.node[k] >= 0) {
      double dn = fmin(fmax(d[k], lb[k]), 1.0);
      if (fx[k]) dn = a.vals[t.node[k]];
      a.d[t.node[k]] = dn;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.st->done = 1;
    a.st->iter = it;
    a.st->reason = reason;
    a.st->last_iter = last;
  }
}

// ------------------------------------------------------------------ host side

// The tiling with the least modelled iteration (microseconds): two waits on the grid, the rows of a tile's nodes,
// and its halo.  False: no tile of at most `most` nodes per block covers the grid.
bool choose_tiling(int NX, int NY, int most, int sms, double node_us, Tiling* out) {
  double best = 1e300;
  const int blocks = std::min(sms, kGridBlocks);
  for (int cx = 1; cx <= blocks; ++cx) {
    const int tx = (NX + cx - 1) / cx;
    if ((NX + tx - 1) / tx != cx) continue;
    for (int cy = 1; cx * cy <= blocks; ++cy) {
      const int ty = (NY + cy - 1) / cy;
      if ((NY + ty - 1) / ty != cy || (long long)tx * ty > most) continue;
      const int G = cx * cy;
      const double c = (G > kGridDirect ? 3.2 : (G > 1 ? 2.0 + 0.02 * G : 0.7)) + node_us * tx * ty + 0.0005 * (2 * (tx + ty) + 4);
      if (c < best) {
        best = c;
        *out = Tiling{NX, NY, tx, ty, cx, cy};
      }
    }
  }
  return best < 1e300;
}

struct DeviceLimits {
  int sms = 0, coop = 0;
};
bool device_limits(DeviceLimits* d) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&d->coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return d->coop && d->sms > 0;
}

// Cooperative launch of one block per tile; PHASTB_UNSUPPORTED when the device refuses it.
template <class K>
int launch_tiles(K kern, const Tiling& g, size_t smem, void** args, cudaStream_t s) {
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) != cudaSuccess ||
      cudaLaunchCooperativeKernel((const void*)kern, dim3(g.tiles_x * g.tiles_y), dim3(kT), args, smem, s) !=
          cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  note_launch();
  return PHASTB_OK;
}

size_t tile_smem(const Tiling& g, int W, int fields, int nc) {
  // rows, fields with their halo, and z of the halo
  return sizeof(double) * ((size_t)W * g.tx * g.ty + (size_t)fields * (g.tx + 2) * (g.ty + 2) +
                           (size_t)nc * (2 * (g.tx + 2) + 2 * g.ty));
}

DamageRows damage_rows(const Q4DamageSys& y) {
  return DamageRows{make_q4_tab<double>(y.g), y.Hq, y.rsh, y.rsh_e, y.gcl0, y.gcl0_e, y.mask};
}

// Zeroes the exchange's slots (in the engines' partials), the error flag and `count` tagged words.
template <class WS>
int reset_sync(const WS& w, Tagged* words, size_t count, cudaStream_t s) {
  int st = cuda_status(cudaMemsetAsync(w.part, 0, grid_slot_bytes(), s));
  if (!st) st = cuda_status(cudaMemsetAsync(w.counter, 0, 4 * sizeof(unsigned), s));
  if (!st) st = cuda_status(cudaMemsetAsync(words, 0, count * sizeof(Tagged), s));
  return st;
}

template <class ROWS>
int run_pcg(const ROWS& rows, const phastb_q4_grid& grid, const PcgWs<double>& w, const double* inv_diag, void* tagged,
            double* x, int maxiter, int check_every, PcgMode mode, double node_us, cudaStream_t s) {
  DeviceLimits lim;
  if (!persistent_pcg_enabled() || !device_limits(&lim)) return PHASTB_UNSUPPORTED;
  constexpr int most = ROWS::NC == 1 ? 4 * kT : 800;  // 800 rows of 256 bytes fill an SM's shared memory
  PcgArgs a;
  std::memset(&a, 0, sizeof(a));
  if (!choose_tiling(grid.nx + 1, grid.ny + 1, most, lim.sms, node_us, &a.g)) return PHASTB_UNSUPPORTED;
  a.maxiter = maxiter;
  a.check_every = check_every;
  a.mode = mode;
  a.r = w.r;
  a.z = static_cast<Tagged*>(tagged);
  a.x = x;
  a.p = w.p;
  a.inv_diag = inv_diag;
  a.slots = reinterpret_cast<Tagged*>(w.part);
  a.err = w.counter;
  a.st = w.st;
  const int nt = a.g.tx * a.g.ty;
  const size_t smem = tile_smem(a.g, ROWS::W, ROWS::NC, ROWS::NC);
  if (smem > kSmemMax || !aligned16(a.z) || !aligned16(a.slots)) return PHASTB_UNSUPPORTED;
  int st = reset_sync(w, a.z, (size_t)ROWS::NC * a.g.NX * a.g.NY, s);
  if (st) return st;
  ROWS r = rows;
  void* args[] = {&r, &a};
  if (nt <= kT) return launch_tiles(q4_pcg_kernel<ROWS, 1>, a.g, smem, args, s);
  if (nt <= 2 * kT) return launch_tiles(q4_pcg_kernel<ROWS, 2>, a.g, smem, args, s);
  if constexpr (ROWS::NC == 1) return launch_tiles(q4_pcg_kernel<ROWS, 4>, a.g, smem, args, s);
  return PHASTB_UNSUPPORTED;
}

static_assert(sizeof(double) * 4 * kMaxPartials >= 4 * kGridValues * kGridBlocks * sizeof(Tagged),
              "the exchange's slots fit the engines' partials");

}  // namespace

int q4_pcg_persistent(const Q4DamageSys& sys, const PcgWs<double>& w, const double* inv_diag, void* tagged, double* x,
                      int maxiter, int check_every, PcgMode mode, cudaStream_t s) {
  return run_pcg(damage_rows(sys), sys.g, w, inv_diag, tagged, x, maxiter, check_every, mode, 0.0006, s);
}

int q4_pcg_persistent(const Q4MechSys& sys, const PcgWs<double>& w, void* tagged, double* x, int maxiter,
                      int check_every, PcgMode mode, cudaStream_t s) {
  // a stress evaluated at the increment itself is no linear operator
  if (sys.m.stress_split == PHASTB_SPLIT_SPECTRAL_STRESS) return PHASTB_UNSUPPORTED;
  const MechRows rows{make_q4_tab<double>(sys.g), make_mat2<double>(sys.m), sys.d, sys.u, sys.mask};
  return run_pcg(rows, sys.g, w, nullptr, tagged, x, maxiter, check_every, mode, 0.002, s);
}

int q4_ppcg_persistent(const Q4DamageSys& sys, const PpcgWs& w, const double* d_prev, const double* d_init,
                       const uint8_t* fixed, const double* vals, double tol, int max_iter, int check_every, double* d,
                       int* info, cudaStream_t s) {
  DeviceLimits lim;
  if (!persistent_pcg_enabled() || !device_limits(&lim)) return PHASTB_UNSUPPORTED;
  PpcgArgs a;
  std::memset(&a, 0, sizeof(a));
  if (!choose_tiling(sys.g.nx + 1, sys.g.ny + 1, 4 * kT, lim.sms, 0.0006, &a.g)) return PHASTB_UNSUPPORTED;
  a.max_iter = max_iter;
  a.check_every = check_every;
  a.tol = tol;
  a.d_prev = d_prev;
  a.d_init = d_init;
  a.fixed = fixed;
  a.vals = vals;
  a.d = d;
  // r, z and p, Ap lie in pairs and are not used here: 16 bytes per node each
  a.pub_z = reinterpret_cast<Tagged*>(w.r);
  a.pub_d = reinterpret_cast<Tagged*>(w.p);
  a.slots = reinterpret_cast<Tagged*>(w.part);
  a.err = w.counter;
  a.st = w.st;
  const int nt = a.g.tx * a.g.ty;
  const size_t smem = tile_smem(a.g, DamageRows::W, 2, 1);
  if (smem > kSmemMax || !aligned16(a.pub_z) || !aligned16(a.pub_d) || !aligned16(a.slots)) return PHASTB_UNSUPPORTED;
  const size_t n = (size_t)a.g.NX * a.g.NY;
  int st = reset_sync(w, a.pub_z, n, s);
  if (!st) st = cuda_status(cudaMemsetAsync(a.pub_d, 0, n * sizeof(Tagged), s));
  if (st) return st;
  DamageRows rows = damage_rows(sys);
  void* args[] = {&rows, &a};
  if (nt <= kT)
    st = launch_tiles(q4_ppcg_kernel<1>, a.g, smem, args, s);
  else if (nt <= 2 * kT)
    st = launch_tiles(q4_ppcg_kernel<2>, a.g, smem, args, s);
  else
    st = launch_tiles(q4_ppcg_kernel<4>, a.g, smem, args, s);
  if (st) return st;
  // the error flag and the state are neighbours: one read
  struct {
    unsigned err[64];
    PpcgState st;
  } h;
  static_assert(offsetof(decltype(h), st) == 256, "the workspace puts the state 256 bytes after the counters");
  if ((st = cuda_status(cudaMemcpyAsync(&h, w.counter, sizeof(h), cudaMemcpyDeviceToHost, s)))) return st;
  if ((st = cuda_status(cudaStreamSynchronize(s)))) return st;
  if (h.err[0]) return PHASTB_ERR_CUDA;  // a wait ran out
  info[0] = h.st.last_iter;
  info[1] = h.st.reason;
  return PHASTB_OK;
}

}  // namespace phastb
