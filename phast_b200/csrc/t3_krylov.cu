// The bound-projected PCG of the T3 damage system in one cooperative launch
// (the rules of ppcg_solve, engine.cuh; element-history models).
//
// A thread owns a node and keeps its row of the assembled operator for the
// whole solve: the distinct neighbours with their coefficients in shared
// memory, formed once from the elements of each colour (a colour touches a node
// at most once, so a table [colour][node] lists a node's elements in the order
// the coloured scatter adds them).  The node's state lives in registers, and so
// does its own copy of each neighbour's direction p, updated with the same beta
// from the neighbour's z, which travels as a tagged word (grid_sync.cuh).  The
// coloured form takes a launch per colour, about 23 of 2.9 us an iteration on a
// mesh with 8 colours; this one is two waits on the grid.  Measured on 35 200
// triangles (17 871 nodes): 4.5 ms with separate launches, 0.6 ms here.
#include <algorithm>
#include <cstring>

#include "engine.cuh"
#include "grid_sync.cuh"

namespace phastb {

bool persistent_pcg_enabled();

namespace {

constexpr int kT = 512;
constexpr int kMaxColours = 14;
constexpr size_t kSmemMax = 220 * 1024;

struct ColourOffsets {
  int off[kMaxColours + 1];
};

// adj[c * n + node] = 4 e + local for the colour-c element at `node` (cleared to -1 before).
__global__ void t3_adjacency_kernel(int n, int n_elems, int colours, ColourOffsets co, const int* __restrict__ elem,
                                    const int* __restrict__ order, int* __restrict__ adj) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n_elems; k += gridDim.x * blockDim.x) {
    int c = 0;
    while (c + 1 < colours && k >= co.off[c + 1]) ++c;
    const int e = order[k];
#pragma unroll
    for (int a = 0; a < 3; ++a) adj[(size_t)c * n + elem[3 * e + a]] = 4 * e + a;
  }
}

struct T3PpcgArgs {
  int n, per, colours, deg;  // per: nodes per block; deg: most neighbours of a node
  int row, pad_;             // row: per rounded up to whole warps
  int max_iter, check_every;
  double tol;
  const int *elem, *adj;
  const double *grad, *areas, *H;
  double gco, gcl0, src;
  const double *gco_e, *gcl0_e, *src_e;
  const double *d_prev, *d_init;
  const uint8_t* fixed;
  const double* vals;
  double* d;
  Tagged *pub_z, *pub_d;  // z, and d when a residual is recomputed, by node
  Tagged* slots;
  unsigned* err;
  PpcgState* st;
};

__device__ __forceinline__ bool bound_active(double d, double lb, double r, bool fixed) {
  const double atol = 1e-14;  // bound_atol (damage_solver.py:3559)
  return ((d <= lb + atol) && (r < 0.0)) || ((d >= 1.0 - atol) && (r > 0.0)) || fixed;
}

__global__ void __launch_bounds__(kT, 1) t3_ppcg_kernel(T3PpcgArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, n = a.n;
  // per neighbour k of the node of thread t, at [k * row + t]: coefficient, p copy, the value that arrived, node
  const int row = a.row;
  double* C = reinterpret_cast<double*>(smem);
  double* P = C + (size_t)a.deg * row;
  double* V = P + (size_t)a.deg * row;
  int* J = reinterpret_cast<int*>(V + (size_t)a.deg * row);
  __shared__ int s_lost;
  if (tid == 0) s_lost = 0;
  GridSync gs{a.slots, a.err, 0ull};
  const int node = blockIdx.x * a.per + tid;
  const bool own = tid < a.per && node < n;
  int deg = 0;
  double diag = 0.0, b = 0.0, mi = 0.0;
  if (own) {
    double mdiag = 0.0;
    for (int c = 0; c < a.colours; ++c) {
      const int q = __ldg(a.adj + (size_t)c * n + node);
      if (q < 0) continue;
      const int e = q >> 2, la = q & 3;
      const double A = __ldg(a.areas + e), He = a.H ? __ldg(a.H + e) : 0.0;
      const double rc = (2.0 * He + (a.gco_e ? __ldg(a.gco_e + e) : a.gco)) * A / 12.0;
      const double kl = a.gcl0_e ? __ldg(a.gcl0_e + e) : a.gcl0;
      const double gx = __ldg(a.grad + 6 * (size_t)e + 2 * la), gy = __ldg(a.grad + 6 * (size_t)e + 2 * la + 1);
      b += (2.0 * He - (a.src_e ? __ldg(a.src_e + e) : a.src)) * A / 3.0;
      mdiag += kl * (A * (gx * gx + gy * gy)) + 2.0 * rc;
      for (int l = 0; l < 3; ++l) {
        const double v = kl * (A * (gx * __ldg(a.grad + 6 * (size_t)e + 2 * l) +
                                    gy * __ldg(a.grad + 6 * (size_t)e + 2 * l + 1))) +
                         (l == la ? 2.0 * rc : rc);
        if (l == la) {
          diag += v;
          continue;
        }
        const int j = __ldg(a.elem + 3 * (size_t)e + l);
        int k = 0;
        while (k < deg && J[k * row + tid] != j) ++k;
        if (k == deg) {
          J[k * row + tid] = j;
          C[k * row + tid] = 0.0;
          ++deg;
        }
        C[k * row + tid] += v;
      }
    }
    mi = 1.0 / (mdiag + 1e-30);
  }
  auto start = [&](int i) {  // the start value of a node
    if (a.fixed && a.fixed[i]) return a.vals[i];
    return a.d_init ? a.d_init[i] : a.d_prev[i];
  };
  const bool fx = own && a.fixed && a.fixed[node];
  double d = 0.0, lb = 0.0, r = 0.0, z = 0.0, p = 0.0;
  bool act = false;
  double v3[3] = {0.0, 0.0, 0.0};  // r . r, b . b, r . z
  if (own) {
    d = start(node);
    lb = fx ? a.vals[node] : a.d_prev[node];
    if (fx) mi = 0.0;
    double y = diag * d;
    for (int k = 0; k < deg; ++k) y += C[k * row + tid] * start(J[k * row + tid]);
    r = fx ? 0.0 : b - y;
    act = bound_active(d, lb, r, fx);
    z = act ? 0.0 : r * mi;
    st_tagged(a.pub_z + node, z, 1);
    v3[0] = r * r;
    v3[1] = b * b;
    v3[2] = act ? 0.0 : r * z;
  }
  int it = 0;
  // this thread's neighbours' words, four polls in flight
  auto take = [&](const Tagged* from, unsigned long long tag) {
    for (int k = 0; k < deg; k += 4) {
      Tagged q[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k + j < deg) q[j] = ld_tagged(from + J[(k + j) * row + tid]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (k + j < deg) {
          if (q[j].tag != tag && !wait_tagged(from + J[(k + j) * row + tid], tag, &q[j].v, a.err)) s_lost = 1;
          V[(k + j) * row + tid] = q[j].v;
        }
      }
    }
  };
  if (!grid_reduce<3, 0, kT>(v3, gs)) return;
  const double r0sq = v3[0];
  const double ref = fmax(fmax(sqrt(v3[1]), sqrt(v3[0])), 1e-30);
  const double tol_sq = (a.tol * ref) * (a.tol * ref);
  double rz = v3[2], beta = 0.0;
  bool reset = true;
  int reason = 1, last = a.max_iter;
  while (it < a.max_iter) {
    // p = z, or z + beta p; zero on the active set (there z is zero, and so is p unless reset)
    double ap = 0.0, v1[3] = {0.0, INFINITY, INFINITY};  // p . Ap, the largest steps up and down
    take(a.pub_z, it + 1);
    if (own) {
      p = act ? 0.0 : (reset ? z : beta * p + z);
      ap = diag * p;
      for (int k = 0; k < deg; ++k) {
        const double pk = reset ? V[k * row + tid] : beta * P[k * row + tid] + V[k * row + tid];
        P[k * row + tid] = pk;
        ap += C[k * row + tid] * pk;
      }
      v1[0] = p * ap;
      if (p > 0.0) v1[1] = (1.0 - d) / p;
      if (p < 0.0) v1[2] = (lb - d) / p;
    }
    if (!grid_reduce<1, 2, kT>(v1, gs) || s_lost) return;
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
    if (own) {
      d = d + alpha * p;
      if (capped)
        d = fmin(fmax(d, lb), 1.0);
      else
        r = r - alpha * ap;
      if (need) st_tagged(a.pub_d + node, d, it);
    }
    if (need) {  // the true residual b - A d, and the active set at it
      take(a.pub_d, it);
      if (own) {
        double y = diag * d;
        for (int k = 0; k < deg; ++k) y += C[k * row + tid] * V[k * row + tid];
        r = fx ? 0.0 : b - y;
        const bool an = bound_active(d, lb, r, fx);
        if (an != act) v2[2] = 1.0;
        act = an;
      }
    }
    if (own) {
      const double rf = act ? 0.0 : r;
      z = act ? 0.0 : rf * mi;
      st_tagged(a.pub_z + node, z, it + 1);
      v2[0] = rf * rf;
      v2[1] = rf * z;
    }
    if (!grid_reduce<3, 0, kT>(v2, gs) || s_lost) return;
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
  if (own) a.d[node] = fx ? a.vals[node] : fmin(fmax(d, lb), 1.0);
  if (blockIdx.x == 0 && tid == 0) {
    a.st->done = 1;
    a.st->iter = it;
    a.st->reason = reason;
    a.st->last_iter = last;
  }
}

}  // namespace

// Bytes behind the engine's workspace for the adjacency table of up to kMaxColours colours.
size_t t3_ppcg_extra_bytes(int n) { return align_up(sizeof(int) * kMaxColours * (size_t)n); }

// ppcg_solve of an element-history damage model on a T3 mesh; `adj` holds t3_ppcg_extra_bytes.
// PHASTB_UNSUPPORTED: too many nodes or colours, a workspace that is not 16-byte aligned (the exchange words are), or
// no cooperative launch; nothing was launched.
int t3_ppcg_persistent(const phastb_t3_mesh& mesh, const phastb_t3_damage_model& md, const double* H, const PpcgWs& w,
                       int* adj, const double* d_prev, const double* d_init, const uint8_t* fixed, const double* vals,
                       double tol, int max_iter, int check_every, double* d, int* info, cudaStream_t s) {
  int dev = 0, sms = 0, coop = 0;
  if (md.nodal_h || !persistent_pcg_enabled() || mesh.n_colors < 1 || mesh.n_colors > kMaxColours)
    return PHASTB_UNSUPPORTED;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  const int n = mesh.n_nodes, most = std::min(sms, kGridBlocks);
  T3PpcgArgs a;
  std::memset(&a, 0, sizeof(a));
  // every SM gets a share of at least 128 nodes; a node has one element per colour at most, with two
  // neighbours each
  const int blocks = std::min(most, std::max(1, (n + 127) / 128));
  a.per = (n + blocks - 1) / blocks;
  a.row = (a.per + 31) / 32 * 32;
  a.deg = 2 * mesh.n_colors;
  const size_t smem = (3 * sizeof(double) + sizeof(int)) * (size_t)a.deg * a.row;
  if (!coop || a.per > kT || smem > kSmemMax || !aligned16(w.r) || !aligned16(w.p) || !aligned16(w.part))
    return PHASTB_UNSUPPORTED;
  const int grid = (n + a.per - 1) / a.per;
  a.n = n;
  a.colours = mesh.n_colors;
  a.max_iter = max_iter;
  a.check_every = check_every;
  a.tol = tol;
  a.elem = mesh.elem;
  a.adj = adj;
  a.grad = mesh.grad;
  a.areas = mesh.areas;
  a.H = H;
  a.gco = md.gc_over_l0;
  a.gcl0 = md.gcl0;
  a.src = md.source;
  a.gco_e = md.gc_over_l0_e;
  a.gcl0_e = md.gcl0_e;
  a.src_e = md.source_e;
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
  int st = cuda_status(cudaMemsetAsync(w.part, 0, grid_slot_bytes(), s));
  if (!st) st = cuda_status(cudaMemsetAsync(w.counter, 0, 4 * sizeof(unsigned), s));
  if (!st) st = cuda_status(cudaMemsetAsync(a.pub_z, 0, (size_t)n * sizeof(Tagged), s));
  if (!st) st = cuda_status(cudaMemsetAsync(a.pub_d, 0, (size_t)n * sizeof(Tagged), s));
  if (!st) st = cuda_status(cudaMemsetAsync(adj, 0xff, sizeof(int) * (size_t)a.colours * n, s));
  if (st) return st;
  ColourOffsets co;
  std::memset(&co, 0, sizeof(co));
  for (int c = 0; c <= mesh.n_colors; ++c) co.off[c] = mesh.color_off[c];
  { note_launch(); t3_adjacency_kernel<<<grid_for(mesh.n_elems), kThreads, 0, s>>>(n, mesh.n_elems, mesh.n_colors, co, mesh.elem, mesh.order, adj); }
  if ((st = last_launch_status())) return st;
  void* args[] = {&a};
  if (cudaFuncSetAttribute(t3_ppcg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) !=
          cudaSuccess ||
      cudaLaunchCooperativeKernel((const void*)t3_ppcg_kernel, dim3(grid), dim3(kT), args, smem, s) != cudaSuccess) {
    cudaGetLastError();
    return PHASTB_UNSUPPORTED;
  }
  note_launch();
  // the error flag and the state are neighbours: one read
  struct {
    unsigned err[64];
    PpcgState st;
  } h;
  if ((st = cuda_status(cudaMemcpyAsync(&h, w.counter, sizeof(h), cudaMemcpyDeviceToHost, s)))) return st;
  if ((st = cuda_status(cudaStreamSynchronize(s)))) return st;
  if (h.err[0]) return PHASTB_ERR_CUDA;  // a wait ran out
  info[0] = h.st.last_iter;
  info[1] = h.st.reason;
  return PHASTB_OK;
}

}  // namespace phastb
