// Device helpers of the marching voxel kernels: periodic wraps, asynchronous
// copies into shared memory, and the scalar damage element in its modal form.
#pragma once
#include "h8_tile.cuh"

namespace phastb {

// Index of a node coordinate along one axis after the periodic wrap; -1 when
// the coordinate lies outside a non-periodic grid.  |c| stays within one
// period because tiles are never wider than the grid.
__device__ __forceinline__ int wrap_node(int c, int n, int r, int periodic) {
  if (periodic) return c < 0 ? c + n : (c >= n ? c - n : c);
  return (c >= 0 && c < r) ? c : -1;
}

__device__ __forceinline__ int wrap_elem(int c, int n, int periodic) {
  if (periodic) return c < 0 ? c + n : (c >= n ? c - n : c);
  return (c >= 0 && c < n) ? c : -1;
}

// Asynchronous global -> shared copies (cp.async, 16 bytes, L2 only).  A thread
// stages the per-element arrays of the NEXT element layer into its own slot of
// a two-buffer shared array and waits for its own group before reading it, so
// no barrier is needed for these slots; both addresses must be 16-byte aligned.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// One word (4 or 8 bytes, naturally aligned) with cp.async.
template <typename T>
__device__ __forceinline__ void cp_async_word(T* smem, const T* gmem) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "cp.async copies 4, 8 or 16 bytes");
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(sizeof(T)) : "memory");
}
// One word, or zero where `live` is false (the source is then not read).
template <typename T>
__device__ __forceinline__ void cp_async_word_or_zero(T* smem, const T* gmem, bool live) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "cp.async copies 4, 8 or 16 bytes");
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const unsigned n = live ? (unsigned)sizeof(T) : 0u;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gmem), "n"(sizeof(T)), "r"(n)
               : "memory");
}

// Staged per-element arrays live chunk-major in shared memory: chunk c (16
// bytes) of the element owned by thread t sits at base + (c * n + t) * 16, so a
// warp reading one chunk touches consecutive 16-byte units (no bank conflicts).
// Copies n_chunks 16-byte chunks of src into chunks c0.. of thread t's column.
__device__ __forceinline__ void stage_chunks(unsigned char* base, int n, int t, int c0, const void* src,
                                             int n_chunks) {
  for (int c = 0; c < n_chunks; ++c)
    cp_async16(base + ((size_t)(c0 + c) * n + t) * 16, static_cast<const unsigned char*>(src) + 16 * c);
}

// Reads W words of thread t's staged column (W * sizeof(T) a multiple of 16).
template <typename T, int W>
__device__ __forceinline__ void load_chunks(const unsigned char* base, int n, int t, T (&out)[W]) {
  using V = typename Vec16<T>::type;
  constexpr int per = 16 / sizeof(T);
#pragma unroll
  for (int c = 0; c < W / per; ++c) {
    const V v = *reinterpret_cast<const V*>(base + ((size_t)c * n + t) * 16);
    const T* pv = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int j = 0; j < per; ++j) out[c * per + j] = pv[j];
  }
}

template <typename T>
__device__ __forceinline__ void ip2(T a0, T a1, T c1, T c2, T& q0, T& q1) {
  q0 = c1 * a0 + c2 * a1;
  q1 = c2 * a0 + c1 * a1;
}

// ---- the scalar damage element
//
// One node layer of the scalar field as an element sees it, in the Haar basis of the face (see Face of
// the elastic action: x, y and mixed differences, the sum as 4 V + R).
template <typename T>
struct DFace {
  T V, R, X, Y, XY;
};
template <typename T>
__device__ __forceinline__ DFace<T> dface(T v0, T v1, T v2, T v3) {
  const T d0 = v1 - v0, d1 = v3 - v2, e0 = v2 - v0, e1 = v3 - v1;
  DFace<T> f;
  f.V = v0;
  f.X = d0 + d1;
  f.Y = e0 + e1;
  f.XY = d1 - d0;
  f.R = f.X + T(2) * e0;
  return f;
}
// An element's share of a node layer's result, in the same basis.
template <typename T>
struct DForce {
  T M, X, Y, XY;
};

// Constants of the element: g = 1/sqrt(3), and 4 scale / (4 h)^2 per axis (the Laplacian's mode factors).
template <typename T>
struct DElemK {
  T g, g2, cx, cy, cz;
};

// scale * [Gc (M / ell + ell L) + 2 (1 - kappa) H-mass] of one element between the faces l and u: adds to lo
// (lower face) and assigns up.  gcw = w scale gc_ell / 64 and chw = w scale 2 (1 - kappa) / 64 weight the Gauss
// points' masses, k2 = 2 w Gc ell the Laplacian.  In the modal basis the interpolation to the Gauss points is
// three butterflies, and the Laplacian of the brick is diagonal: 115 operations, where interpolating the nodal
// values and their gradients takes 300.
template <typename T>
__device__ __forceinline__ void damage_element(const DFace<T>& l, const DFace<T>& u, const T (&h)[8], T gcw, T chw,
                                               T k2, const DElemK<T>& c, DForce<T>& lo, DForce<T>& up) {
  const T Ml = T(4) * l.V + l.R, Mu = T(4) * u.V + u.R;
  const T M = Ml + Mu, X = l.X + u.X, Y = l.Y + u.Y, XY = l.XY + u.XY;
  const T Z = T(4) * (u.V - l.V) + (u.R - l.R), XZ = u.X - l.X, YZ = u.Y - l.Y, XYZ = u.XY - l.XY;
  // values (times 8) at the Gauss points q = qx + 2 qy + 4 qz
  T q[8];
  {
    const T a0 = M - c.g * X, a1 = M + c.g * X, b0 = Y - c.g * XY, b1 = Y + c.g * XY;
    const T s0 = Z - c.g * XZ, s1 = Z + c.g * XZ, t0 = YZ - c.g * XYZ, t1 = YZ + c.g * XYZ;
    const T A0 = a0 - c.g * b0, A1 = a1 - c.g * b1, A2 = a0 + c.g * b0, A3 = a1 + c.g * b1;
    const T B0 = s0 - c.g * t0, B1 = s1 - c.g * t1, B2 = s0 + c.g * t0, B3 = s1 + c.g * t1;
    q[0] = A0 - c.g * B0;
    q[1] = A1 - c.g * B1;
    q[2] = A2 - c.g * B2;
    q[3] = A3 - c.g * B3;
    q[4] = A0 + c.g * B0;
    q[5] = A1 + c.g * B1;
    q[6] = A2 + c.g * B2;
    q[7] = A3 + c.g * B3;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] *= gcw + chw * h[i];
  // transposed: sums and differences over z, y, x, then the factors of g
  const T z0 = q[0] + q[4], z1 = q[1] + q[5], z2 = q[2] + q[6], z3 = q[3] + q[7];
  const T y0 = q[4] - q[0], y1 = q[5] - q[1], y2 = q[6] - q[2], y3 = q[7] - q[3];
  const T zs0 = z0 + z2, zs1 = z1 + z3, zd0 = z2 - z0, zd1 = z3 - z1;
  const T ys0 = y0 + y2, ys1 = y1 + y3, yd0 = y2 - y0, yd1 = y3 - y1;
  const T kx = k2 * c.cx, ky = k2 * c.cy, kz = k2 * c.cz;
  const T fM = zs0 + zs1;
  const T fX = c.g * (zs1 - zs0) + kx * X;
  const T fY = c.g * (zd0 + zd1) + ky * Y;
  const T fXY = c.g2 * ((zd1 - zd0) + (kx + ky) * XY);
  const T fZ = c.g * (ys0 + ys1) + kz * Z;
  const T fXZ = c.g2 * ((ys1 - ys0) + (kx + kz) * XZ);
  const T fYZ = c.g2 * ((yd0 + yd1) + (ky + kz) * YZ);
  const T fXYZ = c.g2 * (c.g * (yd1 - yd0) + c.g2 * ((kx + ky + kz) * XYZ));
  lo.M += fM - fZ;
  lo.X += fX - fXZ;
  lo.Y += fY - fYZ;
  lo.XY += fXY - fXYZ;
  up.M = fM + fZ;
  up.X = fX + fXZ;
  up.Y = fY + fYZ;
  up.XY = fXY + fXYZ;
}

// The four corner values of a node layer's result: corner L = (x side) + 2 (y side).
template <typename T>
__device__ __forceinline__ void dcorners(const DForce<T>& f, T (&c)[4]) {
  const T mm = f.M - f.Y, mp = f.M + f.Y, xm = f.X - f.XY, xp = f.X + f.XY;
  c[0] = mm - xm;
  c[1] = mm + xm;
  c[2] = mp - xp;
  c[3] = mp + xp;
}

template <typename T>
__host__ __device__ inline DElemK<T> damage_elem_k(const VoxGeom& g, double scale) {
  const double q = 0.57735026918962576451;
  return DElemK<T>{T(q), T(1.0 / 3.0), T(scale * 0.25 / (g.hx * g.hx)), T(scale * 0.25 / (g.hy * g.hy)),
                   T(scale * 0.25 / (g.hz * g.hz))};
}

}  // namespace phastb
