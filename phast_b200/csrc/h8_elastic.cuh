// The elastic voxel element in its modal (Haar) form, as the marching kernels evaluate it: a thread goes up an
// element column, forms each node layer's face modes once, keeps them as the lower face of the next element, and
// adds there the forces of the two elements that share the face.
#pragma once
#include "h8_march.cuh"

namespace phastb {

// One node layer as an element sees it: the four corner values of u~ in the Haar basis of the
// face (x difference X, y difference Y, mixed difference XY; the sum M as four times the first
// corner's value V plus differences R, so that only differences of nodal values are ever rounded),
// and 1 - d at the face's four Gauss positions o[qx + 2 qy] (interpolated in x and y).
template <typename T>
struct Face {
  T V[3], R[3], X[3], Y[3], XY[3];
  T o[4];
};

// The element's share of a node layer's forces, in the same Haar basis.
template <typename T>
struct FaceForce {
  T M[3], X[3], Y[3], XY[3];
};

// The face of the corner values v[corner][component], corner = (x side) + 2 (y side).
template <typename T, int W>
__device__ __forceinline__ void elastic_face(const T (&v)[4][W], Face<T>& f) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T d0 = v[1][c] - v[0][c], d1 = v[3][c] - v[2][c];
    const T e0 = v[2][c] - v[0][c], e1 = v[3][c] - v[1][c];
    f.V[c] = v[0][c];
    f.X[c] = d0 + d1;
    f.Y[c] = e0 + e1;
    f.XY[c] = d1 - d0;
    f.R[c] = f.X[c] + T(2) * e0;
  }
}
// 1 - d of the corners at the face's Gauss positions.
template <typename T>
__device__ __forceinline__ void damage_face(T d0, T d1, T d2, T d3, const TileK<T>& k, Face<T>& f) {
  T a0, a1, b0, b1;
  ip2(T(1) - d0, T(1) - d1, k.c1, k.c2, a0, a1);
  ip2(T(1) - d2, T(1) - d3, k.c1, k.c2, b0, b1);
  ip2(a0, b0, k.c1, k.c2, f.o[0], f.o[2]);
  ip2(a1, b1, k.c1, k.c2, f.o[1], f.o[3]);
}
// 1 - d at Gauss point q of the half qz between the faces l and u.
template <typename T>
__device__ __forceinline__ T intact_at(const Face<T>& l, const Face<T>& u, const TileK<T>& k, int qz, int q) {
  return qz ? k.c2 * l.o[q] + k.c1 * u.o[q] : k.c1 * l.o[q] + k.c2 * u.o[q];
}

// Forces of the element between the faces l and u: adds to lo (lower face), assigns up.  half(qz) comes before the
// four Gauss points q of a half, stress(q, ep, sg) gives the weighted stress of the strain ep there, and rows(c,
// sx, sy, sz) receives sum_q sigma for the gradient components d u_c / dx, dy, dz.  STRAIN: the macro strain E6
// enters each strain component once, in the gradient term that component starts from.
template <bool STRAIN, typename T, class Half, class Stress, class Rows>
__device__ __forceinline__ void elastic_element(const Face<T>& fl, const Face<T>& fu, const TileK<T>& k, const T* E6,
                                                Half half, Stress stress, Rows rows, FaceForce<T>& lo,
                                                FaceForce<T>& up) {
  // z modes of the element: sums (X, Y, XY) and differences (Mz, Xz, Yz, XYz) of the two faces
  T X[3], Y[3], XY[3], Mz[3], Xz[3], Yz[3], XYz[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    X[c] = fl.X[c] + fu.X[c];
    Y[c] = fl.Y[c] + fu.Y[c];
    XY[c] = fl.XY[c] + fu.XY[c];
    Mz[c] = T(4) * (fu.V[c] - fl.V[c]) + (fu.R[c] - fl.R[c]);
    Xz[c] = fu.X[c] - fl.X[c];
    Yz[c] = fu.Y[c] - fl.Y[c];
    XYz[c] = fu.XY[c] - fl.XY[c];
  }
  // d u_c / dz at [qy][qx]
  T Dz[3][2][2], Pz[3][2][2];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int qx = 0; qx < 2; ++qx) {
      const T sx = qx ? k.g : -k.g;
      const T A = Mz[c] + sx * Xz[c], B = Yz[c] + sx * XYz[c];
      const T t = k.az * A + (STRAIN ? (c == 0 ? E6[4] : (c == 1 ? E6[3] : E6[2])) : T(0));
      Dz[c][0][qx] = t - k.bz * B;
      Dz[c][1][qx] = t + k.bz * B;
    }
  // sums over the Gauss points of each half (qz = 0, 1) for the transposed gradient
  T Sx[3][2], Sy[3][2], Sxy[3][2];
#pragma unroll
  for (int qz = 0; qz < 2; ++qz) {
    const T sz = qz ? k.g : -k.g;
    T Dx[3][2], Dy[3][2];  // [qy], [qx]
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const T Ax = X[c] + sz * Xz[c], Ay = Y[c] + sz * Yz[c], B = XY[c] + sz * XYz[c];
      const T tx = k.ax * Ax + (STRAIN && c == 0 ? E6[0] : T(0));
      const T ty = k.ay * Ay + (STRAIN && c == 0 ? E6[5] : (STRAIN && c == 1 ? E6[1] : T(0)));
      Dx[c][0] = tx - k.bx * B;
      Dx[c][1] = tx + k.bx * B;
      Dy[c][0] = ty - k.by * B;
      Dy[c][1] = ty + k.by * B;
    }
    half(qz);
    T Px[3][2], Py[3][2];
#pragma unroll
    for (int qy = 0; qy < 2; ++qy)
#pragma unroll
      for (int qx = 0; qx < 2; ++qx) {
        T ep[6], sg[6];
        ep[0] = Dx[0][qy];
        ep[1] = Dy[1][qx];
        ep[2] = Dz[2][qy][qx];
        ep[3] = Dz[1][qy][qx] + Dy[2][qx];
        ep[4] = Dz[0][qy][qx] + Dx[2][qy];
        ep[5] = Dy[0][qx] + Dx[1][qy];
        stress(qx + 2 * qy, ep, sg);
        // first contribution to a sum assigns, the others add
        Px[0][qy] = qx == 0 ? sg[0] : Px[0][qy] + sg[0];
        Px[1][qy] = qx == 0 ? sg[5] : Px[1][qy] + sg[5];
        Px[2][qy] = qx == 0 ? sg[4] : Px[2][qy] + sg[4];
        Py[0][qx] = qy == 0 ? sg[5] : Py[0][qx] + sg[5];
        Py[1][qx] = qy == 0 ? sg[1] : Py[1][qx] + sg[1];
        Py[2][qx] = qy == 0 ? sg[3] : Py[2][qx] + sg[3];
        Pz[0][qy][qx] = qz == 0 ? sg[4] : Pz[0][qy][qx] + sg[4];
        Pz[1][qy][qx] = qz == 0 ? sg[3] : Pz[1][qy][qx] + sg[3];
        Pz[2][qy][qx] = qz == 0 ? sg[2] : Pz[2][qy][qx] + sg[2];
      }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Sx[c][qz] = Px[c][0] + Px[c][1];
      Sy[c][qz] = Py[c][0] + Py[c][1];
      Sxy[c][qz] = k.ax * (Px[c][1] - Px[c][0]) + k.ay * (Py[c][1] - Py[c][0]);
    }
  }
  // transposed gradient: the element's modal forces, split into its two faces
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T p0 = Pz[c][0][0] + Pz[c][0][1], p1 = Pz[c][1][0] + Pz[c][1][1];
    const T m0 = Pz[c][0][1] - Pz[c][0][0], m1 = Pz[c][1][1] - Pz[c][1][0];
    const T T0 = p0 + p1, TY = p1 - p0, TX = m0 + m1, TXY = m1 - m0;
    const T sx = Sx[c][0] + Sx[c][1], sy = Sy[c][0] + Sy[c][1];
    rows(c, sx, sy, T0);
    const T fX = k.ax * sx, fY = k.ay * sy, fXY = k.g * (Sxy[c][0] + Sxy[c][1]);
    const T fM = k.az * T0;
    const T fXz = k.bx * (Sx[c][1] - Sx[c][0]) + k.bz * TX;
    const T fYz = k.by * (Sy[c][1] - Sy[c][0]) + k.bz * TY;
    const T fXYz = k.g * (k.g * (Sxy[c][1] - Sxy[c][0]) + k.bz * TXY);
    lo.M[c] -= fM;
    lo.X[c] += fX - fXz;
    lo.Y[c] += fY - fYz;
    lo.XY[c] += fXY - fXYz;
    up.M[c] = fM;
    up.X[c] = fX + fXz;
    up.Y[c] = fY + fYz;
    up.XY[c] = fXY + fXYz;
  }
}

// Corner forces of a node layer, corner L = (x side) + 2 (y side), component c at fc[(3 L + c) n + t].
template <typename T>
__device__ __forceinline__ void corner_forces(const FaceForce<T>& f, T* fc, int n, int t) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T mm = f.M[c] - f.Y[c], mp = f.M[c] + f.Y[c];
    const T xm = f.X[c] - f.XY[c], xp = f.X[c] + f.XY[c];
    fc[c * n + t] = mm - xm;
    fc[(3 + c) * n + t] = mm + xm;
    fc[(6 + c) * n + t] = mp - xp;
    fc[(9 + c) * n + t] = mp + xp;
  }
}
// A node's sum over the four columns that meet there (their elements t11, t01, t10, t00).
template <typename T>
__device__ __forceinline__ T node_force(const T* fc, int n, int c, int t11, int t01, int t10, int t00) {
  return (fc[c * n + t11] + fc[(3 + c) * n + t01]) + (fc[(6 + c) * n + t10] + fc[(9 + c) * n + t00]);
}

// Weighted isotropic stress of strain ep.
template <typename T>
__device__ __forceinline__ void iso_stress(T lg, T mg, const T (&ep)[6], T (&sg)[6]) {
  const T mg2 = mg + mg;
  const T lt = lg * (ep[0] + ep[1] + ep[2]);
  sg[0] = mg2 * ep[0] + lt;
  sg[1] = mg2 * ep[1] + lt;
  sg[2] = mg2 * ep[2] + lt;
  sg[3] = mg * ep[3];
  sg[4] = mg * ep[4];
  sg[5] = mg * ep[5];
}

}  // namespace phastb
