// Sum-factorised strain and B^T stress of one 2x2x2-Gauss box Hex8 element, one thread per
// element.
//
// Node a = ax + 2 ay + 4 az sits at (+/-1)^3 by its bits, point q = 4 h + 2 by + bz at
// (h, by, bz) -> (+/-) 1/sqrt(3) along (x, y, z).  On a box the nodal interpolation factors
// into one-dimensional sums and differences, and a derivative does not depend on the
// coordinate it is taken along, so the element's 72 derivatives at its 8 points are only 36
// distinct values: the forward pass takes ~180 operations and its transpose ~210, against
// 8 x (72 + 96) for a strain-displacement product per Gauss point.  The points of one x half
// (h) are handled together, so that the live values fit the register file: the second half
// reuses the registers of the first.
#pragma once

#include <cuda_runtime.h>

namespace cib {

// c: 1 / (4 edge) per direction; w: the same times the integration weight; g = 1/sqrt(3).
template <typename T>
struct BoxCoef {
  T cx, cy, cz;
  T wx, wy, wz;
};

template <typename T>
__device__ __forceinline__ BoxCoef<T> box_coef(double hx, double hy, double hz) {
  const double jw = hx * hy * hz / 8.0;
  BoxCoef<T> c;
  c.cx = (T)(0.25 / hx);
  c.cy = (T)(0.25 / hy);
  c.cz = (T)(0.25 / hz);
  c.wx = (T)(0.25 * jw / hx);
  c.wy = (T)(0.25 * jw / hy);
  c.wz = (T)(0.25 * jw / hz);
  return c;
}

// out(a, d, v): v = sum over the 8 points of weight * (B_a^T sigma)_d, with sigma a point's map of
// eps = B u (Voigt xx, yy, zz, yz, xz, xy; engineering shear).  `node(a, d)` returns the nodal
// value; `point.half(h)` is called before the four points of a half (its loads go there);
// `point(p, eps, sig)` maps the strain of point q = 4 h + p to its stress.
template <typename T, typename Node, typename Point, typename Out>
__device__ __forceinline__ void box_element(const BoxCoef<T>& c, const Node& node, Point& point, const Out& out) {
  const T g = (T)0.57735026918962576451;
  const T g2 = (T)(1.0 / 3.0);
  point.half(0);  // its loads overlap the transforms below
  T S[4][3], Q[4][3];  // corner (y, z) = yz & 1, yz >> 1: sum and difference along x
  T X[3][4];           // d u_d / dx at (by, bz) = 2 by + bz (the same in both halves)
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T u0 = node(2 * k, d), u1 = node(2 * k + 1, d);
      S[k][d] = u0 + u1;
      Q[k][d] = u1 - u0;
    }
    const T a = Q[1][d] - Q[0][d], b = Q[3][d] - Q[2][d];
    const T n0 = c.cx * ((Q[0][d] + Q[1][d]) + (Q[2][d] + Q[3][d]));
    const T ny = c.cx * g * (a + b), nz = c.cx * g * ((Q[2][d] - Q[0][d]) + (Q[3][d] - Q[1][d]));
    const T nyz = c.cx * g2 * (b - a);
    const T lo = n0 - ny, hi = n0 + ny, dl = nz - nyz, dh = nz + nyz;
    X[d][0] = lo - dl;
    X[d][1] = lo + dl;
    X[d][2] = hi - dh;
    X[d][3] = hi + dh;
  }
  T FX[3][4];
  T sum[4][3], dif[4][3];  // of the corner: nodes u1 = sum + dif, u0 = sum - dif
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h == 1) point.half(1);
    T Y[3][2], Z[3][2];  // d u_d / dy at bz, d u_d / dz at by
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      T P[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) P[k] = h ? S[k][d] + g * Q[k][d] : S[k][d] - g * Q[k][d];
      const T a = P[1] - P[0], b = P[3] - P[2];
      const T my = c.cy * (a + b), mz = c.cz * ((P[2] - P[0]) + (P[3] - P[1])), myz = g * (b - a);
      Y[d][0] = my - c.cy * myz;
      Y[d][1] = my + c.cy * myz;
      Z[d][0] = mz - c.cz * myz;
      Z[d][1] = mz + c.cz * myz;
    }
    T FY[3][2], FZ[3][2];
#pragma unroll
    for (int by = 0; by < 2; ++by)
#pragma unroll
      for (int bz = 0; bz < 2; ++bz) {
        const int p = 2 * by + bz;
        const T eps[6] = {X[0][p],           Y[1][bz],           Z[2][by],
                          Z[1][by] + Y[2][bz], Z[0][by] + X[2][p], Y[0][bz] + X[1][p]};
        T s[6];
        point(p, eps, s);
        FX[0][p] = h ? FX[0][p] + s[0] : s[0];
        FX[1][p] = h ? FX[1][p] + s[5] : s[5];
        FX[2][p] = h ? FX[2][p] + s[4] : s[4];
        FY[0][bz] = by ? FY[0][bz] + s[5] : s[5];
        FY[1][bz] = by ? FY[1][bz] + s[1] : s[1];
        FY[2][bz] = by ? FY[2][bz] + s[3] : s[3];
        FZ[0][by] = bz ? FZ[0][by] + s[4] : s[4];
        FZ[1][by] = bz ? FZ[1][by] + s[3] : s[3];
        FZ[2][by] = bz ? FZ[2][by] + s[2] : s[2];
      }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const T my = c.wy * (FY[d][0] + FY[d][1]), mz = c.wz * (FZ[d][0] + FZ[d][1]);
      const T myz = g * (c.wy * (FY[d][1] - FY[d][0]) + c.wz * (FZ[d][1] - FZ[d][0]));
      const T t1 = my - myz, t2 = my + myz;
      const T pb[4] = {-t1 - mz, t1 - mz, mz - t2, t2 + mz};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        dif[k][d] = h ? g * (pb[k] - sum[k][d]) : (T)0;
        sum[k][d] = h ? sum[k][d] + pb[k] : pb[k];
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const T a = FX[d][0] + FX[d][1], b = FX[d][2] + FX[d][3];  // by = 0, 1
    const T e = FX[d][1] - FX[d][0], f = FX[d][3] - FX[d][2];
    const T n0 = c.wx * (a + b), ny = c.wx * g * (b - a), nz = c.wx * g * (e + f), nyz = c.wx * g2 * (f - e);
    const T lo = n0 - ny, hi = n0 + ny, dl = nz - nyz, dh = nz + nyz;
    const T qb[4] = {lo - dl, hi - dh, lo + dl, hi + dh};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T t = dif[k][d] + qb[k];
      out(2 * k, d, sum[k][d] - t);
      out(2 * k + 1, d, sum[k][d] + t);
    }
  }
}

// The FP32 element of the linear solves: strain, tangent and B^T stress of all 8 points by
// their strain-displacement products, one thread per element.  Three times the operations of
// box_element, but in the order and rounding of a thread-per-point product with a butterfly
// sum over the points: FP32 Newton steps are solved inexactly and stop on thresholds, so a
// solve that rounds differently can end one iteration earlier or later and leave a visibly
// different (equally valid) fluctuation.  Box gradients have three magnitudes per direction.
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }

template <typename T>
struct BoxGrad {
  T x[3], y[3], z[3];  // (1/8) f f' 2 / edge with 0, 1 or 2 of the factors f = 1 + 1/sqrt(3), else 1 - 1/sqrt(3)
};

template <typename T>
__device__ __forceinline__ BoxGrad<T> box_grad(double hx, double hy, double hz) {
  const T sx = (T)2 / (T)hx, sy = (T)2 / (T)hy, sz = (T)2 / (T)hz;
  const T gp = (T)0.57735026918962576451;
  const T lo = (T)1 - gp, hi = (T)1 + gp;
  const T m[3] = {(T)0.125 * lo * lo, (T)0.125 * lo * hi, (T)0.125 * hi * hi};
  BoxGrad<T> g;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    g.x[k] = m[k] * sx;
    g.y[k] = m[k] * sy;
    g.z[k] = m[k] * sz;
  }
  return g;
}

// dN_a / dx_d at point q (both compile-time after unrolling).
template <typename T>
__device__ __forceinline__ T box_grad_entry(const BoxGrad<T>& g, int a, int q, int d) {
  const int mx = ((a & 1) != 0) == ((q & 4) != 0), my = ((a & 2) != 0) == ((q & 2) != 0),
            mz = ((a & 4) != 0) == ((q & 1) != 0);
  const T v = d == 0 ? g.x[my + mz] : d == 1 ? g.y[mx + mz] : g.z[mx + my];
  return (a & (1 << d)) ? v : -v;
}

template <typename T, typename Node, typename Point, typename Out>
__device__ __forceinline__ void box_element_points(const BoxGrad<T>& g, T w, const Node& node, Point& point,
                                                   const Out& out) {
  T s[8][6];
  {
    T u[8][3];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int d = 0; d < 3; ++d) u[a][d] = node(a, d);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if ((q & 1) == 0) point.pair(q >> 1);
      T exx = 0, eyy = 0, ezz = 0, gyz = 0, gxz = 0, gxy = 0;
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const T gx = box_grad_entry(g, a, q, 0), gy = box_grad_entry(g, a, q, 1), gz = box_grad_entry(g, a, q, 2);
        exx = fma_(gx, u[a][0], exx);
        eyy = fma_(gy, u[a][1], eyy);
        ezz = fma_(gz, u[a][2], ezz);
        gyz = add_(gyz, fma_(gz, u[a][1], mul_(gy, u[a][2])));
        gxz = add_(gxz, fma_(gz, u[a][0], mul_(gx, u[a][2])));
        gxy = add_(gxy, fma_(gy, u[a][0], mul_(gx, u[a][1])));
      }
      const T e[6] = {exx, eyy, ezz, gyz, gxz, gxy};
      point(q & 1, e, s[q]);
    }
  }
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    T f[8][3];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const T gx = box_grad_entry(g, a, q, 0), gy = box_grad_entry(g, a, q, 1), gz = box_grad_entry(g, a, q, 2);
      f[q][0] = mul_(w, fma_(gy, s[q][5], fma_(gx, s[q][0], mul_(gz, s[q][4]))));
      f[q][1] = mul_(w, fma_(gx, s[q][5], fma_(gy, s[q][1], mul_(gz, s[q][3]))));
      f[q][2] = mul_(w, fma_(gx, s[q][4], fma_(gz, s[q][2], mul_(gy, s[q][3]))));
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      out(a, d, ((f[0][d] + f[4][d]) + (f[2][d] + f[6][d])) + ((f[1][d] + f[5][d]) + (f[3][d] + f[7][d])));
  }
}

}  // namespace cib
