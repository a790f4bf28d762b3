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

#include "f32x2.cuh"

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

// The FP32 element in the order and rounding of a sum over nodes at each point and over points
// at each node, two points (2 j, 2 j + 1) to an instruction.  dN_a / dx at the two differs in
// the z factor only: the pair is (x[m + 1], x[m]) at a lower node (bit 2 of a clear) and
// (x[m], x[m + 1]) at an upper one, dN_a / dz is the same at both.  The signs (plus where the
// node's bit is set) go to the displacements; in the divergence a common sign is taken out, so
// that one factor at most is negative.  Rounding is symmetric: the results are those of the
// signed gradients.  Bound by issue slots between the solve's barriers: a batch step of 96 RVEs of
// edges 8 to 24 73 -> 58 ms against one point to an instruction.
template <typename Node, typename Point, typename Out>
__device__ __forceinline__ void box_element_points(const BoxGrad<float>& g, float w, const Node& node, Point& point,
                                                   const Out& out) {
  f32x2 x[2][2], y[2][2], z[3];  // [upper][m]
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    x[0][m] = pack2(g.x[m + 1], g.x[m]);
    x[1][m] = pack2(g.x[m], g.x[m + 1]);
    y[0][m] = pack2(g.y[m + 1], g.y[m]);
    y[1][m] = pack2(g.y[m], g.y[m + 1]);
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) z[m] = pack2(g.z[m], g.z[m]);
  f32x2 s[4][6];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 6; ++k) s[j][k] = 0;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const float u[3] = {node(a, 0), node(a, 1), node(a, 2)};
    f32x2 v[2][3];  // [minus]
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      v[0][d] = pack2(u[d], u[d]);
      v[1][d] = pack2(-u[d], -u[d]);
    }
    const int up = a >> 2, nx = !(a & 1), ny = !(a & 2), nz = !(a & 4);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int mx = ((a & 1) != 0) == ((j & 2) != 0), my = ((a & 2) != 0) == ((j & 1) != 0);
      const f32x2 gx = x[up][my], gy = y[up][mx], gz = z[mx + my];
      s[j][0] = fma2(gx, v[nx][0], s[j][0]);
      s[j][1] = fma2(gy, v[ny][1], s[j][1]);
      s[j][2] = fma2(gz, v[nz][2], s[j][2]);
      s[j][3] = add2(s[j][3], fma2(gz, v[nz][1], mul2(gy, v[ny][2])));
      s[j][4] = add2(s[j][4], fma2(gz, v[nz][0], mul2(gx, v[nx][2])));
      s[j][5] = add2(s[j][5], fma2(gy, v[ny][0], mul2(gx, v[nx][1])));
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    point.pair(j);
    float e[2][6], t[2][6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float2 p = unpack2(s[j][k]);
      e[0][k] = p.x, e[1][k] = p.y;
    }
    point(0, e[0], t[0]);
    point(1, e[1], t[1]);
#pragma unroll
    for (int k = 0; k < 6; ++k) s[j][k] = pack2(t[0][k], t[1][k]);
  }
  // The products with w are added up next: as multiply-adds of a zero that the assembler cannot
  // see (w's sign bit; w > 0), so that it does not fuse them with those additions.
  const float none = __uint_as_float(__float_as_uint(w) & 0x80000000u);
  const f32x2 ww = pack2(w, w), zero = pack2(none, none);
#pragma unroll
  for (int c = 0; c < 4; ++c) {  // which factor has the other sign: none, x, y, z
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int a = h == 0 ? (c == 0 ? 7 : c == 1 ? 6 : c == 2 ? 5 : 3) : (c == 0 ? 0 : c == 1 ? 1 : c == 2 ? 2 : 4);
      const int up = a >> 2;
      f32x2 f[4][3];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int mx = ((a & 1) != 0) == ((j & 2) != 0), my = ((a & 2) != 0) == ((j & 1) != 0);
        const f32x2 gx = c == 1 ? neg2(x[up][my]) : x[up][my], gy = c == 2 ? neg2(y[up][mx]) : y[up][mx],
                    gz = c == 3 ? neg2(z[mx + my]) : z[mx + my];
        f[j][0] = fma2(ww, fma2(gy, s[j][5], fma2(gx, s[j][0], mul2(gz, s[j][4]))), zero);
        f[j][1] = fma2(ww, fma2(gx, s[j][5], fma2(gy, s[j][1], mul2(gz, s[j][3]))), zero);
        f[j][2] = fma2(ww, fma2(gx, s[j][4], fma2(gz, s[j][2], mul2(gy, s[j][3]))), zero);
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float2 p = unpack2(add2(add2(f[0][d], f[2][d]), add2(f[1][d], f[3][d])));
        out(a, d, h == 0 ? p.x + p.y : -(p.x + p.y));
      }
    }
  }
}

}  // namespace cib
