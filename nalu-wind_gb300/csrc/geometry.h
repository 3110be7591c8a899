// Hex8 / Tet4 sub-control-surface area vectors and sub-control volumes of
// one element, shared by the host mesh generator (workload.cpp) and the
// device geometry kernels (geometry.cu). Both are compiled without fused
// multiply-adds (host -ffp-contract=off, device -fmad=false), so the same
// coordinates give the same bits on either side.
#pragma once

#include <cmath>

#include "dd.h"  // NW_HD

namespace nw {

// Vector area of a quadrilateral sub-control surface q0 q1 q2 q3: half the
// cross product of its diagonals. The vector area of a closed polygon
// depends only on its boundary, so this equals, in exact arithmetic, the
// sum over the four triangles fanned around the face centre that
// Quad3DSCS / HexSCS::determinant_scs evaluate (planar or not), with one
// cross product instead of four.
NW_HD void quad_area(const double q[4][3], double a[3]) {
  const double d1[3] = {q[2][0] - q[0][0], q[2][1] - q[0][1], q[2][2] - q[0][2]};
  const double d2[3] = {q[3][0] - q[1][0], q[3][1] - q[1][1], q[3][2] - q[1][2]};
  a[0] = 0.5 * (d1[1] * d2[2] - d1[2] * d2[1]);
  a[1] = 0.5 * (d1[2] * d2[0] - d1[0] * d2[2]);
  a[2] = 0.5 * (d1[0] * d2[1] - d1[1] * d2[0]);
}

// a b + c with one rounding, the same on host and device (the files are
// compiled without contraction, so fused operations are explicit)
NW_HD double geo_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
// o = a x b
NW_HD void geo_cross(const double a[3], const double b[3], double o[3]) {
  o[0] = geo_fma(a[1], b[2], -(a[2] * b[1]));
  o[1] = geo_fma(a[2], b[0], -(a[0] * b[2]));
  o[2] = geo_fma(a[0], b[1], -(a[1] * b[0]));
}
// a . (b x c)
NW_HD double geo_triple(const double a[3], const double b[3], const double c[3]) {
  double x[3];
  geo_cross(b, c, x);
  return geo_fma(a[2], x[2], geo_fma(a[1], x[1], a[0] * x[0]));
}

// Hex8 sub-control surfaces and volumes (HexSCS::determinant_scs,
// HexSCV::determinant_scv, src/master_element/Hex8CVFEM.C:363-389, 565-591)
// from the trilinear map x(u, v, w) of the element, 0 <= u, v, w <= 1.
//
// The reference evaluates each sub-surface as four triangles about its
// centre and each sub-volume by Grandy's formula over its six faces, fanned
// about their centres. The sub-surfaces and the faces of the sub-volumes are
// bilinear patches of the trilinear map; the fans give the patch's vector
// area and enclosed volume exactly, so both equal the integrals of the map:
//   surface  S = int x_v x x_w dv dw      (on u = 1/2, and cyclic)
//   volume   V = int [x_u, x_v, x_w]      (over one octant)
// (brackets: triple product). With the seven difference vectors of the map,
//   A, B, C = mean x_u, x_v, x_w;  P, Q, R = mean x_vw, x_wu, x_uv;  T = x_uvw,
// the integrands are polynomials and the integrals closed forms:
//   S(v, w) = 1/4 (B x C +- 1/4 B x P +- 1/4 P x C), one sign per half, and
//   V = 1/8 ([X Y Z] + 1/48 ([X R Q] + [R Y P] + [Q P Z]))
// with the vectors at the octant's centre: X = x_u(v, w) = A +- R/4 +- Q/4
// +- T/16 (cyclic), P = P +- T/4 and so on; all other terms of the
// determinant are odd about the centre or repeat a vector. That is about
// 520 FP64 operations an element (nine cross products for the twelve
// surfaces, twenty for the eight volumes) against about 5,700 for the fans
// and Grandy's formula. The kernel is bound by the FP64 pipe (2 lanes per SM
// clock), so the operation count is its time: the whole update of 96 x 90 x 45
// hexes went from 4.34 to 0.46 ms.
NW_HD void hex_geometry(const double x[8][3], double scs[12][3], double scv[8]) {
  // a = 4 A, b = 4 B, c = 4 C; p = P, q = Q, r = R; t = T / 4
  double a[3], b[3], c[3], p[3], q[3], r[3], t[3];
  for (int d = 0; d < 3; ++d) {
    const double a0 = x[1][d] - x[0][d], a1 = x[2][d] - x[3][d], a2 = x[5][d] - x[4][d],
                 a3 = x[6][d] - x[7][d];
    const double lo = a0 + a1, hi = a2 + a3, dl = a1 - a0, dh = a3 - a2;
    a[d] = lo + hi;
    q[d] = 0.5 * (hi - lo);
    r[d] = 0.5 * (dl + dh);
    t[d] = 0.25 * (dh - dl);
    const double bl = (x[3][d] - x[0][d]) + (x[2][d] - x[1][d]);
    const double bh = (x[7][d] - x[4][d]) + (x[6][d] - x[5][d]);
    b[d] = bl + bh;
    p[d] = 0.5 * (bh - bl);
    c[d] = ((x[4][d] - x[0][d]) + (x[5][d] - x[1][d])) + ((x[7][d] - x[3][d]) + (x[6][d] - x[2][d]));
  }
  // surfaces: S = 1/64 (b x c +- b x p +- p x c); `m` the low half, `h` the
  // high half of the first coordinate, then the two halves of the second
  const double k = 1.0 / 64.0;
  {
    double f[3], g[3], h[3];
    geo_cross(b, c, f);  // u faces: + v with b x p, + w with p x c
    geo_cross(b, p, g);
    geo_cross(p, c, h);
    for (int d = 0; d < 3; ++d) {
      const double vm = f[d] - g[d], vp = f[d] + g[d];
      scs[0][d] = k * (vm - h[d]);    // edge 0-1
      scs[2][d] = -k * (vp - h[d]);   // edge 2-3, against u
      scs[4][d] = k * (vm + h[d]);    // edge 4-5
      scs[6][d] = -k * (vp + h[d]);   // edge 6-7, against u
    }
    geo_cross(c, a, f);  // v faces: + w with c x q, + u with q x a
    geo_cross(c, q, g);
    geo_cross(q, a, h);
    for (int d = 0; d < 3; ++d) {
      const double wm = f[d] - g[d], wp = f[d] + g[d];
      scs[1][d] = k * (wm + h[d]);   // edge 1-2
      scs[3][d] = k * (wm - h[d]);   // edge 0-3
      scs[5][d] = k * (wp + h[d]);   // edge 5-6
      scs[7][d] = k * (wp - h[d]);   // edge 4-7
    }
    geo_cross(a, b, f);  // w faces: + u with a x r, + v with r x b
    geo_cross(a, r, g);
    geo_cross(r, b, h);
    for (int d = 0; d < 3; ++d) {
      const double um = f[d] - g[d], up = f[d] + g[d];
      scs[8][d] = k * (um - h[d]);    // edge 0-4
      scs[9][d] = k * (up - h[d]);    // edge 1-5
      scs[10][d] = k * (up + h[d]);   // edge 2-6
      scs[11][d] = k * (um + h[d]);   // edge 3-7
    }
  }
  // octant centres: X[v][w] = 4 x_u, Y[w][u] = 4 x_v, Z[u][v] = 4 x_w and
  // the mixed derivatives P[u], Q[v], R[w]
  double X[2][2][3], Y[2][2][3], Z[2][2][3], P[2][3], Q[2][3], R[2][3];
  for (int d = 0; d < 3; ++d) {
    P[0][d] = p[d] - t[d];
    P[1][d] = p[d] + t[d];
    Q[0][d] = q[d] - t[d];
    Q[1][d] = q[d] + t[d];
    R[0][d] = r[d] - t[d];
    R[1][d] = r[d] + t[d];
    // a + s_v r + s_w q + s_v s_w t = (a + s_v r) + s_w Q[v]
    const double am = a[d] - r[d], ap = a[d] + r[d];
    X[0][0][d] = am - Q[0][d];
    X[0][1][d] = am + Q[0][d];
    X[1][0][d] = ap - Q[1][d];
    X[1][1][d] = ap + Q[1][d];
    const double bm = b[d] - p[d], bp = b[d] + p[d];
    Y[0][0][d] = bm - R[0][d];
    Y[0][1][d] = bm + R[0][d];
    Y[1][0][d] = bp - R[1][d];
    Y[1][1][d] = bp + R[1][d];
    const double cm = c[d] - q[d], cp = c[d] + q[d];
    Z[0][0][d] = cm - P[0][d];
    Z[0][1][d] = cm + P[0][d];
    Z[1][0][d] = cp - P[1][d];
    Z[1][1][d] = cp + P[1][d];
  }
  double kx[2][2], ky[2][2], kz[2][2];
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j) {
      kx[i][j] = geo_triple(X[i][j], R[j], Q[i]);  // [v][w]
      ky[i][j] = geo_triple(Y[i][j], P[j], R[i]);  // [w][u]
      kz[i][j] = geo_triple(Z[i][j], Q[j], P[i]);  // [u][v]
    }
  const int node[2][2][2] = {{{0, 4}, {3, 7}}, {{1, 5}, {2, 6}}};  // [u][v][w]
  for (int u = 0; u < 2; ++u)
    for (int v = 0; v < 2; ++v)
      for (int w = 0; w < 2; ++w) {
        const double e = kx[v][w] + ky[w][u] + kz[u][v];
        const double det = geo_triple(X[v][w], Y[w][u], Z[u][v]);
        scv[node[u][v][w]] = (1.0 / 512.0) * geo_fma(1.0 / 3.0, e, det);
      }
}

// Tet4 sub-control geometry (TetSCS::determinant_scs / TetSCV::
// determinant_scv, src/master_element/Tet4CVFEM.C:243-360, 522-620).
//
// Sub-control surfaces: each is the quadrilateral (edge midpoint, face
// centroid, element centroid, face centroid) of one edge, and its vector
// area is half the cross product of its diagonals (quad_area). Both
// diagonals are fixed combinations of the edge vectors e_k = c_k - c_0 (one
// runs from a midpoint or face centroid to the centroid or a face centroid:
// (e_a + e_b - e_c) / 4 or e_k / 3 and the like), so every area is a
// small-integer combination of the three cross products X = e1 x e2,
// Y = e2 x e3, Z = e3 x e1, divided by 24. For the facets of edges
// 0-1, 1-2, 2-0, 0-3, 1-3, 2-3 (the reference's ordering of TetSCS's
// integration points): X + 2Y + Z, Z - Y, X + Y + 2Z, 2X + Y + Z, X - Y,
// X - Z. Equal to the reference's four-triangle fans in exact arithmetic,
// with three cross products instead of twenty-four.
NW_HD void tet_geometry(const double c[4][3], double scs[6][3], double scv[4]) {
  double e1[3], e2[3], e3[3];
  for (int d = 0; d < 3; ++d) {
    e1[d] = c[1][d] - c[0][d];
    e2[d] = c[2][d] - c[0][d];
    e3[d] = c[3][d] - c[0][d];
  }
  const double X[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2],
                       e1[0] * e2[1] - e1[1] * e2[0]};
  const double Y[3] = {e2[1] * e3[2] - e2[2] * e3[1], e2[2] * e3[0] - e2[0] * e3[2],
                       e2[0] * e3[1] - e2[1] * e3[0]};
  const double Z[3] = {e3[1] * e1[2] - e3[2] * e1[1], e3[2] * e1[0] - e3[0] * e1[2],
                       e3[0] * e1[1] - e3[1] * e1[0]};
  const double k = 1.0 / 24.0;
  for (int d = 0; d < 3; ++d) {
    scs[0][d] = k * (X[d] + 2.0 * Y[d] + Z[d]);
    scs[1][d] = k * (Z[d] - Y[d]);
    scs[2][d] = k * (X[d] + Y[d] + 2.0 * Z[d]);
    scs[3][d] = k * (2.0 * X[d] + Y[d] + Z[d]);
    scs[4][d] = k * (X[d] - Y[d]);
    scs[5][d] = k * (X[d] - Z[d]);
  }
  // The four sub-control volumes of a linear tet (node, three edge
  // midpoints, three face centroids, centroid) are its barycentric
  // subdivision: equal quarters of the tet's volume (true for a regular
  // tet by symmetry, and volume ratios are affine invariants). TetSCV
  // evaluates each with Grandy's hexahedron formula, equal in exact
  // arithmetic; the signed volume here, (e1 x e2) . e3 / 6, is taken from
  // the edge vectors, which also avoids that formula's cancellation far
  // from the origin.
  const double det = X[0] * e3[0] + X[1] * e3[1] + X[2] * e3[2];
  const double quarter = det / 24.0;
  for (int ip = 0; ip < 4; ++ip) scv[ip] = quarter;
}


}  // namespace nw
