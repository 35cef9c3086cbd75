// tri_edges.cuh -- free-space elastostatic layers on flat triangles as edge
// integrals contracted with the densities, in global coordinates.
//
// For one triangle (unit normal n, edges with unit tangents t, outward
// in-plane normals nu = t x n) and a target x, the layers are derivatives of
// S = int_T r and N = int_T 1/r (r = |x - y|; derivatives by x):
//   single  u = (2 N s - alpha S.. s) / 2 mu,  strain its symmetric gradient,
//   double  u = b Omega + sum_edges [L w - alpha grad (w . grad E)],  w = b x t,
// alpha = (lam + mu) / (lam + 2 mu), E = int_edge r, L = int_edge 1/r, Omega
// the signed solid angle (the dislocation-loop form of the double layer of a
// constant jump: grad Omega = sum int (rho x t) / r^3 is a line integral too,
// so its strain needs no solid angle).  The single layer's in-plane
// derivatives go to the edges by the divergence theorem (S_a.. = -sum nu_a
// E_..), its normal ones follow from laplacian r = 2 / r.
//
// With rho the target's offset from the edge line, u_A, u_B its coordinates
// along t from the edge's ends A, B and R_A, R_B the distances, every
// derivative of E and L is a combination of L, K3 = int 1/r^3, K5 = int
// 1/r^5 and of end differences of 1/R, 1/R^3, u/R, u/R^3, with tensors built
// from t and rho: no frame, no tables.  L, K3 and K5 are sums of positive
// terms on either side of the foot of the target (rho = 0 included: targets
// collinear with an edge), one division and one logarithm per edge.
//
// Compared with derivative tables of the integrals of r and 1/r in the
// triangle frame (45 entries per pair, as the reference's triartable and
// triabtable, src/triahquad.f:680 and :797, rotated per edge, then contracted,
// the form used before): 1,553 FP64 operations per pair of both layers instead
// of 2,758 and two thirds of the registers.  Errors against 113 bits (rms over
// random and thin triangles, heights down to 1e-4 of the base, with fused
// multiply-adds as on the device) beside those of the tables: off the plane 0.05
// to 1.3 times theirs, near it the double layer's strain up to 1.5; close to a
// vertex 1e-2 to 1e-9 of theirs (u and v from the nearer end of an edge), to an
// edge 0.2 to 1.  In the triangle's plane (every planar fault) the single layer
// 0.3 to 1.5; the double layer's sums over the edges cancel further out: 0.1 to
// 1.8 within 3 edge lengths, 0.6 to 2.2 from 10 to 100 (displacement at 30:
// 1.3e-12 against 0.9e-12).
// On-surface evaluation (target on its own triangle) uses h = 0, Omega = 0: the
// principal value / Hadamard finite part, the reference's iquad = 0 convention
// (src/triahquad.f:4037-4055).
#pragma once
#include "tri_index.cuh"

namespace efmm {

// One triangle in global coordinates with its densities (tree order).
struct __align__(16) TriEdge {
  double v[9];     // vertices
  double t[9];     // unit tangents of the edges 0-1, 1-2, 2-0
  double len[3];   // their lengths
  double n[3];     // unit normal
  double area2;    // twice the area
  double pad;
  double s[3];     // single-layer density
  double b[3];     // double-layer density (jump)
};
static_assert(sizeof(TriEdge) == 256, "TriEdge layout");

EFMM_HD void tri_edge_frame(const double* tv, TriEdge& T) {
#pragma unroll
  for (int c = 0; c < 9; c++) T.v[c] = tv[c];
#pragma unroll
  for (int e = 0; e < 3; e++) {
    const double* a = tv + 3 * e;
    const double* b = tv + 3 * (e == 2 ? 0 : e + 1);
    const double d[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
    const double l = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]), il = 1.0 / l;
    T.len[e] = l;
    for (int c = 0; c < 3; c++) T.t[3 * e + c] = d[c] * il;
  }
  const double u[3] = {tv[3] - tv[0], tv[4] - tv[1], tv[5] - tv[2]};
  const double w[3] = {tv[6] - tv[0], tv[7] - tv[1], tv[8] - tv[2]};
  const double c[3] = {u[1] * w[2] - u[2] * w[1], u[2] * w[0] - u[0] * w[2], u[0] * w[1] - u[1] * w[0]};
  T.area2 = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
  for (int k = 0; k < 3; k++) T.n[k] = c[k] / T.area2;
  T.pad = 0.0;
}

EFMM_HD double te_dot(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
EFMM_HD void te_cross(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
// e (xx yy zz xy xz yz) += symmetric part of f a b^T
EFMM_HD void te_sym(double* e, double f, const double* a, const double* b) {
  const double fa[3] = {f * a[0], f * a[1], f * a[2]}, h = 0.5;
  e[0] += fa[0] * b[0];
  e[1] += fa[1] * b[1];
  e[2] += fa[2] * b[2];
  e[3] += h * (fa[0] * b[1] + fa[1] * b[0]);
  e[4] += h * (fa[0] * b[2] + fa[2] * b[0]);
  e[5] += h * (fa[1] * b[2] + fa[2] * b[1]);
}

// Edge integrals L, K3, K5 for ends at u_A, u_B = u_A - len along the edge
// (target's coordinates), distances RA, RB, squared line distance c2.  All
// three diverge when the target lies on the closed edge and are left out
// there (0, as in the reference, src/triahquad.f:1509); what the edge's ends
// contribute stays: it carries the single layer's displacement, which is
// continuous there.
EFMM_HD void te_line(double len, double uA, double uB, double RA, double RB, double iA, double iB, double c2,
                     double& L, double& K3, double& K5) {
  const bool inside = uA > 0.0 && uB < 0.0;  // the foot of the target lies on the edge
  const double a = fabs(uA), b = fabs(uB), pA = RA + a, pB = RB + b, pp = pA * pB;
  L = K3 = K5 = 0.0;
  if (inside ? c2 == 0.0 : !(pp > 0.0)) return;
  const double q = pA + pB, m = pp + c2;
  // inside: 1 / (c2 q); outside: 1 / (pA pB (pA pB + c2))
  const double inv = 1.0 / (inside ? c2 * q : pp * m);
  if (inside) {
    // R_A + R_B - len = c2 (1 / pA + 1 / pB)
    L = log1p(2.0 * len * pp * inv);
    const double ic = inv * q, xa = a * iA, xb = b * iB, sx = xa + xb;
    K3 = sx * ic;
    K5 = (sx - (xa * xa * xa + xb * xb * xb) * (1.0 / 3.0)) * ic * ic;
  } else {
    // R_A + R_B - len = p_near + c2 / p_far
    const double pf = fmax(pA, pB);
    L = log1p(2.0 * len * pf * pp * inv);
    const double ip = inv * m;  // 1 / (pA pB)
    const double gA = iA * ip * pB, gB = iB * ip * pA;
    const double d = fabs(gA - gB), s = gA + gB;
    K3 = d;
    K5 = d * (s - c2 * (1.0 / 3.0) * (s * s - gA * gB));
  }
}

// Offsets r from the vertices to X, distances R and their reciprocals, 0 at a
// vertex itself (the ends' terms that diverge there are left out as the
// edge's are).  Returns the signed distance from the plane, 0 for the
// centroid (self); measured from the nearest vertex it has the rounding of
// that distance and is 0 at a vertex.
EFMM_HD double te_vertices(const TriEdge& T, const double* X, bool self, double r[3][3], double R[3], double iR[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
#pragma unroll
    for (int c = 0; c < 3; c++) r[k][c] = X[c] - T.v[3 * k + c];
    R[k] = sqrt(te_dot(r[k], r[k]));
    iR[k] = R[k] > 0.0 ? 1.0 / R[k] : 0.0;
  }
  const bool n1 = R[1] < R[0], n2 = R[2] < (n1 ? R[1] : R[0]);
  double d[3];
#pragma unroll
  for (int c = 0; c < 3; c++) d[c] = n2 ? r[2][c] : (n1 ? r[1][c] : r[0][c]);
  return self ? 0.0 : te_dot(d, T.n);
}

// Offset from the nearer end of edge k to X (no dynamic register indexing);
// nb: that is its end B.
EFMM_HD void te_near_end(int k, bool nb, const double r[3][3], double d[3]) {
  const bool i0 = nb ? k == 2 : k == 0, i1 = nb ? k == 0 : k == 1;
#pragma unroll
  for (int c = 0; c < 3; c++) d[c] = i0 ? r[0][c] : (i1 ? r[1][c] : r[2][c]);
}

// Response at X of one triangle: displacement u[3] and strain e[6] (if STR),
// ADDED.  self: X is the triangle's centroid (principal value / finite part).
// i2mu = 1 / 2 mu.
template <bool SL, bool DL>
EFMM_HD void tri_edge_pair(const TriEdge& T, const double* X, bool self, bool str, double al, double i2mu, double* u,
                           double* e) {
  double r[3][3], R[3], iR[3];
  const double h = te_vertices(T, X, self, r, R, iR);
  // signed solid angle (Van Oosterom and Strackee 1983), zero in the plane
  double om = 0.0;
  if (h != 0.0 && (SL || DL)) {
    const double den = R[0] * R[1] * R[2] + te_dot(r[0], r[1]) * R[2] + te_dot(r[0], r[2]) * R[1] +
                       te_dot(r[1], r[2]) * R[0];
    om = 2.0 * atan2(h * T.area2, den);
  }
  // single layer, over the edges: N, the normal components of S s (unn), of
  // S_ijk s_k (in-plane row Mn, normal-normal knn) and of grad grad S (kz)
  double N = 0.0, Mn[3] = {0, 0, 0}, unn = 0.0, knn = 0.0, kz = 0.0;
#pragma unroll 1
  for (int k = 0; k < 3; k++) {
    const double* t = T.t + 3 * k;
    const double len = T.len[k];
    // both ends of the edge; u and v from the nearer one, with its rounding (at
    // an end itself both are exactly 0)
    const double RA = k == 0 ? R[0] : (k == 1 ? R[1] : R[2]);
    const double RB = k == 0 ? R[1] : (k == 1 ? R[2] : R[0]);
    const double iA = k == 0 ? iR[0] : (k == 1 ? iR[1] : iR[2]);
    const double iB = k == 0 ? iR[1] : (k == 1 ? iR[2] : iR[0]);
    const bool nb = RB < RA;
    double d[3], nu[3];
    te_near_end(k, nb, r, d);
    const double ud = te_dot(d, t), uA = nb ? ud + len : ud, uB = nb ? ud : ud - len;
    te_cross(t, T.n, nu);
    const double v = te_dot(d, nu);
    const double rho[3] = {v * nu[0] + h * T.n[0], v * nu[1] + h * T.n[1], v * nu[2] + h * T.n[2]};
    const double c2 = v * v + h * h;
    double L, K3, K5;
    te_line(len, uA, uB, RA, RB, iA, iB, c2, L, K3, K5);
    const double di = iA - iB;
    if (SL) {
      const double* s = T.s;
      const double st = te_dot(s, t), sn = te_dot(s, nu), sr = te_dot(s, rho);
      N -= v * L;
      // grad E = t (R_A - R_B) + rho L; R_A - R_B = (u_A^2 - u_B^2) / (R_A + R_B)
      const double Et = len * (uA + uB) / (RA + RB);
      const double f = i2mu * al * (st * Et + sr * L);
#pragma unroll
      for (int c = 0; c < 3; c++) u[c] += nu[c] * f;
      unn += sn * (h * L);
      if (str) {
        // G = (s . grad) grad E; the edge's part of grad N s + s grad N - al S_ijk s_k
        const double du = uA * iA - uB * iB;
        const double ct = st * du + sr * di - L * st, cr = st * di - K3 * sr;
        double y[3], gn = 0.0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double G = ct * t[c] + cr * rho[c] + L * s[c];
          gn += G * T.n[c];
          y[c] = al * G - 2.0 * L * s[c];
        }
        te_sym(e, i2mu, nu, y);
#pragma unroll
        for (int c = 0; c < 3; c++) Mn[c] -= nu[c] * gn;
        knn -= sn * (L - h * h * K3);
        kz -= v * h * K3;
      }
    }
    if (DL) {
      const double* b = T.b;
      double w[3];
      te_cross(b, t, w);
      const double s = te_dot(w, rho);
      const double fw = (1.0 - al) * L, fr = al * K3 * s, ft = al * s * di;
#pragma unroll
      for (int c = 0; c < 3; c++) u[c] += fw * w[c] + fr * rho[c] - ft * t[c];
      if (str) {
        const double iA3 = iA * iA * iA, iB3 = iB * iB * iB;
        // b (rho x t), rho x t = v n - h nu
        const double g[3] = {v * T.n[0] - h * nu[0], v * T.n[1] - h * nu[1], v * T.n[2] - h * nu[2]};
        te_sym(e, K3, b, g);
        const double q[3] = {K3 * rho[0] - di * t[0], K3 * rho[1] - di * t[1], K3 * rho[2] - di * t[2]};
        te_sym(e, 2.0 * al - 1.0, w, q);
        // al s [K3 (1 - t t) - 3 K5 rho rho + 2 d(1/R^3) t rho + d(u/R^3) t t]
        const double as = al * s, d3 = iA3 - iB3, du3 = uA * iA3 - uB * iB3;
        const double m[3] = {2.0 * d3 * t[0] - 3.0 * K5 * rho[0], 2.0 * d3 * t[1] - 3.0 * K5 * rho[1],
                             2.0 * d3 * t[2] - 3.0 * K5 * rho[2]};
        te_sym(e, as, rho, m);
        te_sym(e, as * (du3 - K3), t, t);
        const double tr = as * K3;
        e[0] += tr;
        e[1] += tr;
        e[2] += tr;
      }
    }
  }
  if (DL)
#pragma unroll
    for (int c = 0; c < 3; c++) u[c] += om * T.b[c];
  if (SL) {
    const double* s = T.s;
    const double* n = T.n;
    const double sn = te_dot(s, n), dnu = -N;  // dnu = sum nu . grad E
    N -= h * om;
    // S s = (edge terms, added above) + n (-unn + sn (2 N + dnu))
    const double fn = al * (unn - sn * (2.0 * N + dnu));
#pragma unroll
    for (int c = 0; c < 3; c++) u[c] += i2mu * (2.0 * N * s[c] + fn * n[c]);
    if (str) {
      // the normal part of grad N, and the normal row and normal-normal term of S_ijk s_k
      const double nn = knn + sn * (kz - 2.0 * om), f = -i2mu * al;
      double y[3];
#pragma unroll
      for (int c = 0; c < 3; c++) y[c] = f * (Mn[c] + nn * n[c]) - 2.0 * i2mu * om * s[c];
      te_sym(e, 1.0, n, y);
    }
  }
}

// The quantities of edge k of T that both layers' unit responses use.
struct TeEdge {
  double t[3], nu[3], rho[3], v, h, RA, RB, uA, uB, iA, iB, L, K3, K5;
};
EFMM_HD void te_edge(const TriEdge& T, int k, const double r[3][3], const double R[3], const double iR[3], double h,
                     TeEdge& g) {
#pragma unroll
  for (int c = 0; c < 3; c++) g.t[c] = T.t[3 * k + c];
  g.RA = k == 0 ? R[0] : (k == 1 ? R[1] : R[2]);
  g.RB = k == 0 ? R[1] : (k == 1 ? R[2] : R[0]);
  g.iA = k == 0 ? iR[0] : (k == 1 ? iR[1] : iR[2]);
  g.iB = k == 0 ? iR[1] : (k == 1 ? iR[2] : iR[0]);
  const bool nb = g.RB < g.RA;
  double d[3];
  te_near_end(k, nb, r, d);
  const double ud = te_dot(d, g.t);
  g.uA = nb ? ud + T.len[k] : ud;
  g.uB = nb ? ud : ud - T.len[k];
  te_cross(g.t, T.n, g.nu);
  g.v = te_dot(d, g.nu);
  g.h = h;
#pragma unroll
  for (int c = 0; c < 3; c++) g.rho[c] = g.v * g.nu[c] + h * T.n[c];
  te_line(T.len[k], g.uA, g.uB, g.RA, g.RB, g.iA, g.iB, g.v * g.v + h * h, g.L, g.K3, g.K5);
}
// e += f sym(e_k, b)
EFMM_HD void te_sym_axis(double* e, int k, double f, const double* b) {
  const double h = 0.5 * f;
  if (k == 0) {
    e[0] += f * b[0]; e[3] += h * b[1]; e[4] += h * b[2];
  } else if (k == 1) {
    e[1] += f * b[1]; e[3] += h * b[0]; e[5] += h * b[2];
  } else {
    e[2] += f * b[2]; e[4] += h * b[0]; e[5] += h * b[1];
  }
}

// Unit responses of one (triangle, target) pair, the stored near-field
// operator of the ITER mode (src/elfmm3dtria_iter_1.f:1559-1760 stores the
// same three unit responses): LAYER 0 single, 1 double; out[KB k + (0..2 u,
// 3..8 strain)] for a unit density along each axis k, KB = 9 with strain, else
// 3.  The arithmetic of tri_edge_pair with the tensors that do not depend on
// the density formed once per edge.
template <int LAYER, bool STR>
EFMM_HD void tri_edge_blocks(const TriEdge& T, const double* X, bool self, double al, double i2mu, double* out) {
  constexpr int KB = STR ? 9 : 3;
  double r[3][3], R[3], iR[3];
  const double h = te_vertices(T, X, self, r, R, iR);
  double om = 0.0;
  if (h != 0.0) {
    const double den = R[0] * R[1] * R[2] + te_dot(r[0], r[1]) * R[2] + te_dot(r[0], r[2]) * R[1] +
                       te_dot(r[1], r[2]) * R[0];
    om = 2.0 * atan2(h * T.area2, den);
  }
  double o[27];
#pragma unroll
  for (int q = 0; q < 27; q++) o[q] = 0.0;
  double N = 0.0, kz = 0.0, unn[3] = {0, 0, 0}, knn[3] = {0, 0, 0};
#pragma unroll 1
  for (int k = 0; k < 3; k++) {
    TeEdge g;
    te_edge(T, k, r, R, iR, h, g);
    const double di = g.iA - g.iB;
    if (LAYER == 1) {
      const double* t = g.t;
      const double d3 = g.iA * g.iA * g.iA - g.iB * g.iB * g.iB;
      const double du3 = g.uA * g.iA * g.iA * g.iA - g.uB * g.iB * g.iB * g.iB;
      double c[3], q[3];
      te_cross(t, g.rho, c);
#pragma unroll
      for (int j = 0; j < 3; j++) q[j] = g.K3 * g.rho[j] - di * t[j];
      double A[6] = {0, 0, 0, 0, 0, 0}, gx[3];
      if (STR) {
        const double m[3] = {2.0 * d3 * t[0] - 3.0 * g.K5 * g.rho[0], 2.0 * d3 * t[1] - 3.0 * g.K5 * g.rho[1],
                             2.0 * d3 * t[2] - 3.0 * g.K5 * g.rho[2]};
        te_sym(A, al, g.rho, m);
        te_sym(A, al * (du3 - g.K3), t, t);
        A[0] += al * g.K3;
        A[1] += al * g.K3;
        A[2] += al * g.K3;
#pragma unroll
        for (int j = 0; j < 3; j++) gx[j] = g.K3 * (g.v * T.n[j] - h * g.nu[j]);
      }
      const double fw = (1.0 - al) * g.L;
#pragma unroll
      for (int j = 0; j < 3; j++) {
        double* u = o + 9 * j;
        double* e = u + 3;
        const int j1 = j == 2 ? 0 : j + 1, j2 = j == 0 ? 2 : j - 1;
        // w = e_j x t: component j1 -t[j2], component j2 t[j1]
        const double s = al * c[j];
        u[0] += s * q[0];
        u[1] += s * q[1];
        u[2] += s * q[2];
        u[j1] -= fw * t[j2];
        u[j2] += fw * t[j1];
        if (STR) {
#pragma unroll
          for (int z = 0; z < 6; z++) e[z] += c[j] * A[z];
          te_sym_axis(e, j1, -(2.0 * al - 1.0) * t[j2], q);
          te_sym_axis(e, j2, (2.0 * al - 1.0) * t[j1], q);
          te_sym_axis(e, j, 1.0, gx);
        }
      }
    } else {
      const double Et = T.len[k] * (g.uA + g.uB) / (g.RA + g.RB), hL = h * g.L;
      const double du = g.uA * g.iA - g.uB * g.iB, kn = g.L - h * h * g.K3;
      N -= g.v * g.L;
      double B[6] = {0, 0, 0, 0, 0, 0}, Tn[6] = {0, 0, 0, 0, 0, 0}, Rn[6] = {0, 0, 0, 0, 0, 0};
      if (STR) {
        kz -= g.v * h * g.K3;
        te_sym(B, i2mu * al, g.nu, T.n);   // in-plane rows' normal column
        te_sym(Tn, i2mu * al, g.nu, g.t);
        te_sym(Rn, i2mu * al, g.nu, g.rho);
      }
#pragma unroll
      for (int j = 0; j < 3; j++) {
        double* u = o + 9 * j;
        double* e = u + 3;
        const double st = g.t[j], sr = g.rho[j];
        const double f = i2mu * al * (st * Et + sr * g.L);
#pragma unroll
        for (int z = 0; z < 3; z++) u[z] += f * g.nu[z];
        unn[j] += g.nu[j] * hL;
        if (STR) {
          const double ct = st * (du - g.L) + sr * di, cr = st * di - g.K3 * sr;
          const double gn = cr * h + g.L * T.n[j];
#pragma unroll
          for (int z = 0; z < 6; z++) e[z] += ct * Tn[z] + cr * Rn[z] + gn * B[z];
          te_sym_axis(e, j, i2mu * (al - 2.0) * g.L, g.nu);
          knn[j] -= g.nu[j] * kn;
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 3; j++) {
    double* u = o + 9 * j;
    double* e = u + 3;
    if (LAYER == 1) {
      u[j] += om;
    } else {
      const double Nh = N - h * om, sn = T.n[j];
      const double fn = i2mu * al * (unn[j] - sn * (2.0 * Nh - N));
#pragma unroll
      for (int z = 0; z < 3; z++) u[z] += fn * T.n[z];
      u[j] += i2mu * 2.0 * Nh;
      if (STR) {
        te_sym(e, -i2mu * al * (knn[j] + sn * (kz - 2.0 * om)), T.n, T.n);
        te_sym_axis(e, j, -2.0 * i2mu * om, T.n);
      }
    }
#pragma unroll
    for (int z = 0; z < KB; z++) out[KB * j + z] = u[z];
  }
}

}  // namespace efmm
