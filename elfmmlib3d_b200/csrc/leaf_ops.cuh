// leaf_ops.cuh -- what the P2M and L2T kernels of a leaf share: the origin of
// the Lame decomposition, the node weights of the expansion columns and the
// image recombination.
#pragma once
#include "common.cuh"
#include "fmm.h"

namespace efmm {

// Origin o of the Lame decomposition for the points of box: the linear
// pass carries the charge (y - o).sigma and the recombination reads
// u_a = (2 - c1) phi_a - c1 (x - o)_j d_a phi_j + d_a Phi_4, which gives the
// same field for every o shared by a source and a target.  In a forest of
// problems (flev >= 0) o is the centre (x, y) of the box's column of level
// flev, so that the FP32 forms see coordinates of the problem's own size
// rather than of its offset in the forest; else o = 0.  o_z is always 0
// (the half-space image formulas read the absolute depth).
__device__ __forceinline__ void lame_origin(const int* ijk, const int* level, int box, const double* c0, double size,
                                            int flev, double o[3]) {
  o[0] = o[1] = o[2] = 0.0;
  const int sh = level[box] - flev;
  if (flev < 0 || sh < 0) return;
  const double w = size / (double)(1 << flev);
  for (int d = 0; d < 2; d++) o[d] = c0[d] - 0.5 * size + (((ijk[3 * box + d] - 1) >> sh) + 0.5) * w;
}

// Node weights of the half-space image columns, 7R per box, column
// kind * R + r for right-hand side r: kinds 0..3 the anti-image passes (the
// free-space passes with the anti-image constants c1, c2 of P2MArgs), 4 and 5
// the two 1/r potentials Phi_a, Phi_c of the C piece, 6 the U potential W of
// the B piece.  Per node 9 weights: charge, dipole (3) and the five
// second-derivative weights (xx - zz, yy - zz, 2xy, 2xz, 2yz of the
// quadrupole tensor).  With f the single-layer density, T the double-layer
// tensor lam (b.n) I + mu (b n^T + n b^T), h = -y_3 the source depth and
// alpha = (lam + mu)/(lam + 2 mu) (sources in the gradient-of-source
// convention of the features):
//   Phi_a: q = -(2 - alpha) f_3, D = -h alpha f - (2 - 2 alpha) T e_3, Q = -h alpha T
//   Phi_c: D = -f, Q = -T
//   W:     D = (f_1, f_2, -f_3), Q = -(S T + T S)/2, S = diag(-1, -1, 1)
// (the B and C pieces of src/mindlinpieces.f:29-520 written as Laplace-type
// potentials; their double layers by differentiation at the source).
__device__ __forceinline__ void img_node_weights(int kind, const double sl[3], const double dl[3], const double nn[3],
                                 const double y[3], const P2MArgs& a, double wv[9]) {
  const double c1 = a.c1, c2 = a.c2, inv2mu = a.inv2mu, al = a.alpha, lam = a.lam, mu = a.mu;
  for (int k = 0; k < 9; k++) wv[k] = 0.0;
  double Qm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  const double dln = dl[0] * nn[0] + dl[1] * nn[1] + dl[2] * nn[2];
  double Tm[3][3];
  for (int k = 0; k < 3; k++)
    for (int l = 0; l < 3; l++) Tm[k][l] = (k == l ? lam * dln : 0.0) + mu * (dl[k] * nn[l] + dl[l] * nn[k]);
  const double h = -y[2];
  if (kind < 3) {
    wv[0] = sl[kind] * inv2mu;
    for (int d = 0; d < 3; d++) wv[1 + d] = 0.5 * (nn[d] * dl[kind] + dl[d] * nn[kind]);
  } else if (kind == 3) {
    const double sly = sl[0] * y[0] + sl[1] * y[1] + sl[2] * y[2];
    const double dly = dl[0] * y[0] + dl[1] * y[1] + dl[2] * y[2];
    const double ny = nn[0] * y[0] + nn[1] * y[1] + nn[2] * y[2];
    wv[0] = sly * c1 * inv2mu + dln * c2;
    for (int d = 0; d < 3; d++) wv[1 + d] = 0.5 * c1 * (nn[d] * dly + dl[d] * ny);
  } else if (kind == 4) {
    wv[0] = -(2.0 - al) * sl[2];
    for (int d = 0; d < 3; d++) wv[1 + d] = -h * al * sl[d] - (2.0 - 2.0 * al) * Tm[2][d];
    for (int k = 0; k < 3; k++)
      for (int l = 0; l < 3; l++) Qm[k][l] = -h * al * Tm[k][l];
  } else if (kind == 5) {
    for (int d = 0; d < 3; d++) wv[1 + d] = -sl[d];
    for (int k = 0; k < 3; k++)
      for (int l = 0; l < 3; l++) Qm[k][l] = -Tm[k][l];
  } else {
    wv[1] = sl[0];
    wv[2] = sl[1];
    wv[3] = -sl[2];
    Qm[0][0] = Tm[0][0]; Qm[1][1] = Tm[1][1]; Qm[2][2] = -Tm[2][2];
    Qm[0][1] = Qm[1][0] = Tm[0][1];
  }
  wv[4] = Qm[0][0] - Qm[2][2];
  wv[5] = Qm[1][1] - Qm[2][2];
  wv[6] = 2.0 * Qm[0][1];
  wv[7] = 2.0 * Qm[0][2];
  wv[8] = 2.0 * Qm[1][2];
}

// Image displacement and strain at the original target from the value,
// gradient and Hessian of the 7 columns at the reflected target x (columns:
// 0..3 anti-image passes, 4 Phi_a, 5 Phi_c, 6 W; org the origin of
// lame_origin); ADDED to U (3) and, if E is set, E (6).
__device__ __forceinline__ void img_recombine(const double x[3], const double org[3], const double pot[7],
                                              const double g[7][3], const double H[7][3][3], double c1, double al,
                                              double imu, double sc,
                                              double* U, double* E) {
  const double x3 = -x[2];
  const double Pv[3] = {g[4][0], g[4][1], -g[4][2] - (2.0 - al) * pot[5]};
  double u[3], Gm[3][3];
  for (int i = 0; i < 3; i++) {
    u[i] = (2.0 - c1) * pot[i] + g[3][i];
    for (int j = 0; j < 3; j++) u[i] -= c1 * (x[j] - org[j]) * g[j][i];
    u[i] += sc * imu * g[6][i] + x3 * imu * Pv[i];
  }
  U[0] += u[0];
  U[1] += u[1];
  U[2] += u[2];
  if (!E) return;
  for (int aa = 0; aa < 3; aa++)
    for (int bb = 0; bb < 3; bb++) {
      double v = (2.0 - c1) * g[aa][bb] - c1 * g[bb][aa] + H[3][aa][bb];
      for (int j = 0; j < 3; j++) v -= c1 * (x[j] - org[j]) * H[j][aa][bb];
      v += sc * imu * H[6][aa][bb];
      const double dP = aa < 2 ? H[4][aa][bb] : -H[4][2][bb] - (2.0 - al) * g[5][bb];
      v += imu * ((bb == 2 ? -Pv[aa] : 0.0) + x3 * dP);
      Gm[aa][bb] = v;  // d u_a / d xb_b
    }
  // d u_a / d x_b = s_b Gm[a][b], s = (1, 1, -1)
  E[0] += Gm[0][0];
  E[1] += Gm[1][1];
  E[2] -= Gm[2][2];
  E[3] += 0.5 * (Gm[0][1] + Gm[1][0]);
  E[4] += 0.5 * (-Gm[0][2] + Gm[2][0]);
  E[5] += 0.5 * (-Gm[1][2] + Gm[2][1]);
}

}  // namespace efmm
