// image_moments.cuh -- the image part of Mindlin's half-space kernels (unit
// forces and unit jumps, displacement and strain) integrated over a triangle
// through moments.
//
// With R = (x1 - y1, x2 - y2, -x3 - y3), r = |R|, h = -y3, alpha =
// (lam + mu) / (lam + 2 mu), tau = (1, 1, -1), sigma = (-1, -1, 1) and
// subscripts for derivatives by R, the image displacement i of a unit force k
// (the three pieces of gen_mindlin.py) is
//
//   G_ki = (2 d_ik V - (2 - alpha) W_ik) / 2 mu + (1 - alpha) / (alpha mu) sigma_k U_ik
//          + x3 / mu (tau_i alpha h V_ik + Q_ki),
//   V = 1 / r, W = r, U = R3 log(r + R3) - r,
//   Q_ki = -(2 - alpha) V_i for k = 3 > i, -(2 - alpha) V_k for i = 3 > k, else 0;
//
// its strain differentiates by x (d/dx_j = tau_j d_j, and x3 itself), the
// jump kernel by y (d/dy_l = -d_l, and h itself, contracted with the elastic
// moduli and the normal).  Everything is a sum of derivatives of V, h V, W
// and U, and those of V and W are monomials of R over odd powers of r: a node
// with weight w adds w R_i R_j .. / r^n to a few dozen moments, and one
// assembly per (target, triangle) pair turns the moments into the 27
// responses.  Traces give the lower moments (sum_k R_k R_k = r^2), h R.. with
// h = R3 + x3 most of the h-weighted ones.  U is harmonic with U_33 = V, so
// per order only its two in-plane angular components are new: with
// w = 1 / (r + R3) and z = R1 + i R2,
//   in-plane U_ab: A z^2, U_abc: -B z^3, U_abcd: C z^4; U_a3: (w / r) z,
//   U_ab3: -A' z^2, U_abc3: B' z^3,
//   A = w^2 / r, B = 2 w^3 / r^2 + w^2 / r^3, C = 6 w^4 / r^3 + 6 w^3 / r^4 + 3 w^2 / r^5,
//   A' = w^2 / r^2 + w / r^3, B' = 2 w^3 / r^3 + 3 w^2 / r^4 + 3 w / r^5.
//
// About 150 FP64 operations per node with one reciprocal square root and one
// division, where the straight-line blocks of mindlin_gen.cuh run thousands
// with some 250 divisions each.
#pragma once
#include "tri_index.cuh"

namespace efmm {

// position of the symmetric component (sorted indices) in a packed table
EFMM_HD constexpr int sx2(int i, int j) {
  const int a = i < j ? i : j, b = i < j ? j : i;
  return a == 0 ? b : (a == 1 ? 2 + b : 5);
}
// counts (n1, n2) of indices 1 and 2 order the packed tables of ranks 3 and 4:
// rank N, component with n0 zeros: the N - n0 others start at (N - n0)(N - n0 + 1) / 2
EFMM_HD constexpr int sx_cnt(int m, int n2) { return m * (m + 1) / 2 + n2; }
EFMM_HD constexpr int sx3(int i, int j, int k) {
  return sx_cnt((i != 0) + (j != 0) + (k != 0), (i == 2) + (j == 2) + (k == 2));
}
EFMM_HD constexpr int sx4(int i, int j, int k, int l) {
  return sx_cnt((i != 0) + (j != 0) + (k != 0) + (l != 0), (i == 2) + (j == 2) + (k == 2) + (l == 2));
}
EFMM_HD double dlt(int i, int j) { return i == j ? 1.0 : 0.0; }

struct ImageConst {
  double al, i2mu, imu, sc;  // alpha, 1 / 2 mu, 1 / mu, (1 - alpha) / (alpha mu)
  double lam, mu;
};
EFMM_HD void image_const(double lam, double mu, ImageConst& c) {
  c.al = (lam + mu) / (lam + 2.0 * mu);
  c.imu = 1.0 / mu;
  c.i2mu = 0.5 * c.imu;
  c.sc = (1.0 - c.al) / c.al * c.imu;
  c.lam = lam;
  c.mu = mu;
}

// Node geometry shared by the layers.
struct ImageNode {
  double R[3], h, ir, ir2, w;
};
EFMM_HD void image_node(const double X[3], const double y[3], ImageNode& g) {
  g.R[0] = X[0] - y[0];
  g.R[1] = X[1] - y[1];
  g.R[2] = -X[2] - y[2];
  g.h = -y[2];
  const double r2 = g.R[0] * g.R[0] + g.R[1] * g.R[1] + g.R[2] * g.R[2];
  const double r = sqrt(r2);
  // one division for both reciprocals
  const double s = r + g.R[2], q = 1.0 / (r * s);
  g.ir = q * s;
  g.ir2 = g.ir * g.ir;
  g.w = q * r;
}

// rank-3 monomials in the packed order, and z^2, z^3 from the in-plane ones
EFMM_HD void image_mono3(const double R[3], double p2[6], double p3[10]) {
  const double a = R[0], b = R[1], c = R[2];
  p2[0] = a * a; p2[1] = a * b; p2[2] = a * c; p2[3] = b * b; p2[4] = b * c; p2[5] = c * c;
  p3[0] = a * p2[0]; p3[1] = b * p2[0]; p3[2] = c * p2[0];
  p3[3] = a * p2[3]; p3[4] = a * p2[4]; p3[5] = a * p2[5];
  p3[6] = b * p2[3]; p3[7] = c * p2[3]; p3[8] = b * p2[5]; p3[9] = c * p2[5];
}

// ---------------------------------------------------------------- moments
// Double layer.  STR: with strain.
template <bool STR>
struct ImageDL {
  // with strain: t3 = RRR / r^5 (10), s3 = RRR / r^7 (10), t4 = RRRR / r^7
  // (15), h4 = h RRRR / r^9 (15); without: t3, s2 = RR / r^5 (6), h3 = h RRR / r^7 (10)
  double t3[10], s3[10], t4[STR ? 15 : 1], h4[STR ? 15 : 1], s2[STR ? 1 : 6];
  double u3[4], u4[4];  // U: (-B z^3), (-A' z^2); (C z^4), (B' z^3)
  EFMM_HD void clear() {
#pragma unroll
    for (int k = 0; k < 10; k++) t3[k] = s3[k] = 0.0;
#pragma unroll
    for (int k = 0; k < (STR ? 15 : 1); k++) t4[k] = h4[k] = 0.0;
#pragma unroll
    for (int k = 0; k < (STR ? 1 : 6); k++) s2[k] = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) u3[k] = u4[k] = 0.0;
  }
  EFMM_HD void add(const ImageNode& g, double wt) {
    double p2[6], p3[10];
    image_mono3(g.R, p2, p3);
    const double ir = g.ir, i2 = g.ir2, w = g.w, w2 = w * w;
    const double c3 = wt * ir * i2, c5 = c3 * i2, c7 = c5 * i2;
#pragma unroll
    for (int k = 0; k < 10; k++) t3[k] += c5 * p3[k];
    const double h7 = g.h * c7;
    const double s37 = STR ? c7 : h7;  // without strain s3 holds h RRR / r^7
#pragma unroll
    for (int k = 0; k < 10; k++) s3[k] += s37 * p3[k];
    const double z2r = p2[0] - p2[3], z2i = 2.0 * p2[1];
    const double z3r = p3[0] - 3.0 * p3[3], z3i = 3.0 * p3[1] - p3[6];
    const double w1 = wt * w * ir;  // wt w / r
    const double Ap = w1 * ir * (w + ir), B = w1 * w * ir * (2.0 * w + ir);
    u3[0] -= B * z3r; u3[1] -= B * z3i;
    u3[2] -= Ap * z2r; u3[3] -= Ap * z2i;
    if (STR) {
      const double h9 = h7 * i2;
      const double a = g.R[0], b = g.R[1], c = g.R[2];
      const double p4[15] = {a * p3[0], b * p3[0], c * p3[0], b * p3[1], b * p3[2], c * p3[2], a * p3[6], a * p3[7],
                             a * p3[8], a * p3[9], b * p3[6], b * p3[7], b * p3[8], b * p3[9], c * p3[9]};
#pragma unroll
      for (int k = 0; k < 15; k++) {
        t4[k] += c7 * p4[k];
        h4[k] += h9 * p4[k];
      }
      const double Bp = w1 * i2 * (2.0 * w2 + 3.0 * ir * (w + ir));
      const double C = w1 * w * i2 * (6.0 * w2 + 3.0 * ir * (2.0 * w + ir));
      u4[0] += C * (z2r * z2r - z2i * z2i); u4[1] += C * (2.0 * z2r * z2i);
      u4[2] += Bp * z3r; u4[3] += Bp * z3i;
    } else {
#pragma unroll
      for (int k = 0; k < 6; k++) s2[k] += c5 * p2[k];
    }
  }
};

// Single layer (with strain; the displacement alone uses a part of it):
// t2 = RR / r^3 (6), t3 = RRR / r^5 (10), s2 = RR / r^5 (6), h3 = h RRR / r^7 (10)
struct ImageSL {
  double t2[6], t3[10], s2[6], h3[10];
  double u2[4], u3[4];  // (A z^2), (w / r z); (-B z^3), (-A' z^2)
  EFMM_HD void clear() {
#pragma unroll
    for (int k = 0; k < 6; k++) t2[k] = s2[k] = 0.0;
#pragma unroll
    for (int k = 0; k < 10; k++) t3[k] = h3[k] = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) u2[k] = u3[k] = 0.0;
  }
  EFMM_HD void add(const ImageNode& g, double wt) {
    double p2[6], p3[10];
    image_mono3(g.R, p2, p3);
    const double ir = g.ir, i2 = g.ir2, w = g.w;
    const double c3 = wt * ir * i2, c5 = c3 * i2, h7 = g.h * c5 * i2;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      t2[k] += c3 * p2[k];
      s2[k] += c5 * p2[k];
    }
#pragma unroll
    for (int k = 0; k < 10; k++) {
      t3[k] += c5 * p3[k];
      h3[k] += h7 * p3[k];
    }
    const double z2r = p2[0] - p2[3], z2i = 2.0 * p2[1];
    const double z3r = p3[0] - 3.0 * p3[3], z3i = 3.0 * p3[1] - p3[6];
    const double w1 = wt * w * ir, A = w1 * w;
    const double Ap = w1 * ir * (w + ir), B = A * ir * (2.0 * w + ir);
    u2[0] += A * z2r; u2[1] += A * z2i;
    u2[2] += w1 * g.R[0]; u2[3] += w1 * g.R[1];
    u3[0] -= B * z3r; u3[1] -= B * z3i;
    u3[2] -= Ap * z2r; u3[3] -= Ap * z2i;
  }
};

// U derivative tables of rank 3 from the angular moments and V_c (V1)
EFMM_HD void image_u3(const double u3[4], const double V1[3], double U3[10]) {
  U3[sx3(0, 1, 1)] = -0.25 * (V1[0] + u3[0]);
  U3[sx3(0, 0, 0)] = -V1[0] - U3[sx3(0, 1, 1)];
  U3[sx3(0, 0, 1)] = 0.25 * (u3[1] - V1[1]);
  U3[sx3(1, 1, 1)] = -V1[1] - U3[sx3(0, 0, 1)];
  U3[sx3(0, 0, 2)] = 0.5 * (u3[2] - V1[2]);
  U3[sx3(1, 1, 2)] = -V1[2] - U3[sx3(0, 0, 2)];
  U3[sx3(0, 1, 2)] = 0.5 * u3[3];
  U3[sx3(0, 2, 2)] = V1[0];
  U3[sx3(1, 2, 2)] = V1[1];
  U3[sx3(2, 2, 2)] = V1[2];
}

// Responses to the three unit jumps (normal nrm): out[9 p + (0..2 u, 3..8
// strain xx yy zz xy xz yz)], ADDED; without strain only u.  x3: the target's.
template <bool STR>
EFMM_HD void image_dl_assemble(const ImageDL<STR>& m, const ImageConst& c, double x3, const double nrm[3],
                               double* out) {
  // V1, V2, W3, U3 and h V3 (hV3 = x3 V3 + R3 V3 with strain)
  double r3[3], V1[3], V2[6], s5[6], W3[10], U3[10], hV3[10];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    r3[i] = m.t3[sx3(i, 0, 0)] + m.t3[sx3(i, 1, 1)] + m.t3[sx3(i, 2, 2)];  // R_i / r^3
    V1[i] = -r3[i];
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = i; j < 3; j++)
      s5[sx2(i, j)] = STR ? m.t4[STR ? sx4(i, j, 0, 0) : 0] + m.t4[STR ? sx4(i, j, 1, 1) : 0] + m.t4[STR ? sx4(i, j, 2, 2) : 0]
                          : m.s2[STR ? 0 : sx2(i, j)];  // RR / r^5
  const double i3 = s5[0] + s5[3] + s5[5];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = i; j < 3; j++) V2[sx2(i, j)] = 3.0 * s5[sx2(i, j)] - dlt(i, j) * i3;
  double s7[3];  // with strain R_k / r^5, without h R_k / r^5
#pragma unroll
  for (int k = 0; k < 3; k++) s7[k] = m.s3[sx3(k, 0, 0)] + m.s3[sx3(k, 1, 1)] + m.s3[sx3(k, 2, 2)];
  double V3[10];  // with strain V3, without h V3
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = i; j < 3; j++)
#pragma unroll
      for (int k = j; k < 3; k++) {
        const int q = sx3(i, j, k);
        W3[q] = 3.0 * m.t3[q] - (dlt(i, j) * r3[k] + dlt(i, k) * r3[j] + dlt(j, k) * r3[i]);
        V3[q] = 3.0 * (dlt(i, j) * s7[k] + dlt(i, k) * s7[j] + dlt(j, k) * s7[i]) - 15.0 * m.s3[q];
        if (STR)
          hV3[q] = x3 * V3[q] + 3.0 * (dlt(i, j) * s5[sx2(k, 2)] + dlt(i, k) * s5[sx2(j, 2)] + dlt(j, k) * s5[sx2(i, 2)]) -
                   15.0 * m.t4[STR ? sx4(i, j, k, 2) : 0];
        else
          hV3[q] = V3[q];
      }
  image_u3(m.u3, V1, U3);
  const double al = c.al, b2 = 2.0 - al;
  const double tau[3] = {1.0, 1.0, -1.0}, sig[3] = {-1.0, -1.0, 1.0};
  // Q_ki,l
  auto Q2 = [&](int k, int i, int l) {
    return (k == 2 && i < 2) ? -b2 * V2[sx2(i, l)] : (i == 2 && k < 2) ? -b2 * V2[sx2(k, l)] : 0.0;
  };
  // P_ki,l + the h derivative: tau_i al (h V_ikl + d_l3 V_ik) + Q_ki,l
  auto P3 = [&](int k, int i, int l) {
    return tau[i] * al * (hV3[sx3(i, k, l)] + dlt(l, 2) * V2[sx2(i, k)]) + Q2(k, i, l);
  };
  // -d G_ki / d y_l
  auto A = [&](int k, int i, int l) {
    return c.i2mu * (2.0 * dlt(i, k) * V1[l] - b2 * W3[sx3(i, k, l)]) + c.sc * sig[k] * U3[sx3(i, k, l)] +
           x3 * c.imu * P3(k, i, l);
  };
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double tr = c.lam * (A(0, i, 0) + A(1, i, 1) + A(2, i, 2));
#pragma unroll
    for (int p = 0; p < 3; p++) {
      double s = 0.0;
#pragma unroll
      for (int l = 0; l < 3; l++) s += nrm[l] * (A(p, i, l) + A(l, i, p));
      out[9 * p + i] -= nrm[p] * tr + c.mu * s;
    }
  }
  if constexpr (STR) {
    double V4h[15], W4[15], U4[15];
    {
      double h7[6], h5;  // h RR / r^7, h / r^5
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++)
          h7[sx2(i, j)] = m.h4[STR ? sx4(i, j, 0, 0) : 0] + m.h4[STR ? sx4(i, j, 1, 1) : 0] + m.h4[STR ? sx4(i, j, 2, 2) : 0];
      h5 = h7[0] + h7[3] + h7[5];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++)
#pragma unroll
          for (int k = j; k < 3; k++)
#pragma unroll
            for (int l = k; l < 3; l++) {
              const int q = STR ? sx4(i, j, k, l) : 0;
              const double dd = dlt(i, j) * dlt(k, l) + dlt(i, k) * dlt(j, l) + dlt(i, l) * dlt(j, k);
              auto d2 = [&](const double* t) {
                return dlt(i, j) * t[sx2(k, l)] + dlt(i, k) * t[sx2(j, l)] + dlt(i, l) * t[sx2(j, k)] +
                       dlt(j, k) * t[sx2(i, l)] + dlt(j, l) * t[sx2(i, k)] + dlt(k, l) * t[sx2(i, j)];
              };
              W4[sx4(i, j, k, l)] = -dd * i3 + 3.0 * d2(s5) - 15.0 * m.t4[q];
              V4h[sx4(i, j, k, l)] = 3.0 * dd * h5 - 15.0 * d2(h7) + 105.0 * m.h4[q];
            }
      const double* u4 = m.u4;
      U4[sx4(0, 0, 1, 1)] = 0.125 * (V2[5] - u4[0]);
      U4[sx4(0, 0, 0, 0)] = -V2[0] - U4[sx4(0, 0, 1, 1)];
      U4[sx4(1, 1, 1, 1)] = -V2[3] - U4[sx4(0, 0, 1, 1)];
      U4[sx4(0, 0, 0, 1)] = 0.5 * (0.25 * u4[1] - V2[1]);
      U4[sx4(0, 1, 1, 1)] = -V2[1] - U4[sx4(0, 0, 0, 1)];
      U4[sx4(0, 1, 1, 2)] = -0.25 * (V2[2] + u4[2]);
      U4[sx4(0, 0, 0, 2)] = -V2[2] - U4[sx4(0, 1, 1, 2)];
      U4[sx4(0, 0, 1, 2)] = 0.25 * (u4[3] - V2[4]);
      U4[sx4(1, 1, 1, 2)] = -V2[4] - U4[sx4(0, 0, 1, 2)];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) U4[sx4(i, j, 2, 2)] = V2[sx2(i, j)];
    }
    auto Q3 = [&](int k, int i, int l, int j) {
      return (k == 2 && i < 2) ? -b2 * V3[sx3(i, l, j)] : (i == 2 && k < 2) ? -b2 * V3[sx3(k, l, j)] : 0.0;
    };
    // -d^2 G_ki / d y_l d x_j
    auto A4 = [&](int k, int i, int l, int j) {
      double s = c.i2mu * (2.0 * dlt(i, k) * V2[sx2(l, j)] - b2 * W4[sx4(i, k, l, j)]) +
                 c.sc * sig[k] * U4[sx4(i, k, l, j)] +
                 x3 * c.imu * (tau[i] * al * (V4h[sx4(i, k, l, j)] + dlt(l, 2) * V3[sx3(i, k, j)]) + Q3(k, i, l, j));
      s *= tau[j];
      if (j == 2) s += c.imu * P3(k, i, l);
      return s;
    };
    // displacement gradients of the three jumps, symmetrised
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const int q = i == j ? i : 2 + i + j;
        const double f = i == j ? 1.0 : 0.5;
        const double tr = c.lam * (A4(0, i, 0, j) + A4(1, i, 1, j) + A4(2, i, 2, j));
#pragma unroll
        for (int p = 0; p < 3; p++) {
          double s = 0.0;
#pragma unroll
          for (int l = 0; l < 3; l++) s += nrm[l] * (A4(p, i, l, j) + A4(l, i, p, j));
          out[9 * p + 3 + q] -= f * (nrm[p] * tr + c.mu * s);
        }
      }
  }
}

// Responses to the three unit forces, as image_dl_assemble.
EFMM_HD void image_sl_assemble(const ImageSL& m, const ImageConst& c, double x3, bool str, double* out) {
  double V1[3], V2[6], W2[6], W3[10], U2[6], U3[10], hV2[6], hV3[10];
  const double V0 = m.t2[0] + m.t2[3] + m.t2[5], i3 = m.s2[0] + m.s2[3] + m.s2[5];
#pragma unroll
  for (int i = 0; i < 3; i++) V1[i] = -(m.t3[sx3(i, 0, 0)] + m.t3[sx3(i, 1, 1)] + m.t3[sx3(i, 2, 2)]);
  const double h3 = x3 * i3 - V1[2];  // h / r^3, h = R3 + x3
  double h5[3];                       // h R_k / r^5
#pragma unroll
  for (int k = 0; k < 3; k++) h5[k] = m.h3[sx3(k, 0, 0)] + m.h3[sx3(k, 1, 1)] + m.h3[sx3(k, 2, 2)];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = i; j < 3; j++) {
      const int q = sx2(i, j);
      V2[q] = 3.0 * m.s2[q] - dlt(i, j) * i3;
      W2[q] = dlt(i, j) * V0 - m.t2[q];
      hV2[q] = 3.0 * (x3 * m.s2[q] + m.t3[sx3(i, j, 2)]) - dlt(i, j) * h3;
#pragma unroll
      for (int k = j; k < 3; k++) {
        const int t = sx3(i, j, k);
        W3[t] = 3.0 * m.t3[t] + (dlt(i, j) * V1[k] + dlt(i, k) * V1[j] + dlt(j, k) * V1[i]);
        hV3[t] = 3.0 * (dlt(i, j) * h5[k] + dlt(i, k) * h5[j] + dlt(j, k) * h5[i]) - 15.0 * m.h3[t];
      }
    }
  U2[sx2(0, 0)] = 0.5 * (m.u2[0] - V0);
  U2[sx2(1, 1)] = -V0 - U2[sx2(0, 0)];
  U2[sx2(0, 1)] = 0.5 * m.u2[1];
  U2[sx2(0, 2)] = m.u2[2];
  U2[sx2(1, 2)] = m.u2[3];
  U2[sx2(2, 2)] = V0;
  image_u3(m.u3, V1, U3);
  const double al = c.al, b2 = 2.0 - al;
  const double tau[3] = {1.0, 1.0, -1.0}, sig[3] = {-1.0, -1.0, 1.0};
  auto P = [&](int k, int i) {
    const double q = (k == 2 && i < 2) ? -b2 * V1[i] : (i == 2 && k < 2) ? -b2 * V1[k] : 0.0;
    return tau[i] * al * hV2[sx2(i, k)] + q;
  };
#pragma unroll
  for (int k = 0; k < 3; k++) {
#pragma unroll
    for (int i = 0; i < 3; i++)
      out[9 * k + i] += c.i2mu * (2.0 * dlt(i, k) * V0 - b2 * W2[sx2(i, k)]) + c.sc * sig[k] * U2[sx2(i, k)] +
                        x3 * c.imu * P(k, i);
    if (!str) continue;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const int q = i == j ? i : 2 + i + j;
        const double f = i == j ? 1.0 : 0.5;
        const double Q = (k == 2 && i < 2) ? -b2 * V2[sx2(i, j)] : (i == 2 && k < 2) ? -b2 * V2[sx2(k, j)] : 0.0;
        double s = c.i2mu * (2.0 * dlt(i, k) * V1[j] - b2 * W3[sx3(i, k, j)]) + c.sc * sig[k] * U3[sx3(i, k, j)] +
                   x3 * c.imu * (tau[i] * al * hV3[sx3(i, k, j)] + Q);
        s *= tau[j];
        if (j == 2) s += c.imu * P(k, i);
        out[9 * k + 3 + q] += f * s;
      }
  }
}

}  // namespace efmm
