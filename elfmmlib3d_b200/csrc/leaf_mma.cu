// leaf_mma.cu -- P2M and L2T of few right-hand sides as FP64 matrix products
// (mma.sync m8n8k4), for the free-space passes and the half-space image
// columns.
//
// P2M.  A leaf's multipole column is sum over quadrature nodes of charge,
// dipole and second-derivative terms of conj(Y_n^m).  A derivative of Y_n^m is
// a combination of Y_{n-1}^{m'} (harmonics.cuh), so the derivatives need not
// be formed per node: the product
//   S[(n, m, re/im)][weight] = sum_nodes Y_n^m(node) weight(node)
// over 16 columns (the charge and dipole weights of the four passes; or the 9
// weights of one image column) is accumulated in registers, and the shifts in
// (n, m) are applied once per leaf to S.
//
// L2T.  The value, gradient and Hessian sums of a local expansion at a point
// are inner products of Y(point) with shifted coefficients of the expansion
// (9 per column), so a chunk of points is the product
//   out[point][column, functional] = sum_(n, m, re/im) Y[point] B,
// B formed from the expansion in shared memory as it is consumed: with the m <
// 0 terms folded onto m >= 0 an element of B is one combination s L_{n+a}^{m+b}
// + t L_{n+a}^{m-b} of two stored parts.  The warps split the rows (n, m) and
// their sums are added at the end.
//
// Both hold the harmonics of 16 points as Y[row][16] in shared memory (rows: the
// re parts of all coefficients, padded to a multiple of 8, then the im parts),
// point p of row c at p ^ 4 (c & 3), which keeps the operand loads of the
// products and the stores of the recurrences free of bank conflicts.
// Half a warp (lane = point) runs the recurrence of one order m, its
// coefficients from a table (no division).
//
// P2M measured, one right-hand side at iprec 2, against per-coefficient
// threads that gathered the shifted harmonics of every node (k_p2m,
// k_p2m_img): 327,680 triangles 39.1 -> 8.7 ms (12 nodes x 768 rows x 16
// columns each: half of the FP64 pipe's time, the recurrences a third of it);
// half-space fault of 49,950 triangles, free-space 7.5 -> 1.5 and image columns
// 14.8 -> 4.7 ms; 1,702 triangles, image 7.4 -> 0.27 ms.  16 warps of 6 row
// tiles instead of 8 of 12 at order 26: 9.4 against 8.7 ms on the large case.
// L2T measured likewise, against a warp per point with lanes over the (n, m)
// terms (k_l2t, k_l2t_img): 577,687 points 25.9 -> 7.9 ms, the fault 9.0 -> 1.3
// ms (both plans), 81,920 + 62,501 points (mixed form) 6.4 -> 1.9 ms; the
// image columns of 2,003 points in 52 leaves 3.2 -> 0.09 ms (0.42 with one CTA
// per leaf); 18,034 triangles at order 39 (8 points per chunk), two
// right-hand sides, image columns 12.6 -> 2.3 ms.
#include <algorithm>

#include "common.cuh"
#include "fmm.h"
#include "kernels.h"
#include "leaf_ops.cuh"

namespace efmm {

namespace {
constexpr Quad12 lm_quad12() {
  Quad12 q{};
  quad12(q);
  return q;
}
__constant__ Quad12 c_quad = lm_quad12();
struct InvFactorials {
  double v[64];
};
constexpr InvFactorials make_ifac() {
  InvFactorials t{};
  t.v[0] = 1.0;
  for (int m = 1; m < 64; m++) t.v[m] = t.v[m - 1] / m;
  return t;
}
__constant__ InvFactorials c_ifac = make_ifac();

__device__ __forceinline__ void dmma(double* d, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Recurrence table: entry (n, m), n > m: ((2n - 1) / ((n - m)(n + m)), 1 /
// ((n - m)(n + m))); (m, m): (1 / m!, 0).  nm: n << 8 | m of every coefficient.
__device__ void harmonic_table(int p, double2* tab, unsigned short* nm) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int n = warp; n <= p; n += nw)
    for (int m = lane; m <= n; m += 32) {
      const int c = n * (n + 1) / 2 + m;
      if (nm) nm[c] = (unsigned short)(n << 8 | m);
      if (m < n) {
        const double inv = 1.0 / ((double)(n - m) * (double)(n + m));
        tab[c] = make_double2((2.0 * n - 1.0) * inv, inv);
      } else {
        tab[c] = make_double2(c_ifac.v[m], 0.0);
      }
    }
}

// Y_n^m(z) of this lane's point `pt` (0..NB-1) for the orders m = h, h + nh,
// .. (h of nh half-warps; every second round backwards, so that a half-warp's
// chains add up to about the same length).
template <int NB>
__device__ __forceinline__ void harmonics_to(double* __restrict__ Y, const double2* __restrict__ tab, int p,
                                             const double z[3], int pt, int h, int nh, int plane) {
  const double r2 = z[0] * z[0] + z[1] * z[1] + z[2] * z[2];
#pragma unroll 1
  for (int round = 0; round * nh <= p; round++) {
    const int m = round * nh + ((round & 1) ? nh - 1 - h : h);
    if (m > p) continue;
    cplx d = {1.0, 0.0}, b = {-0.5 * z[0], -0.5 * z[1]};
    for (int e = m; e; e >>= 1) {
      if (e & 1) d = cmul(d, b);
      b = cmul(b, b);
    }
    int c = m * (m + 1) / 2 + m;
    d = cscale(tab[c].x, d);
    auto put = [&](int cc, cplx v) {
      double* o = Y + cc * NB + ((pt ^ ((cc & 3) << 2)) & (NB - 1));
      o[0] = v.re;
      o[plane] = v.im;
    };
    put(c, d);
    const double zz = z[2];
    cplx y2 = {0.0, 0.0}, y1 = d;
    for (int n = m + 1; n <= p; n++) {
      c += n;
      const double2 t = tab[c];
      const double a = t.x * zz, q = t.y * r2;
      const cplx y = {a * y1.re - q * y2.re, a * y1.im - q * y2.im};
      put(c, y);
      y2 = y1;
      y1 = y;
    }
  }
}
__host__ __device__ constexpr int lm_plane_rows(int nc) { return (nc + 7) & ~7; }
}  // namespace

// ------------------------------------------------------------------------ P2M
// Columns of group g: free space 8 NT g + j -> pass, weight (charge, dipole);
// image, NT = 2: group 0 the four anti-image passes, groups 1..3 the 9 weights
// of columns 4..6; NT = 1: the 16 + 27 columns in groups of 8.
template <int NT, bool IMG>
__device__ __forceinline__ bool p2m_col(int g, int j, int& kind, int& f) {
  if (IMG && NT == 2 && g > 0) {
    kind = 3 + g;
    f = j;
    return j < 9;
  }
  const int c = 8 * NT * g + j;
  if (c < 16) {
    kind = c >> 2;
    f = c & 3;
    return true;
  }
  kind = 4 + (c - 16) / 9;
  f = (c - 16) % 9;
  return IMG && c < 43;
}
__host__ __device__ constexpr int p2m_groups(int nt, bool img) { return img ? (nt == 2 ? 4 : 6) : 2 / nt; }

// One CTA per (leaf, right-hand side and column group, part of the nodes).
// T = double: ADDED to the zeroed expansions; float: stored in the normalised
// basis (one part only).
template <int NW, int MTW, int NT, class T, bool IMG>
__global__ void __launch_bounds__(NW * 32, NW == 8 ? 2 : 1)
k_p2m_mma(const P2MArgs a, int R, long long ubase, T* __restrict__ mpole) {
  constexpr int NB = 16, NC = 8 * NT, WS = NC + 4, NG = p2m_groups(NT, IMG), NTH = NW * 32;
  extern __shared__ __align__(16) double lm_sm[];
  const int box = a.leaves[blockIdx.x], g = blockIdx.y % NG, r = blockIdx.y / NG;
  const int p = a.p, nc = ncoef(p), D = 2 * nc, ncp = lm_plane_rows(nc);
  double* Y = lm_sm;                      // [2 ncp][NB], later the sums [2 ncp][NC]
  double* W = Y + (size_t)2 * ncp * NB;   // [NB][WS]
  double2* tab = reinterpret_cast<double2*>(W + NB * WS);
  double* quad = reinterpret_cast<double*>(tab + nc);  // [12][4]: barycentric coordinates, weight
  const int lev = a.level[box];
  const double s = a.size / (double)(1ull << lev), is = 1.0 / s;
  double c[3];
  for (int d = 0; d < 3; d++) c[d] = a.c0[d] - a.size / 2 + (a.ijk[3 * box + d] - 1) * s + s / 2;
  double org[3];
  lame_origin(a.ijk, a.level, box, a.c0, a.size, a.flev, org);
  const int t0 = a.sstart[box], tn = a.scount[box], nnode = a.points ? tn : 12 * tn;
  const int nbat = (nnode + NB - 1) / NB;
  const int b0 = (int)((long long)nbat * blockIdx.z / gridDim.z), b1 = (int)((long long)nbat * (blockIdx.z + 1) / gridDim.z);
  if (b0 >= b1) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  harmonic_table(p, tab, nullptr);
  if (tid < 48) quad[tid] = (tid & 3) < 3 ? c_quad.b[tid >> 2][tid & 3] : c_quad.w[tid >> 2];
  for (int q = tid; q < NB * WS; q += NTH) W[q] = 0.0;  // columns without a weight stay zero
  // this thread's weight: node wpt of a batch, column wj
  const int wpt = tid & 15, wj = tid >> 4;
  int wkind = 0, wf = 0;
  const bool won = wj < NC && p2m_col<NT, IMG>(g, wj, wkind, wf);
  __syncthreads();
  // position, weight and triangle of a node
  auto node_at = [&](int node, double y[3], double& w) {
    if (a.points) {  // a particle: one node of weight 1
      const int it = t0 + node;
      for (int d = 0; d < 3; d++) y[d] = a.pts[3 * (size_t)it + d];
      w = 1.0;
      return it;
    }
    const int it = t0 + node / 12, iq = node % 12;
    const double* Tr = a.tri + 9 * (size_t)it;
    const double* qb = quad + 4 * iq;
    for (int d = 0; d < 3; d++) y[d] = qb[0] * Tr[d] + qb[1] * Tr[3 + d] + qb[2] * Tr[6 + d];
    const double e1[3] = {Tr[3] - Tr[0], Tr[4] - Tr[1], Tr[5] - Tr[2]};
    const double e2[3] = {Tr[6] - Tr[0], Tr[7] - Tr[1], Tr[8] - Tr[2]};
    const double cr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    w = qb[3] * 0.5 * sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
    return it;
  };
  double acc[MTW][NT][2];
#pragma unroll
  for (int i = 0; i < MTW; i++)
#pragma unroll
    for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int lk = lane & 3, ln = lane >> 2;
  for (int bt = b0; bt < b1; bt++) {
    __syncthreads();  // the table is there; the previous batch is consumed
    {
      const int pt = lane & 15, node = min(bt * NB + pt, nnode - 1);
      double y[3], w;
      node_at(node, y, w);
      const double z[3] = {(y[0] - c[0]) * is, (y[1] - c[1]) * is, (y[2] - c[2]) * is};
      harmonics_to<NB>(Y, tab, p, z, pt, 2 * warp + (lane >> 4), 2 * NW, ncp * NB);
    }
    if (won) {
      const int node = bt * NB + wpt;
      double v = 0.0;
      if (node < nnode) {
        double y[3], w;
        const int it = node_at(node, y, w);
        const long long off = r * a.rstride + it * a.tstride, ds = a.dstride;
        const double* nn = a.nrm + 3 * (size_t)it;
        const double yo[3] = {y[0] - org[0], y[1] - org[1], y[2] - org[2]};
        if (wkind < 3) {  // passes 0..2: charge s_k / 2 mu, dipole (n b_k + b n_k) / 2
          if (wf == 0) {
            if (a.dosl) v = a.ssl[off + wkind * ds] * a.inv2mu;
          } else if (a.dodl) {
            v = 0.5 * (nn[wf - 1] * a.sdl[off + wkind * ds] + a.sdl[off + (wf - 1) * ds] * nn[wkind]);
          }
        } else {
          double sl[3] = {0, 0, 0}, dl[3] = {0, 0, 0}, wv[9];
          if (a.dosl) { sl[0] = a.ssl[off]; sl[1] = a.ssl[off + ds]; sl[2] = a.ssl[off + 2 * ds]; }
          if (a.dodl) { dl[0] = a.sdl[off]; dl[1] = a.sdl[off + ds]; dl[2] = a.sdl[off + 2 * ds]; }
          const double nv[3] = {nn[0], nn[1], nn[2]};
          img_node_weights(IMG ? wkind : 3, sl, dl, nv, yo, a, wv);
#pragma unroll
          for (int k = 0; k < (IMG ? 9 : 4); k++) v = k == wf ? wv[k] : v;
        }
        v *= w;
      }
      W[wpt * WS + wj] = v;
    }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < NB / 4; ks++) {
      double b[NT];
#pragma unroll
      for (int j = 0; j < NT; j++) b[j] = W[(4 * ks + lk) * WS + 8 * j + ln];
#pragma unroll
      for (int i = 0; i < MTW; i++) {
        if (8 * (warp + NW * i) < 2 * ncp) {
          const double av = Y[(8 * (warp + NW * i) + ln) * NB + ((4 * ks + lk) ^ (4 * (ln & 3)))];
#pragma unroll
          for (int j = 0; j < NT; j++) dmma(acc[i][j], av, b[j]);
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < MTW; i++) {
    const int row = 8 * (warp + NW * i) + ln;
    if (row < 2 * ncp)
#pragma unroll
      for (int j = 0; j < NT; j++)
        *reinterpret_cast<double2*>(Y + (size_t)row * NC + 8 * j + 2 * lk) = make_double2(acc[i][j][0], acc[i][j][1]);
  }
  __syncthreads();
  // shifts of the derivative weights: sums S_f of Y (column j0 + f, f0 <= f <
  // f1 in this group) -> the conjugated features' contribution to (n, m)
  auto shifted = [&](int n, int m, int j0, int f0, int f1, double& re, double& im) {
    auto get = [&](int f, int nn, int mm) {
      const int am = mm < 0 ? -mm : mm;
      cplx v = {0.0, 0.0};
      if (nn < 0 || am > nn || f < f0 || f >= f1) return v;
      const int k = nn * (nn + 1) / 2 + am;
      v.re = Y[(size_t)k * NC + j0 + f];
      v.im = Y[(size_t)(ncp + k) * NC + j0 + f];
      if (mm < 0) {
        if (am & 1) v.re = -v.re;
        else v.im = -v.im;
      }
      return v;
    };
    const cplx v0 = get(0, n, m), v3 = get(3, n - 1, m);
    const cplx xb = get(1, n - 1, m + 1), xc = get(1, n - 1, m - 1);
    const cplx yb = get(2, n - 1, m + 1), yc = get(2, n - 1, m - 1);
    re = v0.re + is * (v3.re + 0.5 * (xb.re - xc.re + yb.im + yc.im));
    im = -v0.im + is * (-v3.im - 0.5 * (xb.im - xc.im - yb.re - yc.re));
    if (IMG && f1 > 4) {
      const double h = 0.25 * is * is;
      const cplx a0 = get(4, n - 2, m), ap = get(4, n - 2, m + 2), am = get(4, n - 2, m - 2);
      const cplx b0 = get(5, n - 2, m), bp = get(5, n - 2, m + 2), bm = get(5, n - 2, m - 2);
      const cplx cp = get(6, n - 2, m + 2), cm = get(6, n - 2, m - 2);
      const cplx dp = get(7, n - 2, m + 1), dm = get(7, n - 2, m - 1);
      const cplx ep = get(8, n - 2, m + 1), em = get(8, n - 2, m - 1);
      re += h * (ap.re - 2.0 * a0.re + am.re - bp.re - 2.0 * b0.re - bm.re + cp.im - cm.im +
                 2.0 * (dp.re - dm.re + ep.im + em.im));
      im += h * (-ap.im + 2.0 * a0.im - am.im + bp.im + 2.0 * b0.im + bm.im + cp.re - cm.re +
                 2.0 * (-dp.im + dm.im + ep.re + em.re));
    }
  };
  auto put = [&](int kind, int cc, double re, double im) {
    T* M = IMG ? (kind < 6 ? mpole + ((size_t)box * 6 * R + (size_t)kind * R + r) * D
                           : mpole + ubase + ((size_t)box * R + r) * D)
               : mpole + ((size_t)box * a.C + 4 * r + kind) * D;
    if constexpr (sizeof(T) == 8) {
      atomicAdd(M + 2 * cc, re);
      atomicAdd(M + 2 * cc + 1, im);
    } else {
      const double sr = a.wnorm ? a.wnorm[2 * cc] : 1.0;
      M[2 * cc] = (T)(sr * re);
      M[2 * cc + 1] = (T)(sr * im);
    }
  };
  for (int cc = tid; cc < nc; cc += NTH) {
    int n = (int)((sqrt(8.0 * cc + 1.0) - 1.0) * 0.5);
    while ((n + 1) * (n + 2) / 2 <= cc) n++;
    while (n * (n + 1) / 2 > cc) n--;
    const int m = cc - n * (n + 1) / 2;
    double re, im;
    // the group's columns kind by kind (a kind's weights may end in the next group)
    for (int j = 0; j < NC;) {
      int kind, f;
      if (!p2m_col<NT, IMG>(g, j, kind, f)) break;
      const int nf = kind < 4 ? 4 : 9, f1 = min(nf, f + NC - j);
      shifted(n, m, j - f, f, f1, re, im);
      put(kind, cc, re, im);
      j += f1 - f;
    }
  }
}

static size_t p2m_mma_smem(int p, int nt) {
  const size_t nc = ncoef(p);
  return 8 * (32 * (size_t)lm_plane_rows((int)nc) + 16 * (8 * nt + 4) + 2 * nc + 48);
}

template <class T, bool IMG>
bool launch_p2m_mma(cudaStream_t st, int nleaf, const P2MArgs& a, int R, long long ubase, T* mpole) {
  // 8 warps of 12 row tiles, two CTAs per SM, to order 26; 16 warps of 8 row
  // tiles to order 30; above, 16 warps of 14 row tiles and 8 columns at a
  // time (FP64 only: a column's weights fall in two groups, which add up) to
  // order 39, the last whose harmonics fit in shared memory
  const int p = a.p;
  if (p > 39 || (p > 30 && sizeof(T) == 4)) return false;
  if (nleaf <= 0 || R <= 0) return true;
  const int nt = p > 30 ? 1 : 2, ng = p2m_groups(nt, IMG);
  const size_t smem = p2m_mma_smem(p, nt);
  // parts of the nodes while leaves x groups leave the chip (two CTAs per SM,
  // four rounds) unfilled; each part pays the table and the final shifts
  int parts = 1;
  if (sizeof(T) == 8) parts = std::max(1, std::min(16, (4 * 296) / std::max(1, nleaf * ng * R)));
  const dim3 grid(nleaf, ng * R, parts);
  auto go = [&](auto kern, int threads) {
    EFMM_CUDA_TRY(smem_raise(kern, (int)smem));
    kern<<<grid, threads, smem, st>>>(a, R, ubase, mpole);
    count_launch();
  };
  if (p <= 26) go(k_p2m_mma<8, 12, 2, T, IMG>, 256);
  else if (p <= 30) go(k_p2m_mma<16, 8, 2, T, IMG>, 512);
  else if constexpr (sizeof(T) == 8) go(k_p2m_mma<16, 14, 1, T, IMG>, 512);
  EFMM_CUDA_TRY(cudaGetLastError());
  return true;
}
template bool launch_p2m_mma<double, false>(cudaStream_t, int, const P2MArgs&, int, long long, double*);
template bool launch_p2m_mma<double, true>(cudaStream_t, int, const P2MArgs&, int, long long, double*);
template bool launch_p2m_mma<float, true>(cudaStream_t, int, const P2MArgs&, int, long long, float*);

// ------------------------------------------------------------------------ L2T
// Functionals v of a column (value, d_z, d_zz, the real and imaginary parts of
// d_x + i d_y, of that of d_z, and of (d_x + i d_y)^2): shifts a in n and b in
// m, sign, imaginary part.
struct LmTerm {
  int a, b, sg, im;
};
__constant__ LmTerm c_lm_terms[9] = {{0, 0, 1, 0},  {1, 0, 1, 0},  {2, 0, 1, 0}, {1, 1, -1, 0}, {1, 1, -1, 1},
                                     {2, 1, -1, 0}, {2, 1, -1, 1}, {2, 2, 1, 0}, {2, 2, 1, 1}};

// The expansion rows extended for the shifts: degree N = 0..p + 2 (zero past
// p), orders -2..N, entry N (N + 5) / 2 + M + 2 of a column.
__host__ __device__ constexpr int lm_ext_size(int p) { return (p + 3) * (p + 8) / 2; }

// Doubles of the harmonics of a chunk, or of the 16 warps' sums and their
// total in their place.
__host__ __device__ inline int lm_l2t_y(int p, int nb, int ncol) {
  const int y = 2 * lm_plane_rows(ncoef(p)) * nb, w = 17 * nb * ncol;
  return y > w ? y : w;
}

// One CTA per (leaf, right-hand side, part of the leaf's points), points in
// chunks of NB, 16 warps splitting the product's rows; 9 outputs of a point by
// 9 threads.
template <int NB, bool IMG>
__global__ void __launch_bounds__(512, 1)
k_l2t_mma(const L2TArgs a, int R, long long ubase) {
  constexpr int NW = 16, NTH = NW * 32, NQ = IMG ? 7 : 4, NTL = (9 * NQ + 7) / 8, NC = 8 * NTL, MT = NB / 8;
  extern __shared__ __align__(16) double lm_sm[];
  const int box = a.leaves[blockIdx.x], r = blockIdx.y;
  const int sn = a.do_src ? a.scount[box] : 0, tn = a.do_tgt ? a.tcount[box] : 0, np = sn + tn;
  if ((int)blockIdx.z * NB >= np) return;
  const int p = a.p, nc = ncoef(p), D = 2 * nc, ncp = lm_plane_rows(nc), ext = lm_ext_size(p);
  double* Y = lm_sm;                                  // [2 ncp][NB], later the warps' sums [NW][NB][NC]
  double2* L = reinterpret_cast<double2*>(Y + lm_l2t_y(p, NB, NC));  // [NQ][ext]
  double* S = Y + (size_t)NW * NB * NC;                 // [NB][NC]
  double2* tab = L + NQ * ext;
  unsigned short* nm = reinterpret_cast<unsigned short*>(tab + nc);  // [ncp]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lev = a.level[box];
  const double s = a.size / (double)(1ull << lev), is = 1.0 / s, is2 = is * is;
  double c[3];
  for (int d = 0; d < 3; d++) c[d] = a.c0[d] - a.size / 2 + (a.ijk[3 * box + d] - 1) * s + s / 2;
  double org[3];
  lame_origin(a.ijk, a.level, box, a.c0, a.size, a.flev, org);
  harmonic_table(p, tab, nm);
  for (int q = nc + tid; q < ncp; q += NTH) nm[q] = 0xffff;  // padding rows
  // the extended expansion: thread (column, entry)
  for (int N = warp; N <= p + 2; N += NW)
    for (int i = lane; i < N + 3; i += 32) {
      const int M = i - 2, am = M < 0 ? -M : M;
      const bool in = N <= p && am <= N;
      const int k = 2 * (N * (N + 1) / 2 + am);
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        double2 v = make_double2(0.0, 0.0);
        if (in) {
          const double* src = IMG ? (q < 6 ? a.local + ((size_t)box * 6 * R + (size_t)q * R + r) * D
                                           : a.local + ubase + ((size_t)box * R + r) * D)
                                  : a.local + ((size_t)box * a.C + 4 * r + q) * D;
          v = *reinterpret_cast<const double2*>(src + k);
          if (M < 0) {
            if (am & 1) v.x = -v.x;
            else v.y = -v.y;
          }
        }
        L[q * ext + N * (N + 5) / 2 + i] = v;
      }
    }
  // this lane's columns: offset of the column in L, shifts, signs of the two
  // terms for even (re) and odd (im) rows are resolved per row below
  const int lk = lane & 3, ln = lane >> 2;
  int ta[NTL], tb[NTL], tim[NTL], tq[NTL];
  double tsg[NTL];
#pragma unroll
  for (int j = 0; j < NTL; j++) {
    const int col = 8 * j + ln, q = col / 9, v = col % 9;
    const LmTerm t = c_lm_terms[v];
    ta[j] = t.a;
    tb[j] = t.b;
    tim[j] = t.im;
    tq[j] = q < NQ ? q * ext : 0;
    tsg[j] = q < NQ ? (double)t.sg : 0.0;
  }
  const int s0 = a.sstart[box], t0 = a.tstart[box];
  const int nks = 2 * ncp / 4;
  for (int e0 = blockIdx.z * NB; e0 < np; e0 += gridDim.z * NB) {
    __syncthreads();  // tables and L are there; the last chunk's sums are read
    if (NB == 16 || (lane & 15) < NB) {
      const int pt = lane & (NB - 1), e = min(e0 + pt, np - 1);
      const double* X = e < sn ? a.src_pts + 3 * (size_t)(s0 + e) : a.tgt_pts + 3 * (size_t)(t0 + e - sn);
      const double z[3] = {(X[0] - c[0]) * is, (X[1] - c[1]) * is, (X[2] - c[2]) * is};
      harmonics_to<NB>(Y, tab, p, z, pt, 2 * warp + (lane >> 4), 2 * NW, ncp * NB);
    }
    __syncthreads();
    double acc[MT][NTL][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < NTL; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    // k steps of 4 rows of one part: the re rows first, then the im rows
#pragma unroll 1
    for (int ks = warp; ks < nks; ks += NW) {
      const int row = 4 * ks + lk, part = 4 * ks >= ncp, cc = row - (part ? ncp : 0);
      const int n = nm[cc] >> 8, m = nm[cc] & 255;
      const bool in = nm[cc] != 0xffff;
      // Y past the last coefficient is not there: its operand is zero too
      double av[MT];
#pragma unroll
      for (int i = 0; i < MT; i++)
        av[i] = in ? Y[row * NB + (((8 * i + ln) ^ ((cc & 3) << 2)) & (NB - 1))] : 0.0;
      const double f = m == 0 ? 0.5 : 1.0;
#pragma unroll
      for (int j = 0; j < NTL; j++) {
        double b = 0.0;
        if (in) {
          const int N = n + ta[j];
          const double2* l = L + tq[j] + N * (N + 5) / 2 + m + 2;
          const double2 x = l[tb[j]], z = l[-tb[j]];
          const bool im = (part ^ tim[j]) != 0;
          const double xv = im ? x.y : x.x, zv = im ? z.y : z.x;
          // im = 0: x -+ z (minus for b = 1); im = 1, re rows: x + z for b = 1, x - z for b = 2;
          // im = 1, im rows: -x - z for b = 1, -x + z for b = 2
          const bool neg = tim[j] ? ((tb[j] == 1) == (part != 0)) : tb[j] == 1;
          b = tsg[j] * f * ((tim[j] && part ? -xv : xv) + (neg ? -zv : zv));
        }
#pragma unroll
        for (int i = 0; i < MT; i++) dmma(acc[i][j], av[i], b);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < NTL; j++)
        *reinterpret_cast<double2*>(Y + ((size_t)warp * NB + 8 * i + ln) * NC + 8 * j + 2 * lk) =
            make_double2(acc[i][j][0], acc[i][j][1]);
    __syncthreads();
    for (int q = tid; q < NB * NC; q += NTH) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < NW; w++) v += Y[(size_t)w * NB * NC + q];
      S[q] = v;
    }
    __syncthreads();
    // recombination: thread (point, output)
    for (int q = tid; q < 9 * NB; q += NTH) {
      const int pt = q % NB, o = q / NB, e = e0 + pt;
      if (e >= np) continue;
      const bool is_src = e < sn;
      const int pidx = is_src ? s0 + e : t0 + (e - sn);
      if (o >= 3 && !(is_src ? a.dostrain_src : a.dostrain_tgt)) continue;
      const double* X = is_src ? a.src_pts + 3 * (size_t)pidx : a.tgt_pts + 3 * (size_t)pidx;
      const double x[3] = {X[0], X[1], X[2]};
      const double* Sp = S + (size_t)pt * NC;
      auto grad = [&](int k, int i) { return is * Sp[9 * k + (i == 2 ? 1 : 3 + i)]; };
      auto hess = [&](int k, int i, int j) {
        const double* v = Sp + 9 * k;
        const int ij = i + j;
        double h;
        if (i == j) h = i == 2 ? v[2] : 0.5 * ((i == 0 ? v[7] : -v[7]) - v[2]);
        else h = ij == 1 ? 0.5 * v[8] : (ij == 2 ? v[5] : v[6]);
        return is2 * h;
      };
      const double c1 = a.c1, al = a.alpha, imu = IMG ? 1.0 / a.mu : 0.0, sc = IMG ? (1.0 - al) / al : 0.0, x3 = -x[2];
      if (o < 3) {
        double u = (2.0 - c1) * Sp[9 * o] + grad(3, o);
        for (int j = 0; j < 3; j++) u -= c1 * (x[j] - org[j]) * grad(j, o);
        if (IMG) {
          const double Pv = o < 2 ? grad(4, o) : -grad(4, 2) - (2.0 - al) * Sp[9 * 5];
          u += sc * imu * grad(6, o) + x3 * imu * Pv;
        }
        ((is_src ? a.u_src : a.u_tgt) + 3 * ((is_src ? a.nsrc : a.ntgt) * (long long)r + pidx))[o] += u;
      } else {
        auto G = [&](int i, int b) {  // d u_i / d x_b (image: d u_i / d xb_b)
          double v = (2.0 - c1) * grad(i, b) - c1 * grad(b, i) + hess(3, i, b);
          for (int j = 0; j < 3; j++) v -= c1 * (x[j] - org[j]) * hess(j, i, b);
          if (IMG) {
            v += sc * imu * hess(6, i, b);
            const double dP = i < 2 ? hess(4, i, b) : -hess(4, 2, b) - (2.0 - al) * grad(5, b);
            const double Pv = i < 2 ? grad(4, i) : -grad(4, 2) - (2.0 - al) * Sp[9 * 5];
            v += imu * ((b == 2 ? -Pv : 0.0) + x3 * dP);
          }
          return v;
        };
        const int k = o - 3, i = k < 3 ? k : (k == 5 ? 1 : 0), j = k < 3 ? k : (k == 3 ? 1 : 2);
        double v;
        if (i == j) v = IMG && i == 2 ? -G(2, 2) : G(i, i);
        else v = 0.5 * ((IMG && j == 2 ? -G(i, j) : G(i, j)) + G(j, i));
        ((is_src ? a.e_src : a.e_tgt) + 6 * ((is_src ? a.nsrc : a.ntgt) * (long long)r + pidx))[k] += v;
      }
    }
  }
}

static size_t l2t_mma_smem(int p, int nb, bool img) {
  const int nq = img ? 7 : 4, ncol = 8 * ((9 * nq + 7) / 8), nc = ncoef(p);
  return 8 * ((size_t)lm_l2t_y(p, nb, ncol) + 2 * (size_t)nq * lm_ext_size(p) + 2 * (size_t)nc) +
         2 * (size_t)lm_plane_rows(nc) + 8;
}

bool launch_l2t_mma(cudaStream_t st, int nleaf, const L2TArgs& a, int R, long long ubase, bool image) {
  const int nb = l2t_mma_smem(a.p, 16, image) <= 227 * 1024 ? 16 : 8;
  const size_t smem = l2t_mma_smem(a.p, nb, image);
  if (smem > 227 * 1024) return false;
  if (nleaf <= 0 || R <= 0) return true;
  auto go = [&](auto kern) {
    EFMM_CUDA_TRY(smem_raise(kern, (int)smem));
    // parts while the leaves leave SMs without a CTA (the few, full leaves near
    // the surface that hold an image plan's points)
    const int parts = std::max(1, std::min(16, 2 * 148 / (nleaf * R)));
    kern<<<dim3(nleaf, R, parts), 512, smem, st>>>(a, R, ubase);
    count_launch();
  };
  if (image) {
    if (nb == 16) go(k_l2t_mma<16, true>);
    else go(k_l2t_mma<8, true>);
  } else {
    if (nb == 16) go(k_l2t_mma<16, false>);
    else go(k_l2t_mma<8, false>);
  }
  EFMM_CUDA_TRY(cudaGetLastError());
  return true;
}

}  // namespace efmm
