// nearfield.cu -- analytic near-field kernels (FP64).
//
// The near field of the reference (src/elfmm3dtria.f:968 _evalloc and the
// ITER variant src/elfmm3dtria_iter_1.f:1240-1419) sums, for each evaluation
// point, the exact single/double layer potential of every triangle in the
// source boxes paired with the point's leaf box.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace efmm {

constexpr int NL_MINB = 3;  // resident CTAs per SM the edge-integral kernels' register budget targets

// Edge records of the triangles (tri_edges.cuh) with the densities of
// right-hand side r0 of R (innermost).
__global__ void k_tri_edge_prep(int n, const double* __restrict__ tri, const double* __restrict__ ssl,
                                const double* __restrict__ sdl, int dosl, int dodl, int R, int r0,
                                TriEdge* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double t[9];
#pragma unroll
  for (int c = 0; c < 9; c++) t[c] = tri[9 * (size_t)i + c];
  TriEdge r;
  tri_edge_frame(t, r);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    r.s[c] = dosl ? ssl[(3 * (size_t)i + c) * R + r0] : 0.0;
    r.b[c] = dodl ? sdl[(3 * (size_t)i + c) * R + r0] : 0.0;
  }
  out[i] = r;
}

// Near field of one right-hand side.  Evaluation points of a leaf: its
// sources (sorted centroids, self-aware) then its targets; a work item is a
// few hundred to a few thousand pairs of one leaf (NearTask, the largest
// first), its triangles stream through shared memory in tiles.  The tile's
// triangles are dealt to S = NL_THREADS / points slices of threads: thread
// (point, slice), so 25 points fill 125 of 128 threads, every lane of a slice
// reads the same record (broadcast), and the slices are added once per item.
// Bound by the FP64 pipe: about 760 operations per pair and layer (log1p,
// atan2 and six divisions among them).  One CTA per leaf with one point per
// warp and lanes over the triangles of one box at a time, on derivative
// tables (228 registers, half of the lanes idle), took 104 ms on 327,680
// triangles + 250,007 targets at iprec 2 (165 M pairs) and 2.66 ms on 317 + 41
// (about 20 leaves); this form 19.1 ms and 0.058 ms.  Items instead of
// whole leaves matter where a few leaves hold most pairs (a coarse target
// leaf beside hundreds of fine source boxes): whole leaves took 12.5 ms
// against 6.0 on 81,920 triangles + 62,501 shell targets (55 M pairs).
// Registers for 3 CTAs per SM: 2, 3, 4 and 5 measured 23.6, 18.3, 18.6 and 19.8
// ms on the large case, 1.23, 1.15, 1.31 and 1.54 ms on 5,120 + 1,000 (before
// items, and before points at vertices, on edges and near corners were told
// apart).
// Outputs are ADDED to u (3/pt) and e (6/pt, xx yy zz xy xz yz).
constexpr int NL_THREADS = NEAR_TASK_PTS, NL_TILE = 32, NL_STRIDE = 34;  // record stride (doubles) free of bank conflicts

template <bool SL, bool DL>
__global__ void __launch_bounds__(NL_THREADS, NL_MINB)
k_near_leaf(const NearArgs a, const NearTask* __restrict__ tasks) {
  __shared__ __align__(16) double tile[NL_TILE * NL_STRIDE];
  __shared__ int tidx[NL_TILE];
  const NearTask w = tasks[blockIdx.x];
  const int leaf = a.leaves[w.li], tid = threadIdx.x;
  const int s0 = a.box_src_start[leaf], sn = a.do_src ? a.box_src_count[leaf] : 0, t0 = a.box_tgt_start[leaf];
  const double al = (a.rlam + a.rmu) / (a.rlam + 2.0 * a.rmu), i2mu = 0.5 / a.rmu;
  const int S = NL_THREADS / w.ne, sl = tid / w.ne, e = w.e0 + tid % w.ne;
  const bool on = sl < S;
  const bool is_src = e < sn;
  const int pidx = is_src ? s0 + e : t0 + (e - sn);
  const bool str = is_src ? a.dostrain_src : a.dostrain_tgt;
  double X[3] = {0, 0, 0};
  if (on) {
    const double* P = (is_src ? a.src_pts : a.tgt_pts) + 3 * (size_t)pidx;
    X[0] = P[0]; X[1] = P[1]; X[2] = P[2];
  }
  double u[3] = {0, 0, 0}, ee[6] = {0, 0, 0, 0, 0, 0};
  int left = w.cnt, b = w.r0, k = w.k0;  // range and triangle of the range to stage next
  while (left > 0) {
    __syncthreads();
    int fill = 0;
    while (left > 0 && fill < NL_TILE) {  // tiles fill across ranges
      const int2 rg = a.rng[b];
      const int m = min(min(NL_TILE - fill, rg.y - k), left);
      const int tr0 = rg.x + k;
      const double2* src = reinterpret_cast<const double2*>(a.rec + tr0);
      for (int q = tid; q < 16 * m; q += NL_THREADS)
        reinterpret_cast<double2*>(tile + (fill + q / 16) * NL_STRIDE)[q % 16] = src[q];
      if (tid < m) tidx[fill + tid] = tr0 + tid;
      fill += m;
      left -= m;
      k += m;
      if (k >= rg.y) {
        b++;
        k = 0;
      }
    }
    __syncthreads();
    if (on)
      for (int t = sl; t < fill; t += S) {
        const TriEdge& T = *reinterpret_cast<const TriEdge*>(tile + t * NL_STRIDE);
        tri_edge_pair<SL, DL>(T, X, is_src && tidx[t] == pidx, str, al, i2mu, u, ee);
      }
  }
  // add the slices
  static_assert(NL_TILE * NL_STRIDE >= 8 * NL_THREADS, "reduction space");
  __syncthreads();
  double out[9] = {u[0], u[1], u[2], ee[0], ee[1], ee[2], ee[3], ee[4], ee[5]};
  if (S > 1)
    for (int c0 = 0; c0 < 9; c0 += 8) {  // 8 values at a time through the tile
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (on && c0 + c < 9) tile[c * NL_THREADS + tid] = c0 == 0 ? out[c] : out[8];
      __syncthreads();
      if (on && sl == 0)
#pragma unroll
        for (int c = 0; c < 8; c++)
          if (c0 + c < 9) {
            double v = 0.0;
            for (int q = 0; q < S; q++) v += tile[c * NL_THREADS + q * w.ne + tid];
            if (c0 == 0) out[c] = v;
            else out[8] = v;
          }
      __syncthreads();
    }
  if (on && sl == 0) {
    double* U = (is_src ? a.u_src : a.u_tgt) + 3 * (size_t)pidx;
    double* E = (is_src ? a.e_src : a.e_tgt) + 6 * (size_t)pidx;
    if (w.shared) {
#pragma unroll
      for (int c = 0; c < 3; c++) atomicAdd(U + c, out[c]);
      if (str)
#pragma unroll
        for (int c = 0; c < 6; c++) atomicAdd(E + c, out[3 + c]);
    } else {
#pragma unroll
      for (int c = 0; c < 3; c++) U[c] += out[c];
      if (str)
#pragma unroll
        for (int c = 0; c < 6; c++) E[c] += out[3 + c];
    }
  }
}

// All-pairs direct sum (el3dtriadirecttarg, src/elfmm3dtria.f:1483): a CTA
// holds ND_PTS points, its 16 slices of threads and the CTAs of a cluster share
// the triangles, streamed through shared memory.  The parts are added in a
// fixed order through the cluster's shared memory, so that a call repeats bit
// for bit.  Points [0, nsrc) are the centroids (self pair when the indices
// match), [nsrc, nsrc + ntgt) the targets.  Points per CTA 4 / 8 / 16 / 32 /
// 128: 3.33 / 3.17 / 3.22 / 3.63 / 3.73 ms on 5,120 triangles + 1,000 targets,
// 75 / 73 / 75 / 75 / 82 on 20,480 + 20,000, .104 / .096 / .119 / .122 / .270 on
// 317 + 41 (parts of the triangles added atomically, 128 points: 3.40, 74.7,
// .152).
constexpr int ND_PTS = 8;
template <bool SL, bool DL>
__global__ void __launch_bounds__(NL_THREADS, NL_MINB)
k_direct_all(int ntri, const TriEdge* __restrict__ rec, int nsrc, const double* __restrict__ src_pts, int ntgt,
             const double* __restrict__ tgt_pts, int dostrain_src, int dostrain_tgt, double rlam, double rmu,
             double* __restrict__ u_src, double* __restrict__ e_src, double* __restrict__ u_tgt,
             double* __restrict__ e_tgt) {
  constexpr int P = ND_PTS, S = NL_THREADS / P;
  constexpr int NT = NL_TILE * NL_STRIDE > 9 * NL_THREADS ? NL_TILE * NL_STRIDE : 9 * NL_THREADS;
  __shared__ __align__(16) double tile[NT];  // the triangles, then the threads' sums
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, sl = tid / P, ep = blockIdx.x * P + tid % P;
  const bool on = ep < nsrc + ntgt, is_src = ep < nsrc;
  const int pidx = is_src ? ep : ep - nsrc;
  const bool str = is_src ? dostrain_src : dostrain_tgt;
  const double al = (rlam + rmu) / (rlam + 2.0 * rmu), i2mu = 0.5 / rmu;
  double X[3] = {0, 0, 0};
  if (on) {
    const double* Q = (is_src ? src_pts : tgt_pts) + 3 * (size_t)pidx;
    X[0] = Q[0]; X[1] = Q[1]; X[2] = Q[2];
  }
  const int lo = (int)((long long)ntri * blockIdx.y / gridDim.y);
  const int hi = (int)((long long)ntri * (blockIdx.y + 1) / gridDim.y);
  double u[3] = {0, 0, 0}, ee[6] = {0, 0, 0, 0, 0, 0};
  for (int k0 = lo; k0 < hi; k0 += NL_TILE) {
    const int m = min(NL_TILE, hi - k0);
    __syncthreads();
    const double2* src = reinterpret_cast<const double2*>(rec + k0);
    for (int q = tid; q < 16 * m; q += NL_THREADS)
      reinterpret_cast<double2*>(tile + (q / 16) * NL_STRIDE)[q % 16] = src[q];
    __syncthreads();
    if (on)
      for (int t = sl; t < m; t += S) {
        const TriEdge& T = *reinterpret_cast<const TriEdge*>(tile + t * NL_STRIDE);
        tri_edge_pair<SL, DL>(T, X, is_src && k0 + t == pidx, str, al, i2mu, u, ee);
      }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 3; c++) tile[c * NL_THREADS + tid] = u[c];
#pragma unroll
  for (int c = 0; c < 6; c++) tile[(3 + c) * NL_THREADS + tid] = ee[c];
  cl.sync();
  // (gridDim.y CTAs are the cluster; its first one adds)
  if (blockIdx.y == 0)
    for (int q = tid; q < 9 * P; q += NL_THREADS) {
      const int c = q / P, e = blockIdx.x * P + q % P;
      if (e >= nsrc + ntgt) continue;
      const bool src = e < nsrc;
      if (c >= 3 && !(src ? dostrain_src : dostrain_tgt)) continue;
      double v = 0.0;
      for (int y = 0; y < (int)gridDim.y; y++) {
        const double* part = cl.map_shared_rank(tile, y) + c * NL_THREADS + q % P;
        for (int w = 0; w < S; w++) v += part[w * P];
      }
      const size_t i = src ? e : e - nsrc;
      if (c < 3) (src ? u_src : u_tgt)[3 * i + c] = v;
      else (src ? e_src : e_tgt)[6 * i + c - 3] = v;
    }
  cl.sync();  // the parts stay until they are read
}

// ITER mode, first call: compute and store the unit-density response blocks
// of every near (point, triangle) pair of each leaf.  Layout per leaf:
// [evaluation point][near triangle][K doubles], at base[leaf]; near triangles
// are the concatenated source ranges of the leaf's paired boxes.  Tiles of 64
// triangles of one box, a warp per evaluation point (dealt over gridDim.y
// CTAs), lanes over the tile.
constexpr int NF_TILE = 64, NF_WARPS = 4;

__device__ __forceinline__ void near_pair_blocks(const TriEdge& T, const double* X, bool self, int dosl, int dodl,
                                                 int str, double al, double i2mu, double* out) {
  if (str) {
    if (dosl) {
      tri_edge_blocks<0, true>(T, X, self, al, i2mu, out);
      out += 27;
    }
    if (dodl) tri_edge_blocks<1, true>(T, X, self, al, i2mu, out);
  } else {
    if (dosl) {
      tri_edge_blocks<0, false>(T, X, self, al, i2mu, out);
      out += 9;
    }
    if (dodl) tri_edge_blocks<1, false>(T, X, self, al, i2mu, out);
  }
}

__global__ void __launch_bounds__(NF_WARPS * 32, NL_MINB)
k_near_store(const NearArgs a, const long long* __restrict__ base, const int* __restrict__ ntri,
             int K, double* __restrict__ store) {
  __shared__ __align__(16) double tile[NF_TILE * NL_STRIDE];
  const int leaf = a.leaves[blockIdx.x];
  const int s0 = a.box_src_start[leaf], sn = a.do_src ? a.box_src_count[leaf] : 0;
  const int t0 = a.box_tgt_start[leaf], tn = a.do_tgt ? a.box_tgt_count[leaf] : 0;
  const int nep = sn + tn;
  const int nt = ntri[blockIdx.x];
  const double al = (a.rlam + a.rmu) / (a.rlam + 2.0 * a.rmu), i2mu = 0.5 / a.rmu;
  double* out = store + base[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int pos = 0;  // running index of the leaf's near triangles
  for (int b = a.nb_start[blockIdx.x]; b < a.nb_start[blockIdx.x + 1]; b++) {
    const int sb = a.nb_items[b];
    const int tr0 = a.box_src_start[sb], trn = a.box_src_count[sb];
    for (int k0 = 0; k0 < trn; k0 += NF_TILE) {
      const int cnt = min(NF_TILE, trn - k0);
      __syncthreads();
      const double2* src = reinterpret_cast<const double2*>(a.rec + tr0 + k0);
      for (int q = threadIdx.x; q < 16 * cnt; q += NF_WARPS * 32)
        reinterpret_cast<double2*>(tile + (q / 16) * NL_STRIDE)[q % 16] = src[q];
      __syncthreads();
      for (int e = warp + NF_WARPS * blockIdx.y; e < nep; e += NF_WARPS * gridDim.y) {
        const bool is_src = e < sn;
        const int pidx = is_src ? s0 + e : t0 + (e - sn);
        const double* P = is_src ? a.src_pts + 3 * (size_t)pidx : a.tgt_pts + 3 * (size_t)pidx;
        const double X[3] = {P[0], P[1], P[2]};
        const int str = is_src ? a.dostrain_src : a.dostrain_tgt;
        for (int k = lane; k < cnt; k += 32) {
          const TriEdge& T = *reinterpret_cast<const TriEdge*>(tile + k * NL_STRIDE);
          near_pair_blocks(T, X, is_src && tr0 + k0 + k == pidx, a.dosl, a.dodl, str, al, i2mu,
                           out + ((size_t)e * nt + (pos + k0 + k)) * K);
        }
      }
    }
    pos += trn;
  }
}

// Replay of the stored blocks for R <= RR right-hand sides (densities tree
// order, right-hand side innermost, g0 the first layer stored, g1 the double
// layer when both are), ADDED to the outputs.  A warp streams the stored row
// of one evaluation point: element j of a row is output j % KB of unit
// density j / KB (KB = 3, or 9 with strain), so lane l reads elements l, l +
// 32, .. coalesced, its element i of every group of KB always adds to output
// (l + 32 i) % KB (one accumulator per i, sorted out once per row), and the
// densities are read from shared memory as one flat array at j / KB.  Bound
// by HBM: 8 bytes per RR multiply-adds.  Half-space fault of 49,950 triangles
// at iprec 2, one right-hand side: both replays 3.7 ms (22.3 GB free-space
// store: 6 TB/s, 0.92 of the measured copy rate); with lanes over triangles
// (27 loads 216 bytes apart each) and one CTA per leaf the free-space one took
// 13.3 ms, and the image one, whose few points near the surface have long
// lists, 19.2 ms with one CTA per 8 points (whole lists in this kernel: 0.9).
constexpr int RS_TILE = 1024;  // near triangles whose densities are staged at a time
template <int RR, int KB, int NLAY>
__global__ void __launch_bounds__(256)
k_near_replay(const NearArgs a, const NearTask* __restrict__ tasks, int R,
              const double* __restrict__ g0, const double* __restrict__ g1, int nsrc, int ntgt,
              const long long* __restrict__ base, const int* __restrict__ ntri, const double* __restrict__ store) {
  constexpr int NJ = 3 * NLAY, K = NJ * KB, G = 32 * KB;
  extern __shared__ __align__(16) double rs_sm[];  // [RS_TILE NJ][RR]
  const NearTask w = tasks[blockIdx.x];
  const int leaf = a.leaves[w.li];
  const int s0 = a.box_src_start[leaf], sn = a.do_src ? a.box_src_count[leaf] : 0, t0 = a.box_tgt_start[leaf];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e = w.e0 + warp;
  const bool on = warp < w.ne;
  const double* row = store + base[w.li] + ((size_t)e * ntri[w.li] + w.p0) * K;
  double acc[KB][RR];
  int si[KB];
#pragma unroll
  for (int i = 0; i < KB; i++) {
    si[i] = (lane + 32 * i) / KB;
#pragma unroll
    for (int r = 0; r < RR; r++) acc[i][r] = 0.0;
  }
  int b = w.r0, k = w.k0;  // range and triangle of the range to stage next
  for (int p0 = 0; p0 < w.cnt; p0 += RS_TILE) {
    const int cnt = min(RS_TILE, w.cnt - p0);
    __syncthreads();
    for (int fill = 0; fill < cnt;) {
      const int2 rg = a.rng[b];
      const int m = min(cnt - fill, rg.y - k);
      for (int q = threadIdx.x; q < m * NJ * RR; q += 256) {
        const int t = q / (NJ * RR), jj = (q / RR) % NJ, r = q % RR;
        const double* g = (NLAY == 2 && jj >= 3) ? g1 : g0;
        rs_sm[(size_t)fill * NJ * RR + q] = r < R ? g[((size_t)(rg.x + k + t) * 3 + jj % 3) * R + r] : 0.0;
      }
      fill += m;
      k += m;
      if (k >= rg.y) {
        b++;
        k = 0;
      }
    }
    __syncthreads();
    if (!on) continue;
    const double* B = row + (size_t)p0 * K + lane;
    const int len = cnt * K;
    int j = 0;
    const double* sv = rs_sm;
    for (; j + G <= len; j += G, B += G, sv += 32 * RR) {
      double v[KB];
#pragma unroll
      for (int i = 0; i < KB; i++) v[i] = __ldcs(B + 32 * i);
#pragma unroll
      for (int i = 0; i < KB; i++)
#pragma unroll
        for (int r = 0; r < RR; r++) acc[i][r] += v[i] * sv[si[i] * RR + r];
    }
#pragma unroll
    for (int i = 0; i < KB; i++)
      if (j + 32 * i + lane < len) {
        const double v = __ldcs(B + 32 * i);
#pragma unroll
        for (int r = 0; r < RR; r++) acc[i][r] += v * sv[si[i] * RR + r];
      }
  }
  if (!on) return;
  const bool src = e < sn;
  const int pid = src ? s0 + e : t0 + (e - sn);
  const size_t np = src ? (size_t)nsrc : (size_t)ntgt;
  const bool str = KB == 9 && (src ? a.dostrain_src : a.dostrain_tgt);
#pragma unroll
  for (int r = 0; r < RR; r++) {
    double mine = 0.0;  // output `lane` of this right-hand side
    for (int c = 0; c < KB; c++) {
      double v = 0.0;
#pragma unroll
      for (int i = 0; i < KB; i++) v += (lane + 32 * i) % KB == c ? acc[i][r] : 0.0;
      v = warp_sum(v);
      if (lane == c) mine = v;
    }
    if (r < R) {
      double* o = nullptr;
      if (lane < 3) o = (src ? a.u_src : a.u_tgt) + 3 * (np * r + pid) + lane;
      else if (lane < 9 && str) o = (src ? a.e_src : a.e_tgt) + 6 * (np * r + pid) + lane - 3;
      if (o && w.shared) atomicAdd(o, mine);
      else if (o) *o += mine;
    }
  }
}

// Many right-hand sides at once (densities tree order, right-hand side
// innermost: sigma[(tri * 3 + component) * R + r]).  The pair response to unit densities
// (tri_edge_blocks, as stored by the ITER mode) does not depend on the densities,
// so it is computed once per (point, triangle) pair and contracted with all
// R right-hand sides: per tile of NB_PTS points x NB_TRI triangles, phase 1
// writes the pair blocks to shared memory (one pair per thread), phase 2 is a
// small dense product  out[point][9][R] += block[point][tri][9 x 6] *
// sigma[tri][6][R]  with the outputs held in registers (9 x RB per thread;
// R <= 16 RB).  One CTA per (near leaf, chunk of NB_PTS evaluation points).
constexpr int NB_PTS = NEAR_BATCH_PTS, NB_TRI = 16, NB_THREADS = NB_PTS * NB_TRI;

template <int RB>
__global__ void __launch_bounds__(NB_THREADS)
k_near_batch(const NearArgs a, const NearTask* __restrict__ tasks, int R, int K, int dostrain,
             const double* __restrict__ ssl, const double* __restrict__ sdl, int nsrc, int ntgt) {
  constexpr int RW = 16 * RB;  // right-hand sides held per tile
  __shared__ __align__(16) double tile[NB_TRI * NL_STRIDE];
  __shared__ int tidx[NB_TRI];
  extern __shared__ __align__(16) double nb_sm[];
  double* Bk = nb_sm;                            // [NB_PTS][NB_TRI][K]
  double* Sg = Bk + NB_PTS * NB_TRI * K;         // [NB_TRI][6][RW]
  const NearTask w = tasks[blockIdx.x];
  const int leaf = a.leaves[w.li];
  const int s0 = a.box_src_start[leaf], sn = a.do_src ? a.box_src_count[leaf] : 0, t0 = a.box_tgt_start[leaf];
  const int tid = threadIdx.x;
  const int pp = tid / NB_TRI, tt = tid % NB_TRI;  // phase 1: (point, triangle)
  const int rr = tid % 16, pq = tid / 16;          // phase 2: (point, rhs lane)
  const double al = (a.rlam + a.rmu) / (a.rlam + 2.0 * a.rmu), i2mu = 0.5 / a.rmu;
  // phase-1 point
  const int e1 = w.e0 + pp;
  const bool ok1 = pp < w.ne;
  const bool src1 = e1 < sn;
  const int pid1 = ok1 ? (src1 ? s0 + e1 : t0 + (e1 - sn)) : 0;
  double X[3] = {0, 0, 0};
  if (ok1) {
    const double* P = src1 ? a.src_pts + 3 * (size_t)pid1 : a.tgt_pts + 3 * (size_t)pid1;
    X[0] = P[0]; X[1] = P[1]; X[2] = P[2];
  }
  double acc[9][RB];
#pragma unroll
  for (int c = 0; c < 9; c++)
#pragma unroll
    for (int k = 0; k < RB; k++) acc[c][k] = 0.0;
  int left = w.cnt, b = w.r0, k = w.k0;  // range and triangle of the range to stage next
  while (left > 0) {
    __syncthreads();
    int cnt = 0;
    while (left > 0 && cnt < NB_TRI) {  // tiles fill across ranges
      const int2 rg = a.rng[b];
      const int m = min(min(NB_TRI - cnt, rg.y - k), left), tr0 = rg.x + k;
      const double2* src = reinterpret_cast<const double2*>(a.rec + tr0);
      for (int q = tid; q < 16 * m; q += NB_THREADS)
        reinterpret_cast<double2*>(tile + (cnt + q / 16) * NL_STRIDE)[q % 16] = src[q];
      if (tid < m) tidx[cnt + tid] = tr0 + tid;
      cnt += m;
      left -= m;
      k += m;
      if (k >= rg.y) {
        b++;
        k = 0;
      }
    }
    __syncthreads();
    for (int q = tid; q < NB_TRI * 6 * RW; q += NB_THREADS) {
      const int t = q / (6 * RW), j = (q / RW) % 6, r = q % RW;
      const int layer = j / 3, d = j % 3;
      double v = 0.0;
      if (t < cnt && r < R && (layer == 0 ? a.dosl : a.dodl)) {
        const double* sg = layer == 0 ? ssl : sdl;
        v = sg[((size_t)tidx[t] * 3 + d) * R + r];
      }
      Sg[q] = v;
    }
    {
      double* o = Bk + (pp * NB_TRI + tt) * K;
      if (ok1 && tt < cnt) {
        const TriEdge& T = *reinterpret_cast<const TriEdge*>(tile + tt * NL_STRIDE);
        near_pair_blocks(T, X, src1 && tidx[tt] == pid1, a.dosl, a.dodl, dostrain, al, i2mu, o);
      } else {
        for (int q = 0; q < K; q++) o[q] = 0.0;
      }
    }
    __syncthreads();
    for (int t = 0; t < cnt; t++) {
      const double* Bt = Bk + (pq * NB_TRI + t) * K;
      int q0 = 0;
      for (int j = 0; j < 6; j++) {
        if ((j < 3 && !a.dosl) || (j >= 3 && !a.dodl)) continue;
        double sv[RB];
#pragma unroll
        for (int q = 0; q < RB; q++) sv[q] = Sg[(t * 6 + j) * RW + rr + 16 * q];
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
          for (int q = 0; q < RB; q++) acc[c][q] += Bt[q0 + c] * sv[q];
        q0 += 3;
        if (dostrain) {
#pragma unroll
          for (int c = 0; c < 6; c++)
#pragma unroll
            for (int q = 0; q < RB; q++) acc[3 + c][q] += Bt[q0 + c] * sv[q];
          q0 += 6;
        }
      }
    }
  }
  const int e2 = w.e0 + pq;
  if (pq >= w.ne) return;
  const bool src2 = e2 < sn;
  const int pid2 = src2 ? s0 + e2 : t0 + (e2 - sn);
  const size_t np = src2 ? (size_t)nsrc : (size_t)ntgt;
  const bool ds2 = src2 ? a.dostrain_src : a.dostrain_tgt;
#pragma unroll
  for (int k = 0; k < RB; k++) {
    const int r = rr + 16 * k;
    if (r >= R) continue;
    double* U = (src2 ? a.u_src : a.u_tgt) + 3 * (np * r + pid2);
    double* E = (src2 ? a.e_src : a.e_tgt) + 6 * (np * r + pid2);
    if (w.shared) {
#pragma unroll
      for (int c = 0; c < 3; c++) atomicAdd(U + c, acc[c][k]);
      if (ds2)
#pragma unroll
        for (int c = 0; c < 6; c++) atomicAdd(E + c, acc[3 + c][k]);
    } else {
#pragma unroll
      for (int c = 0; c < 3; c++) U[c] += acc[c][k];
      if (ds2)
#pragma unroll
        for (int c = 0; c < 6; c++) E[c] += acc[3 + c][k];
    }
  }
}

// Batched replay of the stored near field, specialised on the layer count
// NLAY (1: one layer, 2: both) and strain STR: compile-time block size
// K = 3 NLAY (3 + 6 STR), only the enabled layers' densities staged, every
// inner loop unrolled.  Same tiling as k_near_batch (work items of 8 points, 16
// triangles per tile, 9 x RB outputs per thread).  Items instead of whole
// lists: the image replay of 64 right-hand sides on 18,034 triangles, where few
// points have near triangles, 10.5 -> 2.8 ms.  The next tile's triangles are
// looked up while this one's are read, so that a tile costs two barriers, and
// the densities are read before the store: 5 right-hand sides, near field alone
// of 5,120 triangles + 1,000 targets 12.5 ms (three barriers 21, the store
// first 23).
template <int RB, int NLAY, int STR>
__global__ void __launch_bounds__(NB_THREADS)
k_near_replay_batch(const NearArgs a, const NearTask* __restrict__ tasks, int R,
                    const double* __restrict__ sg0, const double* __restrict__ sg1, int nsrc, int ntgt,
                    const long long* __restrict__ sbase, const int* __restrict__ sntri,
                    const double* __restrict__ store) {
  constexpr int RW = 16 * RB, NJ = 3 * NLAY, KB = 3 + 6 * STR, K = NJ * KB;
  extern __shared__ __align__(16) double rb_sm[];
  double* Bk = rb_sm;                     // [NB_PTS][NB_TRI][K]
  double* Sg = Bk + NB_PTS * NB_TRI * K;  // [NB_TRI][NJ][RW]
  __shared__ int tidx[2][NB_TRI];  // this tile's triangles and the next one's
  const NearTask w = tasks[blockIdx.x];
  const int leaf = a.leaves[w.li];
  const int s0 = a.box_src_start[leaf], sn = a.do_src ? a.box_src_count[leaf] : 0, t0 = a.box_tgt_start[leaf];
  const int tid = threadIdx.x;
  const int rr = tid % 16, pq = tid / 16;
  const int nt = sntri[w.li];
  const double* src = store + sbase[w.li] + ((size_t)w.e0 * nt + w.p0) * K;
  double acc[KB][RB];
#pragma unroll
  for (int c = 0; c < KB; c++)
#pragma unroll
    for (int k = 0; k < RB; k++) acc[c][k] = 0.0;
  int b = w.r0, k = w.k0;  // range and triangle of the range to stage next
  auto stage = [&](int pos, int* to) {  // the triangles of the tile at pos, across ranges
    const int cnt = min(NB_TRI, w.cnt - pos);
    for (int fill = 0; fill < cnt;) {
      const int2 rg = a.rng[b];
      const int m = min(cnt - fill, rg.y - k);
      if (tid < m) to[fill + tid] = rg.x + k + tid;
      fill += m;
      k += m;
      if (k >= rg.y) {
        b++;
        k = 0;
      }
    }
  };
  stage(0, tidx[0]);
  for (int pos = 0; pos < w.cnt; pos += NB_TRI) {
    const int cnt = min(NB_TRI, w.cnt - pos), cur = (pos / NB_TRI) & 1;
    __syncthreads();
    for (int q = tid; q < NB_TRI * NJ * RW; q += NB_THREADS) {
      const int t = q / (NJ * RW), j = (q / RW) % NJ, r = q % RW;
      const double* sg = (NLAY == 2 && j >= 3) ? sg1 : sg0;
      double v = 0.0;
      if (t < cnt && r < R) v = sg[((size_t)tidx[cur][t] * 3 + (j % 3)) * R + r];
      Sg[q] = v;
    }
    for (int q = tid; q < NB_PTS * NB_TRI * K; q += NB_THREADS) {
      const int pt = q / (NB_TRI * K), rem = q % (NB_TRI * K);
      double v = 0.0;
      if (pt < w.ne && rem < cnt * K) v = __ldcs(src + ((size_t)pt * nt + pos) * K + rem);
      Bk[q] = v;
    }
    if (pos + NB_TRI < w.cnt) stage(pos + NB_TRI, tidx[cur ^ 1]);
    __syncthreads();
    const double* Bp = Bk + pq * NB_TRI * K;
#pragma unroll 2
    for (int t = 0; t < cnt; t++) {
      const double* Bt = Bp + t * K;
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        double sv[RB];
#pragma unroll
        for (int q = 0; q < RB; q++) sv[q] = Sg[(t * NJ + j) * RW + rr + 16 * q];
#pragma unroll
        for (int c = 0; c < KB; c++) {
          const double bv = Bt[j * KB + c];
#pragma unroll
          for (int q = 0; q < RB; q++) acc[c][q] += bv * sv[q];
        }
      }
    }
  }
  const int e2 = w.e0 + pq;
  if (pq >= w.ne) return;
  const bool src2 = e2 < sn;
  const int pid2 = src2 ? s0 + e2 : t0 + (e2 - sn);
  const size_t np = src2 ? (size_t)nsrc : (size_t)ntgt;
  const bool ds2 = src2 ? a.dostrain_src : a.dostrain_tgt;
#pragma unroll
  for (int k = 0; k < RB; k++) {
    const int r = rr + 16 * k;
    if (r >= R) continue;
    double* U = (src2 ? a.u_src : a.u_tgt) + 3 * (np * r + pid2);
    double* E = (src2 ? a.e_src : a.e_tgt) + 6 * (np * r + pid2);
    if (w.shared) {
#pragma unroll
      for (int c = 0; c < 3; c++) atomicAdd(U + c, acc[c][k]);
      if (STR && ds2)
#pragma unroll
        for (int c = 0; c < 6; c++) atomicAdd(E + c, acc[STR ? 3 + c : 0][k]);
    } else {
#pragma unroll
      for (int c = 0; c < 3; c++) U[c] += acc[c][k];
      if (STR && ds2)
#pragma unroll
        for (int c = 0; c < 6; c++) E[c] += acc[STR ? 3 + c : 0][k];
    }
  }
}

// ------------------------------------- stored near field on the tensor cores
// Mixed-precision replay of the ITER store as one dense product per leaf:
// out[row][r] = sum_k A[k][row] S[r][k] with k = NJ t + j (near triangle t,
// density component j of the NJ = 3 x layers stored) and row = KB e + c
// (evaluation point e, output c of KB = 3 (+ 6 strain)).  A is the FP64
// store converted once to FP32 in this layout (same per-leaf offsets, lda =
// KB x points); S the leaf's near densities gathered per right-hand side;
// the product runs on the tensor cores (gemm_product<float>) and the
// results are added to the FP64 outputs.

// Position of the leaf's own triangles in its near list (-1 if absent):
// the self pairs (source point e, near triangle self + e) are applied in
// FP64 from the FP64 store (k_near_self64), not through the FP32 copy.
__device__ __forceinline__ int near_self_pos(const NearArgs& a, int i, int leaf) {
  int pos = 0;
  for (int b = a.nb_start[i]; b < a.nb_start[i + 1]; b++) {
    const int sb = a.nb_items[b];
    if (sb == leaf) return pos;
    pos += a.box_src_count[sb];
  }
  return -1;
}

// FP64 store [point][near triangle][K] -> FP32 [NJ t + j][KB e + c], per leaf
// at fbase[i] with rows of ceil4(KB x points) floats (padding zero; self
// pairs zero).
__global__ void __launch_bounds__(256)
k_near_store_tc(const NearArgs a, const long long* __restrict__ base, const long long* __restrict__ fbase,
                const int* __restrict__ ntri, int K, int KB, const double* __restrict__ store,
                float* __restrict__ out) {
  const int i = blockIdx.x, leaf = a.leaves[i];
  const int sn = a.do_src ? a.box_src_count[leaf] : 0;
  const int nep = sn + (a.do_tgt ? a.box_tgt_count[leaf] : 0);
  const long long nt = ntri[i], M = (long long)KB * nep, Mp = (M + 3) & ~3LL, NJ = K / KB, tot = nep * nt * K;
  const int self = near_self_pos(a, i, leaf);
  const double* src = store + base[i];
  float* dst = out + fbase[i];
  for (long long q = blockIdx.y * (long long)blockDim.x + threadIdx.x; q < tot; q += (long long)gridDim.y * blockDim.x) {
    const long long e = q / (nt * K), rem = q % (nt * K), t = rem / K, jc = rem % K;
    const long long j = jc / KB, c = jc % KB;
    const bool is_self = e < sn && self >= 0 && t == self + e;
    dst[(t * NJ + j) * Mp + e * KB + c] = is_self ? 0.0f : (float)src[q];
  }
  // the padding of each row
  const long long pad = Mp - M, rows = nt * NJ;
  for (long long q = blockIdx.y * (long long)blockDim.x + threadIdx.x; q < rows * pad;
       q += (long long)gridDim.y * blockDim.x)
    dst[(q / pad) * Mp + M + q % pad] = 0.0f;
}

// FP64 store [point][near triangle][K] -> tiles of the pre-split store: per
// leaf at tbase[i], tile (mt, kt) at (mt nkt + kt) 8192 floats holding rows
// 128 mt.. (KB e + c) and k 32 kt.. (NJ t + j) of A, the TF32 head of each
// element then its tail, in the canonical K-major layout (element (row, k)
// at (k % 4) + 4 (row % 8) + 32 (k / 4) + 256 (row / 8)); zero past M and K
// and at the self pairs (applied in FP64).  CTAs (leaf, blockIdx.y) over the
// leaf's tiles; the stores are coalesced, the loads gather from runs of the
// pair blocks.
__global__ void __launch_bounds__(256)
k_near_split_store(const NearArgs a, const long long* __restrict__ base, const long long* __restrict__ tbase,
                   const int* __restrict__ ntri, int K, int KB, const double* __restrict__ store,
                   float* __restrict__ out) {
  const int i = blockIdx.x, leaf = a.leaves[i];
  const int sn = a.do_src ? a.box_src_count[leaf] : 0;
  const int nep = sn + (a.do_tgt ? a.box_tgt_count[leaf] : 0);
  const long long nt = ntri[i], NJ = K / KB, M = (long long)KB * nep, KK = NJ * nt;
  const long long nmt = (M + 127) / 128, nkt = (KK + 31) / 32;
  const int self = near_self_pos(a, i, leaf);
  const double* src = store + base[i];
  float* dst = out + tbase[i];
  for (long long tile = blockIdx.y; tile < nmt * nkt; tile += gridDim.y) {
    const long long mt = tile / nkt, kt = tile % nkt;
    float* o = dst + tile * 8192;
    for (int q = threadIdx.x; q < 4096; q += blockDim.x) {
      const int k = (q & 3) | (((q >> 5) & 7) << 2), m = ((q >> 2) & 7) | ((q >> 8) << 3);
      const long long row = 128 * mt + m, kk = 32 * kt + k;
      float v = 0.0f;
      if (row < M && kk < KK) {
        const long long e = row / KB, c = row % KB, t = kk / NJ, j = kk % NJ;
        if (!(e < sn && self >= 0 && t == self + e)) v = (float)src[(e * nt + t) * K + j * KB + c];
      }
      const float h = tf32_head(v);
      o[q] = h;
      o[4096 + q] = v - h;
    }
  }
}

// Near densities of each leaf as pre-split tiles of 64 columns (right-hand
// sides) x 32 k (k = NJ t + j over the leaf's near triangles t, components
// j), TF32 head then tail, canonical layout: per leaf at sbase[i], tile (ct,
// kt) at (ct nkt + kt) 4096 floats; positions past R or K written as zeros.
// CTAs (leaf, blockIdx.y) over the leaf's tiles: the triangle of each k is
// found by walking the leaf's near boxes, the densities are read 64
// right-hand sides at a time (coalesced) into shared memory (rows of 72
// floats: neither phase has bank conflicts) and written in tile order.
__global__ void __launch_bounds__(256)
k_near_sigma_split(const NearArgs a, int R, int NJ, const double* __restrict__ g0, const double* __restrict__ g1,
                   const long long* __restrict__ sbase, const int* __restrict__ ntri, float* __restrict__ S) {
  __shared__ float sv[32][72];
  __shared__ int tri_k[32];
  const int i = blockIdx.x;
  const int K = NJ * ntri[i], nkt = (K + 31) / 32, nct = (R + 63) / 64;
  float* o = S + sbase[i];
  for (int tile = blockIdx.y; tile < nct * nkt; tile += gridDim.y) {
    const int ct = tile / nkt, kt = tile % nkt;
    __syncthreads();  // the previous tile's reads of sv and tri_k are done
    if (threadIdx.x < 32) {
      const int kk = 32 * kt + threadIdx.x;
      int tri = -1;
      if (kk < K) {
        int u = kk / NJ;
        for (int b = a.nb_start[i]; b < a.nb_start[i + 1]; b++) {
          const int sb = a.nb_items[b], cnt = a.box_src_count[sb];
          if (u < cnt) {
            tri = a.box_src_start[sb] + u;
            break;
          }
          u -= cnt;
        }
      }
      tri_k[threadIdx.x] = tri;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 2048; q += blockDim.x) {
      const int n = q & 63, k = q >> 6, r = 64 * ct + n, tri = tri_k[k];
      float v = 0.0f;
      if (tri >= 0 && r < R) {
        const int j = (32 * kt + k) % NJ;
        v = (float)(j >= 3 ? g1 : g0)[((size_t)tri * 3 + (j % 3)) * R + r];
      }
      sv[k][n] = v;
    }
    __syncthreads();
    float* t = o + (long long)tile * 4096;
    for (int q = threadIdx.x; q < 2048; q += blockDim.x) {
      const int k = (q & 3) | (((q >> 5) & 7) << 2), n = ((q >> 2) & 7) | ((q >> 8) << 3);
      const float v = sv[k][n], h = tf32_head(v);
      t[q] = h;
      t[2048 + q] = v - h;
    }
  }
}

// The self pairs of the mixed replay in FP64: per source point of the leaf
// (thread) and group of SELF_RB right-hand sides (blockIdx.y), the FP64
// stored block (NJ density components x KB outputs, read once into
// registers) times the FP64 densities of the point's own triangle, ADDED to
// the outputs.
constexpr int SELF_RB = 8;
template <int NJ, int KB>
__global__ void __launch_bounds__(128)
k_near_self64(const NearArgs a, int R, const double* __restrict__ g0, const double* __restrict__ g1,
              const long long* __restrict__ base, const int* __restrict__ ntri, const double* __restrict__ store,
              int nsrc) {
  constexpr int K = NJ * KB;
  const int i = blockIdx.x, r0 = blockIdx.y * SELF_RB, leaf = a.leaves[i];
  const int s0 = a.box_src_start[leaf], sn = a.do_src ? a.box_src_count[leaf] : 0;
  const int self = near_self_pos(a, i, leaf);
  if (self < 0) return;
  const long long nt = ntri[i];
  const int rn = min(SELF_RB, R - r0);
  for (int e = threadIdx.x; e < sn; e += blockDim.x) {
    const int pid = s0 + e;
    const double* blk = store + base[i] + ((long long)e * nt + self + e) * K;
    double bk[K];
#pragma unroll
    for (int k = 0; k < K; k++) bk[k] = blk[k];
    for (int rr = 0; rr < rn; rr++) {
      const int r = r0 + rr;
      double out[KB];
#pragma unroll
      for (int c = 0; c < KB; c++) out[c] = 0.0;
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const double sv = (j >= 3 ? g1 : g0)[((size_t)pid * 3 + (j % 3)) * R + r];
#pragma unroll
        for (int c = 0; c < KB; c++) out[c] += bk[j * KB + c] * sv;
      }
      double* U = a.u_src + 3 * ((size_t)nsrc * r + pid);
#pragma unroll
      for (int c = 0; c < 3; c++) U[c] += out[c];
      if (KB == 9 && a.dostrain_src) {
        double* E = a.e_src + 6 * ((size_t)nsrc * r + pid);
#pragma unroll
        for (int c = 0; c < 6; c++) E[c] += out[3 + c];
      }
    }
  }
}

static void launch_near_self64(cudaStream_t st, const NearArgs& a, int R, int NJ, int KB, const double* g0,
                               const double* g1, const long long* base, const int* ntri, const double* store,
                               int nsrc) {
  const dim3 grid(a.nleaf, (R + SELF_RB - 1) / SELF_RB);
  if (NJ == 3 && KB == 3)
    k_near_self64<3, 3><<<grid, 128, 0, st>>>(a, R, g0, g1, base, ntri, store, nsrc);
  else if (NJ == 3 && KB == 9)
    k_near_self64<3, 9><<<grid, 128, 0, st>>>(a, R, g0, g1, base, ntri, store, nsrc);
  else if (NJ == 6 && KB == 3)
    k_near_self64<6, 3><<<grid, 128, 0, st>>>(a, R, g0, g1, base, ntri, store, nsrc);
  else if (NJ == 6 && KB == 9)
    k_near_self64<6, 9><<<grid, 128, 0, st>>>(a, R, g0, g1, base, ntri, store, nsrc);
  else
    throw CudaError{(int)cudaErrorInvalidValue};
  count_launch();
}

// Near densities of each leaf as the B operand: S[r][NJ t + j] at soff[leaf]
// (row length ntri NJ rounded up to 4), from sigma[(tri 3 + comp) R + r]
// (g0: the first layer stored, g1: the double layer when both are).
__global__ void __launch_bounds__(256)
k_near_sigma_tc(const NearArgs a, int R, int NJ, const double* __restrict__ g0, const double* __restrict__ g1,
                const long long* __restrict__ soff, const int* __restrict__ ntri, float* __restrict__ S) {
  const int i = blockIdx.x;
  const int K = NJ * ntri[i], Kp = (K + 3) & ~3;
  float* o = S + soff[i];
  int pos = 0;
  for (int b = a.nb_start[i]; b < a.nb_start[i + 1]; b++) {
    const int sb = a.nb_items[b];
    const int tr0 = a.box_src_start[sb], trn = a.box_src_count[sb];
    for (int q = threadIdx.x; q < trn * NJ * R; q += blockDim.x) {
      const int r = q / (trn * NJ), k = q % (trn * NJ), t = k / NJ, j = k % NJ;
      const double* sg = j >= 3 ? g1 : g0;
      o[(size_t)r * Kp + (size_t)(pos + t) * NJ + j] = (float)sg[((size_t)(tr0 + t) * 3 + (j % 3)) * R + r];
    }
    pos += trn;
  }
}

// Add the products C[r][KB e + c] (per leaf at coff) to the outputs.
__global__ void __launch_bounds__(256)
k_near_scatter_tc(const NearArgs a, int R, int KB, const long long* __restrict__ coff, const double* __restrict__ C,
                  int nsrc, int ntgt) {
  const int i = blockIdx.x, r = blockIdx.y, leaf = a.leaves[i];
  const int s0 = a.box_src_start[leaf], sn = a.do_src ? a.box_src_count[leaf] : 0;
  const int t0 = a.box_tgt_start[leaf], tn = a.do_tgt ? a.box_tgt_count[leaf] : 0;
  const int M = KB * (sn + tn);
  const double* Cr = C + coff[i] + (size_t)r * M;
  for (int row = threadIdx.x; row < M; row += blockDim.x) {
    const int e = row / KB, c = row % KB;
    const bool src = e < sn;
    const int pid = src ? s0 + e : t0 + (e - sn);
    const size_t np = src ? (size_t)nsrc : (size_t)ntgt;
    const double v = Cr[row];
    if (c < 3) {
      (src ? a.u_src : a.u_tgt)[3 * (np * r + pid) + c] += v;
    } else if (src ? a.dostrain_src : a.dostrain_tgt) {
      (src ? a.e_src : a.e_tgt)[6 * (np * r + pid) + (c - 3)] += v;
    }
  }
}

void launch_near_store_tc(cudaStream_t st, const NearArgs& a, const long long* base, const long long* fbase,
                          const int* ntri, int K, int KB, const double* store, float* out) {
  if (a.nleaf <= 0) return;
  k_near_store_tc<<<dim3(a.nleaf, 64), 256, 0, st>>>(a, base, fbase, ntri, K, KB, store, out);
  count_launch();
  EFMM_CUDA_TRY(cudaGetLastError());
}

void launch_near_split_store(cudaStream_t st, const NearArgs& a, const long long* base, const long long* tbase,
                             const int* ntri, int K, int KB, const double* store, float* out) {
  if (a.nleaf <= 0) return;
  k_near_split_store<<<dim3(a.nleaf, 32), 256, 0, st>>>(a, base, tbase, ntri, K, KB, store, out);
  count_launch();
  EFMM_CUDA_TRY(cudaGetLastError());
}

void launch_near_split(cudaStream_t st, const NearArgs& a, int R, int NJ, int KB, const double* g0,
                       const double* g1, const long long* sbase, const int* ntri, float* S, int ntask,
                       const BulkTask* tasks, const float* A, const long long* coff, double* C, int nsrc, int ntgt,
                       const long long* base, const double* store, int* err, cudaEvent_t* ev) {
  if (a.nleaf <= 0 || R <= 0) return;
  k_near_sigma_split<<<dim3(a.nleaf, 8), 256, 0, st>>>(a, R, NJ, g0, g1, sbase, ntri, S);
  count_launch();
  if (ev) EFMM_CUDA_TRY(cudaEventRecord(ev[0], st));
  launch_tc_bulk<double>(st, ntask, tasks, A, S, C, err, 64);
  if (ev) EFMM_CUDA_TRY(cudaEventRecord(ev[1], st));
  k_near_scatter_tc<<<dim3(a.nleaf, R), 256, 0, st>>>(a, R, KB, coff, C, nsrc, ntgt);
  count_launch();
  if (a.do_src) {
    launch_near_self64(st, a, R, NJ, KB, g0, g1, base, ntri, store, nsrc);
  }
  EFMM_CUDA_TRY(cudaGetLastError());
}

void launch_near_tc(cudaStream_t st, const NearArgs& a, int R, int NJ, int KB, const double* g0, const double* g1,
                    const long long* soff, const int* ntri, float* S, int ntask, const GemmTask* tasks,
                    const float* A, const long long* coff, double* C, int nsrc, int ntgt, const long long* base,
                    const double* store) {
  if (a.nleaf <= 0 || R <= 0) return;
  k_near_sigma_tc<<<a.nleaf, 256, 0, st>>>(a, R, NJ, g0, g1, soff, ntri, S);
  count_launch();
  launch_gemm_tc(st, ntask, tasks, A, S, C, tc_err_ptr(), R <= 64 ? 64 : 128);
  k_near_scatter_tc<<<dim3(a.nleaf, R), 256, 0, st>>>(a, R, KB, coff, C, nsrc, ntgt);
  count_launch();
  if (a.do_src) {
    launch_near_self64(st, a, R, NJ, KB, g0, g1, base, ntri, store, nsrc);
  }
  EFMM_CUDA_TRY(cudaGetLastError());
}

// ---------------------------------------------------------------- launchers
void launch_tri_edge_prep(cudaStream_t st, int n, const double* tri, const double* ssl, const double* sdl, int dosl,
                          int dodl, TriEdge* out, int R, int r) {
  if (n <= 0) return;
  k_tri_edge_prep<<<(n + 127) / 128, 128, 0, st>>>(n, tri, ssl, sdl, dosl, dodl, R, r, out); count_launch();
}

void launch_near_leaf(cudaStream_t st, const NearArgs& a, int ntask, const NearTask* tasks) {
  if (ntask <= 0) return;
  if (a.dosl && a.dodl)
    k_near_leaf<true, true><<<ntask, NL_THREADS, 0, st>>>(a, tasks);
  else if (a.dosl)
    k_near_leaf<true, false><<<ntask, NL_THREADS, 0, st>>>(a, tasks);
  else
    k_near_leaf<false, true><<<ntask, NL_THREADS, 0, st>>>(a, tasks);
  count_launch();
}

void launch_near_store(cudaStream_t st, const NearArgs& a, const long long* base, const int* ntri, int K,
                       double* store) {
  if (a.nleaf <= 0) return;
  k_near_store<<<dim3(a.nleaf, 16), NF_WARPS * 32, 0, st>>>(a, base, ntri, K, store); count_launch();
}

void launch_near_batch(cudaStream_t st, const NearArgs& a, int ntask, const NearTask* tasks, int R, int dostrain,
                       const double* ssl, const double* sdl, int nsrc, int ntgt) {
  if (ntask <= 0 || R <= 0) return;
  if (R > 64) throw CudaError{(int)cudaErrorInvalidValue};
  const int K = (a.dosl + a.dodl) * 3 * (3 + 6 * dostrain);
  const int RB = (R + 15) / 16;
  const int smem = (int)(sizeof(double) * (NB_PTS * NB_TRI * K + NB_TRI * 6 * 16 * RB));
  auto go = [&](auto kern) {
    EFMM_CUDA_TRY(smem_raise(kern, (int)(smem)));
    kern<<<ntask, NB_THREADS, smem, st>>>(a, tasks, R, K, dostrain, ssl, sdl, nsrc, ntgt);
    count_launch();
  };
  switch (RB) {
    case 1: go(k_near_batch<1>); break;
    case 2: go(k_near_batch<2>); break;
    case 3: go(k_near_batch<3>); break;
    default: go(k_near_batch<4>); break;
  }
  EFMM_CUDA_TRY(cudaGetLastError());
}

// Up to this many right-hand sides the store is streamed (k_near_replay):
// 18,034 triangles, iprec 3 (about 16 GB): 3.4 ms for 2 and 6.3 for 4 against
// 8.7 ms of k_near_replay_batch for any number up to 16.
constexpr int NEAR_STREAM_R = 4;
void launch_near_replay_batch(cudaStream_t st, const NearArgs& a, int ntask, const NearTask* tasks, int R,
                              int dostrain, const double* ssl, const double* sdl, int nsrc, int ntgt,
                              const long long* sbase, const int* sntri, const double* store) {
  // without a layer the store is empty (K = 0) and there is nothing to add
  if (ntask <= 0 || R <= 0 || !(a.dosl || a.dodl)) return;
  if (R > 64) throw CudaError{(int)cudaErrorInvalidValue};
  const int nlay = a.dosl + a.dodl, str = dostrain, K = nlay * 3 * (3 + 6 * dostrain), RB = (R + 15) / 16;
  const double* g0 = a.dosl ? ssl : sdl;
  const double* g1 = sdl;
  if (R <= NEAR_STREAM_R) {  // one read of the store, one warp per point
    const int rr = R == 1 ? 1 : (R == 2 ? 2 : 4);
    auto stream = [&](auto kern) {
      const int sm = RS_TILE * 3 * nlay * rr * (int)sizeof(double);
      EFMM_CUDA_TRY(smem_raise(kern, sm));
      kern<<<ntask, 256, sm, st>>>(a, tasks, R, g0, g1, nsrc, ntgt, sbase, sntri, store);
      count_launch();
    };
#define EFMM_RR(RRV)                                             \
  if (nlay == 1 && !str) stream(k_near_replay<RRV, 3, 1>);       \
  else if (nlay == 1) stream(k_near_replay<RRV, 9, 1>);          \
  else if (!str) stream(k_near_replay<RRV, 3, 2>);               \
  else stream(k_near_replay<RRV, 9, 2>);
    if (rr == 1) { EFMM_RR(1) }
    else if (rr == 2) { EFMM_RR(2) }
    else { EFMM_RR(4) }
#undef EFMM_RR
    EFMM_CUDA_TRY(cudaGetLastError());
    return;
  }
  const int smem = (int)(sizeof(double) * (NB_PTS * NB_TRI * K + NB_TRI * 3 * nlay * 16 * RB));
  auto go = [&](auto kern) {
    EFMM_CUDA_TRY(smem_raise(kern, (int)(smem)));
    kern<<<ntask, NB_THREADS, smem, st>>>(a, tasks, R, g0, g1, nsrc, ntgt, sbase, sntri, store);
    count_launch();
  };
#define EFMM_RB(RBV)                                                        \
  if (nlay == 1 && !str) go(k_near_replay_batch<RBV, 1, 0>);                \
  else if (nlay == 1) go(k_near_replay_batch<RBV, 1, 1>);                   \
  else if (!str) go(k_near_replay_batch<RBV, 2, 0>);                        \
  else go(k_near_replay_batch<RBV, 2, 1>);
  switch (RB) {
    case 1: EFMM_RB(1) break;
    case 2: EFMM_RB(2) break;
    case 3: EFMM_RB(3) break;
    default: EFMM_RB(4) break;
  }
#undef EFMM_RB
  EFMM_CUDA_TRY(cudaGetLastError());
}

void launch_direct_all(cudaStream_t st, int ntri, const TriEdge* rec, int nsrc, const double* src_pts, int ntgt,
                       const double* tgt_pts, int dosl, int dodl, int dostrain_src, int dostrain_tgt, double rlam,
                       double rmu, double* u_src, double* e_src, double* u_tgt, double* e_tgt) {
  const int nep = nsrc + ntgt;
  if (nep <= 0) return;
  // up to 8 CTAs (a cluster) share the triangles of a block of points so that
  // few points still cover the chip about three times (3 CTAs per SM), but no
  // part of fewer than about 16
  const int nb = (nep + ND_PTS - 1) / ND_PTS;
  const int parts = std::max(1, std::min({(3 * 3 * 148 + nb - 1) / nb, (ntri + 15) / 16, 8}));
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1;
  at.val.clusterDim.y = parts;
  at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nb, parts);
  cfg.blockDim = dim3(NL_THREADS);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  auto go = [&](auto kern) {
    EFMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, ntri, rec, nsrc, src_pts, ntgt, tgt_pts, dostrain_src,
                                     dostrain_tgt, rlam, rmu, u_src, e_src, u_tgt, e_tgt));
  };
  if (dosl && dodl)
    go(k_direct_all<true, true>);
  else if (dosl)
    go(k_direct_all<true, false>);
  else
    go(k_direct_all<false, true>);
  count_launch();
}

}  // namespace efmm
