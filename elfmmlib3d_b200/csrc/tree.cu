// tree.cu -- adaptive oct-tree and interaction lists on the GPU.
//
// Reproduces the boxes, point orders and lists of the reference builder
// d3tstrcr (src/d3tstrcr.f:31, d3tallbem :1249, lists d3tlsts :702 / d3tlst31
// :919) for the same points:
//   * the root is the bounding cube of sources and targets (Mindlin variant:
//     centred on z = 0, side >= 2 max|z|, src/d3tstrcr_mindlin.f:1380);
//   * a box splits while it holds more than nbox sources or nbox targets;
//   * points are partitioned stably by z, then y, then x against the box
//     centre (coordinate > centre goes to the upper child), child digit
//     d = ix + 2 iy + 4 iz, empty children are skipped, boxes are numbered
//     breadth-first;
//   * box centres use the reference's floating-point expression (no FMA).
// One level at a time: the points of a splitting box are partitioned stably by
// their digit (one CTA per box; where a box holds more than PART_MAX points, a
// stable radix sort of all points by (start of box, digit) instead), and
// children are created from the per-box digit counts.
// Lists: 5 (colleagues) and 2 from the parent's colleagues' children, 1 and 3
// from a depth-first walk below each leaf's colleagues, 4 as the dual of 3.
//
// Forest (no counterpart in the reference): many independent problems in one
// tree.  The caller places problem k in its own column of boxes of level L
// (grid position (i, j) of that level, all k) and gives the root cube; every
// box above level L splits, and boxes of different columns are never
// colleagues, so every list stays inside one problem and each problem sees
// the FMM of the subtree below its column.
#include <vector>
#include <algorithm>
#include "common.cuh"
#include "devbuf.h"
#include "sort.h"
#include "tree.h"

namespace efmm {

// reference box centre, src/d3tstrcr.f:1682 (d3tcentf) without contraction
__device__ __forceinline__ double centf(double c0, double size, double side, int i) {
  double x0 = __dsub_rn(c0, size / 2.0);
  double t = __dmul_rn((double)(i - 1), side);
  return __dadd_rn(__dadd_rn(x0, t), side / 2.0);
}

__global__ void k_bbox(int n, const double* __restrict__ p, double* out /* 6: mins, maxs */) {
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int c = 0; c < 3; c++) {
      double v = p[3 * (size_t)i + c];
      mn[c] = fmin(mn[c], v);
      mx[c] = fmax(mx[c], v);
    }
  for (int c = 0; c < 3; c++) {
    for (int o = 16; o > 0; o >>= 1) {
      mn[c] = fmin(mn[c], __shfl_xor_sync(0xffffffffu, mn[c], o));
      mx[c] = fmax(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    for (int c = 0; c < 3; c++) {
      // monotone integer images of doubles for atomic min/max
      unsigned long long* o = reinterpret_cast<unsigned long long*>(out);
      auto enc = [](double v) {
        unsigned long long b = __double_as_longlong(v);
        return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
      };
      atomicMin(o + c, enc(mn[c]));
      atomicMax(o + 3 + c, enc(mx[c]));
    }
  }
}

// every box of a level below `force` splits (the levels above a forest's
// problems), others while they hold more than nbox sources or targets
__global__ void k_split(int lo, int hi, int nbox, int force, const int* __restrict__ scount,
                        const int* __restrict__ tcount, int* __restrict__ split, int* __restrict__ cs,
                        int* __restrict__ ct) {
  int b = lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= hi) return;
  split[b - lo] = (force || scount[b] > nbox || tcount[b] > nbox) ? 1 : 0;
  for (int d = 0; d < 8; d++) cs[8 * (b - lo) + d] = ct[8 * (b - lo) + d] = 0;
}

// the root box and the points' initial order
__global__ void k_root(int n, int nt, int* __restrict__ level, int* __restrict__ ijk, int* __restrict__ parent,
                       int* __restrict__ kids, int* __restrict__ nkids, int* __restrict__ sstart,
                       int* __restrict__ scount, int* __restrict__ tstart, int* __restrict__ tcount,
                       int* __restrict__ iz, int* __restrict__ izt, int* __restrict__ pbs, int* __restrict__ pbt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    level[0] = nkids[0] = sstart[0] = tstart[0] = 0;
    ijk[0] = ijk[1] = ijk[2] = 1;
    parent[0] = -1;
    for (int q = 0; q < 8; q++) kids[q] = -1;
    scount[0] = n;
    tcount[0] = nt;
  }
  if (i < n) {
    iz[i] = i;
    pbs[i] = 0;
  }
  if (i < nt) {
    izt[i] = i;
    pbt[i] = 0;
  }
}

// digit of every point of a splitting box (8: other points), the radix path's
// key (keys not null), and the counts per (split box, digit), added once per
// group of a warp's points with the same box and digit
__global__ void k_digits(int n, const double* __restrict__ pts, const int* __restrict__ perm,
                         const int* __restrict__ pbox, const int* __restrict__ level, int lev,
                         int lo, const int* __restrict__ split, const int* __restrict__ ijk,
                         double c0x, double c0y, double c0z, double size, double side,
                         unsigned char* __restrict__ digit, int* __restrict__ cnt) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int d = 8, b = 0;
  if (i < n) {
    b = pbox[i];
    if (level[b] == lev && split[b - lo]) {
      int j = perm[i];
      double cx = centf(c0x, size, side, ijk[3 * b]);
      double cy = centf(c0y, size, side, ijk[3 * b + 1]);
      double cz = centf(c0z, size, side, ijk[3 * b + 2]);
      int ix = pts[3 * (size_t)j] > cx, iy = pts[3 * (size_t)j + 1] > cy, iz = pts[3 * (size_t)j + 2] > cz;
      d = ix + 2 * iy + 4 * iz;
    }
    digit[i] = (unsigned char)d;
  }
  const int g = d < 8 ? 8 * (b - lo) + d : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, g);
  if (g >= 0 && (__ffs(peers) - 1) == (int)(threadIdx.x & 31)) atomicAdd(&cnt[g], __popc(peers));
}

__global__ void k_digit_keys(int n, const int* __restrict__ pbox, const int* __restrict__ bstart,
                             const unsigned char* __restrict__ digit, unsigned long long* __restrict__ keys) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = ((unsigned long long)bstart[pbox[i]] << 3) | (digit[i] & 7);
}

// Stable partition of the points of one splitting box per CTA by their digit:
// out[start + digits below + equal digits before] = in, and the points' new
// boxes (children in digit order, empty ones skipped, from hi + off).  Rounds
// of blockDim points: ranks within a warp by ballot, over the warps and rounds
// by counters in shared memory.
// Bound by the rounds of one CTA in turn (about 2.4 us per 1,024 points), as the
// radix sort is by its launches: 39 us against 79 for all levels of 16,000
// points, 71 against 57 (radix at the top level only) for 32,000 and 126
// against 66 for 64,000, hence the line at 16,384 points in one box.
constexpr int PART_MAX = 16384;
__global__ void __launch_bounds__(1024)
k_partition(int lo, int hi, const int* __restrict__ split, const int* __restrict__ start,
            const int* __restrict__ count, const int* __restrict__ cnt, const int* __restrict__ cs,
            const int* __restrict__ ct, const int* __restrict__ off, const unsigned char* __restrict__ digit,
            const int* __restrict__ in, int* __restrict__ out, int* __restrict__ pbox) {
  __shared__ int wc[32][8], run[8], child[8];
  const int k = blockIdx.x;
  if (!split[k]) return;
  const int s = start[lo + k], c = count[lo + k], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = blockDim.x >> 5;
  if (tid == 0) {
    int p = s, q = hi + off[k];
    for (int d = 0; d < 8; d++) {
      run[d] = p;
      p += cnt[8 * k + d];
      child[d] = q;
      q += (cs[8 * k + d] + ct[8 * k + d]) > 0;
    }
  }
  for (int r0 = 0; r0 < c; r0 += blockDim.x) {
    const int i = r0 + tid;
    const int d = i < c ? digit[s + i] : 8;
    int rank = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const unsigned m = __ballot_sync(0xffffffffu, d == q);
      if (d == q) rank = __popc(m & ((1u << lane) - 1u));
      if (lane == q) wc[warp][q] = __popc(m);
    }
    __syncthreads();
    if (tid < 8) {  // first position of digit tid per warp
      int p = run[tid];
      for (int w = 0; w < nw; w++) {
        const int t = wc[w][tid];
        wc[w][tid] = p;
        p += t;
      }
      run[tid] = p;
    }
    __syncthreads();
    if (d < 8) {
      const int pos = wc[warp][d] + rank;
      out[pos] = in[s + i];
      pbox[pos] = child[d];
    }
    __syncthreads();
  }
}

// [0] new boxes of the level, [1] the largest splitting box's points
__global__ void k_level_info(int nl, const int* __restrict__ nch, const int* __restrict__ off,
                             const int* __restrict__ split, const int* __restrict__ scount,
                             const int* __restrict__ tcount, int* __restrict__ info) {
  __shared__ int mx;
  if (threadIdx.x == 0) mx = 0;
  __syncthreads();
  int m = 0;
  for (int k = threadIdx.x; k < nl; k += blockDim.x)
    if (split[k]) m = max(m, max(scount[k], tcount[k]));
  atomicMax(&mx, m);
  __syncthreads();
  if (threadIdx.x == 0) {
    info[0] = nch[nl - 1] + off[nl - 1];
    info[1] = mx;
  }
}

__global__ void k_nchild(int nlev, const int* __restrict__ split, const int* __restrict__ cs,
                         const int* __restrict__ ct, int* __restrict__ nch) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nlev) return;
  int c = 0;
  if (split[k])
    for (int d = 0; d < 8; d++) c += (cs[8 * k + d] + ct[8 * k + d]) > 0;
  nch[k] = c;
}

__global__ void k_children(int lo, int hi, int lev, const int* __restrict__ split,
                           const int* __restrict__ cs, const int* __restrict__ ct,
                           const int* __restrict__ off, int* __restrict__ level, int* __restrict__ ijk,
                           int* __restrict__ parent, int* __restrict__ kids, int* __restrict__ nkids,
                           int* __restrict__ sstart, int* __restrict__ scount,
                           int* __restrict__ tstart, int* __restrict__ tcount) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  int b = lo + k;
  if (b >= hi || !split[k]) return;
  int id = hi + off[k];
  int s = sstart[b], t = tstart[b];
  int q = 0;
  for (int d = 0; d < 8; d++) {
    int a = cs[8 * k + d], c = ct[8 * k + d];
    if (a + c > 0) {
      int ch = id + q;
      level[ch] = lev + 1;
      ijk[3 * ch] = 2 * (ijk[3 * b] - 1) + 1 + (d & 1);
      ijk[3 * ch + 1] = 2 * (ijk[3 * b + 1] - 1) + 1 + ((d >> 1) & 1);
      ijk[3 * ch + 2] = 2 * (ijk[3 * b + 2] - 1) + 1 + ((d >> 2) & 1);
      parent[ch] = b;
      nkids[ch] = 0;
      for (int z = 0; z < 8; z++) kids[8 * ch + z] = -1;
      sstart[ch] = s;
      scount[ch] = a;
      tstart[ch] = t;
      tcount[ch] = c;
      kids[8 * b + q] = ch;
      q++;
    }
    s += a;
    t += c;
  }
  nkids[b] = q;
}

// point -> box for the new children (one warp per child)
__global__ void k_pbox(int lo, int hi, const int* __restrict__ start, const int* __restrict__ count,
                       int* __restrict__ pbox) {
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  int b = lo + w;
  if (b >= hi) return;
  int s = start[b], c = count[b];
  for (int i = lane; i < c; i += 32) pbox[s + i] = b;
}

// --------------------------------------------------------------------------
// lists
// --------------------------------------------------------------------------
// reference touch test d3tifint (src/d3tstrcr.f:1082) on box corners
__device__ __forceinline__ void box_corner(const double* c0, double size, int lev, const int* ijk,
                                           double* mn, double* mx) {
  double side = size / (double)(1ull << lev);
  for (int d = 0; d < 3; d++) {
    double c = centf(c0[d], size, side, ijk[d]);
    mn[d] = __dsub_rn(c, side / 2.0);
    mx[d] = __dadd_rn(mn[d], side);
  }
}
__device__ bool touch(const TreeDev& T, int a, int b) {
  double mn1[3], mx1[3], mn2[3], mx2[3];
  box_corner(T.c0, T.size, T.level[a], T.ijk + 3 * a, mn1, mx1);
  box_corner(T.c0, T.size, T.level[b], T.ijk + 3 * b, mn2, mx2);
  double eps = mx1[0] - mn1[0];
  eps = fmin(eps, mx2[0] - mn2[0]);
  eps = fmin(eps, mx2[1] - mn2[1]);
  eps = fmin(eps, mx2[2] - mn2[2]);
  eps = fmin(eps, mx1[1] - mn1[1]);
  eps = fmin(eps, mx1[2] - mn1[2]);
  eps = eps / 10000.0;
  for (int d = 0; d < 3; d++) {
    if (mn1[d] > mx2[d] + eps) return false;
    if (mn2[d] > mx1[d] + eps) return false;
  }
  return true;
}

// Problem of box b in a forest: its grid column (i, j) at level T.flev, -1
// above that level (boxes that hold several problems); 0 without a forest.
__device__ __forceinline__ int fcol(const TreeDev& T, int b) {
  if (T.flev < 0) return 0;
  const int l = T.level[b];
  if (l < T.flev) return -1;
  const int sh = l - T.flev;
  return ((T.ijk[3 * b] - 1) >> sh) + (((T.ijk[3 * b + 1] - 1) >> sh) << T.flev);
}

// Candidates of list 5 and 2 of box b, one warp: the children of the parent's
// colleagues and of the parent itself, 4 (colleague) x 8 (child) lanes at a
// time, in that order.  visit(chunk's kid, is it a colleague, is it in list 2).
template <class F>
__device__ __forceinline__ void list52_walk(const TreeDev& T, int b, int lane, F visit) {
  const int dad = T.parent[b], nd = T.ncoll[dad], fb = fcol(T, b);
  for (int i0 = 0; i0 <= nd; i0 += 4) {
    const int i = i0 + (lane >> 3), q = lane & 7;
    int kid = -1;
    if (i <= nd) {
      const int c = i == 0 ? dad : T.coll[27 * dad + i - 1];
      if (q < T.nkids[c]) kid = T.kids[8 * c + q];
    }
    bool is5 = false, is2 = false;
    if (kid >= 0 && kid != b) {
      const int fk = fcol(T, kid);
      const bool t = touch(T, kid, b);
      is5 = t && fk == fb;
      is2 = !t && fk == fb && fb >= 0;
    }
    visit(kid, is5, is2);
  }
}

// list 5 (27 slots per box, one warp per box) and the number of list-2
// entries, for the boxes of one level.  In a forest, boxes of different
// problems are neither colleagues nor in list 2, and the boxes above the
// problems' level (colleagues among themselves, so that the level below finds
// its colleagues) have no list 2.
__global__ void k_list5(TreeDev T, int lo, int hi, int* __restrict__ l2cnt) {
  const int b = lo + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (b >= hi) return;
  int nc = 0, n2 = 0;
  list52_walk(T, b, lane, [&](int kid, bool is5, bool is2) {
    const unsigned m5 = __ballot_sync(0xffffffffu, is5), m2 = __ballot_sync(0xffffffffu, is2);
    if (is5) T.coll[27 * b + nc + __popc(m5 & ((1u << lane) - 1u))] = kid;
    nc += __popc(m5);
    n2 += __popc(m2);
  });
  if (lane == 0) {
    T.ncoll[b] = nc;
    l2cnt[b] = n2;
  }
}

// list 2 of every box in ascending order at start[b] (at most 27 x 8 - 27
// entries, sorted in shared memory by rank)
constexpr int L2_WARPS = 4, L2_MAX = 224;
__global__ void __launch_bounds__(L2_WARPS * 32)
k_list2(TreeDev T, int nb, const int* __restrict__ start, int* __restrict__ items) {
  __shared__ int buf[L2_WARPS][L2_MAX];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, b = 1 + blockIdx.x * L2_WARPS + w;
  if (b >= nb) return;
  int* it = buf[w];
  int n = 0;
  list52_walk(T, b, lane, [&](int kid, bool, bool is2) {
    const unsigned m2 = __ballot_sync(0xffffffffu, is2);
    if (is2) it[n + __popc(m2 & ((1u << lane) - 1u))] = kid;
    n += __popc(m2);
  });
  __syncwarp();
  int* o = items + start[b];
  for (int k = lane; k < n; k += 32) {
    const int v = it[k];
    int r = 0;
    for (int j = 0; j < n; j++) r += it[j] < v;
    o[r] = v;
  }
}

// d3tlst31: depth-first walk below the colleagues of a leaf, one warp per leaf
// with a colleague per lane.  FILL = false counts the list-1 entries (both
// directions when levels differ), list-3 entries and the dual list-4 ones per
// row; FILL = true writes them at the rows' cursors (any order: the rows are
// sorted afterwards).
template <bool FILL>
__global__ void k_list13(TreeDev T, int nb, int* __restrict__ c1, int* __restrict__ c3, int* __restrict__ c4,
                         int* __restrict__ i1, int* __restrict__ i3, int* __restrict__ i4) {
  const int ib = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (ib >= nb || T.nkids[ib] != 0 || T.level[ib] == 0 || lane >= T.ncoll[ib]) return;
  int n1 = 0, n3 = 0;
  auto add1 = [&](int a, int b) {
    if (FILL) i1[atomicAdd(c1 + a, 1)] = b;
    else if (a == ib) n1++;
    else atomicAdd(c1 + a, 1);
  };
  int stk_box[64], stk_n[64];
  const int j0 = T.coll[27 * ib + lane];
  int is = 0, j = j0;
  stk_box[0] = j;
  stk_n[0] = T.nkids[j];
  for (int guard = 0; guard < (1 << 26); guard++) {
    if (!touch(T, ib, j)) {
      if (FILL) {
        i3[atomicAdd(c3 + ib, 1)] = j;
        i4[atomicAdd(c4 + j, 1)] = ib;
      } else {
        n3++;
        atomicAdd(c4 + j, 1);
      }
      is--;
      stk_n[is]--;
      j = stk_box[is];
      continue;
    }
    if (T.nkids[j] == 0) {
      add1(ib, j);
      if (T.level[j] != T.level[ib]) add1(j, ib);
      if (j == j0) break;
      is--;
      stk_n[is]--;
      j = stk_box[is];
      continue;
    }
    int ns = stk_n[is];
    if (ns == 0) {
      if (j == j0) break;
      is--;
      stk_n[is]--;
      j = stk_box[is];
      continue;
    }
    j = T.kids[8 * j + ns - 1];
    is++;
    if (is >= 64) break;  // deeper than 64 levels below a colleague: cannot happen for < 64-level trees
    stk_box[is] = j;
    stk_n[is] = T.nkids[j];
  }
  if (!FILL) {
    if (n1) atomicAdd(c1 + ib, n1);
    if (n3) atomicAdd(c3 + ib, n3);
  }
}

// Sums and the longest row of three count arrays of nb rows (+ the scan's
// last element): info[0..2] totals, info[3] the longest row; info[4] the
// entries of list 2.
__global__ void k_list_info(int nb, const int* __restrict__ c1, const int* __restrict__ c3,
                            const int* __restrict__ c4, const int* __restrict__ o1, const int* __restrict__ o3,
                            const int* __restrict__ o4, const int* __restrict__ o2, int* __restrict__ info) {
  __shared__ int mx;
  if (threadIdx.x == 0) mx = 0;
  __syncthreads();
  int m = 0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) m = max(m, max(c1[b], max(c3[b], c4[b])));
  atomicMax(&mx, m);
  __syncthreads();
  if (threadIdx.x == 0) {
    info[0] = o1[nb];
    info[1] = o3[nb];
    info[2] = o4[nb];
    info[3] = mx;
    info[4] = o2[nb];
  }
}

// Rows of a CSR sorted ascending by rank (out of place): a warp per row of at
// most ROW_WARP entries, CTAs of 512 threads for longer ones.
constexpr int ROW_WARP = 512;
__global__ void k_row_sort(int nb, const int* __restrict__ start, const int* __restrict__ in, int* __restrict__ out) {
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b >= nb) return;
  const int s = start[b], n = start[b + 1] - s;
  if (n > ROW_WARP) return;
  for (int k = lane; k < n; k += 32) {
    const int v = in[s + k];
    int r = 0;
    for (int j = 0; j < n; j++) {
      const int u = in[s + j];
      r += u < v || (u == v && j < k);
    }
    out[s + r] = v;
  }
}
// 512 rows per CTA column; the chunks of a long row are spread over blockIdx.y
// (a row's cost grows with the square of its length)
__global__ void __launch_bounds__(512)
k_row_sort_long(int nb, const int* __restrict__ start, const int* __restrict__ in, int* __restrict__ out) {
  __shared__ int tile[512], rows[512], nrow;
  const int tid = threadIdx.x, b = blockIdx.x * 512 + tid;
  if (tid == 0) nrow = 0;
  __syncthreads();
  if (b < nb && start[b + 1] - start[b] > ROW_WARP) rows[atomicAdd(&nrow, 1)] = b;
  __syncthreads();
  for (int q = 0; q < nrow; q++) {
    const int s = start[rows[q]], n = start[rows[q] + 1] - s;
    for (int k0 = 512 * blockIdx.y; k0 < n; k0 += 512 * gridDim.y) {
      const int k = k0 + tid;
      const int v = k < n ? in[s + k] : 0;
      int r = 0;
      for (int j0 = 0; j0 < n; j0 += 512) {
        __syncthreads();
        if (j0 + tid < n) tile[tid] = in[s + j0 + tid];
        __syncthreads();
        const int m = min(512, n - j0);
        for (int j = 0; j < m; j++) r += tile[j] < v || (tile[j] == v && j0 + j < k);
      }
      if (k < n) out[s + r] = v;
    }
  }
}

// --------------------------------------------------------------------------
// host orchestration
// --------------------------------------------------------------------------
template <class T>
static std::vector<T> to_host(const T* d, size_t n, cudaStream_t st) {
  std::vector<T> h(n);
  if (n) EFMM_CUDA_TRY(cudaMemcpyAsync(h.data(), d, n * sizeof(T), cudaMemcpyDeviceToHost, st));
  EFMM_CUDA_TRY(cudaStreamSynchronize(st));
  return h;
}

static void exclusive_scan(cudaStream_t st, const int* in, int* out, int n, DevBuf<char>& tmp) {
  if (n <= 0) return;
  const size_t bytes = scan_scratch_bytes(n);
  if (bytes > tmp.size()) tmp.resize(bytes);
  exclusive_scan_dev(st, in, out, n, tmp.get());
}

// stable sort of (key, value) pairs whose keys are below 2^bits (sort.cu)
static void sort_pairs(cudaStream_t st, const unsigned long long* kin, unsigned long long* kout, const int* vin,
                       int* vout, int n, const std::vector<int>& shifts, DevBuf<char>& tmp) {
  if (n <= 0) return;
  const size_t bytes = radix_scratch_bytes(n);
  if (bytes > tmp.size()) tmp.resize(bytes);
  radix_sort_pairs(st, kin, kout, vin, vout, n, shifts.data(), (int)shifts.size(), tmp.get());
}

// The reference's root (src/d3tstrcr.f:31 d3tstrcr, src/d3tstrcr_mindlin.f:
// 1380): centre and side of the bounding cube of sources and targets; the
// Mindlin variant centres it on z = 0 with side >= 2 max|z|.
static void bounding_root(cudaStream_t st, int n, const double* d_src, int nt, const double* d_tgt, int mindlin,
                          DevBuf<double>& bb, double* c0, double& size) {
  bb.resize(6);
  unsigned long long init[6];
  for (int c = 0; c < 3; c++) {
    init[c] = ~0ull;
    init[3 + c] = 0ull;
  }
  EFMM_CUDA_TRY(cudaMemcpyAsync(bb.get(), init, sizeof(init), cudaMemcpyHostToDevice, st));
  k_bbox<<<148, 256, 0, st>>>(n, d_src, bb.get()); count_launch();
  if (nt > 0) { k_bbox<<<148, 256, 0, st>>>(nt, d_tgt, bb.get()); count_launch(); }
  std::vector<unsigned long long> hb = to_host((unsigned long long*)bb.get(), 6, st);
  double mn[3], mx[3];
  for (int c = 0; c < 3; c++) {
    auto dec = [](unsigned long long b) {
      unsigned long long r = (b & 0x8000000000000000ull) ? (b & 0x7fffffffffffffffull) : ~b;
      double v;
      memcpy(&v, &r, 8);
      return v;
    };
    mn[c] = dec(hb[c]);
    mx[c] = dec(hb[3 + c]);
  }
  size = mx[0] - mn[0];
  const double sy = mx[1] - mn[1], sz = mx[2] - mn[2];
  if (sy > size) size = sy;
  if (sz > size) size = sz;
  for (int c = 0; c < 3; c++) c0[c] = (mn[c] + mx[c]) / 2;
  if (mindlin) {
    const double distz = fabs(mn[2]) > fabs(mx[2]) ? fabs(mn[2]) : fabs(mx[2]);
    c0[2] = 0.0;
    if (2 * distz > size) size = 2 * distz;
  }
}

int build_tree(cudaStream_t st, int n, const double* d_src, int nt, const double* d_tgt, int nbox,
               int mindlin, Tree& tr, const double* forest) {
  if (n < 1) return IER_BADARG;
  TreeScratch& S = tr.scr;
  DevBuf<char>& tmp = S.tmp;
  tr.n = n;
  tr.nt = nt;
  tr.flev = -1;
  double size = 0.0;
  if (forest) {
    if (!(forest[3] > 0.0) || forest[4] < 1.0 || forest[4] > 15.0) return IER_BADARG;
    for (int c = 0; c < 3; c++) tr.c0[c] = forest[c];
    size = forest[3];
    tr.flev = (int)forest[4];
  }
  // ---- root: the given cube of a forest, else the points' bounding cube
  if (!forest) bounding_root(st, n, d_src, nt, d_tgt, mindlin, S.bb, tr.c0, size);
  tr.size = size;

  // ---- boxes (grown per level)
  size_t cap = 1024;
  auto growall = [&](size_t m) {
    tr.level.grow(m, st);
    tr.ijk.grow(3 * m, st);
    tr.parent.grow(m, st);
    tr.kids.grow(8 * m, st);
    tr.nkids.grow(m, st);
    tr.sstart.grow(m, st);
    tr.scount.grow(m, st);
    tr.tstart.grow(m, st);
    tr.tcount.grow(m, st);
  };
  growall(cap);
  // ---- points
  tr.iz.resize(n);
  tr.izt.resize(nt);
  DevBuf<int>&pbs = S.pbs, &pbt = S.pbt, &izs2 = S.izs2, &izt2 = S.izt2, &split = S.split, &cs = S.cs,
              &ct = S.ct, &nch = S.nch, &off = S.off;
  DevBuf<unsigned long long>&ks = S.ks, &ks2 = S.ks2;
  DevBuf<unsigned char>&ds = S.ds, &dt = S.dt;
  pbs.resize(n);
  pbt.resize(nt);
  izs2.resize(n);
  izt2.resize(nt);
  ds.resize(n);
  dt.resize(nt);
  S.info.resize(8);
  const int nmax = std::max(n, nt);
  k_root<<<(nmax + 255) / 256, 256, 0, st>>>(n, nt, tr.level.get(), tr.ijk.get(), tr.parent.get(), tr.kids.get(),
                                             tr.nkids.get(), tr.sstart.get(), tr.scount.get(), tr.tstart.get(),
                                             tr.tcount.get(), tr.iz.get(), tr.izt.get(), pbs.get(), pbt.get());
  count_launch();
  int lo = 0, hi = 1, nlev = 0;
  tr.laddr.clear();
  tr.laddr.push_back({0, 1});
  // The reference allows 198 levels but its integer box indices overflow past
  // ~30; only more than nbox coincident points get that deep, so subdivision
  // stops at MAX_LEVELS (boxes at that level stay leaves).
  const int MAX_LEVELS = 50;
  for (int lev = 0; lev < MAX_LEVELS; lev++) {
    int nl = hi - lo;
    split.resize(nl);
    cs.resize(8 * (size_t)nl);
    ct.resize(8 * (size_t)nl);
    nch.resize(nl);
    off.resize(nl);
    k_split<<<(nl + 255) / 256, 256, 0, st>>>(lo, hi, nbox, lev < tr.flev ? 1 : 0, tr.scount.get(),
                                              tr.tcount.get(), split.get(), cs.get(), ct.get()); count_launch();
    double side = size / (double)(1ull << lev);
    k_digits<<<(n + 255) / 256, 256, 0, st>>>(n, d_src, tr.iz.get(), pbs.get(), tr.level.get(), lev, lo,
                                              split.get(), tr.ijk.get(), tr.c0[0], tr.c0[1], tr.c0[2], size, side,
                                              ds.get(), cs.get()); count_launch();
    if (nt > 0)
      k_digits<<<(nt + 255) / 256, 256, 0, st>>>(nt, d_tgt, tr.izt.get(), pbt.get(), tr.level.get(), lev,
                                                 lo, split.get(), tr.ijk.get(), tr.c0[0], tr.c0[1], tr.c0[2], size,
                                                 side, dt.get(), ct.get()); count_launch();
    k_nchild<<<(nl + 255) / 256, 256, 0, st>>>(nl, split.get(), cs.get(), ct.get(), nch.get()); count_launch();
    exclusive_scan(st, nch.get(), off.get(), nl, tmp);
    k_level_info<<<1, 1024, 0, st>>>(nl, nch.get(), off.get(), split.get(), tr.scount.get() + lo,
                                     tr.tcount.get() + lo, S.info.get()); count_launch();
    int info[2];
    EFMM_CUDA_TRY(cudaMemcpyAsync(info, S.info.get(), sizeof(info), cudaMemcpyDeviceToHost, st));
    EFMM_CUDA_TRY(cudaStreamSynchronize(st));
    const int nnew = info[0];
    if (nnew == 0) break;
    growall(hi + nnew);
    // stable partition of the points by (box start, digit)
    const bool radix = info[1] > PART_MAX;
    int bits = 3;
    while ((1ll << (bits - 3)) <= (long long)nmax && bits < 64) bits++;
    auto reorder = [&](int m, DevBuf<int>& perm, DevBuf<int>& perm2, DevBuf<int>& pb, const DevBuf<int>& start,
                       const DevBuf<int>& count, const DevBuf<unsigned char>& dg, const DevBuf<int>& cnt) {
      if (m <= 0) return;
      if (radix) {
        ks.resize(m);
        ks2.resize(m);
        k_digit_keys<<<(m + 255) / 256, 256, 0, st>>>(m, pb.get(), start.get(), dg.get(), ks.get()); count_launch();
        std::vector<int> shifts;
        for (int b = 0; b < bits; b += 8) shifts.push_back(b);
        sort_pairs(st, ks.get(), ks2.get(), perm.get(), perm2.get(), m, shifts, tmp);
      } else {
        EFMM_CUDA_TRY(cudaMemcpyAsync(perm2.get(), perm.get(), 4 * (size_t)m, cudaMemcpyDeviceToDevice, st));
        const int per = m / nl, threads = per > 512 ? 1024 : (per > 96 ? 256 : 64);
        k_partition<<<nl, threads, 0, st>>>(lo, hi, split.get(), start.get(), count.get(), cnt.get(), cs.get(),
                                            ct.get(), off.get(), dg.get(), perm.get(), perm2.get(), pb.get());
        count_launch();
      }
      perm.swap(perm2);
    };
    reorder(n, tr.iz, izs2, pbs, tr.sstart, tr.scount, ds, cs);
    reorder(nt, tr.izt, izt2, pbt, tr.tstart, tr.tcount, dt, ct);
    k_children<<<(nl + 127) / 128, 128, 0, st>>>(lo, hi, lev, split.get(), cs.get(), ct.get(), off.get(),
                                                 tr.level.get(), tr.ijk.get(), tr.parent.get(), tr.kids.get(),
                                                 tr.nkids.get(), tr.sstart.get(), tr.scount.get(),
                                                 tr.tstart.get(), tr.tcount.get()); count_launch();
    int nh = hi + nnew;
    if (radix) {
      k_pbox<<<(nnew * 32 + 255) / 256, 256, 0, st>>>(hi, nh, tr.sstart.get(), tr.scount.get(), pbs.get()); count_launch();
      if (nt > 0)
        k_pbox<<<(nnew * 32 + 255) / 256, 256, 0, st>>>(hi, nh, tr.tstart.get(), tr.tcount.get(), pbt.get()); count_launch();
    }
    tr.laddr.push_back({hi, nnew});
    lo = hi;
    hi = nh;
    nlev = lev + 1;
  }
  tr.nboxes = hi;
  tr.nlev = nlev;
  return IER_OK;
}

int build_lists(cudaStream_t st, Tree& tr) {
  TreeScratch& S = tr.scr;
  DevBuf<char>& tmp = S.tmp;
  const int nb = tr.nboxes;
  tr.coll.resize(27 * (size_t)nb);
  tr.ncoll.resize(nb);
  tr.ncoll.zero(st);
  // counts of the rows of lists 2, 1, 3, 4 (one more: the scans' totals)
  DevBuf<int>& cnt = S.cnt;
  cnt.resize(4 * (size_t)(nb + 1));
  cnt.zero(st);
  int *c2 = cnt.get(), *c1 = c2 + nb + 1, *c3 = c1 + nb + 1, *c4 = c3 + nb + 1;
  TreeDev T = tr.dev();
  // list 5 and the size of list 2, level by level (colleagues of the parent must exist)
  for (int lev = 1; lev <= tr.nlev; lev++) {
    const int lo = tr.laddr[lev].first, n = tr.laddr[lev].second;
    k_list5<<<(n + 3) / 4, 128, 0, st>>>(T, lo, lo + n, c2); count_launch();
  }
  k_list13<false><<<(nb + 3) / 4, 128, 0, st>>>(T, nb, c1, c3, c4, nullptr, nullptr, nullptr); count_launch();
  for (DevBuf<int>* b : {&tr.l2_start, &tr.l1_start, &tr.l3_start, &tr.l4_start}) b->resize(nb + 1);
  exclusive_scan(st, c2, tr.l2_start.get(), nb + 1, tmp);
  exclusive_scan(st, c1, tr.l1_start.get(), nb + 1, tmp);
  exclusive_scan(st, c3, tr.l3_start.get(), nb + 1, tmp);
  exclusive_scan(st, c4, tr.l4_start.get(), nb + 1, tmp);
  S.info.resize(8);
  k_list_info<<<1, 1024, 0, st>>>(nb, c1, c3, c4, tr.l1_start.get(), tr.l3_start.get(), tr.l4_start.get(),
                                  tr.l2_start.get(), S.info.get()); count_launch();
  int info[5];
  EFMM_CUDA_TRY(cudaMemcpyAsync(info, S.info.get(), sizeof(info), cudaMemcpyDeviceToHost, st));
  EFMM_CUDA_TRY(cudaStreamSynchronize(st));
  tr.l2_items.resize(info[4]);
  if (nb > 1) { k_list2<<<(nb - 1 + L2_WARPS - 1) / L2_WARPS, L2_WARPS * 32, 0, st>>>(T, nb, tr.l2_start.get(), tr.l2_items.get()); count_launch(); }
  // lists 1, 3 and 4: the rows filled in any order from cursors, then sorted
  DevBuf<int>&u1 = S.u1, &u3 = S.u3, &u4 = S.u4, &cur = S.cur;
  u1.resize(info[0]);
  u3.resize(info[1]);
  u4.resize(info[2]);
  cur.resize(3 * (size_t)(nb + 1));
  int *q1 = cur.get(), *q3 = q1 + nb + 1, *q4 = q3 + nb + 1;
  EFMM_CUDA_TRY(cudaMemcpyAsync(q1, tr.l1_start.get(), 4 * (size_t)nb, cudaMemcpyDeviceToDevice, st));
  EFMM_CUDA_TRY(cudaMemcpyAsync(q3, tr.l3_start.get(), 4 * (size_t)nb, cudaMemcpyDeviceToDevice, st));
  EFMM_CUDA_TRY(cudaMemcpyAsync(q4, tr.l4_start.get(), 4 * (size_t)nb, cudaMemcpyDeviceToDevice, st));
  k_list13<true><<<(nb + 3) / 4, 128, 0, st>>>(T, nb, q1, q3, q4, u1.get(), u3.get(), u4.get()); count_launch();
  auto sort_rows = [&](DevBuf<int>& start, DevBuf<int>& from, DevBuf<int>& items, int tot) {
    items.resize(tot);
    if (tot == 0) return;
    k_row_sort<<<(nb + 3) / 4, 128, 0, st>>>(nb, start.get(), from.get(), items.get()); count_launch();
    if (info[3] > ROW_WARP) { k_row_sort_long<<<dim3((nb + 511) / 512, std::min((info[3] + 511) / 512, 64)), 512, 0, st>>>(nb, start.get(), from.get(), items.get()); count_launch(); }
  };
  sort_rows(tr.l1_start, u1, tr.l1_items, info[0]);
  sort_rows(tr.l3_start, u3, tr.l3_items, info[1]);
  sort_rows(tr.l4_start, u4, tr.l4_items, info[2]);
  EFMM_CUDA_TRY(cudaGetLastError());
  return IER_OK;
}

}  // namespace efmm
