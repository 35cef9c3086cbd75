// rot_mma.cu -- the FP64 translations (M2M, M2L, L2L) in the parity-split
// factored form on the FP64 tensor cores.
//
// A translation by an offset is Rz, Ry, the shift along z, Ry back, Rz back
// (rotations.cu).  Rz mixes only the (re, im) pair of a coefficient; Ry is an
// (n+1)^2 re block and an n^2 im block per degree n, the shift a re and an im
// block of p - m + 1 rows per order m: 43 k multiply-adds per column at p = 26,
// against 79 k for full blocks.  Each block times the columns of a group is a
// small matrix product, done with mma.sync m8n8k4 (FP64 accumulation; the
// FP64 pipe's rate, but one operand load per 16 multiply-adds of a lane
// instead of per one or two, which is what bounds a plain FMA kernel here).
//
// One CTA per 8 NT columns of one group, all five factors in place in shared
// memory: row n^2 + m holds the re part of coefficient (n, m), row n^2 + n + m
// the im part (m >= 1), so every block's rows step by 1 (Ry) or by one degree
// (shift).  Column c of a row is stored at c ^ 4 ((n + m) & 3): the four rows a
// warp reads per k step (consecutive n + m) and the rows it writes fall in
// distinct banks.  A warp owns whole blocks (re or im of one degree or order,
// assigned by size on the host), keeps a block's results in registers until
// all its inputs are read, and takes the operator from L2 in fragment order
// (256 contiguous bytes per 8 x 4 tile, zero padded, one k step ahead).
//
// Columns per CTA: 32 while the rows fit (p <= 29), else 16; fewer where a
// launch's groups are so small that most of a tile would be padding.
//
// What bounds it is the FP64 tensor pipe and, between its bursts, the latency
// of L2: a warp's next block has its first operator fragments loaded during
// the last k step of the block before (across the barriers of the stages
// too), and the sources of four staging steps are in flight together (two
// cost 6 %); without both 29.7 ms instead of 25.5 on the first case below.
// Atomics laid out so that a warp fills whole lines (half as many columns per
// instruction) cost 6 %: the final pass is bound by instructions.
//
// Measured (all M2M + M2L + L2L launches of a pass) against full (re, im)
// blocks on plain FP64 FMAs, 8 columns per CTA (bound by L2 latency): 327,680
// triangles + 250,007 targets at iprec 2 (1.33 M box pairs x 4 columns) 78.5
// -> 25.5 ms; 16 right-hand sides on 9,973 + 2,003 30.6 -> 10.0 ms (8.9e10
// multiply-adds, 0.50 of the measured DGEMM rate, padding to 8 x 4 tiles not
// counted); 20,011 particles 14.5 -> 4.6 ms; 20,480 triangles at iprec 1 3.9
// -> 1.1 ms.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "fmm.h"
#include "rotations.h"

namespace efmm {

// doubles of a packed block of r rows: ceil(r / 8) x ceil(r / 4) tiles of 32
__host__ __device__ constexpr int rm_size(int r) { return ((r + 7) / 8) * ((r + 3) / 4) * 32; }
struct RmPrefix {
  int s[RM_PMAX + 3];  // s[R] = sum of rm_size(1..R)
};
constexpr RmPrefix make_rm_prefix() {
  RmPrefix t{};
  for (int r = 1; r <= RM_PMAX + 2; r++) t.s[r] = t.s[r - 1] + rm_size(r);
  return t;
}
static constexpr RmPrefix h_rm = make_rm_prefix();
__constant__ RmPrefix c_rm = make_rm_prefix();

// Group layout (doubles) at base: Rz [4 (p+1)], Ry, shift, Ry back (each
// rm_stage doubles), Rz back [4 (p+1)].  A stage: the re blocks in order of
// r = 1..p+1 rows, then the im blocks of r = 1..p rows.
__host__ __device__ inline int rm_stage(const RmPrefix& t, int p) { return t.s[p + 1] + t.s[p]; }
long long rm_group_size(int p) { return 8LL * (p + 1) + 3LL * rm_stage(h_rm, p); }
long long rm_stage_size(int p) { return rm_stage(h_rm, p); }
long long rm_block_off(int p, int r, int part) { return (part ? h_rm.s[p + 1] : 0) + h_rm.s[r - 1]; }

// Warp lists: for order p and nw warps, the units (r rows, part) of a stage,
// code r | part << 7, dealt longest first onto the least loaded warp; the
// list of warp w at w * RM_UNITS of the order's table, ended by 0.
void build_rm_sched(int nw, std::vector<unsigned char>& out) {
  out.assign((size_t)(RM_PMAX + 1) * nw * RM_UNITS, 0);
  for (int p = 0; p <= RM_PMAX; p++) {
    std::vector<int> load(nw, 0), cnt(nw, 0);
    for (int r = p + 1; r >= 1; r--)
      for (int part = 0; part < (r <= p ? 2 : 1); part++) {
        int best = -1;
        for (int w = 0; w < nw; w++)
          if (cnt[w] < RM_UNITS - 1 && (best < 0 || load[w] < load[best])) best = w;
        out[((size_t)p * nw + best) * RM_UNITS + cnt[best]++] = (unsigned char)(r | part << 7);
        load[best] += rm_size(r) / 32 + 6;
      }
  }
}

__device__ __forceinline__ void dmma(double* d, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Operator fragments of a block's first k step, for up to RM_MT row tiles
template <int NT>
constexpr int RM_MT = NT == 4 ? 4 : 6;
template <int NT>
__device__ __forceinline__ void rm_first(double (&an)[RM_MT<NT>], const double* __restrict__ A, int mt, int lane) {
#pragma unroll
  for (int a = 0; a < RM_MT<NT>; a++)
    if (a < mt) an[a] = __ldg(A + lane + 32 * a);
}

// One block of r <= 8 MT rows: stage 1 (shift) rows (m + i)^2 + m + part (m +
// i), else rb + i; key of row i: kb + i.  an holds its first fragments and
// leaves with those of the warp's next block (An, mtn row tiles; none: 0).
template <int MT, int NT>
__device__ __forceinline__ void rm_block(double* __restrict__ X, const double* __restrict__ A, int r, bool shift,
                                         int rb, int m, int part, int kb, int lane, double (&an)[RM_MT<NT>],
                                         const double* __restrict__ An, int mtn) {
  constexpr int NC = 8 * NT;
  const int lk = lane & 3, ln = lane >> 2;
  auto row = [&](int i) {
    const int n = m + i;
    return shift ? n * n + m + part * n : rb + i;
  };
  double acc[MT][NT][2];
#pragma unroll
  for (int a = 0; a < MT; a++)
#pragma unroll
    for (int b = 0; b < NT; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
  const int kt = (r + 3) >> 2;
  const double* Al = A + lane;
  const int cx = ln ^ (((kb + lk) & 3) << 2);  // swizzled column of n-tile 0 in this lane's input rows
#pragma unroll 2
  for (int k = 0; k < kt; k++) {
    double ac[MT], b[NT];
#pragma unroll
    for (int a = 0; a < MT; a++) ac[a] = an[a];
    Al += 32 * MT;
    if (k + 1 < kt) {
#pragma unroll
      for (int a = 0; a < MT; a++) an[a] = __ldg(Al + 32 * a);
    } else {
      rm_first<NT>(an, An, mtn, lane);
    }
    // rows past the block's last are met by zero operator columns
    const double* xr = X + (size_t)row(min(4 * k + lk, r - 1)) * NC;
#pragma unroll
    for (int j = 0; j < NT; j++) b[j] = xr[NT == 1 ? (cx & 7) : ((8 * j) ^ cx)];
#pragma unroll
    for (int a = 0; a < MT; a++)
#pragma unroll
      for (int j = 0; j < NT; j++) dmma(acc[a][j], ac[a], b[j]);
  }
  __syncwarp();
#pragma unroll
  for (int a = 0; a < MT; a++) {
    const int i = 8 * a + ln;
    if (i < r) {
      double* xr = X + (size_t)row(i) * NC;
      const int sw = ((kb + i) & 3) << 2;
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const int c = (8 * j + 2 * lk) ^ sw;
        *reinterpret_cast<double2*>(xr + (NT == 1 ? (c & 7) : c)) = make_double2(acc[a][j][0], acc[a][j][1]);
      }
    }
  }
  __syncwarp();
}

template <int NT, int NW>
__global__ void __launch_bounds__(NW * 32, NW == 8 ? 2 : 1)
k_translate_mma(const TransTask* __restrict__ tasks, const TransPair* __restrict__ pairs,
                const RotMOp* __restrict__ ops, const double* __restrict__ pool,
                const unsigned char* __restrict__ sched, int D, int C, const double* __restrict__ src,
                double* __restrict__ dst) {
  constexpr int NC = 8 * NT;
  extern __shared__ __align__(16) unsigned char rm_smem_[];
  const TransTask t = tasks[blockIdx.x];
  const RotMOp op = ops[t.group];
  const int p = op.p, nc = (p + 1) * (p + 2) / 2;
  double* X = reinterpret_cast<double*>(rm_smem_);  // [(p+1)^2][NC]
  double* alpha = X + (size_t)(p + 1) * (p + 1) * NC;
  long long* sb = reinterpret_cast<long long*>(alpha + NC);  // source and destination columns
  long long* db = sb + NC;
  unsigned short* nm = reinterpret_cast<unsigned short*>(db + NC);  // [nc]: n << 8 | m
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < NC) {
    const int col = t.col0 + tid;
    long long b = -1, d = -1;
    double al = 0.0;
    if (col < t.ncols) {
      const TransPair pr = pairs[t.pair0 + col / C];
      b = ((long long)pr.src * C + col % C) * D;
      d = ((long long)pr.dst * C + col % C) * D;
      al = pr.alpha;
    }
    sb[tid] = b;
    db[tid] = d;
    alpha[tid] = al;
  }
  for (int n = warp; n <= p; n += NW)
    for (int m = lane; m <= n; m += 32) nm[n * (n + 1) / 2 + m] = (unsigned short)(n << 8 | m);
  __syncthreads();
  const double* g0 = pool + op.base;
  const int nst = rm_stage(c_rm, p), ncg = (nc + 7) / 8;
  const unsigned char* list = sched + ((size_t)p * NW + warp) * RM_UNITS;
  // operator of unit code x of stage st, and the fragments of the first one
  auto oper = [&](int st, int x) {
    return g0 + 4 * (p + 1) + (size_t)st * nst + ((x >> 7) ? c_rm.s[p + 1] : 0) + c_rm.s[(x & 127) - 1];
  };
  double an[RM_MT<NT>];
  if (list[0]) rm_first<NT>(an, oper(0, list[0]), ((list[0] & 127) + 7) >> 3, lane);
  // sources with Rz: lane (coefficient of 8, column of 4), both parts, the
  // loads of RM_U steps in flight together
  constexpr int RM_U = 4;
  for (int q0 = warp; q0 < ncg * (NC / 4); q0 += RM_U * NW) {
    double2 v[RM_U], R0[RM_U], R1[RM_U];
    int at[RM_U];  // n << 16 | m << 8 | column, -1: none
#pragma unroll
    for (int u = 0; u < RM_U; u++) {
      const int q = q0 + u * NW, c = (q % ncg) * 8 + (lane & 7), j = (q / ncg) * 4 + (lane >> 3);
      at[u] = -1;
      if (q >= ncg * (NC / 4) || c >= nc) continue;
      at[u] = nm[c] << 8 | j;
      const int m = nm[c] & 255;
      const long long b = sb[j];
      v[u] = b >= 0 ? __ldg(reinterpret_cast<const double2*>(src + b) + c) : make_double2(0.0, 0.0);
      R0[u] = __ldg(reinterpret_cast<const double2*>(g0 + 4 * m));
      R1[u] = __ldg(reinterpret_cast<const double2*>(g0 + 4 * m + 2));
    }
#pragma unroll
    for (int u = 0; u < RM_U; u++) {
      if (at[u] < 0) continue;
      const int n = at[u] >> 16, m = at[u] >> 8 & 255, j = at[u] & 255;
      const int cs = (j ^ (((n + m) & 3) << 2)) & (NC - 1);
      X[(size_t)(n * n + m) * NC + cs] = R0[u].x * v[u].x + R0[u].y * v[u].y;
      if (m > 0) X[(size_t)(n * n + n + m) * NC + cs] = R1[u].x * v[u].x + R1[u].y * v[u].y;
    }
  }
#pragma unroll 1
  for (int st = 0; st < 3; st++) {
    __syncthreads();
#pragma unroll 1
    for (int u = 0; list[u]; u++) {
      const int r = list[u] & 127, part = list[u] >> 7;
      const double* A = oper(st, list[u]);
      // the warp's next block, of this stage or the first of the next
      const int xn = list[u + 1] ? list[u + 1] : (st < 2 ? list[0] : 0), mtn = ((xn & 127) + 7) >> 3;
      const double* An = xn ? oper(list[u + 1] ? st : st + 1, xn) : A;
      const bool shift = st == 1;
      // Ry: degree n = r - 1 (re) or r (im, orders 1..n); shift: order m = p + 1 - r
      const int n = r - 1 + part, m = p + 1 - r;
      const int rb = n * n + (part ? n + 1 : 0), kb = shift ? 2 * m : n + part;
      switch ((r + 7) >> 3) {
        case 1: rm_block<1, NT>(X, A, r, shift, rb, m, part, kb, lane, an, An, mtn); break;
        case 2: rm_block<2, NT>(X, A, r, shift, rb, m, part, kb, lane, an, An, mtn); break;
        case 3: rm_block<3, NT>(X, A, r, shift, rb, m, part, kb, lane, an, An, mtn); break;
        case 4: rm_block<4, NT>(X, A, r, shift, rb, m, part, kb, lane, an, An, mtn); break;
        case 5: if constexpr (NT < 4) rm_block<5, NT>(X, A, r, shift, rb, m, part, kb, lane, an, An, mtn); break;
        default: if constexpr (NT < 4) rm_block<6, NT>(X, A, r, shift, rb, m, part, kb, lane, an, An, mtn); break;
      }
    }
  }
  __syncthreads();
  // Rz back, pair factor, into the destinations
  const double* rzb = g0 + 4 * (p + 1) + 3 * (size_t)nst;
  for (int q = warp; q < ncg * (NC / 4); q += NW) {
    const int c = (q % ncg) * 8 + (lane & 7), j = (q / ncg) * 4 + (lane >> 3);
    if (c >= nc || db[j] < 0) continue;
    const int n = nm[c] >> 8, m = nm[c] & 255;
    const int cs = (j ^ (((n + m) & 3) << 2)) & (NC - 1);
    const double re = X[(size_t)(n * n + m) * NC + cs], im = m > 0 ? X[(size_t)(n * n + n + m) * NC + cs] : 0.0;
    const double2 R0 = __ldg(reinterpret_cast<const double2*>(rzb + 4 * m));
    const double2 R1 = __ldg(reinterpret_cast<const double2*>(rzb + 4 * m + 2));
    double* d = dst + db[j] + 2 * c;
    const double al = alpha[j];
    atomicAdd(d, al * (R0.x * re + R0.y * im));
    if (m > 0) atomicAdd(d + 1, al * (R1.x * re + R1.y * im));
  }
}

static size_t rm_smem(int p, int nt) {
  return 8 * nt * (size_t)(8 * (p + 1) * (p + 1) + 24) + 2 * (size_t)((p + 1) * (p + 2) / 2);
}
bool rot_mma_ok(int p) { return p <= RM_PMAX && rm_smem(p, 2) <= 227 * 1024; }

// n-tiles per CTA for groups of order p whose columns average `cols`: 4 while
// the rows fit, less where a half-empty tile would waste more than it shares
int rot_mma_tiles(int p, double cols) {
  int nt = rm_smem(p, 4) <= 227 * 1024 ? 4 : 2;
  while (nt > 1 && cols < 6.0 * nt) nt /= 2;
  return nt;
}

// 16 warps where one CTA fills an SM's shared memory, two CTAs of 8 below
bool rot_mma_big(int p, int nt) { return rm_smem(p, nt) > 110 * 1024; }

void launch_translate_mma(cudaStream_t st, int ntask, const TransTask* tasks, const TransPair* pairs,
                          const RotMOp* ops, const double* pool, const unsigned char* sched16,
                          const unsigned char* sched8, int D, int C, int pmax, int nt, const double* src,
                          double* dst) {
  if (ntask <= 0) return;
  const size_t smem = rm_smem(pmax, nt);
  auto go = [&](auto kern, int nw, const unsigned char* sched) {
    EFMM_CUDA_TRY(smem_raise(kern, (int)smem));
    kern<<<ntask, nw * 32, smem, st>>>(tasks, pairs, ops, pool, sched, D, C, src, dst);
    count_launch();
  };
  const bool big = rot_mma_big(pmax, nt);
  if (nt == 4) {
    if (big) go(k_translate_mma<4, 16>, 16, sched16);
    else go(k_translate_mma<4, 8>, 8, sched8);
  } else if (nt == 2) {
    if (big) go(k_translate_mma<2, 16>, 16, sched16);
    else go(k_translate_mma<2, 8>, 8, sched8);
  } else {
    if (big) go(k_translate_mma<1, 16>, 16, sched16);
    else go(k_translate_mma<1, 8>, 8, sched8);
  }
  EFMM_CUDA_TRY(cudaGetLastError());
}

}  // namespace efmm
