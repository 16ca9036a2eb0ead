// The multigrid V-cycle on the coarse levels as one dense matrix.
//
// On a level l of few active rows the V-cycle from a zero start (TMultiGrid3D::Cycle,
// src/FE/MultiGrid3D.C:423-669: damped Jacobi sweeps, defect, restriction, the cycle below,
// prolongation, damped Jacobi sweeps, exact solve at the bottom) is a linear map of the level's
// right-hand side, x = B f with B an n_l x n_l matrix that depends on the assembled levels
// 0..l, the transfers and the cycle's parameters only.  B is formed once per assembly, in FP64,
// by running that cycle on the unit vectors (vcycle_matrix_kernel: every CTA takes a few columns
// through all levels with its vectors in shared memory), and each cycle then applies it with one
// dense product (dense_cycle_kernel) where it launched 3 + pre + post kernels per level.
// The coarse levels are bound by launch and load latency, not by bytes: a 961 x 961 FP64 matrix
// (7.4 MB) is read from L2 by all SMs at once, its first entries before the predecessor of the
// product has finished.  Measured per solve, the launched levels against the dense product
// (formation included): CD2D Q1 64^2 (28 launches of each FGMRES iteration saved) 1415 -> 959 us,
// CD2D Q2 192^2 4280 -> 3810, CD3D Q2 32^3 mixed 3734 -> 3630.  Mixed solves that may end
// unconverged keep the launched FP32 levels (sums_keep_order in solve.cu).
#pragma once

#include "internal.h"

// Largest active block that becomes a dense matrix: formation takes 20 us at 121 rows, 50-90 us at
// 529-961 and grows with rows times nonzeros (1,331 rows of 12^3 trilinear cells would need two
// waves of CTAs), the product 2 us at 121 rows and 4.5 us at 961; a launched level costs about
// 7 x 1.5-2.5 us per cycle.
constexpr int kDenseRows = 1024;
constexpr int kVMaxLevels = 12;
constexpr int kVThreads = 1024;
constexpr size_t kVSharedBytes = 220 * 1024; // of a CTA, at most (vcycle_layout); below kMaxDynShared

struct VLevel
{
  int na = 0;
  const int *rp = nullptr, *kc = nullptr, *dirst = nullptr;
  const double *a = nullptr, *diag = nullptr;
  // transfers between this level (fine) and the one below: P by rows of this level, R = P^T by
  // rows of the level below
  const int *prp = nullptr, *pkc = nullptr, *rrp = nullptr, *rkc = nullptr;
  const double *pv = nullptr, *rv = nullptr;
  int row = 1, prow = 1, rrow = 1; // mean entries per row of A, P and R
  // offsets (per column) of the level's two iterates and its right-hand side in shared memory
  int buf[2] = {0, 0}, f = 0;
  int winv = 0; // offset of omega / diagonal, behind the columns
};

struct VCycleArgs
{
  int top = 0, pre = 0, post = 0;
  int cols = 0; // doubles of shared memory per column
  double omega = 0, damp = 1;
  VLevel lev[kVMaxLevels];
  const double *cinv = nullptr; // inverse of the coarsest active block
  double *B = nullptr;          // n_top x n_top, row-major
};

// shared-memory layout: per column two iterates per level and the right-hand sides below the top
// (the top's are unit vectors), then omega / diagonal of every level and two flags per row of the
// top; returns the bytes of C columns
inline size_t vcycle_layout(VCycleArgs &v, int C)
{
  int o = 0, w = 0;
  for (int l = 0; l <= v.top; l++)
  {
    VLevel &L = v.lev[l];
    for (int &b : L.buf) { b = o; o += L.na; }
    L.f = o;
    if (l < v.top) o += L.na;
    L.winv = w;
    if (l > 0) w += L.na;
  }
  v.cols = o;
  return sizeof(double) * ((size_t)o * C + w) + 2 * (size_t)v.lev[v.top].na;
}

// what a pass over the rows of a level computes from s = (row of A, R or P) x
enum { V_SWEEP = 0, V_DEFECT = 1, V_RESTRICT = 2, V_PROLONG = 3 };

// operands of a pass: a CSR matrix (row r: entries [rp[r], re[r])), the vectors' leading
// dimensions (x: ldx, the others: rows) and, on the top level, unit vectors for f
struct VPass
{
  int rows, cols, unit; // unit: first column of this CTA's unit right-hand sides, -1: f is stored
  const int *rp, *re, *kc;
  const double *a, *winv;
  const double *x, *f;
  double *y;
  // rows of x (in) and y (out) that can be nonzero: the sweeps that start from unit vectors only
  // reach a few rings of rows around them (null: all)
  const unsigned char *nz;
  unsigned char *nz_out;
  double scale; // the damping factor (prolongation); winv: omega / diagonal (sweep)
};

// One pass for the CTA's C columns, TPR lanes per row: kVBatch entries of a lane are loaded at
// once, entries with a column at or beyond p.cols (Dirichlet columns, which carry zeros) are
// skipped.  The lanes of a row add up by passing on half of their columns at each step, so a lane
// ends with C / TPR columns (at least one) and their epilogue.
constexpr int kVBatch = 8;
template <int C, int TPR, int MODE> __device__ __forceinline__ void v_pass_tpr(const VPass &p)
{
  constexpr int OWN = C > TPR ? C / TPR : 1, DUP = TPR > C ? TPR / C : 1; // columns a lane ends with, lanes per column
  const int lane = threadIdx.x & (TPR - 1);
  const int warp_row = (int)(threadIdx.x & ~31) / TPR;
  for (int base = 0; base + warp_row < p.rows; base += kVThreads / TPR)
  {
    const int r = base + (int)threadIdx.x / TPR;
    const bool ok = r < p.rows;
    const int b = ok ? __ldg(p.rp + r) : 0, e = ok ? __ldg(p.re + r) : 0;
    const double w = MODE == V_SWEEP ? (ok ? p.winv[r] : 0.0) : p.scale;
    double s[C];
#pragma unroll
    for (int c = 0; c < C; c++) s[c] = 0.0;
    bool reached = false;
    for (int j0 = b + lane; j0 < e; j0 += TPR * kVBatch)
    {
      int k[kVBatch];
      double v[kVBatch];
#pragma unroll
      for (int u = 0; u < kVBatch; u++)
      {
        k[u] = j0 + u * TPR < e ? __ldg(p.kc + j0 + u * TPR) : p.cols;
        v[u] = j0 + u * TPR < e ? __ldg(p.a + j0 + u * TPR) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kVBatch; u++)
        if (k[u] < p.cols && (!p.nz || p.nz[k[u]]))
        {
          reached = true;
          const double *x = p.x + k[u];
#pragma unroll
          for (int c = 0; c < C; c++) s[c] += v[u] * x[c * p.cols];
        }
    }
    if (p.nz)
    {
      const unsigned m = __ballot_sync(0xffffffffu, reached);
      if (p.nz_out && ok && lane == 0)
        p.nz_out[r] = (m >> (threadIdx.x & 31 & ~(TPR - 1)) & (TPR == 32 ? 0xffffffffu : (1u << (TPR & 31)) - 1)) != 0;
    }
    int c0 = 0, cnt = C;
#pragma unroll
    for (int o = TPR >> 1; o > 0; o >>= 1)
    {
      if (cnt > 1)
      {
        const int half = cnt >> 1;
        const bool hi = lane & o;
#pragma unroll
        for (int c = 0; c < C / 2; c++)
          if (c < half)
          {
            const double keep = hi ? s[c + half] : s[c], give = hi ? s[c] : s[c + half];
            s[c] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        c0 += hi ? half : 0;
        cnt = half;
      }
      else
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
    }
    if (!ok || (DUP > 1 && (lane & (DUP - 1)))) continue;
#pragma unroll
    for (int c = 0; c < OWN; c++)
    {
      const int i = (c0 + c) * p.rows + r;
      if (MODE == V_RESTRICT)
        p.y[i] = s[c];
      else if (MODE == V_PROLONG)
        p.y[i] += w * s[c];
      else
      {
        const double t = (p.unit < 0 ? p.f[i] : r == p.unit + c0 + c ? 1.0 : 0.0) - s[c];
        p.y[i] = MODE == V_DEFECT ? t : p.x[i] + w * t;
      }
    }
  }
  __syncthreads();
}

// lanes per row: about kVBatch entries a lane, more where the level has too few rows to occupy
// the CTA
template <int C, int MODE> __device__ __forceinline__ void v_pass(const VPass &p, int entries)
{
  int t = 1;
  while (t < 32 && (p.rows * t * 2 <= kVThreads || t * kVBatch < entries)) t *= 2;
  if (t <= 2) v_pass_tpr<C, 2, MODE>(p);
  else if (t == 4) v_pass_tpr<C, 4, MODE>(p);
  else if (t <= 16) v_pass_tpr<C, 16, MODE>(p);
  else v_pass_tpr<C, 32, MODE>(p);
}

// One CTA forms C columns of B, its vectors in shared memory, column-major.  Dirichlet rows and
// columns carry zeros throughout a coarse cycle and are skipped.  (8 columns at 1,024 threads leave 64
// registers a thread: 52 bytes of spill stores, 128 of loads.)
template <int C>
__global__ void __launch_bounds__(kVThreads, 1) vcycle_matrix_kernel(const __grid_constant__ VCycleArgs v)
{
  CD_PDL_ENTRY();
  extern __shared__ double vsm[];
  const int tid = threadIdx.x, col0 = blockIdx.x * C, top = v.top;
  // iterate `q` and right-hand side of level l; the sweeps alternate between the two iterates
  auto iter = [&](int l, int q) { return vsm + (size_t)v.lev[l].buf[q] * C; };
  auto frhs = [&](int l) { return vsm + (size_t)v.lev[l].f * C; };
  auto winv = [&](int l) { return vsm + (size_t)v.cols * C + v.lev[l].winv; };
  for (int l = 1; l <= top; l++)
    for (int r = tid; r < v.lev[l].na; r += kVThreads) winv(l)[r] = v.omega / __ldg(v.lev[l].diag + r);
  __syncthreads();
  const int after_pre = v.pre > 1 ? (v.pre - 1) & 1 : 0, after_post = (after_pre + v.post) & 1;
  auto matrix = [&](int l, int src) {
    const VLevel &L = v.lev[l];
    VPass p;
    p.rows = p.cols = L.na;
    p.unit = l == top ? col0 : -1;
    p.rp = L.rp;
    p.re = L.dirst;
    p.kc = L.kc;
    p.a = L.a;
    p.winv = winv(l);
    p.x = iter(l, src);
    p.y = iter(l, 1 - src);
    p.f = frhs(l);
    p.nz = nullptr;
    p.nz_out = nullptr;
    p.scale = v.damp;
    return p;
  };
  unsigned char *nz[2]; // reached rows of the top level's two iterates
  nz[0] = (unsigned char *)(winv(top) + v.lev[top].na);
  nz[1] = nz[0] + v.lev[top].na;
  for (int l = top; l > 0; l--)
  {
    const VLevel &L = v.lev[l];
    const int na = L.na;
    const bool unit = l == top;
    // the first sweep from zero is omega f / d
    double *x0 = iter(l, 0);
    const double *f = frhs(l);
    for (int r = tid; r < na; r += kVThreads)
    {
      const double w = v.pre > 0 ? winv(l)[r] : 0.0;
      if (unit) nz[0][r] = r >= col0 && r < col0 + C;
#pragma unroll
      for (int c = 0; c < C; c++) x0[c * na + r] = unit ? (r == col0 + c ? w : 0.0) : w * f[c * na + r];
    }
    __syncthreads();
    for (int k = 1; k < v.pre; k++)
    {
      VPass p = matrix(l, (k - 1) & 1);
      if (unit) p.nz = nz[(k - 1) & 1], p.nz_out = nz[k & 1];
      v_pass<C, V_SWEEP>(p, L.row);
    }
    VPass p = matrix(l, after_pre);
    if (unit) p.nz = nz[after_pre], p.nz_out = nz[1 - after_pre];
    v_pass<C, V_DEFECT>(p, L.row);
    // right-hand side below: R times the defect
    p = matrix(l, 1 - after_pre);
    if (unit) p.nz = nz[1 - after_pre];
    p.rows = v.lev[l - 1].na;
    p.rp = L.rrp;
    p.re = L.rrp + 1;
    p.kc = L.rkc;
    p.a = L.rv;
    p.y = frhs(l - 1);
    v_pass<C, V_RESTRICT>(p, L.rrow);
  }
  {
    // the exact solve at the bottom
    const int n0 = v.lev[0].na;
    const double *f = frhs(0);
    double *x = iter(0, after_post);
    for (int i = tid; i < n0 * C; i += kVThreads)
    {
      const int c = i / n0, r = i - c * n0;
      double s = 0.0;
#pragma unroll 8
      for (int j = 0; j < n0; j++) s += __ldg(v.cinv + (size_t)r * n0 + j) * f[c * n0 + j];
      x[i] = s;
    }
    __syncthreads();
  }
  for (int l = 1; l <= top; l++)
  {
    const VLevel &L = v.lev[l];
    VPass p = matrix(l, after_pre);
    p.cols = v.lev[l - 1].na;
    p.rp = L.prp;
    p.re = L.prp + 1;
    p.kc = L.pkc;
    p.a = L.pv;
    p.x = iter(l - 1, after_post);
    p.y = iter(l, after_pre);
    v_pass<C, V_PROLONG>(p, L.prow);
    for (int k = 0; k < v.post; k++) v_pass<C, V_SWEEP>(matrix(l, (after_pre + k) & 1), L.row);
  }
  const double *x = iter(top, after_post);
  const int na = v.lev[top].na;
  for (int i = tid; i < na * C; i += kVThreads)
  {
    const int r = i / C, c = i - r * C;
    if (col0 + c < na) v.B[(size_t)r * na + col0 + c] = x[c * na + r];
  }
}

// sol = B f on the active rows, one warp per row; the first kDensePre entries of a lane are
// loaded before the wait (no kernel of a cycle writes B)
constexpr int kDensePre = 16;
template <typename T>
__global__ void __launch_bounds__(256) dense_cycle_kernel(int na, const double *__restrict__ B,
                                                          const T *__restrict__ f, T *__restrict__ sol, int pre)
{
  const int lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (!pre) CD_PDL_ENTRY();
  const double *row = B + (size_t)(r < na ? r : 0) * na;
  double b[kDensePre];
#pragma unroll
  for (int u = 0; u < kDensePre; u++) b[u] = lane + 32 * u < na ? __ldg(row + lane + 32 * u) : 0.0;
  if (pre) CD_PDL_ENTRY();
  if (r >= na) return;
  double s = 0.0;
#pragma unroll
  for (int u = 0; u < kDensePre; u++)
    if (lane + 32 * u < na) s += b[u] * (double)f[lane + 32 * u];
#pragma unroll 8
  for (int j = lane + 32 * kDensePre; j < na; j += 32) s += __ldg(row + j) * (double)f[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) sol[r] = (T)s;
}
