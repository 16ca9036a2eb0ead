// Inverse of the coarsest level's active block, at most 32 rows, by one warp.
//
// In-place Gauss-Jordan with partial pivoting is a chain of n steps of seven phases; with a block
// per matrix every phase ended in a block barrier (2.3 us a step: 17 us for 9 rows, 63 us for 27).
// Here lane j owns column j of the matrix in shared memory, read straight from the CSR entries,
// and the phases are separated by warp synchronisation.  Every element goes through the same
// operations in the same order as in the block form (gj_invert_kernel), which keeps the larger
// blocks, so the inverse is the same to the last bit.  9 rows: 17.4 ->
// 9.6 us with the copy to a dense block and the flag's fill gone; where it stands in a chain: CD2D Q2
// 192^2 (25 rows) 3,228 -> 3,175 us a solve, time step 128^2 Q2 (9 rows) 1,030 -> 1,012; 27 rows
// beside the assembly of a 32^3 level, where one warp gets little of a busy SM: no change.
#pragma once

#include "internal.h"

constexpr int kGjWarpRows = 32;

static __global__ void __launch_bounds__(32) gj_warp_kernel(int n, const int *__restrict__ rp,
                                                            const int *__restrict__ dirst, const int *__restrict__ kc,
                                                            const double *__restrict__ a, double *__restrict__ inv,
                                                            int *__restrict__ flag)
{
  CD_PDL_ENTRY();
  constexpr int LD = kGjWarpRows + 1, U = 8; // LD: rows and columns without bank conflicts
  __shared__ double S[kGjWarpRows * LD];
  __shared__ int piv[kGjWarpRows];
  const int lane = threadIdx.x;
  const bool col = lane < n;
  for (int i = 0; i < n; i++) S[i * LD + lane] = 0.0;
  __syncwarp();
  // a row's active entries [rp, dirst) are at most n; U rows at a time, so that their loads overlap
  const int rb = col ? rp[lane] : 0, re = col ? dirst[lane] : 0;
  for (int i0 = 0; i0 < n; i0 += U)
  {
    int c[U];
    double v[U];
#pragma unroll
    for (int u = 0; u < U; u++)
    {
      const int b = __shfl_sync(0xffffffffu, rb, (i0 + u) & 31), e = __shfl_sync(0xffffffffu, re, (i0 + u) & 31);
      const bool in = i0 + u < n && b + lane < e;
      c[u] = in ? kc[b + lane] : n;
      v[u] = in ? a[b + lane] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (c[u] < n) S[(i0 + u) * LD + c[u]] = v[u];
  }
  __syncwarp();
  bool singular = false;
  for (int k = 0; k < n; k++)
  {
    // largest magnitude of column k in rows k..n-1, lowest row on ties: magnitudes order like
    // their bits, so two reductions of 32-bit words and a ballot find it
    const double m = lane >= k && col ? fabs(S[lane * LD + k]) : 0.0;
    const bool in = lane >= k && col && m == m;
    const unsigned hi = in ? (unsigned)__double2hiint(m) : 0u, mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = in && hi == mh ? (unsigned)__double2loint(m) : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
    const unsigned best = __ballot_sync(0xffffffffu, in && hi == mh && lo == ml);
    const int p = best ? __ffs(best) - 1 : n;
    singular = singular || !(mh | ml);
    if (lane == 0) piv[k] = p;
    if (p >= n) continue; // no comparable entry in the column
    double akj = col ? S[p * LD + lane] : 0.0;
    const double pivot = S[p * LD + k];
    __syncwarp();
    if (p != k && col) S[p * LD + lane] = S[k * LD + lane];
    akj = (lane == k ? 1.0 : akj) / pivot;
    if (col) S[k * LD + lane] = akj;
    __syncwarp();
    const double akk = S[k * LD + k];
    if (col && lane != k)
      for (int i0 = 0; i0 < n; i0 += U) // (rows beyond n, below kGjWarpRows, are read and not used)
      {
        double f[U], t[U];
#pragma unroll
        for (int u = 0; u < U; u++)
        {
          f[u] = S[(i0 + u) * LD + k];
          t[u] = S[(i0 + u) * LD + lane];
        }
#pragma unroll
        for (int u = 0; u < U; u++)
          if (i0 + u < n && i0 + u != k && f[u] != 0.0) S[(i0 + u) * LD + lane] = t[u] - f[u] * akj;
      }
    __syncwarp();
    if (col && lane != k) S[lane * LD + k] = -S[lane * LD + k] * akk;
    __syncwarp();
  }
  // undo the row interchanges as column interchanges, last first
  for (int k = n - 1; k >= 0; k--)
  {
    const int p = piv[k];
    if (p != k && p < n && col)
    {
      const double t = S[lane * LD + k];
      S[lane * LD + k] = S[lane * LD + p];
      S[lane * LD + p] = t;
    }
  }
  __syncwarp();
  for (int i = 0; i < n; i++)
    if (col) inv[(size_t)i * n + lane] = S[i * LD + lane];
  if (lane == 0) flag[0] = singular ? 1 : 0;
}
