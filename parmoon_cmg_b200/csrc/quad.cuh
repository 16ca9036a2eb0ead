// Local matrices and right-hand sides by Gauss quadrature, for cells that are not affine and
// coefficients that vary in space: the reference's per-point local forms (src/FE/ConvDiff2D.C:
// 32-162, src/FE/ConvDiff3D.C:61-190) with the assembly's own Gauss rule.  Writes nbf * nbf matrix
// entries then nbf right-hand side entries per cell.
//
// In reference coordinates every form is
//   A_ij = sum_q sum_ab C_ab(q) D_a phi_i(q) D_b phi_j(q),   F_i = sum_q sum_a f_a(q) D_a phi_i(q)
// with D_a the value and the reference derivatives (2D SUPG: the trial side also has second
// derivatives), and C, f the weight, geometry and coefficients of a point: for every cell they are
// evaluated once per point, and basis and rule are tensor products of one-dimensional tables, so
// the sums over the points are taken one direction at a time.
//   * Q2 hexahedra (quad27_kernel): 5 cells per block pass; the three directions are contracted
//     one after the other through shared memory, 32,000 FMAs per cell instead of the 47,000
//     points x entries with 10 FMAs each.  24^3 deformed cells, table coefficients: 1,900 us for
//     one entry and point at a time, now 144 us (FP64 pipe 40 %, bound by the latency of the
//     stages at two blocks per SM; 4 barriers per 5 cells).
//   * the other elements (quad_lane_kernel): 32 cells per block pass, lane = cell, warp = local
//     row i; a thread forms its row's sums over the trial functions direction by direction in
//     registers, without a barrier between the coefficients and the copy out.  160^2 Q2 cells,
//     SUPG, table coefficients: 358 us with one cell per block pass, now 40 us; 128^2 Galerkin
//     (and its coarser levels) 37.9 us per level on average, now 7.9.
#pragma once

#include "internal.h"

enum { QF_MASS = 0, QF_GALERKIN = 1, QF_SUPG = 2 };

struct QuadArgs
{
  int n_cells, affine_all;
  Coef co;
  const double *coords, *tab; // tab: n_cells x nq x 6 (kind TABLE)
  double *out;
  QuadTab t;
};

// geometry and coefficients of one Gauss point
template <int DIM> struct QuadPoint
{
  double m, k[6], delta, Ji[DIM * DIM];
  double beta[DIM]; // J^-1 b
  template <int NV>
  __device__ __forceinline__ void eval(const QuadArgs &a, const double *V, const double *rec, const double *xi, double w,
                                       bool supg)
  {
    double x[3], J[9], Jx[9];
    d_ref_map(DIM, NV, a.affine_all != 0, V, xi, x, J);
    const double det = d_invert(DIM, J, Jx);
#pragma unroll
    for (int i = 0; i < DIM * DIM; i++) Ji[i] = Jx[i];
    m = w * fabs(det);
    coef_at(a.co, rec, x, k);
#pragma unroll
    for (int e = 0; e < DIM; e++)
    {
      double s = 0;
#pragma unroll
      for (int r = 0; r < DIM; r++) s += Ji[e * DIM + r] * k[1 + r];
      beta[e] = s;
    }
    delta = supg ? sdfem_delta(d_diameter(DIM, V), k[0], k[1], k[2], DIM == 3 ? k[3] : 0.0, a.co.delta0, a.co.poly_degree)
                 : 0.0;
  }
  // G_ef = sum_r Ji[e][r] Ji[f][r]
  __device__ __forceinline__ double metric(int e, int f) const
  {
    double s = 0;
#pragma unroll
    for (int r = 0; r < DIM; r++) s += Ji[e * DIM + r] * Ji[f * DIM + r];
    return s;
  }
};

// ---------------------------------------------------------------------------
// Q1 quadrilaterals and hexahedra, Q2 quadrilaterals
// ---------------------------------------------------------------------------
template <int DIM, int P, int FORM> struct QuadLane
{
  static constexpr int N1 = P + 1, Q1 = P == 1 ? 3 : 4, NB = DIM == 2 ? N1 * N1 : N1 * N1 * N1,
                       NQ = DIM == 2 ? Q1 * Q1 : Q1 * Q1 * Q1, NV = 1 << DIM, PER = NB * NB + NB;
  static constexpr bool LAP = DIM == 2 && FORM == QF_SUPG; // the residual's Laplacian
  // fields of a point: C_00, C_0s, C_rs (all DIM^2), C_r0, the Laplacian's -m delta eps beta_r and
  // G_00, G_11, 2 G_01, then f_0 and f_r
  static constexpr int C00 = 0, C0S = 1, CRS = C0S + DIM, CR0 = FORM == QF_MASS ? 1 : CRS + DIM * DIM,
                       LB = CR0 + (FORM == QF_SUPG ? DIM : 0), LG = LB + (LAP ? 2 : 0), F0 = LG + (LAP ? 3 : 0),
                       NF = F0 + (FORM == QF_SUPG ? 1 + DIM : 1);
  static constexpr int LD = 33; // cells of a field and point, padded
  static constexpr int OUT_LD = PER + 1;
  static constexpr int FIELDS = NF * NQ * LD, OUT = 32 * OUT_LD, BIG = FIELDS > OUT ? FIELDS : OUT;
  static constexpr int THREADS = 32 * NB;
  static constexpr int TEST = NQ * NB * (DIM + 1); // D_a phi_i at the points
  static constexpr size_t smem() { return sizeof(double) * (size_t)(BIG + TEST); }
};

template <int DIM, int P, int FORM>
__global__ void __launch_bounds__(QuadLane<DIM, P, FORM>::THREADS) quad_lane_kernel(const __grid_constant__ QuadArgs a)
{
  using T = QuadLane<DIM, P, FORM>;
  constexpr int N1 = T::N1, Q1 = T::Q1, NB = T::NB, NQ = T::NQ, NV = T::NV, LD = T::LD;
  CD_PDL_ENTRY();
  extern __shared__ double qsm[];
  double *fld = qsm, *test = qsm + T::BIG;
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < NQ * NB; e += T::THREADS)
  {
    const int q = e / NB, i = e - q * NB;
    const int qi[3] = {q % Q1, q / Q1 % Q1, q / (Q1 * Q1)}, ii[3] = {i % N1, i / N1 % N1, i / (N1 * N1)};
    for (int d = 0; d <= DIM; d++)
    {
      double v = 1.0;
      for (int b = 0; b < DIM; b++) v *= d == b + 1 ? a.t.G[qi[b]][ii[b]] : a.t.B[qi[b]][ii[b]];
      test[e * (DIM + 1) + d] = v;
    }
  }
  const int groups = (a.n_cells + 31) / 32;
  for (int grp = blockIdx.x; grp < groups; grp += gridDim.x)
  {
    const int c0 = grp * 32, nc = min(32, a.n_cells - c0);
    __syncthreads(); // the previous group's results have left the shared tile (first: the tables)
    // the points' fields; neighbouring threads take neighbouring points of a cell
    for (int e = threadIdx.x; e < nc * NQ; e += T::THREADS)
    {
      const int lc = e / NQ, q = e - lc * NQ;
      const int qx = q % Q1, qy = q / Q1 % Q1, qz = q / (Q1 * Q1);
      const double xi[3] = {a.t.x[qx], a.t.x[qy], DIM == 3 ? a.t.x[qz] : 0.0};
      double V[NV * DIM];
      const double *Vg = a.coords + (size_t)(c0 + lc) * NV * DIM;
#pragma unroll
      for (int k = 0; k < NV * DIM; k++) V[k] = __ldg(Vg + k);
      QuadPoint<DIM> p;
      p.template eval<NV>(a, V, a.tab ? a.tab + ((size_t)(c0 + lc) * NQ + q) * 6 : nullptr, xi,
                          a.t.w[qx] * a.t.w[qy] * (DIM == 3 ? a.t.w[qz] : 1.0), FORM == QF_SUPG);
      double *o = fld + q * LD + lc;
      auto put = [&](int f, double v) { o[f * NQ * LD] = v; };
      if constexpr (FORM == QF_MASS)
        put(T::C00, p.m);
      else
      {
        const double md = p.m * p.delta, me = p.m * p.k[0];
        put(T::C00, p.m * p.k[4]);
        double lb[2] = {0, 0}, gam[2] = {0, 0}, g01 = 0;
        if constexpr (T::LAP)
        {
          // Laplacian G_00 d_00 + G_11 d_11 + 2 G_01 (d_01 - gamma . grad): on a bilinear cell
          // x = .. + c3 xi eta the mixed derivative carries grad(phi) . c3
          // (QuadBilinear::GetOrigValues, src/FE/QuadBilinear.C:531-549)
          g01 = 2.0 * p.metric(0, 1);
#pragma unroll
          for (int r = 0; r < 2; r++)
          {
            lb[r] = -md * p.k[0] * p.beta[r];
            put(T::LB + r, lb[r]);
            if (!a.affine_all)
#pragma unroll
              for (int s = 0; s < 2; s++) gam[s] += p.Ji[s * 2 + r] * 0.25 * (V[r] - V[2 + r] + V[4 + r] - V[6 + r]);
          }
          put(T::LG, p.metric(0, 0));
          put(T::LG + 1, p.metric(1, 1));
          put(T::LG + 2, g01);
        }
#pragma unroll
        for (int s = 0; s < DIM; s++)
        {
          put(T::C0S + s, p.m * p.beta[s]);
#pragma unroll
          for (int r = 0; r < DIM; r++)
          {
            double v = me * p.metric(r, s);
            if (FORM == QF_SUPG) v += md * p.beta[r] * p.beta[s];
            if constexpr (T::LAP) v -= lb[r] * g01 * gam[s];
            put(T::CRS + r * DIM + s, v);
          }
          if (FORM == QF_SUPG)
          {
            put(T::CR0 + s, md * p.k[4] * p.beta[s]);
            put(T::F0 + 1 + s, md * p.k[5] * p.beta[s]);
          }
        }
      }
      put(T::F0, p.m * p.k[5]);
    }
    __syncthreads();
    // row `row` of cell `lane`: the trial sums direction by direction, x innermost
    double A[NB], F = 0.0;
#pragma unroll
    for (int j = 0; j < NB; j++) A[j] = 0.0;
    const double *ti = test + row * (DIM + 1);
    auto point = [&](int q, double (&t)[DIM + 1], double (&l)[3]) {
      // coefficients of the trial side: t_b = sum_a C_ab D_a phi_i, l: of the second derivatives
      const double *c = fld + q * LD + lane, *d = ti + q * NB * (DIM + 1);
      auto C = [&](int f) { return c[f * NQ * LD]; };
      const double ph = d[0];
      t[0] = C(T::C00) * ph;
      F += C(T::F0) * ph;
      if constexpr (FORM != QF_MASS)
      {
#pragma unroll
        for (int s = 0; s < DIM; s++)
        {
          double v = C(T::C0S + s) * ph;
#pragma unroll
          for (int r = 0; r < DIM; r++) v += C(T::CRS + r * DIM + s) * d[1 + r];
          t[1 + s] = v;
          if (FORM == QF_SUPG)
          {
            t[0] += C(T::CR0 + s) * d[1 + s];
            F += C(T::F0 + 1 + s) * d[1 + s];
          }
        }
        if constexpr (T::LAP)
        {
          const double bg = C(T::LB) * d[1] + C(T::LB + 1) * d[2];
#pragma unroll
          for (int s = 0; s < 3; s++) l[s] = bg * C(T::LG + s);
        }
      }
    };
    if constexpr (DIM == 2)
    {
#pragma unroll
      for (int qy = 0; qy < Q1; qy++)
      {
        double uv[N1], uy[N1], uyy[N1]; // trial x sums of the terms without, with d_y and d_yy
#pragma unroll
        for (int j = 0; j < N1; j++) uv[j] = uy[j] = uyy[j] = 0.0;
#pragma unroll
        for (int qx = 0; qx < Q1; qx++)
        {
          double t[DIM + 1], l[3];
          point(qy * Q1 + qx, t, l);
#pragma unroll
          for (int j = 0; j < N1; j++)
          {
            uv[j] += t[0] * a.t.B[qx][j];
            if constexpr (FORM != QF_MASS)
            {
              uv[j] += t[1] * a.t.G[qx][j];
              uy[j] += t[2] * a.t.B[qx][j];
            }
            if constexpr (T::LAP)
            {
              if (P == 2) uv[j] += l[0] * a.t.H[qx][j];
              uy[j] += l[2] * a.t.G[qx][j];
              if (P == 2) uyy[j] += l[1] * a.t.B[qx][j];
            }
          }
        }
#pragma unroll
        for (int jy = 0; jy < N1; jy++)
#pragma unroll
          for (int j = 0; j < N1; j++)
          {
            double s = A[jy * N1 + j] + uv[j] * a.t.B[qy][jy];
            if constexpr (FORM != QF_MASS) s += uy[j] * a.t.G[qy][jy];
            if constexpr (T::LAP && P == 2) s += uyy[j] * a.t.H[qy][jy];
            A[jy * N1 + j] = s;
          }
      }
    }
    else
    {
#pragma unroll
      for (int qz = 0; qz < Q1; qz++)
      {
        double wv[N1][N1], wz[N1][N1];
#pragma unroll
        for (int jy = 0; jy < N1; jy++)
#pragma unroll
          for (int j = 0; j < N1; j++) wv[jy][j] = wz[jy][j] = 0.0;
#pragma unroll
        for (int qy = 0; qy < Q1; qy++)
        {
          double uv[N1], uy[N1], uz[N1];
#pragma unroll
          for (int j = 0; j < N1; j++) uv[j] = uy[j] = uz[j] = 0.0;
#pragma unroll
          for (int qx = 0; qx < Q1; qx++)
          {
            double t[DIM + 1], l[3];
            point((qz * Q1 + qy) * Q1 + qx, t, l);
#pragma unroll
            for (int j = 0; j < N1; j++)
            {
              uv[j] += t[0] * a.t.B[qx][j];
              if constexpr (FORM != QF_MASS)
              {
                uv[j] += t[1] * a.t.G[qx][j];
                uy[j] += t[2] * a.t.B[qx][j];
                uz[j] += t[3] * a.t.B[qx][j];
              }
            }
          }
#pragma unroll
          for (int jy = 0; jy < N1; jy++)
#pragma unroll
            for (int j = 0; j < N1; j++)
            {
              wv[jy][j] += uv[j] * a.t.B[qy][jy];
              if constexpr (FORM != QF_MASS)
              {
                wv[jy][j] += uy[j] * a.t.G[qy][jy];
                wz[jy][j] += uz[j] * a.t.B[qy][jy];
              }
            }
        }
#pragma unroll
        for (int jz = 0; jz < N1; jz++)
#pragma unroll
          for (int jy = 0; jy < N1; jy++)
#pragma unroll
            for (int j = 0; j < N1; j++)
            {
              double s = A[(jz * N1 + jy) * N1 + j] + wv[jy][j] * a.t.B[qz][jz];
              if constexpr (FORM != QF_MASS) s += wz[jy][j] * a.t.G[qz][jz];
              A[(jz * N1 + jy) * N1 + j] = s;
            }
      }
    }
    __syncthreads(); // the fields' space takes the results
    double *os = qsm + lane * T::OUT_LD;
#pragma unroll
    for (int j = 0; j < NB; j++) os[row * NB + j] = A[j];
    os[NB * NB + row] = F;
    __syncthreads();
    double *og = a.out + (size_t)c0 * T::PER;
    for (int e = threadIdx.x; e < nc * T::PER; e += T::THREADS) og[e] = qsm[e / T::PER * T::OUT_LD + e % T::PER];
  }
}

// ---------------------------------------------------------------------------
// Q2 hexahedra
// ---------------------------------------------------------------------------
// (two blocks per SM leave 128 registers: 32-40 bytes of spill stores, 36-52 of loads, by form)
constexpr int kQ27Cells = 5, kQ27Threads = 256;

// products of one-dimensional functions at the points: [q][i * 3 + j], i the test function
struct QuadPairs
{
  double BB[4][9], BG[4][9], GB[4][9], GG[4][9];
};

// fields of a point: C_00, C_0x..z, C_xx C_yy C_zz C_xy C_xz C_yz, (SUPG) C_x0..z0, f_0, (SUPG) f_x..z
template <int FORM> struct Quad27
{
  static constexpr int CR0 = 10, F0 = FORM == QF_MASS ? 1 : FORM == QF_GALERKIN ? 10 : 13,
                       NF = F0 + (FORM == QF_SUPG ? 4 : 1);
  static constexpr int T1 = (FORM == QF_MASS ? 1 : 8) * 144, T2 = (FORM == QF_MASS ? 1 : 4) * 324;
  // per cell: region 1 the fields, then the sums over z and y; region 2 the sums over z, then the
  // results
  static constexpr int R1 = NF * 64 > T2 ? NF * 64 : T2, R2 = T1 > 756 ? T1 : 756;
  static constexpr size_t smem() { return sizeof(double) * (size_t)(kQ27Cells * (R1 + R2 + 27) + 4 * 4 * 9); }
};

template <int FORM>
__global__ void __launch_bounds__(kQ27Threads, 2) quad27_kernel(const __grid_constant__ QuadArgs a,
                                                                const __grid_constant__ QuadPairs pr)
{
  using T = Quad27<FORM>;
  CD_PDL_ENTRY();
  extern __shared__ double qsm[];
  double *reg1 = qsm, *reg2 = qsm + kQ27Cells * T::R1, *rhs = reg2 + kQ27Cells * T::R2, *pairs = rhs + kQ27Cells * 27;
  const int tid = threadIdx.x;
  if (tid < 144) pairs[tid] = (&pr.BB[0][0])[tid]; // [type][q][pair]
  const int groups = (a.n_cells + kQ27Cells - 1) / kQ27Cells;
  for (int grp = blockIdx.x; grp < groups; grp += gridDim.x)
  {
    const int c0 = grp * kQ27Cells, nc = min(kQ27Cells, a.n_cells - c0);
    // the points' fields
    for (int e = tid; e < nc * 64; e += kQ27Threads)
    {
      const int lc = e >> 6, q = e & 63, qx = q & 3, qy = q >> 2 & 3, qz = q >> 4;
      const double xi[3] = {a.t.x[qx], a.t.x[qy], a.t.x[qz]};
      double V[24];
      const double *Vg = a.coords + (size_t)(c0 + lc) * 24;
#pragma unroll
      for (int k = 0; k < 24; k++) V[k] = __ldg(Vg + k);
      QuadPoint<3> p;
      p.template eval<8>(a, V, a.tab ? a.tab + ((size_t)(c0 + lc) * 64 + q) * 6 : nullptr, xi,
                         a.t.w[qx] * a.t.w[qy] * a.t.w[qz], FORM == QF_SUPG);
      double *o = reg1 + lc * T::R1 + q;
      if constexpr (FORM == QF_MASS)
        o[0] = p.m;
      else
      {
        const double me = p.m * p.k[0], md = p.m * p.delta;
        o[0] = p.m * p.k[4];
#pragma unroll
        for (int s = 0; s < 3; s++)
        {
          o[(1 + s) * 64] = p.m * p.beta[s];
          if (FORM == QF_SUPG)
          {
            o[(T::CR0 + s) * 64] = md * p.k[4] * p.beta[s];
            o[(T::F0 + 1 + s) * 64] = md * p.k[5] * p.beta[s];
          }
        }
        constexpr int er[6] = {0, 1, 2, 0, 0, 1}, es[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
        for (int u = 0; u < 6; u++)
        {
          double v = me * p.metric(er[u], es[u]);
          if (FORM == QF_SUPG) v += md * p.beta[er[u]] * p.beta[es[u]];
          o[(4 + u) * 64] = v;
        }
      }
      o[T::F0 * 64] = p.m * p.k[5];
    }
    __syncthreads();
    // z: thread = (cell, qy, iz, qx); for the three jz the sums over qz, by the x and y
    // derivatives of test and trial function (v: neither): vv vx vy xv yv xx xy yy
    if (tid < nc * 48)
    {
      const int lc = tid / 48, it = tid - lc * 48, qx = it & 3, iz = it / 4 % 3, qy = it / 12;
      const double *c = reg1 + lc * T::R1 + qy * 4 + qx;
      double s[8][3];
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int j = 0; j < 3; j++) s[u][j] = 0.0;
#pragma unroll
      for (int qz = 0; qz < 4; qz++)
      {
        const double *cq = c + qz * 16, *pq = pairs + qz * 9 + iz * 3;
        auto C = [&](int f) { return cq[f * 64]; };
        if constexpr (FORM == QF_MASS)
        {
          const double c00 = C(0);
#pragma unroll
          for (int j = 0; j < 3; j++) s[0][j] += c00 * pq[j];
        }
        else
        {
          const double c00 = C(0), c0x = C(1), c0y = C(2), c0z = C(3), cxx = C(4), cyy = C(5), czz = C(6), cxy = C(7),
                       cxz = C(8), cyz = C(9);
          double cx0 = 0, cy0 = 0, cz0 = 0;
          if (FORM == QF_SUPG) cx0 = C(T::CR0), cy0 = C(T::CR0 + 1), cz0 = C(T::CR0 + 2);
#pragma unroll
          for (int j = 0; j < 3; j++)
          {
            const double bb = pq[j], bg = pq[36 + j], gb = pq[72 + j], gg = pq[108 + j];
            s[0][j] += c00 * bb + c0z * bg + czz * gg;
            s[1][j] += c0x * bb + cxz * gb;
            s[2][j] += c0y * bb + cyz * gb;
            s[3][j] += cxz * bg;
            s[4][j] += cyz * bg;
            s[5][j] += cxx * bb;
            s[6][j] += cxy * bb;
            s[7][j] += cyy * bb;
            if (FORM == QF_SUPG)
            {
              s[0][j] += cz0 * gb;
              s[3][j] += cx0 * bb;
              s[4][j] += cy0 * bb;
            }
          }
        }
      }
      double *o = reg2 + lc * T::R2 + (qy * 9 + iz * 3) * 4 + qx; // [sum][qy][iz jz][qx]
#pragma unroll
      for (int u = 0; u < (FORM == QF_MASS ? 1 : 8); u++)
#pragma unroll
        for (int j = 0; j < 3; j++) o[u * 144 + j * 4] = s[u][j];
    }
    // right-hand side, thread = (cell, i)
    if (tid < nc * 27)
    {
      const int lc = tid / 27, i = tid - lc * 27, ix = i % 3, iy = i / 3 % 3, iz = i / 9;
      const double *f = reg1 + lc * T::R1 + T::F0 * 64;
      double s = 0.0;
#pragma unroll 1
      for (int qz = 0; qz < 4; qz++)
#pragma unroll 1
        for (int qy = 0; qy < 4; qy++)
        {
          const double by = a.t.B[qy][iy], bz = a.t.B[qz][iz];
          double s0 = 0.0, sx = 0.0;
#pragma unroll
          for (int qx = 0; qx < 4; qx++)
          {
            const int q = qz * 16 + qy * 4 + qx;
            double v = f[q] * by * bz;
            if (FORM == QF_SUPG)
            {
              v += f[128 + q] * a.t.G[qy][iy] * bz + f[192 + q] * by * a.t.G[qz][iz];
              sx += f[64 + q] * a.t.G[qx][ix];
            }
            s0 += v * a.t.B[qx][ix];
          }
          s += s0 + sx * by * bz;
        }
      rhs[lc * 27 + i] = s;
    }
    __syncthreads();
    // y: thread = (cell, iz jz, qx); for the nine (iy, jy) the sums over qy, by the x derivatives
    if (tid < nc * 36)
    {
      const int lc = tid / 36, it = tid - lc * 36, pz = it >> 2, qx = it & 3;
      const double *c = reg2 + lc * T::R2 + it;
      double s[4][9];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int p = 0; p < 9; p++) s[u][p] = 0.0;
#pragma unroll
      for (int qy = 0; qy < 4; qy++)
      {
        double v[8];
#pragma unroll
        for (int u = 0; u < (FORM == QF_MASS ? 1 : 8); u++) v[u] = c[u * 144 + qy * 36];
#pragma unroll
        for (int p = 0; p < 9; p++)
        {
          s[0][p] += v[0] * pr.BB[qy][p];
          if constexpr (FORM != QF_MASS)
          {
            s[0][p] += v[2] * pr.BG[qy][p] + v[4] * pr.GB[qy][p] + v[7] * pr.GG[qy][p];
            s[1][p] += v[1] * pr.BB[qy][p] + v[6] * pr.GB[qy][p];
            s[2][p] += v[3] * pr.BB[qy][p] + v[6] * pr.BG[qy][p];
            s[3][p] += v[5] * pr.BB[qy][p];
          }
        }
      }
      double *o = reg1 + lc * T::R1 + qx * 81 + pz; // [sum][qx][iy jy][iz jz]
#pragma unroll
      for (int u = 0; u < (FORM == QF_MASS ? 1 : 4); u++)
#pragma unroll
        for (int p = 0; p < 9; p++) o[u * 324 + p * 9] = s[u][p];
    }
    __syncthreads();
    // x: thread = (cell, iy jy, iz jz); the nine (ix, jx)
    for (int e = tid; e < nc * 81; e += kQ27Threads)
    {
      const int lc = e / 81, it = e - lc * 81, py = it / 9, pz = it - py * 9;
      const double *c = reg1 + lc * T::R1 + it;
      double s[9];
#pragma unroll
      for (int p = 0; p < 9; p++) s[p] = 0.0;
#pragma unroll
      for (int qx = 0; qx < 4; qx++)
      {
        double v[4];
#pragma unroll
        for (int u = 0; u < (FORM == QF_MASS ? 1 : 4); u++) v[u] = c[u * 324 + qx * 81];
#pragma unroll
        for (int p = 0; p < 9; p++)
        {
          s[p] += v[0] * pr.BB[qx][p];
          if constexpr (FORM != QF_MASS) s[p] += v[1] * pr.BG[qx][p] + v[2] * pr.GB[qx][p] + v[3] * pr.GG[qx][p];
        }
      }
      double *o = reg2 + lc * T::R2 + (py / 3 * 3 + pz / 3 * 9) * 27 + py % 3 * 3 + pz % 3 * 9;
#pragma unroll
      for (int p = 0; p < 9; p++) o[p / 3 * 27 + p % 3] = s[p];
    }
    __syncthreads();
    double *og = a.out + (size_t)c0 * 756;
    for (int e = tid; e < nc * 756; e += kQ27Threads)
    {
      const int lc = e / 756, k = e - lc * 756;
      og[e] = k < 729 ? reg2[lc * T::R2 + k] : rhs[lc * 27 + k - 729];
    }
  }
}
