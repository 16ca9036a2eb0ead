// Time-dependent convection-diffusion (theta schemes) on top of a multigrid hierarchy:
// the GPU counterpart of TSystemTCD2D (src/System/SystemTCD2D.C) -- AssembleMRhs,
// AssembleARhs, AssembleSystMat, Solve, RestoreMassMat -- with the multigrid-preconditioned
// FGMRES of libcdgpu as the solver on every level.
//
// The mass matrix is kept and updated in place exactly like the reference's sqmatrixM:
//   M <- M - tau*theta2*A                    (MatAdd, Blas2.C:132, active rows only)
//   B  = tau*theta3*f_old + tau*theta4*f + M_active u_old;  B, u on Dirichlet rows <- f
//   M <- M + (tau*theta2 + tau*theta1)*A     (the system matrix)
//   solve M u = B
//   M <- M - tau*theta1*A                    (RestoreMassMat)
// so the rounding of every update is the reference's; all of it but the solve is one pass over
// the entries (tcd_system_kernel).
#include <algorithm>
#include <cmath>

#include "internal.h"

struct Tcd
{
  Hierarchy *h = nullptr;
  int disctype = CDGPU_GALERKIN;
  std::vector<double *> M, A; // per level, same CSR pattern as the level's space
  double *d_f_old = nullptr, *d_f = nullptr, *d_B = nullptr, *d_x = nullptr;
  bool have_mass = false, have_stiff = false;
  // BoundValue at the finest level's Dirichlet DOFs for the next assemblies (empty = 0)
  std::vector<double> h_dir;
};

static std::vector<Tcd *> &tcds(cdgpu_ctx *ctx) { return ctx->tcds; }

void free_tcd(Tcd *t)
{
  if (!t) return;
  for (double *p : t->M) cudaFree(p);
  for (double *p : t->A) cudaFree(p);
  double *v[] = {t->d_f_old, t->d_f, t->d_B, t->d_x};
  for (double *p : v)
    if (p) cudaFree(p);
  delete t;
}

// One step's matrix work on every level, and the finest right-hand side, in one pass over the
// entries (8 lanes per row, so the entries of a warp's rows are read and written as whole
// lines; up to four entries per lane in flight).  Entry by entry, with M read once:
//   m  = M - tau theta2 A           (where the level takes this update)
//   s += m x                        (finest level: the row's share of B)
//   m += c A                        (the system matrix: FP64, FP32 and diagonal copies)
//   M <- m - tau theta1 A           (what RestoreMassMat leaves; the solve reads the copies)
// each update rounded as the separate passes of MatAdd round it.  Dirichlet rows keep M and
// take B = f; their x = f comes in a launch of its own, the active rows read the old x.
// Bound by DRAM/L2 bytes (40 per entry) on large levels and by launches on small ones:
// 128^2 Q2 cells on 7 levels, a step's matrix work took 24 launches (a MatAdd before, in and
// after the solve and an install kernel per level, one thread per row in the latter):
// 155 us, now 2 launches, 17 us.
constexpr int kTcdLevels = 32; // levels of one launch (the argument's size stays below 4 KB)
constexpr int kTcdRows = 32;   // rows of a block

struct TcdLevel
{
  const int *rp, *kc;
  const double *A;
  double *M, *a, *diag;
  float *a32, *diag32;
  double c; // of the second update
  int n, n_active, block0, half;
};

struct TcdArgs
{
  int levels, fine; // fine: lev[0] is the finest level
  int in_order;     // the right-hand side's sums over a row's entries one after the other
  double c_half, c_restore, c3, c4;
  const double *f_old, *f, *x;
  double *B;
  TcdLevel lev[kTcdLevels];
};

__global__ void __launch_bounds__(256) tcd_system_kernel(const __grid_constant__ TcdArgs p)
{
  CD_PDL_ENTRY();
  constexpr int U = 4;
  int k = 0;
  while (k + 1 < p.levels && (int)blockIdx.x >= p.lev[k + 1].block0) k++;
  const TcdLevel &l = p.lev[k];
  const int lane = threadIdx.x % 8, r = ((int)blockIdx.x - l.block0) * kTcdRows + threadIdx.x / 8;
  const bool valid = r < l.n, active = r < l.n_active, rhs = p.fine && k == 0 && active;
  const int j1 = valid ? l.rp[r + 1] : 0;
  double s = 0;
  const bool in_order = rhs && p.in_order;
  if (in_order) // every lane the whole row, before any entry of M is replaced
    for (int j = l.rp[r]; j < j1; j++)
    {
      double v = l.M[j];
      if (l.half) v += p.c_half * l.A[j];
      s += v * p.x[l.kc[j]];
    }
  __syncwarp();
  for (int j0 = valid ? l.rp[r] + lane : 0; j0 < j1; j0 += 8 * U)
  {
    double m[U], a[U], x[U];
    int col[U];
#pragma unroll
    for (int q = 0; q < U; q++)
    {
      const int j = j0 + 8 * q;
      const bool in = j < j1;
      col[q] = in ? l.kc[j] : -1;
      m[q] = in ? l.M[j] : 0.0;
      a[q] = in && active ? l.A[j] : 0.0;
    }
    if (rhs)
#pragma unroll
      for (int q = 0; q < U; q++) x[q] = col[q] >= 0 ? p.x[col[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < U; q++)
    {
      const int j = j0 + 8 * q;
      if (j >= j1) break;
      double v = m[q];
      if (active)
      {
        if (l.half) v += p.c_half * a[q];
        if (rhs && !in_order) s += v * x[q];
        v += l.c * a[q];
        double back = v;
        back += p.c_restore * a[q];
        l.M[j] = back;
      }
      l.a[j] = v;
      l.a32[j] = (float)v;
      if (col[q] == r) { l.diag[r] = v; l.diag32[r] = (float)v; }
    }
  }
  if (!p.fine || k != 0) return; // block-uniform
  if (!p.in_order) // block-uniform
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, 8);
  if (lane != 0 || !valid) return;
  double b = 0.0;
  b += p.c3 * p.f_old[r];
  b += p.c4 * p.f[r];
  p.B[r] = active ? b + s : p.f[r];
}

__global__ void dirichlet_copy_kernel(int n, int n_active, const double *__restrict__ f, double *__restrict__ x)
{
  CD_PDL_ENTRY();
  int r = n_active + blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) x[r] = f[r];
}

static Tcd *get_tcd(cdgpu_ctx *ctx, int id)
{
  auto &v = tcds(ctx);
  return id >= 0 && id < (int)v.size() ? v[id] : nullptr;
}

// assemble one form on every level and keep the values in dst[l]; the finest right-hand
// side goes to rhs_dst
static int assemble_into(cdgpu_ctx *ctx, Tcd &t, int disctype, std::vector<double *> &dst, double *rhs_dst)
{
  // finest level first: while it runs, the launches of the small levels are queued behind it
  for (size_t l = t.h->lev.size(); l-- > 0;)
  {
    Space &s = *t.h->lev[l].sp;
    const bool fine = l + 1 == t.h->lev.size();
    const double *dir = fine && !t.h_dir.empty() ? t.h_dir.data() : nullptr;
    int rc = assemble_space(ctx, s, disctype, dir, false);
    if (rc) return rc;
    CD_CUDA(ctx, cudaMemcpyAsync(dst[l], s.d_a, sizeof(double) * s.nnz, cudaMemcpyDeviceToDevice, ctx->stream));
    if (l + 1 == t.h->lev.size() && rhs_dst)
      CD_CUDA(ctx, cudaMemcpyAsync(rhs_dst, s.d_rhs, sizeof(double) * s.n_dof, cudaMemcpyDeviceToDevice,
                                   ctx->stream));
  }
  return assemble_check(ctx);
}

extern "C" {

int cdgpu_tcd_create(cdgpu_ctx *ctx, int mg_id, int disctype, int *tcd_id)
{
  if (!ctx || mg_id < 0 || mg_id >= (int)ctx->mgs.size() || !tcd_id)
    return fail(ctx, CDGPU_ERR_INVALID, "tcd_create: bad argument");
  if (disctype != CDGPU_GALERKIN)
    return fail(ctx, CDGPU_ERR_UNSUPPORTED, "tcd_create: only the Galerkin time-dependent forms are implemented");
  cudaSetDevice(ctx->device);
  Tcd *t = new Tcd();
  t->h = ctx->mgs[mg_id];
  t->disctype = disctype;
  int rc;
  for (auto &L : t->h->lev)
  {
    double *m = nullptr, *a = nullptr;
    if ((rc = dev_alloc(ctx, &m, L.sp->nnz)) || (rc = dev_alloc(ctx, &a, L.sp->nnz))) return rc;
    t->M.push_back(m);
    t->A.push_back(a);
  }
  int n = t->h->lev.back().sp->n_dof;
  if ((rc = dev_alloc(ctx, &t->d_f_old, n)) || (rc = dev_alloc(ctx, &t->d_f, n)) || (rc = dev_alloc(ctx, &t->d_B, n)) ||
      (rc = dev_alloc(ctx, &t->d_x, n)))
    return rc;
  tcds(ctx).push_back(t);
  *tcd_id = (int)tcds(ctx).size() - 1;
  return CDGPU_OK;
}

// the boundary values that the reference's assembly takes from BoundValue at the current
// time (Assemble3D / Assemble2D set the Dirichlet entries of rhs), for the finest level's
// Dirichlet DOFs [n_active, n_dof); NULL returns to zero values
int cdgpu_tcd_set_dirichlet(cdgpu_ctx *ctx, int tcd_id, const double *h_dirichlet)
{
  Tcd *t = get_tcd(ctx, tcd_id);
  if (!t) return fail(ctx, CDGPU_ERR_INVALID, "tcd_set_dirichlet: bad id");
  const Space &f = *t->h->lev.back().sp;
  if (!h_dirichlet)
    t->h_dir.clear();
  else
    t->h_dir.assign(h_dirichlet, h_dirichlet + (f.n_dof - f.n_active));
  return CDGPU_OK;
}

// TSystemTCD2D::AssembleMRhs (SystemTCD2D.C:94-123): mass matrices of every level; the
// finest (f, phi) becomes the current right-hand side
int cdgpu_tcd_assemble_mass(cdgpu_ctx *ctx, int tcd_id)
{
  Tcd *t = get_tcd(ctx, tcd_id);
  if (!t) return fail(ctx, CDGPU_ERR_INVALID, "tcd_assemble_mass: bad id");
  cudaSetDevice(ctx->device);
  int rc = assemble_into(ctx, *t, CDGPU_MASS, t->M, t->d_f);
  if (rc) return rc;
  t->have_mass = true;
  return CDGPU_OK;
}

// TSystemTCD2D::AssembleARhs (SystemTCD2D.C:124-153) after the time loop's
// memcpy(oldrhs, rhs) (2DPrograms/TCD2D_ParMooN.C:265)
int cdgpu_tcd_assemble_stiffness(cdgpu_ctx *ctx, int tcd_id)
{
  Tcd *t = get_tcd(ctx, tcd_id);
  if (!t) return fail(ctx, CDGPU_ERR_INVALID, "tcd_assemble_stiffness: bad id");
  cudaSetDevice(ctx->device);
  int n = t->h->lev.back().sp->n_dof;
  CD_CUDA(ctx, cudaMemcpyAsync(t->d_f_old, t->d_f, sizeof(double) * n, cudaMemcpyDeviceToDevice, ctx->stream));
  int rc = assemble_into(ctx, *t, t->disctype, t->A, t->d_f);
  if (rc) return rc;
  t->have_stiff = true;
  return CDGPU_OK;
}

// AssembleSystMat (SystemTCD2D.C:154-186) + Solve + RestoreMassMat (187-210) for one step
int cdgpu_tcd_step_device(cdgpu_ctx *ctx, int tcd_id, const cdgpu_solver_params *p, double tau,
                          double theta1, double theta2, double theta3, double theta4, double *d_sol,
                          cdgpu_solve_info *info)
{
  Tcd *t = get_tcd(ctx, tcd_id);
  if (!t || !p || !d_sol) return fail(ctx, CDGPU_ERR_INVALID, "tcd_step: bad argument");
  if (!t->have_mass || !t->have_stiff) return fail(ctx, CDGPU_ERR_INVALID, "tcd_step: assemble mass and stiffness first");
  cudaSetDevice(ctx->device);
  Hierarchy &h = *t->h;
  const int L = (int)h.lev.size();
  const Space &f = *h.lev[L - 1].sp;
  // 2D (SystemTCD2D.C): M <- M - tau theta2 A on every level, so that the coarse levels get
  // the finest level's sequence of updates; 3D (SystemTCD3D.C:257-278): on the finest level
  // only, the coarser levels' system matrices are M + tau theta1 A
  const bool fine_only = f.dim == 3;
  // finest level first, in the blocks of one launch
  for (int top = L - 1; top >= 0;)
  {
    TcdArgs a;
    a.levels = 0;
    a.fine = top == L - 1;
    a.in_order = step_keeps_order(f, p->precision);
    a.c_half = -tau * theta2;
    a.c_restore = -tau * theta1;
    a.c3 = tau * theta3;
    a.c4 = tau * theta4;
    a.f_old = t->d_f_old;
    a.f = t->d_f;
    a.x = d_sol;
    a.B = t->d_B;
    long blocks = 0;
    for (; top >= 0 && a.levels < kTcdLevels; top--)
    {
      Space &s = *h.lev[top].sp;
      const bool half = !(fine_only && top < L - 1);
      const double c = half ? -a.c_half + tau * theta1 : tau * theta1;
      a.lev[a.levels++] = {s.d_row_ptr, s.d_kcol, t->A[top], t->M[top], s.d_a, s.d_diag, s.d_a32, s.d_diag32, c,
                           s.n_dof, s.n_active, (int)blocks, half ? 1 : 0};
      blocks += (s.n_dof + kTcdRows - 1) / kTcdRows;
      s.mf_T = 0; // the system matrix is a combination, not one affine assembly
      s.assembly_version++;
    }
    (void)cd_launch(tcd_system_kernel, (unsigned)std::max(1L, blocks), 256, 0, ctx->stream, a);
    CD_LAUNCHED(ctx);
  }
  if (f.n_dof > f.n_active)
  {
    (void)cd_launch(dirichlet_copy_kernel, (f.n_dof - f.n_active + 255) / 256, 256, 0, ctx->stream, f.n_dof, f.n_active, t->d_f,
                                                                                     d_sol);
    CD_LAUNCHED(ctx);
  }
  cdgpu_solve_info local{};
  return run_solve(ctx, h, *p, t->d_B, d_sol, info ? info : &local, true);
}

int cdgpu_tcd_step(cdgpu_ctx *ctx, int tcd_id, const cdgpu_solver_params *p, double tau, double theta1,
                   double theta2, double theta3, double theta4, double *h_sol, cdgpu_solve_info *info)
{
  Tcd *t = get_tcd(ctx, tcd_id);
  if (!t || !h_sol) return fail(ctx, CDGPU_ERR_INVALID, "tcd_step: bad argument");
  cudaSetDevice(ctx->device);
  int n = t->h->lev.back().sp->n_dof;
  CD_CUDA(ctx, cudaMemcpyAsync(t->d_x, h_sol, sizeof(double) * n, cudaMemcpyHostToDevice, ctx->stream));
  int rc = cdgpu_tcd_step_device(ctx, tcd_id, p, tau, theta1, theta2, theta3, theta4, t->d_x, info);
  if (rc) return rc;
  CD_CUDA(ctx, cudaMemcpyAsync(h_sol, t->d_x, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream));
  CD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return CDGPU_OK;
}

// copies of one level's mass matrix M (as updated in place), stiffness matrix A and the system
// matrix the last step's solve used (the level's installed entries), each nullable; like
// TSystemTCD2D's sqmatrixM / sqmatrixA members (include/System/SystemTCD2D.h)
int cdgpu_tcd_matrices(cdgpu_ctx *ctx, int tcd_id, int level, double *h_M, double *h_A, double *h_S)
{
  Tcd *t = get_tcd(ctx, tcd_id);
  if (!t || level < 0 || level >= (int)t->h->lev.size()) return fail(ctx, CDGPU_ERR_INVALID, "tcd_matrices: bad argument");
  if ((h_M && !t->have_mass) || (h_A && !t->have_stiff)) return fail(ctx, CDGPU_ERR_INVALID, "tcd_matrices: not assembled");
  const Space &s = *t->h->lev[level].sp;
  if (h_S && !s.assembled) return fail(ctx, CDGPU_ERR_INVALID, "tcd_matrices: no system matrix yet");
  cudaSetDevice(ctx->device);
  const size_t bytes = sizeof(double) * s.nnz;
  if (h_M) CD_CUDA(ctx, cudaMemcpyAsync(h_M, t->M[level], bytes, cudaMemcpyDeviceToHost, ctx->stream));
  if (h_A) CD_CUDA(ctx, cudaMemcpyAsync(h_A, t->A[level], bytes, cudaMemcpyDeviceToHost, ctx->stream));
  if (h_S) CD_CUDA(ctx, cudaMemcpyAsync(h_S, s.d_a, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  CD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return CDGPU_OK;
}

// the current finest right-hand side (f, phi) of the last assembly, to the host
int cdgpu_tcd_rhs(cdgpu_ctx *ctx, int tcd_id, double *h_rhs)
{
  Tcd *t = get_tcd(ctx, tcd_id);
  if (!t || !h_rhs) return fail(ctx, CDGPU_ERR_INVALID, "tcd_rhs: bad argument");
  int n = t->h->lev.back().sp->n_dof;
  CD_CUDA(ctx, cudaMemcpyAsync(h_rhs, t->d_f, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream));
  CD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return CDGPU_OK;
}

} // extern "C"
