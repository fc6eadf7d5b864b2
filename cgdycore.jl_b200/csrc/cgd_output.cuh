// cgd_output.cuh - interpolation of the state to the output sub-cells.
//
// The reference writes its VTK output from OrdPrint x OrdPrint sub-cells per
// element and layer: each cell value is the element's GLL interpolant at the
// cell centre, Inter[I,J,iP,jP] = L_iP(xi_I) L_jP(eta_J)
// (src/Outputs/vtkSphere.jl:199-219), applied to the nodal values gathered
// through Glob (InterpolateKernel!, src/Outputs/vtkOutputKernel.jl:49-74).
// k_cells evaluates the same sums in the same order, several quantities at once:
//
//   InterpolateKernel!     cCell = sum_(jP,iP) Inter * c
//   InterpolateRhoKernel!  cCell = sum_(jP,iP) Inter * c / rhoc     (:97-121)
//   of the pressure or the potential temperature     ("Pres" and "Th")
//   InterpolateWBKernel!   layer-mean w, the surface w from no normal flow (:123-159)
//   InterpolateRotKernel!  element-local vertical vorticity         (:1-47)
//
// The reference's vorticity kernel accumulates with atomics (unordered); here
// every sum runs in ascending node order: the curl at node (i,j) is
// sum_I D(i,I) tx(I,j) followed by sum_J D(j,J) ty(i,J), from 0.
// Inter is Fortran-ordered (OrdPrint, OrdPrint, N, N); cCell is
// (OrdPrint, OrdPrint, nz, NF).
#pragma once
#include "cgd_kernels.cuh"

namespace cgd {

constexpr int OUT_MAX_PRINT = 8;   // OrdPrint <= 8

__device__ __forceinline__ double pott_dry(const GP &P, double rho, double p)
{
  // the dry model's Pressure (src/Models/Equation.jl:24-32), evaluated by
  // PressureKernel! into Cache.AuxG[:,:,1] (p) and [:,:,3]
  const double T = p / (P.Rd * rho);
  return pow(P.p0 / p, P.kappa) * T;   // (p0/p)^(Rd/Cpd) * T
}

// What a cell value interpolates.
enum { CELL_C = 0, CELL_C_RHO, CELL_PRES, CELL_POTT, CELL_WB, CELL_VORT };

// One launch's quantities: cell array k (n values each, back to back) is kind
// op[k].op of the columns c (and, for CELL_WB, u, v; for CELL_VORT, u and v).
constexpr int CELL_MAX = 16;
struct CellOp {
  int op;
  const double *c, *u, *v;
};
struct CellArgs {
  CellOp f[CELL_MAX];
  int n;
  const double *rho, *rhoth;   // (nz, NumG); what CELL_C_RHO divides by, what the pressure is of
};

// n / d with r = 1 / d: the correctly rounded quotient by two Newton
// corrections of n r, whose residuals are exact; outside the range where they
// are, the division itself.
__device__ __forceinline__ double exact_quotient(double n, double d, double r)
{
  double q = n * r;
  const double a = fabs(q);
  if (a > 1e-280 && a < 1e280) {
    q = __fma_rn(__fma_rn(-q, d, n), r, q);
    return __fma_rn(__fma_rn(-q, d, n), r, q);
  }
  return n == 0.0 ? q : n / d;
}

// One CTA per (element, tile of LT levels), numbered in one dimension: more than
// 65535 elements are taken.  The nodal values of every
// quantity are formed once, by one thread per (node, level), level fastest
// (runs of consecutive levels of a column), into shared planes; then the
// threads, each holding one sub-cell's N^2 weights in registers, walk the
// (quantity, level) pairs and write runs of consecutive cells.  One kernel
// per quantity and one thread per cell, as before, gathered the columns again
// for every sub-cell, evaluated the pressure's exp and log N^2 times for each,
// and wrote OrdPrint^2 values apart: nPanel 30, nz 45, nine quantities on
// 4 x 4 sub-cells 4.80 ms.
template <int N>
struct CellCfg {
  static constexpr int DoF = N * N, LT = 256 / DoF;
  static constexpr int RS = (DoF + 2) & ~1;   // row of a plane: even, so that two nodes are one 16-byte load
  static constexpr int PL = LT * RS;
  static size_t smem(int nq) { return ((size_t)(nq + 4) * PL) * sizeof(double); }   // planes, rho, 1/rho, tx, ty
};

template <int N>
__global__ void __launch_bounds__(256, N == 5 ? 3 : 4) k_cells(const GP P, const CellArgs A, const double *__restrict__ inter, int OP,
                                               double *__restrict__ cell)
{
  using CF = CellCfg<N>;
  constexpr int DoF = CF::DoF, LT = CF::LT, RS = CF::RS, PL = CF::PL;
  extern __shared__ __align__(16) double sc[];
  double *srho = sc + (size_t)A.n * PL, *srr = srho + PL, *tx = srr + PL, *ty = tx + PL;
  const int nz = P.nz, OP2 = OP * OP;
  const int tiles = (nz + LT - 1) / LT, IF = blockIdx.x / tiles, l0 = (blockIdx.x % tiles) * LT;
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT, l = l0 + lvl;
  const bool act = ID < DoF && l < nz;
  const size_t cs = (size_t)DoF * nz;
  const int si = lvl * RS + ID;
  const double *mt = P.met + ((size_t)IF * NCOMP * DoF + ID) * nz + l;
  size_t o = 0;
  double rho = 1.0, p = 0.0, pt = 0.0;
  int vort = -1;
  if (act) {
    o = l + (size_t)nz * P.glob[(size_t)IF * DoF + ID];
    bool need_rho = false, need_p = false, div_rho = false, need_pt = false;
    for (int k = 0; k < A.n; ++k) {
      need_rho = need_rho || A.f[k].op == CELL_C_RHO || A.f[k].op == CELL_POTT;
      need_p = need_p || A.f[k].op == CELL_PRES || A.f[k].op == CELL_POTT;
      div_rho = div_rho || A.f[k].op == CELL_C_RHO;
      need_pt = need_pt || A.f[k].op == CELL_POTT;
    }
    if (need_rho) rho = A.rho[o];
    if (div_rho) {
      srho[si] = rho;
      srr[si] = 1.0 / rho;
    }
    if (need_p) p = pressure_dry(P, A.rhoth[o]);
    if (need_pt) pt = pott_dry(P, rho, p);
  }
  // the columns' values first, all of a thread's loads in flight at once
  double x[CELL_MAX];
#pragma unroll
  for (int k = 0; k < CELL_MAX; ++k) {
    x[k] = 0.0;
    if (act && k < A.n && A.f[k].c && A.f[k].op != CELL_WB) x[k] = A.f[k].c[o];
  }
#pragma unroll
  for (int k = 0; k < CELL_MAX; ++k) {
    if (act && k < A.n) {
      const int op = A.f[k].op;
      sc[(size_t)k * PL + si] = op == CELL_PRES ? p : op == CELL_POTT ? pt : x[k];
    }
  }
  for (int k = 0; k < A.n; ++k) {
    const CellOp f = A.f[k];
    if (f.op == CELL_VORT) {   // uniform: at most one per launch
      vort = k;
      if (act) {
        const double u = f.u[o], v = f.v[o];
        tx[si] = (mt[C_D11_0 * cs] + mt[C_D11_1 * cs]) * v - (mt[C_D12_0 * cs] + mt[C_D12_1 * cs]) * u;
        ty[si] = (mt[C_D21_0 * cs] + mt[C_D21_1 * cs]) * v - (mt[C_D22_0 * cs] + mt[C_D22_1 * cs]) * u;
      }
    } else if (f.op == CELL_WB && act) {
      // 0.5 (w(l) + w(l-1)), in the lowest layer 0.5 (w(1) + w0) with w0 =
      // -(u d31 + v d32) / d33 of the lower node (no normal flow); the
      // reference halves the weight, the same value
      const double below = l == 0 ? -(f.u[o] * mt[C_D31_0 * cs] + f.v[o] * mt[C_D32_0 * cs]) / mt[C_D33_0 * cs] : f.c[o - 1];
      sc[(size_t)k * PL + si] = 0.5 * (f.c[o] + below);
    }
  }
  __syncthreads();
  if (vort >= 0) {
    if (act) {
      const int i = ID % N, j = ID / N, row = lvl * RS;
      double acc = 0.0;
#pragma unroll
      for (int I = 0; I < N; ++I) acc += P.D[i + N * I] * tx[row + I + N * j];
#pragma unroll
      for (int J = 0; J < N; ++J) acc += P.D[j + N * J] * ty[row + i + N * J];
      sc[(size_t)vort * PL + si] = acc / (mt[C_J0 * cs] + mt[C_J1 * cs]);
    }
    __syncthreads();
  }
  // the cells: thread t holds the weights of sub-cell t % OP2
  const int step = 256 / OP2;          // (quantity, level) pairs in flight
  const int cI = t % OP2, p0 = t / OP2;
  if (p0 >= step) return;
  double w[DoF];
#pragma unroll
  for (int n = 0; n < DoF; ++n) w[n] = inter[cI + (size_t)OP2 * n];
  const int nl = min(LT, nz - l0);
  const size_t per = (size_t)OP2 * nz * P.NF;
  double *out = cell + cI + (size_t)OP2 * (l0 + (size_t)nz * IF);
  for (int q = p0; q < A.n * nl; q += step) {
    const int k = q / nl, lz = q - k * nl;
    const double *s = sc + (size_t)k * PL + lz * RS;
    double acc = 0.0;
    if (A.f[k].op == CELL_C_RHO) {
      const double *sr = srho + lz * RS, *si2 = srr + lz * RS;
#pragma unroll
      for (int n = 0; n < DoF; ++n) acc += exact_quotient(w[n] * s[n], sr[n], si2[n]);
    } else {
      const double2 *s2 = reinterpret_cast<const double2 *>(s);
#pragma unroll
      for (int n = 0; n + 1 < DoF; n += 2) {
        const double2 x = s2[n / 2];
        acc += w[n] * x.x;
        acc += w[n + 1] * x.y;
      }
      if (DoF % 2) acc += w[DoF - 1] * s[DoF - 1];
    }
    out[(size_t)k * per + (size_t)lz * OP2] = acc;
  }
}

}  // namespace cgd
