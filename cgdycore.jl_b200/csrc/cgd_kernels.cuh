// cgd_kernels.cuh - sm_100a kernels of the FP64 hot path.
//
// Layouts in HBM
//   state U, Temp1, F, k   (nz, NumG, NV) level fastest (the reference layout)
//   met                    [IF][comp][ID][nz]  21 components per element node
//                          and level (14 used dXdxI entries, J bottom/top,
//                          2*Omega*sin(lat) at the layer midpoint, the four
//                          J-only coefficients of RecU4 at the interface above)
//   C  (contributions)     [IF][slot][ID][nz]  element-local DSS inputs; NV + 1
//                          slots (the tendency fields, then the lower-node
//                          part of the phase-2 w contribution, one level down)
//   M                      (nz, NumG, 2)
//
// Direct-stiffness summation is an owner gather: the element kernels write
// every element-node contribution to C, and one thread per (global DOF,
// level) sums the contributions of the element nodes that share the DOF in
// ascending (element, node) order.  No atomics: results are bit-reproducible
// and equal to the CPU restatement's.
//
// Every floating-point expression below is written in the reference's
// evaluation order (see CGD_FAST below for the two builds).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>
#include "../../include/cgd_math.h"

// Two builds come from this source, both compiled without multiply-add
// contraction (-fmad=false).  The exact build evaluates the reference's
// expressions literally - every division is a division - so results are
// bit-identical to the CPU restatement.  The fast build (CGD_FAST) replaces
// the final division of a chain by the time-invariant sums J0+J1 (element
// Jacobian) and M0+M1 (lumped mass), or by rho, with a multiply by a
// reciprocal computed once per node and level (one rounding more, at the
// end of the chain).
#ifdef CGD_FAST
#define CGD_DIVJ(x) ((x) * rJs)
#define CGD_DIVM(x) ((x) * rMC)
#else
#define CGD_DIVJ(x) ((x) / Js)
#define CGD_DIVM(x) ((x) / MC)
#endif

namespace cgd {

// Arithmetic of the horizontal derivative sums, generic in the compute type R.
// For R = double the expressions are the reference's, unfused, in its order
// (acc + c*x; acc + (c1*x1 + c2*x2)); for R = float (the mixed form) they are
// fused multiply-adds.
__device__ __forceinline__ double rsum1(double acc, double c, double x) { return acc + c * x; }
__device__ __forceinline__ double rsum2(double acc, double c1, double x1, double c2, double x2)
{
  return acc + (c1 * x1 + c2 * x2);
}
__device__ __forceinline__ float rsum1(float acc, float c, float x) { return __fmaf_rn(c, x, acc); }
__device__ __forceinline__ float rsum2(float acc, float c1, float x1, float c2, float x2)
{
  return __fmaf_rn(c1, x1, __fmaf_rn(c2, x2, acc));
}

// 8- and 4-byte asynchronous copies global -> shared (cp.async, sm_80 and
// later) and the wait for all of a thread's copies
__device__ __forceinline__ void cp_async8(double *smem_dst, const double *gsrc)
{
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Ask for the bytes at p in L2 (whole 16-byte units, from the one p lies in)
__device__ __forceinline__ void l2_prefetch(const void *p, size_t bytes)
{
  const size_t a = (size_t)p & ~(size_t)15, e = ((size_t)p + bytes) & ~(size_t)15;
  if (e > a)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(__cvta_generic_to_global((const void *)a)),
                 "r"((unsigned)(e - a)));
}

constexpr int NCOMP = 21;
enum {
  C_D11_0 = 0, C_D11_1, C_D12_0, C_D12_1, C_D21_0, C_D21_1, C_D22_0, C_D22_1,
  C_D31_0, C_D31_1, C_D32_0, C_D32_1, C_D33_0, C_D33_1, C_J0, C_J1, C_FCOR,
  // RecU4 coefficients of the interface above the level (they depend on J only):
  // kR, kL of the left state and kL, kR of the right state
  C_RK0, C_RK1, C_RK2, C_RK3
};
// flat product grids (cgd_flat.cuh): horizontal factors of an element node:
// dXdxI(1:2,1:2) and J over z(l), z / J, dXdxI(3,3), 2*Omega*sin(lat), z / M
enum { H_11 = 0, H_12, H_21, H_22, H_RJ, H_J, H_33, H_FC, H_RM, H_N };
constexpr int MAXTR = 4;
constexpr int MAXNV = 5 + MAXTR;

// Everything a kernel needs about the grid, passed by value.
struct GP {
  int N, DoF, nz, NF, NumG, NumTr, NV;
  int NC;                   // contribution slots per element node: NV fields + the lower-node w of phase 2
  int rev;                  // walk the elements or columns of a launch from the last to the first (stage_piece)
  int IF0;                  // first element of a launch over a range of elements (k_hypervisc1, k_phase2)
  const double *met;        // [IF][comp][ID][nz]
  const double *M;          // (nz, NumG, 2)
  const double *dz;         // (nz, NumG)
  const int *glob;          // [IF*DoF + ID], 0-based
  const int *inv_ptr;       // NumG + 1
  const long long *inv_off; // (IF*NC*DoF + ID)*nz for every contributor
  const long long *inv_tab; // 4 per DOF: its first four inv_off entries, -1 past the count (-1 first: > 4)
  const int4 *etab;         // per element node the inv_tab row of its DOF, in units of nz
  const unsigned char *own; // per element node: 1 at the DOF's first contributor of this process
  int flat;                 // the grid is a flat product grid: the next two hold its factors
  const double *hm;         // [IF][H_N][ID]
  const double *zl;         // [6+2N][nz]: z (layer thickness over the first), 1/z, RecU4 coefficients (4),
                            // slope residue of node index I (N: sum of the layer's nodes; N: half the difference over z)
  double D[25], DW[25];     // D[i + N*j] = DS[i,j]
  const double *pref;       // mixed form: per-level FP64 reference pressure and theta
  const double *thref;
  double Grav, Rd, p0, kappa, nuCurl, nuGrad, nuDiv;
  // column physics of the tendency tail (cgd_set_physics): the dry
  // Held-Suarez forcing and the Rayleigh damping of w near the top
  int held_suarez, damping;
  double hs[8];             // k_a, k_f, k_s, DeltaT_y, DeltaTh_z, T_equator, T_min, sigma_b
  const double *coslat, *sinlat;   // (NumG) latitude of each column's surface node
  const double *dampc;             // (nz, NumG) damping rate at the layer midpoint
};

// The element of a launch with one blockIdx.y per element
__device__ __forceinline__ int launch_element(const GP &P)
{
  return P.IF0 + (int)(P.rev ? gridDim.y - 1 - blockIdx.y : blockIdx.y);
}

// Rosenbrock-W coefficients (src/Integration/RosenbrockMethod.jl:26-47).
struct RK {
  double a[3][3], c[3][3], m[3], gamma;
};

__device__ __forceinline__ double pressure_dry(const GP &P, double rhoth)
{
  // src/Models/Equation.jl:25-38, fast_powGPU (Equation.jl:79)
  return P.p0 * cgd_exp(1.0 / (1.0 - P.kappa) * cgd_log(P.Rd * rhoth / P.p0));
}

// The column physics of the tendency tail at level l of column g
// (src/GPU/FcnGPU.jl:953-966): ForceKernel! with the dry Held-Suarez Force
// (src/GPU/OperatorKernel.jl:1073-1080, src/Examples/initial.jl:513-531) and
// DampKernel! with DampingW (OperatorKernel.jl:1061-1071,
// src/GPU/dampingGPU.jl:1-19), for the state values rho, u, v, w, rho*theta
// and the pressure p there: adds to f[1] (u), f[2] (v), f[3] (w), f[4]
// (rho*theta).  fast_powGPU(x, y) = exp(y log x) (src/Models/Equation.jl:79).
__device__ __forceinline__ void physics_terms(const GP &P, int l, int g, double rho, double u, double v, double w,
                                              double rhoth, double p, double *f)
{
  if (P.held_suarez) {
    const double k_a = P.hs[0], k_f = P.hs[1], k_s = P.hs[2], DeltaT_y = P.hs[3], DeltaTh_z = P.hs[4];
    const double T_equator = P.hs[5], T_min = P.hs[6], sigma_b = P.hs[7];
    const double Sigma = p / P.p0;
    const double SigmaPowKappa = cgd_exp(P.kappa * cgd_log(Sigma));
    const double height_factor = cgd_max(0.0, (Sigma - sigma_b) / (1.0 - sigma_b));
    const double coslat = P.coslat[g], sinlat = P.sinlat[g];
    f[1] += -(k_f * height_factor) * u;
    f[2] += -(k_f * height_factor) * v;
    const double kT = k_a + (k_s - k_a) * height_factor * coslat * coslat * coslat * coslat;
    double Teq = (T_equator - DeltaT_y * sinlat * sinlat - DeltaTh_z * cgd_log(Sigma) * coslat * coslat) *
                 SigmaPowKappa;
    Teq = cgd_max(T_min, Teq);
    const double T = p / (rho * P.Rd);
    const double DeltaT = kT * (T - Teq);
    f[4] += -rhoth / T * DeltaT;
  }
  if (P.damping) f[3] += -P.dampc[l + (size_t)P.nz * g] * w;
}

// ---------------------------------------------------------------------------
// Phase 1: HyperViscKernel! + HyperViscTracerKernel!
// (src/GPU/ViscKernel.jl:1-84,169-218).  One CTA per (element, tile of LT
// levels); thread (node, level).  Purely horizontal: no vertical halo.
// R is the compute type of the derivative sums: double, or float for the
// mixed form, where theta enters as its perturbation from the level's FP64
// reference value.
// ---------------------------------------------------------------------------
// shared arrays of phase 1: planes 0-3 curl/contra of (u,v), 4 theta, 5-8
// the first derivatives, then per tracer its ratio and the two components of
// its gradient, each LT levels x DoF nodes
template <int N, int NT, typename R, int LT_ = 256 / (N * N)>
struct HV1Smem {
  static constexpr int DoF = N * N, LT = LT_;
  // row stride of a plane, odd: the levels of a half warp, a row apart, fall
  // into different banks (with the 16 of p = 3 they all shared one)
  static constexpr int RS = DoF | 1;
  static constexpr int PLANES = 9 + 3 * NT;
  static constexpr size_t BYTES = (size_t)PLANES * LT * RS * sizeof(R);
};

// Level tile of k_hypervisc1.  At p = 4 in FP64, 16 levels (400 threads,
// three CTAs per SM): a warp then reads runs of 16 consecutive levels of two
// nodes instead of 10 levels of three or four, so the metric and state loads
// touch fewer L1 lines: 0.416 -> 0.310 ms on the drop-in grid.  Elsewhere 256 / N^2 levels (256
// threads, four CTAs per SM), which the FP32 form also keeps (0.286 ms against
// 0.316 ms with 16 levels).
template <int N, typename R>
struct HV1Tile {
  static constexpr bool WIDE = N == 5 && sizeof(R) == sizeof(double);
  static constexpr int LT = WIDE ? 16 : 256 / (N * N);
  static constexpr int THREADS = WIDE ? LT * N * N : 256;
  static constexpr int MINB = WIDE ? 3 : 4;
};

// Phase 1 also forms the pressure (Pr, unless null): rho*theta is at hand, and
// the exp and log run beside a kernel that the shared-memory pipe bounds.  A
// DOF's value is written by its first element node.  A kernel of its own took
// 0.041 ms per stage on the drop-in grid (now 0.027 ms more in phase 1) and 6 of
// 150 us per step on the smallest configurations.
__device__ __forceinline__ void stage_pressure(const GP &P, double *Pr, int n, int g, int l, double rhoth)
{
  if (Pr && P.own[n]) Pr[l + (size_t)P.nz * g] = pressure_dry(P, rhoth);
}

// sbuf: the shared arrays (a kernel's dynamic buffer)
template <int N, int NT, typename R, int LT = 256 / (N * N)>
__device__ __forceinline__ void hypervisc1_body(const GP &P, const double *__restrict__ U, double *__restrict__ C,
                                                double *__restrict__ Pr, const int tile, const int IF, R *sbuf)
{
  constexpr bool MIX = sizeof(R) == sizeof(float);
  constexpr int DoF = N * N, RS = HV1Smem<N, NT, R, LT>::RS;
  R(*s)[LT * RS] = reinterpret_cast<R(*)[LT * RS]>(sbuf);
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT;
  const int I = ID % N, Jn = ID / N;
  const int l = tile * LT + lvl;
  const int nz = P.nz, NumG = P.NumG;
  const bool act = (ID < DoF) && (l < nz);
  const int si = lvl * RS + ID, row = lvl * RS;
  const size_t cs = (size_t)DoF * nz;
  int g = 0;
  R d11 = 0, d12 = 0, d21 = 0, d22 = 0;
  double JsD = 1, MCD = 1;
  R DI[N], DJ[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    DI[k] = (R)P.D[I + N * k];
    DJ[k] = (R)P.D[Jn + N * k];
  }
  const double *mt = P.met + ((size_t)IF * NCOMP * DoF + ID) * nz + l;
  if (act) {
    g = P.glob[IF * DoF + ID];
    d11 = (R)(mt[C_D11_0 * cs] + mt[C_D11_1 * cs]);
    d12 = (R)(mt[C_D12_0 * cs] + mt[C_D12_1 * cs]);
    d21 = (R)(mt[C_D21_0 * cs] + mt[C_D21_1 * cs]);
    d22 = (R)(mt[C_D22_0 * cs] + mt[C_D22_1 * cs]);
    JsD = mt[C_J0 * cs] + mt[C_J1 * cs];
    const double *Ug = U + l + (size_t)nz * g;
    const size_t fs = (size_t)nz * NumG;
    const R u = (R)Ug[1 * fs], v = (R)Ug[2 * fs];
    s[0][si] = d11 * v - d12 * u;   // Curl12
    s[1][si] = d21 * v - d22 * u;
    s[2][si] = d11 * u + d12 * v;   // Contra12
    s[3][si] = d21 * u + d22 * v;
    if (MIX) s[4][si] = (R)(Ug[4 * fs] / Ug[0] - P.thref[l]);
    else s[4][si] = (R)(Ug[4 * fs] / Ug[0]);
#pragma unroll
    for (int q = 0; q < NT; ++q) s[9 + 3 * q][si] = (R)(Ug[(5 + q) * fs] / Ug[0]);
    MCD = P.M[l + (size_t)nz * g] + P.M[l + (size_t)nz * (g + (size_t)NumG)];
    stage_pressure(P, Pr, IF * DoF + ID, g, l, Ug[4 * fs]);
  }
  const R Js = (R)JsD, MC = (R)MCD;
  const R rJs = (R)(1.0 / JsD), rMC = (R)(1.0 / MCD);
  (void)rJs; (void)rMC; (void)Js; (void)MC;
  __syncthreads();
  if (act) {
    const R *uC = s[0] + row, *vC = s[1] + row, *uD = s[2] + row, *vD = s[3] + row, *Th = s[4] + row;
    R Dxc = DI[0] * Th[N * Jn];
    R Dyc = DJ[0] * Th[I];
    R cu = DI[0] * uC[N * Jn] + DJ[0] * vC[I];
    R dv = DI[0] * uD[N * Jn] + DJ[0] * vD[I];
#pragma unroll
    for (int k = 1; k < N; ++k) {
      Dxc = rsum1(Dxc, DI[k], Th[k + N * Jn]);
      Dyc = rsum1(Dyc, DJ[k], Th[I + N * k]);
      cu = rsum2(cu, DI[k], uC[k + N * Jn], DJ[k], vC[I + N * k]);
      dv = rsum2(dv, DI[k], uD[k + N * Jn], DJ[k], vD[I + N * k]);
    }
    s[5][si] = CGD_DIVJ(cu);
    s[6][si] = CGD_DIVJ(dv);
    R GradDx = CGD_DIVJ(d11 * Dxc + d21 * Dyc);   // Grad12 with J
    R GradDy = CGD_DIVJ(d12 * Dxc + d22 * Dyc);
    s[7][si] = d11 * GradDx + d12 * GradDy;         // Contra12
    s[8][si] = d21 * GradDx + d22 * GradDy;
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      const R *Tr = s[9 + 3 * q] + row;
      R Dxt = DI[0] * Tr[N * Jn];
      R Dyt = DJ[0] * Tr[I];
#pragma unroll
      for (int k = 1; k < N; ++k) {
        Dxt = rsum1(Dxt, DI[k], Tr[k + N * Jn]);
        Dyt = rsum1(Dyt, DJ[k], Tr[I + N * k]);
      }
      R GDx = CGD_DIVJ(d11 * Dxt + d21 * Dyt);
      R GDy = CGD_DIVJ(d12 * Dxt + d22 * Dyt);
      s[10 + 3 * q][si] = d11 * GDx + d12 * GDy;
      s[11 + 3 * q][si] = d21 * GDx + d22 * GDy;
    }
  }
  __syncthreads();
  using CT = typename std::conditional<MIX, float, double>::type;   // stored contributions
  CT *out = reinterpret_cast<CT *>(C) + ((size_t)IF * P.NC * DoF + ID) * nz + l;
  R WI[N], WJ[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    WI[k] = (R)P.DW[I + N * k];
    WJ[k] = (R)P.DW[Jn + N * k];
  }
  if (act) {
    const R *Cu = s[5] + row, *Dv = s[6] + row, *Cx = s[7] + row, *Cy = s[8] + row;
    R DxCurl = WI[0] * Cu[N * Jn], DyCurl = WJ[0] * Cu[I];
    R DxDiv = WI[0] * Dv[N * Jn], DyDiv = WJ[0] * Dv[I];
    R DivTh = WI[0] * Cx[N * Jn] + WJ[0] * Cy[I];
#pragma unroll
    for (int k = 1; k < N; ++k) {
      DxCurl = rsum1(DxCurl, WI[k], Cu[k + N * Jn]);
      DyCurl = rsum1(DyCurl, WJ[k], Cu[I + N * k]);
      DxDiv = rsum1(DxDiv, WI[k], Dv[k + N * Jn]);
      DyDiv = rsum1(DyDiv, WJ[k], Dv[I + N * k]);
      DivTh = rsum2(DivTh, WI[k], Cx[k + N * Jn], WJ[k], Cy[I + N * k]);
    }
    R FuC = d12 * DxCurl + d22 * DyCurl;       // Rot12
    R FvC = -d11 * DxCurl - d21 * DyCurl;
    R FuD = d11 * DxDiv + d21 * DyDiv;         // Grad12
    R FvD = d12 * DxDiv + d22 * DyDiv;
    out[0 * cs] = (CT)CGD_DIVM(-FuC);
    out[1 * cs] = (CT)CGD_DIVM(-FvC);
    out[2 * cs] = (CT)CGD_DIVM(FuD);
    out[3 * cs] = (CT)CGD_DIVM(FvD);
    out[4 * cs] = (CT)CGD_DIVM(DivTh);
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      const R *Tx = s[10 + 3 * q] + row, *Ty = s[11 + 3 * q] + row;
      R DivTr = WI[0] * Tx[N * Jn] + WJ[0] * Ty[I];
#pragma unroll
      for (int k = 1; k < N; ++k) DivTr = rsum2(DivTr, WI[k], Tx[k + N * Jn], WJ[k], Ty[I + N * k]);
      out[(5 + q) * cs] = (CT)CGD_DIVM(DivTr);
    }
  }
}

// Shared arrays: HV1Smem<N, NT, R, HV1Tile<N, R>::LT>::BYTES of dynamic shared memory.
template <int N, int NT, typename R>
__global__ void __launch_bounds__(HV1Tile<N, R>::THREADS, HV1Tile<N, R>::MINB)
    k_hypervisc1(const GP P, const double *__restrict__ U, double *__restrict__ C, double *__restrict__ Pr)
{
  extern __shared__ __align__(16) unsigned char hv1_dyn[];
  hypervisc1_body<N, NT, R, HV1Tile<N, R>::LT>(P, U, C, Pr, blockIdx.x, launch_element(P),
                                               reinterpret_cast<R *>(hv1_dyn));
}

// Contributions and the phase-1 cache: double, or float in the mixed form
// (C32, a compile-time choice of every kernel that reads or writes them).
template <bool C32>
__device__ __forceinline__ double cload(const double *C, long long i)
{
  return C32 ? (double)reinterpret_cast<const float *>(C)[i] : C[i];
}

// Sum over the NQ contributors (element-node offsets o) of one global DOF at
// one level, for every field, each sum from 0.0 in ascending order.
// WSPLIT (the phase-2 tendency): a node's contribution to w at interface l is
// its upper part (slot 3, level l) plus its lower part (slot NV, stored at
// level l), zero at the top level.
template <int NQ, bool WSPLIT, bool C32>
__device__ __forceinline__ void gather_nq(const GP &P, const double *__restrict__ C, const long long *o, bool wtop,
                                          size_t fstr, double *acc)
{
  double wlo[NQ];
  if (WSPLIT) {
#pragma unroll
    for (int j = 0; j < NQ; ++j) wlo[j] = !wtop ? cload<C32>(C, o[j] + P.NV * fstr) : 0.0;
  }
#pragma unroll
  for (int f = 0; f < MAXNV; ++f) {
    if (f < P.NV) {
      double x[NQ];
#pragma unroll
      for (int j = 0; j < NQ; ++j) x[j] = !(WSPLIT && f == 3 && wtop) ? cload<C32>(C, o[j] + f * fstr) : 0.0;
      if (WSPLIT && f == 3) {
#pragma unroll
        for (int j = 0; j < NQ; ++j) x[j] = wtop ? 0.0 : x[j] + wlo[j];
      }
      double a = 0.0;
#pragma unroll
      for (int j = 0; j < NQ; ++j) a += x[j];
      acc[f] = a;
    }
  }
}

// Sum the contributions of the element nodes sharing global DOF g at level l
// (ascending element, node order) for every field.  Every cubed-sphere node
// has 1 to 4 contributors; each count has its own fully unrolled path (the
// count is uniform over a column, so over a warp of the column kernel), whose
// loads are all independent.
template <bool WSPLIT, bool C32>
__device__ __forceinline__ void gather_node(const GP &P, const double *__restrict__ C, int g, int l, size_t fstr,
                                            double *acc)
{
  // one 32-byte row of the table gives the count and the offsets, so the
  // contribution loads wait on a single index load
  const longlong2 *t = reinterpret_cast<const longlong2 *>(P.inv_tab) + 2 * (size_t)g;
  const longlong2 ta = t[0], tb = t[1];
  const bool wtop = WSPLIT && l == P.nz - 1;
  long long o[4] = {ta.x + l, ta.y + l, tb.x + l, tb.y + l};
  const int nq = ta.x < 0 ? 0 : 1 + (ta.y >= 0) + (tb.x >= 0) + (tb.y >= 0);
  switch (nq) {
    case 1:
      gather_nq<1, WSPLIT, C32>(P, C, o, wtop, fstr, acc);
      return;
    case 2:
      gather_nq<2, WSPLIT, C32>(P, C, o, wtop, fstr, acc);
      return;
    case 3:
      gather_nq<3, WSPLIT, C32>(P, C, o, wtop, fstr, acc);
      return;
    case 4:
      gather_nq<4, WSPLIT, C32>(P, C, o, wtop, fstr, acc);
      return;
    default:
      break;
  }
  const int q0 = P.inv_ptr[g], q1 = P.inv_ptr[g + 1];
#pragma unroll
  for (int f = 0; f < MAXNV; ++f) {
    if (f < P.NV) {
      double a = 0.0;
      for (int q = q0; q < q1; ++q) {
        const long long oq = P.inv_off[q] + l;
        double x = cload<C32>(C, oq + f * fstr);
        if (WSPLIT && f == 3) x = wtop ? 0.0 : x + cload<C32>(C, oq + P.NV * fstr);
        a += x;
      }
      acc[f] = a;
    }
  }
}

// ---------------------------------------------------------------------------
// Owner gather (DSS): out(l, g, f) = sum over contributors in ascending
// (element, node) order.  Thread per (g, l), level fastest.
// ---------------------------------------------------------------------------
template <bool WSPLIT, bool C32>
__global__ void __launch_bounds__(256) k_gather(const GP P, const double *__restrict__ C,
                                                double *__restrict__ out)
{
  const int nz = P.nz;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (long long)nz * P.NumG) return;
  const int g = (int)(tid / nz), l = (int)(tid % nz);
  double acc[MAXNV];
  gather_node<WSPLIT, C32>(P, C, g, l, (size_t)P.DoF * nz, acc);
#pragma unroll
  for (int f = 0; f < MAXNV; ++f)
    if (f < P.NV) out[l + (long long)nz * (g + (long long)P.NumG * f)] = acc[f];
}

// The DSS'd phase-1 cache of element node n (= IF*DoF + ID) at level l, fields
// F0 .. F0+NF-1, summed from the contributions C1 as gather_node sums them
// (ascending contributors, from 0.0; the mixed form rounds the sum to FP32).
// Phase 2 forms it itself: 1.96 contributor reads an element node, mostly from
// L2, instead of a kernel that wrote the summed cache (0.11 ms per stage on the
// drop-in grid) and its read.
template <bool C32, int F0, int NFLD, typename R>
__device__ __forceinline__ void cache_sums(const GP &P, const double *__restrict__ C1, int n, int l, R *c)
{
  using CT = typename std::conditional<C32, float, double>::type;
  const CT *C = reinterpret_cast<const CT *>(C1);
  const size_t fstr = (size_t)P.DoF * P.nz;
  const int4 e = P.etab[n];
  if (e.x >= 0) {
    const CT *p0 = C + (size_t)e.x * P.nz + l, *p1 = C + (size_t)max(e.y, 0) * P.nz + l;
    const CT *p2 = C + (size_t)max(e.z, 0) * P.nz + l, *p3 = C + (size_t)max(e.w, 0) * P.nz + l;
#pragma unroll
    for (int f = 0; f < NFLD; ++f) {
      const size_t o = (F0 + f) * fstr;
      const double x0 = p0[o];
      const double x1 = e.y >= 0 ? (double)p1[o] : 0.0, x2 = e.z >= 0 ? (double)p2[o] : 0.0;
      const double x3 = e.w >= 0 ? (double)p3[o] : 0.0;
      c[f] = (R)((((0.0 + x0) + x1) + x2) + x3);
    }
    return;
  }
  const int g = P.glob[n];
#pragma unroll
  for (int f = 0; f < NFLD; ++f) {
    double a = 0.0;
    for (int q = P.inv_ptr[g]; q < P.inv_ptr[g + 1]; ++q) a += (double)C[P.inv_off[q] + l + (F0 + f) * fstr];
    c[f] = (R)a;
  }
}

// ---------------------------------------------------------------------------
// Column part of a Rosenbrock-W stage, fused (one warp per column, lanes over
// levels): owner gather of the tendency, stage corrections
// fV = F + sum_j c_ij/dt k_j, the vertical acoustic Jacobian of the step's
// initial state (JacSchurKernel!, src/DyCore/JacSchur.jl:29-75), the Schur
// tridiagonal system (TriDiagKernel!, SchurSolveFKernel!, triSolve!,
// SchurSolveBKernel!: src/Integration/SchurSolve.jl:1-114) and the stage
// update of RosenbrockSchur! (src/Integration/RosenbrockSchur.jl:13-32).
// MODE 0: stage 1 -> k1, Vst = Vn + a21 k1; the Jacobian bands are formed
//         and kept (level fastest) for stages 2 and 3
// MODE 1: stage 2 -> k2, Vst = (Vn + a31 k1) + a32 k2
// MODE 2: stage 3 -> Vout = ((Vn + m1 k1) + m2 k2) + m3 k3   (Vout may alias Vn)
// MODE 3: standalone Schur solve with stored bands: k, v updated (cgd_schur_solve)
// Only rho, w and rho*theta enter the Schur system; every other field has
// k = fac * fV and is finished right after its gather.
// ---------------------------------------------------------------------------
struct ColArgs {
  const double *C;       // contributions of phase 2 (MODE 0..2)
  const double *Vn;      // step initial state (MODE 0..2)
  // MODE 1 reads k1; MODE 2 k1 and k2, or (COL_KSUM) their sum alone from k2
  const double *k1, *k2;
  double *kout;          // MODE 0,1,3 (MODE 1 with COL_KSUM: k1 + k2)
  double *k2out;         // MODE 1 with COL_KSUM: k2 itself, for the adjoint's tape (else null)
  double *Vout;          // MODE 0,1 (stage state), 2 (new state)
  double *v;             // MODE 3: right-hand side (overwritten)
  // MODE 3: the four Jacobian bands JRhoW, JWRho, JWRhoTh, JRhoThW, each
  // (2, nz-1, NumG) in the reference layout (the JCache arrays)
  const double *jb4[4];
  double *jbg;           // MODE 0 writes, 1-2 read: [8][NumG][nz-1] bands of the step
  // MODE 0..2 with column physics: the stage state the tendency is of and its
  // pressure (Vs may be Vout: each lane reads its own levels before writing them)
  const double *Vs, *ps;
  double dt, fac;
  double cd[2];          // c[MODE][j] / dt
  double ifac, ifac2;    // 1 / fac, 1 / fac / fac
  RK rk;

  void set_dt(int mode, double dt_, double fac_)
  {
    dt = dt_;
    fac = fac_;
    ifac = 1.0 / fac;
    ifac2 = ifac / fac;
    for (int j = 0; j < 2; ++j) cd[j] = mode <= 2 ? rk.c[mode][j] / dt : 0.0;
  }
};

// The third stage needs k1 and k2 only in c31/dt k1 + c32/dt k2, m1 k1 + m2 k2,
// and the SSP-Knoth scheme has c31 = c32, m1 = m2 and a31 = a32
// (src/Integration/RosenbrockMethod.jl:26-47).  The fast build's second stage
// therefore keeps k1 + k2 instead of k2: one array less to read in the third.
#ifdef CGD_FAST
constexpr bool COL_KSUM = true;
#else
constexpr bool COL_KSUM = false;
#endif

constexpr int COL_WARPS = 8;
// Per warp: fv of rho, w, rho*theta and 8 bands, each nz long; tri[3] and x
// take the rows of JWRho and JWRhoTh, which are dead by then, and the first
// stage has two more rows.  (15 rows before: the second and third stage took
// 0.368/0.362 ms instead of 0.353/0.345 on the drop-in grid, and at nz 64,
// where only three CTAs fitted an SM, 1.45/1.42 instead of 1.24/1.18 ms on
// nPanel 60.  Copying the step's initial rho, w, rho*theta into shared memory
// at the start, for the update at the end, is slower than reading them there.)
template <int MODE>
constexpr int COL_ARR = MODE == 0 ? 13 : 11;
constexpr int COL_ARR_MAX = COL_ARR<0>;
// CTAs per SM the column kernel's registers are sized for: five for the first
// stage (48 registers; 0.474 -> 0.464 ms on the drop-in grid), four for the
// others (64 registers; five cost them 4-20 %)
template <int MODE>
constexpr int col_min_blocks() { return MODE == 0 ? 5 : 4; }

// dPresdRhoTh (src/Models/Equation.jl:33-36) of one level
__device__ __forceinline__ double dpdrhoth(const GP &P, double RhoTh0)
{
  const double RhoTh = RhoTh0 + 0.0;
  return P.Rd * cgd_pow(P.Rd * RhoTh / P.p0, P.kappa / (1.0 - P.kappa));
}

__device__ __forceinline__ void jac_bands(const GP &P, double RhoL, double RhoR, double RhoThL0, double RhoThR0,
                                          double dPdThL, double dPdThR, double dzL, double dzR, double *jb)
{
  // JacSchurKernel! (src/DyCore/JacSchur.jl:40-73); AuxG[:,:,4] == 0 for Dry
  double RhoThL = RhoThL0 + 0.0, RhoThR = RhoThR0 + 0.0;
  double RhoF = (RhoL * dzL + RhoR * dzR) / (dzL + dzR);
  jb[0] = -RhoF / dzL;             // JRhoW[1]
  jb[1] = RhoF / dzR;              // JRhoW[2]
  jb[4] = -dPdThR / RhoF / (0.5 * (dzL + dzR));   // JWRhoTh[1]
  jb[5] = dPdThL / RhoF / (0.5 * (dzL + dzR));    // JWRhoTh[2]
  jb[2] = -P.Grav * dzR / RhoF / (dzL + dzR);     // JWRho[1]
  jb[3] = -P.Grav * dzL / RhoF / (dzL + dzR);     // JWRho[2]
  double RhoThF = (RhoThL * dzL + RhoThR * dzR) / (dzL + dzR);
  jb[6] = -RhoThF / dzL;           // JRhoThW[1]
  jb[7] = RhoThF / dzR;            // JRhoThW[2]
}

#ifdef CGD_FAST
// jac_bands with reciprocals shared by its quotients: riL, riR the
// reciprocals of dzL and dzR (two divisions instead of fifteen)
__device__ __forceinline__ void jac_bands_rcp(const GP &P, double RhoL, double RhoR, double RhoThL, double RhoThR,
                                              double dPdThL, double dPdThR, double dzL, double dzR, double riL,
                                              double riR, double *jb)
{
  const double dzs = dzL + dzR, rs = 1.0 / dzs, num = RhoL * dzL + RhoR * dzR;
  const double RhoF = num * rs, rF = dzs * (1.0 / num);   // rF = 1 / RhoF
  jb[0] = -RhoF * riL;
  jb[1] = RhoF * riR;
  const double q = rF * rs, w = 2.0 * q, b = P.Grav * q;
  jb[4] = -dPdThR * w;
  jb[5] = dPdThL * w;
  jb[2] = -b * dzR;
  jb[3] = -b * dzL;
  const double RhoThF = (RhoThL * dzL + RhoThR * dzR) * rs;
  jb[6] = -RhoThF * riL;
  jb[7] = RhoThF * riR;
}
#endif

// Solve M x = b for one column with the warp's 32 lanes (the fast build's
// triSolve!).  M(i,i) = t1(i), M(i+1,i) = t2(i), M(i,i+1) = t0(i+1), n <= 64
// rows; lane L holds rows 2L and 2L+1.  The Thomas recurrences become scans:
//   pivots d(i) = t1(i) - t2(i-1) t0(i) / d(i-1) = p(i)/q(i), (p, q) the first
//     column of the product M_i ... M_0 with M_i = [[t1(i), -t2(i-1) t0(i)], [1, 0]]
//     (products rescaled by powers of two, which is exact);
//   forward b'(i) = b(i) - t2(i-1)/d(i-1) b'(i-1), an affine prefix scan;
//   back x(i) = (b'(i) - t0(i+1) x(i+1)) / d(i), an affine suffix scan.
struct Mat2 {
  double a, b, c, d;
};
__device__ __forceinline__ Mat2 mat2_mul(const Mat2 &x, const Mat2 &y)
{
  return {x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
}
// m scaled by 2^-e, e the binary exponent of its largest entry (largest |entry|
// = f 2^e, 0.5 <= f < 1).  When that entry is a normal number whose 2^-e is
// normal too (biased exponent 1 .. 2044), the scaling is one multiply by 2^-e,
// assembled from the exponent bits: a multiply by an exact power of two is
// the single correctly rounded x 2^-e, so it equals ldexp(x, -e) bit for bit.
// Other magnitudes (zero, subnormal, near overflow, not finite) take
// frexp/ldexp.
__device__ __forceinline__ Mat2 mat2_scaled(Mat2 m)
{
  const double mx = fmax(fmax(fabs(m.a), fabs(m.b)), fmax(fabs(m.c), fabs(m.d)));
  const int be = (int)((unsigned long long)__double_as_longlong(mx) >> 52);   // mx >= 0: no sign bit
  if (be >= 1 && be <= 2044) {
    // e = be - 1022; 2^-e has the biased exponent 1023 - e = 2045 - be
    const double sc = __longlong_as_double((long long)(2045 - be) << 52);
    m.a *= sc; m.b *= sc; m.c *= sc; m.d *= sc;
  } else if (mx > 0.0) {
    int e;
    frexp(mx, &e);
    m.a = ldexp(m.a, -e); m.b = ldexp(m.b, -e); m.c = ldexp(m.c, -e); m.d = ldexp(m.d, -e);
  }
  return m;
}
__device__ __forceinline__ Mat2 mat2_shfl_up(const Mat2 &m, int k)
{
  return {__shfl_up_sync(0xffffffffu, m.a, k), __shfl_up_sync(0xffffffffu, m.b, k),
          __shfl_up_sync(0xffffffffu, m.c, k), __shfl_up_sync(0xffffffffu, m.d, k)};
}
__device__ __forceinline__ void warp_tri_solve(const double *t0, const double *t1, const double *t2,
                                               const double *b, double *x, int n, int lane)
{
  constexpr unsigned FULL = 0xffffffffu;
  const Mat2 I2 = {1.0, 0.0, 0.0, 1.0};
  const int i0 = 2 * lane, i1 = i0 + 1;
  auto mi = [&](int i) -> Mat2 {
    if (i >= n) return I2;
    return {t1[i], i > 0 ? -t2[i - 1] * t0[i] : 0.0, 1.0, 0.0};
  };
  const Mat2 A0 = mi(i0), A1 = mi(i1);
  // pivots
  Mat2 S = mat2_scaled(mat2_mul(A1, A0));
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    Mat2 Sp = mat2_shfl_up(S, k);
    if (lane < k) Sp = I2;
    S = mat2_scaled(mat2_mul(S, Sp));
  }
  Mat2 E = mat2_shfl_up(S, 1);
  if (lane == 0) E = I2;
  const Mat2 P0 = mat2_scaled(mat2_mul(A0, E));
  const Mat2 P1 = mat2_scaled(mat2_mul(A1, P0));
  const double r0 = i0 < n ? P0.c / P0.a : 0.0;   // 1 / d(i0)
  const double r1 = i1 < n ? P1.c / P1.a : 0.0;   // 1 / d(i1)
  // forward substitution
  const double rprev = __shfl_up_sync(FULL, r1, 1);   // 1 / d(i0 - 1)
  const double a0 = i0 < n ? (i0 > 0 ? -t2[i0 - 1] * rprev : 0.0) : 1.0;
  const double a1 = i1 < n ? -t2[i0] * r0 : 1.0;
  const double c0 = i0 < n ? b[i0] : 0.0, c1 = i1 < n ? b[i1] : 0.0;
  double CA = a1 * a0, CB = a1 * c0 + c1;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    double pA = __shfl_up_sync(FULL, CA, k), pB = __shfl_up_sync(FULL, CB, k);
    if (lane < k) { pA = 1.0; pB = 0.0; }
    CB = CA * pB + CB;
    CA = CA * pA;
  }
  double yprev = __shfl_up_sync(FULL, CB, 1);
  if (lane == 0) yprev = 0.0;
  const double bp0 = a0 * yprev + c0, bp1 = a1 * bp0 + c1;
  // back substitution
  const double al0 = i0 + 1 < n ? -t0[i0 + 1] * r0 : 0.0, be0 = bp0 * r0;
  const double al1 = i1 + 1 < n ? -t0[i1 + 1] * r1 : 0.0, be1 = bp1 * r1;
  CA = al0 * al1;
  CB = al0 * be1 + be0;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    double nA = __shfl_down_sync(FULL, CA, k), nB = __shfl_down_sync(FULL, CB, k);
    if (lane + k >= 32) { nA = 1.0; nB = 0.0; }
    CB = CA * nB + CB;
    CA = CA * nA;
  }
  double xnext = __shfl_down_sync(FULL, CB, 1);
  if (lane == 31) xnext = 0.0;
  const double x1v = al1 * xnext + be1, x0v = al0 * x1v + be0;
  if (i0 < n) x[i0] = x0v;
  if (i1 < n) x[i1] = x1v;
}

// The update of the second and third stage at state entry o: k of the stage,
// x1 = k1 (third stage with COL_KSUM: k1 + k2), x2 = k2.
template <int MODE>
__device__ __forceinline__ void stage_update(const ColArgs &A, size_t o, double vn, double x1, double x2, double k)
{
  if (MODE == 1) {
    if (COL_KSUM) {
      const double ks = x1 + k;
      A.kout[o] = ks;
      if (A.k2out) A.k2out[o] = k;
      A.Vout[o] = vn + A.rk.a[2][0] * ks;
    } else {
      A.kout[o] = k;
      A.Vout[o] = vn + A.rk.a[2][0] * x1 + A.rk.a[2][1] * k;
    }
  } else {
    if (COL_KSUM) A.Vout[o] = vn + A.rk.m[0] * x1 + A.rk.m[2] * k;
    else A.Vout[o] = vn + A.rk.m[0] * x1 + A.rk.m[1] * x2 + A.rk.m[2] * k;
  }
}

// A column's loads come in four rounds (table row, levels 0-31, 32-63, update)
// that each wait for DRAM; the kernel moved 3.9 TB/s so.  Each warp therefore
// starts with requests for all of its column's contributions, one row of nz
// levels per lane, and the first warp for the CTA's columns of the states and
// stage quantities, which lie side by side.  Column stages of one step, nPanel
// 30, nz 45, NumTr 2: 0.387 + 0.415 + 0.384 -> 0.371 + 0.368 + 0.362 ms;
// nPanel 60, nz 64: 1.86 + 1.83 + 1.73 -> 1.58 + 1.45 + 1.42 ms.  A launch of
// less than one wave (four CTAs an SM) finds its data in L2: nPanel 6, nz 10
// 14.5 -> 16.5 us with the requests.  (Plain prefetches of the second round's
// and the update's lines: no gain; requests one wave ahead: slower, 0.50 ms.)
constexpr int COL_PREFETCH_MIN = 4 * 148;

template <int MODE, bool C32>
__device__ __forceinline__ void column_prefetch(const GP &P, const ColArgs &A, int g0, int warp, int lane)
{
  const int nz = P.nz, NV = P.NV, g = g0 + warp;
  const longlong2 *t = reinterpret_cast<const longlong2 *>(P.inv_tab) + 2 * (size_t)g;
  const longlong2 ta = t[0], tb = t[1];
  for (int r = lane; r < 4 * (NV + 1); r += 32) {
    const int j = r & 3, f = r >> 2;
    const long long off = j == 0 ? ta.x : j == 1 ? ta.y : j == 2 ? tb.x : tb.y;
    const size_t es = C32 ? sizeof(float) : sizeof(double);
    if (off >= 0) l2_prefetch(reinterpret_cast<const char *>(A.C) + (off + (size_t)f * P.DoF * nz) * es, nz * es);
  }
  if (warp > 0) return;
  const int rows = NV * (MODE == 0 ? 1 : MODE == 2 && !COL_KSUM ? 3 : 2), cols = min(COL_WARPS, P.NumG - g0);
  for (int r = lane; r < rows; r += 32) {
    const int q = r / NV, f = r % NV;
    const double *a = q == 0 ? A.Vn : q == 2 || (MODE == 2 && COL_KSUM) ? A.k2 : A.k1;
    l2_prefetch(a + (size_t)nz * (g0 + (size_t)f * P.NumG), (size_t)cols * nz * sizeof(double));
  }
}

template <int MODE, bool C32>
__device__ __forceinline__ void column_body(const GP &P, const ColArgs &A, const int bx)
{
  extern __shared__ double csm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g0 = bx * COL_WARPS;
  const int g = g0 + warp;
  const int nz = P.nz, n = nz - 1, NV = P.NV, NumG = P.NumG;
  const bool valid = g < NumG;   // no early return: the block synchronises below
  const int LS = nz;                    // per-warp arrays of nz entries
  double *sw = csm + (size_t)warp * COL_ARR<MODE> * LS;
  double *fv = sw;                      // [3][nz]: rho, w, rho*theta
  double *jb = sw + 3 * LS;             // [8][nz]
  double *tri = jb + 2 * LS;            // [3][nz], over JWRho, JWRhoTh
  double *xs = jb + 5 * LS;             // [nz], over JWRhoTh
  double *tmp = jb + 8 * LS;            // [2][nz], first stage
  const size_t fs = (size_t)nz * NumG;
  const double fac = A.fac;
  // k1, k2 of the Schur fields (rho, w, rho*theta), kept for the update
  double s1[2][3], s2[2][3];

  // stages 2 and 3: the stored bands of the step are copied into the warp's
  // band rows first, so that they are in flight with the gather's loads
  if ((MODE == 1 || MODE == 2) && valid) {
    const size_t js = (size_t)NumG * n;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int l = lane + 32 * it;
      if (l >= n) continue;
      const double *jg = A.jbg + (size_t)g * n + l;
#pragma unroll
      for (int r = 0; r < 8; ++r) cp_async8(jb + r * LS + l, jg + r * js);
    }
  }

  if (MODE <= 2 && valid && gridDim.x >= COL_PREFETCH_MIN) column_prefetch<MODE, C32>(P, A, g0, warp, lane);

  // 1. tendency (owner gather) + stage corrections; fields outside the Schur
  //    system finished here; bands
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int l = lane + 32 * it;
    if (!valid || l >= nz) continue;
    const size_t o0 = l + (size_t)nz * g;
    if (MODE <= 2) {
      const size_t fstr = (size_t)P.DoF * nz;
      double gacc[MAXNV];
      gather_node<true, C32>(P, A.C, g, l, fstr, gacc);
      if (P.held_suarez || P.damping) {   // the tendency tail, at the stage state
        const double *vs = A.Vs + o0;
        physics_terms(P, l, g, vs[0], vs[fs], vs[2 * fs], vs[3 * fs], vs[4 * fs], A.ps[o0], gacc);
      }
#pragma unroll
      for (int f = 0; f < MAXNV; ++f) {
        if (f >= NV) break;
        const size_t o = o0 + f * fs;
        double x = gacc[f];
        double x1 = 0.0, x2 = 0.0;
        if (MODE == 2 && COL_KSUM) {
          x1 = A.k2[o];
          x = x + A.cd[0] * x1;
        } else {
          if (MODE >= 1) {
            x1 = A.k1[o];
            x = x + A.cd[0] * x1;
          }
          if (MODE >= 2) {
            x2 = A.k2[o];
            x = x + A.cd[1] * x2;
          }
        }
        if (f == 0 || f == 3 || f == 4) {
          const int sf = f == 0 ? 0 : f - 2;   // 0, 1, 2
          fv[sf * LS + l] = x;
          s1[it][sf] = x1;
          s2[it][sf] = x2;
        } else {
          const double k = fac * x;
          const double vn = A.Vn[o];
          if (MODE == 0) {
            A.kout[o] = k;
            A.Vout[o] = vn + A.rk.a[1][0] * k;
          } else {
            stage_update<MODE>(A, o, vn, x1, x2, k);
          }
        }
      }
      if (MODE == 0) {
        // dPresdRhoTh once per level, shared with the interface below
#ifdef CGD_FAST
        // Rd (Rd rhotheta / p0)^(kappa/(1-kappa)) = p / rhotheta with the pressure at hand (0 at 0)
        const double rth = A.Vn[o0 + 4 * fs];
        tmp[l] = rth != 0.0 ? A.ps[o0] / rth : 0.0;
        tmp[LS + l] = 1.0 / P.dz[o0];
#else
        tmp[l] = dpdrhoth(P, A.Vn[o0 + 4 * fs]);
#endif
      }
    } else {
      fv[l] = A.v[o0];
      fv[LS + l] = A.v[o0 + 3 * fs];
      fv[2 * LS + l] = A.v[o0 + 4 * fs];
      for (int f = 1; f < NV; ++f)
        if (f != 3 && f != 4) A.kout[o0 + f * fs] = fac * A.v[o0 + f * fs];
      if (l < n) {
        for (int arr = 0; arr < 4; ++arr)
          for (int r = 0; r < 2; ++r) jb[(2 * arr + r) * LS + l] = A.jb4[arr][r + 2 * (l + (size_t)n * g)];
      }
    }
  }
  if (MODE == 1 || MODE == 2) cp_async_wait_all();   // this lane's band copies; the warp sync below publishes them
  if (MODE == 0) {
    __syncwarp();
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int l = lane + 32 * it;
      if (!valid || l >= n) continue;
      double *jg = A.jbg + (size_t)g * n + l;
      const size_t js = (size_t)NumG * n;
      if (MODE == 0) {
        double b[8];
        const double *V0 = A.Vn + (size_t)nz * g;
#ifdef CGD_FAST
        jac_bands_rcp(P, V0[l], V0[l + 1], V0[l + 4 * fs], V0[l + 1 + 4 * fs], tmp[l], tmp[l + 1],
                      P.dz[l + (size_t)nz * g], P.dz[l + 1 + (size_t)nz * g], tmp[LS + l], tmp[LS + l + 1], b);
#else
        jac_bands(P, V0[l], V0[l + 1], V0[l + 4 * fs], V0[l + 1 + 4 * fs], tmp[l], tmp[l + 1],
                  P.dz[l + (size_t)nz * g], P.dz[l + 1 + (size_t)nz * g], b);
#endif
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          jb[r * LS + l] = b[r];
          jg[r * js] = b[r];
        }
      }
    }
  }
  __syncwarp();
  // jb rows: 0,1 JRhoW ; 2,3 JWRho ; 4,5 JWRhoTh ; 6,7 JRhoThW  (row r = Julia index r%2+1)
#define JB(arr, r, i) jb[((arr) * 2 + (r)) * LS + (i)]
#define FV0(i) fv[(i)]
#define FV3(i) fv[LS + (i)]
#define FV4(i) fv[2 * LS + (i)]
  const double invfac2 = A.ifac2;
  double v3new[2] = {0.0, 0.0}, tq[2][3];
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int l = lane + 32 * it;
    if (valid && l < n) {   // TriDiagKernel!
      double t0, t1, t2;
      t1 = invfac2 - JB(1, 1, l) * JB(0, 0, l) - JB(1, 0, l) * JB(0, 1, l) -
           JB(2, 1, l) * JB(3, 0, l) - JB(2, 0, l) * JB(3, 1, l);
      if (l == 0) t0 = 0.0;
      else t0 = -JB(1, 0, l - 1) * JB(0, 0, l) - JB(2, 0, l - 1) * JB(3, 0, l);
      if (l == n - 1) t2 = 0.0;
      else t2 = -JB(1, 1, l + 1) * JB(0, 1, l) - JB(2, 1, l + 1) * JB(3, 1, l);
      tq[it][0] = t0; tq[it][1] = t1; tq[it][2] = t2;
      // SchurSolveFKernel!
#ifdef CGD_FAST
      const double v3 = FV3(l) * A.ifac;
#else
      const double v3 = FV3(l) / fac;
#endif
      v3new[it] = v3 + JB(1, 1, l) * FV0(l) + JB(1, 0, l) * FV0(l + 1) +
                  JB(2, 1, l) * FV4(l) + JB(2, 0, l) * FV4(l + 1);
    }
  }
  __syncwarp();
#pragma unroll
  for (int it = 0; it < 2; ++it)
    if (valid && lane + 32 * it < n) {
      FV3(lane + 32 * it) = v3new[it];
#pragma unroll
      for (int r = 0; r < 3; ++r) tri[r * LS + lane + 32 * it] = tq[it][r];
    }
#ifdef CGD_FAST
  // triSolve! as three warp scans over the column's levels (fast build);
  // the result differs from the sequential sweep by rounding only
  __syncwarp();
  if (!valid) return;   // warp-uniform; nothing below synchronises the block
  warp_tri_solve(tri, tri + LS, tri + 2 * LS, fv + LS, xs, n, lane);
  __syncwarp();
#else
  __syncthreads();
  // triSolve! (Thomas), b = FV3, x = xs: the serial sweeps of the block's
  // columns run concurrently, one per lane of the first warp
  if (threadIdx.x < COL_WARPS && g0 + (int)threadIdx.x < NumG) {
    double *sc = csm + (size_t)threadIdx.x * COL_ARR<MODE> * LS;
    double *b = sc + LS;
    const double *tr = sc + 5 * LS;
    double *x = sc + 8 * LS;
    x[0] = tr[LS + 0];
    for (int i = 0; i < n - 1; ++i) {
      const double m = tr[2 * LS + i] / x[i];   // the reference's tri[3,i]/x[i], used twice
      x[i + 1] = tr[LS + i + 1] - m * tr[i + 1];
      b[i + 1] = b[i + 1] - m * b[i];
    }
    x[n - 1] = b[n - 1] / x[n - 1];
    for (int i = n - 2; i >= 0; --i) x[i] = (b[i] - tr[i + 1] * x[i + 1]) / x[i];
  }
  __syncthreads();
#endif
  if (!valid) return;
  // SchurSolveBKernel! and the stage update of rho, w, rho*theta; each lane
  // owns levels lane and lane + 32
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int l = lane + 32 * it;
    if (l >= nz) continue;
    const double kw = l < n ? xs[l] : 0.0;
    double v0 = FV0(l), v4 = FV4(l);
    if (l == 0) {
      v0 += JB(0, 0, l) * xs[l];
      v4 += JB(3, 0, l) * xs[l];
    } else if (l == nz - 1) {
      v0 += JB(0, 1, l - 1) * xs[l - 1];
      v4 += JB(3, 1, l - 1) * xs[l - 1];
    } else {
      v0 += JB(0, 0, l) * xs[l] + JB(0, 1, l - 1) * xs[l - 1];
      v4 += JB(3, 0, l) * xs[l] + JB(3, 1, l - 1) * xs[l - 1];
    }
    const size_t o0 = l + (size_t)nz * g;
    if (MODE == 3) {
      // v after SchurSolveF/B (the Thomas sweep works on a copy, as in
      // SchurSolveTriKernel!'s shared-memory vCol)
      A.v[o0] = v0;
      A.v[o0 + 4 * fs] = v4;
      if (l < n) A.v[o0 + 3 * fs] = it == 0 ? v3new[0] : v3new[1];
    }
    const double kk[3] = {fac * v0, kw, fac * v4};
#pragma unroll
    for (int sf = 0; sf < 3; ++sf) {
      const int f = sf == 0 ? 0 : sf + 2;
      const size_t o = o0 + f * fs;
      const double k = kk[sf];
      if (MODE == 0) {
        const double vn = A.Vn[o];
        A.kout[o] = k;
        A.Vout[o] = vn + A.rk.a[1][0] * k;
      } else if (MODE <= 2) {
        // Vout may alias Vn: this lane alone reads index o and then writes it
        stage_update<MODE>(A, o, A.Vn[o], s1[it][sf], s2[it][sf], k);
        if (MODE == 2 && A.kout) A.kout[o] = k;   // the last stage's k of rho, w, rho*theta (adjoint replay only)
      } else {
        A.kout[o] = k;
      }
    }
  }
#undef JB
#undef FV0
#undef FV3
#undef FV4
}

template <int MODE, bool C32>
__global__ void __launch_bounds__(32 * COL_WARPS, col_min_blocks<MODE>()) k_column(const GP P, const ColArgs A)
{
  column_body<MODE, C32>(P, A, P.rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
}

// The kernels below are defined by the forward translation unit only (the
// adjoint's, cgd_adjoint.cu, includes this header for its device functions).
#ifndef CGD_ADJOINT_TU
// Mixed form: the FP64 reference profile of pressure and theta, the
// horizontal mean of each level of a state (one CTA per level, fixed-order
// tree reduction, so the profile is reproducible).
__global__ void __launch_bounds__(256) k_refprof(const GP P, const double *__restrict__ U, double *__restrict__ pref,
                                                 double *__restrict__ thref)
{
  __shared__ double sp[256], st[256];
  const int l = blockIdx.x, nz = P.nz, NumG = P.NumG;
  const size_t fs = (size_t)nz * NumG;
  double a = 0.0, b = 0.0;
  for (int g = threadIdx.x; g < NumG; g += blockDim.x) {
    const double rho = U[l + (size_t)nz * g], rth = U[l + (size_t)nz * g + 4 * fs];
    a += pressure_dry(P, rth);
    b += rth / rho;
  }
  sp[threadIdx.x] = a;
  st[threadIdx.x] = b;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sp[threadIdx.x] += sp[threadIdx.x + w];
      st[threadIdx.x] += st[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    pref[l] = sp[0] / NumG;
    thref[l] = st[0] / NumG;
  }
}

// The four band arrays of the reference's JCache (JRhoW, JWRho, JWRhoTh,
// JRhoThW), each (2, nz-1, NumG).
struct Bands4 {
  double *b[4];
};

// The column physics added to a tendency F of the state U with pressure p
// (cgd_rhs): one thread per column-level.
__global__ void __launch_bounds__(256) k_physics(const GP P, const double *__restrict__ U,
                                                 const double *__restrict__ p, double *__restrict__ F)
{
  const long long S = (long long)P.nz * P.NumG;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S) return;
  const int g = (int)(t / P.nz), l = (int)(t - (long long)g * P.nz);
  double f[5] = {0.0, F[t + S], F[t + 2 * S], F[t + 3 * S], F[t + 4 * S]};
  physics_terms(P, l, g, U[t], U[t + S], U[t + 2 * S], U[t + 3 * S], U[t + 4 * S], p[t], f);
  F[t + S] = f[1];
  F[t + 2 * S] = f[2];
  F[t + 3 * S] = f[3];
  F[t + 4 * S] = f[4];
}

// Jacobian bands into memory (cgd_jac): one thread per (level, column), which
// evaluates dp/d(rho theta) of its level and takes the upper level's from the
// next thread, and writes the bands of the interface above, a pair (16 bytes)
// per store; out2 (null entries: none) takes a copy for the caller.  nPanel 20,
// nz 37: 47 us and four copies of the bands before; now 64 us for
// all (70 us with single stores).
__global__ void __launch_bounds__(256) k_jac(const GP P, const double *__restrict__ U, const Bands4 out,
                                             const Bands4 out2)
{
  __shared__ double dp[257];
  const int nz = P.nz, n = nz - 1, t = threadIdx.x;
  const long long tid = (long long)blockIdx.x * 256 + t, S = (long long)nz * P.NumG;
  const bool in = tid < S;
  if (in) dp[t] = dpdrhoth(P, U[tid + 4 * S]);
  if (t == 255 && tid + 1 < S) dp[256] = dpdrhoth(P, U[tid + 1 + 4 * S]);
  __syncthreads();
  if (!in) return;
  const long long g = tid / nz;
  const int l = (int)(tid - g * nz);
  if (l == n) return;
  double b[8];
  jac_bands(P, U[tid], U[tid + 1], U[tid + 4 * S], U[tid + 1 + 4 * S], dp[t], dp[t + 1], P.dz[tid], P.dz[tid + 1], b);
  const size_t o = l + (size_t)n * g;
#pragma unroll
  for (int arr = 0; arr < 4; ++arr) {
    const double2 b2 = {b[2 * arr], b[2 * arr + 1]};
    reinterpret_cast<double2 *>(out.b[arr])[o] = b2;
    if (out2.b[arr]) reinterpret_cast<double2 *>(out2.b[arr])[o] = b2;
  }
}

__device__ __forceinline__ void pressure_body(const GP &P, const double *__restrict__ U, double *__restrict__ p,
                                              const long long tid)
{
  const long long S = (long long)P.nz * P.NumG;
  if (tid >= S) return;
  p[tid] = pressure_dry(P, U[tid + 4 * S]);
}

__global__ void __launch_bounds__(256) k_pressure(const GP P, const double *__restrict__ U, double *__restrict__ p)
{
  pressure_body(P, U, p, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// 1 if any entry is not finite
__global__ void k_nonfinite(const double *__restrict__ x, long long n, int *__restrict__ flag)
{
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  int bad = 0;
  for (; i < n; i += stride) {
    double v = x[i];
    if (!(v - v == 0.0)) bad = 1;
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

// deterministic two-level reduction of sum(rho*MMass): per-block partials in
// fixed order, then one block sums the partials in order
__global__ void k_mass_partial(const double *__restrict__ rho, const double *__restrict__ mm, long long n,
                               double *__restrict__ part)
{
  __shared__ double sh[256];
  long long chunk = (n + gridDim.x - 1) / gridDim.x;
  long long b0 = blockIdx.x * chunk, b1 = b0 + chunk < n ? b0 + chunk : n;
  double acc = 0.0;
  for (long long i = b0 + threadIdx.x; i < b1; i += blockDim.x) acc += rho[i] * mm[i];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void k_mass_final(const double *__restrict__ part, int nb, double *__restrict__ out)
{
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double acc = 0.0;
    for (int i = 0; i < nb; ++i) acc += part[i];
    out[0] = acc;
  }
}

#endif  // CGD_ADJOINT_TU

} // namespace cgd
