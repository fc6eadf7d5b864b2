// cgd_output.cuh - interpolation of the state to sub-cells for the output files.
//
// Each element and layer is divided into OrdPrint x OrdPrint sub-cells; the
// cell value of a quantity c is the interpolating polynomial at the sub-cell
// centre, Inter[I,J,iP,jP] = L_iP(xi_I) L_jP(eta_J)
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
//
// Two launches.  k_cells_nodal forms what is not a column of the state: the
// pressure and the potential temperature once per column and level, the
// vorticity once per element node and level, the surface w once per element
// node (only those asked for; no launch for none).  k_cells then is a thread per
// (element, level) and quantity, which gathers the N^2 nodal values (neighbouring
// threads: neighbouring levels of one column) and keeps up to 25 sub-cells' sums
// in registers.  One kernel with the nodal values of every quantity in shared
// planes, as before, spent its time in the chain index - columns - pow - barrier -
// curl - barrier - sums of 10 levels a CTA; with one sub-cell, or one quantity,
// most of its threads idled.  Calls on nPanel 30, p 4, nz 45, two tracers, us:
//
//                      OrdPrint 1        OrdPrint 4        OrdPrint 8
//   nine quantities    966 -> 312        941 -> 475        1841 -> 1223
//   rho alone          204 -> 39         218 -> 52
//   a tracer alone     656 -> 55         351 -> 95
//   vorticity alone    311 -> 145        327 -> 161
//
// and nPanel 60, nz 64, seven quantities, OrdPrint 1 2718 -> 1260; nPanel 6, nz 10
// 37 -> 36 (of these some 25 us are the call's own).  k_cells_nodal moves
// 4.0 TB/s, most of it the vorticity's metric (nPanel 20: 87 us under a profiler),
// k_cells 3.1 TB/s (50 us), waiting for its gathers.
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

// Levels of a vorticity tile; threads (node, level), level fastest.
template <int N>
struct NodalCfg {
  static constexpr int DoF = N * N, LT = N == 2 ? 32 : 16, RS = DoF | 1, THREADS = LT * DoF;
};

// What k_cells_nodal forms (null: not wanted): columns p and th of rho and
// rhoth; the surface w, -(a d31 + b d32) / d33 of the lowest lower node (no
// normal flow), [IF][ID], for (a, b) = (u, u) in w0[0] and (u, v) in w0[1]; the
// vorticity rot ([IF][ID][nz]) of u and v.  The first colblocks CTAs take the
// columns (bound by exp, log and pow), the next w0blocks the surface, the others
// a tile of an element each (bound by its ten metric values a node and level).
struct NodalArgs {
  const double *rho, *rhoth, *u, *v;
  double *p, *th, *w0[2], *rot;
  unsigned colblocks, w0blocks;
};

// COLS: more than the vorticity (without the others' code it alone takes 97 instead
// of 110 us on nPanel 60, p 1, nz 40)
template <int N, bool COLS>
__global__ void __launch_bounds__(NodalCfg<N>::THREADS) k_cells_nodal(const GP P, const NodalArgs A)
{
  using CF = NodalCfg<N>;
  constexpr int DoF = CF::DoF, LT = CF::LT, RS = CF::RS;
  const int nz = P.nz, t = threadIdx.x;
  asm volatile("griddepcontrol.launch_dependents;\n");   // k_cells waits for this grid's end itself
  if (COLS && blockIdx.x < A.colblocks) {
    const size_t i = (size_t)blockIdx.x * CF::THREADS + t;
    if (i >= (size_t)nz * P.NumG) return;
    const double p = pressure_dry(P, A.rhoth[i]);
    if (A.p) A.p[i] = p;
    if (A.th) A.th[i] = pott_dry(P, A.rho[i], p);
    return;
  }
  if (COLS && blockIdx.x < A.colblocks + A.w0blocks) {
    const int n = (blockIdx.x - A.colblocks) * CF::THREADS + t;
    if (n >= P.NF * DoF) return;
    const size_t o = (size_t)nz * P.glob[n], cs = (size_t)DoF * nz;
    const double *m = P.met + ((size_t)(n / DoF) * NCOMP * DoF + n % DoF) * nz;
    const double u = A.u[o], d31 = m[C_D31_0 * cs], d32 = m[C_D32_0 * cs], d33 = m[C_D33_0 * cs];
    if (A.w0[0]) A.w0[0][n] = -(u * d31 + u * d32) / d33;
    if (A.w0[1]) A.w0[1][n] = -(u * d31 + A.v[o] * d32) / d33;
    return;
  }
  __shared__ double tx[LT * RS], ty[LT * RS];
  const unsigned b = COLS ? blockIdx.x - A.colblocks - A.w0blocks : blockIdx.x, tiles = (nz + LT - 1) / LT;
  const int IF = b / tiles, lvl = t % LT, ID = t / LT, l = (b % tiles) * LT + lvl;
  const bool act = l < nz;
  const int i = ID % N, j = ID / N, row = lvl * RS;
  double J = 1.0;
  if (act) {
    const size_t cs = (size_t)DoF * nz, o = l + (size_t)nz * P.glob[(size_t)IF * DoF + ID];
    const double *mt = P.met + ((size_t)IF * NCOMP * DoF + ID) * nz + l;
    const double u = A.u[o], v = A.v[o];
    tx[row + ID] = (mt[C_D11_0 * cs] + mt[C_D11_1 * cs]) * v - (mt[C_D12_0 * cs] + mt[C_D12_1 * cs]) * u;
    ty[row + ID] = (mt[C_D21_0 * cs] + mt[C_D21_1 * cs]) * v - (mt[C_D22_0 * cs] + mt[C_D22_1 * cs]) * u;
    J = mt[C_J0 * cs] + mt[C_J1 * cs];
  }
  __syncthreads();
  if (!act) return;
  double acc = 0.0;
#pragma unroll
  for (int I = 0; I < N; ++I) acc += P.D[i + N * I] * tx[row + I + N * j];
#pragma unroll
  for (int k = 0; k < N; ++k) acc += P.D[j + N * k] * ty[row + i + N * k];
  A.rot[((size_t)IF * DoF + ID) * nz + l] = acc / J;
}

// What a cell value interpolates: a column c, c over rho, the layer mean of the
// column c = w with w0 at the surface, or the element-node array c.
enum { CELL_C = 0, CELL_C_RHO, CELL_WB, CELL_NODE };

// One launch's quantities: cell array k (n values each, back to back) is kind
// op of f[k].
constexpr int CELL_MAX = 16;
struct CellOp {
  int op;
  const double *c, *w0;
};
struct CellArgs {
  CellOp f[CELL_MAX];
  const double *rho;   // (nz, NumG), what CELL_C_RHO divides by
};

// n / d with r = 1 / d: the correctly rounded quotient by two Newton
// corrections of n r, whose residuals are exact (Markstein's theorem: from an
// approximation within one unit in the last place, with r correctly rounded,
// the second is correctly rounded).  For n zero or in 2^-400 .. 2^500 and d in
// 2^-400 .. 2^400, where nothing overflows or loses bits to underflow.
__device__ __forceinline__ double exact_quotient(double n, double d, double r)
{
  double q = n * r;
  q = __fma_rn(__fma_rn(-q, d, n), r, q);
  return __fma_rn(__fma_rn(-q, d, n), r, q);
}

// |x| in 2^lo .. 2^hi (below 2^(hi+1)), zero too where it may be.
__device__ __forceinline__ bool in_range(double x, int lo, int hi, bool zero)
{
  const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
  return (e >= lo && e <= hi) || (zero && x == 0.0);
}

constexpr int CELL_THREADS = 128;

// CH sub-cells a thread; blockIdx.y: quantity; blockIdx.x: group of CH sub-cells
// (fastest, so that the groups' halves of a cache line come together), pairs.
// CH > 1: the weights are read from shared memory, as broadcasts, and the sums go
// out through it, a warp's in runs of CH values.
template <int N, int CH>
__global__ void __launch_bounds__(CELL_THREADS, CH == 1 ? 8 : CH <= 9 ? 6 : CH <= 18 ? 5 : 4) k_cells(const GP P, const CellArgs A, const double *__restrict__ inter,
                                                        int OP2, double *__restrict__ cell)
{
  constexpr int DoF = N * N, CS = CH | 1;
  __shared__ __align__(16) double sw[CH > 1 ? DoF * CH : 1];
  __shared__ double so[CH > 1 ? CELL_THREADS * CS : 1];
  const int nz = P.nz, t = threadIdx.x, groups = (OP2 + CH - 1) / CH;
  const int c0 = blockIdx.x % groups * CH, nc = min(CH, OP2 - c0);
  const long long total = (long long)nz * P.NF, first = (long long)(blockIdx.x / groups) * CELL_THREADS;
  const bool in = first + t < total;
  const long long x = in ? first + t : total - 1;
  const int IF = (int)(x / nz), l = (int)(x - (long long)IF * nz);
  const int *gl = P.glob + (size_t)IF * DoF;
  if (CH > 1) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(gl));   // while the weights come
  bool plain = true;   // every weight zero or in 2^-100 .. 2^99
  if (CH > 1) {
    for (int y = t; y < DoF * CH; y += CELL_THREADS) {
      const int n = y / CH, c = y % CH;
      const double w = c < nc ? inter[c0 + c + (size_t)OP2 * n] : 0.0;
      sw[y] = w;
      plain = plain && in_range(w, -100, 98, true);
    }
    plain = __syncthreads_and(plain);
  }
  auto weight = [&](int n, int c) { return CH > 1 ? sw[n * CH + c] : inter[c0 + (size_t)OP2 * n]; };
  const CellOp f = A.f[blockIdx.y];
  asm volatile("griddepcontrol.wait;\n" ::: "memory");   // k_cells_nodal's arrays
  double acc[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) acc[c] = 0.0;
  // sum of weight * value(n) over the nodes in ascending order
  auto sums = [&](auto &&value) {
#pragma unroll
    for (int n = 0; n < DoF; ++n) {
      const double y = value(n);
#pragma unroll
      for (int c = 0; c < CH; ++c) acc[c] += weight(n, c) * y;
    }
  };
  // the same with divisions: a row's loads first (their slow paths keep loads
  // from being moved ahead of them)
  auto rows = [&](auto &&load, auto &&add) {
#pragma unroll 1
    for (int jn = 0; jn < N; ++jn) {
      double z[N][2];
#pragma unroll
      for (int k = 0; k < N; ++k) load(jn * N + k, z[k]);
#pragma unroll
      for (int k = 0; k < N; ++k) add(jn * N + k, z[k]);
    }
  };
  if (f.op == CELL_C) {
    sums([&](int n) { return f.c[l + (size_t)nz * gl[n]]; });
  } else if (f.op == CELL_NODE) {
    const double *e = f.c + (size_t)IF * DoF * nz + l;
    sums([&](int n) { return e[(size_t)n * nz]; });
  } else if (f.op == CELL_WB) {
    // the reference halves the weight, the same value
    sums([&](int n) {
      const size_t o = l + (size_t)nz * gl[n];
      const double *below = l > 0 ? f.c + o - 1 : f.w0 + IF * DoF + n;
      return 0.5 * (f.c[o] + *below);
    });
  } else if (CH == 1) {
    rows([&](int n, double *z) {
      const size_t o = l + (size_t)nz * gl[n];
      z[0] = f.c[o]; z[1] = A.rho[o];
    }, [&](int n, const double *z) { acc[0] += weight(n, 0) * z[0] / z[1]; });
  } else {
    // one division a node instead of one a sub-cell, with the same quotients
    rows([&](int n, double *z) {
      const size_t o = l + (size_t)nz * gl[n];
      z[0] = f.c[o]; z[1] = A.rho[o];
    }, [&](int n, const double *z) {
      const double y = z[0], d = z[1];
      if (plain && in_range(d, -400, 399, false) && in_range(y, -300, 399, true)) {
        const double r = 1.0 / d;
#pragma unroll
        for (int c = 0; c < CH; ++c) acc[c] += exact_quotient(weight(n, c) * y, d, r);
      } else {
#pragma unroll 1
        for (int c = 0; c < nc; ++c) so[t * CS + c] = weight(n, c) * y / d;
#pragma unroll
        for (int c = 0; c < CH; ++c) acc[c] += so[t * CS + c];
      }
    });
  }
  double *out = cell + (size_t)blockIdx.y * OP2 * total;
  if (CH == 1) {
    if (in) out[x * OP2 + c0] = acc[0];
    return;
  }
  const int warp = t & ~31, lane = t & 31;
#pragma unroll
  for (int c = 0; c < CH; ++c) so[t * CS + c] = acc[c];
  __syncwarp();
  const int pairs = (int)min(32LL, total - first - warp);   // (element, level) pairs of this warp
  double *ow = out + (first + warp) * OP2 + c0;
  if (OP2 == CH) {
    for (int y = lane; y < pairs * CH; y += 32) ow[y] = so[warp * CS + (CS == CH ? y : y / CH * CS + y % CH)];
  } else {
    for (int y = lane; y < pairs * CH; y += 32) {
      const int r = y / CH, c = y % CH;
      if (c < nc) ow[(size_t)r * OP2 + c] = so[(warp + r) * CS + c];
    }
  }
}

}  // namespace cgd
