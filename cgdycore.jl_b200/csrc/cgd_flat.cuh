// cgd_flat.cuh - phase 1 and phase 2 of the tendency on a flat product grid
// (fast build).
//
// Without orography every element-node metric of the sphere is a horizontal
// factor times the layer thickness: dXdxI(1:2,1:2) = h z(l) and J = hJ z(l) on
// both nodes of a layer, dXdxI(3,3) = h33, M = m z(l), and the slopes
// dXdxI(3,1:2) of the levels are rounding residue, 1e-16 of h33, the same
// function of I and of J in every element.  z then drops
// out of every horizontal operator (a derivative sum runs over one level, and
// each is divided by J or by M):
//
//   curl, divergence, gradients  D (h .) / hJ            instead of D (d .) / J
//   weak forms, flux divergences D (h .) / m             instead of D (d .) / M
//   the w-dependent curls        X(l) = D (h w(l)) serves the upper node of
//                                level l and the lower node of level l + 1
//
// so the 21 metric values a node and level are replaced by eight a node
// and a few a level, which stay in L1, and half of the w-curl sums go.  The
// slopes' residue is kept where it stands beside small differences of large
// terms, in gravity along the level and in the curl of (u, v): without it the
// u and v tendencies are 1e-12 of their size away from the arrays' own, with
// it as near as the general kernels (5e-13, the rounding of the pressure
// sums).  Elsewhere it is below the rounding of the terms it adds to.  The
// grid set-up checks that the caller's arrays have this form to rounding
// (k_flat_check, FLAT_TOL); any other grid, and the exact build, run the
// general kernels (hypervisc1_body, phase2_body).
//
// Same tiles, roles and planes as cgd_phase2.cuh.  nPanel 30, p 4, nz 45, two
// tracers: phase 1 0.310 -> 0.238 ms (91 % of the L1/shared pipe's peak), phase
// 2 1.224 -> 0.749 ms (67 % of it, 26 warps an SM waiting for loads and
// barriers); before the pressure (phase 1, 0.027 ms) and the cache sums (phase
// 2, 0.07 ms) came in from kernels of 0.041 and 0.115 ms.  Tried: a thread per row
// of nodes with the x sums in registers, half the shared loads but 10 to 15
// warps an SM: 1.29 ms.
#pragma once
#include "cgd_phase2.cuh"

namespace cgd {

constexpr double FLAT_TOL = 2e-15;   // relative

// n / d with r = 1 / d shared by several quotients: one Newton correction of
// n r keeps the quotient's error at a rounding of the division's
__device__ __forceinline__ double ratio_of(double n, double d, double r)
{
  const double q = n * r;
  return fma(fma(-q, d, n), r, q);
}

// The layers' table zl: z from the nodes of the first element (their mean J, as
// cgd_set_layers documents it), or the caller's zin; 1/z, the RecU4
// coefficients and the slope residue.  One CTA of 64 threads.
__global__ void __launch_bounds__(64) k_flat_layers(const GP P, const double *__restrict__ zin,
                                                    double *__restrict__ zl)
{
  __shared__ double zs[64];
  const int l = threadIdx.x, nz = P.nz, DoF = P.DoF, N = P.N;
  const size_t cs = (size_t)DoF * nz;
  const double *me = P.met;   // element 0
  if (l < nz) {
    double a = 0.0, b = 0.0;
    for (int ID = 0; ID < DoF; ++ID) {
      a += me[C_J0 * cs + (size_t)ID * nz + l];
      b += me[C_J0 * cs + (size_t)ID * nz];
    }
    zs[l] = zin ? zin[l] : a / b;
  }
  __syncthreads();
  if (l >= nz) return;
  zl[l] = zs[l];
  zl[nz + l] = 1.0 / zs[l];
  double rk[4] = {0.0, 0.0, 0.0, 0.0};
  if (l < nz - 1) {   // RecU4 (OperatorKernel.jl:1044-1059) with J = hJ z
    const double LL = zs[l > 0 ? l - 1 : 0], L = zs[l], R = zs[l + 1], RR = zs[l + 2 < nz ? l + 2 : nz - 1];
    rk[0] = (L / (L + R)) * ((LL + L) / (LL + L + R));
    rk[1] = (L / (LL + L)) * (R / (LL + L + R));
    rk[2] = (R / (R + L)) * ((RR + R) / (L + R + RR));
    rk[3] = (R / (RR + R)) * (L / (L + R + RR));
  }
  for (int c = 0; c < 4; ++c) zl[(2 + c) * nz + l] = rk[c];
  // slope residue: dXdxI(3,1) = -(h11 f(I) + h21 f(J)), (3,2) = -(h12 f(I) +
  // h22 f(J)) with f(I, level, node) = sum_k DS[I,k] height, the same in every
  // element; from the nodes (I, 0).  Kept: the sum over the two nodes of a
  // layer and half their difference over z, in single precision (1e-23 of d33
  // off, and the same digits whichever element they come from)
  for (int I = 0; I < N; ++I) {
    const double *m = me + (size_t)I * nz + l;
    const double h11 = m[C_D11_0 * cs], h12 = m[C_D12_0 * cs], h21 = m[C_D21_0 * cs], h22 = m[C_D22_0 * cs];
    const double rd = zs[l] / (h11 * h22 - h12 * h21);
    double f[2];
    for (int k = 0; k < 2; ++k) f[k] = (h21 * m[(C_D32_0 + k) * cs] - h22 * m[(C_D31_0 + k) * cs]) * rd;
    zl[(size_t)(6 + I) * nz + l] = (float)(f[0] + f[1]);
    zl[(size_t)(6 + N + I) * nz + l] = (float)(0.5 * (f[1] - f[0]) / zs[l]);
  }
}

// The element nodes' factors, each the mean over the levels of what the arrays
// hold, nearer to their common value than any one rounded entry.  One CTA per
// element: the entries come in runs of levels, a thread then sums a node's in
// their order.  (A thread reading its node's entries itself, nz apart from the
// next thread's, took 0.20 ms on the mean of nPanel 16, 24 and 32 at nz 30 to 64.)
__global__ void __launch_bounds__(256) k_flat_factors(const GP P, double *__restrict__ hm)
{
  __shared__ double s[25 * 65];
  const int IF = blockIdx.x, t = threadIdx.x, nz = P.nz, DoF = P.DoF;
  const size_t cs = (size_t)DoF * nz;
  const double *m = P.met + (size_t)IF * NCOMP * cs;
  double *o = hm + (size_t)IF * H_N * DoF + t;
  double sz = 0.0;
  for (int l = 0; l < nz; ++l) sz += P.zl[l];
  // sum over the levels of x + y, for node t
  auto total = [&](auto &&x, auto &&y) {
    __syncthreads();
    for (int i = t; i < DoF * nz; i += 256) s[i / nz * 65 + i % nz] = x(i) + y(i);
    __syncthreads();
    double a = 0.0;
    if (t < DoF)
      for (int l = 0; l < nz; ++l) a += s[t * 65 + l];
    return a;
  };
  auto mean = [&](int c) {   // of both nodes of the layers, over z
    return 0.5 * total([&](int i) { return m[c * cs + i]; }, [&](int i) { return m[(c + 1) * cs + i]; }) / sz;
  };
  for (int c = 0; c < 4; ++c) {
    const double h = mean(C_D11_0 + 2 * c);
    if (t < DoF) o[(H_11 + c) * DoF] = h;
  }
  const double hJ = mean(C_J0);
  auto mass = [&](int i, int k) { return P.M[i % nz + (size_t)nz * (P.glob[IF * DoF + i / nz] + (size_t)k * P.NumG)]; };
  const double a = total([&](int i) { return mass(i, 0); }, [&](int i) { return mass(i, 1); });
  if (t >= DoF) return;
  o[H_J * DoF] = hJ;
  o[H_RJ * DoF] = 1.0 / hJ;
  o[H_33 * DoF] = m[C_D33_0 * cs + (size_t)t * nz];
  o[H_FC * DoF] = m[C_FCOR * cs + (size_t)t * nz];
  o[H_RM * DoF] = 2.0 * sz / a;
}

// Sets *bad unless every entry of the metric and the lumped mass is its
// product of factors to FLAT_TOL.  One thread per element node and level.
__global__ void __launch_bounds__(256) k_flat_check(const GP P, double Omega2, int *__restrict__ bad)
{
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nz = P.nz, DoF = P.DoF;
  const size_t cs = (size_t)DoF * nz;
  const long long ne = (long long)P.NF * DoF * nz;
  auto differ = [](double a, double b, double scale) { return !(fabs(a - b) <= FLAT_TOL * scale); };
  if (t >= ne) return;
  {
    const int l = (int)(t % nz);
    const long long n = t / nz;
    const int ID = (int)(n % DoF), IF = (int)(n / DoF);
    const double *m = P.met + ((size_t)IF * NCOMP * DoF + ID) * nz + l;
    const double *h = P.hm + (size_t)IF * H_N * DoF + ID;
    const double *zt = P.zl;
    const double z = zt[l], h33 = h[H_33 * DoF], hJ = h[H_J * DoF];
    double mx = 0.0;
    for (int c = 0; c < 4; ++c) mx = fmax(mx, fabs(h[(H_11 + c) * DoF]));
    bool b = !(h33 > 0.0) || !(hJ > 0.0) || !(z > 0.0);
    for (int c = 0; c < 4; ++c)
      for (int k = 0; k < 2; ++k) b = b || differ(m[(C_D11_0 + 2 * c + k) * cs], h[(H_11 + c) * DoF] * z, mx * z);
    for (int k = 0; k < 2; ++k) {
      b = b || differ(m[(C_J0 + k) * cs], hJ * z, hJ * z) || differ(m[(C_D33_0 + k) * cs], h33, h33);
      b = b || differ(m[(C_D31_0 + k) * cs], 0.0, h33) || differ(m[(C_D32_0 + k) * cs], 0.0, h33);
    }
    // the slope residue against its factors: to a hundredth of a rounding of d33
    const double *sl = zt + (size_t)6 * nz + l;
    const int I = ID % P.N, J = ID / P.N;
    const double sI = sl[I * nz], sJ = sl[J * nz];
    const double dI = 2.0 * z * sl[(P.N + I) * nz], dJ = 2.0 * z * sl[(P.N + J) * nz];
    for (int c = 0; c < 2; ++c) {
      const double a = h[(H_11 + c) * DoF], bb = h[(H_21 + c) * DoF];
      const double m0 = m[(C_D31_0 + 2 * c) * cs], m1 = m[(C_D31_0 + 2 * c + 1) * cs];
      b = b || !(fabs(m0 + m1 + (a * sI + bb * sJ)) <= 1e-18 * h33);
      b = b || !(fabs(m1 - m0 + (a * dI + bb * dJ)) <= 1e-18 * h33);
    }
    b = b || differ(m[C_FCOR * cs], h[H_FC * DoF], Omega2);
    if (l < nz - 1)
      for (int c = 0; c < 4; ++c) b = b || differ(m[(C_RK0 + c) * cs], zt[(2 + c) * nz + l], 1.0);
    const size_t o = l + (size_t)nz * P.glob[IF * DoF + ID];
    const double rm = h[H_RM * DoF], x0 = P.M[o] * rm, x1 = P.M[o + (size_t)nz * P.NumG] * rm;
    b = b || !(rm > 0.0) || differ(x0, z, z) || differ(x1, z, z);
    if (b) *bad = 1;
  }
}

// ---------------------------------------------------------------------------
// Phase 1 (ViscKernel.jl:1-84,169-218): curl, divergence, Laplacians.
// ---------------------------------------------------------------------------
template <int N, int NT, typename R, int LT>
__device__ __forceinline__ void hypervisc1_flat(const GP &P, const double *__restrict__ U, double *__restrict__ C,
                                                double *__restrict__ Pr, const int tile, const int IF, R *sbuf)
{
  constexpr bool MIX = sizeof(R) == sizeof(float);
  using CT = typename std::conditional<MIX, float, double>::type;
  constexpr int DoF = N * N, RS = HV1Smem<N, NT, R, LT>::RS;
  R(*s)[LT * RS] = reinterpret_cast<R(*)[LT * RS]>(sbuf);
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT;
  const int I = ID % N, Jn = ID / N;
  const int l = tile * LT + lvl;
  const int nz = P.nz;
  const bool act = (ID < DoF) && (l < nz);
  const int row = lvl * RS, si = row + ID;
  const size_t cs = (size_t)DoF * nz;
  R h11 = 0, h12 = 0, h21 = 0, h22 = 0, rJ = 0, rm = 0;
  if (act) {
    const int g = P.glob[IF * DoF + ID];
    const double *h = P.hm + (size_t)IF * H_N * DoF + ID;
    h11 = (R)h[H_11 * DoF]; h12 = (R)h[H_12 * DoF]; h21 = (R)h[H_21 * DoF]; h22 = (R)h[H_22 * DoF];
    rJ = (R)h[H_RJ * DoF];
    rm = (R)h[H_RM * DoF];
    const double *Ug = U + l + (size_t)nz * g;
    const size_t fs = (size_t)nz * P.NumG;
    const R u = (R)Ug[1 * fs], v = (R)Ug[2 * fs];
    const double rho = Ug[0], rr = 1.0 / rho;
    s[0][si] = h11 * v - h12 * u;   // Curl12
    s[1][si] = h21 * v - h22 * u;
    s[2][si] = h11 * u + h12 * v;   // Contra12
    s[3][si] = h21 * u + h22 * v;
    s[4][si] = (R)(ratio_of(Ug[4 * fs], rho, rr) - (MIX ? P.thref[l] : 0.0));
#pragma unroll
    for (int q = 0; q < NT; ++q) s[9 + 3 * q][si] = (R)ratio_of(Ug[(5 + q) * fs], rho, rr);
    stage_pressure(P, Pr, IF * DoF + ID, g, l, Ug[4 * fs]);
  }
  __syncthreads();
  if (act) {
    R DI[N], DJ[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      DI[k] = (R)P.D[I + N * k];
      DJ[k] = (R)P.D[Jn + N * k];
    }
    const R *uC = s[0] + row, *vC = s[1] + row, *uD = s[2] + row, *vD = s[3] + row;
    R cu = DI[0] * uC[N * Jn] + DJ[0] * vC[I];
    R dv = DI[0] * uD[N * Jn] + DJ[0] * vD[I];
#pragma unroll
    for (int k = 1; k < N; ++k) {
      cu = fsum2(cu, DI[k], uC[k + N * Jn], DJ[k], vC[I + N * k]);
      dv = fsum2(dv, DI[k], uD[k + N * Jn], DJ[k], vD[I + N * k]);
    }
    s[5][si] = cu * rJ;
    s[6][si] = dv * rJ;
#pragma unroll
    for (int q = 0; q < 1 + NT; ++q) {
      const R *c = s[q == 0 ? 4 : 6 + 3 * q] + row;
      R Dx = DI[0] * c[N * Jn], Dy = DJ[0] * c[I];
#pragma unroll
      for (int k = 1; k < N; ++k) {
        Dx = fsum1(Dx, DI[k], c[k + N * Jn]);
        Dy = fsum1(Dy, DJ[k], c[I + N * k]);
      }
      const R Gx = (h11 * Dx + h21 * Dy) * rJ;   // Grad12 with J
      const R Gy = (h12 * Dx + h22 * Dy) * rJ;
      s[7 + 3 * q][si] = h11 * Gx + h12 * Gy;    // Contra12
      s[8 + 3 * q][si] = h21 * Gx + h22 * Gy;
    }
  }
  __syncthreads();
  if (!act) return;
  R WI[N], WJ[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    WI[k] = (R)P.DW[I + N * k];
    WJ[k] = (R)P.DW[Jn + N * k];
  }
  CT *out = reinterpret_cast<CT *>(C) + ((size_t)IF * P.NC * DoF + ID) * nz + l;
  const R *Cu = s[5] + row, *Dv = s[6] + row;
  R DxCurl = WI[0] * Cu[N * Jn], DyCurl = WJ[0] * Cu[I];
  R DxDiv = WI[0] * Dv[N * Jn], DyDiv = WJ[0] * Dv[I];
#pragma unroll
  for (int k = 1; k < N; ++k) {
    DxCurl = fsum1(DxCurl, WI[k], Cu[k + N * Jn]);
    DyCurl = fsum1(DyCurl, WJ[k], Cu[I + N * k]);
    DxDiv = fsum1(DxDiv, WI[k], Dv[k + N * Jn]);
    DyDiv = fsum1(DyDiv, WJ[k], Dv[I + N * k]);
  }
  out[0 * cs] = (CT)(-(h12 * DxCurl + h22 * DyCurl) * rm);   // Rot12
  out[1 * cs] = (CT)((h11 * DxCurl + h21 * DyCurl) * rm);
  out[2 * cs] = (CT)((h11 * DxDiv + h21 * DyDiv) * rm);      // Grad12
  out[3 * cs] = (CT)((h12 * DxDiv + h22 * DyDiv) * rm);
#pragma unroll
  for (int q = 0; q < 1 + NT; ++q) {
    const R *x = s[7 + 3 * q] + row, *y = s[8 + 3 * q] + row;
    R Lap = WI[0] * x[N * Jn] + WJ[0] * y[I];
#pragma unroll
    for (int k = 1; k < N; ++k) Lap = fsum2(Lap, WI[k], x[k + N * Jn], WJ[k], y[I + N * k]);
    out[(4 + q) * cs] = (CT)(Lap * rm);
  }
}

// ---------------------------------------------------------------------------
// Phase 2
// ---------------------------------------------------------------------------
template <int N, int NT, typename R, int LT_ = p2_levels<N>()>
struct P2Flat {
  using G = P2Cfg<N, NT, R, LT_>;
  static constexpr int DoF = G::DoF, LT = LT_, RS = G::RS, PL = G::PL, NS = G::NS, THREADS = G::THREADS;
  static constexpr bool MIX = G::MIX;
  // scalars: ratios of the tile and two halo levels on each side, the mass
  // flux of interface L0-1 and its 1 + NS halo fluxes (double); planes as in
  // the general kernel
  static constexpr size_t S_BYTES = ((size_t)NS * (LT + 4) * RS + (size_t)(2 + NS) * RS) * sizeof(double) +
                                    (size_t)(3 * NS + 2 + (MIX ? NS : 0)) * PL * sizeof(R);
  // momentum: the w-curls of level L0-1 (2); planes: cache (4), h w of the
  // tile and of level L0-1 (4, LT + 1 rows), the curl of (u, v) (2), K, the
  // pressure, second round (2)
  static constexpr int M_PLANES = 4 + 2 + 2 + 2;
  static constexpr size_t M_BYTES = ((size_t)2 * RS + (size_t)M_PLANES * PL + (size_t)4 * (PL + RS)) * sizeof(R);
  static constexpr size_t SMEM = S_BYTES > M_BYTES ? S_BYTES : M_BYTES;
  static constexpr int MINB = G::MINB, MINB_S = 1280 / THREADS;
};

template <int N, int NT, typename R, int LT, int TH>
__device__ __forceinline__ void phase2_scalars_flat(const GP &P, const double *__restrict__ U,
                                                    const double *__restrict__ C1, double *__restrict__ C,
                                                    const int L0, const int IF, double *sm)
{
  using CF = P2Flat<N, NT, R, LT>;
  constexpr bool MIX = CF::MIX;
  constexpr int DoF = CF::DoF, RS = CF::RS, PL = CF::PL, NS = CF::NS, CR = LT + 4;
  using CT = typename std::conditional<MIX, float, double>::type;   // stored cache and contributions
  const int nz = P.nz;
  const size_t cs = (size_t)DoF * nz, fs = (size_t)nz * P.NumG;
  double *cth = sm;                              // [NS][CR][RS] ratios, rows L0-2 .. L0+LT+1
  double *f0 = cth + (size_t)NS * CR * RS;       // mass flux of interface L0-1
  double *fxh = f0 + RS;                         // [1+NS][RS] fluxes of interface L0-1
  R *sc = reinterpret_cast<R *>(fxh + (size_t)(1 + NS) * RS);   // [NS] cache
  R *scon = sc + (size_t)NS * PL;                // [2] contravariant mass flux
  R *s2 = scon + (size_t)2 * PL;                 // [2 NS] second round
  R *sq = s2 + (size_t)2 * NS * PL;              // [NS] ratios as R (mixed form)
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT;
  const int l = L0 + lvl;
  const bool act = ID < DoF && l < nz;
  const int I = ID % N, Jn = ID / N;
  const int row = lvl * RS, si = row + ID;
  const double *hn = P.hm + (size_t)IF * H_N * DoF + ID;
  const unsigned lanes = block_lanes<TH>();

  // ---------------- operands of the first round, vertical halo ----------------
  // halo: thread t < 4 DoF takes node t / 4 of level L0-2, L0-1, L0+LT or
  // L0+LT+1; its loads are issued first, beside the thread's own
  static_assert(4 * DoF <= TH, "one halo slot per thread");
  const int hID = t >> 2, hr = (t & 3) < 2 ? (t & 3) : LT + (t & 3), hl = L0 - 2 + hr;
  const bool hs = t < 4 * DoF && hl >= 0 && hl < nz;
  double hrho = 1.0, hq[NS], hw = 0.0, ha = 0.0;
  if (hs) {
    const double *Ug = U + (size_t)nz * P.glob[IF * DoF + hID] + hl;
    hrho = Ug[0];
#pragma unroll
    for (int q = 0; q < NS; ++q) hq[q] = Ug[(4 + q) * fs];
    if ((t & 3) == 1) { hw = Ug[3 * fs]; ha = Ug[1]; }
  }
  double rho = 1.0, F0 = 0.0, rm = 0.0;
  R h11 = 0, h12 = 0, h21 = 0, h22 = 0;
  if (act) {
    const int g = P.glob[IF * DoF + ID];
    const double *Ug = U + (size_t)nz * g + l;
    R ca[NS];
    cache_sums<MIX, 4, NS>(P, C1, IF * DoF + ID, l, ca);
    rho = Ug[0];
    const double u = Ug[fs], v = Ug[2 * fs];
    F0 = Ug[3 * fs] * (rho + (l < nz - 1 ? Ug[1] : 0.0));   // mass flux of interface l over d33
    const double a11 = hn[H_11 * DoF], a12 = hn[H_12 * DoF], a21 = hn[H_21 * DoF], a22 = hn[H_22 * DoF];
    rm = hn[H_RM * DoF];
    const double rr = 1.0 / rho;
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      sc[q * PL + si] = ca[q];
      const double c = ratio_of(Ug[(4 + q) * fs], rho, rr);
      cth[(q * CR + lvl + 2) * RS + ID] = c;
      if (MIX) sq[q * PL + si] = (R)c;
    }
    scon[si] = (R)(-rho * (a11 * u + a12 * v));           // Contra12(-Rho, u, v)
    scon[PL + si] = (R)(-rho * (a21 * u + a22 * v));
    h11 = (R)a11; h12 = (R)a12; h21 = (R)a21; h22 = (R)a22;
  }
  if (hs) {
    const double rr = 1.0 / hrho;
#pragma unroll
    for (int q = 0; q < NS; ++q) cth[(q * CR + hr) * RS + hID] = ratio_of(hq[q], hrho, rr);
    if ((t & 3) == 1) f0[hID] = hw * (hrho + ha);
  }
  __syncthreads();

  // ---------------- vertical fluxes of interface l (over d33) ----------------
  auto fluxes = [&](int il, int pl, int n, double w, double *f) {
    const bool up = w > 0.0;
    const double *k = P.zl + (size_t)(up ? 2 : 4) * nz + il;
    const double kc = k[0], ks = k[nz];
    const int far = up ? (il > 0 ? pl - 1 : pl) : (il + 2 < nz ? pl + 2 : pl + 1);
    f[0] = w;
#pragma unroll
    for (int q = 0; q < NS; ++q)
      f[1 + q] = upwind_flux(cth + (size_t)q * CR * RS + n, RS, up ? pl : pl + 1, up ? pl + 1 : pl, far, kc, ks, w);
  };
  double Ft[1 + NS];
#pragma unroll
  for (int q = 0; q < 1 + NS; ++q) Ft[q] = 0.0;
  if (act && l < nz - 1) fluxes(l, lvl + 2, ID, F0, Ft);
  if (L0 > 0 && t < DoF) {   // the interface below the tile
    double f[1 + NS];
    fluxes(L0 - 1, 1, t, f0[t], f);
#pragma unroll
    for (int q = 0; q < 1 + NS; ++q) fxh[q * RS + t] = f[q];
  }

  // ---------------- first derivatives, flux divergences ----------------
  R DivRho = 0, Div[NS];
  if (act) {
    R DI[N], DJ[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      DI[k] = (R)P.D[I + N * k];
      DJ[k] = (R)P.D[Jn + N * k];
    }
    const R rJ = (R)hn[H_RJ * DoF];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const R *c = sc + q * PL + row;
      R Dx = DI[0] * c[N * Jn], Dy = DJ[0] * c[I];
#pragma unroll
      for (int k = 1; k < N; ++k) {
        Dx = fsum1(Dx, DI[k], c[k + N * Jn]);
        Dy = fsum1(Dy, DJ[k], c[I + N * k]);
      }
      const R Gx = (h11 * Dx + h21 * Dy) * rJ;
      const R Gy = (h12 * Dx + h22 * Dy) * rJ;
      s2[(2 * q) * PL + si] = (R)(rho * (h11 * Gx + h12 * Gy));   // (in FP64 in the mixed form too)
      s2[(2 * q + 1) * PL + si] = (R)(rho * (h21 * Gx + h22 * Gy));
    }
    // D (rho u) at the summed nodes, shared by rho and every scalar
    const R *uc = scon + row, *vc = scon + PL + row;
    R mx[N], my[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      mx[k] = DI[k] * uc[k + N * Jn];
      my[k] = DJ[k] * vc[I + N * k];
    }
    DivRho = mx[0] + my[0];
#pragma unroll
    for (int k = 1; k < N; ++k) DivRho = DivRho + (mx[k] + my[k]);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      if constexpr (MIX) {
        const R *c = sq + q * PL + row;
        Div[q] = mx[0] * c[N * Jn] + my[0] * c[I];
#pragma unroll
        for (int k = 1; k < N; ++k) Div[q] = rsum2(Div[q], mx[k], c[k + N * Jn], my[k], c[I + N * k]);
      } else {
        const double *c = cth + (size_t)(q * CR + lvl + 2) * RS;
        Div[q] = mx[0] * c[N * Jn] + my[0] * c[I];
#pragma unroll
        for (int k = 1; k < N; ++k) Div[q] = fsum2(Div[q], mx[k], c[k + N * Jn], my[k], c[I + N * k]);
      }
    }
  }
  __syncthreads();

  // ---------------- weak derivatives; contributions ----------------
  double Fb[1 + NS];
#pragma unroll
  for (int q = 0; q < 1 + NS; ++q) Fb[q] = __shfl_up_sync(lanes, Ft[q], 1, LT);
  if (!act) return;
  if (lvl == 0) {
#pragma unroll
    for (int q = 0; q < 1 + NS; ++q) Fb[q] = l > 0 ? fxh[q * RS + ID] : 0.0;
  }
  // vertical fluxes: F d33 / (2 m z)
  const double fz = 0.5 * rm * hn[H_33 * DoF] * P.zl[nz + l];
  CT *out = reinterpret_cast<CT *>(C) + ((size_t)IF * P.NC * DoF + ID) * nz + l;
  out[0] = (CT)(0.5 * fz * (Fb[0] - Ft[0]) + rm * DivRho);
  R WI[N], WJ[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    WI[k] = (R)P.DW[I + N * k];
    WJ[k] = (R)P.DW[Jn + N * k];
  }
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const R *x = s2 + (2 * q) * PL + row, *y = s2 + (2 * q + 1) * PL + row;
    R Lap = WI[0] * x[N * Jn] + WJ[0] * y[I];
#pragma unroll
    for (int k = 1; k < N; ++k) Lap = fsum2(Lap, WI[k], x[k + N * Jn], WJ[k], y[I + N * k]);
    out[(4 + q) * cs] = (CT)(fz * (Fb[1 + q] - Ft[1 + q]) + rm * (Div[q] - P.nuDiv * Lap));
  }
}

template <int N, int NT, typename R, int LT, int TH>
__device__ __forceinline__ void phase2_momentum_flat(const GP &P, const double *__restrict__ U,
                                                     const double *__restrict__ Pr, const double *__restrict__ C1,
                                                     double *__restrict__ C, const int L0, const int IF, double *sm)
{
  using CF = P2Flat<N, NT, R, LT>;
  constexpr bool MIX = CF::MIX;
  constexpr int DoF = CF::DoF, RS = CF::RS, PL = CF::PL;
  using CT = typename std::conditional<MIX, float, double>::type;
  const int nz = P.nz;
  const size_t cs = (size_t)DoF * nz, fs = (size_t)nz * P.NumG;
  R *s = reinterpret_cast<R *>(sm);
  constexpr int S_C = 4, S_K = 6, S_P = 7, S_2 = 8;   // first plane of each group
  R *sw = s + (size_t)CF::M_PLANES * PL;              // [4][LT+1][RS]: -h12 w, -h22 w, -h11 w, -h21 w; row 0 is level L0-1
  R *xh = sw + (size_t)4 * (PL + RS);                 // [2][RS]: the w-curls of level L0-1
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT;
  const int l = L0 + lvl;
  const bool act = ID < DoF && l < nz;
  const int I = ID % N, Jn = ID / N;
  const int row = lvl * RS, si = row + ID;
  const double *hn = P.hm + (size_t)IF * H_N * DoF + ID;
  const unsigned lanes = block_lanes<TH>();
#define SP(q) s[(q) * PL + si]
#define SWP(q, r, id) sw[((q) * (LT + 1) + (r)) * RS + (id)]

  // ---------------- operands of the first round ----------------
  double rho = 1.0, u = 0.0, v = 0.0, wh = 0.0, wl = 0.0, pr = 0.0, rm = 0.0;
  // rho, u, v, p of level l + 1; u, v of level l - 1; rho z of levels l - 1, l, l + 1
  double ua = 0.0, va = 0.0, pa = 0.0, ub = 0.0, vb = 0.0, sa = 1.0, sb = 1.0;
  if (act) {
    const int g = P.glob[IF * DoF + ID];
    const double *Ug = U + (size_t)nz * g + l;
    R ca[4];
    cache_sums<MIX, 0, 4>(P, C1, IF * DoF + ID, l, ca);
    rho = Ug[0]; u = Ug[fs]; v = Ug[2 * fs]; wh = Ug[3 * fs];
    const double *pg = Pr + (size_t)nz * g + l;
    pr = pg[0];
    const double zr = rho * P.zl[l];
    if (l > 0) {   // below: the same cache lines as the own level's
      wl = Ug[3 * fs - 1];
      ub = Ug[fs - 1]; vb = Ug[2 * fs - 1];
      sb = Ug[-1] * P.zl[l - 1] + zr;
    }
    if (l < nz - 1) {
      ua = Ug[fs + 1]; va = Ug[2 * fs + 1]; pa = pg[1];
      sa = zr + Ug[1] * P.zl[l + 1];
    }
    rm = hn[H_RM * DoF];
    const double a11 = hn[H_11 * DoF], a12 = hn[H_12 * DoF], a21 = hn[H_21 * DoF], a22 = hn[H_22 * DoF];
    const R h11 = (R)a11, h12 = (R)a12, h21 = (R)a21, h22 = (R)a22;
    const R c1 = ca[0], c2 = ca[1], c3 = ca[2], c4 = ca[3];
    SP(0) = h11 * c2 - h12 * c1;       // Curl12(Cache1, Cache2)
    SP(1) = h21 * c2 - h22 * c1;
    SP(2) = h11 * c3 + h12 * c4;       // Contra12(Cache3, Cache4)
    SP(3) = h21 * c3 + h22 * c4;
    const R whR = (R)wh, uR = (R)u, vR = (R)v;
    SWP(0, lvl + 1, ID) = -h12 * whR; SWP(1, lvl + 1, ID) = -h22 * whR;   // tempuZ1, tempuZ2
    SWP(2, lvl + 1, ID) = -h11 * whR; SWP(3, lvl + 1, ID) = -h21 * whR;   // tempvZ1, tempvZ2
    if (lvl == 0) {
      const R w1 = (R)wl;
      SWP(0, 0, ID) = -h12 * w1; SWP(1, 0, ID) = -h22 * w1;
      SWP(2, 0, ID) = -h11 * w1; SWP(3, 0, ID) = -h21 * w1;
    }
    SP(S_C + 0) = h12 * uR - h11 * vR;   // tempwZ1
    SP(S_C + 1) = h22 * uR - h21 * vR;   // tempwZ2
    SP(S_K) = (R)((u * u + v * v) + 0.5 * (wl * wl + wh * wh));   // K of both nodes
    // pressure (the mixed form: its perturbation from the level's FP64 reference)
    SP(S_P) = (R)(pr - (MIX ? P.pref[l] : 0.0));
  }
  __syncthreads();

  // ---------------- first derivatives ----------------
  R U2 = 0, V2 = 0, W = 0, KX = 0, KY = 0, PX = 0, PY = 0;
  if (act) {
    R DI[N], DJ[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      DI[k] = (R)P.D[I + N * k];
      DJ[k] = (R)P.D[Jn + N * k];
    }
    const R *x0 = s + row + N * Jn, *y0 = s + row + I;   // row Jn and column I of a plane
#define DX(q, k) x0[(q) * PL + (k)]
#define DY(q, k) y0[(q) * PL + N * (k)]
    const R rJ = (R)hn[H_RJ * DoF];
    R cu = DI[0] * DX(0, 0) + DJ[0] * DY(1, 0);
    R dv = DI[0] * DX(2, 0) + DJ[0] * DY(3, 0);
#pragma unroll
    for (int k = 1; k < N; ++k) {
      cu = fsum2(cu, DI[k], DX(0, k), DJ[k], DY(1, k));
      dv = fsum2(dv, DI[k], DX(2, k), DJ[k], DY(3, k));
    }
    SP(S_2 + 0) = cu * rJ;
    SP(S_2 + 1) = dv * rJ;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      U2 = fsum2(U2, DI[k], SWP(0, lvl + 1, k + N * Jn), DJ[k], SWP(1, lvl + 1, I + N * k));
      V2 = fsum2(V2, DI[k], SWP(2, lvl + 1, k + N * Jn), DJ[k], SWP(3, lvl + 1, I + N * k));
      W = fsum2(W, DI[k], DX(S_C + 0, k), DJ[k], DY(S_C + 1, k));
    }
    // the levels' slope residue in the curl of (u, v)
    const double *sd = P.zl + (size_t)(6 + N) * nz + l;
    W = fsum2(W, (R)-sd[I * nz], SP(S_C + 0), (R)-sd[Jn * nz], SP(S_C + 1));
    KX = DI[0] * DX(S_K, 0); KY = DJ[0] * DY(S_K, 0);
    PX = DI[0] * DX(S_P, 0); PY = DJ[0] * DY(S_P, 0);
#pragma unroll
    for (int k = 1; k < N; ++k) {
      KX = fsum1(KX, DI[k], DX(S_K, k));
      KY = fsum1(KY, DJ[k], DY(S_K, k));
      PX = rsum1(PX, DI[k], DX(S_P, k));
      PY = rsum1(PY, DJ[k], DY(S_P, k));
    }
  }
  if (L0 > 0 && t < DoF) {   // the w-curls of the level below the tile
    const int In = t % N, Jt = t / N;
    R x = 0, y = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const R di = (R)P.D[In + N * k], dj = (R)P.D[Jt + N * k];
      x = fsum2(x, di, SWP(0, 0, k + N * Jt), dj, SWP(1, 0, In + N * k));
      y = fsum2(y, di, SWP(2, 0, k + N * Jt), dj, SWP(3, 0, In + N * k));
    }
    xh[t] = x;
    xh[RS + t] = y;
  }
  __syncthreads();

  // ---------------- contributions ----------------
  R U1 = __shfl_up_sync(lanes, U2, 1, LT), V1 = __shfl_up_sync(lanes, V2, 1, LT);
  if (!act) return;
  if (lvl == 0) {
    U1 = l > 0 ? xh[ID] : (R)0;
    V1 = l > 0 ? xh[RS + ID] : (R)0;
  }
  const bool top = l < nz - 1, bot = l > 0;
  CT *out = reinterpret_cast<CT *>(C) + ((size_t)IF * P.NC * DoF + ID) * nz + l;
  const double h33 = hn[H_33 * DoF], hJ = hn[H_J * DoF], z = P.zl[l];
  // w: upper node (interface l) and lower node (interface l - 1)
  {
    const double q = 0.5 * (u * u + v * v);
    double whi = 0.0;
    if (top) {
      const double dK = 0.5 * (ua * ua + va * va) - q + 0.5 * (wh * wh - wl * wl);
      const double kin = rho * (z * (u * V2 + v * U2) + 0.5 * h33 * (u * (ua - u) + v * (va - v) - dK));
      whi = (kin - (h33 * (pa - pr) + P.Grav * hJ * sa)) * (rm / sa);
    }
    out[3 * cs] = (CT)whi;
    if (bot) {
      const double dK = q - 0.5 * (ub * ub + vb * vb) + 0.5 * (wh * wh - wl * wl);
      const double kin = rho * (z * (u * V1 + v * U1) + 0.5 * h33 * (u * (u - ub) + v * (v - vb) - dK));
      out[(size_t)P.NV * cs - 1] = (CT)(kin * (rm / sb));   // slot NV, one level down
    }
  }
  // u, v: hyperviscosity, momentum, gradients
  {
    R WI[N], WJ[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      WI[k] = (R)P.DW[I + N * k];
      WJ[k] = (R)P.DW[Jn + N * k];
    }
    const R *x0 = s + row + N * Jn, *y0 = s + row + I;
    R DxCurl = WI[0] * DX(S_2 + 0, 0), DyCurl = WJ[0] * DY(S_2 + 0, 0);
    R DxDiv = WI[0] * DX(S_2 + 1, 0), DyDiv = WJ[0] * DY(S_2 + 1, 0);
#pragma unroll
    for (int k = 1; k < N; ++k) {
      DxCurl = fsum1(DxCurl, WI[k], DX(S_2 + 0, k));
      DyCurl = fsum1(DyCurl, WJ[k], DY(S_2 + 0, k));
      DxDiv = fsum1(DxDiv, WI[k], DX(S_2 + 1, k));
      DyDiv = fsum1(DyDiv, WJ[k], DY(S_2 + 1, k));
    }
    const double h11 = hn[H_11 * DoF], h12 = hn[H_12 * DoF], h21 = hn[H_21 * DoF], h22 = hn[H_22 * DoF];
    const double hv_u = P.nuCurl * (h12 * DxCurl + h22 * DyCurl) - P.nuGrad * (h11 * DxDiv + h21 * DyDiv);
    const double hv_v = -P.nuCurl * (h11 * DxCurl + h21 * DyCurl) - P.nuGrad * (h12 * DxDiv + h22 * DyDiv);
    // vertical advection: 0.5 d33 (u(l) - u(l-1)) and so on, over 2 z
    const double fz = 0.25 * h33 * P.zl[nz + l];
    const double dub = bot ? u - ub : 0.0, dvb = bot ? v - vb : 0.0;
    const double dua = top ? ua - u : 0.0, dva = top ? va - v : 0.0;
    const double fc = hn[H_FC * DoF] * hJ, rr = 1.0 / rho;
    const double mom_u = -v * W - 0.5 * (wl * V1 + wh * V2) + v * fc - fz * (wl * dub + wh * dua);
    const double mom_v = u * W - 0.5 * (wl * U1 + wh * U2) - u * fc - fz * (wl * dvb + wh * dva);
    // pressure gradient over rho, and gravity along the levels' slope residue
    const double gs = 0.5 * P.Grav * hJ / h33;
    const double *ss = P.zl + (size_t)6 * nz + l;
    const double px = PX * rr + gs * ss[I * nz], py = PY * rr + gs * ss[Jn * nz];
    const double gr_u = -0.5 * (h11 * KX + h21 * KY) - (h11 * px + h21 * py);
    const double gr_v = -0.5 * (h12 * KX + h22 * KY) - (h12 * px + h22 * py);
    out[cs] = (CT)(rm * (hv_u + mom_u + gr_u));
    out[2 * cs] = (CT)(rm * (hv_v + mom_v + gr_v));
  }
#undef DX
#undef DY
#undef SP
#undef SWP
}

// item: 2 * tile + role (even: momentum, odd: scalars); TH: threads of the block
template <int N, int NT, typename R, int LT = p2_levels<N>(), int TH = P2Flat<N, NT, R, LT>::THREADS>
__device__ __forceinline__ void phase2_flat(const GP &P, const double *__restrict__ U, const double *__restrict__ Pr,
                                            const double *__restrict__ C1, double *__restrict__ C, const int item,
                                            const int IF)
{
  extern __shared__ double sm[];
  const int L0 = (item >> 1) * LT;
  if (item & 1) phase2_scalars_flat<N, NT, R, LT, TH>(P, U, C1, C, L0, IF, sm);
  else phase2_momentum_flat<N, NT, R, LT, TH>(P, U, Pr, C1, C, L0, IF, sm);
}

template <int N, int NT, typename R>
__global__ void __launch_bounds__(HV1Tile<N, R>::THREADS, HV1Tile<N, R>::MINB)
    k_hypervisc1_flat(const GP P, const double *__restrict__ U, double *__restrict__ C, double *__restrict__ Pr)
{
  extern __shared__ __align__(16) unsigned char hv1_dyn[];
  hypervisc1_flat<N, NT, R, HV1Tile<N, R>::LT>(P, U, C, Pr, blockIdx.x, launch_element(P),
                                               reinterpret_cast<R *>(hv1_dyn));
}

template <int N, int NT, typename R>
__global__ void __launch_bounds__(P2Flat<N, NT, R>::THREADS, P2Flat<N, NT, R>::MINB)
    k_phase2_flat(const GP P, const double *__restrict__ U, const double *__restrict__ Pr,
                  const double *__restrict__ C1, double *__restrict__ C)
{
  phase2_flat<N, NT, R>(P, U, Pr, C1, C, blockIdx.x, launch_element(P));
}

// The roles in launches of their own: the scalars' needs fewer registers, so
// that half as many CTAs again fit an SM (48 registers; at p = 4 three CTAs
// instead of two), which one launch of both cannot use.  Against it stand the
// second launch's start and tail.  The crossover lies at as many threads of a
// role for every p, later with tracers, which take registers and shared memory
// of the scalars' gain, and earlier in the mixed form.  One launch / two, us:
//
//              no tracer                      two tracers
//   p 4        1.23 M threads 131 / 132       1.92 M threads 244 / 250
//              1.92 M         201 / 199       4.87 M         599 / 595
//              17.3 M        1754 / 1641      17.3 M        2140 / 2069
//   p 4 mixed  1.04 M threads 103 / 101       1.04 M threads 125 / 124
//   p 2        1.04 M threads 95.2 / 95.9     2.33 M threads 253 / 255
//              1.75 M         159 / 157       4.15 M         444 / 438
//   p 1        1.04 M threads 70.3 / 70.7     1.38 M threads 117 / 119
//              1.38 M         94.2 / 91.5     2.46 M         204 / 202
//
// (A line at 4096 CTAs, whatever their size, cost up to 7 % at p 1 and 2.)  The
// momentum role at 48 registers spills and takes longer (0.89 for 0.79 ms of
// both, drop-in grid).
template <int N, int NT, typename R>
constexpr long long p2_split_threads() { return (sizeof(R) == sizeof(float) ? 500000LL : 750000LL) * (2 + NT); }

template <int N, typename R>
__global__ void __launch_bounds__(P2Flat<N, 0, R>::THREADS, P2Flat<N, 0, R>::MINB)
    k_phase2_momentum(const GP P, const double *__restrict__ U, const double *__restrict__ Pr,
                      const double *__restrict__ C1, double *__restrict__ C)
{
  extern __shared__ double sm[];
  using F = P2Flat<N, 0, R>;   // (the role is the same with tracers)
  phase2_momentum_flat<N, 0, R, F::LT, F::THREADS>(P, U, Pr, C1, C, blockIdx.x * F::LT, launch_element(P), sm);
}

template <int N, int NT, typename R>
__global__ void __launch_bounds__(P2Flat<N, NT, R>::THREADS, P2Flat<N, NT, R>::MINB_S)
    k_phase2_scalars(const GP P, const double *__restrict__ U, const double *__restrict__ C1, double *__restrict__ C)
{
  extern __shared__ double sm[];
  using F = P2Flat<N, NT, R>;
  phase2_scalars_flat<N, NT, R, F::LT, F::THREADS>(P, U, C1, C, blockIdx.x * F::LT, launch_element(P), sm);
}

}  // namespace cgd
