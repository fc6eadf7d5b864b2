// cgd_phase2.cuh - the fused tendency kernel (phase 2 of the RHS).
//
// One CTA per (element, tile of LT levels, role); one thread per (node,
// level), level fastest, so the state, metric and cache loads and the
// contribution stores are runs of consecutive levels.  Two roles share the
// work of a tile, each with about half of the tendency's live state:
//
//   scalars   hyperviscosity of theta and the tracers, the limited vertical
//             fluxes and the horizontal flux divergences -> contributions to
//             rho, rho*theta and the tracers
//   momentum  hyperviscosity of u and v, vector-invariant momentum + Coriolis,
//             kinetic-energy and pressure gradients with gravity
//             -> contributions to u, v and w
//
// The operands of the horizontal D/DW sums go through shared planes of
// LT x N^2 values (row stride odd, so that the 16 levels of a half warp fall
// into different banks); every operand of a round is written before one CTA
// barrier, so a role needs two barriers.  Values of the neighbouring levels
// come from the neighbouring lanes (shuffles within the LT lanes of a node)
// and, at the tile's ends, from halo rows that a few threads form beforehand.
//
// Bound by the L1/shared pipe and by the latency of its loads and barriers (61 %
// of the pipe's peak, 98 M shared-load and 72 M global-load wavefronts a launch,
// before it summed the phase-1 contributions itself).  One thread per (node,
// level) instead of one warp per level with 25 of 32 lanes, two roles at 72
// registers (26 warps an SM) instead of one at 128 (16 warps): nPanel 30, p 4, nz
// 45, two tracers 1.327 -> 1.224 ms, mixed form 1.247 -> 1.166 ms, nPanel 60, nz 64
// 5.65 -> 4.69 ms; with the phase-1 sums, which a kernel of 0.11 ms formed before,
// 1.226, 1.137 and 5.01 ms.
//
// The vertical momentum equation lives on interfaces: the contribution of
// the element node to w at interface l is hi(l) + lo(l+1), hi from the upper
// node of level l and lo from the lower node of level l+1.  Each level writes
// its hi into field 3 of the contribution buffer and its lo into the extra
// slot NV, one level down; the owner gather adds the pair per contributor.
//
// Expressions are the reference's (ViscKernel.jl:86-167,277-327,
// MomentumKernel.jl:1-178, GradKineticKernel.jl:1-129,
// OperatorKernel.jl:637-760) with the CPU restatement's per-node contribution
// order.  The exact build evaluates them term by term in its order; the fast
// build fuses the multiply-adds of the derivative sums, except those of the
// pressure (its 1e5 Pa make the balanced u, v tendencies small residuals:
// fused sums move them by 5e-12 relative), and sums the two vertical halves
// of the w-row curl before differentiating them.
#pragma once
#include "cgd_kernels.cuh"

namespace cgd {

// fused multiply-adds of the fast build's derivative sums (rsum1, rsum2 in the
// exact build)
template <typename R>
__device__ __forceinline__ R fsum1(R acc, R c, R x)
{
#ifdef CGD_FAST
  return fma(c, x, acc);
#else
  return rsum1(acc, c, x);
#endif
}
template <typename R>
__device__ __forceinline__ R fsum2(R acc, R c1, R x1, R c2, R x2)
{
#ifdef CGD_FAST
  return fma(c1, x1, fma(c2, x2, acc));
#else
  return rsum2(acc, c1, x1, c2, x2);
#endif
}

// RecU4's limiter max(0, min(r, min(k r + c, 1))) (OperatorKernel.jl:1044-1059)
// with selects that keep the reference's values for every r, a NaN r giving
// NaN, at a third of the instructions of cgd_min/cgd_max.
__device__ __forceinline__ double upwind_limit(double r, double k, double c)
{
  const double lin = k * r + c;
  const double m2 = lin > 1.0 ? 1.0 : lin;
  const double m1 = m2 < r ? m2 : r;
  return m1 <= 0.0 ? 0.0 : m1;
}

// The limited upwind flux of one interface, 0.25 ((|w| + w) cFL + (-|w| + w) cFR):
// one of the two factors is zero and the other 2 w, so only the upwind side's
// reconstruction is formed (the same value: the factors are exact).  c: the
// ratios of the node, rows rs apart; u1, d1 the rows of the upwind and the
// downwind level, u2 the row beyond the upwind one.
__device__ __forceinline__ double upwind_flux(const double *c, int rs, int u1, int d1, int u2, double kc, double ks,
                                              double w)
{
  const double c1 = c[u1 * rs], dc = c[d1 * rs] - c1;
  const double r = (c1 - c[u2 * rs]) / (dc + 1.e-20);
  return 0.5 * (w * (c1 + upwind_limit(r, ks, kc) * dc));
}

// A load the compiler may not merge with an earlier one of the same address:
// the metric of a thread's node is read again (from L1) where it is needed
// instead of being held in registers across a barrier.
__device__ __forceinline__ double ld_again(const double *p)
{
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];\n" : "=d"(v) : "l"(p));
  return v;
}

// Level tile of phase 2: LT levels of one element, a power of two (the lanes
// of a node exchange levels by shuffles of width LT).
template <int N>
constexpr int p2_levels() { return N == 2 ? 32 : 16; }

#ifdef CGD_FAST
constexpr int P2_WPLANES = 2;   // the curl of (u, v): both vertical halves summed
#else
constexpr int P2_WPLANES = 4;
#endif

template <int N, int NT, typename R, int LT_ = p2_levels<N>()>
struct P2Cfg {
  static constexpr int DoF = N * N, LT = LT_;
  static constexpr int RS = DoF | 1;             // row stride of a plane
  static constexpr int PL = LT * RS;             // values of a plane
  static constexpr int NS = 1 + NT;              // theta and the tracers
  static constexpr int LC = LT;
  static constexpr int THREADS = LT * DoF;
  static constexpr bool MIX = sizeof(R) == sizeof(float);
  // scalars: ratios of the tile and two halo levels on each side (double),
  // three halo rows of mass-flux parts, 1 + NS halo fluxes; planes: cache,
  // contravariant mass flux (2), second-round operands (2 per scalar), and in
  // the mixed form the ratios as R
  static constexpr size_t S_BYTES = ((size_t)NS * (LT + 4) * RS + (size_t)(3 + 1 + NS) * RS) * sizeof(double) +
                                    (size_t)(3 * NS + 2 + (MIX ? NS : 0)) * PL * sizeof(R);
  // momentum: 13 halo rows (double); planes: cache (4), w times the metric
  // (8), the curl of (u, v), K of both nodes, pressure, second round (2)
  static constexpr int M_PLANES = 4 + 8 + P2_WPLANES + 3 + 2;
  static constexpr size_t M_BYTES = (size_t)13 * RS * sizeof(double) + (size_t)M_PLANES * PL * sizeof(R);
  static constexpr size_t SMEM = S_BYTES > M_BYTES ? S_BYTES : M_BYTES;
  // CTAs per SM the registers are sized for: 25 warps of at most 80 registers a thread
  static constexpr int MINB = 800 / THREADS;
};

// items of the tiles of one element: two roles per tile
template <typename CF>
__host__ __device__ constexpr int p2_items(int nz) { return 2 * ((nz + CF::LT - 1) / CF::LT); }

// lanes of this thread's warp that exist in a block of TH threads
template <int TH>
__device__ __forceinline__ unsigned block_lanes()
{
  return (TH % 32 != 0 && (int)threadIdx.x / 32 == TH / 32) ? (1u << (TH % 32)) - 1u : 0xffffffffu;
}

template <int N, int NT, typename R, int LT, int TH>
__device__ __forceinline__ void phase2_scalars(const GP &P, const double *__restrict__ U,
                                               const double *__restrict__ C1, double *__restrict__ C, const int L0,
                                               const int IF, double *sm)
{
  using CF = P2Cfg<N, NT, R, LT>;
  constexpr bool MIX = CF::MIX;
  constexpr int DoF = CF::DoF, RS = CF::RS, PL = CF::PL, NS = CF::NS, CR = LT + 4;
  using CT = typename std::conditional<MIX, float, double>::type;   // stored cache and contributions
  const int nz = P.nz, NumG = P.NumG;
  const size_t cs = (size_t)DoF * nz, fs = (size_t)nz * NumG;
  double *cth = sm;                              // [NS][CR][RS] ratios, rows L0-2 .. L0+LT+1
  double *aa = cth + (size_t)NS * CR * RS;       // upper mass-flux part of level L0-1
  double *bl = aa + RS;                          // lower part of level L0
  double *bh = bl + RS;                          // lower part of level L0+LT
  double *fxh = bh + RS;                         // [1+NS][RS] fluxes of interface L0-1
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
  const double *mt = P.met + ((size_t)IF * NCOMP * DoF + ID) * nz + l;

  // ---------------- operands of the first round, vertical halo ----------------
  double rho = 1.0, A = 0.0, B = 0.0, JsD = 1.0, MCD = 1.0;
  double d11s = 0.0, d12s = 0.0, d21s = 0.0, d22s = 0.0;
  if (act) {
    const int g = P.glob[IF * DoF + ID];
    const double *Ug = U + (size_t)nz * g + l;
    R ca[NS];
    cache_sums<MIX, 4, NS>(P, C1, IF * DoF + ID, l, ca);
    rho = Ug[0];
    const double u = Ug[fs], v = Ug[2 * fs], wh = Ug[3 * fs], wm = l > 0 ? Ug[3 * fs - 1] : 0.0;
    d11s = mt[C_D11_0 * cs] + mt[C_D11_1 * cs];
    d12s = mt[C_D12_0 * cs] + mt[C_D12_1 * cs];
    d21s = mt[C_D21_0 * cs] + mt[C_D21_1 * cs];
    d22s = mt[C_D22_0 * cs] + mt[C_D22_1 * cs];
    JsD = mt[C_J0 * cs] + mt[C_J1 * cs];
    MCD = P.M[l + (size_t)nz * g] + P.M[l + (size_t)nz * (g + (size_t)NumG)];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      sc[q * PL + si] = ca[q];
      const double c = Ug[(4 + q) * fs] / rho;
      cth[(q * CR + lvl + 2) * RS + ID] = c;
      if (MIX) sq[q * PL + si] = (R)c;
    }
    scon[si] = (R)(-rho * (d11s * u + d12s * v));           // Contra12(-Rho, u, v)
    scon[PL + si] = (R)(-rho * (d21s * u + d22s * v));
    // the two parts of the vertical mass flux: of interface l from this
    // level, and of interface l - 1 from this level
    A = rho * (mt[C_D31_1 * cs] * u + mt[C_D32_1 * cs] * v + mt[C_D33_1 * cs] * wh);
    B = rho * (mt[C_D31_0 * cs] * u + mt[C_D32_0 * cs] * v + mt[C_D33_0 * cs] * wm);
    if (lvl == 0) bl[ID] = B;
  }
  for (int s = t; s < 4 * DoF; s += TH) {   // levels L0-2, L0-1, L0+LT, L0+LT+1
    const int n = s >> 2, h = s & 3, r = h < 2 ? h : LT + h;
    const int lev = L0 - 2 + r;
    if (lev < 0 || lev >= nz) continue;
    const double *Ug = U + (size_t)nz * P.glob[IF * DoF + n] + lev;
    const double rh = Ug[0];
#pragma unroll
    for (int q = 0; q < NS; ++q) cth[(q * CR + r) * RS + n] = Ug[(4 + q) * fs] / rh;
    const double *m = P.met + ((size_t)IF * NCOMP * DoF + n) * nz + lev;
    if (h == 1)
      aa[n] = rh * (m[C_D31_1 * cs] * Ug[fs] + m[C_D32_1 * cs] * Ug[2 * fs] + m[C_D33_1 * cs] * Ug[3 * fs]);
    else if (h == 2)
      bh[n] = rh * (m[C_D31_0 * cs] * Ug[fs] + m[C_D32_0 * cs] * Ug[2 * fs] + m[C_D33_0 * cs] * Ug[3 * fs - 1]);
  }
  __syncthreads();

  // ---------------- vertical fluxes of interface l ----------------
  // wCon and the limited upwind fluxes between levels il and il + 1, row pl
  // of the ratios holding level il, m the metric of that level
  auto fluxes = [&](int il, int pl, int n, const double *m, double wCon, double *f) {
    const bool up = wCon > 0.0;
    const double kc = m[(up ? C_RK0 : C_RK2) * cs], ks = m[(up ? C_RK1 : C_RK3) * cs];
    const int far = up ? (il > 0 ? pl - 1 : pl) : (il + 2 < nz ? pl + 2 : pl + 1);
    f[0] = wCon;
#pragma unroll
    for (int q = 0; q < NS; ++q)
      f[1 + q] = upwind_flux(cth + (size_t)q * CR * RS + n, RS, up ? pl : pl + 1, up ? pl + 1 : pl, far, kc, ks, wCon);
  };
  const unsigned lanes = block_lanes<TH>();
  double Ft[1 + NS];
#pragma unroll
  for (int q = 0; q < 1 + NS; ++q) Ft[q] = 0.0;
  {
    double Bup = __shfl_down_sync(lanes, B, 1, LT);
    if (act && l < nz - 1) {
      if (lvl == LT - 1) Bup = bh[ID];
      fluxes(l, lvl + 2, ID, mt, A + Bup, Ft);
    }
  }
  if (L0 > 0 && t < DoF) {   // the interface below the tile
    double f[1 + NS];
    fluxes(L0 - 1, 1, t, P.met + ((size_t)IF * NCOMP * DoF + t) * nz + L0 - 1, aa[t] + bl[t], f);
#pragma unroll
    for (int q = 0; q < 1 + NS; ++q) fxh[q * RS + t] = f[q];
  }

  // ---------------- first derivatives, flux divergences ----------------
  const R Js = (R)JsD, rJs = (R)(1.0 / JsD);
  (void)Js; (void)rJs;
  R DivRho = 0, Div[NS];
  if (act) {
    R DI[N], DJ[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      DI[k] = (R)P.D[I + N * k];
      DJ[k] = (R)P.D[Jn + N * k];
    }
    const R d11 = (R)d11s, d12 = (R)d12s, d21 = (R)d21s, d22 = (R)d22s;
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const R *c = sc + q * PL + row;
      R Dxc = DI[0] * c[N * Jn], Dyc = DJ[0] * c[I];
#pragma unroll
      for (int k = 1; k < N; ++k) {
        Dxc = fsum1(Dxc, DI[k], c[k + N * Jn]);
        Dyc = fsum1(Dyc, DJ[k], c[I + N * k]);
      }
      const R GradDx = CGD_DIVJ(d11 * Dxc + d21 * Dyc);
      const R GradDy = CGD_DIVJ(d12 * Dxc + d22 * Dyc);
      s2[(2 * q) * PL + si] = rho * (d11 * GradDx + d12 * GradDy);
      s2[(2 * q + 1) * PL + si] = rho * (d21 * GradDx + d22 * GradDy);
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
  // accumulated in the restatement's order: rho: flux top, flux bottom,
  // horizontal divergence; rho*theta and tracers: hyperviscosity, flux top,
  // flux bottom, horizontal divergence
  double Fb[1 + NS];
#pragma unroll
  for (int q = 0; q < 1 + NS; ++q) Fb[q] = __shfl_up_sync(lanes, Ft[q], 1, LT);
  if (!act) return;
  const bool top = l < nz - 1, bot = l > 0;
  if (lvl == 0 && bot) {
#pragma unroll
    for (int q = 0; q < 1 + NS; ++q) Fb[q] = fxh[q * RS + ID];
  }
  const double MC = MCD, rMC = 1.0 / MCD;
  (void)MC; (void)rMC;
  CT *out = reinterpret_cast<CT *>(C) + ((size_t)IF * P.NC * DoF + ID) * nz + l;
  double acc = 0.0;
  if (top) acc += CGD_DIVM(-(0.5 * Ft[0]));
  if (bot) acc += CGD_DIVM(0.5 * Fb[0]);
  acc += CGD_DIVM(DivRho);
  out[0] = (CT)acc;
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
    acc = 0.0;
    acc += CGD_DIVM(-P.nuDiv * Lap);
    if (top) acc += CGD_DIVM(-Ft[1 + q]);
    if (bot) acc += CGD_DIVM(Fb[1 + q]);
    acc += CGD_DIVM(Div[q]);
    out[(4 + q) * cs] = (CT)acc;
  }
}

template <int N, int NT, typename R, int LT, int TH>
__device__ __forceinline__ void phase2_momentum(const GP &P, const double *__restrict__ U,
                                                const double *__restrict__ Pr, const double *__restrict__ C1,
                                                double *__restrict__ C, const int L0, const int IF, double *sm)
{
  using CF = P2Cfg<N, NT, R, LT>;
  constexpr bool MIX = CF::MIX;
  constexpr int DoF = CF::DoF, RS = CF::RS, PL = CF::PL;
  using CT = typename std::conditional<MIX, float, double>::type;
  const int nz = P.nz, NumG = P.NumG;
  const size_t cs = (size_t)DoF * nz, fs = (size_t)nz * NumG;
  // halo rows: of level L0-1 tu1, tv1, tw1, K2, rho M1; of level L0+LT tu0,
  // tv0, tw0, K1, rho M0, p, d33 (lower node), rho J0
  double *hb = sm, *ha = sm + 5 * RS;
  R *s = reinterpret_cast<R *>(sm + 13 * RS);
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT;
  const int l = L0 + lvl;
  const bool act = ID < DoF && l < nz;
  const int I = ID % N, Jn = ID / N;
  const int row = lvl * RS, si = row + ID;
  const double *mt = P.met + ((size_t)IF * NCOMP * DoF + ID) * nz + l;
  constexpr int S_W = 4, S_C = 12, S_K = 12 + P2_WPLANES, S_2 = S_K + 3;   // first plane of each group
#define SP(q) s[(q) * PL + si]

  // ---------------- operands of the first round, vertical halo ----------------
  int g = 0;
  double rho = 1.0, u = 0.0, v = 0.0, wh = 0.0, wl = 0.0, pr = 0.0;
  double tu0 = 0.0, tv0 = 0.0, tw0 = 0.0, tu1 = 0.0, tv1 = 0.0, tw1 = 0.0;
  if (act) {
    g = P.glob[IF * DoF + ID];
    const double *Ug = U + (size_t)nz * g + l;
    R ca[4];
    cache_sums<MIX, 0, 4>(P, C1, IF * DoF + ID, l, ca);
    rho = Ug[0]; u = Ug[fs]; v = Ug[2 * fs]; wh = Ug[3 * fs];
    pr = Pr[l + (size_t)nz * g];
    const double c110 = mt[C_D11_0 * cs], c111 = mt[C_D11_1 * cs], c120 = mt[C_D12_0 * cs], c121 = mt[C_D12_1 * cs];
    const double c210 = mt[C_D21_0 * cs], c211 = mt[C_D21_1 * cs], c220 = mt[C_D22_0 * cs], c221 = mt[C_D22_1 * cs];
    const double e310 = mt[C_D31_0 * cs], e311 = mt[C_D31_1 * cs], e320 = mt[C_D32_0 * cs], e321 = mt[C_D32_1 * cs];
    const double e330 = mt[C_D33_0 * cs], e331 = mt[C_D33_1 * cs];
    // surface w from no normal flow (MomentumKernel.jl:35-36)
    wl = l == 0 ? -(e310 * u + e320 * v) / e330 : Ug[3 * fs - 1];
    {
      const R d11 = (R)(c110 + c111), d12 = (R)(c120 + c121), d21 = (R)(c210 + c211), d22 = (R)(c220 + c221);
      const R c1 = ca[0], c2 = ca[1], c3 = ca[2], c4 = ca[3];
      SP(0) = d11 * c2 - d12 * c1;       // Curl12(Cache1, Cache2)
      SP(1) = d21 * c2 - d22 * c1;
      SP(2) = d11 * c3 + d12 * c4;       // Contra12(Cache3, Cache4)
      SP(3) = d21 * c3 + d22 * c4;
    }
    {
      const R d110 = (R)c110, d111 = (R)c111, d120 = (R)c120, d121 = (R)c121;
      const R d210 = (R)c210, d211 = (R)c211, d220 = (R)c220, d221 = (R)c221;
      const R wlR = (R)wl, whR = (R)wh, uR = (R)u, vR = (R)v;
      SP(S_W + 0) = -d120 * wlR; SP(S_W + 1) = -d220 * wlR;   // tempuZ1, tempuZ2 (lower)
      SP(S_W + 2) = -d121 * whR; SP(S_W + 3) = -d221 * whR;   // (upper)
      SP(S_W + 4) = -d110 * wlR; SP(S_W + 5) = -d210 * wlR;   // tempvZ1, tempvZ2 (lower)
      SP(S_W + 6) = -d111 * whR; SP(S_W + 7) = -d211 * whR;   // (upper)
#ifdef CGD_FAST
      SP(S_C + 0) = (R)(c120 + c121) * uR - (R)(c110 + c111) * vR;   // tempwZ1, both nodes
      SP(S_C + 1) = (R)(c220 + c221) * uR - (R)(c210 + c211) * vR;   // tempwZ2
#else
      SP(S_C + 0) = d120 * uR - d110 * vR;                    // tempwZ1
      SP(S_C + 1) = d220 * uR - d210 * vR;                    // tempwZ2
      SP(S_C + 2) = d121 * uR - d111 * vR;
      SP(S_C + 3) = d221 * uR - d211 * vR;
#endif
    }
    SP(S_K + 0) = (R)(0.5 * (u * u + v * v) + 0.5 * (wl * wl));   // K on the bottom node
    SP(S_K + 1) = (R)(0.5 * (u * u + v * v) + 0.5 * (wh * wh));   // K on the top node
    // pressure (the mixed form: its perturbation from the level's FP64 reference)
    SP(S_K + 2) = (R)(pr - (MIX ? P.pref[l] : 0.0));
    tu0 = e330 * v - e320 * wl; tu1 = e331 * v - e321 * wh;
    tv0 = e330 * u - e310 * wl; tv1 = e331 * u - e311 * wh;
    tw0 = e320 * u - e310 * v; tw1 = e321 * u - e311 * v;
  }
  for (int x = t; x < 2 * DoF; x += TH) {
    const int n = x >> 1, above = x & 1;
    const int lev = above ? L0 + LT : L0 - 1;
    if (lev < 0 || lev >= nz) continue;
    const int gn = P.glob[IF * DoF + n];
    const double *Ug = U + (size_t)nz * gn + lev;
    const double *m = P.met + ((size_t)IF * NCOMP * DoF + n) * nz + lev + (above ? 0 : cs);   // node 0 or 1 of the level
    const double r1 = Ug[0], u1 = Ug[fs], v1 = Ug[2 * fs], w1 = above ? Ug[3 * fs - 1] : Ug[3 * fs];
    const double a31 = m[C_D31_0 * cs], a32 = m[C_D32_0 * cs], a33 = m[C_D33_0 * cs];
    double *h = (above ? ha : hb) + n;
    h[0] = a33 * v1 - a32 * w1;
    h[RS] = a33 * u1 - a31 * w1;
    h[2 * RS] = a32 * u1 - a31 * v1;
    h[3 * RS] = 0.5 * (u1 * u1 + v1 * v1) + 0.5 * (w1 * w1);
    h[4 * RS] = r1 * P.M[lev + (size_t)nz * (gn + (above ? 0 : (size_t)NumG))];
    if (above) {
      h[5 * RS] = Pr[lev + (size_t)nz * gn];
      h[6 * RS] = a33;
      h[7 * RS] = r1 * m[C_J0 * cs];
    }
  }
  __syncthreads();

  // ---------------- terms that couple the levels ----------------
  const bool top = act && l < nz - 1, bot = act && l > 0;
  const unsigned lanes = block_lanes<TH>();
  double FU = 0.0, FV = 0.0, FW1 = 0.0, FW2 = 0.0, den_hi = 1.0, den_lo = 1.0;
  const double K1s = 0.5 * (u * u + v * v) + 0.5 * (wl * wl);   // K on the bottom node
  const double K2s = 0.5 * (u * u + v * v) + 0.5 * (wh * wh);   // K on the top node
  double K2b = 0.0, K1a = 0.0, Gradp = 0.0, M0 = 1.0, M1 = 0.0, J0 = 0.5, J1 = 0.5;
  {
    double e330 = 1.0, e331 = 1.0;
    if (act) {
      M0 = P.M[l + (size_t)nz * g];
      M1 = P.M[l + (size_t)nz * (g + (size_t)NumG)];
      J0 = mt[C_J0 * cs];
      J1 = mt[C_J1 * cs];
      e330 = ld_again(mt + C_D33_0 * cs);
      e331 = ld_again(mt + C_D33_1 * cs);
    }
    const double rM0 = rho * M0, rM1 = rho * M1, rJ0 = rho * J0;
    double a = __shfl_up_sync(lanes, tu1, 1, LT), b = __shfl_up_sync(lanes, tv1, 1, LT);
    double c = __shfl_up_sync(lanes, tw1, 1, LT), k = __shfl_up_sync(lanes, K2s, 1, LT);
    double m = __shfl_up_sync(lanes, rM1, 1, LT);
    if (bot) {
      if (lvl == 0) { a = hb[ID]; b = hb[RS + ID]; c = hb[2 * RS + ID]; k = hb[3 * RS + ID]; m = hb[4 * RS + ID]; }
      const double FluxUZ = 0.5 * (tu0 - a);
      const double FluxVZ = 0.5 * (tv0 - b);
      const double FluxWZ = 0.5 * (tw0 - c);
      FU += (-v * FluxWZ - wl * FluxVZ);
      FV += (u * FluxWZ - wl * FluxUZ);
      FW1 += (u * FluxVZ + v * FluxUZ);
      den_lo = m + rM0;
      K2b = k;
    }
    a = __shfl_down_sync(lanes, tu0, 1, LT);
    b = __shfl_down_sync(lanes, tv0, 1, LT);
    c = __shfl_down_sync(lanes, tw0, 1, LT);
    k = __shfl_down_sync(lanes, K1s, 1, LT);
    m = __shfl_down_sync(lanes, rM0, 1, LT);
    double pa = __shfl_down_sync(lanes, pr, 1, LT), ea = __shfl_down_sync(lanes, e330, 1, LT);
    double ja = __shfl_down_sync(lanes, rJ0, 1, LT);
    if (top) {
      if (lvl == LT - 1) {
        a = ha[ID]; b = ha[RS + ID]; c = ha[2 * RS + ID]; k = ha[3 * RS + ID]; m = ha[4 * RS + ID];
        pa = ha[5 * RS + ID]; ea = ha[6 * RS + ID]; ja = ha[7 * RS + ID];
      }
      const double FluxUZt = 0.5 * (a - tu1);
      const double FluxVZt = 0.5 * (b - tv1);
      const double FluxWZt = 0.5 * (c - tw1);
      FU += (-v * FluxWZt - wh * FluxVZt);
      FV += (u * FluxWZt - wh * FluxUZt);
      FW2 += (u * FluxVZt + v * FluxUZt);
      den_hi = m + rM1;
      K1a = k;
      const double GZ = 0.5 * (pa - pr);
      const double Gradw = GZ * (e331 + ea);
      Gradp = -(Gradw + P.Grav * (rho * J1 + ja));
    }
  }
  const double JsD = J0 + J1, MCD = M0 + M1;
  const double rMC = 1.0 / MCD, MC = MCD;
  const R rJs = (R)(1.0 / JsD), Js = (R)JsD;
  (void)rMC; (void)MC; (void)rJs; (void)Js;

  // ---------------- first derivatives ----------------
#ifdef CGD_FAST
#define CGD_DIVW(x, d) ((x) * (1.0 / (d)))
#define CGD_DIVR(x) ((x) * (1.0 / rho))
#else
#define CGD_DIVW(x, d) ((x) / (d))
#define CGD_DIVR(x) ((x) / rho)
#endif
  double mom_u = 0.0, mom_v = 0.0, grad_u = 0.0, grad_v = 0.0;
  if (act) {
    CT *out = reinterpret_cast<CT *>(C) + ((size_t)IF * P.NC * DoF + ID) * nz + l;
    R DI[N], DJ[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      DI[k] = (R)P.D[I + N * k];
      DJ[k] = (R)P.D[Jn + N * k];
    }
    const R *x0 = s + row + N * Jn, *y0 = s + row + I;   // row Jn and column I of a plane
#define DX(q, k) x0[(q) * PL + (k)]
#define DY(q, k) y0[(q) * PL + N * (k)]
    // hyperviscosity: first derivatives of the DSS'd cache
    {
      R cu = DI[0] * DX(0, 0) + DJ[0] * DY(1, 0);
      R dv = DI[0] * DX(2, 0) + DJ[0] * DY(3, 0);
#pragma unroll
      for (int k = 1; k < N; ++k) {
        cu = fsum2(cu, DI[k], DX(0, k), DJ[k], DY(1, k));
        dv = fsum2(dv, DI[k], DX(2, k), DJ[k], DY(3, k));
      }
      SP(S_2 + 0) = CGD_DIVJ(cu);
      SP(S_2 + 1) = CGD_DIVJ(dv);
    }
    // vector-invariant momentum
    double whi = 0.0, wlo = 0.0;
    {
      R U1 = (R)(0.5 * (tu1 - tu0)), U2 = U1;
      R V1 = (R)(0.5 * (tv1 - tv0)), V2 = V1;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        U1 = fsum2(U1, DI[k], DX(S_W + 0, k), DJ[k], DY(S_W + 1, k));
        U2 = fsum2(U2, DI[k], DX(S_W + 2, k), DJ[k], DY(S_W + 3, k));
        V1 = fsum2(V1, DI[k], DX(S_W + 4, k), DJ[k], DY(S_W + 5, k));
        V2 = fsum2(V2, DI[k], DX(S_W + 6, k), DJ[k], DY(S_W + 7, k));
      }
      const double fc = mt[C_FCOR * cs];
      const double FuCor = v * fc, FvCor = -u * fc, FwCor = 0.0;
      FU += FuCor * JsD;
      FV += FvCor * JsD;
      FW1 += FwCor * J0;
      FW2 += FwCor * J1;
#ifdef CGD_FAST
      R W = (R)(tw1 - tw0);
#pragma unroll
      for (int k = 0; k < N; ++k) W = fsum2(W, DI[k], DX(S_C + 0, k), DJ[k], DY(S_C + 1, k));
      mom_u = CGD_DIVM(-v * W - wl * V1 - wh * V2 + FU);
      mom_v = CGD_DIVM(u * W - wl * U1 - wh * U2 + FV);
#else
      R W1 = (R)(0.5 * (tw1 - tw0)), W2 = W1;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        W1 = fsum2(W1, DI[k], DX(S_C + 0, k), DJ[k], DY(S_C + 1, k));
        W2 = fsum2(W2, DI[k], DX(S_C + 2, k), DJ[k], DY(S_C + 3, k));
      }
      mom_u = CGD_DIVM(-v * W1 - wl * V1 - v * W2 - wh * V2 + FU);
      mom_v = CGD_DIVM(u * W1 - wl * U1 + u * W2 - wh * U2 + FV);
#endif
      if (top) whi = CGD_DIVW(rho * (u * V2 + v * U2 + FW2), den_hi);
      if (bot) wlo = CGD_DIVW(rho * (u * V1 + v * U1 + FW1), den_lo);
    }
    // kinetic-energy and pressure gradients
    {
      R DXp = DI[0] * DX(S_K + 2, 0), DYp = DJ[0] * DY(S_K + 2, 0);
      R DXK1 = DI[0] * DX(S_K + 0, 0), DYK1 = DJ[0] * DY(S_K + 0, 0);
      R DXK2 = DI[0] * DX(S_K + 1, 0), DYK2 = DJ[0] * DY(S_K + 1, 0);
#pragma unroll
      for (int k = 1; k < N; ++k) {
        DXK1 = fsum1(DXK1, DI[k], DX(S_K + 0, k));
        DYK1 = fsum1(DYK1, DJ[k], DY(S_K + 0, k));
        DXK2 = fsum1(DXK2, DI[k], DX(S_K + 1, k));
        DYK2 = fsum1(DYK2, DJ[k], DY(S_K + 1, k));
        DXp = rsum1(DXp, DI[k], DX(S_K + 2, k));
        DYp = rsum1(DYp, DJ[k], DY(S_K + 2, k));
      }
      const double d110 = ld_again(mt + C_D11_0 * cs), d111 = ld_again(mt + C_D11_1 * cs);
      const double d120 = ld_again(mt + C_D12_0 * cs), d121 = ld_again(mt + C_D12_1 * cs);
      const double d210 = ld_again(mt + C_D21_0 * cs), d211 = ld_again(mt + C_D21_1 * cs);
      const double d220 = ld_again(mt + C_D22_0 * cs), d221 = ld_again(mt + C_D22_1 * cs);
      const double e310 = ld_again(mt + C_D31_0 * cs), e311 = ld_again(mt + C_D31_1 * cs);
      const double e320 = ld_again(mt + C_D32_0 * cs), e321 = ld_again(mt + C_D32_1 * cs);
      const double e330 = ld_again(mt + C_D33_0 * cs), e331 = ld_again(mt + C_D33_1 * cs);
      double GuF1 = -(d110 * DXK1 + d210 * DYK1);
      double GvF1 = -(d120 * DXK1 + d220 * DYK1);
      double GuF2 = -(d111 * DXK2 + d211 * DYK2);
      double GvF2 = -(d121 * DXK2 + d221 * DYK2);
      double Gradu = (d110 + d111) * DXp + (d210 + d211) * DYp;
      double Gradv = (d120 + d121) * DXp + (d220 + d221) * DYp;
      double GZ = -P.Grav * rho * JsD / (e330 + e331);
      Gradu += GZ * (e310 + e311);
      Gradv += GZ * (e320 + e321);
      // kinetic-energy jumps to the neighbour levels
      double GwF2 = 0.0;
      if (bot) {
        GZ = 0.5 * (K1s - K2b);
        GuF1 += -GZ * e310;
        GvF1 += -GZ * e320;
      }
      if (top) {
        GZ = 0.5 * (K1a - K2s);
        GuF2 += -GZ * e311;
        GvF2 += -GZ * e321;
        GwF2 += -rho * GZ * e331;
      }
      GZ = 0.5 * (K2s - K1s);
      GuF2 += -GZ * e311;
      GuF1 += -GZ * e310;
      GvF2 += -GZ * e321;
      GvF1 += -GZ * e320;
      GwF2 += -rho * GZ * e331;
      grad_u = CGD_DIVM(GuF1 + GuF2 - CGD_DIVR(Gradu));
      grad_v = CGD_DIVM(GvF1 + GvF2 - CGD_DIVR(Gradv));
      // w: upper node of l (interface l) and lower node of l (interface l-1)
      if (top) whi = whi + CGD_DIVW(GwF2 + Gradp, den_hi);
      if (bot) {
        double GwF1 = 0.0;
        double GZa = 0.5 * (K1s - K2b);
        GwF1 += -rho * GZa * e330;
        GZa = 0.5 * (K2s - K1s);
        GwF1 += -rho * GZa * e330;
        wlo = wlo + CGD_DIVW(GwF1, den_lo);
      }
    }
    out[3 * cs] = (CT)whi;
    if (bot) out[(size_t)P.NV * cs - 1] = (CT)wlo;   // slot NV, one level down
  }
  __syncthreads();

  // ---------------- weak derivatives of the hyperviscosity; contributions of u, v ----------------
  if (!act) return;
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
    const R d11 = (R)(ld_again(mt + C_D11_0 * cs) + ld_again(mt + C_D11_1 * cs));
    const R d12 = (R)(ld_again(mt + C_D12_0 * cs) + ld_again(mt + C_D12_1 * cs));
    const R d21 = (R)(ld_again(mt + C_D21_0 * cs) + ld_again(mt + C_D21_1 * cs));
    const R d22 = (R)(ld_again(mt + C_D22_0 * cs) + ld_again(mt + C_D22_1 * cs));
    const R FuC = d12 * DxCurl + d22 * DyCurl;
    const R FvC = -d11 * DxCurl - d21 * DyCurl;
    const R FuD = d11 * DxDiv + d21 * DyDiv;
    const R FvD = d12 * DxDiv + d22 * DyDiv;
    double acc_u = 0.0, acc_v = 0.0;
    acc_u += CGD_DIVM(-(-P.nuCurl * FuC + P.nuGrad * FuD));
    acc_v += CGD_DIVM(-(-P.nuCurl * FvC + P.nuGrad * FvD));
    acc_u += mom_u;
    acc_v += mom_v;
    acc_u += grad_u;
    acc_v += grad_v;
    CT *out = reinterpret_cast<CT *>(C) + ((size_t)IF * P.NC * DoF + ID) * nz + l;
    out[cs] = (CT)acc_u;
    out[2 * cs] = (CT)acc_v;
  }
#undef DX
#undef DY
#undef SP
#undef CGD_DIVW
#undef CGD_DIVR
}

// item: 2 * tile + role (even: momentum, odd: scalars); TH: threads of the block
template <int N, int NT, typename R, int LT = p2_levels<N>(), int TH = P2Cfg<N, NT, R, LT>::THREADS>
__device__ __forceinline__ void phase2_body(const GP &P, const double *__restrict__ U, const double *__restrict__ Pr,
                                            const double *__restrict__ C1, double *__restrict__ C, const int item,
                                            const int IF)
{
  extern __shared__ double sm[];
  const int L0 = (item >> 1) * LT;
  if (item & 1) phase2_scalars<N, NT, R, LT, TH>(P, U, C1, C, L0, IF, sm);
  else phase2_momentum<N, NT, R, LT, TH>(P, U, Pr, C1, C, L0, IF, sm);
}

template <int N, int NT, typename R>
__global__ void __launch_bounds__(P2Cfg<N, NT, R>::THREADS, P2Cfg<N, NT, R>::MINB)
    k_phase2(const GP P, const double *__restrict__ U, const double *__restrict__ Pr, const double *__restrict__ C1,
             double *__restrict__ C)
{
  phase2_body<N, NT, R>(P, U, Pr, C1, C, blockIdx.x, launch_element(P));
}

}  // namespace cgd
