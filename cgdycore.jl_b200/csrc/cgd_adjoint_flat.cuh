// cgd_adjoint_flat.cuh - the reverse of phase 2 on a flat product grid (the
// fast build; cgd_flat.cuh has the forward and the factors).
//
// The forward's layout: one CTA per (element, tile of LT levels, role), one
// thread per (node, level), level fastest; the scalars role reverses the
// contributions to rho and rho*theta, the momentum role those to u, v and w.
// Each recomputes the forward sums that its chain rule needs, puts the adjoints
// of every derivative sum into shared planes and forms the transposed sums
// (D^T, DW^T; a plane that feeds both is read once).  What a level's terms give
// to the neighbouring levels goes to the neighbouring lanes by shuffles, and
// at the tile's ends to memory, so a thread adds each of its level's state
// adjoints to LU once, with the level's other element nodes (global atomics,
// runs of consecutive levels).  The general kernel (k_phase2_adj) sums them by
// FP64 atomics in shared memory, about 50 a node and level, which are
// compare-and-swap loops.  nPanel 30, p 4, nz 45, no tracer: 2.33 -> 1.05 ms,
// and the adjoint of a step 14.7 -> 9.5 ms; registers capped for two CTAs an
// SM, with spills, beat one CTA an SM without them (10.5 ms a step).  The levels' slope residue (1e-16 of dXdxI(3,3)) is
// not differentiated.
#pragma once
#include "cgd_phase2.cuh"

namespace cgd {

template <int N>
struct AdjFlat {
  static constexpr int DoF = N * N, LT = p2_levels<N>(), RS = DoF | 1, PL = LT * RS, THREADS = LT * DoF;
  // scalars: theta of the tile and of two halo levels on each side; lambda_rho
  // and lambda_theta over M, the cache, the second round (2)
  static constexpr size_t S_BYTES = ((size_t)(LT + 4) * RS + (size_t)5 * PL) * sizeof(double);
  // momentum: forward operands h w (4, LT + 1 rows), curl of (u, v) (2), p;
  // adjoints of the w-curls (2, LT + 1 rows), of the curl of (u, v), K (2),
  // pressure (2), hyperviscous curl (2), second round (2)
  static constexpr size_t M_BYTES = ((size_t)6 * (PL + RS) + (size_t)12 * PL) * sizeof(double);
  static constexpr size_t SMEM = S_BYTES > M_BYTES ? S_BYTES : M_BYTES;
  static constexpr int MINB = 800 / THREADS;
};

// phi = max(0, min(r, min(k r + c, 1))) and its derivative in r (the branches
// of lim_phi in cgd_adjoint.cuh)
__device__ __forceinline__ double upwind_limit_d(double r, double k, double c, double &dphi)
{
  const double lin = k * r + c;
  double m = lin, dm = k;
  if (1.0 < lin) { m = 1.0; dm = 0.0; }
  if (!(m < r)) { m = r; dm = 1.0; }
  if (m > 0.0) { dphi = dm; return m; }
  dphi = 0.0;
  return 0.0;
}

template <int N>
__device__ __forceinline__ void phase2_scalars_adj(const GP &P, const double *__restrict__ U,
                                                   const double *__restrict__ T1, const double *__restrict__ LF,
                                                   double *__restrict__ LU, double *__restrict__ LT1, const int L0,
                                                   const int IF, double *sm)
{
  using CF = AdjFlat<N>;
  constexpr int DoF = CF::DoF, RS = CF::RS, PL = CF::PL, LT = CF::LT, TH = CF::THREADS;
  const int nz = P.nz;
  const size_t fs = (size_t)nz * P.NumG;
  double *th = sm;                    // [LT+4][RS] theta, rows L0-2 .. L0+LT+1
  double *s = th + (size_t)(LT + 4) * RS;   // planes: 0 lambda_rho/m, 1 lambda_theta/m, 2 cache, 3-4 second round
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT;
  const int l = L0 + lvl;
  const bool act = l < nz;
  const int I = ID % N, Jn = ID / N;
  const int row = lvl * RS, si = row + ID;
  const double *hn = P.hm + (size_t)IF * H_N * DoF + ID;
  const unsigned lanes = block_lanes<TH>();
  const int g = P.glob[IF * DoF + ID];
  const double *Ug = U + (size_t)nz * g + l, *Lg = LF + (size_t)nz * g + l;
  double *Og = LU + (size_t)nz * g + l;
  // halo: thread t < 4 DoF takes node t / 4 of level L0-2, L0-1, L0+LT or L0+LT+1
  static_assert(4 * DoF <= TH, "one halo slot per thread");
  const int hID = t >> 2, hr = (t & 3) < 2 ? (t & 3) : LT + (t & 3), hl = L0 - 2 + hr;
  const bool hs = t < 4 * DoF && hl >= 0 && hl < nz;
  double hrho = 1.0, hrth = 0.0;
  if (hs) {
    const double *Un = U + (size_t)nz * P.glob[IF * DoF + hID] + hl;
    hrho = Un[0];
    hrth = Un[4 * fs];
  }
  double rho = 1.0, u = 0.0, v = 0.0, wh = 0.0, thl = 0.0, ar = 0.0, at = 0.0;
  if (act) {
    const double rm = hn[H_RM * DoF];
    rho = Ug[0]; u = Ug[fs]; v = Ug[2 * fs]; wh = Ug[3 * fs];
    thl = Ug[4 * fs] / rho;
    ar = rm * Lg[0];
    at = rm * Lg[4 * fs];
    th[(lvl + 2) * RS + ID] = thl;
    s[si] = ar;
    s[PL + si] = at;
    s[2 * PL + si] = T1[(size_t)nz * g + l + 4 * fs];
  }
  if (hs) th[hr * RS + hID] = hrth / hrho;
  // neighbours above: state and lambda over z of level l + 1
  double ra = __shfl_down_sync(lanes, rho, 1, LT), ua = __shfl_down_sync(lanes, u, 1, LT);
  double va = __shfl_down_sync(lanes, v, 1, LT), ara = __shfl_down_sync(lanes, ar, 1, LT);
  double ata = __shfl_down_sync(lanes, at, 1, LT);
  const bool top = act && l < nz - 1;
  if (top && lvl == LT - 1) {
    const double rm = hn[H_RM * DoF];
    ra = Ug[1]; ua = Ug[fs + 1]; va = Ug[2 * fs + 1];
    ara = rm * Lg[1];
    ata = rm * Lg[4 * fs + 1];
  }
  __syncthreads();
  // ---------------- the interface above level l ----------------
  // F0 = w (rho + rho_a); contributions 0.5 fz (Fb0 - Ft0), fz (Fb1 - Ft1), fz = d33 / (2 m z)
  double br = 0.0, bw = 0.0, tm = 0.0, t0 = 0.0, t1 = 0.0, t2 = 0.0;   // to rho (l and l+1), w; theta of l-1 .. l+2
  if (top) {
    const double hz = 0.5 * hn[H_33 * DoF];
    const double aF0r = 0.5 * hz * (ara * P.zl[nz + l + 1] - ar * P.zl[nz + l]);
    const double aF = hz * (ata * P.zl[nz + l + 1] - at * P.zl[nz + l]);
    const double F0 = wh * (rho + ra);
    // a mass flux within rounding of its own terms has no direction: the
    // symmetric slope (see k_phase2_adj)
    const double mag = rho * (fabs(u) + fabs(v) + fabs(wh)) + ra * (fabs(ua) + fabs(va) + fabs(wh));
    const int sg = fabs(F0) <= 1e-13 * mag ? 0 : (F0 > 0.0 ? 1 : -1);
    const double *c = th + (lvl + 2) * RS + ID;
    double cf = 0.0;   // dF1 / dF0
#pragma unroll
    for (int side = 0; side < 2; ++side) {   // 0: from level l, 1: from level l + 1
      if (sg != 0 && (sg > 0) != (side == 0)) continue;
      const int far = side == 0 ? (l > 0 ? -1 : 0) : (l + 2 < nz ? 2 : 1);
      const double cu = c[side * RS], cd = c[(1 - side) * RS], dc = cd - cu, num = cu - c[far * RS];
      const double iden = 1.0 / (dc + 1.e-20), r = num * iden;
      const double *k = P.zl + (size_t)(side == 0 ? 2 : 4) * nz + l;
      double dphi;
      const double phi = upwind_limit_d(r, k[nz], k[0], dphi);
      const double cF = cu + phi * dc;
      cf += (sg == 0 ? 0.25 : 0.5) * cF;
      if (sg == 0) continue;
      const double ac = 0.5 * F0 * aF;
      const double an = dphi * dc * ac * iden, ad = -an * r;   // adjoints of num and of the denominator
      const double au = (1.0 - phi) * ac + an - ad, adn = phi * ac + ad;
      if (side == 0) {
        t0 += au; t1 += adn;
        if (far < 0) tm -= an; else t0 -= an;
      } else {
        t1 += au; t0 += adn;
        if (far == 2) t2 -= an; else t1 -= an;
      }
    }
    const double aF0 = aF0r + cf * aF;
    bw = (rho + ra) * aF0;
    br = wh * aF0;
  }
  // what level l gets from the interfaces of its neighbours
  const double br_b = __shfl_up_sync(lanes, br, 1, LT), t1_b = __shfl_up_sync(lanes, t1, 1, LT);
  const double t2_b = __shfl_up_sync(lanes, t2, 2, LT), tm_a = __shfl_down_sync(lanes, tm, 1, LT);
  double a_th = t0, a_r = br, a_u = 0.0, a_v = 0.0;
  if (lvl > 0) { a_th += t1_b; a_r += br_b; }
  if (lvl > 1) a_th += t2_b;
  if (lvl < LT - 1) a_th += tm_a;
  // and what goes to levels outside the tile
  auto out_theta = [&](int d, double x) {   // theta of level l + d
    const double r = x / Ug[d];
    atomicAdd(Og + 4 * fs + d, r);
    atomicAdd(Og + d, -r * th[(lvl + 2 + d) * RS + ID]);
  };
  if (act) {
    if (lvl == 0 && l > 0 && tm != 0.0) out_theta(-1, tm);
    if (top && lvl == LT - 1) {
      out_theta(1, t1);
      atomicAdd(Og + 1, br);
    }
    if (lvl >= LT - 2 && l + 2 < nz && t2 != 0.0) out_theta(2, t2);
  }
  // ---------------- transposed sums ----------------
  const double h11 = hn[H_11 * DoF], h12 = hn[H_12 * DoF], h21 = hn[H_21 * DoF], h22 = hn[H_22 * DoF];
  if (act) {
    double xr = 0, yr = 0, xt = 0, yt = 0, X = 0, Y = 0, Dx = 0, Dy = 0;
    const double *x0 = s + row + N * Jn, *y0 = s + row + I;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double dtI = P.D[k + N * I], dtJ = P.D[k + N * Jn];
      const double bx = x0[PL + k], by = y0[PL + N * k];
      xr += dtI * x0[k];
      yr += dtJ * y0[N * k];
      xt += dtI * bx;
      yt += dtJ * by;
      X += P.DW[k + N * I] * bx;
      Y += P.DW[k + N * Jn] * by;
      Dx += P.D[I + N * k] * x0[2 * PL + k];
      Dy += P.D[Jn + N * k] * y0[2 * PL + N * k];
    }
    // flux divergences
    const double cu = h11 * u + h12 * v, cv = h21 * u + h22 * v;
    const double auc = xr + thl * xt, avc = yr + thl * yt;
    a_th -= rho * (cu * xt + cv * yt);
    a_r -= cu * auc + cv * avc;
    a_u -= rho * (h11 * auc + h21 * avc);
    a_v -= rho * (h12 * auc + h22 * avc);
    // hyperviscosity of theta: X, Y the sums of the Laplacian's adjoint
    const double rJ = hn[H_RJ * DoF], nu = -P.nuDiv;
    const double aGx = nu * (h11 * X + h21 * Y), aGy = nu * (h12 * X + h22 * Y);
    a_r += rJ * ((h11 * Dx + h21 * Dy) * aGx + (h12 * Dx + h22 * Dy) * aGy);
    s[3 * PL + si] = rho * rJ * (h11 * aGx + h12 * aGy);
    s[4 * PL + si] = rho * rJ * (h21 * aGx + h22 * aGy);
    // the state adjoint of this level
    const double q = a_th / rho;
    atomicAdd(Og, a_r - q * thl);
    atomicAdd(Og + fs, a_u);
    atomicAdd(Og + 2 * fs, a_v);
    if (top) atomicAdd(Og + 3 * fs, bw);
    atomicAdd(Og + 4 * fs, q);
  }
  __syncthreads();
  if (!act) return;
  double c5 = 0;
  const double *x0 = s + row + N * Jn, *y0 = s + row + I;
#pragma unroll
  for (int k = 0; k < N; ++k)
    c5 += P.D[k + N * I] * x0[3 * PL + k] + P.D[k + N * Jn] * y0[4 * PL + N * k];
  atomicAdd(LT1 + (size_t)nz * g + l + 4 * fs, c5);
}

template <int N>
__device__ __forceinline__ void phase2_momentum_adj(const GP &P, const double *__restrict__ U,
                                                    const double *__restrict__ Pr, const double *__restrict__ LF,
                                                    double *__restrict__ LU, double *__restrict__ LT1, const int L0,
                                                    const int IF, double *sm)
{
  using CF = AdjFlat<N>;
  constexpr int DoF = CF::DoF, RS = CF::RS, PL = CF::PL, LT = CF::LT, TH = CF::THREADS, PW = PL + RS;
  const int nz = P.nz;
  const size_t fs = (size_t)nz * P.NumG;
  double *fw = sm;             // [4][LT+1][RS]: -h12 w, -h22 w, -h11 w, -h21 w; row 0 is level L0-1
  double *aw = fw + 4 * PW;    // [2][LT+1][RS]: adjoints of the w-curls U, V of the levels L0-1 .. L0+LT-1
  double *s = aw + 2 * PW;     // planes: 0-1 curl operands, 2 p, 3 W, 4-5 K, 6-7 pressure, 8-9 curl, 10-11 second round
  const int t = threadIdx.x;
  const int lvl = t % LT, ID = t / LT;
  const int l = L0 + lvl;
  const bool act = l < nz, top = l < nz - 1, bot = act && l > 0;
  const int I = ID % N, Jn = ID / N;
  const int row = lvl * RS, si = row + ID;
  const double *hn = P.hm + (size_t)IF * H_N * DoF + ID;
  const unsigned lanes = block_lanes<TH>();
  const int g = P.glob[IF * DoF + ID];
  const double *Ug = U + (size_t)nz * g + l, *Lg = LF + (size_t)nz * g + l, *pg = Pr + (size_t)nz * g + l;
  double *Og = LU + (size_t)nz * g + l;
  const double h11 = hn[H_11 * DoF], h12 = hn[H_12 * DoF], h21 = hn[H_21 * DoF], h22 = hn[H_22 * DoF];
  double rho = 1.0, u = 0.0, v = 0.0, wh = 0.0, pr = 0.0;
  if (act) {
    rho = Ug[0]; u = Ug[fs]; v = Ug[2 * fs]; wh = Ug[3 * fs]; pr = pg[0];
    fw[row + RS + ID] = -h12 * wh;
    fw[PW + row + RS + ID] = -h22 * wh;
    fw[2 * PW + row + RS + ID] = -h11 * wh;
    fw[3 * PW + row + RS + ID] = -h21 * wh;
    s[si] = h12 * u - h11 * v;
    s[PL + si] = h22 * u - h21 * v;
    s[2 * PL + si] = pr;
  }
  // neighbouring levels
  double wl = __shfl_up_sync(lanes, wh, 1, LT), ub = __shfl_up_sync(lanes, u, 1, LT);
  double vb = __shfl_up_sync(lanes, v, 1, LT), rb = __shfl_up_sync(lanes, rho, 1, LT);
  double ua = __shfl_down_sync(lanes, u, 1, LT), va = __shfl_down_sync(lanes, v, 1, LT);
  double ra = __shfl_down_sync(lanes, rho, 1, LT), pa = __shfl_down_sync(lanes, pr, 1, LT);
  if (lvl == 0) {
    wl = 0.0;
    if (bot) { wl = Ug[3 * fs - 1]; ub = Ug[fs - 1]; vb = Ug[2 * fs - 1]; rb = Ug[-1]; }
    fw[ID] = -h12 * wl;
    fw[PW + ID] = -h22 * wl;
    fw[2 * PW + ID] = -h11 * wl;
    fw[3 * PW + ID] = -h21 * wl;
  }
  if (act && top && lvl == LT - 1) { ra = Ug[1]; ua = Ug[fs + 1]; va = Ug[2 * fs + 1]; pa = pg[1]; }
  __syncthreads();

  // ---------------- forward sums ----------------
  const double rr = 1.0 / rho;
  double U2 = 0, V2 = 0, U1 = 0, V1 = 0, W = 0, PX = 0, PY = 0;
  if (act) {
    const double *x0 = s + row + N * Jn, *y0 = s + row + I;
    const double *fx = fw + row + RS + N * Jn, *fy = fw + row + RS + I;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double dI = P.D[I + N * k], dJ = P.D[Jn + N * k];
      U2 += dI * fx[k] + dJ * fy[PW + N * k];
      V2 += dI * fx[2 * PW + k] + dJ * fy[3 * PW + N * k];
      W += dI * x0[k] + dJ * y0[PL + N * k];
      PX += dI * x0[2 * PL + k];
      PY += dJ * y0[2 * PL + N * k];
    }
  }
  U1 = __shfl_up_sync(lanes, U2, 1, LT);
  V1 = __shfl_up_sync(lanes, V2, 1, LT);
  if (lvl == 0 && act) {   // the w-curls of the level below the tile
    U1 = V1 = 0.0;
    const double *fx = fw + N * Jn, *fy = fw + I;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double dI = P.D[I + N * k], dJ = P.D[Jn + N * k];
      U1 += dI * fx[k] + dJ * fy[PW + N * k];
      V1 += dI * fx[2 * PW + k] + dJ * fy[3 * PW + N * k];
    }
  }
  // ---------------- pointwise adjoints ----------------
  // of rho, u, v, w (upper interface), p of this level; _a, _b: what levels
  // l + 1 and l - 1 get; a_wl: of w at the lower interface
  double a_r = 0, a_u = 0, a_v = 0, a_w = 0, a_wl = 0, a_p = 0;
  double r_a = 0, u_a = 0, v_a = 0, p_a = 0, r_b = 0, u_b = 0, v_b = 0;
  double aU1 = 0, aV1 = 0, aU2 = 0, aV2 = 0;
  if (act) {
    const double rm = hn[H_RM * DoF], h33 = hn[H_33 * DoF], hJ = hn[H_J * DoF], z = P.zl[l];
    const double su = rm * Lg[fs], sv = rm * Lg[2 * fs];
    const double fc = hn[H_FC * DoF] * hJ, fz = 0.25 * h33 * P.zl[nz + l], zr = rho * z;
    s[3 * PL + si] = u * sv - v * su;   // W
    a_v += (fc - W) * su;
    a_u += (W - fc) * sv;
    aV1 = -0.5 * wl * su; aV2 = -0.5 * wh * su;
    aU1 = -0.5 * wl * sv; aU2 = -0.5 * wh * sv;
    a_wl -= 0.5 * (V1 * su + U1 * sv);
    a_w -= 0.5 * (V2 * su + U2 * sv);
    if (bot) {   // -fz wl (u - ub)
      const double x = fz * wl;
      a_u -= x * su; u_b += x * su;
      a_v -= x * sv; v_b += x * sv;
      a_wl -= fz * ((u - ub) * su + (v - vb) * sv);
    }
    if (top) {   // -fz wh (ua - u)
      const double x = fz * wh;
      u_a -= x * su; a_u += x * su;
      v_a -= x * sv; a_v += x * sv;
      a_w -= fz * ((ua - u) * su + (va - v) * sv);
    }
    const double kx = -0.5 * (h11 * su + h12 * sv), ky = -0.5 * (h21 * su + h22 * sv);
    s[4 * PL + si] = kx;
    s[5 * PL + si] = ky;
    s[6 * PL + si] = 2.0 * kx * rr;
    s[7 * PL + si] = 2.0 * ky * rr;
    a_r -= 2.0 * (kx * PX + ky * PY) * rr * rr;
    s[8 * PL + si] = P.nuCurl * (h12 * su - h11 * sv);
    s[9 * PL + si] = P.nuCurl * (h22 * su - h21 * sv);
    if (top) {   // w at interface l from its upper node
      const double za = P.zl[l + 1], sa = zr + ra * za, isa = 1.0 / sa, lw = Lg[3 * fs], a = lw * rm * isa;
      const double hh = 0.5 * h33;
      const double T = u * (ua - u) + v * (va - v) - 0.5 * (ua * ua + va * va) + 0.5 * (u * u + v * v) -
                       0.5 * (wh * wh - wl * wl);
      const double B = z * (u * V2 + v * U2) + hh * T;
      const double whi = (rho * B - (h33 * (pa - pr) + P.Grav * hJ * sa)) * (rm * isa);
      a_r += B * a;
      const double e = zr * a, f = hh * rho * a;
      aV2 += u * e; aU2 += v * e;
      a_u += V2 * e + f * (ua - u); u_a += f * (u - ua);
      a_v += U2 * e + f * (va - v); v_a += f * (v - va);
      a_w -= f * wh; a_wl += f * wl;
      p_a -= h33 * a; a_p += h33 * a;
      const double as = -lw * isa * (whi + P.Grav * hJ * rm);
      a_r += z * as; r_a += za * as;
    }
    if (bot) {   // w at interface l - 1 from its lower node
      const double zb = P.zl[l - 1], sb = rb * zb + zr, isb = 1.0 / sb, lw = Lg[3 * fs - 1], b = lw * rm * isb;
      const double hh = 0.5 * h33;
      const double T = u * (u - ub) + v * (v - vb) - 0.5 * (u * u + v * v) + 0.5 * (ub * ub + vb * vb) -
                       0.5 * (wh * wh - wl * wl);
      const double B = z * (u * V1 + v * U1) + hh * T;
      a_r += B * b;
      const double e = zr * b, f = hh * rho * b;
      aV1 += u * e; aU1 += v * e;
      a_u += V1 * e + f * (u - ub); u_b += f * (ub - u);
      a_v += U1 * e + f * (v - vb); v_b += f * (vb - v);
      a_w -= f * wh; a_wl += f * wl;
      const double as = -b * rho * B * isb;
      a_r += z * as; r_b += zb * as;
    }
  }
  {   // the w-curl of a level serves its upper node and the lower node above
    const double U1a = __shfl_down_sync(lanes, aU1, 1, LT), V1a = __shfl_down_sync(lanes, aV1, 1, LT);
    if (act) {
      const bool in = top && lvl < LT - 1;
      aw[row + RS + ID] = aU2 + (in ? U1a : 0.0);
      aw[PW + row + RS + ID] = aV2 + (in ? V1a : 0.0);
      if (lvl == 0) {
        aw[ID] = aU1;
        aw[PW + ID] = aV1;
      }
    }
  }
  __syncthreads();
  // ---------------- transposed sums ----------------
  if (act) {
    double xU = 0, yU = 0, xV = 0, yV = 0, xW = 0, yW = 0, K = 0, p = 0, dv = 0, cu = 0;
    const double *x0 = s + row + N * Jn, *y0 = s + row + I;
    const double *ax = aw + row + RS + N * Jn, *ay = aw + row + RS + I;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double dI = P.D[k + N * I], dJ = P.D[k + N * Jn], wI = P.DW[k + N * I], wJ = P.DW[k + N * Jn];
      xU += dI * ax[k];
      yU += dJ * ay[N * k];
      xV += dI * ax[PW + k];
      yV += dJ * ay[PW + N * k];
      xW += dI * x0[3 * PL + k];
      yW += dJ * y0[3 * PL + N * k];
      const double kx = x0[4 * PL + k], ky = y0[5 * PL + N * k];
      K += dI * kx + dJ * ky;
      dv += wI * kx + wJ * ky;
      p += dI * x0[6 * PL + k] + dJ * y0[7 * PL + N * k];
      cu += wI * x0[8 * PL + k] + wJ * y0[9 * PL + N * k];
    }
    a_w -= h12 * xU + h22 * yU + h11 * xV + h21 * yV;
    a_u += h12 * xW + h22 * yW + 2.0 * u * K;
    a_v += 2.0 * v * K - h11 * xW - h21 * yW;
    a_wl += wl * K;
    a_w += wh * K;
    a_p += p;
    const double rJ = hn[H_RJ * DoF];
    s[10 * PL + si] = cu * rJ;
    s[11 * PL + si] = 2.0 * P.nuGrad * dv * rJ;
    if (lvl == 0 && bot) {   // the w-curl of the level below the tile, from this level's lower node
      double x = 0, y = 0, x2 = 0, y2 = 0;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const double dI = P.D[k + N * I], dJ = P.D[k + N * Jn];
        x += dI * aw[k + N * Jn];
        y += dJ * aw[I + N * k];
        x2 += dI * aw[PW + k + N * Jn];
        y2 += dJ * aw[PW + I + N * k];
      }
      a_wl -= h12 * x + h22 * y + h11 * x2 + h21 * y2;
    }
  }
  // ---------------- to the neighbouring levels, and the state adjoint ----------------
  {
    const double r0 = __shfl_up_sync(lanes, r_a, 1, LT), u0 = __shfl_up_sync(lanes, u_a, 1, LT);
    const double v0 = __shfl_up_sync(lanes, v_a, 1, LT), p0 = __shfl_up_sync(lanes, p_a, 1, LT);
    const double r1 = __shfl_down_sync(lanes, r_b, 1, LT), u1 = __shfl_down_sync(lanes, u_b, 1, LT);
    const double v1 = __shfl_down_sync(lanes, v_b, 1, LT), w1 = __shfl_down_sync(lanes, a_wl, 1, LT);
    if (act) {
      const double dpd = 1.0 / (1.0 - P.kappa);   // p / (rho*theta) times this: dp/d(rho*theta)
      if (lvl > 0) { a_r += r0; a_u += u0; a_v += v0; a_p += p0; }
      if (lvl < LT - 1 && top) { a_r += r1; a_u += u1; a_v += v1; a_w += w1; }
      atomicAdd(Og, a_r);
      atomicAdd(Og + fs, a_u);
      atomicAdd(Og + 2 * fs, a_v);
      atomicAdd(Og + 3 * fs, a_w);
      atomicAdd(Og + 4 * fs, a_p * dpd * pr / Ug[4 * fs]);
      if (lvl == 0 && bot) {
        atomicAdd(Og - 1, r_b);
        atomicAdd(Og + fs - 1, u_b);
        atomicAdd(Og + 2 * fs - 1, v_b);
        atomicAdd(Og + 3 * fs - 1, a_wl);
      }
      if (lvl == LT - 1 && top) {
        atomicAdd(Og + 1, r_a);
        atomicAdd(Og + fs + 1, u_a);
        atomicAdd(Og + 2 * fs + 1, v_a);
        atomicAdd(Og + 4 * fs + 1, p_a * dpd * pa / Ug[4 * fs + 1]);
      }
    }
  }
  __syncthreads();
  if (!act) return;
  // ---------------- the cache ----------------
  double a1 = 0, a2 = 0, a3 = 0, a4 = 0;
  const double *x0 = s + row + N * Jn, *y0 = s + row + I;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double dI = P.D[k + N * I], dJ = P.D[k + N * Jn];
    a1 += dI * x0[10 * PL + k];
    a2 += dJ * y0[10 * PL + N * k];
    a3 += dI * x0[11 * PL + k];
    a4 += dJ * y0[11 * PL + N * k];
  }
  double *T = LT1 + (size_t)nz * g + l;
  atomicAdd(T, -h12 * a1 - h22 * a2);
  atomicAdd(T + fs, h11 * a1 + h21 * a2);
  atomicAdd(T + 2 * fs, h11 * a3 + h21 * a4);
  atomicAdd(T + 3 * fs, h12 * a3 + h22 * a4);
}

// blockIdx.x: 2 * tile + role (even: momentum, odd: scalars)
template <int N>
__global__ void __launch_bounds__(AdjFlat<N>::THREADS, AdjFlat<N>::MINB)
    k_phase2_adj_flat(const GP P, const double *__restrict__ U, const double *__restrict__ Pr,
                      const double *__restrict__ T1, const double *__restrict__ LF, double *__restrict__ LU,
                      double *__restrict__ LT1)
{
  extern __shared__ double sm[];
  const int L0 = (blockIdx.x >> 1) * AdjFlat<N>::LT;
  if (blockIdx.x & 1) phase2_scalars_adj<N>(P, U, T1, LF, LU, LT1, L0, blockIdx.y, sm);
  else phase2_momentum_adj<N>(P, U, Pr, LF, LU, LT1, L0, blockIdx.y, sm);
}

}  // namespace cgd
