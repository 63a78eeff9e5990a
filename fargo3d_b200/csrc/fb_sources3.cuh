// fb_sources3.cuh -- the source stage of 3D spherical disks (algogas.c:30-120:
// pressure, potential, CorrectVtheta, SubStep1_x/y/z, visctensor_sph.c:141-213,
// addviscosity_sph.c:74-126, SubStep2_a/b) in FP64 arithmetic.
//
// A CTA owns a TX x TY tile of columns (azimuth x radius) and marches over
// layers (colatitude): the inputs of layers k-1, k, k+1 stay in shared memory,
// each layer is loaded once, its potential formed once and each stress once
// per cell and halo.  (One tile per layer loads three layers and forms the
// potential of two and every stress of two for each layer it writes.)  The
// next layer's inputs are loaded (cp.async) while this one is computed.
// Divisors that depend on the row, the row and layer, or the column and layer
// only (radii, zone sizes, r sin(theta)) are inverted once into a table and
// the quotients taken with divk, which rounds as '/' does.  FP32 storage is
// not bound to the reference's rounding: its quotients are products with the
// tabulated reciprocals, and three sums of densities are its only per-cell
// divisors besides the SubStep1 weights (5 divisions a cell instead of 17).
#pragma once
#include <atomic>

#include "fb_kernels.cuh"

namespace fb {

// Rows of a tile: FP64 8 (256 threads, 128 registers at 2 CTAs: 737 us at
// 512x256x48, 6 rows 780); FP32 storage 6 (192 threads, 168 registers: 535 us, 8
// rows spill: 578).
constexpr int S3_TX = 32, S3_W = S3_TX + 2;
template <typename S>
struct S3 {
  static constexpr int TY = sizeof(S) == 8 ? 8 : 6, T = S3_TX * TY;
  static constexpr int H = TY + 2, P = S3_W * H;   // a plane with its halo
};
// row-and-layer divisors and their reciprocals
enum { S3_RS, S3_RDZ, S3_RDM, S3_RSI, S3_YDM, S3_YS, S3_NT };
// layer scalars: sin / cos of Zmed and Zmin, face factors, faces and centres
// with their neighbours', reciprocals
enum { L3_SZM, L3_SZMM, L3_CZM, L3_SZI, L3_SZIP, L3_CZI, L3_SYK, L3_SXK, L3_SZK, L3_SZKP, L3_ZI, L3_ZIP, L3_ZIM, L3_ZM,
       L3_ZMM, L3_ISZM, L3_ISYK, L3_N };
template <typename S>
struct S3Shared {
  static constexpr int S3_H = S3<S>::H, S3_P = S3<S>::P;
  static_assert(S3_NT * S3_H <= 64 && S3_W <= 40, "the threads that fill the tables");
  double rho[4][S3_P], cs[4][S3_P], u[4][S3_P], vy[4][S3_P], vz[4][S3_P], pot[2][S3_P];   // layer k in k & 3
  double xx[2][S3_P], zz[2][S3_P], xz[2][S3_P], zy[2][S3_P], yy[S3_P], yx[S3_P];
  double t[3][S3_NT][S3_H], it[3][S3_NT][S3_H];   // layer k in k % 3
  double lay[3][L3_N], bg[3][S3_H];
  double vd[3][S3_W], ivd[3][S3_W];               // Syk Sxi and its reciprocal
  float raw[sizeof(S) == 4 ? 5 : 1][sizeof(S) == 4 ? S3_P : 1];   // FP32 storage: the next layer as stored
  double sxi[S3_W], idx[S3_W], dxm[S3_W], cx[S3_W], sx[S3_W];   // columns: Sxi, 1 / Sxi, cos and sin of Xmed
  // rows: Ymin(j+1) - Ymin(j) and Ymed(j) - Ymed(j-1) with their reciprocals,
  // radii, face areas, 1 / Vol, viscosity factors
  double dyi[S3_H], idyi[S3_H], dym[S3_H], idym[S3_H], ym[S3_H], iym[S3_H], yi[S3_H], iyi[S3_H];
  double sxj[S3_H], syj[S3_H + 1], szj[S3_H], ivj[S3_H], visc[S3_H], viscm[S3_H], pst[S3_H];
  double ind[FB_MAXPLANETS];
  fb_scalars sc;
};

// one element from global to shared memory, asynchronously
template <typename S>
__device__ __forceinline__ void cp_el(S *dst, const S *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "n"(sizeof(S))
               : "memory");
}
template <typename S>
__device__ __forceinline__ void b_sources_sph(const Dims &m, const Geo<double> &g, const S *__restrict__ rho,
    const S *__restrict__ cs, const S *__restrict__ vx, const S *__restrict__ vy, const S *__restrict__ vz,
    S *__restrict__ vxt, S *__restrict__ vyt, S *__restrict__ vzt, const fb_scalars *__restrict__ scp, int dust,
    int viscous, const double *__restrict__ vbg, int bx, int by, int k0, int k1) {
  extern __shared__ __align__(16) unsigned char s3_raw[];
  S3Shared<S> &s = *reinterpret_cast<S3Shared<S> *>(s3_raw);
  constexpr int S3_TY = S3<S>::TY, S3_T = S3<S>::T, S3_H = S3<S>::H, S3_P = S3<S>::P;
  static_assert((S3_T == 192 || S3_T == 256) && S3_TX + 1 + S3_TY <= 64, "warps in pairs for the halo's work");
  constexpr bool FAST = sizeof(S) == 4;   // FP32 storage: the fast potential
  const int i0 = bx * S3_TX, j0 = FB_NGH + by * S3_TY, tid = threadIdx.x;
  for (int w = tid; w < (int)(sizeof(fb_scalars) / 8); w += S3_T)
    reinterpret_cast<double *>(&s.sc)[w] = reinterpret_cast<const double *>(scp)[w];
  if (tid < S3_H) {
    const int j = min(j0 - 1 + tid, m.sy - 1);
    s.dyi[tid] = ld(g.ymin + j + 1) - ld(g.ymin + j);
    s.idyi[tid] = 1.0 / s.dyi[tid];
    s.ym[tid] = ld(g.ymed + j); s.iym[tid] = ld(g.inv_ymed + j);
    s.yi[tid] = ld(g.ymin + j); s.iyi[tid] = ld(g.inv_ymin + j);
    s.dym[tid] = j > 0 ? ld(g.ymed + j) - ld(g.ymed + j - 1) : 0.0; s.idym[tid] = ld(g.inv_dymed + j);
    s.sxj[tid] = ld(g.sxj + j); s.szj[tid] = ld(g.szj + j); s.ivj[tid] = ld(g.invvj + j);
    s.syj[tid] = ld(g.syj + j);
    if (tid == S3_H - 1) s.syj[S3_H] = ld(g.syj + min(j + 1, m.sy - 1));
    s.visc[tid] = ld(g.visc_j + j); s.viscm[tid] = ld(g.viscm_j + j); s.pst[tid] = ld(g.pot_star + j);
  } else if (tid >= 64 && tid < 64 + S3_W) {
    const int c = tid - 64, i = wrapx(min(i0 - 1 + c, m.nx), m.nx);
    s.sxi[c] = ld(g.sxi + i); s.idx[c] = ld(g.invdiffxmed + i);
    s.dxm[c] = ld(g.xmin + min(i + 1, m.nx)) - ld(g.xmin + i);
    s.cx[c] = ld(g.cos_xmed + i); s.sx[c] = ld(g.sin_xmed + i);
  }
  __syncthreads();
  // FP64: 1 / d^3 of each planet
  if (tid < s.sc.nplanets) s.ind[tid] = (FAST ? s.sc.pmass[tid] : 1.0) / s.sc.pdist3[tid];
  const double dt = s.sc.dt, domega = s.sc.domega, of = s.sc.omegaframe, nu = s.sc.nu, alpha = s.sc.alpha;
  // the one or two plane elements this thread loads
  constexpr int NE = (S3_P + S3_T - 1) / S3_T;
  bool ein[NE];
  long long eo[NE];
#pragma unroll
  for (int n = 0; n < NE; n++) {
    const int e = tid + n * S3_T, lj = e / S3_W, li = e - lj * S3_W, j = j0 - 1 + lj;
    ein[n] = e < S3_P && j < m.sy && i0 - 1 + li <= m.nx;
    eo[n] = m.l(wrapx(min(i0 - 1 + li, m.nx), m.nx), min(j, m.sy - 1), 0);
  }
  double szn;
  // layer k's inputs: FP64 straight into plane k & 3 (which no layer still in
  // work reads), FP32 into a buffer of their own
  auto fetch = [&](int k) {
    const long long o = (long long)k * m.stride;
    szn = ld(g.sin_zmed + k);
#pragma unroll
    for (int n = 0; n < NE; n++)
      if (ein[n]) {
        const long long l = eo[n] + o;
        const int e = tid + n * S3_T;
        if constexpr (FAST) {
          cp_el(&s.raw[0][e], rho + l); cp_el(&s.raw[1][e], cs + l); cp_el(&s.raw[2][e], vx + l);
          cp_el(&s.raw[3][e], vy + l); cp_el(&s.raw[4][e], vz + l);
        } else {
          const int p = k & 3;
          cp_el(&s.rho[p][e], rho + l); cp_el(&s.cs[p][e], cs + l); cp_el(&s.u[p][e], vx + l);
          cp_el(&s.vy[p][e], vy + l); cp_el(&s.vz[p][e], vz + l);
        }
      }
  };
  auto put = [&](int k) {     // plane k & 3 completed; CorrectVtheta (correct_vtheta.c:55-60)
    const int p = k & 3;
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int n = 0; n < NE; n++)
      if (ein[n]) {
        const int e = tid + n * S3_T;
        if constexpr (FAST) {
          s.rho[p][e] = s.raw[0][e];
          s.cs[p][e] = s.raw[1][e];
          const double u = s.raw[2][e] + s.bg[k % 3][e / S3_W];   // stored less the ring's background
          s.u[p][e] = u - domega * s.ym[e / S3_W] * szn;
          s.vy[p][e] = s.raw[3][e];
          s.vz[p][e] = s.raw[4][e];
        } else {
          s.u[p][e] -= domega * s.ym[e / S3_W] * szn;
        }
      }
  };
  auto tables = [&](int k) {  // layer k's divisors and scalars
    const int w = tid - (S3_T - 64), c = tid - 64;
    if (w >= 0 && w < S3_NT * S3_H) {
      const int r = w / S3_H, lj = w - r * S3_H;
      const double ym = s.ym[lj], yi = s.yi[lj];
      const double dzm = ld(g.zmed + k) - ld(g.zmed + k - 1);
      double d;
      switch (r) {
        case S3_RS: d = ld(g.sin_zmed + k) * ym; break;
        case S3_RDZ: d = ym * (ld(g.zmin + k + 1) - ld(g.zmin + k)); break;
        case S3_RDM: d = ym * dzm; break;
        case S3_RSI: d = ld(g.sin_zmin + k) * ym; break;
        case S3_YDM: d = yi * dzm; break;
        default: d = yi * ld(g.sin_zmed + k); break;
      }
      s.t[k % 3][r][lj] = d;
      s.it[k % 3][r][lj] = 1.0 / d;
    } else if (c >= 0 && c < S3_W) {
      const double d = ld(g.syk + k) * s.sxi[c];
      s.vd[k % 3][c] = d;
      s.ivd[k % 3][c] = 1.0 / d;
    } else if (tid >= 104 && tid < 104 + L3_N) {
      const int r = tid - 104;
      const double *a;
      switch (r) {
        case L3_SZMM: a = g.sin_zmed + k - 1; break;
        case L3_CZM: a = g.cos_zmed + k; break;
        case L3_SZI: a = g.sin_zmin + k; break;
        case L3_SZIP: a = g.sin_zmin + k + 1; break;
        case L3_CZI: a = g.cos_zmin + k; break;
        case L3_SXK: a = g.sxk + k; break;
        case L3_SZK: a = g.szk + k; break;
        case L3_SZKP: a = g.szk + k + 1; break;
        case L3_ZI: a = g.zmin + k; break;
        case L3_ZIP: a = g.zmin + k + 1; break;
        case L3_ZIM: a = g.zmin + k - 1; break;
        case L3_ZM: a = g.zmed + k; break;
        case L3_ZMM: a = g.zmed + k - 1; break;
        case L3_SYK: case L3_ISYK: a = g.syk + k; break;
        default: a = g.sin_zmed + k; break;
      }
      const double d = ld(a);
      s.lay[k % 3][r] = r >= L3_ISZM ? 1.0 / d : d;
    } else if (FAST && tid < S3_H) {   // the rings' backgrounds
      s.bg[k % 3][tid] = bg_at(vbg, min(j0 - 1 + tid, m.sy - 1) + k * m.sy);
    }
  };
  // potential.c:51-208; FP32 storage: the indirect term with m / d^3 (ind), the
  // planets' terms with an FP64 reciprocal root
  auto potential = [&](int k, int e, int li, int lj) {
    const double *L = s.lay[k % 3];
    const double ym = s.ym[lj], XC = ym * s.cx[li] * L[L3_SZM], YC = ym * s.sx[li] * L[L3_SZM], ZC = ym * L[L3_CZM];
    double pot = s.pst[lj];
    for (int n = 0; n < s.sc.nplanets; n++) {
      const double mp = s.sc.pmass[n], xp = s.sc.px[n], yp = s.sc.py[n], zp = s.sc.pz[n];
      const double dist = (XC - xp) * (XC - xp) + (YC - yp) * (YC - yp) + (ZC - zp) * (ZC - zp);
      if (FAST) {
        if (s.sc.indirect_term) pot += s.ind[n] * (XC * xp + YC * yp + ZC * zp);
        pot -= mp * rsqrt(dist + s.sc.psmooth2[n]);
      } else {
        if (s.sc.indirect_term) pot += divk(mp * (XC * xp + YC * yp + ZC * zp), s.sc.pdist3[n], s.ind[n]);
        pot += -mp / sqrt(dist + s.sc.psmooth2[n]);
      }
    }
    s.pot[k & 1][e] = pot;
  };
  // x / d with id = 1 / d
  auto quo = [](double x, double d, double id) -> double { return FAST ? x * id : divk(x, d, id); };
  // tau_phiphi, tau_thth (and tau_rr) of layer k, from planes k and k + 1
  auto diag = [&](int k, bool yy, int e, int li, int lj) {
    const int p = k & 3, pp = (k + 1) & 3, q = k & 1, tq = k % 3;
    const double *L = s.lay[tq];
    const double szm = L[L3_SZM], czm = L[L3_CZM], syk = L[L3_SYK], sxk = L[L3_SXK], szk = L[L3_SZK], szkp = L[L3_SZKP];
    const double c = s.cs[p][e], r = s.rho[p][e];
    const double visc = m.alpha ? alpha * c * c * s.visc[lj] : nu;
    const double sxi = s.sxi[li], ym = s.ym[lj];
    const double u0 = s.u[p][e], dvx = s.u[p][e + 1] - u0;
    const double vy0 = s.vy[p][e], vyp = s.vy[p][e + S3_W], vz0 = s.vz[p][e], vzp = s.vz[pp][e];
    const double szj = s.szj[lj];
    double div_v = 0.0;
    div_v += dvx * s.sxj[lj] * sxk;
    div_v += (vyp * s.syj[lj + 1] * syk * sxi - vy0 * s.syj[lj] * syk * sxi);
    div_v += (vzp * szj * szkp * sxi - vz0 * szj * szk * sxi);
    const double ix = s.idx[li];   // uniform spacing: 1 / Sxi
    if (FAST) div_v *= (2.0 / 3.0) * s.ivj[lj] * L[L3_ISYK] * ix;
    else div_v *= divk((2.0 / 3.0) * s.ivj[lj], s.vd[tq][li], s.ivd[tq][li]);
    double txx = visc * r * ((FAST ? 2.0 * dvx * ix * s.iym[lj] * L[L3_ISZM] : 2.0 * dvx / (sxi * ym * szm)) - div_v);
    txx += quo(visc * r * (vyp + vy0), ym, s.iym[lj]);
    txx += quo(visc * r * (vzp + vz0) * czm, s.t[tq][S3_RS][lj], s.it[tq][S3_RS][lj]);
    double tzz = visc * r * (quo(2.0 * (vzp - vz0), s.t[tq][S3_RDZ][lj], s.it[tq][S3_RDZ][lj]) - div_v);
    tzz += quo(visc * r * (vy0 + vyp), ym, s.iym[lj]);
    s.xx[q][e] = txx;
    s.zz[q][e] = tzz;
    if (yy) s.yy[e] = visc * r * (quo(2.0 * (vyp - vy0), s.dyi[lj], s.idyi[lj]) - div_v);
  };
  // tau_phith and tau_rth of the lower faces of layer k, from planes k - 1 and k
  auto offd = [&](int k, int e, int li, int lj) {
    const int p = k & 3, pm = (k + 3) & 3, q = k & 1, tq = k % 3;
    const double *L = s.lay[tq], *Lm = s.lay[(k + 2) % 3];
    const double c0 = s.cs[p][e], cz = s.cs[pm][e];
    double visczm = nu, visczmym = nu;
    if (m.alpha) {
      const double s2 = c0 + cz + s.cs[p][e - 1] + s.cs[pm][e - 1];
      visczm = alpha * 0.0625 * s2 * s2 * s.visc[lj];
      const double s3 = c0 + cz + s.cs[p][e - S3_W] + s.cs[pm][e - S3_W];
      visczmym = alpha * 0.0625 * s3 * s3 * s.viscm[lj];
    }
    const double r = s.rho[p][e], rz = s.rho[pm][e], vz0 = s.vz[p][e];
    s.xz[q][e] = visczm * 0.25 * (r + rz + s.rho[p][e - 1] + s.rho[pm][e - 1]) *
                 (quo((quo(s.u[p][e], L[L3_SZM], L[L3_ISZM]) - quo(s.u[pm][e], Lm[L3_SZM], Lm[L3_ISZM])) * L[L3_SZI],
                       s.t[tq][S3_RDM][lj], s.it[tq][S3_RDM][lj]) +
                  (quo((vz0 - s.vz[p][e - 1]) * s.idx[li], s.t[tq][S3_RSI][lj], s.it[tq][S3_RSI][lj])));
    const double vzm = s.vz[p][e - S3_W];
    s.zy[q][e] = visczmym * 0.25 * (r + s.rho[p][e - S3_W] + rz + s.rho[pm][e - S3_W]) *
                 (quo(vz0 - vzm, s.dym[lj], s.idym[lj]) -
                  quo(0.5 * (vz0 + vzm), s.yi[lj], s.iyi[lj]) +
                  quo(s.vy[p][e] - s.vy[pm][e], s.t[tq][S3_YDM][lj], s.it[tq][S3_YDM][lj]));
  };
  // tau_rphi of layer k
  auto offd_yx = [&](int k, int e, int li, int lj) {
    const int p = k & 3, tq = k % 3;
    double viscm = nu;
    if (m.alpha) {
      const double s1 = s.cs[p][e] + s.cs[p][e - 1] + s.cs[p][e - S3_W] + s.cs[p][e - S3_W - 1];
      viscm = alpha * 0.0625 * s1 * s1 * s.viscm[lj];
    }
    const double u0 = s.u[p][e], um = s.u[p][e - S3_W];
    s.yx[e] = viscm * 0.25 * (s.rho[p][e] + s.rho[p][e - 1] + s.rho[p][e - S3_W] + s.rho[p][e - S3_W - 1]) *
              (quo((s.vy[p][e] - s.vy[p][e - 1]) * s.idx[li], s.t[tq][S3_YS][lj], s.it[tq][S3_YS][lj]) +
               quo(u0 - um, s.dym[lj], s.idym[lj]) -
               quo(0.5 * (u0 + um), s.yi[lj], s.iyi[lj]));
  };
  // This thread's own cell and, for the halo's 33 + TY elements of each
  // quantity (the lower row and column for the potential and the diagonal
  // stresses, the upper ones for the others), one element that belongs to a
  // pair of warps each, so that no warp has all of them to do.  (With the
  // plane's elements dealt to the threads in turn, three warps of six did all
  // of them, the rest waited; with the layer's scalars, whose loads and
  // divisions each warp had repeated, in tables, and the inputs by cp.async:
  // 512x256x48 FP64 844 -> 780 us, FP32 storage 612 -> 535.)
  const int li = (tid & (S3_TX - 1)) + 1, lj = tid / S3_TX + 1, e = lj * S3_W + li;
  const bool own = i0 + li - 1 <= m.nx && j0 + lj - 1 < m.sy;
  const int pair = tid >> 6, x = tid & 63, hi = pair >= 2;
  const int xj = x <= S3_TX ? (hi ? S3_TY + 1 : 0) : x - S3_TX, xi = x <= S3_TX ? x + hi : (hi ? S3_TX + 1 : 0);
  const int xe = xj * S3_W + xi;
  const bool extra = x <= S3_TX + S3_TY && i0 - 1 + xi <= m.nx && j0 - 1 + xj < m.sy;
  // layers k0 - 1 and k0, the stresses of the one below the first
  fetch(k0 - 1);
  tables(k0 - 1);
  tables(k0);
  __syncthreads();   // sc.ind, tables
  put(k0 - 1);
  fetch(k0);
  put(k0);
  __syncthreads();
  if (own) potential(k0 - 1, e, li, lj);
  if (extra && pair == 0) potential(k0 - 1, xe, xi, xj);
  if (viscous) {
    if (own) diag(k0 - 1, false, e, li, lj);
    if (extra && pair == 1) diag(k0 - 1, false, xe, xi, xj);
  }
  tables(k0 + 1);
  fetch(k0 + 1);
  __syncthreads();
  if (viscous) {
    if (own) offd(k0, e, li, lj);
    if (extra && pair == S3_T / 64 - 1) offd(k0, xe, xi, xj);
  }
  const int i = i0 + li - 1, j = j0 + lj - 1;
  const bool mine = i < m.nx && j <= m.ny + FB_NGH - 1;
  const double ym = s.ym[lj], ymm = s.ym[lj - 1], yi = s.yi[lj], yip = s.yi[lj + 1], yim = s.yi[lj - 1];
  const double iym = s.iym[lj], iyi = s.iyi[lj], idym = s.idym[lj], dym = ym - ymm;
  const double sxi = s.sxi[li], sxim = s.sxi[li - 1], idx = s.idx[li];
  const double dxmed = 0.5 * (sxi + sxim);
  for (int k = k0; k < k1; k++) {
    const int p = k & 3, pp = (k + 1) & 3, pm = (k + 3) & 3, q = k & 1, qn = q ^ 1, tq = k % 3;
    put(k + 1);
    __syncthreads();
    if (k + 1 < k1) {
      fetch(k + 2);
      tables(k + 2);   // slot (k - 1) % 3, which nothing reads any more
    }
    if (own) {
      potential(k, e, li, lj);
      if (viscous) {
        diag(k, true, e, li, lj);
        offd_yx(k, e, li, lj);
        offd(k + 1, e, li, lj);
      }
    }
    if (extra) {
      if (pair == 0) {
        potential(k, xe, xi, xj);
      } else if (viscous) {
        if (pair == 1) {
          diag(k, true, xe, xi, xj);
        } else {
          if (pair == 2) offd_yx(k, xe, xi, xj);
          if (pair == S3_T / 64 - 1) offd(k + 1, xe, xi, xj);
        }
      }
    }
    __syncthreads();
    if (mine) {
      const long long l = m.l(i, j, k);
      const double r = s.rho[p][e], rxm = s.rho[p][e - 1], rym = s.rho[p][e - S3_W], rzm = s.rho[pm][e];
      auto P = [&](int a, int x) -> double { const double c = s.cs[a][x]; return s.rho[a][x] * c * c; };
      const double *L = s.lay[tq];   // layer k's slot only: k - 1's may be layer k + 2's by now
      const double zi = L[L3_ZI], zip = L[L3_ZIP], zim = L[L3_ZIM], zm = L[L3_ZM], zmm = L[L3_ZMM];
      const double szm = L[L3_SZM], czm = L[L3_CZM], szi = L[L3_SZI], czi = L[L3_CZI];
      const double izx = FAST ? idx * s.it[tq][S3_RS][lj] : divk(divk(idx, ym, iym), szm, L[L3_ISZM]);
      const double rdm = s.t[tq][S3_RDM][lj], irdm = s.it[tq][S3_RDM][lj], rsi = s.t[tq][S3_RSI][lj], irsi = s.it[tq][S3_RSI][lj];
      const double u0 = s.u[p][e], v0 = s.vy[p][e], w0 = s.vz[p][e];
      const double p0 = P(p, e), pot0 = s.pot[q][e];
      // SubStep1_x
      const double sx = rxm + r, isx = FAST ? 1.0 / sx : 0.0;
      const double dx_ = r * sxi + rxm * sxim, idx_ = FAST ? isx * idx : 1.0 / dx_;
      const double dtorx = quo(2. * dt, dx_, idx_) * dxmed;
      double ax = u0;
      if (!dust) ax -= dtorx * (p0 - P(p, e - 1)) * izx;
      ax -= ((pot0 - s.pot[q][e - 1]) * dt) * izx;
      // SubStep1_y (spherical branch, substep1_y.c:212-217)
      const double dy_ = r * (yip - yi) + rym * (yi - yim), idy_ = 1.0 / dy_;
      const double dtory = quo(2.0 * dt, dy_, idy_) * dym;
      double ay = v0;
      if (!dust) ay -= quo(dtory * (p0 - P(p, e - S3_W)), dym, idym);
      {
        double vphi = 0.25 * (u0 + s.u[p][e + 1] + s.u[p][e - S3_W] + s.u[p][e - S3_W + 1]);
        vphi += yi * szm * of;
        const double vzz = 0.25 * (w0 + s.vz[pp][e] + s.vz[p][e - S3_W] + s.vz[pp][e - S3_W]);
        ay += quo(vphi * vphi + vzz * vzz, yi, iyi) * dt;
      }
      ay -= quo((pot0 - s.pot[q][e - S3_W]) * dt, dym, idym);
      // SubStep1_z (spherical branch, substep1_z.c:172-180)
      const double dz_ = r * (zip - zi) + rzm * (zi - zim), idz_ = 1.0 / dz_;
      const double dtorz = quo(2.0 * dt, dz_, idz_) * (zm - zmm);
      double vphz = 0.25 * (u0 + s.u[p][e + 1] + s.u[pm][e] + s.u[pm][e + 1]);
      vphz += ym * szi * of;
      double az = w0;
      if (!dust) az -= quo(dtorz * (p0 - P(pm, e)), rdm, irdm);
      az += quo(vphz * vphz * czi, rsi, irsi) * dt;
      az -= quo((pot0 - s.pot[qn][e]) * dt, rdm, irdm);
      if (viscous) {
        // addviscosity_sph
        const double txx = s.xx[q][e], sy = r + rym, sz = r + rzm, t2 = 2.0;
        const double yx0 = s.yx[e], yxp = s.yx[e + S3_W], xz0 = s.xz[q][e], xzp = s.xz[qn][e];
        const double zy0 = s.zy[q][e], zyp = s.zy[qn][e], zz0 = s.zz[q][e];
        const double dyi = yip - yi, dzi = zip - zi;
        if constexpr (!FAST) {
          ax += t2 * (txx - s.xx[q][e - 1]) * izx / sx * dt;
          ax += t2 * (yip * yip * yxp - yi * yi * yx0) / (dyi * ym * ym * sx) * dt;
          ax += (yxp + yx0) / (sx * ym) * dt;
          ax += t2 * (xzp - xz0) / (dzi * ym * sx) * dt;
          ax += t2 * (xzp + xz0) * czm / (szm * ym * sx) * dt;

          ay += t2 * (ym * ym * s.yy[e] - ymm * ymm * s.yy[e - S3_W]) / (dym * sy * yi * yi) * dt;
          ay += t2 * (s.yx[e + 1] - yx0) / (s.dxm[li] * yi * szm * sy) * dt;
          const double ys = yi * sy, iys = 1.0 / ys;
          ay -= quo(txx + s.xx[q][e - S3_W], ys, iys) * dt;
          ay -= quo(zz0 + s.zz[q][e - S3_W], ys, iys) * dt;
          ay += t2 * (zyp * L[L3_SZIP] - zy0 * szi) / (dzi * yi * szm * sy) * dt;

          az += t2 * (zz0 * szm - s.zz[qn][e] * L[L3_SZMM]) / ((zm - zmm) * ym * szi * sz) * dt;
          az += t2 * (s.xz[q][e + 1] - xz0) / ((sxi * ym * szi) * sz) * dt;
          az += t2 * (yip * yip * yip * s.zy[q][e + S3_W] - yi * yi * yi * zy0) / (dyi * ym * ym * ym * sz) * dt;
          az -= (txx + s.xx[qn][e]) * czi / (ym * szi * sz) * dt;
        } else {
          const double isy = 1.0 / sy, isz = 1.0 / sz, idyi = s.idyi[lj], iym2 = iym * iym;
          const double irs = s.it[tq][S3_RS][lj], irdz = s.it[tq][S3_RDZ][lj], iys = s.it[tq][S3_YS][lj];
          ax += dt * isx * (t2 * (txx - s.xx[q][e - 1]) * izx + t2 * (yip * yip * yxp - yi * yi * yx0) * (idyi * iym2) +
                            (yxp + yx0) * iym + t2 * (xzp - xz0) * irdz + t2 * (xzp + xz0) * czm * irs);
          ay += dt * isy * (t2 * (ym * ym * s.yy[e] - ymm * ymm * s.yy[e - S3_W]) * (idym * iyi * iyi) +
                            t2 * (s.yx[e + 1] - yx0) * (idx * iys) -
                            (txx + s.xx[q][e - S3_W] + zz0 + s.zz[q][e - S3_W]) * iyi +
                            t2 * (zyp * L[L3_SZIP] - zy0 * szi) * (ym * irdz * iys));
          az += dt * isz * (t2 * (zz0 * szm - s.zz[qn][e] * L[L3_SZMM]) * (irdm * ym * irsi) +
                            t2 * (s.xz[q][e + 1] - xz0) * (idx * irsi) +
                            t2 * (yip * yip * yip * s.zy[q][e + S3_W] - yi * yi * yi * zy0) * (idyi * iym2 * iym) -
                            (txx + s.xx[qn][e]) * czi * irsi);
        }
      }
      // SubStep2_a / SubStep2_b
      const double c2 = FB_CVNR;
      auto art = [&](double rr, double dv) { return dv < 0.0 ? c2 * c2 * rr * dv * dv : 0.0; };
      const double qx = art(r, s.u[p][e + 1] - u0), qxm = art(rxm, u0 - s.u[p][e - 1]);
      const double qy = art(r, s.vy[p][e + S3_W] - v0), qym = art(rym, v0 - s.vy[p][e - S3_W]);
      const double qz = art(r, s.vz[pp][e] - w0), qzm = art(rzm, w0 - s.vz[pm][e]);
      ax += quo(-2.0 * dt * dxmed * (qx - qxm), dx_, idx_) * izx;
      ay += quo(-2.0 * (qy - qym), dy_, idy_) * dt;
      az += quo(quo(-2.0 * (zm - zmm) * (qz - qzm), dz_, idz_) * dt, rdm, irdm);
      vxt[l] = FAST ? (S)(ax - s.bg[tq][lj]) : (S)ax;
      vyt[l] = (S)ay;
      vzt[l] = (S)az;
    }
    // no barrier here: the next layer's plane is one that this output does not
    // read, and its stresses wait for the barrier after it
  }
}

// layers a CTA marches over: long marches where the tiles alone fill the chip
// (2 resident CTAs on 148 SMs, several times over), short ones on small meshes;
// each march loads and forms one layer more than it writes
__host__ __device__ inline int s3_layers(long long tiles_layers, int nz) {
  long long k = tiles_layers / (148 * 2 * 3);
  if (k < 2) k = 2;
  if (k > 16) k = 16;
  const int segs = (int)((nz + k - 1) / k);
  return (nz + segs - 1) / segs;
}
__host__ __device__ inline int s3_ty(int precision) { return precision == FB_FP64 ? S3<double>::TY : S3<float>::TY; }
__host__ __device__ inline int s3_tiles(const fb_disk_dev &D) {
  const int ty = s3_ty(D.precision);
  return ((D.nx + S3_TX - 1) / S3_TX) * ((D.ny + ty - 1) / ty);
}
#ifndef FB_S3_MINB
#define FB_S3_MINB 2
#endif
template <typename S>
__global__ void __launch_bounds__(S3<S>::T, FB_S3_MINB) k_sources_sph(const __grid_constant__ fb_disk_dev D, int layers) {
  const Dims m = dims_of(D);
  const int segs = (m.nz + layers - 1) / layers, f = blockIdx.z / segs, k0 = FB_NGH + (blockIdx.z - f * segs) * layers;
  const fb_fluid_dev &F = D.fl[f];
  b_sources_sph<S>(m, geo_of<double>(D.geomd), (const S *)F.rho, (const S *)F.cs, (const S *)F.vx, (const S *)F.vy,
                   (const S *)F.vz, (S *)F.vxt, (S *)F.vyt, (S *)F.vzt, D.scal_dev, F.dust, !F.dust, F.vbg, blockIdx.x,
                   blockIdx.y, k0, min(k0 + layers, m.nz + FB_NGH));
}
// the kernel's shared memory is above the default limit: allowed once per
// device (idempotent, so threads may race to it)
template <auto Kernel, typename S>
inline int s3_allow(int device) {
  static std::atomic<unsigned long long> done{0};   // one per kernel
  const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
  if (bit && (done.load() & bit)) return 0;
  const int e = (int)cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(S3Shared<S>));
  if (!e) done.fetch_or(bit);
  return e;
}

}  // namespace fb
