// fb_sources32.cuh -- the source stage of FP32 2D cylindrical disks
// (algogas.c:30-120: ComputePressureFieldIso, the planets' potential,
// CorrectVtheta, SubStep1_x/y, visctensor_cyl + addviscosity_cyl, SubStep2_a/b)
// in FP32 arithmetic.  Cells pass through registers and shuffles; shared memory
// holds what a row contributes and the planets, formed once per CTA before its
// one barrier.
//
// Layout of the work: a warp owns 32 consecutive columns (azimuthal cells) of
// a ring and marches over 2 to 16 rows (s32_rows), keeping j-1, j, j+1 of its
// column in registers; the neighbours i-1 / i+1 come from the adjacent lanes
// by shuffle.  Lanes 0 and 31 are halo lanes: they compute what their
// neighbours need but write nothing, so a warp writes 30 columns.  Every
// quantity (pressure, planet potential, the three viscous stresses) is formed
// once per cell and row, none is staged or recomputed for a tile halo.
//
// Why FP32 is safe here: FP32 disks store v_phi relative to a per-ring
// background vbg (fb_fluid_dev), so no large velocity enters the arithmetic.
// What remains large is the background's own radial balance -- centrifugal
// (B^2 / r) against the star's gravity, with B = vbg + r OMEGAFRAME on the
// face -- two O(1) terms whose difference is O(h^2).  That difference is
// formed per row in FP64 (K_j below) and only the perturbation terms,
// (2 B + d) d / r with d the small relative velocity, the planets' potential
// and the pressure gradient, are formed in FP32.  Likewise the background's
// r-phi shear enters tau_r_phi as one per-row constant (fb_fluid_dev shear_bg,
// formed in FP64).  The planets' potential is the only potential evaluated
// per cell: the star's -GM/r cancels in the x differences and is part of
// K_j in the y difference.
#pragma once
#include "fb_kernels.cuh"

namespace fb {

constexpr int S32_WARPS = 4;                       // warps per CTA
constexpr int S32_OUT = 30;                        // columns written per warp (lanes 1..30)
constexpr int S32_COLS = S32_WARPS * S32_OUT;      // columns per CTA
constexpr int S32_NS = 16;                         // most rows per CTA
// resident CTAs per SM the kernel is compiled for (register cap 64 at 8)
#ifndef FB_S32_MINB
#define FB_S32_MINB 8
#endif

// one row of a column: density, sound speed, relative azimuthal velocity
// (CorrectVtheta applied), radial velocity, pressure, planets' potential
struct Cell32 {
  float r, c, u, vy, p, pot;
};

__device__ __forceinline__ float lane_m(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }    // column i-1
__device__ __forceinline__ float lane_p(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }  // column i+1

// The planets of one step in FP32, formed once per CTA: position, mass,
// smoothing^2 + z^2 and the indirect-term factor m / d^3 (0 without it).
struct Planet32 {
  float x, y, m, s2z, ind;
};

// What a row contributes to the stencil, formed once per CTA and row and read
// as four broadcast 16-byte words: the radii and their reciprocals, the face
// areas and zone size, the viscosity factors, the background's balance K and
// velocity B on the lower face, and the factors of the viscous accelerations
// (addviscosity_cyl.c:106-124).  Reading the tables and dividing by them in
// every lane took a third of the kernel's instructions.
struct Row32 {
  float ym, iym, iyi, idym;       // Ymed, 1/Ymed, 1/Ymin, 1/(Ymed(j)-Ymed(j-1))
  float syj, sxj, isxj, f23;      // SurfY, zone size and its reciprocal, (2/3) InvVol / Sxi
  float visc, viscm, shb, yi2;    // alpha-nu factors, background shear, Ymin^2
  float K, B, ax2, ay1;           // 2 / (zone Ymed^2), 2 / ((Ymed(j)-Ymed(j-1)) Ymin)
};

// planets' potential (potential.c:51-208 without the star's term), FP32
__device__ __forceinline__ float pot_planets32(const Planet32 *sp, int np, float XC, float YC) {
  float pot = 0.0f;
  for (int n = 0; n < np; n++) {
    const Planet32 p = sp[n];
    const float dx = XC - p.x, dy = YC - p.y;
    pot += p.ind * (XC * p.x + YC * p.y);
    pot -= p.m * rsqrtf(dx * dx + dy * dy + p.s2z);
  }
  return pot;
}

__device__ __forceinline__ void b_sources_cyl32(const Dims m, const Geo<float> g, const Geo<double> gd,
    const float *__restrict__ rho, const float *__restrict__ cs, const float *__restrict__ vx,
    const float *__restrict__ vy, float *__restrict__ vxt, float *__restrict__ vyt,
    const fb_scalars *__restrict__ sc, int dust, int viscous, const double *__restrict__ vbg,
    const float *__restrict__ shear_bg, const double *__restrict__ tab, int rows, uint3 bid) {
  __shared__ Planet32 s_pl[FB_MAXPLANETS];
  __shared__ __align__(16) Row32 s_row[S32_NS + 2];   // rows j0 - 1 .. j1
  const int j0 = FB_NGH + (int)bid.y * rows, j1 = min(j0 + rows, m.ny + FB_NGH);
  if (j0 >= j1) return;
  const int np = sc->nplanets;
  const double dtd = sc->dt, of = sc->omegaframe;
  const float sxi0 = ld(g.sxi + 0), idx0 = ld(g.invdiffxmed + 0);
  if ((int)threadIdx.x < np) {
    const int n = threadIdx.x;
    Planet32 p;
    p.x = (float)sc->px[n];
    p.y = (float)sc->py[n];
    p.m = (float)sc->pmass[n];
    p.s2z = (float)(sc->psmooth2[n] + sc->pz[n] * sc->pz[n]);
    p.ind = sc->indirect_term ? (float)(sc->pmass[n] / sc->pdist3[n]) : 0.0f;
    s_pl[n] = p;
  }
  if ((int)threadIdx.x >= 32 && (int)threadIdx.x - 32 < j1 - j0 + 2) {
    const int q = threadIdx.x - 32, j = j0 - 1 + q;   // 2 .. ny + 3: j - 1 and j + 1 are stored rows
    Row32 R;
    R.ym = ld(g.ymed + j); R.iym = ld(g.inv_ymed + j); R.iyi = ld(g.inv_ymin + j); R.idym = ld(g.inv_dymed + j);
    R.syj = ld(g.syj + j); R.sxj = ld(g.sxj + j); R.isxj = 1.0f / R.sxj;
    R.f23 = (2.0f / 3.0f) * ld(g.invvj + j) / sxi0;
    R.visc = ld(g.visc_j + j); R.viscm = ld(g.viscm_j + j); R.shb = ld(shear_bg + j);
    const float yi = ld(g.ymin + j);
    R.yi2 = yi * yi;
    // the background's balance on face j: K = B^2 / r - d(Phi_star)/dr,
    // B = (vbg(j) + vbg(j-1)) / 2 + Ymin(j) OMEGAFRAME, in FP64
    const double Bd = 0.5 * (bg_at(vbg, j) + bg_at(vbg, j - 1)) + ld(gd.ymin + j) * of;
    R.K = (float)(Bd * Bd * ld(gd.inv_ymin + j) - (ld(gd.pot_star + j) - ld(gd.pot_star + j - 1)) * ld(gd.inv_dymed + j));
    R.B = (float)Bd;
    R.ax2 = 2.0f * R.iym * R.iym * R.isxj;
    R.ay1 = 2.0f * R.idym * R.iyi;
    s_row[q] = R;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int iu = (int)(bid.x * S32_WARPS + w) * S32_OUT - 1 + lane;   // unwrapped column of this lane
  const int i = ((iu % m.nx) + m.nx) % m.nx;
  const bool writes = lane >= 1 && lane <= S32_OUT && iu < m.nx;
  if ((int)(bid.x * S32_WARPS + w) * S32_OUT - 1 >= m.nx) return;   // the whole warp lies past the ring
  const float dt = (float)dtd, domega = (float)sc->domega, nu = (float)sc->nu, alpha = (float)sc->alpha;
  const float cx = ld(g.cos_xmed + i), sx = ld(g.sin_xmed + i), isx2 = 2.0f / sxi0;
  const float cv2 = (float)(FB_CVNR * FB_CVNR);
  const float *pr = rho + m.l(i, j0 - 1, 0), *pc = cs + m.l(i, j0 - 1, 0), *pu = vx + m.l(i, j0 - 1, 0),
              *pv = vy + m.l(i, j0 - 1, 0);
  float *ou = vxt + m.l(i, j0, 0), *ov = vyt + m.l(i, j0, 0);
  float in[4];
  auto fetch = [&]() {   // the next row's inputs
    in[0] = *pr; in[1] = *pc; in[2] = *pu; in[3] = *pv;
    pr += m.pitch; pc += m.pitch; pu += m.pitch; pv += m.pitch;
  };
  auto form = [&](const Row32 &R) -> Cell32 {
    Cell32 o;
    o.r = in[0];
    o.c = in[1];
    o.u = in[2] - domega * R.ym;     // CorrectVtheta (correct_vtheta.c:55-60)
    o.vy = in[3];
    o.p = o.r * o.c * o.c;           // ComputePressureFieldIso
    o.pot = pot_planets32(s_pl, np, R.ym * cx, R.ym * sx);
    return o;
  };
  // tau_phi_phi and tau_r_r of the row (visctensor_cyl.c): C its cells, vyp
  // the radial velocity of the row above, uxp the velocity of column i + 1
  auto diag = [&](const Row32 &R, float syjp, const Cell32 &C, float vyp, float uxp, float &txx, float &tyy) {
    const float mu = (m.alpha ? alpha * C.c * C.c * R.visc : nu) * C.r;
    const float dux = uxp - C.u, dvy = vyp - C.vy;
    const float div_v = (dux * R.sxj + (vyp * syjp * sxi0 - C.vy * R.syj * sxi0)) * R.f23;
    txx = mu * (2.0f * dux * (idx0 * R.iym) - div_v + (vyp + C.vy) * R.iym);
    tyy = mu * (2.0f * dvy * R.isxj - div_v);
  };
  // tau_r_phi at the corner (i - 1/2, j - 1/2) from rows j (C) and j - 1 (Cm)
  auto corner = [&](const Row32 &R, const Cell32 &C, const Cell32 &Cm) -> float {
    const float rs = C.r + Cm.r, rxs = lane_m(rs), vyxm = lane_m(C.vy);
    float viscm = nu;
    if (m.alpha) {
      const float cc = C.c + Cm.c, s4 = cc + lane_m(cc);
      viscm = alpha * 0.0625f * s4 * s4 * R.viscm;
    }
    return viscm * 0.25f * (rs + rxs) *
           ((C.vy - vyxm) * idx0 * R.iyi + (C.u - Cm.u) * R.idym - 0.5f * (C.u + Cm.u) * R.iyi + R.shb);
  };
  // rows j0 - 1 and j0; the stresses of row j0 - 1 and the corner of row j0
  fetch();
  Cell32 A = form(s_row[0]);
  fetch();
  Cell32 C0 = form(s_row[1]);
  fetch();
  float uxp = lane_p(C0.u), umxp = lane_p(A.u);
  float txx_m = 0.f, tyy_m = 0.f, tyx_c = 0.f;
  if (viscous) {
    diag(s_row[0], s_row[1].syj, A, C0.vy, umxp, txx_m, tyy_m);
    tyx_c = corner(s_row[1], C0, A);
  }
  for (int j = j0; j < j1; j++) {
    const Row32 &R = s_row[j - j0 + 1], &Rp = s_row[j - j0 + 2];
    const Cell32 P = form(Rp);
    if (j + 1 < j1) fetch();
    float txx_c = 0.f, tyy_c = 0.f, tyx_p = 0.f;
    if (viscous) {
      diag(R, Rp.syj, C0, P.vy, uxp, txx_c, tyy_c);
      tyx_p = corner(Rp, P, C0);
    }
    // neighbours by shuffle (every lane takes part)
    const float rxm = lane_m(C0.r), pxm = lane_m(C0.p), potxm = lane_m(C0.pot);
    const float uxm = lane_m(C0.u), upxp = lane_p(P.u);
    const float txx_xm = lane_m(txx_c), tyx_xp = lane_p(tyx_c);
    const float r = C0.r, rym = A.r;
    const float izx = idx0 * R.iym;
    const float sxm = s_row[j - j0].sxj;
    const float irx = __fdividef(1.0f, r + rxm);   // 1 / (rho + rho_{i-1}) (uniform azimuthal spacing)
    const float ideny = __fdividef(1.0f, r * R.sxj + rym * sxm);
    // artificial viscosity (substep2_a.c:107-129): negative differences only
    const float du = fminf(uxp - C0.u, 0.0f), dum = fminf(C0.u - uxm, 0.0f);
    const float dv = fminf(P.vy - C0.vy, 0.0f), dvm = fminf(C0.vy - A.vy, 0.0f);
    const float qx = cv2 * (r * du * du - rxm * dum * dum), qy = cv2 * (r * dv * dv - rym * dvm * dvm);
    // SubStep1_x (substep1_x.c:107-117), SubStep2
    float fx = (dust ? 0.0f : C0.p - pxm) + qx, fy = (dust ? 0.0f : C0.p - A.p) + qy;
    float ax = -2.0f * irx * fx * izx - (C0.pot - potxm) * izx;
    // SubStep1_y (substep1_y.c:146-192, cylindrical)
    const float d = 0.25f * (C0.u + uxp + A.u + umxp);
    float ay = R.K + (2.0f * R.B + d) * d * R.iyi - (C0.pot - A.pot) * R.idym - 2.0f * ideny * fy;
    if (viscous) {
      // addviscosity_cyl (addviscosity_cyl.c:106-124)
      const float iry = __fdividef(1.0f, r + rym);
      ax += irx * (2.0f * (txx_c - txx_xm) * izx + (Rp.yi2 * tyx_p - R.yi2 * tyx_c) * R.ax2);
      ay += iry * ((R.ym * tyy_c - s_row[j - j0].ym * tyy_m) * R.ay1 +
                   ((tyx_xp - tyx_c) * isx2 - (txx_c + txx_m)) * R.iyi);
    }
    if (writes) {
      const float u1 = fmaf(ax, dt, C0.u), v1 = fmaf(ay, dt, C0.vy);   // relative to the background, as the state
      *ou = u1;
      *ov = j == FB_NGH && m.bclo ? 0.0f : v1;
      if (edge_row(m, j)) ghosts_of_row<float>(m, gd.ymed, tab, vbg, of, i, j, nullptr, vxt, vyt, nullptr, r, u1, v1, 0.0f);
    }
    ou += m.pitch;
    ov += m.pitch;
    A = C0;
    C0 = P;
    umxp = uxp;
    uxp = upxp;
    txx_m = txx_c;
    tyy_m = tyy_c;
    tyx_c = tyx_p;
  }
}

// rows a warp marches over: 16 where that fills the chip (148 SMs x 32
// resident warps), fewer on small meshes; a march forms two rows more than it
// writes
__host__ __device__ inline int s32_rows(long long cells) {
  const long long r = cells / (30ll * 148 * 32);
  return r < 2 ? 2 : (r > S32_NS ? S32_NS : (int)r);
}

static __global__ void __launch_bounds__(S32_WARPS * 32, FB_S32_MINB) k_sources_cyl32(const __grid_constant__ fb_disk_dev D, int rows) {
  const fb_fluid_dev &F = D.fl[blockIdx.z];
  b_sources_cyl32(dims_of(D), geo_of<float>(D.geom), geo_of<double>(D.geomd), (const float *)F.rho,
                  (const float *)F.cs, (const float *)F.vx, (const float *)F.vy, (float *)F.vxt, (float *)F.vyt,
                  D.scal_dev, F.dust, !F.dust, F.vbg, (const float *)F.shear_bg, D.bnd_tab, rows, blockIdx);
}

// ---------------------------------------------------------------------------
// CFL time step of FP32 2D disks (cfl.c:135-258, cfl_b.c:14-39) whose rings
// are no multiple of four cells: 128 columns x CFL32_R rows, a lane per column
// marching over the rows with every load of the tile issued up front (the
// kernel is a stream of four fields; it is bound by how many loads are in
// flight), the x neighbour's vx by shuffle, the next row's vy reused.  The
// tile's minimum (with the shear limits of its rows) is folded into the
// disk's by cfl_commit; non-finite limits and non-positive densities set the
// disk's flag word.
constexpr int CFL32_R = 8;

__device__ __forceinline__ void b_cfl_cyl32(const Dims m, const Geo<float> g, const float *__restrict__ rho,
    const float *__restrict__ cs, const float *__restrict__ vx, const float *__restrict__ vy,
    const double *__restrict__ vxmed, const double *__restrict__ vbg, float nu, float alpha, double cfl_num,
    double mindx, unsigned long long *__restrict__ dtmin, uint3 bid) {
  const int lane = threadIdx.x & 31;
  const int i = (int)bid.x * blockDim.x + threadIdx.x;
  const int j0 = FB_NGH + (int)bid.y * CFL32_R;
  const int nr = min(CFL32_R, m.ny + FB_NGH - j0);
  const bool act = i < m.nx;
  const int ic = act ? i : m.nx - 1;
  const int ixp = ic < m.nx - 1 ? ic + 1 : 0;
  float r[CFL32_R], c[CFL32_R], u[CFL32_R], v[CFL32_R + 1], uxp_edge[CFL32_R];
#pragma unroll
  for (int q = 0; q < CFL32_R; q++) {
    const int j = j0 + min(q, nr - 1);
    const long long l = m.l(ic, j, 0);
    r[q] = rho[l];
    c[q] = cs[l];
    u[q] = vx[l];
    v[q] = vy[l];
    uxp_edge[q] = (lane == 31 || ic == m.nx - 1) ? vx[m.l(ixp, j, 0)] : 0.0f;
  }
  v[CFL32_R] = vy[m.l(ic, j0 + nr, 0)];
  const float cflf = (float)cfl_num;
  const float izx0 = ld(g.invdiffxmed + 0);
  float mn = 1e20f;
  bool bad = false;
#pragma unroll
  for (int q = 0; q < CFL32_R; q++) {
    const int j = j0 + min(q, nr - 1);
    float uxp = lane_p(u[q]);
    if (lane == 31 || ic == m.nx - 1) uxp = uxp_edge[q];
    const float vyp = q + 1 < nr ? v[q + 1] : v[CFL32_R];
    const float vmf = (float)(vxmed[j] - bg_at(vbg, j));
    const float izx = izx0 * ld(g.inv_ymed + j), izy = 1.0f / ld(g.sxj + j);
    const float visc = m.alpha ? alpha * c[q] * c[q] * ld(g.visc_j + j) : nu;
    const float mx7 = fmaxf(izx, izy);
    const float c1 = fabsf(c[q]) * mx7;
    const float c2 = fmaxf(fabsf(u[q] - vmf), fabsf(uxp - vmf)) * izx;
    const float c3 = fmaxf(fabsf(v[q]), fabsf(vyp)) * izy;
    const float c5 = fmaxf(fabsf(uxp - u[q]) * izx, fabsf(vyp - v[q]) * izy) * (4.0f * (float)FB_CVNR);
    const float c7 = 4.0f * visc * (mx7 * mx7);
    const float dtc = cflf * rsqrtf(c1 * c1 + c2 * c2 + c3 * c3 + c5 * c5 + c7 * c7);
    if (act && q < nr) {
      bad |= !(dtc == dtc) || !(r[q] > 0.0f);
      mn = fminf(mn, dtc);
    }
  }
  double mnd = (double)mn;
  if ((int)threadIdx.x < nr) {   // the shear limits of the tile's rows (a MIN: repeats are harmless)
    const int j = j0 + threadIdx.x;
    const double shear = cfl_shear(g, vxmed, cfl_num, mindx, j, j);
    if (shear < mnd) mnd = shear;
  }
  if (bad) atomicOr(dtmin + 1, 1ull);
  cfl_commit(mnd, dtmin);
}

// ---------------------------------------------------------------------------
// CFL limits of FP32 2D disks whose rings hold a multiple of four cells: a
// thread takes Q32_K quads of four consecutive cells, Q32_T quads apart, with
// 16-byte loads, so that a CTA's fixed costs (its descriptor, the fold of its
// minimum: 40 % of the instructions with one quad a thread) are paid once per
// Q32_K Q32_T quads.  The loop is not unrolled: the loads of the resident
// warps hide each other, and two quads at once cost a third of them (68 us
// against 62 for one).  The x neighbour of a quad's last cell comes from the
// next lane when that lane holds the adjacent cells of the same row, else from
// one load; the row above (vy) by a second 16-byte load.  Per cell the
// arithmetic of b_cfl_cyl32.
constexpr int Q32_T = 128, Q32_K = 4;
__device__ __forceinline__ float4 ld4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float q4(const float4 &a, int k) { return k == 0 ? a.x : (k == 1 ? a.y : (k == 2 ? a.z : a.w)); }

__device__ __forceinline__ void b_cfl_cyl32q(const Dims &m, const Geo<float> &g, const float *__restrict__ rho,
    const float *__restrict__ cs, const float *__restrict__ vx, const float *__restrict__ vy,
    const double *__restrict__ vxmed, const double *__restrict__ vbg, float nu, float alpha, double cfl_num,
    double mindx, unsigned long long *__restrict__ dtmin, int blk) {
  const int lane = threadIdx.x & 31;
  const int qpr = m.nx >> 2, nq = qpr * m.ny;
  const float cflf = (float)cfl_num, izx0 = ld(g.invdiffxmed + 0);
  float mx = 0.0f;   // the largest sum of squares; the limit is cfl / sqrt of it
  double mnd = 1e20;
  bool bad = false, shears = false;
#pragma unroll 1
  for (int e = 0; e < Q32_K; e++) {
    const int t0 = (blk * Q32_K + e) * Q32_T;
    if (t0 >= nq) break;
    // quads past the disk's last repeat it (a minimum does not mind)
    const int t = min(t0 + (int)threadIdx.x, nq - 1);
    const int j = FB_NGH + t / qpr, q = t - (j - FB_NGH) * qpr;
    const long long l = m.l(4 * q, j, 0);
    const float4 r4 = ld4(rho + l), c4 = ld4(cs + l), u4 = ld4(vx + l), v4 = ld4(vy + l), vp4 = ld4(vy + l + m.pitch);
    // vx of cell 4q + 4: the next lane's first cell, or a load (ring wrap, warp edge, repeats)
    float uxp3 = __shfl_down_sync(0xffffffffu, u4.x, 1);
    if (lane == 31 || q == qpr - 1) uxp3 = vx[q == qpr - 1 ? m.l(0, j, 0) : l + 4];
    const float vmf = (float)(vxmed[j] - bg_at(vbg, j));
    const float izx = izx0 * ld(g.inv_ymed + j), izy = 1.0f / ld(g.sxj + j);
    const float vj = alpha * ld(g.visc_j + j);
    const float mx7 = fmaxf(izx, izy), m2 = 4.0f * mx7 * mx7;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float c = q4(c4, k), u = q4(u4, k), v = q4(v4, k), vyp = q4(vp4, k);
      const float uxp = k < 3 ? q4(u4, k + 1) : uxp3;
      const float c1 = c * mx7;
      const float c2 = fmaxf(fabsf(u - vmf), fabsf(uxp - vmf)) * izx;
      const float c3 = fmaxf(fabsf(v), fabsf(vyp)) * izy;
      const float c5 = fmaxf(fabsf(uxp - u) * izx, fabsf(vyp - v) * izy) * (4.0f * (float)FB_CVNR);
      const float c7 = (m.alpha ? vj * c * c : nu) * m2;
      const float sum = c1 * c1 + c2 * c2 + c3 * c3 + c5 * c5 + c7 * c7;
      bad |= !(sum == sum) || !(q4(r4, k) > 0.0f);
      mx = fmaxf(mx, sum);
    }
    if (q == 0) {   // the shear limit of row j (once per row; repeats are harmless)
      const double shear = cfl_shear(g, vxmed, cfl_num, mindx, j, j);
      if (shear < mnd) mnd = shear;
      shears = true;
    }
  }
  const float mn = cflf * rsqrtf(mx);   // infinite where nothing moves
  if (bad) atomicOr(dtmin + 1, 1ull);
  // block minimum, folded into the disk's: the cells' limits as the bits of
  // non-negative floats, the few shear limits in FP64
  __shared__ double wm[Q32_T / 32];
  const unsigned bits = __reduce_min_sync(0xffffffffu, __float_as_uint(mn));
  if (__any_sync(0xffffffffu, shears))
    for (int o = 16; o > 0; o >>= 1) mnd = fmin(mnd, __shfl_xor_sync(0xffffffffu, mnd, o));
  if (lane == 0) wm[threadIdx.x >> 5] = fmin((double)__uint_as_float(bits), mnd);
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = wm[0];
#pragma unroll
    for (int w = 1; w < Q32_T / 32; w++) v = fmin(v, wm[w]);
    if (v > 0.0) atomicMin(dtmin, (unsigned long long)__double_as_longlong(v));
  }
}
static __global__ void __launch_bounds__(Q32_T) k_cfl_cyl32q(const __grid_constant__ fb_disk_dev D) {
  const fb_fluid_dev &F = D.fl[blockIdx.y];
  b_cfl_cyl32q(dims_of(D), geo_of<float>(D.geom), (const float *)F.rho, (const float *)F.cs, (const float *)F.vx,
               (const float *)F.vy, F.vxmed, F.vbg, (float)D.scal_dev->nu, (float)D.scal_dev->alpha, D.cfl, D.mindx,
               (unsigned long long *)D.dtmin, blockIdx.x);
  cfl_report(D);
}
static __global__ void __launch_bounds__(128) k_cfl_cyl32(const __grid_constant__ fb_disk_dev D) {
  const fb_fluid_dev &F = D.fl[blockIdx.z];
  b_cfl_cyl32(dims_of(D), geo_of<float>(D.geom), (const float *)F.rho, (const float *)F.cs, (const float *)F.vx,
              (const float *)F.vy, F.vxmed, F.vbg, (float)D.scal_dev->nu, (float)D.scal_dev->alpha, D.cfl, D.mindx,
              (unsigned long long *)D.dtmin, blockIdx);
  cfl_report(D);
}
__host__ __device__ inline int cfl32q_ctas(int nx, int ny) {
  return (nx / 4 * ny + Q32_T * Q32_K - 1) / (Q32_T * Q32_K);
}

}  // namespace fb
