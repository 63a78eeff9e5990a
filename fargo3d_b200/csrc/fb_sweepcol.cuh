// fb_sweepcol.cuh -- the radial and colatitude sweeps (TransportY/TransportZ,
// transport.c:24-46, for the density and every momentum: momenta_x/y/z,
// DivideByRho, VanLeerY/Z_a/_b, UpdateY/Z, UpdateDensityY/Z).
//
// A thread marches along one column over a segment of cells and keeps, of the
// density and of each of its quantities, only what the current face needs:
// each cell is loaded once, each specific momentum, slope and face value
// formed once.  (A window per segment in registers forms the halo cells'
// again: at 4 cells a segment twice the divisions by the density and half as
// many slopes again.)  The next cell's inputs are loaded a face ahead.
//
// FP64 keeps the reference's operations and order; divisors shared by several
// quotients (zone sizes, the density under the momenta, the cell volume) are
// inverted once (divk).  A thread carries at most 4 quantities beside the
// density, which 128 registers hold; 3D disks run two groups of three as
// separate CTAs, each of which advances the density for its own fluxes.
//
// FP32: the azimuthal momenta are relative to the frame and the ring
// background (fb_fluid_dev): the limiter sees the neighbour differences of
// the full specific momentum, l(c) = R (OMEGAFRAME R + vbg) restored from
// tables, and a face flux carries the upwind cell's offset from the updated
// cell's times the mass flux, so no large momentum is formed and cancelled.
#pragma once
#include "fb_kernels.cuh"

namespace fb {

// quantities: 0 Mpx, 1 Mmx, 2 Mpy, 3 Mmy, 4 Mpz, 5 Mmz, 6 the energy
template <typename T>
struct ColArgs {
  const T *rho, *vxt, *vyt, *vzt;
  const T *q[6];   // !FROMV: the momenta
  const T *e;      // the energy of adiabatic disks
  const T *dl;     // FP32: neighbour differences of vbg R along the sweep
  T *o_rho, *o[6], *o_e;
};
constexpr int COL_T = 128;   // columns per CTA

// DIR 0: along y (t2 is the layer k), 1: along z (t2 is the row j).  Q0, NQ:
// the quantities this CTA carries; FROMV: the momenta are formed from rho and
// V_temp; NE: the energy too.  Cells [c0, c1) of column (i, t2).
template <typename T, int DIR, int Q0, int NQ, bool FROMV, bool NE>
__device__ __forceinline__ void b_sweep_colm(const Dims &m, const Geo<T> &g, const ColArgs<T> &A, int i, int t2, int c0,
                                             int c1, const fb_scalars *__restrict__ scp) {
  constexpr bool F64 = sizeof(T) == 8;
  constexpr int NA = NQ + (NE ? 1 : 0);
  constexpr bool FLAT32 = !F64 && NQ == 4;   // the FP32 2D sweep
  const T dt = (T)scp->dt, of = (T)scp->omegaframe;
  const long long step = DIR == 0 ? (long long)m.pitch : m.stride;
  const long long base = DIR == 0 ? m.l(i, 0, t2) : m.l(i, t2, 0);
  const long long dxp = i < m.nx - 1 ? 1 : 1 - m.nx;   // to cell i + 1
  const T sxi = ld(g.sxi + (F64 ? i : 0));             // FP32 disks: uniform azimuthal spacing
  const T syk0 = DIR == 0 ? ld(g.syk + t2) : (T)0, ym0 = DIR == 1 ? ld(g.ymed + t2) : (T)0;
  const T szj0 = DIR == 1 ? ld(g.szj + t2) : (T)0, ivj0 = DIR == 1 ? ld(g.invvj + t2) : (T)0;
  const T st0 = DIR == 0 ? (m.sph ? ld(g.sin_zmed + t2) : (T)1) : (T)0;
  // cylindrical radius and Ymed of cell c
  auto ymed = [&](int c) -> T { return DIR == 0 ? ld(g.ymed + c) : ym0; };
  auto radius = [&](int c) -> T {
    if (FLAT32 || !m.sph) return ymed(c);
    return ymed(c) * (DIR == 0 ? st0 : ld(g.sin_zmed + c));
  };
  // FP32 2D: the row's zone size as it was differenced in double; a difference
  // of two FP32 edges is off by up to 6e-8 Ymin / zone, the same in every step
  auto zone = [&](int c) -> T {
    if (FLAT32) return ld(g.sxj + c);
    return DIR == 0 ? zsy(g, c) : zsz(m, g, t2, c);
  };
  // v Surf(c) (define.h:228-235, the macro's association); Syk = 1 in 2D
  auto surf = [&](T v, int c) -> T {
    if (DIR == 0) {
      const T x = v * ld(g.syj + c);
      return (m.is3d ? x * syk0 : x) * sxi;
    }
    return v * szj0 * ld(g.szk + c) * sxi;
  };
  const T ud0 = DIR == 0 ? syk0 * sxi : (T)0, iu0 = DIR == 0 ? (T)1.0 / ud0 : (T)0;
  // OMEGAFRAME (R^2(c) - R^2(c-1)) + (vbg R)(c) - (vbg R)(c-1)
  auto offs = [&](int c) -> T {
    T x;
    if (FLAT32 || !m.sph) x = ld(g.dr2_j + c);
    else if (DIR == 0) x = ld(g.dr2_j + c) * ld(g.s2_k + t2);
    else x = ld(g.r2_j + t2) * ld(g.ds2_k + c);
    return of * x + (A.dl ? ld(A.dl + (DIR == 0 ? c + t2 * m.sy : t2 + c * m.sy)) : (T)0);
  };

  // raw inputs of a cell; in[NA + 1]: rho, then one value per quantity (the
  // momentum, or with FROMV the velocity it is formed from)
  // (with FROMV the velocity on the cell's lower face along the sweep is the
  // one on the upper face of the cell below, vlo --
  // in FP64; in FP32, whose loop is bound by its instructions, carrying it over
  // costs more than the load: 64 disks 113 -> 130 us)
  constexpr int QUP = DIR == 0 ? 2 : 4;                          // the quantity read on the upper face
  constexpr bool UPS = F64 && FROMV && Q0 <= QUP && Q0 + NQ > QUP + 1;  // this CTA carries it and its lower twin
  T vlo = 0;
  auto load = [&](int c, T *in) {
    const long long l = base + (long long)c * step;
    in[0] = A.rho[l];
#pragma unroll
    for (int n = 0; n < NQ; n++) {
      const int q = Q0 + n;
      if (!FROMV) in[1 + n] = A.q[q][l];
      else if (q == 0) in[1 + n] = A.vxt[l + dxp];
      else if (q == 1) in[1 + n] = A.vxt[l];
      else if (q == 2) in[1 + n] = A.vyt[l + m.pitch];
      else if (q == 3) in[1 + n] = DIR == 0 && UPS ? vlo : A.vyt[l];
      else if (q == 4) in[1 + n] = A.vzt[l + m.stride];
      else in[1 + n] = DIR == 1 && UPS ? vlo : A.vzt[l];
    }
    if (NE) in[1 + NQ] = A.e[l];
  };
  // cell c's density r, momenta raw[] and specific momenta a[] from in[].
  // FP64: raw as the reference forms it and its quotient by the density;
  // FP32 with FROMV: the specific momentum directly, raw = a r at the update
  auto form = [&](int c, const T *in, T &r, T *raw, T *a) {
    r = in[0];
    const T ir = (T)1.0 / r;
    T R = 0, y = 0;
    if (FROMV && Q0 <= 1) R = radius(c);
    if (FROMV && m.sph) y = ymed(c);
#pragma unroll
    for (int n = 0; n < NA; n++) {
      const int q = n < NQ ? Q0 + n : 6;
      const T x = in[1 + n];
      if (!FROMV || q == 6) {
        raw[n] = x;
      } else if (F64) {
        if (q <= 1) raw[n] = (x + R * of) * R * r;
        else if (q <= 3) raw[n] = x * r;
        else raw[n] = m.sph ? x * r * y : x * r;
      } else {
        a[n] = q <= 1 ? x * R : (q <= 3 || !m.sph ? x : x * y);
        continue;
      }
      if constexpr (F64) a[n] = divk(raw[n], r, ir);
      else a[n] = raw[n] * ir;
    }
  };
  auto harm = [&](T dqm, T dqp) -> T {
    const T p = dqp * dqm;
    if (F64) {
      const bool none = p <= (T)0;
      const T w = ((T)2. * dqp * dqm) / (none ? (T)1 : dqm + dqp);
      return none ? (T)0 : w;
    }
    return p <= (T)0 ? (T)0 : (p + p) / (dqm + dqp);
  };
  auto quot = [&](T x, T y, T z) -> T {   // x / y, z = 1 / y
    if constexpr (F64) return divk(x, y, z);
    else return x * z;
  };
  constexpr bool KEEP = F64 || !FROMV;   // raw momenta are kept
  T in_[NA + 1];
  T r_m, r_0, r_p, dr_0, sr_m, Fr = 0;
  T a_m[NA], a_0[NA], a_p[NA], dq_0[NA], s_m[NA], F_m[NA], w_m[KEEP ? NA : 1], w_0[KEEP ? NA : 1], w_p[NA];
  T z_m, z_0, off_0 = 0, off_p = 0;
  // the velocity at the current face (with UPS the lower-face value of the cell
  // above it, which came with that cell)
  const T *vface = DIR == 0 ? A.vyt : A.vzt;
  T v_n;
  {
    T r_b, a_b[NA];   // cell c0 - 2
    if (UPS) vlo = (DIR == 0 ? A.vyt : A.vzt)[base + (long long)(c0 - 2) * step];
    load(c0 - 2, in_);
    form(c0 - 2, in_, r_b, w_p, a_b);
    if (UPS) vlo = in_[1 + QUP - Q0];
    load(c0 - 1, in_);
    form(c0 - 1, in_, r_m, w_p, a_m);
    if (UPS) vlo = in_[1 + QUP - Q0];
#pragma unroll
    for (int n = 0; n < NA; n++) if (KEEP) w_m[KEEP ? n : 0] = w_p[n];
    load(c0, in_);
    form(c0, in_, r_0, w_p, a_0);
    if (UPS) { vlo = in_[1 + QUP - Q0]; v_n = in_[1 + QUP + 1 - Q0]; }
#pragma unroll
    for (int n = 0; n < NA; n++) if (KEEP) w_0[KEEP ? n : 0] = w_p[n];
    load(c0 + 1, in_);
    z_m = zone(c0 - 1);
    z_0 = zone(c0);
    const T iz_m = (T)1.0 / z_m, iz_0 = (T)1.0 / z_0;
    T off_m = 0;
    if (!F64 && Q0 == 0) { off_m = offs(c0 - 1); off_0 = offs(c0); }
    const T dr_m = quot(r_m - r_b, z_m, iz_m);
    dr_0 = quot(r_0 - r_m, z_0, iz_0);
    sr_m = harm(dr_m, dr_0);
#pragma unroll
    for (int n = 0; n < NA; n++) {
      const bool rel = !F64 && Q0 + n <= 1 && n < NQ;
      const T dm = quot(a_m[n] - a_b[n] + (rel ? off_m : (T)0), z_m, iz_m);
      dq_0[n] = quot(a_0[n] - a_m[n] + (rel ? off_0 : (T)0), z_0, iz_0);
      s_m[n] = harm(dm, dq_0[n]);
      F_m[n] = 0;
    }
  }
  if (!UPS) v_n = vface[base + (long long)c0 * step];
#pragma unroll 1
  for (int f = c0; f <= c1; f++) {   // the face between cells f - 1 and f
    const T v = v_n;
    form(f + 1, in_, r_p, w_p, a_p);
    if (UPS) { vlo = in_[1 + QUP - Q0]; v_n = in_[1 + QUP + 1 - Q0]; }
    if (f < c1) {   // the next face's inputs
      load(f + 2, in_);
      if (!UPS) v_n = vface[base + (long long)(f + 1) * step];
    }
    const T z_p = zone(f + 1), iz_p = (T)1.0 / z_p;
    if (!F64 && Q0 == 0) off_p = offs(f + 1);
    const bool up = v > (T)0.;
    // VanLeer*_b: 0.5 (zone(upwind) -+ v dt)
    const T h = up ? (T)0.5 * (z_m - v * dt) : (T)0.5 * (z_0 + v * dt);
    const T dr_p = quot(r_p - r_0, z_p, iz_p), sr_0 = harm(dr_0, dr_p);
    const T rs = up ? r_m + h * sr_m : r_0 - h * sr_0;
    const int c = f - 1;   // the cell that face f completes
    const bool upd = f > c0;
    const long long l = base + (long long)c * step;
    T ud = ud0, iu = iu0, ivj = ivj0;
    if (DIR == 0) ivj = ld(g.invvj + c);
    if (DIR == 1) { ud = ld(g.syk + c) * sxi; iu = (T)1.0 / ud; }
    const T fin = F64 ? (T)0 : dt * ivj * iu;
    auto finish = [&](T fl) -> T {   // flux dt InvVol
      if constexpr (F64) return divk(fl * dt * ivj, ud, iu);
      else return fl * fin;
    };
    {
      const T fr = surf(v * rs, f);
      if (upd && (Q0 == 0)) A.o_rho[l] = r_m + finish(Fr - fr);
      Fr = fr;
    }
#pragma unroll
    for (int n = 0; n < NA; n++) {
      const int q = n < NQ ? Q0 + n : 6;
      const bool rel = !F64 && q <= 1;
      const T dq_p = quot(a_p[n] - a_0[n] + (rel ? off_p : (T)0), z_p, iz_p);
      const T s_0 = harm(dq_0[n], dq_p);
      const T qs = up ? a_m[n] + h * s_m[n] : a_0[n] - h * s_0;
      T fo, fi;   // the flux out of cell f - 1 and into cell f
      if (rel) {
        const T mass = Fr;
        fo = mass * (up ? qs : qs + off_0);
        fi = mass * (up ? qs - off_0 : qs);
      } else if (F64) {
        fo = fi = surf(v * qs * rs, f);
      } else {
        fo = fi = Fr * qs;
      }
      if (upd) {
        T *o = q == 6 ? A.o_e : A.o[q];
        const T raw = KEEP ? w_m[KEEP ? n : 0] : a_m[n] * r_m;
        o[l] = raw + finish(F_m[n] - fo);
      }
      F_m[n] = fi;
      a_m[n] = a_0[n]; a_0[n] = a_p[n];
      dq_0[n] = dq_p;
      s_m[n] = s_0;
      if (KEEP) { w_m[KEEP ? n : 0] = w_0[KEEP ? n : 0]; w_0[KEEP ? n : 0] = w_p[n]; }
    }
    r_m = r_0; r_0 = r_p;
    dr_0 = dr_p;
    sr_m = sr_0;
    z_m = z_0; z_0 = z_p;
    off_0 = off_p;
  }
}

// cells per segment: a segment of n cells forms n + 4 of them, so segments
// are long where the columns alone fill the chip (148 SMs x 512 threads) and
// short, down to 2 cells, where the mesh is small; a disk's set tile
// (fb_disk_set_tiles) comes first
__host__ __device__ inline int col_rows(long long columns, int cells, int set) {
  if (set) return set;
  const long long r = columns * cells / (148 * 512);
  return r < 2 ? 2 : (r > 16 ? 16 : (int)r);
}

template <typename T>
__host__ __device__ inline ColArgs<T> col_args(const fb_disk_dev &D, const fb_fluid_dev &F, int dir) {
  ColArgs<T> a;
  const bool y3 = D.is3d && dir == 0;   // the 3D Y sweep reads the Z sweep's set A and writes set B
  a.rho = (const T *)(y3 ? F.rho_a : F.rho);
  a.vxt = (const T *)F.vxt; a.vyt = (const T *)F.vyt; a.vzt = (const T *)F.vzt;
  const void *in[6] = {F.mpx, F.mmx, F.mpy, F.mmy, F.mpz, F.mmz};
  void *out[6] = {y3 ? F.mpx_b : F.mpx, y3 ? F.mmx_b : F.mmx, y3 ? F.mpy_b : F.mpy,
                  y3 ? F.mmy_b : F.mmy, y3 ? F.mpz_b : F.mpz, y3 ? F.mmz_b : F.mmz};
  for (int q = 0; q < 6; q++) { a.q[q] = (const T *)in[q]; a.o[q] = (T *)out[q]; }
  a.o_rho = (T *)(y3 ? F.rho_b : F.rho_a);
  a.e = (const T *)F.cs;
  a.o_e = (T *)F.e_a;
  a.dl = (const T *)(dir == 0 ? F.dlb_y : F.dlb_z);
  return a;
}
// resident CTAs of COL_T threads the sweep is compiled for
#ifndef FB_CM64_MINB
#define FB_CM64_MINB 4
#endif
// FP32: 2D at 8 (64 disks 113 -> 108 us against 6), 3D, with two quantities
// more, at 6 (512x256x48 230 us, 8 spills: 257)
template <typename T, bool IS3D>
constexpr int colm_minb() { return sizeof(T) == 8 ? FB_CM64_MINB : (IS3D ? 6 : 8); }
// blk: (column block, t2, segment x groups)
template <typename T, int DIR, bool IS3D, bool NE>
__device__ __forceinline__ void colm_cta(const Dims &m, const Geo<T> &g, const ColArgs<T> &A, int rows, uint3 bid,
                                         const fb_scalars *__restrict__ scp) {
  const int i = (int)bid.x * COL_T + threadIdx.x;
  if (i >= m.nx) return;
  const int clo = FB_NGH - 1, chi = (DIR == 0 ? m.ny : m.nz) + FB_NGH - 1;
  const int t2 = (int)bid.y + (IS3D && DIR == 0 ? FB_NGH - 1 : 0);
  if constexpr (!IS3D) {
    const int c0 = clo + (int)bid.z * rows;
    if (c0 > chi) return;
    b_sweep_colm<T, 0, 0, 4, true, NE>(m, g, A, i, 0, c0, min(c0 + rows, chi + 1), scp);
  } else if constexpr (sizeof(T) == 4) {
    const int c0 = clo + (int)bid.z * rows;
    if (c0 > chi) return;
    b_sweep_colm<T, DIR, 0, 6, DIR == 1, false>(m, g, A, i, t2, c0, min(c0 + rows, chi + 1), scp);
  } else {
    const int c0 = clo + (int)(bid.z >> 1) * rows;
    if (c0 > chi) return;
    const int c1 = min(c0 + rows, chi + 1);
    if ((bid.z & 1) == 0) b_sweep_colm<T, DIR, 0, 3, DIR == 1, false>(m, g, A, i, t2, c0, c1, scp);
    else b_sweep_colm<T, DIR, 3, 3, DIR == 1, false>(m, g, A, i, t2, c0, c1, scp);
  }
}
template <typename T, int DIR, bool IS3D, bool NE>
__global__ void __launch_bounds__(COL_T, colm_minb<T, IS3D>())
    k_sweep_colm(const __grid_constant__ fb_disk_dev D, int rows) {
  const int gz = gridDim.z / D.nfluids, f = blockIdx.z / gz;
  colm_cta<T, DIR, IS3D, NE>(dims_of(D), geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), col_args<T>(D, D.fl[f], DIR), rows,
                             make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - f * gz), D.scal_dev);
}
// grid of a sweep: columns, transverse index (3D Z: rows 0 .. sy-2; Y: layers
// Nghz-1 ..), segments (x 2 groups in FP64 3D)
__host__ __device__ inline dim3 colm_grid(const fb_disk_dev &D, int dir, int rows) {
  const int n = (dir == 0 ? D.ny : D.nz) + 1;
  const int segs = (n + rows - 1) / rows;
  return dim3((D.nx + COL_T - 1) / COL_T, !D.is3d ? 1 : (dir == 0 ? D.nz + 1 : D.sy - 1),
              D.is3d && D.precision == FB_FP64 ? 2 * segs : segs);
}
__host__ __device__ inline int colm_rows(const fb_disk_dev &D, int dir) {
  return col_rows((long long)D.nx * (!D.is3d ? 1 : (dir == 0 ? D.nz + 1 : D.sy - 1)), (dir == 0 ? D.ny : D.nz) + 1,
                  D.tile_ns);
}

}  // namespace fb
