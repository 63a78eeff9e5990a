// fb_sweepx.cuh -- the azimuthal sweep (transport.c:129-158: FARGO residual
// with van Leer, the uniform rest with PPA, the integer shift) on registers,
// fused in 2D with NewVelocity_x/y and StockholmBoundary.
//
// Layout of the work: a warp owns a strip of N = 32 C consecutive cells of a
// ring, C per lane, and marches over rings.  Both advection passes run in
// registers: neighbours within a lane are registers, those across lanes
// shuffles, so every specific momentum, slope, edge and face value is formed
// once per cell and no shared-memory round trip or barrier separates the
// stages.  The stencil of the two passes reaches 5 cells to either side (6 to
// the left with newvel_x), so of the N cells the outer halo lanes are
// computed but not written: XS<C>::W are.  A ring of exactly N cells needs no
// halo (the shuffles wrap around).
//
// The strip is a range of OUTPUT columns: AdvectSHIFT moves cell i to
// i + nshift(ring), so the warp reads its cells from column - nshift.  Rows
// of one warp are then aligned in their outputs, and newvel_y finds the row
// below in the same lane's registers from the previous ring (the ring before
// a warp's first one is advected once more for its density and Mpy only).
//
// Ring pieces arrive by bulk copies (TMA) into a two-stage buffer of the warp
// while the previous ring is computed; each wait is bounded.  Rings whose
// rows are not 16-byte multiples are read with plain loads.
#pragma once
#include "fb_kernels.cuh"

namespace fb {

template <int C>
struct XS {
  static constexpr int N = 32 * C;                  // cells a warp holds
  static constexpr int HL = 6;                      // left halo; at least 5 cells follow the written ones
  static constexpr int W = (N - HL - 5) / 2 * 2;    // columns written: an even number, from an even column
};
// strips of a ring
template <int C>
__host__ __device__ inline int xs_strips(int nx) {
  return nx == XS<C>::N ? 1 : (nx + XS<C>::W - 1) / XS<C>::W;
}
constexpr int XS_WARPS = 4;   // warps per CTA (independent of one another)
// cells per lane: the strips are as wide as the registers allow (FP64 128,
// FP32 96 a thread), because the halo is a fixed number of cells
template <typename T>
struct XsC { static constexpr int C = sizeof(T) == 8 ? 2 : 4; };
// elements of one staged ring piece: N cells from a 16-byte boundary
template <typename T, int C>
struct XsRow { static constexpr int E = 16 / (int)sizeof(T), LEN = XS<C>::N + E; };
// dynamic shared memory: two stages of (rho, nq momenta, vxt) per warp
template <typename T, int C>
__host__ __device__ inline size_t xs_smem(int nq) {
  return (size_t)XS_WARPS * 2 * (nq + 2) * XsRow<T, C>::LEN * sizeof(T);
}

template <typename T>
struct XsArgs {
  const T *rho, *vxt;        // transported density, V_temp
  const T *q[6];             // transported momenta (the energy of adiabatic disks as the fifth)
  T *o_rho, *o[6];           // not fused: the advected quantities
  T *s_rho, *s_vx, *s_vy, *s_e;   // fused (2D): the new state
  const T *rho0, *vx0, *vy0; // Stockholm profiles
  const double *ramps;
  const double *tab, *vbg, *ymed;   // ghosts: boundary factors, background, Ymed
  int stockholm;
  const double *vxmed_t;     // ring means of V_temp
  const int *nshift;         // integer shift of each ring (ring_shift)
  const float4 *ringx;       // FP32 rings' scalars (ring_shift)
};

template <typename V>
__device__ __forceinline__ V from_left(V v, int lane) { return __shfl_sync(0xffffffffu, v, (lane + 31) & 31); }
template <typename V>
__device__ __forceinline__ V from_right(V v, int lane) { return __shfl_sync(0xffffffffu, v, (lane + 1) & 31); }

// ---- FP64: the reference's operations in its order ------------------------
// Scalars of a lane's C cells / lower faces for both passes of one ring.
template <int C>
struct XsRing64 {
  double z[C], iz[C], iu[C];    // zone size, its reciprocal; 1 / (syk sxi)
  double iu_d[C];               // syk sxi
  double v0[C], h0[C];          // residual velocity; 0.5 (zone(up) -+ v dt)
  double v1[C], ks[C], kk[C];   // rest velocity, |v| dt / zone, ks (1 - ks)
  double s1, s2, s3, s4;        // sxj, sxk, dt, invvj
  bool flat;                    // 2D: sxk = 1
};
// fl Surf dt / Vol (update_x.c) in the reference's order
template <int C>
__device__ __forceinline__ double xs_upd(const XsRing64<C> &R, double fl, int u) {
  double x = fl * R.s1;
  if (!R.flat) x = x * R.s2;
  return divk(x * R.s3 * R.s4, R.iu_d[u], R.iu[u]);
}
// van Leer face values (vanleer_x_a/_b) at the C lower faces of the cells a
template <int C>
__device__ __forceinline__ void xs_vl(const XsRing64<C> &R, const double *a, int lane, double *qs) {
  double dq[C + 1], s[C];
  const double am = from_left(a[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++) dq[u] = divk(a[u] - (u ? a[u - 1] : am), R.z[u], R.iz[u]);
  dq[C] = from_right(dq[0], lane);
#pragma unroll
  for (int u = 0; u < C; u++) {
    const double dqm = dq[u], dqp = dq[u + 1];
    const bool none = dqp * dqm <= 0.0;
    const double w = (2. * dqp * dqm) / (none ? 1.0 : dqm + dqp);
    s[u] = none ? 0.0 : w;
  }
  const double sm = from_left(s[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++) {
    const double al = u ? a[u - 1] : am, sl = u ? s[u - 1] : sm;
    qs[u] = R.v0[u] > 0.0 ? al + R.h0[u] * sl : a[u] - R.h0[u] * s[u];
  }
}
// PPA face values (fargo_ppa_a..d)
template <int C>
__device__ __forceinline__ void xs_ppa(const XsRing64<C> &R, const double *a, int lane, double *qs) {
  double d[C + 1], s[C], e[C + 1], L[C], Rr[C];
  const double am = from_left(a[C - 1], lane), ap = from_right(a[0], lane);
#pragma unroll
  for (int u = 0; u <= C; u++) d[u] = (u < C ? a[u] : ap) - (u ? a[u - 1] : am);
#pragma unroll
  for (int u = 0; u < C; u++) {
    const double sl = 0.5 * ((u < C - 1 ? a[u + 1] : ap) - (u ? a[u - 1] : am));
    double w = fabs(sl);
    const double t1 = 2.0 * fabs(d[u]), t2 = 2.0 * fabs(d[u + 1]);
    if (t1 < w) w = t1;
    if (t2 < w) w = t2;
    s[u] = d[u + 1] * d[u] <= 0.0 ? 0.0 : (sl < 0 ? -w : w);
  }
  const double sm = from_left(s[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++)
    e[u] = (u ? a[u - 1] : am) + 0.5 * d[u] - (1.0 / 6.0) * (s[u] - (u ? s[u - 1] : sm));
  e[C] = from_right(e[0], lane);
#pragma unroll
  for (int u = 0; u < C; u++) {
    double l = e[u], r = e[u + 1];
    if ((r - a[u]) * (a[u] - l) < 0.0) { l = a[u]; r = a[u]; }
    const double diff = r - l, cord = a[u] - 0.5 * (l + r), x = 6.0 * diff * cord;
    if (x > diff * diff) l = 3.0 * a[u] - 2.0 * r;
    if (-diff * diff > x) r = 3.0 * a[u] - 2.0 * l;
    L[u] = l;
    Rr[u] = r;
  }
  const double Lm = from_left(L[C - 1], lane), Rm = from_left(Rr[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++) {
    const bool up = R.v1[u] > 0.0;   // upwind: the cell below the face
    const double a0 = up ? (u ? a[u - 1] : am) : a[u];
    const double l = up ? (u ? L[u - 1] : Lm) : L[u], r = up ? (u ? Rr[u - 1] : Rm) : Rr[u];
    const double ed = up ? r : l;
    double x = ed + R.ks[u] * (a0 - ed);
    x += R.kk[u] * (2.0 * a0 - r - l);
    qs[u] = x;
  }
}

// ---- FP32: uniform zones; slopes in undivided differences, the PPA's edges
// as deviations from the cell (no cancellation), the update factor in the last
// fused product of each pass.  Algebraically the stages above.
template <int C>
struct XsRing32 {
  float h0[C];        // 0.5 (1 - cr) upwind below, -0.5 (1 + cr) above
  float f0[C];        // residual velocity
  bool up0[C];
  float ks;           // |v| dt / z of the rest velocity
};
template <int C>
__device__ __forceinline__ void xs_vl(const XsRing32<C> &R, const float *a, int lane, float *qs) {
  float dq[C + 1], s[C];
  const float am = from_left(a[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++) dq[u] = a[u] - (u ? a[u - 1] : am);
  dq[C] = from_right(dq[0], lane);
#pragma unroll
  for (int u = 0; u < C; u++) {
    const float p = dq[u] * dq[u + 1];
    s[u] = p <= 0.0f ? 0.0f : __fdividef(p + p, dq[u] + dq[u + 1]);
  }
  const float sm = from_left(s[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++) {
    const float al = u ? a[u - 1] : am, sl = u ? s[u - 1] : sm;
    qs[u] = fmaf(R.h0[u], R.up0[u] ? sl : s[u], R.up0[u] ? al : a[u]);
  }
}
// The rest velocity is one value per ring: each cell is upwind of one face,
// the one above it (UP) or below it.  g[u]: cell u's value at that face.
template <int C, bool UP>
__device__ __forceinline__ void xs_ppa32(float ks, const float *a, int lane, float *g) {
  float d[C + 1], s[C], t[C + 1];
  const float am = from_left(a[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++) d[u] = a[u] - (u ? a[u - 1] : am);
  d[C] = from_right(d[0], lane);
#pragma unroll
  for (int u = 0; u < C; u++) {   // the MC slope
    const float w = fminf(0.5f * fabsf(d[u] + d[u + 1]), 2.0f * fminf(fabsf(d[u]), fabsf(d[u + 1])));
    s[u] = d[u] * d[u + 1] <= 0.0f ? 0.0f : copysignf(w, d[u]);
  }
  const float sm = from_left(s[C - 1], lane);
#pragma unroll
  for (int u = 0; u < C; u++) t[u] = s[u] - (u ? s[u - 1] : sm);
  t[C] = from_right(t[0], lane);
  const float k1 = 1.0f - ks;
#pragma unroll
  for (int u = 0; u < C; u++) {
    // right edge - a and a - left edge; the parabola's limits (fargo_ppa_c):
    // opposite signs flatten, either deviation is at most twice the other
    const float dr = fmaf(-1.0f / 6.0f, t[u + 1], 0.5f * d[u + 1]), dl = fmaf(1.0f / 6.0f, t[u], 0.5f * d[u]);
    const float mr = fminf(fabsf(dr), 2.0f * fabsf(dl)), ml = fminf(fabsf(dl), 2.0f * fabsf(dr));
    const float w = UP ? k1 * fmaf(ks, ml - mr, mr) : k1 * fmaf(ks, mr - ml, ml);
    const float x = copysignf(w, UP ? dr : -dr);
    g[u] = dr * dl <= 0.0f ? a[u] : a[u] + x;
  }
}

// ---- staging ----------------------------------------------------------------
__device__ __forceinline__ void xs_bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ bool xs_wait(uint32_t bar, uint32_t parity, long long limit) {
  uint32_t done = 0;
  for (long long it = 0; it < limit && !done; it++)
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// this lane's C cells of a staged row, whose first cell sits sh elements in
template <typename T, int C>
__device__ __forceinline__ void xs_take(const T *row, int sh, int lane, T *a) {
  // one scalar load per cell: the lanes' cells are C apart, which costs the
  // shared memory C-way conflicts but no selects (the first cell's place in
  // its 16 bytes differs from ring to ring)
#pragma unroll
  for (int u = 0; u < C; u++) a[u] = row[sh + lane * C + u];
}

// One warp: strip `strip` of the rings [r0, r1) (ring = jlo + r % nj, klo + r / nj).
// NV: 2D, fused with NewVelocity / Stockholm; the ring before r0 is advected
// too, for its density and Mpy.  NQ: transported quantities besides rho.
template <typename T, int C, int NQ, bool NV>
__device__ __forceinline__ void b_sweep_xs(const Dims &m, const Geo<T> &g, const XsArgs<T> &A, int jlo, int klo, int nj,
                                           int strip, int r0, int r1, const fb_scalars *__restrict__ scp,
                                           unsigned long long *__restrict__ errflag, long long wait_limit) {
  using X = XS<C>;
  constexpr int E = XsRow<T, C>::E, LEN = XsRow<T, C>::LEN, NA = NQ + 2;
  extern __shared__ __align__(16) unsigned char xs_raw[];
  __shared__ __align__(8) unsigned long long xs_bar[XS_WARPS][2];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nx = m.nx;
  const bool whole = nx == X::N;
  T *stage = reinterpret_cast<T *>(xs_raw) + (size_t)w * 2 * NA * LEN;
  const int rf = NV ? r0 - 1 : r0;
  const int o0 = whole ? 0 : strip * X::W - X::HL;   // output column of the strip's first cell (unwrapped)
  auto array = [&](int a) -> const T * { return a == 0 ? A.rho : (a <= NQ ? A.q[a - 1] : A.vxt); };
  bool bulk = ((size_t)nx * sizeof(T)) % 16 == 0;
  {
    uintptr_t p = 0;
#pragma unroll
    for (int a = 0; a < NA; a++) p |= (uintptr_t)array(a);
    bulk = bulk && (p & 15) == 0;
  }
  auto ring_jk = [&](int r, int &j, int &k) {
    j = jlo + (NV ? r : r % nj);
    k = NV ? 0 : (m.is3d ? klo + r / nj : 0);
  };
  // the input column of ring r's first cell: output column - shift, mod nx
  auto first_col = [&](int r) {
    int j, k;
    ring_jk(r, j, k);
    int c = o0 - A.nshift[j + k * m.sy];
    while (c < 0) c += nx;
    return c;
  };
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(&xs_bar[w][0]);
  if (bulk) {
    if (lane == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
  }
  // copies of ring r's pieces into stage s, one array per lane: LEN cells
  // from the 16-byte boundary at or below the first column, around the ring's
  // end
  const T *mine = array(0);
#pragma unroll
  for (int a = 1; a < NA; a++) mine = lane == a ? array(a) : mine;
  auto issue = [&](int r, int s, int fc) {
    if (lane >= NA) return;
    int j, k, c = fc & ~(E - 1);
    ring_jk(r, j, k);
    const uint32_t bar = bar0 + 8 * s;
    if (lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                   ::"r"(bar), "r"((uint32_t)(NA * LEN * sizeof(T))) : "memory");
    const T *src = mine + m.l(0, j, k);
    uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage + (size_t)(s * NA + lane) * LEN);
    for (int left = LEN; left > 0;) {
      const int n = min(left, nx - c);
      xs_bulk(dst, src + c, (uint32_t)(n * sizeof(T)), bar);
      dst += (uint32_t)(n * sizeof(T));
      left -= n;
      c = 0;
    }
  };
  // the first columns of this ring and of the next are known a ring ahead
  int fc = first_col(rf), fc1 = rf + 1 < r1 ? first_col(rf + 1) : 0;
  if (bulk) issue(rf, 0, fc);
  const double dtd = scp->dt;
  const T dt = (T)dtd, of = (T)scp->omegaframe;
  const double idt = 1.0 / dtd;
  const T dof = sizeof(T) == 4 ? (T)(scp->omegaframe - scp->omegaframe0) : of - (T)scp->omegaframe0;
  // output column of this lane's first cell; lanes that write
  const int oc = o0 + lane * C;
  // which of this lane's cells the strip writes, two at a time: stores are
  // 2-cell words where rows are 16-byte aligned
  auto in_strip = [&](int u) -> bool {
    const int p = lane * C + u;
    return (whole || (p >= X::HL && p < X::HL + X::W)) && oc + u < nx;
  };
  auto put = [&](T *o, const T *x) {   // o: the row's place of column oc
    if (bulk && C % 2 == 0) {
#pragma unroll
      for (int u = 0; u < C; u += 2)
        if (in_strip(u)) {
          if constexpr (sizeof(T) == 8) reinterpret_cast<double2 *>(o + u)[0] = make_double2(x[u], x[u + 1]);
          else reinterpret_cast<float2 *>(o + u)[0] = make_float2(x[u], x[u + 1]);
        }
    } else {
#pragma unroll
      for (int u = 0; u < C; u++)
        if (in_strip(u)) o[u] = x[u];
    }
  };
  T r_m[C], py_m[C], sx_o[C], sxm_o = 0;   // NV: the row below; Sxi of the output columns
  if (NV && sizeof(T) == 8) {
#pragma unroll
    for (int u = 0; u < C; u++) {
      int c = (oc + u) % nx;
      sx_o[u] = ld(g.sxi + (c < 0 ? c + nx : c));
    }
    sxm_o = from_left(sx_o[C - 1], lane);
  }
#pragma unroll
  for (int u = 0; u < C; u++) { r_m[u] = py_m[u] = 0; }

  for (int r = rf; r < r1; r++) {
    const int s = (r - rf) & 1;
    const bool pre = NV && r < r0;
    int j, k;
    ring_jk(r, j, k);
    const int sh = fc & (E - 1);
    const int fc2 = r + 2 < r1 ? first_col(r + 2) : 0;
    if (bulk) {
      __syncwarp();   // every lane is done with the other stage
      if (r + 1 < r1) issue(r + 1, s ^ 1, fc1);
      // Bounded wait (wait_limit polls).  A warp that gives up flags the disk
      // (its next step reports it; a batch freezes it), waits again --
      // boundedly -- for its copies in flight, so that it does not leave while
      // the copy engine still writes its stage, and returns without writing.
      const bool ok = xs_wait(bar0 + 8 * s, ((r - rf) >> 1) & 1, wait_limit);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicOr(errflag, 2ull);
        xs_wait(bar0 + 8 * s, ((r - rf) >> 1) & 1, 1ll << 22);
        if (r + 1 < r1) xs_wait(bar0 + 8 * (s ^ 1), ((r + 1 - rf) >> 1) & 1, 1ll << 22);
        __syncwarp();
        return;
      }
    }
    int col[C];   // input columns of this lane's cells
    if (sizeof(T) == 8 || !bulk) {
      int c = fc + lane * C;
      while (c >= nx) c -= nx;
#pragma unroll
      for (int u = 0; u < C; u++) {
        col[u] = c;
        c = c + 1 < nx ? c + 1 : 0;
      }
    }
    const long long l0 = m.l(0, j, k);
    auto take = [&](int a, T *x) {
      if (bulk) {
        xs_take<T, C>(stage + (size_t)(s * NA + a) * LEN, sh, lane, x);
      } else {
        const T *row = array(a) + l0;
#pragma unroll
        for (int u = 0; u < C; u++) x[u] = row[col[u]];
      }
    };
    T vt[C], rho[C];
    take(NA - 1, vt);
    take(0, rho);
    T out_r[C], outq[NQ][C];
    if constexpr (sizeof(T) == 8) {
      XsRing64<C> R;
      const double vm = A.vxmed_t[j + k * m.sy], vmdt = vm * dtd;
      R.s1 = ld(g.sxj + j); R.s2 = ld(g.sxk + k); R.s3 = dt; R.s4 = ld(g.invvj + j);
      R.flat = !m.is3d;
      const double ym = ld(g.ymed + j), st = m.sph ? ld(g.sin_zmed + k) : 1.0, syk = ld(g.syk + k);
#pragma unroll
      for (int u = 0; u < C; u++) {
        const double sx = ld(g.sxi + col[u]);
        R.z[u] = m.sph ? sx * ym * st : sx * ym;
        R.iz[u] = 1.0 / R.z[u];
        R.iu_d[u] = syk * sx;
        R.iu[u] = 1.0 / R.iu_d[u];
      }
      const double zm = from_left(R.z[C - 1], lane);
#pragma unroll
      for (int u = 0; u < C; u++) {
        R.v0[u] = vt[u] - vm;   // residual
        R.h0[u] = R.v0[u] > 0.0 ? 0.5 * ((u ? R.z[u - 1] : zm) - R.v0[u] * dt) : 0.5 * (R.z[u] + R.v0[u] * dt);
        const double nt = divk(vmdt, R.z[u], R.iz[u]), nr = floor(nt + 0.5);   // compute_residual.c:68-73
        R.v1[u] = divk((nt - nr) * R.z[u], dtd, idt);
        R.ks[u] = divk(fabs(R.v1[u]) * dt, R.z[u], R.iz[u]);
        R.kk[u] = R.ks[u] * (1.0 - R.ks[u]);
      }
      double rs0[C], rs1[C], rho1[C], ir0[C], ir1[C], fl[C + 1];
      xs_vl<C>(R, rho, lane, rs0);
#pragma unroll
      for (int u = 0; u < C; u++) fl[u] = R.v0[u] * rs0[u];
      fl[C] = from_right(fl[0], lane);
#pragma unroll
      for (int u = 0; u < C; u++) {
        rho1[u] = rho[u] + xs_upd<C>(R, fl[u] - fl[u + 1], u);
        ir0[u] = 1.0 / rho[u];
        ir1[u] = 1.0 / rho1[u];
      }
      xs_ppa<C>(R, rho1, lane, rs1);
#pragma unroll
      for (int u = 0; u < C; u++) fl[u] = R.v1[u] * rs1[u];
      fl[C] = from_right(fl[0], lane);
#pragma unroll
      for (int u = 0; u < C; u++) out_r[u] = rho1[u] + xs_upd<C>(R, fl[u] - fl[u + 1], u);
#pragma unroll (NV ? NQ : 1)
      for (int q = 0; q < NQ; q++) {
        if (pre && q != 2) continue;
        double x[C], a[C], qs[C];
        take(1 + q, x);
#pragma unroll
        for (int u = 0; u < C; u++) a[u] = divk(x[u], rho[u], ir0[u]);   // DivideByRho
        xs_vl<C>(R, a, lane, qs);
#pragma unroll
        for (int u = 0; u < C; u++) fl[u] = R.v0[u] * qs[u] * rs0[u];
        fl[C] = from_right(fl[0], lane);
#pragma unroll
        for (int u = 0; u < C; u++) {
          x[u] = x[u] + xs_upd<C>(R, fl[u] - fl[u + 1], u);
          a[u] = divk(x[u], rho1[u], ir1[u]);
        }
        xs_ppa<C>(R, a, lane, qs);
#pragma unroll
        for (int u = 0; u < C; u++) fl[u] = R.v1[u] * qs[u] * rs1[u];
        fl[C] = from_right(fl[0], lane);
#pragma unroll
        for (int u = 0; u < C; u++) x[u] = x[u] + xs_upd<C>(R, fl[u] - fl[u + 1], u);
        if constexpr (NV) {
#pragma unroll
          for (int u = 0; u < C; u++) outq[q][u] = x[u];
        } else {
          put(A.o[q] + l0 + oc, x);
        }
      }
    } else {
      XsRing32<C> R;
      const float4 rx = A.ringx[j + k * m.sy];
      const float upd = rx.w;
      const bool up = rx.y > 0.0f;
      R.ks = fabsf(rx.y) * rx.z;
      const float f1 = rx.y;
#pragma unroll
      for (int u = 0; u < C; u++) {
        const float v = vt[u] - rx.x, cr = v * rx.z;
        R.up0[u] = v > 0.0f;
        R.h0[u] = R.up0[u] ? 0.5f * (1.0f - cr) : -0.5f * (1.0f + cr);
        R.f0[u] = v;
      }
      // van Leer pass and rest pass of one quantity: x += upd times the flux
      // differences; the flux of rho is f0 / f1 times its face value, of a
      // momentum the density's flux times its own
      auto faces1 = [&](const float *a, float *fl) {   // PPA values at the C + 1 faces
        float gq[C];
        if (up) {
          xs_ppa32<C, true>(R.ks, a, lane, gq);
          fl[0] = from_left(gq[C - 1], lane);
#pragma unroll
          for (int u = 0; u < C; u++) fl[u + 1] = gq[u];
        } else {
          xs_ppa32<C, false>(R.ks, a, lane, gq);
#pragma unroll
          for (int u = 0; u < C; u++) fl[u] = gq[u];
          fl[C] = from_right(gq[0], lane);
        }
      };
      float qs[C], fl[C + 1], m0[C], m1[C + 1], rho1[C], ir0[C], ir1[C];
      xs_vl<C>(R, rho, lane, qs);
#pragma unroll
      for (int u = 0; u < C; u++) m0[u] = R.f0[u] * qs[u];
      fl[C] = from_right(m0[0], lane);
#pragma unroll
      for (int u = 0; u < C; u++) {
        rho1[u] = fmaf(m0[u] - (u < C - 1 ? m0[u + 1] : fl[C]), upd, rho[u]);
        ir0[u] = __fdividef(1.0f, rho[u]);
        ir1[u] = __fdividef(1.0f, rho1[u]);
      }
      faces1(rho1, m1);
#pragma unroll
      for (int u = 0; u <= C; u++) m1[u] *= f1;
#pragma unroll
      for (int u = 0; u < C; u++) out_r[u] = fmaf(m1[u] - m1[u + 1], upd, rho1[u]);
#pragma unroll (NV ? NQ : 1)
      for (int q = 0; q < NQ; q++) {
        if (pre && q != 2) continue;
        float x[C], a[C];
        take(1 + q, x);
#pragma unroll
        for (int u = 0; u < C; u++) a[u] = x[u] * ir0[u];   // DivideByRho
        xs_vl<C>(R, a, lane, qs);
#pragma unroll
        for (int u = 0; u < C; u++) fl[u] = m0[u] * qs[u];
        fl[C] = from_right(fl[0], lane);
#pragma unroll
        for (int u = 0; u < C; u++) {
          x[u] = fmaf(fl[u] - fl[u + 1], upd, x[u]);
          a[u] = x[u] * ir1[u];
        }
        faces1(a, fl);
#pragma unroll
        for (int u = 0; u <= C; u++) fl[u] *= m1[u];
#pragma unroll
        for (int u = 0; u < C; u++) x[u] = fmaf(fl[u] - fl[u + 1], upd, x[u]);
        if constexpr (NV) {
#pragma unroll
          for (int u = 0; u < C; u++) outq[q][u] = x[u];
        } else {
          put(A.o[q] + l0 + oc, x);
        }
      }
    }
    if constexpr (!NV) {
      put(A.o_rho + l0 + oc, out_r);
    } else {
      if (!pre) {
        // NewVelocity_x/y (newvel_x.c:81, newvel_y.c:70) of row j
        const T rxm = from_left(out_r[C - 1], lane), pxm = from_left(outq[0][C - 1], lane);
        const T ivj = ld(g.invvj + j), ivjm = ld(g.invvj + j - 1), rc = ld(g.ymed + j);
        T nr[C], nvx[C], nvy[C];
        if constexpr (sizeof(T) == 8) {
          const double iv = 1.0 / ivj, ivm = 1.0 / ivjm, syk = ld(g.syk + k);
          double vl[C];   // r syk sxi / ivj of this row's cells
#pragma unroll
          for (int u = 0; u < C; u++) vl[u] = divk(out_r[u] * syk * sx_o[u], ivj, iv);
          const double vlm = from_left(vl[C - 1], lane);
#pragma unroll
          for (int u = 0; u < C; u++) {
            const double px = u ? outq[0][u - 1] : pxm, sxm = u ? sx_o[u - 1] : sxm_o;
            double x = (divk(outq[1][u] * syk * sx_o[u], ivj, iv) + divk(px * syk * sxm, ivj, iv)) /
                       ((vl[u] + (u ? vl[u - 1] : vlm)) * rc);
            x -= of * rc;
            nvx[u] = x;
            nvy[u] = (divk(outq[3][u] * syk * sx_o[u], ivj, iv) + divk(py_m[u] * syk * sx_o[u], ivjm, ivm)) /
                     (vl[u] + divk(r_m[u] * syk * sx_o[u], ivjm, ivm));
            nr[u] = out_r[u];
          }
        } else {
          // the factors common to numerator and denominator cancelled; the
          // azimuthal momenta are relative to the frame and the background
#pragma unroll
          for (int u = 0; u < C; u++) {
            nvx[u] = div_rn(outq[1][u] + (u ? outq[0][u - 1] : pxm), (out_r[u] + (u ? out_r[u - 1] : rxm)) * rc);
            nvy[u] = div_rn(outq[3][u] * ivjm + py_m[u] * ivj, out_r[u] * ivjm + r_m[u] * ivj);
            nr[u] = out_r[u];
          }
        }
        if (A.stockholm) {   // stockholm.c:129-185
          const T ramp = (T)A.ramps[j];
          if (ramp > (T)0.0) {
            const T taud = ld(g.tau_j + j) / ramp, den = dt + taud;
            T vx0t = A.vx0[j];
            vx0t -= dof * rc;
#pragma unroll
            for (int u = 0; u < C; u++) {
              nr[u] = (nr[u] * taud + A.rho0[j] * dt) / den;
              nvx[u] = (nvx[u] * taud + vx0t * dt) / den;
              nvy[u] = (nvy[u] * taud + A.vy0[j] * dt) / den;
            }
          }
        }
        const long long l = l0 + oc;
        put(A.s_rho + l, nr);
        put(A.s_vx + l, nvx);
        // the transported energy (stockholm.c leaves it alone)
        if (NQ == 5 && A.s_e) put(A.s_e + l, outq[NQ - 1]);
        if (edge_row(m, j)) {
#pragma unroll
          for (int u = 0; u < C; u++)
            if (in_strip(u))
              ghosts_of_row<T>(m, A.ymed, A.tab, A.vbg, scp->omegaframe, oc + u, j, A.s_rho, A.s_vx, A.s_vy,
                               NQ == 5 ? A.s_e : (T *)nullptr, nr[u], nvx[u], nvy[u], NQ == 5 ? outq[NQ - 1][u] : (T)0);
          if (j == FB_NGH && m.bclo) {
#pragma unroll
            for (int u = 0; u < C; u++) nvy[u] = 0;
          }
        }
        put(A.s_vy + l, nvy);
      }
#pragma unroll
      for (int u = 0; u < C; u++) {
        r_m[u] = out_r[u];
        py_m[u] = outq[2][u];
      }
    }
    fc = fc1;
    fc1 = fc2;
  }
}

// rings a warp marches over: enough warps to fill the chip twice over
// (148 SMs x 16 resident warps) before longer marches, which save the fused
// sweep the extra ring per march (2 of its 5 quantities) and the pipeline's
// first load
__host__ __device__ inline int xs_rows(long long strip_rings) {
  const long long r = strip_rings / (148 * 16 * 2);
  return r < 1 ? 1 : (r > 8 ? 8 : (int)r);
}
__host__ __device__ inline int xs_ctas(int strips, int rings, int rows) {
  return (strips * ((rings + rows - 1) / rows) + XS_WARPS - 1) / XS_WARPS;
}

template <typename T>
__host__ __device__ inline XsArgs<T> xs_args(const fb_disk_dev &D, const fb_fluid_dev &F) {
  XsArgs<T> a;
  const bool b = D.is3d;
  a.rho = (const T *)(b ? F.rho_b : F.rho_a);
  a.vxt = (const T *)F.vxt;
  const void *in[6] = {b ? F.mpx_b : F.mpx, b ? F.mmx_b : F.mmx, b ? F.mpy_b : F.mpy,
                       b ? F.mmy_b : F.mmy, b ? F.mpz_b : F.e_a, F.mmz_b};
  // 3D: back into set A, which the Y sweep has consumed
  void *out[6] = {F.mpx, F.mmx, F.mpy, F.mmy, F.mpz, F.mmz};
  for (int q = 0; q < 6; q++) { a.q[q] = (const T *)in[q]; a.o[q] = (T *)out[q]; }
  a.o_rho = (T *)F.rho_a;
  a.s_rho = (T *)F.rho; a.s_vx = (T *)F.vx; a.s_vy = (T *)F.vy;
  a.s_e = D.adiabatic ? (T *)F.cs : nullptr;
  a.rho0 = (const T *)F.rho0; a.vx0 = (const T *)F.vx0; a.vy0 = (const T *)F.vy0;
  a.ramps = D.ramps;
  a.tab = D.bnd_tab; a.vbg = F.vbg; a.ymed = (const double *)D.geomd.ymed;
  a.stockholm = D.stockholm;
  a.vxmed_t = F.vxmed_t;
  a.nshift = F.nshift;
  a.ringx = (const float4 *)F.ringx;
  return a;
}
// rings of the sweep: 2D (fused) the active rows, the row below the first
// being advected too; 3D rows Nghy-1 .. of layers Nghz-1 ..
__host__ __device__ inline int xs_rings(const fb_disk_dev &D) { return D.is3d ? (D.ny + 1) * (D.nz + 1) : D.ny; }

// CTA bx of a disk: its warps take strip wid % strips of `rows` rings each,
// segment wid / strips of them, wid = XS_WARPS bx + warp
template <typename T, int NQ, bool NV>
__device__ __forceinline__ void xs_cta(const Dims &m, const Geo<T> &g, const XsArgs<T> &A,
                                       const fb_scalars *__restrict__ scp, unsigned long long *__restrict__ errflag,
                                       long long wait_limit, int bx, int rows) {
  constexpr int C = XsC<T>::C;
  const int strips = xs_strips<C>(m.nx), wid = bx * XS_WARPS + (threadIdx.x >> 5);
  const int rings = m.is3d ? (m.ny + 1) * (m.nz + 1) : m.ny, seg = wid / strips, strip = wid - seg * strips;
  const int first = NV ? 1 : 0;   // NV: ring 0 is the ghost row below the active ones
  const int r0 = first + seg * rows, r1 = min(r0 + rows, first + rings);
  if (r0 >= r1) return;
  b_sweep_xs<T, C, NQ, NV>(m, g, A, FB_NGH - 1, FB_NGH - 1, m.ny + 1, strip, r0, r1, scp, errflag, wait_limit);
}
// resident CTAs of 128 threads the sweep is compiled for
#ifndef FB_XS64_MINB
#define FB_XS64_MINB 4
#endif
#ifndef FB_XS32_MINB
#define FB_XS32_MINB 5
#endif
template <typename T, int NQ, bool NV>
__global__ void __launch_bounds__(32 * XS_WARPS, sizeof(T) == 8 ? FB_XS64_MINB : FB_XS32_MINB)
    k_sweep_xs(const __grid_constant__ fb_disk_dev D, int rows) {
  xs_cta<T, NQ, NV>(dims_of(D), geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), xs_args<T>(D, D.fl[blockIdx.y]),
                    D.scal_dev, (unsigned long long *)D.dtmin + 1, wait_limit(D), blockIdx.x, rows);
}

}  // namespace fb
