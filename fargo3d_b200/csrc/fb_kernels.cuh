// fb_kernels.cuh -- the hydro-step kernels, templated on the field precision.
//
// Stage kernels of one hydro step (FARGO3D main.c:361-448):
//   rowsum      ring sums of v_phi * dphi (ComputeVmed, compute_vmed.c:10-39)
//   cfl         per-cell time step, CFL minimum and shear limit (cfl.c, cfl_b.c)
//   sources     pressure, potential, SubStep1, viscous stress, SubStep2 fused in a
//               shared-memory tile (algogas.c:30-120); 3D: fb_sources3.cuh, FP32 2D:
//               fb_sources32.cuh
//   bnd         ghost rows / layers (generated boundaries, algogas.c:11-27) where the
//               stage before does not fill them
//   sweep_z/y   conservative upwind van Leer transport along a column, one thread
//               per column marching in its direction (transport.c:24-46, 84-127;
//               fb_sweepcol.cuh)
//   sweep_x     a warp per strip of a ring: FARGO residual, van Leer, PPA and integer
//               shift in registers, 2D with the new velocities (transport.c:129-158;
//               fb_sweepx.cuh)
//   newvel      3D: new velocities and Stockholm damping (newvel_*.c, stockholm.c)
//
// Floating-point expressions follow the reference's evaluation order exactly
// (including the order implied by its geometry macros), so the FP64
// instantiation, compiled without FMA contraction, reproduces the CPU build.
#pragma once
#include <type_traits>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "fb_dev.h"

#define FB_CVNR 1.41
#define FB_NGH 3

namespace fb {

template <typename T>
struct Geo {
  const T *xmin, *ymin, *zmin, *xmed, *ymed, *zmed, *invdiffxmed;
  const T *sxi, *sxj, *syj, *szj, *sxk, *syk, *szk, *invvj;
  const T *sin_zmed, *cos_zmed, *sin_zmin, *cos_zmin;
  const T *cos_xmed, *sin_xmed;
  const T *visc_j, *viscm_j, *tau_j;
  const T *r2_j, *dr2_j, *s2_k, *ds2_k;
  const T *inv_ymed, *inv_ymin, *inv_dymed, *pot_star;
};

template <typename T>
__host__ __device__ inline Geo<T> geo_of(const fb_geom_dev &g) {
  Geo<T> o;
  o.xmin = (const T *)g.xmin; o.ymin = (const T *)g.ymin; o.zmin = (const T *)g.zmin;
  o.xmed = (const T *)g.xmed; o.ymed = (const T *)g.ymed; o.zmed = (const T *)g.zmed;
  o.invdiffxmed = (const T *)g.invdiffxmed; o.sxi = (const T *)g.sxi;
  o.sxj = (const T *)g.sxj; o.syj = (const T *)g.syj; o.szj = (const T *)g.szj;
  o.sxk = (const T *)g.sxk; o.syk = (const T *)g.syk; o.szk = (const T *)g.szk;
  o.invvj = (const T *)g.invvj;
  o.sin_zmed = (const T *)g.sin_zmed; o.cos_zmed = (const T *)g.cos_zmed;
  o.sin_zmin = (const T *)g.sin_zmin; o.cos_zmin = (const T *)g.cos_zmin;
  o.cos_xmed = (const T *)g.cos_xmed; o.sin_xmed = (const T *)g.sin_xmed;
  o.visc_j = (const T *)g.visc_j; o.viscm_j = (const T *)g.viscm_j; o.tau_j = (const T *)g.tau_j;
  o.r2_j = (const T *)g.r2_j; o.dr2_j = (const T *)g.dr2_j; o.s2_k = (const T *)g.s2_k; o.ds2_k = (const T *)g.ds2_k;
  o.inv_ymed = (const T *)g.inv_ymed; o.inv_ymin = (const T *)g.inv_ymin; o.inv_dymed = (const T *)g.inv_dymed;
  o.pot_star = (const T *)g.pot_star;
  return o;
}

template <typename T>
__device__ __forceinline__ T ld(const T *p) { return __ldg(p); }

struct Dims {
  int nx, ny, nz, sy, sz, pitch;
  long long stride;
  int is3d, sph, alpha;
  int adiab;        // ADIABATIC: the cs field holds the internal energy e
  double gam;       // GAMMA
  int bclo, bchi;   // the radial edges are the mesh's own (boundary templates) or a slab's
  __device__ __forceinline__ long long l(int i, int j, int k) const {
    return (long long)i + (long long)j * pitch + (long long)k * stride;
  }
};

__host__ __device__ inline Dims dims_of(const fb_disk_dev &d) {
  Dims m;
  m.nx = d.nx; m.ny = d.ny; m.nz = d.nz; m.sy = d.sy; m.sz = d.sz; m.pitch = d.pitch;
  m.stride = d.stride; m.is3d = d.is3d; m.sph = d.spherical; m.alpha = d.alpha_visc;
  m.adiab = d.adiabatic; m.gam = d.gamma;
  m.bclo = d.bc_lo; m.bchi = d.bc_hi;
  return m;
}

__device__ __forceinline__ int wrapx(int i, int nx) { return i < 0 ? i + nx : (i >= nx ? i - nx : i); }

// x / y given z = RN(1 / y): Markstein's product and two fused steps.  With z
// the correctly rounded reciprocal the result is RN(x / y) for every x and y
// whose quotient and remainder stay in the normal range (|x| above 2^-969):
// the first product is within 1.5 ulp, the remainder after it is exact where
// the quotient is near a rounding boundary, and a quotient of two 53-bit
// numbers keeps 2^-106 / y from every boundary.  3 FP64 issue slots against
// 12.6 for '/' (measured), so divisors shared by several numerators (zone
// sizes, the density under the momenta) are inverted once.
__device__ __forceinline__ double divk(double x, double y, double z) {
  const double q = x * z;
  return __fma_rn(__fma_rn(-y, q, x), z, q);
}

// RN(n / d): a Newton step on the approximate reciprocal gives RN(1 / d) (on
// sm_100a for every mantissa, from exponent -110 to 110; test_gpu_div.py), and
// with that the product and one residual step round as the division does
// (Markstein), as long as quotient and remainder stay in the normal range.
// NewVelocity divides by it: an error to one side would add up in a cell from
// step to step.  64 disks' azimuthal sweep 208 us with the approximate
// reciprocal alone (not always rounded so), 212 with the step, 215 with
// __fdiv_rn; a 512x256x48 step 1102, 1102, 1117.
__device__ __forceinline__ float recip_rn(float d) {
  const float z = __fdividef(1.0f, d);
  return fmaf(fmaf(-d, z, 1.0f), z, z);
}
__device__ __forceinline__ float div_rn(float n, float d) {
  const float z = recip_rn(d), q = n * z;
  return fmaf(fmaf(-d, q, n), z, q);
}

template <typename T>
__device__ __forceinline__ T zsx(const Dims &m, const Geo<T> &g, int i, int j, int k) {
  // zone_size_x (define.h:262-273)
  if (m.sph) return (ld(g.sxi + i) * ld(g.ymed + j) * ld(g.sin_zmed + k));
  return (ld(g.sxi + i) * ld(g.ymed + j));
}

// The ring's integer shift modulo the ring (compute_residual.c:68-73 at cell
// 0, advect_shift.c:49-54) and, for FP32 rings (uniform azimuthal spacing), the
// sweep's scalars: the mean less the background, the uniform rest velocity,
// dt / zone size and the update factor dt Surf / Vol, all formed in FP64.
__device__ __forceinline__ void ring_shift(const Dims &m, const Geo<double> &gd, double dt, double vm, double vb,
                                           int ring, int *__restrict__ nshift, float4 *__restrict__ ringx) {
  const int j = ring % m.sy, k = ring / m.sy;
  const double zx = zsx(m, gd, 0, j, k);
  const double nt = vm * dt / zx, nr = floor(nt + 0.5);
  const int ns = (int)nr % m.nx;
  nshift[ring] = ns < 0 ? ns + m.nx : ns;
  if (ringx)
    ringx[ring] = make_float4((float)(vm - vb), (float)((nt - nr) * zx / dt), (float)(dt / zx),
                              (float)(ld(gd.sxj + j) * ld(gd.sxk + k) * dt * ld(gd.invvj + j) /
                                      (ld(gd.syk + k) * ld(gd.sxi + 0))));
}

// in-order sum of n shared doubles onto acc, loads ahead of the additions
__device__ __forceinline__ double add_in_order(double acc, const double *v, int n) {
  int e = 0;
  for (; e + 16 <= n; e += 16) {
    double t[16];
#pragma unroll
    for (int u = 0; u < 16; u++) t[u] = v[e + u];
#pragma unroll
    for (int u = 0; u < 16; u++) acc = acc + t[u];
  }
  for (; e < n; e++) acc = acc + v[e];
  return acc;
}

// ---------------------------------------------------------------------------
// Ordered ring sums (ComputeVweight + reduction_SUM, compute_vmed.c:42-97,
// reduction_generic.c:5-23): vmed[j,k] = (sum_i v[i] * (xmin[i+1]-xmin[i])) /
// (XMAX - XMIN), accumulated sequentially in i as the reference does.
// A warp owns R rings: its lanes load and weight a chunk of each, a chunk
// ahead, into the warp's shared memory, and lane r adds ring r's chunk in
// order -- a chain of nx additions, 8.7 cycles each, which bounds the kernel.
// R = 1 where the rings are few (2D: a warp per ring spreads them over the
// chip), 8 where they are many (3D), so that one addition issues for 8 rings.
constexpr int RS_WARPS = 4;
template <int R>
__device__ __forceinline__ void b_rowsum(const Dims &m, const Geo<double> &gd, const double *__restrict__ v,
                                         double *__restrict__ out, double xlen, int blk,
                                         const fb_scalars *__restrict__ sc, int *__restrict__ nshift) {
  constexpr int CH = R == 1 ? 256 : 64, PL = CH / 32;   // cells of a chunk, per lane
  __shared__ double buf[RS_WARPS][R][CH + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nring = m.sy * m.sz, r0 = (blk * RS_WARPS + w) * R;
  if (r0 >= nring) return;
  double val[R][PL], acc = 0.0;
  auto fetch = [&](int c0) {
#pragma unroll
    for (int rr = 0; rr < R; rr++) {
      const int ring = min(r0 + rr, nring - 1), j = ring % m.sy, k = ring / m.sy;
      const double *row = v + m.l(0, j, k);
#pragma unroll
      for (int u = 0; u < PL; u++) {
        const int i = min(c0 + u * 32 + lane, m.nx - 1);
        val[rr][u] = row[i];
      }
    }
  };
  fetch(0);
  for (int c0 = 0; c0 < m.nx; c0 += CH) {
    const int cw = min(CH, m.nx - c0);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < PL; u++) {
      const int i = min(c0 + u * 32 + lane, m.nx - 1);
      const double dx = ld(gd.xmin + i + 1) - ld(gd.xmin + i);
#pragma unroll
      for (int rr = 0; rr < R; rr++) buf[w][rr][u * 32 + lane] = val[rr][u] * dx;
    }
    __syncwarp();
    if (c0 + CH < m.nx) fetch(c0 + CH);
    if (lane < R) acc = add_in_order(acc, buf[w][lane], cw);
  }
  if (lane < R && r0 + lane < nring) {
    out[r0 + lane] = acc / xlen;
    if (nshift) ring_shift(m, gd, sc->dt, acc / xlen, 0.0, r0 + lane, nshift, nullptr);
  }
}
// rings per warp, and the CTAs of a disk
__host__ __device__ inline int rs_rings(int nring) { return nring < 148 * 32 ? 1 : 8; }
__host__ __device__ inline int rs_ctas(int nring) {
  const int per = RS_WARPS * rs_rings(nring);
  return (nring + per - 1) / per;
}
// Order-free ring sums (FP32 storage): a warp owns RW_R rings, lanes striding
// over all of them at once with FP64 accumulators, then a shuffle tree each,
// and lane r finishes ring r: the divisions of the mean and of the azimuthal
// sweep's shift (a chain of some 600 cycles) run for RW_R rings side by side.
// vbg: the ring's background azimuthal velocity (FP32 disks store v - vbg),
// added back so the mean is that of the full velocity.
constexpr int RW_R = 4, RW_WARPS = 8;
template <typename S>
__device__ __forceinline__ void b_rowsum_warp(const Dims &m, const Geo<double> &gd, const S *__restrict__ v,
                                              double *__restrict__ out, double xlen, const double *__restrict__ vbg,
                                              int blk, const fb_scalars *__restrict__ sc, int *__restrict__ nshift,
                                              float4 *__restrict__ ringx) {
  const int lane = threadIdx.x & 31, r0 = (blk * RW_WARPS + (threadIdx.x >> 5)) * RW_R, nring = m.sy * m.sz;
  if (r0 >= nring) return;
  double acc[RW_R];
  const S *row[RW_R];
#pragma unroll
  for (int r = 0; r < RW_R; r++) {
    const int ring = min(r0 + r, nring - 1), j = ring % m.sy, k = ring / m.sy;
    row[r] = v + m.l(0, j, k);
    acc[r] = 0.0;
  }
  // rings of a multiple of 4 cells: float4 loads, the uniform azimuthal
  // spacing factored out of the sum
  const bool quad = sizeof(S) == 4 && (m.nx & 3) == 0 && (((uintptr_t)v) & 15) == 0;
  if (quad) {
    for (int q = lane; q < (m.nx >> 2); q += 32) {
      float4 x[RW_R];
#pragma unroll
      for (int r = 0; r < RW_R; r++) x[r] = reinterpret_cast<const float4 *>(row[r])[q];
#pragma unroll
      for (int r = 0; r < RW_R; r++) acc[r] += ((double)x[r].x + (double)x[r].y) + ((double)x[r].z + (double)x[r].w);
    }
  } else {
    for (int i = lane; i < m.nx; i += 32) {
      const double dx = ld(gd.xmin + i + 1) - ld(gd.xmin + i);
#pragma unroll
      for (int r = 0; r < RW_R; r++) acc[r] += (double)row[r][i] * dx;
    }
  }
  double mine = 0.0;
#pragma unroll
  for (int r = 0; r < RW_R; r++) {
    for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
    if (lane == r) mine = acc[r];
  }
  const int ring = r0 + lane;
  if (lane < RW_R && ring < nring) {
    if (quad) mine *= ld(gd.xmin + 1) - ld(gd.xmin + 0);
    const double vb = vbg ? vbg[ring] : 0.0, mean = mine / xlen + vb;
    out[ring] = mean;
    if (nshift) ring_shift(m, gd, sc->dt, mean, vb, ring, nshift, ringx);
  }
}
__host__ __device__ inline int rw_ctas(int nring) { return (nring + RW_WARPS * RW_R - 1) / (RW_WARPS * RW_R); }

// The background of an FP32 fluid at ring (j, k) (0 without one).
__device__ __forceinline__ double bg_at(const double *__restrict__ vbg, int ring) {
  return vbg ? vbg[ring] : 0.0;
}

// The host's part of a one-disk step reaches the device without copies of its
// own: the first kernel's first CTA reads the scalars, the CFL minimum's
// start value and the disk force's points from the disk's page-locked slot
// while the others sum rings, and the last CFL CTA to finish writes the
// minimum, the flags and the accelerations back to it, then the sequence
// number the host waits for.  (Four copies a step cost about 2 us of the
// device and as much of the host each.)
__device__ __forceinline__ void begin_upload(const fb_disk_dev &D) {
  if (blockIdx.x != 0 || blockIdx.y != 0) return;
  constexpr int NS = sizeof(fb_scalars) / 8;
  const double *h = D.pin + PIN_BEGIN / 8;
  double *dst = reinterpret_cast<double *>(D.scal_dev);
  for (int w = threadIdx.x; w < NS; w += blockDim.x) dst[w] = __ldcv(h + w);
  if (threadIdx.x == 32) {
    D.dtmin[0] = __ldcv(h + NS);
    D.dtmin[3] = __ldcv(h + NS + 1);
  }
  if (D.feeldisk)
    for (int w = threadIdx.x; w < 4 * FB_MAXPLANETS; w += blockDim.x) D.pts[w] = __ldcv(D.pin + PIN_PTS / 8 + w);
}
__device__ __forceinline__ void cfl_report(const fb_disk_dev &D) {
  if (threadIdx.x != 0) return;   // the thread that folded the CTA's minimum, after the CTA's barrier
  unsigned long long *dm = reinterpret_cast<unsigned long long *>(D.dtmin);
  __threadfence();
  const unsigned long long n = (unsigned long long)gridDim.x * gridDim.y * gridDim.z;
  if (atomicAdd(dm + 2, 1ull) != n - 1) return;
  __threadfence();
  dm[2] = 0ull;
  volatile double *h = D.pin;
  const volatile double *d = D.dtmin;
  h[0] = d[0];
  h[1] = d[1];
  if (D.feeldisk)
    for (int w = 0; w < 3 * FB_MAXPLANETS; w++) h[8 + w] = D.facc[w];
  __threadfence_system();
  h[2] = d[3];
}

// One-disk kernels take the disk's descriptor and all its fluids in one
// launch: the slowest grid index counts the fluids, which share no data
// within a stage.
template <typename S>
__global__ void __launch_bounds__(32 * RW_WARPS) k_rowsum_warp(const __grid_constant__ fb_disk_dev D, int which) {
  if (which == 0) begin_upload(D);
  const fb_fluid_dev &F = D.fl[blockIdx.y];
  b_rowsum_warp<S>(dims_of(D), geo_of<double>(D.geomd), (const S *)(which ? F.vxt : F.vx), which ? F.vxmed_t : F.vxmed,
                   D.xlen, F.vbg, blockIdx.x, D.scal_dev, which ? F.nshift : nullptr, (float4 *)F.ringx);
}

static __global__ void __launch_bounds__(32 * RS_WARPS) k_rowsum(const __grid_constant__ fb_disk_dev D, int which) {
  if (which == 0) begin_upload(D);
  const fb_fluid_dev &F = D.fl[blockIdx.y];
  const Dims m = dims_of(D);
  const double *v = (const double *)(which ? F.vxt : F.vx);
  double *out = which ? F.vxmed_t : F.vxmed;
  int *ns = which ? F.nshift : nullptr;
  if (rs_rings(m.sy * m.sz) == 1) b_rowsum<1>(m, geo_of<double>(D.geomd), v, out, D.xlen, blockIdx.x, D.scal_dev, ns);
  else b_rowsum<8>(m, geo_of<double>(D.geomd), v, out, D.xlen, blockIdx.x, D.scal_dev, ns);
}

// ---------------------------------------------------------------------------
// CFL (cfl.c:135-258) and cfl_b's shear limit (cfl_b.c:14-39).  One CTA per
// active ring; the ring minimum (including its shear limit) is folded into a
// device-wide minimum held as the bit pattern of a positive double.
__device__ __forceinline__ double dmax2(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double dmax3(double a, double b, double c) {
  return (((a) > (b) ? (a) : (b)) > (c) ? ((a) > (b) ? (a) : (b)) : (c));
}
__device__ __forceinline__ float dmax2(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float dmax3(float a, float b, float c) {
  return (((a) > (b) ? (a) : (b)) > (c) ? ((a) > (b) ? (a) : (b)) : (c));
}

template <typename T>
__device__ __forceinline__ T zsy(const Geo<T> &g, int j) { return (ld(g.ymin + j + 1) - ld(g.ymin + j)); }
template <typename T>
__device__ __forceinline__ T zsz(const Dims &m, const Geo<T> &g, int j, int k) {
  if (m.sph) return ((ld(g.zmin + k + 1) - ld(g.zmin + k)) * ld(g.ymed + j));
  return (ld(g.zmin + k + 1) - ld(g.zmin + k));
}

// The radial and colatitude zone sizes of a ring and their reciprocals.
template <typename T>
struct CflRing { T y, iy, z, iz; };
template <typename T>
__device__ __forceinline__ CflRing<T> cfl_zones(const Dims &m, const Geo<T> &g, int j, int k) {
  CflRing<T> z;
  z.y = zsy(g, j);
  z.iy = (T)1.0 / z.y;
  z.z = m.is3d ? zsz(m, g, j, k) : (T)1;
  z.iz = (T)1.0 / z.z;
  return z;
}

// A cell's inputs, loaded apart from the work on them so that the loads of
// several cells, and of the ring's zones, are under way together.
template <typename S>
struct CflIn { S r, c, v, vp, y, yp, z, zp; };
template <typename S>
__device__ __forceinline__ CflIn<S> cfl_load(const Dims &m, const S *__restrict__ rho, const S *__restrict__ cs,
                                             const S *__restrict__ vx, const S *__restrict__ vy,
                                             const S *__restrict__ vz, int i, int j, int k) {
  const long long l = m.l(i, j, k);
  CflIn<S> q;
  q.r = rho[l]; q.c = cs[l];
  q.v = vx[l]; q.vp = vx[(i < m.nx - 1) ? l + 1 : l - (m.nx - 1)];
  q.y = vy[l]; q.yp = vy[l + m.pitch];
  q.z = m.is3d ? vz[l] : (S)0; q.zp = m.is3d ? vz[l + m.stride] : (S)0;
  return q;
}

// The sum under the root of one cell's time-step limit (cfl.c:142-250).  The
// limit, cfl / sqrt(sum), falls monotonically with the sum in rounded
// arithmetic too, so the smallest limit is that of the largest sum: one root
// and one division a thread instead of a cell.  `bad` collects the failure
// flags (a non-finite limit or a non-positive density).
template <typename T, typename S>
__device__ __forceinline__ T cfl_sum(const Dims &m, const Geo<T> &g, const CflIn<S> &q, double vm, T nu, T alpha, int i,
                                     int j, int k, const CflRing<T> &z, bool &bad) {
  const T vxx = q.v - (T)vm, vxxp = q.vp - (T)vm;
  const T c = q.c;
  T ss2 = c * c;
  T visc;
  if (m.alpha) visc = alpha * c * c * ld(g.visc_j + j);
  else visc = nu;
  if (m.adiab) {   // cs holds the internal energy (cfl.c:164-172)
    const T gm = (T)m.gam;
    ss2 = gm * (gm - (T)1) * c / (T)q.r;
    if (m.alpha) visc = alpha * gm * (gm - (T)1.0) * c / (T)q.r * ld(g.visc_j + j);
  }
  // isothermal: the root of a rounded square is the magnitude, exactly
  const T ss = m.adiab ? sqrt(ss2) : fabs(c);
  const T zx = zsx(m, g, i, j, k);
  // quotients by the zone sizes from their reciprocals, which the viscous
  // limit needs anyway (c7); z.y, z.z: the ring's, formed once per thread
  const T ix = (T)1.0 / zx;
  auto by = [](T x, T y, T iy) -> T {
    if constexpr (sizeof(T) == 8) return divk(x, y, iy);
    else return x * iy;
  };
  T c1c = 0, c4 = 0, c5c = 0, c7c = 0;
  const T c1a = by(ss, zx, ix), c1b = by(ss, z.y, z.iy);
  if (m.is3d) c1c = by(ss, z.z, z.iz);
  const T c1 = (T)dmax3(c1a, c1b, c1c);
  const T c2 = by((T)(dmax2(fabs(vxx), fabs(vxxp))), zx, ix);
  const T vyl = q.y, vyp = q.yp;
  const T c3 = by((T)(dmax2(fabs(vyl), fabs(vyp))), z.y, z.iy);
  const T c5a = by(fabs((T)(q.vp - q.v)), zx, ix);
  const T c5b = by(fabs(vyp - vyl), z.y, z.iy);
  if (m.is3d) {
    const T vzl = q.z, vzp = q.zp;
    c4 = by((T)(dmax2(fabs(vzl), fabs(vzp))), z.z, z.iz);
    c5c = by(fabs(vzp - vzl), z.z, z.iz);
    c7c = z.iz;
  }
  const T c5 = (T)dmax3(c5a, c5b, c5c) * (T)4.0 * (T)FB_CVNR;
  const T mx7 = (T)dmax3(ix, z.iy, c7c);
  const T c7 = (T)4.0 * visc * (mx7 * mx7);
  const T zero = 0;
  const T sum = c1 * c1 + c2 * c2 + c3 * c3 + c4 * c4 + c5 * c5 + zero * zero + c7 * c7 + zero * zero + zero * zero +
                zero * zero;
  bad |= !(sum == sum) || !(q.r > (S)0);
  return sum;
}

// Shear limit of ring j (cfl_b.c:20-31).
template <typename T>
__device__ __forceinline__ double cfl_shear(const Geo<T> &g, const double *__restrict__ vxmed, double cfl_num,
                                            double mindx, int jk, int j) {
  return cfl_num * mindx / fabs(vxmed[jk] / (double)ld(g.ymed + j) - vxmed[jk + 1] / (double)ld(g.ymed + j + 1));
}

// This thread's share of ring (j, k): the minimum of its cells' limits (and,
// for thread 0, the ring's shear limit); non-finite steps or non-positive
// densities raise the flag word dtmin[1].  Two cells a thread at a time, the
// first two loaded before the ring's zones are formed: the kernel waits for
// memory most of its time (512x256x48 FP64 161 -> 112 us, FP32 storage
// 107 -> 71, against a root a cell and cell after cell).
template <typename T, typename S = T>
__device__ __forceinline__ double cfl_ring(Dims m, Geo<T> g, const S *__restrict__ rho, const S *__restrict__ cs,
                                           const S *__restrict__ vx, const S *__restrict__ vy,
                                           const S *__restrict__ vz, const double *__restrict__ vxmed,
                                           const fb_scalars *__restrict__ sc, double cfl_num, double mindx,
                                           unsigned long long *__restrict__ dtmin, int j, int k,
                                           const double *__restrict__ vbg) {
  const int step = 2 * blockDim.x;
  int i = threadIdx.x;
  CflIn<S> a = cfl_load<S>(m, rho, cs, vx, vy, vz, min(i, m.nx - 1), j, k);
  CflIn<S> b = cfl_load<S>(m, rho, cs, vx, vy, vz, min(i + (int)blockDim.x, m.nx - 1), j, k);
  // FP32 disks hold vx less the ring's background: the mean less it too
  const double vm = vxmed[j + k * m.sy] - bg_at(vbg, j + k * m.sy);
  const T nu = (T)sc->nu, alpha = (T)sc->alpha;
  const CflRing<T> z = cfl_zones(m, g, j, k);
  T mx = 0;
  bool bad = false;
  for (; i < m.nx; i += step) {   // past the ring's end: its last cell, again
    const int ib = min(i + (int)blockDim.x, m.nx - 1);
    const T sa = cfl_sum<T, S>(m, g, a, vm, nu, alpha, i, j, k, z, bad);
    const T sb = cfl_sum<T, S>(m, g, b, vm, nu, alpha, ib, j, k, z, bad);
    mx = fmax(mx, fmax(sa, sb));
    if (i + step < m.nx) {
      a = cfl_load<S>(m, rho, cs, vx, vy, vz, i + step, j, k);
      b = cfl_load<S>(m, rho, cs, vx, vy, vz, min(i + step + (int)blockDim.x, m.nx - 1), j, k);
    }
  }
  double mn = fmin(1e20, (double)((T)cfl_num / sqrt(mx)));
  // failure detection: the host or the batch scalar kernel reacts to dtmin[1]
  if (bad) atomicOr(dtmin + 1, 1ull);
  if (threadIdx.x == 0) {
    const double shear = cfl_shear(g, vxmed, cfl_num, mindx, j + k * m.sy, j);
    if (shear < mn) mn = shear;
  }
  return mn;
}

// Block minimum of the threads' shares, folded into the device-wide minimum.
__device__ __forceinline__ void cfl_commit(double mn, unsigned long long *__restrict__ dtmin) {
  for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  __shared__ double wm[32];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = mn;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < (blockDim.x >> 5) ? wm[threadIdx.x] : 1e20;
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0 && v > 0.0) atomicMin(dtmin, (unsigned long long)__double_as_longlong(v));
  }
}

// one CTA per ring (four rings a CTA, one after the other: 138 -> 169 us at
// 512x256x48), as many resident as hide the loads without spilling
// (512x256x48: FP64 173 us at 2, 134, 112 at 4, 116, 126 at 6; FP32 storage 89
// at 4, 77, 71 at 6)
template <typename T, typename S>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 4 : 6) k_cfl(const __grid_constant__ fb_disk_dev D) {
  const fb_fluid_dev &F = D.fl[blockIdx.z];
  const Dims m = dims_of(D);
  unsigned long long *dtmin = (unsigned long long *)D.dtmin;
  cfl_commit(cfl_ring<T, S>(m, geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), (const S *)F.rho, (const S *)F.cs,
                            (const S *)F.vx, (const S *)F.vy, (const S *)F.vz, F.vxmed, D.scal_dev, D.cfl, D.mindx,
                            dtmin, FB_NGH + blockIdx.x, m.is3d ? FB_NGH + blockIdx.y : 0, F.vbg),
             dtmin);
  cfl_report(D);
}

// ---------------------------------------------------------------------------
// Ghost cells from the setups' boundary templates (std/boundaries.txt with
// setups/fargo/fargo.bound in 2D and setups/p3disof/p3disof.bound in 3D;
// index rules of scripts/boundparser.py:360-398).  All libm factors of the
// templates are tabulated on the host.  Table layout (doubles):
//   [0,6)  rho power factor per (side, ghost row)   [6,12) sqrt factor
//   [12,18) 3D radial v_phi correction factor        [18,18+6*sz) 3D exp factor
//   then 6*sy colatitude density factors, then 6 colatitude v_phi factors.
struct BndTab {
  const double *t;
  int sy, sz;
  __device__ double rhof(int s, int jj) const { return t[s * 3 + jj]; }
  __device__ double sqf(int s, int jj) const { return t[6 + s * 3 + jj]; }
  __device__ double cf(int s, int jj) const { return t[12 + s * 3 + jj]; }
  __device__ double rhoe(int s, int jj, int k) const { return t[18 + (s * 3 + jj) * sz + k]; }
  __device__ double zrho(int s, int kk, int j) const { return t[18 + 6 * sz + (s * 3 + kk) * sy + j]; }
  __device__ double zw(int s, int kk) const { return t[18 + 6 * sz + 6 * sy + s * 3 + kk]; }
};

// 2D disks fill their radial ghosts from the kernels that write the mirrored
// active rows (the source stage V_temp's, but for adiabatic disks, whose
// SubStep3 reads the outer edge face before it is filled; the azimuthal sweep
// the state's) instead of in a launch of their own: the ghosts of column i that
// row j's value determines, with b_bnd_y's formulas.  A disk has at least four
// rows (fb_disk_create), of which one may mirror to both sides.
// rho, e: null for V_temp / isothermal disks.  The caller stores vy = 0 on the
// lower edge face (row Nghy) itself.
template <typename S>
__device__ __forceinline__ void ghosts_of_row(const Dims &m, const double *__restrict__ ymed, const double *__restrict__ tab,
                                              const double *__restrict__ vbg, double of, int i, int j, S *rho, S *vx,
                                              S *vy, S *e, S r, S u, S v, S en) {
  const double ya = ld(ymed + j);
  auto mirror = [&](int s, int jj, int jgh) {
    const long long g = m.l(i, jgh, 0);
    const double yg = ld(ymed + jgh), f = tab[6 + s * 3 + jj];
    if (rho) rho[g] = r * tab[s * 3 + jj];
    if constexpr (sizeof(S) == 4)   // vx less the rings' backgrounds
      vx[g] = (((double)u + (vbg ? vbg[j] : 0.0)) + ya * of) * f - yg * of - (vbg ? vbg[jgh] : 0.0);
    else vx[g] = (u + ya * of) * f - yg * of;
    if (e) e[g] = en;
  };
  if (m.bclo) {
    if (j <= 5) mirror(0, 5 - j, 5 - j);
    if (j >= 4 && j <= 6) vy[m.l(i, 6 - j, 0)] = -v;
  }
  const int up = m.ny + FB_NGH - 1 - j;
  if (m.bchi && up <= 2) {
    mirror(1, up, m.ny + FB_NGH + up);
    if (up < 2) vy[m.l(i, m.ny + FB_NGH + 1 + up, 0)] = -v;
    if (up == 0) vy[m.l(i, m.ny + FB_NGH, 0)] = 0;
  }
}
// whether row j of a 2D disk determines ghosts
__device__ __forceinline__ bool edge_row(const Dims &m, int j) { return j <= 6 || j >= m.ny; }

// ---------------------------------------------------------------------------
// Sources, 2D cylindrical (algogas.c:30-120): ComputePressureFieldIso,
// compute_potential's Potential, CorrectVtheta, SubStep1_x/y, visctensor_cyl,
// addviscosity_cyl, SubStep2_a/b, fused over a TX x TY tile of active cells,
// FP64 in the reference's operations and order.
// Inputs (rho, cs, v, P, Pot) are staged with a one-cell halo; the stress
// tensor is computed once per point into shared memory.  The kernel is bound
// by its FP64 divisions (12.6 issue slots each): those by a row's or column's
// geometry or by a planet's constants take a tabulated reciprocal (divk), and
// the density sums that several terms divide by are inverted once.
constexpr int SRC2_TX = 32, SRC2_TY = 8;
__device__ __forceinline__ void b_sources_cyl(const Dims &m, const Geo<double> &g, const double *__restrict__ rho,
    const double *__restrict__ cs, const double *__restrict__ vx, const double *__restrict__ vy,
    double *__restrict__ vxt, double *__restrict__ vyt, const fb_scalars *__restrict__ scp, int dust, int viscous,
    double *__restrict__ et, const double *__restrict__ tab, int bx, int by) {
  constexpr int TX = SRC2_TX, TY = SRC2_TY, W = TX + 2, H = TY + 2;
  __shared__ double s_rho[H][W], s_cs[H][W], s_vx[H][W], s_vy[H][W], s_p[H][W], s_pot[H][W];
  __shared__ double s_txx[H][W], s_tyy[H][W], s_tyx[H][W];
  __shared__ fb_scalars sc;
  __shared__ double s_id3[FB_MAXPLANETS];          // 1 / d^3 of the planets
  __shared__ double s_iyi[H];                      // 1 / (Ymin(j+1) - Ymin(j))
  const int i0 = bx * TX, j0 = FB_NGH + by * TY;
  const int tid = threadIdx.x;
  for (int w = tid; w < (int)(sizeof(fb_scalars) / 8); w += TX * TY)
    reinterpret_cast<double *>(&sc)[w] = reinterpret_cast<const double *>(scp)[w];
  if (tid >= 64 && tid < 64 + H) {
    const int j = min(j0 - 1 + tid - 64, m.sy - 1);
    s_iyi[tid - 64] = 1.0 / (ld(g.ymin + j + 1) - ld(g.ymin + j));
  }
  if (tid >= 128 && tid < 128 + FB_MAXPLANETS && tid - 128 < scp->nplanets) s_id3[tid - 128] = 1.0 / scp->pdist3[tid - 128];
  __syncthreads();
  const double dt = sc.dt, domega = sc.domega, of = sc.omegaframe;
  // stage inputs; vx carries CorrectVtheta (correct_vtheta.c:55-60)
  for (int e = tid; e < H * W; e += TX * TY) {
    const int lj = e / W, li = e - lj * W;
    const int j = j0 - 1 + lj, i = wrapx(i0 - 1 + li, m.nx);
    if (j < m.sy && i0 - 1 + li <= m.nx) {
      const long long l = m.l(i, j, 0);
      const double r = rho[l], c = cs[l], ym = ld(g.ymed + j);
      s_rho[lj][li] = r;
      s_cs[lj][li] = c;
      s_vx[lj][li] = vx[l] - domega * ym;
      s_vy[lj][li] = vy[l];
      // ComputePressureFieldIso, or ComputePressureFieldAd (CompPresAd.c:54)
      // where cs holds the internal energy
      s_p[lj][li] = m.adiab ? (m.gam - 1.0) * c : r * c * c;
      // Potential (potential.c:51-208); the star's term is the row table's
      const double XC = ym * ld(g.cos_xmed + i), YC = ym * ld(g.sin_xmed + i), ZC = ld(g.zmed + 0);
      double pot = ld(g.pot_star + j);
      for (int n = 0; n < sc.nplanets; n++) {
        const double mp = sc.pmass[n], xp = sc.px[n], yp = sc.py[n], zp = sc.pz[n];
        const double dist = ((XC - xp) * (XC - xp) + (YC - yp) * (YC - yp) + (ZC - zp) * (ZC - zp));
        if (sc.indirect_term) pot += divk(mp * (XC * xp + YC * yp + ZC * zp), sc.pdist3[n], s_id3[n]);
        pot += -1.0 * mp / sqrt(dist + sc.psmooth2[n]);
      }
      s_pot[lj][li] = pot;
    }
  }
  __syncthreads();
  auto by_ymin = [&](double x, int j) { return divk(x, ld(g.ymin + j), ld(g.inv_ymin + j)); };
  auto by_dymed = [&](double x, int j) { return divk(x, ld(g.ymed + j) - ld(g.ymed + j - 1), ld(g.inv_dymed + j)); };
  if (viscous) {
    const double nu = sc.nu, alpha = sc.alpha, syk = ld(g.syk + 0), sxk = ld(g.sxk + 0);
    for (int e = tid; e < H * W; e += TX * TY) {
      const int lj = e / W, li = e - lj * W;
      const int j = j0 - 1 + lj, i = wrapx(i0 - 1 + li, m.nx);
      if (j >= m.sy - 1 || i0 - 1 + li > m.nx) continue;
      // tau_xx, tau_yy at (li in [0,TX], lj in [0,TY]); tau_yx at (li,lj >= 1)
      double visc = nu, viscm = nu;
      if (m.alpha && lj >= 1 && li >= 1) {
        const double e0 = s_cs[lj][li], ex = s_cs[lj][li - 1], ey = s_cs[lj - 1][li], exy = s_cs[lj - 1][li - 1];
        if (m.adiab)   // visctensor_cyl.c:148 (cs = internal energy)
          viscm = alpha * m.gam * (m.gam - 1.0) * (e0 + ex + ey + exy) /
                  (s_rho[lj][li] + s_rho[lj][li - 1] + s_rho[lj - 1][li] + s_rho[lj - 1][li - 1]) * ld(g.viscm_j + j);
        else
          viscm = alpha * 0.0625 * (e0 + ex + ey + exy) * (e0 + ex + ey + exy) * ld(g.viscm_j + j);
      }
      if (m.alpha) {
        if (m.adiab)   // visctensor_cyl.c:147
          visc = alpha * m.gam * (m.gam - 1.0) * s_cs[lj][li] / s_rho[lj][li] * ld(g.visc_j + j);
        else
          visc = alpha * s_cs[lj][li] * s_cs[lj][li] * ld(g.visc_j + j);
      }
      if (li <= TX && lj <= TY) {
        const double r = s_rho[lj][li], sxi = ld(g.sxi + i), ym = ld(g.ymed + j);
        const double dvx = s_vx[lj][li + 1] - s_vx[lj][li], vy0 = s_vy[lj][li], vyp = s_vy[lj + 1][li];
        double div_v = 0.0;
        div_v += dvx * ld(g.sxj + j) * sxk;
        div_v += (vyp * ld(g.syj + j + 1) * syk * sxi - vy0 * ld(g.syj + j) * syk * sxi);
        div_v *= (2.0 / 3.0) * ld(g.invvj + j) / (syk * sxi);
        double txx = visc * r * (2.0 * dvx / (sxi * ym) - div_v);
        txx += divk(visc * r * (vyp + vy0), ym, ld(g.inv_ymed + j));
        s_txx[lj][li] = txx;
        s_tyy[lj][li] = visc * r * (divk(2.0 * (vyp - vy0), ld(g.ymin + j + 1) - ld(g.ymin + j), s_iyi[lj]) - div_v);
      }
      if (li >= 1 && lj >= 1) {
        s_tyx[lj][li] = viscm * 0.25 *
                        (s_rho[lj][li] + s_rho[lj][li - 1] + s_rho[lj - 1][li] + s_rho[lj - 1][li - 1]) *
                        (by_ymin((s_vy[lj][li] - s_vy[lj][li - 1]) * ld(g.invdiffxmed + i), j) +
                         by_dymed(s_vx[lj][li] - s_vx[lj - 1][li], j) -
                         by_ymin(0.5 * (s_vx[lj][li] + s_vx[lj - 1][li]), j));
      }
    }
    __syncthreads();
  }
  const int lx = tid & (TX - 1), ly = tid / TX, li = lx + 1, lj = ly + 1;
  const int i = i0 + lx, j = j0 + ly;
  // adiabatic disks also need V_temp of row Ny+3, the outer edge face, which
  // SubStep3 reads before the ghost fill (substep1_y.c: j < Ny+2*NGHY-1)
  if (i >= m.nx || j > m.ny + FB_NGH - 1 + m.adiab) return;
  const int im = wrapx(i - 1, m.nx);
  const long long l = m.l(i, j, 0);
  const double r = s_rho[lj][li], rxm = s_rho[lj][li - 1], rym = s_rho[lj - 1][li];
  const double ym = ld(g.ymed + j), ymm = ld(g.ymed + j - 1), yi = ld(g.ymin + j), yip = ld(g.ymin + j + 1),
               yim = ld(g.ymin + j - 1), dym = ym - ymm, idym = ld(g.inv_dymed + j);
  const double izx = divk(ld(g.invdiffxmed + i), ym, ld(g.inv_ymed + j));
  // SubStep1_x (substep1_x.c:107-117)
  const double sxi = ld(g.sxi + i), sxim = ld(g.sxi + im);
  const double dxmed = 0.5 * (sxi + sxim);
  const double dx_ = r * sxi + rxm * sxim, idx_ = 1.0 / dx_;
  const double dtorx = divk(2. * dt, dx_, idx_) * dxmed;
  double ax = s_vx[lj][li];
  if (!dust) ax -= dtorx * (s_p[lj][li] - s_p[lj][li - 1]) * izx;
  ax -= ((s_pot[lj][li] - s_pot[lj][li - 1]) * dt) * izx;
  // SubStep1_y (substep1_y.c:146-192, cylindrical)
  const double dy_ = r * (yip - yi) + rym * (yi - yim), idy_ = 1.0 / dy_;
  const double dtory = divk(2.0 * dt, dy_, idy_) * dym;
  double ay = s_vy[lj][li];
  if (!dust) ay -= divk(dtory * (s_p[lj][li] - s_p[lj - 1][li]), dym, idym);
  double vphi = 0.25 * (s_vx[lj][li] + s_vx[lj][li + 1] + s_vx[lj - 1][li] + s_vx[lj - 1][li + 1]);
  vphi += yi * of;
  ay += by_ymin(vphi * vphi, j) * dt;
  ay -= divk((s_pot[lj][li] - s_pot[lj - 1][li]) * dt, dym, idym);
  if (viscous) {
    // addviscosity_cyl (addviscosity_cyl.c:106-124)
    const double sx = r + rxm, sy = r + rym;
    ax += 2.0 * (s_txx[lj][li] - s_txx[lj][li - 1]) * izx / sx * dt;
    ax += 2.0 * (yip * yip * s_tyx[lj + 1][li] - yi * yi * s_tyx[lj][li]) / ((yip - yi) * ym * ym * sx) * dt;
    ay += 2.0 * (ym * s_tyy[lj][li] - ymm * s_tyy[lj - 1][li]) / (dym * sy * yi) * dt;
    ay += 2.0 * (s_tyx[lj][li + 1] - s_tyx[lj][li]) / ((ld(g.xmin + i + 1) - ld(g.xmin + i)) * yi * sy) * dt;
    ay -= (s_txx[lj][li] + s_txx[lj - 1][li]) / (yi * sy) * dt;
  }
  // SubStep2_a / SubStep2_b (substep2_a.c:107-129, substep2_b.c:150-175)
  auto art = [&](double rr, double dv) { return dv < 0.0 ? FB_CVNR * FB_CVNR * rr * dv * dv : 0.0; };
  const double dvx = s_vx[lj][li + 1] - s_vx[lj][li], dvy = s_vy[lj + 1][li] - s_vy[lj][li];
  const double qx = art(r, dvx), qxm = art(rxm, s_vx[lj][li] - s_vx[lj][li - 1]);
  const double qy = art(r, dvy), qym = art(rym, s_vy[lj][li] - s_vy[lj - 1][li]);
  ax += divk(-2.0 * dt * dxmed * (qx - qxm), dx_, idx_) * izx;
  ay += divk(-2.0 * (qy - qym), dy_, idy_) * dt;
  vxt[l] = ax;
  if (!m.adiab) {
    vyt[l] = j == FB_NGH && m.bclo ? 0.0 : ay;
    if (edge_row(m, j)) ghosts_of_row<double>(m, g.ymed, tab, nullptr, of, i, j, nullptr, vxt, vyt, nullptr, r, ax, ay, 0.0);
  } else {
    vyt[l] = ay;
  }
  if (m.adiab && !dust && et) {
    // SubStep2_b (substep2_b.c:161-178): the artificial viscosity's heating,
    // with the velocities the step started from (after CorrectVtheta)
    double en = s_cs[lj][li];
    en += -dt * (qx * dvx / (sxi * ym));
    en += -dt * divk(qy * dvy, yip - yi, s_iyi[lj]);
    et[l] = en;
  }
}

static __global__ void __launch_bounds__(SRC2_TX *SRC2_TY, 2) k_sources_cyl(const __grid_constant__ fb_disk_dev D) {
  const fb_fluid_dev &F = D.fl[blockIdx.z];
  b_sources_cyl(dims_of(D), geo_of<double>(D.geomd), (const double *)F.rho, (const double *)F.cs, (const double *)F.vx,
                (const double *)F.vy, (double *)F.vxt, (double *)F.vyt, D.scal_dev, F.dust, !F.dust, (double *)F.et,
                D.bnd_tab, blockIdx.x, blockIdx.y);
}

}  // namespace fb

namespace fb {

// ---------------------------------------------------------------------------
// Dust diffusion (DustDiffusion_Main, dust_diffusion_main.c:3-28), 2D
// cylindrical: each dust fluid's density diffuses down the gradient of its
// concentration c = rho_d / (rho_d + rho_g) with the gas's diffusivity --
// Nu (VISCOSITY) or Alpha cs^2 / Omega_K (ALPHAVISCOSITY, isothermal), at cell
// centres and at the radial faces (dust_diffusion_coefficients.c:94-120) --
// rho_d += dt div(D grad c) in the reference's operation order
// (dust_diffusion_core.c:132-185), into a buffer, for the active rows.
template <typename T, typename S>
__global__ void __launch_bounds__(128) k_dust_diffusion(const __grid_constant__ fb_disk_dev D) {
  const fb_fluid_dev &F = D.fl[1 + blockIdx.z];
  const S *__restrict__ rd = (const S *)F.rho, *__restrict__ rg = (const S *)D.fl[0].rho,
                       *__restrict__ csg = (const S *)D.fl[0].cs;
  S *__restrict__ out = (S *)F.rho_a;
  const fb_scalars *__restrict__ scp = D.scal_dev;
  const Dims m = dims_of(D);
  const Geo<T> g = geo_of<T>(D.geomd);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = FB_NGH + blockIdx.y;
  if (i >= m.nx) return;
  const T dt = (T)scp->dt, nu = (T)scp->nu, alpha = (T)scp->alpha;
  const long long l = m.l(i, j, 0);
  const int ixp = i < m.nx - 1 ? i + 1 : 0;
  const long long lxp = (i < m.nx - 1) ? l + 1 : l - (m.nx - 1), lxm = i > 0 ? l - 1 : l + (m.nx - 1);
  const long long lyp = l + m.pitch, lym = l - m.pitch;
  // Sdiffyczc at a cell of row jj, Sdiffyfzc at the lower face of row jj
  auto sdc = [&](long long ll, int jj) -> T {
    if (!m.alpha) return nu;
    const T ss2 = (T)csg[ll] * (T)csg[ll];
    const T r3 = ld(g.ymed + jj) * ld(g.ymed + jj) * ld(g.ymed + jj);
    return alpha * ss2 / sqrt((T)1.0 * (T)1.0 / r3);
  };
  auto sdf = [&](long long ll, int jj) -> T {
    if (!m.alpha) return nu;
    T ssf2;
    if (jj == 0) ssf2 = (T)csg[ll] * (T)csg[ll];
    else ssf2 = (T)0.5 * ((T)csg[ll] + (T)csg[ll - m.pitch]) * (T)0.5 * ((T)csg[ll] + (T)csg[ll - m.pitch]);
    const T r3 = ld(g.ymin + jj) * ld(g.ymin + jj) * ld(g.ymin + jj);
    return alpha * ssf2 / sqrt((T)1.0 * (T)1.0 / r3);
  };
  const T d0 = rd[l], g0 = rg[l];
  T update = 0.0;
  const T c = d0 / (d0 + g0);
  const T dxmin = ld(g.xmin + i + 1) - ld(g.xmin + i);
  const T dxmedp = (T)1.0 / ld(g.invdiffxmed + ixp), dxmedm = (T)1.0 / ld(g.invdiffxmed + i);
  const T dxp = rd[lxp], gxp = rg[lxp], dxm = rd[lxm], gxm = rg[lxm];
  const T d1 = (T)0.25 * (d0 + g0 + dxp + gxp) * (sdc(lxp, j) + sdc(l, j));
  const T d2 = (T)0.25 * (d0 + g0 + dxm + gxm) * (sdc(lxm, j) + sdc(l, j));
  const T cxp = dxp / (dxp + gxp), cxm = dxm / (dxm + gxm);
  const T ym = ld(g.ymed + j), ymp = ld(g.ymed + j + 1), ymm = ld(g.ymed + j - 1);
  const T yi = ld(g.ymin + j), yip = ld(g.ymin + j + 1);
  update += (T)1.0 / ym / ym / (dxmin) * (d1 * (cxp - c) / (dxmedp) - (d2 * (c - cxm)) / (dxmedm));
  const T dyp = rd[lyp], gyp = rg[lyp], dym = rd[lym], gym = rg[lym];
  const T d3 = (T)0.5 * (d0 + g0 + dyp + gyp) * sdf(lyp, j + 1);
  const T d4 = (T)0.5 * (d0 + g0 + dym + gym) * sdf(l, j);
  const T cyp = dyp / (dyp + gyp), cym = dym / (dym + gym);
  update += (T)1.0 / ym / (yip - yi) * (yip * d3 * (cyp - c) / (ymp - ym) - (yi * d4 * (c - cym)) / (ym - ymm));
  out[l] = d0 + dt * update;
}

// copy_field(Density, Pressure) of DustDiffusion_Main for the active rows
template <typename S>
__global__ void __launch_bounds__(128) k_copy_rows(const __grid_constant__ fb_disk_dev D) {
  const Dims m = dims_of(D);
  const S *__restrict__ src = (const S *)D.fl[1 + blockIdx.z].rho_a;
  S *__restrict__ dst = (S *)D.fl[1 + blockIdx.z].rho;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nx) return;
  const long long l = m.l(i, FB_NGH + blockIdx.y, 0);
  dst[l] = src[l];
}

// FillGhosts(DENS): the density's radial ghosts only (KEPLERIAN2DDENS)
template <typename T, typename S>
__global__ void k_bnd_rho_y(const __grid_constant__ fb_disk_dev D) {
  const Dims m = dims_of(D);
  const double *__restrict__ tab = D.bnd_tab;
  S *__restrict__ rho = (S *)D.fl[1 + blockIdx.z].rho;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int jj = blockIdx.y % 3, s = blockIdx.y / 3;
  if (i >= m.nx) return;
  const int jgh = s == 0 ? jj : m.ny + FB_NGH + jj, jact = s == 0 ? 2 * FB_NGH - jj - 1 : m.ny + FB_NGH - 1 - jj;
  rho[m.l(i, jgh, 0)] = rho[m.l(i, jact, 0)] * (T)tab[s * 3 + jj];
}

// ---------------------------------------------------------------------------
// SubStep3 (substep3.c:79-118), adiabatic disks: the compression work of the
// source step, e *= (1 - theta) / (1 + theta) with theta = dt (GAMMA - 1)
// div(V_temp) / (2 Vol), on the energy after SubStep2_b (et) into the Energy
// field, for the active rows (the ghosts are refilled after it).  The
// divergence uses the macros' unparenthesised products (SurfX, SurfY,
// InvVol: define.h:228-235) in the reference's order.
template <typename T>
__global__ void __launch_bounds__(128) k_substep3(const __grid_constant__ fb_disk_dev D) {
  const fb_fluid_dev &F = D.fl[blockIdx.z];
  const T *__restrict__ et = (const T *)F.et, *__restrict__ vxt = (const T *)F.vxt, *__restrict__ vyt = (const T *)F.vyt;
  T *__restrict__ e = (T *)F.cs;
  const fb_scalars *__restrict__ scp = D.scal_dev;
  const Dims m = dims_of(D);
  const Geo<T> g = geo_of<T>(D.geomd);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = FB_NGH + blockIdx.y, k = 0;
  if (i >= m.nx) return;
  const T dt = (T)scp->dt;
  const long long l = m.l(i, j, k);
  const long long lxp = (i < m.nx - 1) ? l + 1 : l - (m.nx - 1);
  T div_v = 0.0;
  div_v += (vxt[lxp] - vxt[l]) * ld(g.sxj + j) * ld(g.sxk + k);
  div_v += (vyt[l + m.pitch] * ld(g.syj + j + 1) * ld(g.syk + k) * ld(g.sxi + i) -
            vyt[l] * ld(g.syj + j) * ld(g.syk + k) * ld(g.sxi + i));
  const T term = (T)0.5 * dt * ((T)m.gam - (T)1.) * div_v * ld(g.invvj + j) / (ld(g.syk + k) * ld(g.sxi + i));
  e[l] = et[l] * (((T)1.0 - term) / ((T)1.0 + term));
}

// ---------------------------------------------------------------------------
// Radial sides: one thread per (i, ghost row jj, side s, layer k).
template <typename T, typename S = T>
__device__ __forceinline__ void b_bnd_y(Dims m, Geo<T> g, BndTab tb, S *__restrict__ rho, S *__restrict__ vx,
                        S *__restrict__ vy, S *__restrict__ vz, const fb_scalars *__restrict__ scp,
                        int do_rho, const double *__restrict__ vbg, uint3 bid, S *__restrict__ energy = nullptr) {
  const int i = bid.x * blockDim.x + threadIdx.x;
  const int jj = bid.y % 3, s = bid.y / 3, k = bid.z;
  if (i >= m.nx) return;
  // a slab's inner edge takes its ghosts from the neighbouring slab
  if ((s == 0 && !m.bclo) || (s == 1 && !m.bchi)) return;
  const T of = (T)scp->omegaframe;
  const int nghy = FB_NGH, ny = m.ny;
  int jgh, jact, jlacts, jnull;
  if (s == 0) { jgh = jj; jact = 2 * nghy - jj - 1; jlacts = 2 * nghy - jj; jnull = nghy; }
  else { jgh = ny + nghy + jj; jact = ny + nghy - 1 - jj; jlacts = jact; jnull = ny + nghy; }
  const long long lgh = m.l(i, jgh, k), lact = m.l(i, jact, k);
  const T yact = ld(g.ymed + jact), ygh = ld(g.ymed + jgh);
  // FP32 storage: vx less the ring backgrounds of the active and ghost rows
  constexpr bool BG = sizeof(S) < sizeof(T);
  const T vact = BG ? (T)vx[lact] + (T)bg_at(vbg, jact + k * m.sy) : (T)vx[lact];
  const T bgh = BG ? (T)bg_at(vbg, jgh + k * m.sy) : (T)0;
  if (!m.is3d) {
    if (do_rho) rho[lgh] = rho[lact] * (T)tb.rhof(s, jj);
    if (BG) vx[lgh] = (vact + yact * of) * (T)tb.sqf(s, jj) - ygh * of - bgh;
    else vx[lgh] = (vx[lact] + yact * of) * (T)tb.sqf(s, jj) - ygh * of;
  } else {
    const T sz = ld(g.sin_zmed + k);
    if (do_rho) rho[lgh] = rho[lact] * (T)tb.rhof(s, jj) * (T)tb.rhoe(s, jj, k);
    if (BG) vx[lgh] = (vact + of * yact * sz) * (T)tb.sqf(s, jj) * (T)tb.cf(s, jj) - ygh * of * sz - bgh;
    else vx[lgh] = (vx[lact] + of * yact * sz) * (T)tb.sqf(s, jj) * (T)tb.cf(s, jj) - ygh * of * sz;
  }
  // Energy of adiabatic disks: SYMMETRIC (the ghost mirrors the active cell)
  if (energy) energy[lgh] = energy[lact];
  // Vy: ANTISYMMETRIC, staggered in y (|-a|0|a|)
  if (s == 0) vy[lgh] = -vy[m.l(i, jlacts, k)];
  else if (jj < nghy - 1) vy[m.l(i, ny + nghy + 1 + jj, k)] = -vy[m.l(i, jlacts, k)];
  vy[m.l(i, jnull, k)] = 0;
  // Vz: SYMMETRIC, centred in y
  if (m.is3d) vz[lgh] = vz[lact];
}
template <typename T, typename S = T>
__global__ void k_bnd_y(const __grid_constant__ fb_disk_dev D, int vtemp) {
  const Dims m = dims_of(D);
  const int f = blockIdx.z / m.sz;
  const fb_fluid_dev &F = D.fl[f];
  // adiabatic disks: the energy's ghosts too, after the sources and at the end
  b_bnd_y<T, S>(m, geo_of<T>(D.geomd), BndTab{D.bnd_tab, m.sy, m.sz}, (S *)F.rho, (S *)(vtemp ? F.vxt : F.vx),
                (S *)(vtemp ? F.vyt : F.vy), (S *)(vtemp ? F.vzt : F.vz), D.scal_dev, !vtemp, F.vbg,
                make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - f * m.sz), m.adiab ? (S *)F.cs : (S *)nullptr);
}

// Colatitude sides (3D): one thread per (i, j, ghost layer kk, side s).
template <typename T, typename S = T>
__device__ __forceinline__ void b_bnd_z(Dims m, Geo<T> g, BndTab tb, S *__restrict__ rho, S *__restrict__ vx,
                        S *__restrict__ vy, S *__restrict__ vz, const fb_scalars *__restrict__ scp,
                        int do_rho, const double *__restrict__ vbg, uint3 bid) {
  const int i = bid.x * blockDim.x + threadIdx.x;
  const int j = bid.y, kk = bid.z % 3, s = bid.z / 3;
  if (i >= m.nx) return;
  const T of = (T)scp->omegaframe;
  const int nghz = FB_NGH, nz = m.nz;
  int kgh, kact, klacts, knull;
  if (s == 0) { kgh = kk; kact = 2 * nghz - kk - 1; klacts = 2 * nghz - kk; knull = nghz; }
  else { kgh = nz + nghz + kk; kact = nz + nghz - 1 - kk; klacts = kact; knull = nz + nghz; }
  const long long lgh = m.l(i, j, kgh), lact = m.l(i, j, kact);
  const T ym = ld(g.ymed + j);
  if (do_rho) rho[lgh] = rho[lact] * (T)tb.zrho(s, kk, j);
  if (sizeof(S) < sizeof(T)) {  // FP32 storage: vx less the ring backgrounds
    const T vact = (T)vx[lact] + (T)bg_at(vbg, j + kact * m.sy);
    vx[lgh] = (vact + of * ym * ld(g.sin_zmed + kact)) * (T)tb.zw(s, kk) - ym * of * ld(g.sin_zmed + kgh) -
              (T)bg_at(vbg, j + kgh * m.sy);
  } else {
    vx[lgh] = (vx[lact] + of * ym * ld(g.sin_zmed + kact)) * (T)tb.zw(s, kk) - ym * of * ld(g.sin_zmed + kgh);
  }
  vy[lgh] = vy[lact];
  if (s == 0) vz[lgh] = -vz[m.l(i, j, klacts)];
  else if (kk < nghz - 1) vz[m.l(i, j, nz + nghz + 1 + kk)] = -vz[m.l(i, j, klacts)];
  vz[m.l(i, j, knull)] = 0;
}
template <typename T, typename S = T>
__global__ void k_bnd_z(const __grid_constant__ fb_disk_dev D, int vtemp) {
  const Dims m = dims_of(D);
  const int f = blockIdx.z / 6;
  const fb_fluid_dev &F = D.fl[f];
  b_bnd_z<T, S>(m, geo_of<T>(D.geomd), BndTab{D.bnd_tab, m.sy, m.sz}, (S *)F.rho, (S *)(vtemp ? F.vxt : F.vx),
                (S *)(vtemp ? F.vyt : F.vy), (S *)(vtemp ? F.vzt : F.vz), D.scal_dev, !vtemp, F.vbg,
                make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - f * 6));
}

}  // namespace fb

namespace fb {

// ---------------------------------------------------------------------------
// NewVelocity_x/y/z (newvel_x.c:81, newvel_y.c:70, newvel_z.c:66-69) and
// StockholmBoundary (stockholm.c:129-185) on the active cells of 3D disks;
// writes the new state (rho, vx, vy, vz).  2D: fused in fb_sweepx.cuh.
template <typename T, typename S = T>
__device__ __forceinline__ void b_newvel(Dims m, Geo<T> g, const S *__restrict__ rt, const S *__restrict__ mpx,
                                                const S *__restrict__ mmx, const S *__restrict__ mpy,
                                                const S *__restrict__ mmy, const S *__restrict__ mpz,
                                                const S *__restrict__ mmz, S *__restrict__ rho, S *__restrict__ vx,
                                                S *__restrict__ vy, S *__restrict__ vz, const S *__restrict__ rho0,
                                                const S *__restrict__ vx0, const S *__restrict__ vy0,
                                                const S *__restrict__ vz0, const double *__restrict__ ramps,
                                                int stockholm, const fb_scalars *__restrict__ scp, uint3 bid) {
  const int i = bid.x * blockDim.x + threadIdx.x;
  const int j = FB_NGH + bid.y;
  const int k = FB_NGH + bid.z;
  if (i >= m.nx) return;
  const long long l = m.l(i, j, k);
  const int im = i > 0 ? i - 1 : m.nx - 1;
  const long long lxm = i > 0 ? l - 1 : l + (m.nx - 1);
  const T of = (T)scp->omegaframe;
  const T syk = ld(g.syk + k), sxi = ld(g.sxi + i), sxim = ld(g.sxi + im), ivj = ld(g.invvj + j);
  const T r = rt[l];
  T nvx, nvy, nvz;
  if constexpr (sizeof(S) == 4) {
    // FP32 storage: the same averages with the factors common to numerator
    // and denominator (Syk, InvVj) cancelled, one correctly rounded division
    // per component (a biased division would add the same error to a cell
    // step after step); the azimuthal momenta are frame-relative, so the
    // OMEGAFRAME * R term is not subtracted.
    const T rc = m.sph ? ld(g.ymed + j) * ld(g.sin_zmed + k) : ld(g.ymed + j);
    nvx = div_rn((T)mmx[l] * sxi + (T)mpx[lxm] * sxim, (r * sxi + (T)rt[lxm] * sxim) * rc);
    const T ivjm = ld(g.invvj + j - 1);
    const long long lym = l - m.pitch;
    nvy = div_rn((T)mmy[l] * ivjm + (T)mpy[lym] * ivj, r * ivjm + (T)rt[lym] * ivj);
    const T sykm = ld(g.syk + k - 1);
    const long long lzm = l - m.stride;
    nvz = div_rn((T)mmz[l] * syk + (T)mpz[lzm] * sykm, r * syk + (T)rt[lzm] * sykm);
    if (m.sph) nvz = div_rn(nvz, ld(g.ymed + j));
  } else {
    // the cells' volumes (times Sxi) are shared by the averages, and the
    // quotients by InvVj taken from its reciprocal
    const T rc = m.sph ? ld(g.ymed + j) * ld(g.sin_zmed + k) : ld(g.ymed + j);
    const T iv = (T)1.0 / ivj, ivjm = ld(g.invvj + j - 1), ivm = (T)1.0 / ivjm;
    const T w0 = divk(r * syk * sxi, ivj, iv);
    nvx = (divk(mmx[l] * syk * sxi, ivj, iv) + divk(mpx[lxm] * syk * sxim, ivj, iv)) /
          ((w0 + divk(rt[lxm] * syk * sxim, ivj, iv)) * rc);
    nvx -= of * rc;
    const long long lym = l - m.pitch;
    nvy = (divk(mmy[l] * syk * sxi, ivj, iv) + divk(mpy[lym] * syk * sxi, ivjm, ivm)) /
          (w0 + divk(rt[lym] * syk * sxi, ivjm, ivm));
    const T sykm = ld(g.syk + k - 1);
    const long long lzm = l - m.stride;
    nvz = (divk(mmz[l] * syk * sxi, ivj, iv) + divk(mpz[lzm] * sykm * sxi, ivj, iv)) /
          (w0 + divk(rt[lzm] * sykm * sxi, ivj, iv));
    if (m.sph) nvz = divk(nvz, ld(g.ymed + j), ld(g.inv_ymed + j));
  }
  T nr = r;
  if (stockholm) {
    const double dtd = scp->dt;
    const T dt = (T)dtd;
    const double rampy = ramps[j], rampz = ramps[m.sy + k], rampzz = ramps[m.sy + m.sz + k];
    const T ramp = (T)(rampy + rampz), rampi = (T)(rampy + rampzz);
    const T tau = ld(g.tau_j + j);
    const int l2 = j + k * m.sy;
    if (ramp > (T)0.0) {
      const T taud = tau / ramp;
      nr = (nr * taud + rho0[l2] * dt) / (dt + taud);
      T radius = ld(g.ymed + j);
      if (m.sph) radius *= ld(g.sin_zmed + k);
      T vx0t = vx0[l2];
      vx0t -= (of - (T)scp->omegaframe0) * radius;
      nvx = (nvx * taud + vx0t * dt) / (dt + taud);
      nvy = (nvy * taud + vy0[l2] * dt) / (dt + taud);
    }
    if (rampi > (T)0.0) {
      const T taud = tau / rampi;
      nvz = (nvz * taud + vz0[l2] * dt) / (dt + taud);
    }
  }
  rho[l] = nr;
  vx[l] = nvx;
  vy[l] = nvy;
  vz[l] = nvz;
}
template <typename T, typename S = T>
__global__ void __launch_bounds__(256) k_newvel(const __grid_constant__ fb_disk_dev D) {
  const Dims m = dims_of(D);
  const int f = blockIdx.z / m.nz;
  const fb_fluid_dev &F = D.fl[f];
  b_newvel<T, S>(m, geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), (const S *)F.rho_a, (const S *)F.mpx,
                 (const S *)F.mmx, (const S *)F.mpy, (const S *)F.mmy, (const S *)F.mpz, (const S *)F.mmz, (S *)F.rho,
                 (S *)F.vx, (S *)F.vy, (S *)F.vz, (const S *)F.rho0, (const S *)F.vx0, (const S *)F.vy0,
                 (const S *)F.vz0, D.ramps, D.stockholm, D.scal_dev,
                 make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - f * m.nz));
}

}  // namespace fb

namespace fb {

// ---------------------------------------------------------------------------
// Implicit drag between the N fluids (Collisions(dt, 1): collisions.c:10-189,
// collision_kernel.h:11-94, gauss.h:1-45), on V_temp after every fluid's
// sources.  One thread per cell (i, j >= 1[, k >= 1]) solves, for each
// direction, the N x N system of the face between the cell and its lower
// neighbour along that direction:
//   M[o][p] (o != p) = -dt W a[p][o] rho_p / rho_o  (p > o),  -dt W a[p][o]  (p < o)
//   M[p][p]          = 1 + dt W sum_{q != p} (q > p ? a[q][p] rho_q / rho_p : a[q][p])
// with face-averaged densities, W = sqrt(G M / r^3) at Ymed (x, z faces) or
// Ymin (y faces), by Gaussian elimination with the reference's row pivoting
// (the search compares |m| with the signed value last kept) and back
// substitution, in the reference's operation order.  The directions touch
// different velocity fields, so solving them in one thread per cell gives the
// reference's direction-by-direction result.
template <typename T, int N, typename S>
__device__ __forceinline__ void b_collisions(const fb_disk_dev &D, Dims m, Geo<double> gd, const fb_scalars *scp,
                                             uint3 bid) {
  const int i = bid.x * blockDim.x + threadIdx.x;
  const int j = 1 + bid.y, k = m.is3d ? 1 + bid.z : 0;
  if (i >= m.nx) return;
  const T dt = (T)scp->dt;
  const long long l = m.l(i, j, k);
  const int ndir = m.is3d ? 3 : 2;
  for (int dir = 0; dir < ndir; dir++) {
    const long long lm = dir == 0 ? (i > 0 ? l - 1 : l + (m.nx - 1)) : (dir == 1 ? l - m.pitch : l - m.stride);
    const T y = (T)(dir == 1 ? ld(gd.ymin + j) : ld(gd.ymed + j));
    const T w = sqrt((T)1.0 / (y * y * y));  // G = MSTAR = 1 (fondam.h)
    if constexpr (sizeof(S) < sizeof(T)) {
      // FP32 storage is not bound to the reference's elimination: only the
      // gas and each dust couple (ColRate, colrate.c:10-23), so with
      // k_f = dt W / St / (1 + dt W / St) the system's solution is the
      // density-weighted mean v_g = (rho_g b_g + sum rho_f k_f b_f) /
      // (rho_g + sum rho_f k_f), v_f = b_f + k_f (v_g - b_f): one division
      // a face besides the rows' k_f, in FP64 as the elimination was (768 x
      // 256, 5 fluids: 66 us of 35 divisions a face)
      T kf[N], b[N];
      const T bg = dir == 0 ? (T)1 : (T)0;   // the drag acts on the full azimuthal velocities
      T num = 0, den = 0;
#pragma unroll
      for (int f = 0; f < N; f++) {
        const S *r = (const S *)D.fl[f].rho;
        const S *v = (const S *)(dir == 0 ? D.fl[f].vxt : (dir == 1 ? D.fl[f].vyt : D.fl[f].vzt));
        const T e = f ? dt * w * (T)D.alpha[f] : (T)0;
        kf[f] = f ? e / ((T)1.0 + e) : (T)1;
        b[f] = (T)v[l] + bg * (T)bg_at(D.fl[f].vbg, j + k * m.sy);
        const T rk = (T)0.5 * ((T)r[l] + (T)r[lm]) * kf[f];
        num += rk * b[f];
        den += rk;
      }
      const T vg = num / den;
#pragma unroll
      for (int f = 0; f < N; f++) {
        S *v = (S *)(dir == 0 ? D.fl[f].vxt : (dir == 1 ? D.fl[f].vyt : D.fl[f].vzt));
        v[l] = (S)(b[f] + kf[f] * (vg - b[f]) - bg * (T)bg_at(D.fl[f].vbg, j + k * m.sy));
      }
      continue;
    }
    T rf[N], M[N * N], b[N];
#pragma unroll
    for (int f = 0; f < N; f++) {
      const S *r = (const S *)D.fl[f].rho;
      rf[f] = (T)0.5 * ((T)r[l] + (T)r[lm]);
    }
#pragma unroll
    for (int o = 0; o < N; o++) {
#pragma unroll
      for (int p = 0; p < N; p++) {
        if (p != o) {
          if (p > o) M[p + o * N] = -dt * w * (T)D.alpha[p + o * N] * rf[p] / rf[o];
          else M[p + o * N] = -dt * w * (T)D.alpha[p + o * N];
        } else {
          T sum = (T)0.0;
#pragma unroll
          for (int q = 0; q < N; q++) {
            if (q == p) continue;
            if (q > p) sum += (T)D.alpha[q + p * N] * rf[q] / rf[p];
            else sum += (T)D.alpha[q + p * N];
          }
          M[p + p * N] = (T)1.0 + dt * w * sum;
        }
      }
      const S *v = (const S *)(dir == 0 ? D.fl[o].vxt : (dir == 1 ? D.fl[o].vyt : D.fl[o].vzt));
      b[o] = (T)v[l];
    }
#pragma unroll
    for (int ir = 0; ir < N - 1; ir++) {
      T mx = (T)-1;
      int irm = ir;
#pragma unroll
      for (int ir2 = ir; ir2 < N; ir2++)
        if (fabs(M[ir + ir2 * N]) >= mx) { mx = M[ir + ir2 * N]; irm = ir2; }
      if (irm != ir) {
#pragma unroll
        for (int ic = 0; ic < N; ic++) {
          // row exchange by predicated copies keeps the matrix in registers
          T a = M[ic + ir * N];
#pragma unroll
          for (int r2 = ir + 1; r2 < N; r2++)
            if (r2 == irm) { M[ic + ir * N] = M[ic + r2 * N]; M[ic + r2 * N] = a; }
        }
        T a = b[ir];
#pragma unroll
        for (int r2 = ir + 1; r2 < N; r2++)
          if (r2 == irm) { b[ir] = b[r2]; b[r2] = a; }
      }
#pragma unroll
      for (int ir2 = ir + 1; ir2 < N; ir2++) {
        const T factor = M[ir + ir2 * N] / M[ir + ir * N];
#pragma unroll
        for (int ic = 0; ic < N; ic++) M[ic + ir2 * N] -= M[ic + ir * N] * factor;
        b[ir2] -= b[ir] * factor;
      }
    }
#pragma unroll
    for (int ir = N - 1; ir > -1; ir--) {
#pragma unroll
      for (int ic = N - 1; ic > ir; ic--) b[ir] -= M[ic + ir * N] * b[ic];
      b[ir] /= M[ir + ir * N];
    }
#pragma unroll
    for (int o = 0; o < N; o++) {
      S *v = (S *)(dir == 0 ? D.fl[o].vxt : (dir == 1 ? D.fl[o].vyt : D.fl[o].vzt));
      v[l] = (S)b[o];
    }
  }
}

template <typename T, int N, typename S>
__global__ void __launch_bounds__(128) k_collisions(const __grid_constant__ fb_disk_dev D) {
  b_collisions<T, N, S>(D, dims_of(D), geo_of<double>(D.geomd), D.scal_dev, blockIdx);
}

// ---------------------------------------------------------------------------
// The disk's gravitational acceleration at a point (x, y, z) with smoothing
// rs: ComputeAccel (planets.c:62-84) over _ComputeForce_cpu
// (compute_force.c:16-219), in FP64 and in the reference's summation order:
// each active ring's cells in order of i (reduction_SUM), then the rings in
// order of k then j (reduction_full_SUM), the inner rings (up to the point's
// radius) and the outer ones separately.  Density = the sum of the fluids'
// densities in fluid order (ComputeTotalDensity).
//
// One CTA per ring: its threads form the cells' terms (a square root and two
// divisions each) side by side in shared memory, and one lane per component
// adds them in order, a chain of nx dependent additions (8.7 cycles each).
// One lane per ring doing both took 280 us of the 632 us that two planets at
// 512 x 256 cost, its terms' latencies all in a row.
constexpr int DF_T = 128, DF_CH = 512;   // threads; cells per pass
template <typename S>
__device__ __forceinline__ void b_disk_force_rings(const fb_disk_dev &D, double x, double y, double z, double rs,
                                                   double *__restrict__ ring3, int r) {
  __shared__ double term[3][DF_CH];
  const Dims m = dims_of(D);
  const Geo<double> gd = geo_of<double>(D.geomd);
  if (r >= m.ny * (m.is3d ? m.nz : 1)) return;
  const int j = FB_NGH + r % m.ny, k = m.is3d ? FB_NGH + r / m.ny : 0;
  const double ym = ld(gd.ymed + j), syk = ld(gd.syk + k), ivj = ld(gd.invvj + j);
  const int warp = threadIdx.x >> 5;   // lane 0 of warp c sums component c
  double acc = 0.0;
  for (int c0 = 0; c0 < m.nx; c0 += DF_CH) {
    const int n = min(DF_CH, m.nx - c0);
    for (int e = threadIdx.x; e < n; e += DF_T) {
      const int i = c0 + e;
      const long long l = m.l(i, j, k);
      double dens = 0.0;
      for (int f = 0; f < D.nfluids; f++) dens += (double)((const S *)D.fl[f].rho)[l];
      const double cellmass = syk * ld(gd.sxi + i) / ivj * dens;
      double dx, dy, dz;
      if (m.sph) {
        dx = ym * ld(gd.cos_xmed + i) * ld(gd.sin_zmed + k) - x;
        dy = ym * ld(gd.sin_xmed + i) * ld(gd.sin_zmed + k) - y;
        dz = ym * ld(gd.cos_zmed + k) - z;
      } else {
        dx = ym * ld(gd.cos_xmed + i) - x;
        dy = ym * ld(gd.sin_xmed + i) - y;
        dz = ld(gd.zmed + k) - z;
      }
      double dist2 = dx * dx + dy * dy + dz * dz;
      dist2 += rs * rs;
      const double distance = sqrt(dist2);
      double inv3 = 1.0 / (dist2 * distance);
      inv3 *= 1.0 * cellmass;  // G = 1
      term[0][e] = dx * inv3;
      term[1][e] = dy * inv3;
      term[2][e] = dz * inv3;
    }
    __syncthreads();
    if (warp < 3 && (threadIdx.x & 31) == 0) acc = add_in_order(acc, term[warp], n);
    __syncthreads();
  }
  if (warp < 3 && (threadIdx.x & 31) == 0) ring3[(size_t)warp * (m.sy * m.sz) + j + k * m.sy] = acc;
}
template <typename S>
__global__ void __launch_bounds__(DF_T) k_disk_force_rings(const __grid_constant__ fb_disk_dev D,
                                                           const double *__restrict__ pt, double *__restrict__ ring3) {
  b_disk_force_rings<S>(D, pt[0], pt[1], pt[2], pt[3], ring3, blockIdx.x);
}

// fold the ring sums into inner + outer (compute_force.c:161-214): one CTA of
// DF_T threads stages the rings in order, six lanes (a component's inner or
// outer part each, in warps of their own) add them
__device__ __forceinline__ void b_disk_force_fold(const fb_disk_dev &D, double x, double y, double z,
                                                  const double *__restrict__ ring3, double *__restrict__ out3) {
  __shared__ double v[3][DF_CH];
  __shared__ double part[6];
  const Dims m = dims_of(D);
  const Geo<double> gd = geo_of<double>(D.geomd);
  const int nz = m.is3d ? m.nz : 1, k0 = m.is3d ? FB_NGH : 0, n2 = m.sy * m.sz;
  const double aa = sqrt(x * x + y * y + z * z);
  const int index = (int)(((aa - ld(gd.ymin + FB_NGH)) / (ld(gd.ymin + m.ny + FB_NGH + 1) - ld(gd.ymin + FB_NGH))) *
                          (double)m.ny) + FB_NGH;
  // rows [FB_NGH, split) are inner, [split, ny + FB_NGH) outer
  const int split = index < FB_NGH ? FB_NGH : min(index, m.ny + FB_NGH);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool adds = warp < 3 && lane < 2;   // component warp; lane 0 inner, 1 outer
  double acc = 0.0;
  for (int part_ = 0; part_ < 2; part_++) {   // all layers' inner rows, then all layers' outer rows
    const int lo = part_ ? split : FB_NGH, w = (part_ ? m.ny + FB_NGH : split) - lo;
    const long long tot = (long long)w * nz;
    for (long long e0 = 0; e0 < tot; e0 += DF_CH) {
      const int n = (int)min((long long)DF_CH, tot - e0);
      for (int e = threadIdx.x; e < n; e += DF_T) {
        const long long q = e0 + e;
        const int k = k0 + (int)(q / w), j = lo + (int)(q % w);
#pragma unroll
        for (int c = 0; c < 3; c++) v[c][e] = ring3[(size_t)c * n2 + j + k * m.sy];
      }
      __syncthreads();
      if (adds && lane == part_) acc = add_in_order(acc, v[warp], n);
      __syncthreads();
    }
  }
  if (adds) part[2 * warp + lane] = acc;
  __syncthreads();
  if (threadIdx.x < 3) out3[threadIdx.x] = part[2 * threadIdx.x] + part[2 * threadIdx.x + 1];
}
static __global__ void __launch_bounds__(DF_T) k_disk_force_fold(const __grid_constant__ fb_disk_dev D,
                                                                 const double *__restrict__ pt,
                                                                 const double *__restrict__ ring3,
                                                                 double *__restrict__ out3) {
  b_disk_force_fold(D, pt[0], pt[1], pt[2], ring3, out3);
}

// ---------------------------------------------------------------------------
// Mass of one fluid, ComputeMass (LowTasks.c:709-748): the sum over the active
// cells of rho * Vol(i, j, k), Vol = Syk(k) * Sxi(i) / InvVj(j) (define.h:229),
// in FP64 with compensation (Neumaier), so its rounding error does not grow
// with the cell count and a change of the total at round-off level is
// visible.  One warp per active ring writes the ring's (sum, compensation);
// one CTA folds the rings in a fixed order.
__device__ __forceinline__ void neumaier_add(double &s, double &c, double v) {
  const double t = s + v;
  if (fabs(s) >= fabs(v)) c += (s - t) + v;
  else c += (v - t) + s;
  s = t;
}
// (s, c) += (s2, c2) with the rounding error of s + s2 kept
__device__ __forceinline__ void neumaier_merge(double &s, double &c, double s2, double c2) {
  neumaier_add(s, c, s2);
  c += c2;
}

template <typename S>
__global__ void __launch_bounds__(256) k_mass_rings(Dims m, Geo<double> gd, const S *__restrict__ rho,
                                                    double *__restrict__ part) {
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= m.ny * (m.is3d ? m.nz : 1)) return;
  const int j = FB_NGH + r % m.ny, k = m.is3d ? FB_NGH + r / m.ny : 0;
  const double syk = ld(gd.syk + k), ivj = ld(gd.invvj + j);
  double s = 0.0, c = 0.0;
  for (int i = lane; i < m.nx; i += 32) neumaier_add(s, c, (double)rho[m.l(i, j, k)] * (syk * ld(gd.sxi + i) / ivj));
  for (int o = 16; o > 0; o >>= 1) {
    const double s2 = __shfl_xor_sync(0xffffffffu, s, o), c2 = __shfl_xor_sync(0xffffffffu, c, o);
    // both lanes of a pair fold in the same order (lower lane first)
    if (lane & o) { double t = s2, tc = c2; neumaier_merge(t, tc, s, c); s = t; c = tc; }
    else neumaier_merge(s, c, s2, c2);
  }
  if (lane == 0) { part[2 * r] = s; part[2 * r + 1] = c; }
}

static __global__ void __launch_bounds__(256) k_mass_fold(const double *__restrict__ part, int n, double *__restrict__ out) {
  __shared__ double ss[256], cc[256];
  double s = 0.0, c = 0.0;
  for (int r = threadIdx.x; r < n; r += 256) neumaier_merge(s, c, part[2 * r], part[2 * r + 1]);
  ss[threadIdx.x] = s;
  cc[threadIdx.x] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    double S = 0.0, Cc = 0.0;
    for (int t = 0; t < 256; t++) neumaier_merge(S, Cc, ss[t], cc[t]);
    *out = S + Cc;
  }
}

// The rings a step takes, a limit of the interface: an azimuthal tile of 1, 2,
// 4, 8 or 16 cells a thread (fb_disk_set_tiles) that divides them into at most
// 256 threads and whose rings, two buffers of every quantity, fit an SM's shared
// memory.  The strips of the sweep would take any ring.
inline bool ring_fits(const fb_disk_dev &d) {
  int c = d.tile_cx;
  const int cs[5] = {4, 8, 16, 2, 1};   // the default: the first that fits
  for (int t = 0; t < 5 && !c; t++)
    if (d.nx % cs[t] == 0 && d.nx / cs[t] <= 256) c = cs[t];
  if (c == 0) return false;
  const size_t esz = d.precision == FB_FP64 ? 8 : 4, nq = d.is3d ? 6 : (d.adiabatic ? 5 : 4);
  return (size_t)(256 / (d.nx / c)) * (d.nx + 16 / esz) * (2 * (1 + nq) + 1) * esz <= 227 * 1024;
}
// polls of the staged-load wait before a disk is flagged (fb_disk_set_wait_limit)
__host__ __device__ inline long long wait_limit(const fb_disk_dev &d) {
  return d.wait_limit > 0 ? d.wait_limit : (d.wait_limit < 0 ? 0 : (1ll << 22));
}

}  // namespace fb

#include "fb_sources32.cuh"
#include "fb_sources3.cuh"
#include "fb_sweepcol.cuh"
#include "fb_sweepx.cuh"
