// fb_batch.cuh -- batched stage kernels and the step launcher (see fb_batch.cu),
// included by the per-precision translation units fb_batch_f64.cu and
// fb_batch_f32.cu.
#pragma once
#include <cuda_runtime.h>


#include <stdlib.h>
#include <string.h>
#include <vector>

#include "fargo_b200.h"
#include "fb_kernels.cuh"
#include "fb_psys.h"

namespace fb {

enum { ST_ROWSUM, ST_CFL, ST_SOURCES, ST_BND_Z, ST_BND_Y, ST_COLL, ST_Z, ST_Y, ST_X, ST_NEWVEL, ST_FORCE, ST_CFL4,
       ST_N };

// tile shapes shared with the one-disk launchers (fb_launch.cuh)
// CFL_R rings per CFL CTA and NV_R rows per NewVelocity CTA: enough work per
// CTA to amortise its descriptor loads
constexpr int CFL_R = 4, NV_R = 4;
constexpr int BND_BX = 128, NV_BX = 128;

// FP32 2D CFL of rings that are no multiple of four cells (kb_cfl_cyl32): 6
// CTAs of 128 threads per SM (80 registers); on the 64-disk workload 0.090 ->
// 0.061 ms against the unconstrained 147
#ifndef FB_CFL32_MINB
#define FB_CFL32_MINB 6
#endif
#define FB_TILE                                        \
  const int4 w = items[blockIdx.x];                    \
  const int f = blockIdx.y;   /* fluid */              \
  const fb_disk_dev &D = ds[w.x];                      \
  const fb_scalars *scp = D.scal_dev;                  \
  if (scp->skip) return;                               \
  const uint3 bid = make_uint3(w.y, w.z, w.w);         \
  const fb_fluid_dev &F = D.fl[f];                     \
  (void)F;

template <typename S>
__global__ void __launch_bounds__(sizeof(S) == 8 ? 32 * RS_WARPS : 32 * RW_WARPS, sizeof(S) == 8 ? 1 : 4) kb_rowsum(const fb_disk_dev *ds, const int4 *items, int which) {
  FB_TILE
  const Dims m = dims_of(D);
  const S *v = (const S *)(which == 0 ? F.vx : F.vxt);
  double *out = which == 0 ? F.vxmed : F.vxmed_t;
  int *ns = which == 0 ? nullptr : F.nshift;   // V_temp: the azimuthal sweep's shift too
  if constexpr (sizeof(S) == 8) {
    // bid.y: rings per warp, 1 or 8 (the sum does not depend on it)
    if (bid.y == 1) b_rowsum<1>(m, geo_of<double>(D.geomd), v, out, D.xlen, (int)bid.x, scp, ns);
    else b_rowsum<8>(m, geo_of<double>(D.geomd), v, out, D.xlen, (int)bid.x, scp, ns);
  } else {
    b_rowsum_warp<S>(m, geo_of<double>(D.geomd), v, out, D.xlen, F.vbg, (int)bid.x, scp, ns, (float4 *)F.ringx);
  }
}

template <typename T, typename S>
__global__ void __launch_bounds__(256, 3) kb_cfl(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  // CFL_R rings per CTA, one minimum folded per CTA
  const Dims m = dims_of(D);
  const Geo<T> g = geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom);
  const int k = m.is3d ? FB_NGH + (int)bid.y : 0;
  const int j0 = FB_NGH + (int)bid.x * CFL_R;
  const int nr = min(CFL_R, m.ny + FB_NGH - j0);
  const T nu = (T)scp->nu, alpha = (T)scp->alpha;
  unsigned long long *dtmin = (unsigned long long *)D.dtmin;
  // the rings' zones and means, formed once
  __shared__ CflRing<T> zs[CFL_R];
  __shared__ double vms[CFL_R];
  if ((int)threadIdx.x < nr) {
    const int j = j0 + threadIdx.x;
    zs[threadIdx.x] = cfl_zones(m, g, j, k);
    vms[threadIdx.x] = F.vxmed[j + k * m.sy] - bg_at(F.vbg, j + k * m.sy);
  }
  T mx = 0;
  bool bad = false;
  // the CTA's cells, ring after ring, spread over all its threads (rings of
  // 128 cells keep all 256 busy), two at a time; max and OR do not depend on
  // the order (16 FP64 disks 90 -> 40 us,
  // against a root and the zones a cell; 43 at 4 CTAs, 50 at 2)
  const int cells = nr * m.nx;
  auto load = [&](int q, int &i, int &r) {
    q = min(q, cells - 1);
    r = q / m.nx;
    i = q - r * m.nx;
    return cfl_load<S>(m, (const S *)F.rho, (const S *)F.cs, (const S *)F.vx, (const S *)F.vy, (const S *)F.vz, i, j0 + r, k);
  };
  int ia, ra, ib, rb, q = threadIdx.x;
  CflIn<S> a = load(q, ia, ra), b = load(q + blockDim.x, ib, rb);
  __syncthreads();
  for (; q < cells; q += 2 * blockDim.x) {   // past the end: the last cell, again
    const T sa = cfl_sum<T, S>(m, g, a, vms[ra], nu, alpha, ia, j0 + ra, k, zs[ra], bad);
    const T sb = cfl_sum<T, S>(m, g, b, vms[rb], nu, alpha, ib, j0 + rb, k, zs[rb], bad);
    mx = fmax(mx, fmax(sa, sb));
    if (q + 2 * (int)blockDim.x < cells) {
      a = load(q + 2 * blockDim.x, ia, ra);
      b = load(q + 3 * blockDim.x, ib, rb);
    }
  }
  double mn = fmin(1e20, (double)((T)D.cfl / sqrt(mx)));
  if (bad) atomicOr(dtmin + 1, 1ull);
  if ((int)threadIdx.x < nr) {
    const int j = j0 + threadIdx.x;
    const double shear = cfl_shear(g, F.vxmed, D.cfl, D.mindx, j + k * m.sy, j);
    if (shear < mn) mn = shear;
  }
  cfl_commit(mn, dtmin);
}

// FP32 2D: 128 columns x CFL32_R rows a tile (fb_sources32.cuh)
static __global__ void __launch_bounds__(128, FB_CFL32_MINB) kb_cfl_cyl32(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  b_cfl_cyl32(dims_of(D), geo_of<float>(D.geom), (const float *)F.rho, (const float *)F.cs, (const float *)F.vx,
              (const float *)F.vy, F.vxmed, F.vbg, (float)scp->nu, (float)scp->alpha, D.cfl, D.mindx,
              (unsigned long long *)D.dtmin, bid);
}

static __global__ void __launch_bounds__(SRC2_TX *SRC2_TY, 2) kb_sources_cyl(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  b_sources_cyl(dims_of(D), geo_of<double>(D.geomd), (const double *)F.rho, (const double *)F.cs, (const double *)F.vx,
                (const double *)F.vy, (double *)F.vxt, (double *)F.vyt, scp, F.dust, !F.dust, (double *)nullptr,
                D.bnd_tab, (int)bid.x, (int)bid.y);
}

// FP32 storage, 2D: FP32 arithmetic, column-marching warps (fb_sources32.cuh)
static __global__ void __launch_bounds__(S32_WARPS * 32, FB_S32_MINB) kb_sources_cyl32(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  b_sources_cyl32(dims_of(D), geo_of<float>(D.geom), geo_of<double>(D.geomd), (const float *)F.rho,
                  (const float *)F.cs, (const float *)F.vx, (const float *)F.vy, (float *)F.vxt, (float *)F.vyt, scp,
                  F.dust, !F.dust, F.vbg, (const float *)F.shear_bg, D.bnd_tab, (int)bid.z, bid);
}

// 3D (fb_sources3.cuh); an item is (disk, tile x, tile y, segment | layers per segment << 16)
template <typename S>
__global__ void __launch_bounds__(S3<S>::T, FB_S3_MINB) kb_sources_sph(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  const Dims m = dims_of(D);
  const int layers = (int)(bid.z >> 16), k0 = FB_NGH + (int)(bid.z & 0xffff) * layers;
  b_sources_sph<S>(m, geo_of<double>(D.geomd), (const S *)F.rho, (const S *)F.cs, (const S *)F.vx, (const S *)F.vy,
                   (const S *)F.vz, (S *)F.vxt, (S *)F.vyt, (S *)F.vzt, scp, F.dust, !F.dust, F.vbg, (int)bid.x,
                   (int)bid.y, k0, min(k0 + layers, m.nz + FB_NGH));
}

template <typename T, typename S>
__global__ void kb_bnd(const fb_disk_dev *ds, const int4 *items, int vtemp, int zside) {
  FB_TILE
  Dims m = dims_of(D);
  BndTab tb{D.bnd_tab, m.sy, m.sz};
  S *vx = (S *)(vtemp ? F.vxt : F.vx), *vy = (S *)(vtemp ? F.vyt : F.vy), *vz = (S *)(vtemp ? F.vzt : F.vz);
  if (zside) b_bnd_z<T, S>(m, geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), tb, (S *)F.rho, vx, vy, vz, scp, !vtemp, F.vbg, bid);
  else b_bnd_y<T, S>(m, geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), tb, (S *)F.rho, vx, vy, vz, scp, !vtemp, F.vbg, bid);
}

template <typename T, int N, typename S>
__global__ void __launch_bounds__(128) kb_collisions(const fb_disk_dev *ds, const int4 *items) {
  const int4 w = items[blockIdx.x];
  const fb_disk_dev &D = ds[w.x];
  if (D.scal_dev->skip) return;
  b_collisions<T, N, S>(D, dims_of(D), geo_of<double>(D.geomd), D.scal_dev, make_uint3(w.y, w.z, w.w));
}

// column sweeps (fb_sweepcol.cuh); an item is (disk, column block, t2 | cells
// per segment << 24, segment)
template <typename T, int DIR, bool IS3D>
__global__ void __launch_bounds__(COL_T, colm_minb<T, IS3D>()) kb_sweep_colm(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  colm_cta<T, DIR, IS3D, false>(dims_of(D), geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), col_args<T>(D, F, DIR),
                                (int)(bid.y >> 24), make_uint3(bid.x, bid.y & 0xffffff, bid.z), scp);
}

// azimuthal sweep (fb_sweepx.cuh), in 2D with NewVelocity and Stockholm;
// an item is (disk, CTA, rings per warp)
template <typename T, int NQ, bool NV>
__global__ void __launch_bounds__(32 * XS_WARPS, sizeof(T) == 8 ? FB_XS64_MINB : FB_XS32_MINB) kb_sweep_xs(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  xs_cta<T, NQ, NV>(dims_of(D), geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom), xs_args<T>(D, F), scp,
                    (unsigned long long *)D.dtmin + 1, wait_limit(D), (int)bid.x, (int)bid.y);
}

// 3D disks
template <typename T, typename S>
__global__ void __launch_bounds__(NV_BX) kb_newvel(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  Dims m = dims_of(D);
  const Geo<T> g = geo_of<T>(sizeof(T) == 8 ? D.geomd : D.geom);
  for (int r = 0; r < NV_R; r++) {   // NV_R rows per CTA
    const uint3 rb = make_uint3(bid.x, bid.y * NV_R + r, bid.z);
    if ((int)rb.y >= m.ny) break;
    b_newvel<T, S>(m, g, (const S *)F.rho_a, (const S *)F.mpx, (const S *)F.mmx, (const S *)F.mpy, (const S *)F.mmy,
                   (const S *)F.mpz, (const S *)F.mmz, (S *)F.rho, (S *)F.vx, (S *)F.vy, (S *)F.vz,
                   (const S *)F.rho0, (const S *)F.vx0, (const S *)F.vy0, (const S *)F.vz0, D.ramps, D.stockholm,
                   scp, rb);
  }
}

// FP32 2D: four cells a thread (fb_sources32.cuh)
static __global__ void __launch_bounds__(Q32_T, 8) kb_cfl_cyl32q(const fb_disk_dev *ds, const int4 *items) {
  FB_TILE
  b_cfl_cyl32q(dims_of(D), geo_of<float>(D.geom), (const float *)F.rho, (const float *)F.cs, (const float *)F.vx,
               (const float *)F.vy, F.vxmed, F.vbg, (float)scp->nu, (float)scp->alpha, D.cfl, D.mindx,
               (unsigned long long *)D.dtmin, (int)bid.x);
}
// The disk's acceleration at planet n of every disk whose planet n feels the
// disk (ComputeAccel for AdvanceSystemFromDisk, planets.c:86-114), from the
// density and planets at the start of the step: the ring sums (one CTA per
// ring, the reference's order), then one CTA per disk folds them.  The
// smoothing is the planet's (compute_potential's RocheSmoothing or the
// flared thickness), formed on the device.
__device__ __forceinline__ bool force_planet(const fb_disk_dev &D, const fb_psys &S, int n, double &x, double &y,
                                             double &z, double &rs) {
  if (!D.feeldisk || n >= S.np || !S.feeldisk[n]) return false;
  x = S.px[n]; y = S.py[n]; z = S.pz[n];
  const double r = sqrt(x * x + y * y + z * z), mp = S.pmass[n];
  if (S.roche_smoothing != 0) rs = r * pow(mp / 3. / FB_MSTAR, 1. / 3.) * S.roche_smoothing;
  else rs = S.aspectratio * pow(r / FB_R0, S.flaringindex) * r * S.thickness_smoothing;
  return true;
}
template <typename S>
static __global__ void __launch_bounds__(DF_T) kb_disk_force_rings(const fb_disk_dev *ds, const fb_psys *ps,
                                                                  const int4 *items, int n) {
  const int4 w = items[blockIdx.x];
  const fb_disk_dev &D = ds[w.x];
  if (D.scal_dev->skip) return;
  double x, y, z, rs;
  if (!force_planet(D, ps[w.x], n, x, y, z, rs)) return;
  b_disk_force_rings<S>(D, x, y, z, rs, D.ring3, w.y);
}
static __global__ void __launch_bounds__(DF_T) kb_disk_force_fold(const fb_disk_dev *ds, const fb_psys *ps, const int *dl, int n) {
  const int i = dl ? dl[blockIdx.x] : (int)blockIdx.x;
  const fb_disk_dev &D = ds[i];
  if (D.nx == 0 || D.scal_dev->skip) return;
  double x, y, z, rs;
  if (!force_planet(D, ps[i], n, x, y, z, rs)) return;
  b_disk_force_fold(D, x, y, z, D.ring3, D.facc + 3 * n);
}

// The scalar work of the step for every disk of the list dl (all n disks when
// dl is null), one thread per disk; then the
// CFL minimum is reset for the next step.  dtmin[1] carries the kernels'
// non-finite flag.  A disk with an end time uses it as its DT interval, so
// its last step is clipped to land on it; that step still runs in full, and
// the disk is frozen (FB_DONE) when the next step's scalar work finds it
// there.  Empty slots (zeroed descriptors) are passed over.
static __global__ void kb_scalars(const fb_disk_dev *ds, fb_psys *ps, const int *dl, int n, double DT) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int i = dl ? dl[t] : t;
  const fb_disk_dev &D = ds[i];
  if (D.nx == 0) return;
  unsigned long long *dm = (unsigned long long *)D.dtmin;
  // in place: a step touches a tenth of either structure
  fb_scalars *sc = D.scal_dev;
  fb_psys *S = ps + i;
  if (!sc->skip) {
    const double cflmin = __longlong_as_double((long long)dm[0]);
    if (S->status == FB_DONE) {
      sc->skip = 1;
    } else if (dm[1] != 0ull) {
      S->status = FB_ERR_NONFINITE;
      sc->skip = 1;
    } else if (fb_psys_step(S, cflmin, S->t_end > 0.0 ? S->t_end : DT, sc, D.feeldisk ? D.facc : nullptr) < 0.0) {
      sc->skip = 1;
    } else if (S->t_end > 0.0 && S->dtemp >= S->t_end) {
      S->status = FB_DONE;
    }
  }
  dm[0] = 0x4415AF1D78B58C40ULL;  // 1e20, the MIN reduction start (define.h:165)
}

}  // namespace fb

using namespace fb;

#define FB_MAX_CHAINS 8
/* FP32 batches step as 4 concurrent chains (64 disks: 0.460 -> 0.402 ms a step
   against one); FP64 batches, whose stage kernels fill the GPU on
   their own, as one */
#define FB_DEFAULT_CHAINS_F32 4
#define FB_DEFAULT_CHAINS_F64 1

// Slots: state[i] 0 empty, 1 reserved (created, not activated), 2 active.
// n is the capacity; the work lists cover the active slots only.
struct fb_batch {
  int n, precision, device, is3d, nfluids;
  std::vector<int> state;
  std::vector<double> t_end;
  int dirty;
  char *arena;   // one allocation lent to the members of fb_batch_create (or null)
  cudaStream_t stream;
  std::vector<fb_disk *> disks;
  fb_disk_dev *d_disks;
  fb_psys *d_psys;
  int4 *items[ST_N];
  int nitems[ST_N];
  /* concurrent step chains: the active disks split into nchains groups of
     about equal cells, each group stepped on its own stream with its own work
     lists (chain c: citems[c], its disks cdisks[c]), so that one group's
     latency-bound launches (the scalar step, reductions, boundaries, launch
     tails) overlap another's throughput-bound ones */
  void *lists;    /* one device allocation holding every work list below */
  void *h_act;    /* page-locked staging of the members' activation uploads */
  int force_np;   /* planet indices that feel the disk in some member (0: none) */
  int nchains;
  cudaStream_t cstream[FB_MAX_CHAINS];
  cudaEvent_t ev_fork, ev_join[FB_MAX_CHAINS];
  int4 *citems[FB_MAX_CHAINS][ST_N];
  int ncitems[FB_MAX_CHAINS][ST_N];
  int *cdisks[FB_MAX_CHAINS];
  int ncdisks[FB_MAX_CHAINS];
  std::vector<int> chain_of;
  long long columns[2];   /* the column sweeps' work: columns of the active disks, and the longest's cells */
  int cells[2];
  int rings;    /* rings of the active disks */
  long long tile_layers;   /* the 3D source stage's tiles x layers */
  int rows_x;   /* rings a warp of the azimuthal sweep marches over */
  cudaGraphExec_t exec;
  int graph_steps;
  double graph_dt;
};

static int tiles(fb_batch *B, int st, std::vector<int4> &v, int chain = -1) {
  for (int di = 0; di < B->n; di++) {
    if (B->state[di] != 2) continue;
    if (chain >= 0 && B->chain_of[di] != chain) continue;
    const fb_disk_dev &D = *fb_disk_internal_dev(B->disks[di]);
    const int nx = D.nx, ny = D.ny, nz = D.nz, sy = D.sy, sz = D.sz;
    // FP32 2D disks whose rings hold a multiple of 4 cells: CFL four cells a
    // thread (fb_sources32.cuh)
    const bool quad = !D.is3d && B->precision == FB_FP32 && nx % 4 == 0;
    dim3 g(1, 1, 1);
    switch (st) {
      case ST_ROWSUM:
        if (B->precision == FB_FP64) {   // rings per warp from the whole batch's rings
          const int R = rs_rings(B->rings), per = RS_WARPS * R;
          for (int x = 0; x < (sy * sz + per - 1) / per; x++) v.push_back(make_int4(di, x, R, 0));
          g = dim3(0);
        } else {
          g = dim3(rw_ctas(sy * sz));
        }
        break;
      case ST_CFL:
        if (quad) g = dim3(0);
        else if (!D.is3d && B->precision == FB_FP32) g = dim3((nx + 127) / 128, (ny + CFL32_R - 1) / CFL32_R);
        else g = dim3((ny + CFL_R - 1) / CFL_R, D.is3d ? nz : 1);
        break;
      case ST_SOURCES:
        if (D.is3d) {   // layers per march from the whole batch's work (the results do not depend on it)
          const int layers = s3_layers(B->tile_layers, nz), ty = s3_ty(B->precision);
          for (int z = 0; z < (nz + layers - 1) / layers; z++)
            for (int y = 0; y < (ny + ty - 1) / ty; y++)
              for (int x = 0; x < (nx + S3_TX - 1) / S3_TX; x++) v.push_back(make_int4(di, x, y, z | layers << 16));
          g = dim3(0);
        }
        else if (B->precision == FB_FP32) {   // rows per march from the whole batch's cells, as the item's z
          const int rows = s32_rows(B->columns[0] * B->cells[0] * B->nfluids);
          for (int y = 0; y < (ny + rows - 1) / rows; y++)
            for (int x = 0; x < (nx + S32_COLS - 1) / S32_COLS; x++) v.push_back(make_int4(di, x, y, rows));
          g = dim3(0);
        }
        else g = dim3((nx + SRC2_TX - 1) / SRC2_TX, (ny + SRC2_TY - 1) / SRC2_TY);
        break;
      case ST_BND_Z: g = D.is3d ? dim3((nx + BND_BX - 1) / BND_BX, sy, 6) : dim3(0); break;
      case ST_BND_Y: g = D.is3d ? dim3((nx + BND_BX - 1) / BND_BX, 6, sz) : dim3(0); break;
      case ST_COLL: g = D.nfluids > 1 ? dim3((nx + 127) / 128, sy - 1, D.is3d ? sz - 1 : 1) : dim3(0); break;
      case ST_Z: case ST_Y: {
        if (st == ST_Z && !D.is3d) { g = dim3(0); break; }
        const int dir = st == ST_Y ? 0 : 1;
        // segments from the whole batch's columns (the results do not depend on them)
        const int rows = col_rows(B->columns[dir], B->cells[dir], D.tile_ns);
        const dim3 t = colm_grid(D, dir, rows);
        for (unsigned z = 0; z < t.z; z++)
          for (unsigned y = 0; y < t.y; y++)
            for (unsigned x = 0; x < t.x; x++) v.push_back(make_int4(di, (int)x, (int)(y | (unsigned)rows << 24), (int)z));
        g = dim3(0);
        break;
      }
      case ST_X: {
        const int strips = B->precision == FB_FP64 ? xs_strips<XsC<double>::C>(nx) : xs_strips<XsC<float>::C>(nx);
        const int n = xs_ctas(strips, xs_rings(D), B->rows_x);
        for (int x = 0; x < n; x++) v.push_back(make_int4(di, x, B->rows_x, 0));
        g = dim3(0);
        break;
      }
      case ST_FORCE: {
        const int nr = ny * (D.is3d ? nz : 1);
        g = D.feeldisk ? dim3(nr) : dim3(0);
        break;
      }
      case ST_CFL4:
        g = quad ? dim3(cfl32q_ctas(nx, ny)) : dim3(0);
        break;
      case ST_NEWVEL:
        g = D.is3d ? dim3((nx + NV_BX - 1) / NV_BX, (ny + NV_R - 1) / NV_R, nz) : dim3(0);
        break;
    }
    for (unsigned z = 0; z < g.z; z++)
      for (unsigned y = 0; y < g.y; y++)
        for (unsigned x = 0; x < g.x; x++) v.push_back(make_int4(di, (int)x, (int)y, (int)z));
  }
  return (int)v.size();
}

// optional per-launch timing of an eager (uncaptured) step
struct Prof {
  cudaEvent_t ev[40];
  const char *name[40];
  int n;
};
extern Prof *g_prof;
static void pmark(cudaStream_t st, const char *name) {
  if (!g_prof || g_prof->n >= 40) return;
  cudaEventCreate(&g_prof->ev[g_prof->n]);
  cudaEventRecord(g_prof->ev[g_prof->n], st);
  g_prof->name[g_prof->n++] = name;
}

// T: compute type of the source stage; TC, TX, TN, TF: of the column sweeps,
// the azimuthal sweep, NewVelocity and the CFL's per-cell limits (its
// minimum is always FP64); S: storage type.
// chain < 0: every active disk on the batch's stream (one chain); else the
// disks of that chain on its stream.
template <typename T, typename S, typename TC = T, typename TX = T, typename TN = T, typename TF = T>
static int launch_step(fb_batch *B, double DT, int chain) {
  int4 *const *items = chain < 0 ? B->items : B->citems[chain];
  const int *nitems = chain < 0 ? B->nitems : B->ncitems[chain];
  if (nitems[ST_ROWSUM] == 0) return 0;  // no active disk
  cudaStream_t st = chain < 0 ? B->stream : B->cstream[chain];
  pmark(st, "start");
  const fb_disk_dev *ds = B->d_disks;
  const int nf = B->nfluids;
  auto grid = [&](int s) { return dim3((unsigned)nitems[s], (unsigned)nf); };
  kb_rowsum<S><<<grid(ST_ROWSUM), sizeof(S) == 8 ? 32 * RS_WARPS : 32 * RW_WARPS, 0, st>>>(ds, items[ST_ROWSUM], 0);
  pmark(st, "rowsum");
  if (nitems[ST_CFL4]) kb_cfl_cyl32q<<<grid(ST_CFL4), Q32_T, 0, st>>>(ds, items[ST_CFL4]);
  if (nitems[ST_CFL]) {
    if (!B->is3d && sizeof(S) == 4) kb_cfl_cyl32<<<grid(ST_CFL), 128, 0, st>>>(ds, items[ST_CFL]);
    else kb_cfl<TF, S><<<grid(ST_CFL), 256, 0, st>>>(ds, items[ST_CFL]);
  }
  pmark(st, "cfl");
  {
    const int nd = chain < 0 ? B->n : B->ncdisks[chain];
    const int *dl = chain < 0 ? nullptr : B->cdisks[chain];
    if (nitems[ST_FORCE]) {   // planets that feel the disk, one planet index at a time
      for (int n = 0; n < B->force_np; n++) {
        kb_disk_force_rings<S><<<dim3((unsigned)nitems[ST_FORCE]), DF_T, 0, st>>>(ds, B->d_psys, items[ST_FORCE], n);
        kb_disk_force_fold<<<nd, DF_T, 0, st>>>(ds, B->d_psys, dl, n);
      }
      pmark(st, "disk_force");
    }
    kb_scalars<<<(nd + 63) / 64, 64, 0, st>>>(ds, B->d_psys, dl, nd, DT);
  }
  pmark(st, "scalars");
  if (B->is3d) {
    const int e = s3_allow<kb_sources_sph<S>, S>(B->device);
    if (e) return e;
    kb_sources_sph<S><<<grid(ST_SOURCES), S3<S>::T, sizeof(S3Shared<S>), st>>>(ds, items[ST_SOURCES]);
  } else if constexpr (sizeof(S) == 4) {
    kb_sources_cyl32<<<grid(ST_SOURCES), S32_WARPS * 32, 0, st>>>(ds, items[ST_SOURCES]);
  } else {
    kb_sources_cyl<<<grid(ST_SOURCES), SRC2_TX * SRC2_TY, 0, st>>>(ds, items[ST_SOURCES]);
  }
  pmark(st, "sources");
  if (B->is3d) {   // 2D: within the source stage
    kb_bnd<T, S><<<grid(ST_BND_Z), BND_BX, 0, st>>>(ds, items[ST_BND_Z], 1, 1);
    kb_bnd<T, S><<<grid(ST_BND_Y), BND_BX, 0, st>>>(ds, items[ST_BND_Y], 1, 0);
    pmark(st, "bnd_vtemp");
  }
  if (nf > 1 && nitems[ST_COLL]) {  // implicit drag between the fluids
    const int4 *it = items[ST_COLL];
    switch (nf) {
      case 2: kb_collisions<T, 2, S><<<dim3((unsigned)nitems[ST_COLL]), 128, 0, st>>>(ds, it); break;
      case 3: kb_collisions<T, 3, S><<<dim3((unsigned)nitems[ST_COLL]), 128, 0, st>>>(ds, it); break;
      case 4: kb_collisions<T, 4, S><<<dim3((unsigned)nitems[ST_COLL]), 128, 0, st>>>(ds, it); break;
      case 5: kb_collisions<T, 5, S><<<dim3((unsigned)nitems[ST_COLL]), 128, 0, st>>>(ds, it); break;
      case 6: kb_collisions<T, 6, S><<<dim3((unsigned)nitems[ST_COLL]), 128, 0, st>>>(ds, it); break;
      case 7: kb_collisions<T, 7, S><<<dim3((unsigned)nitems[ST_COLL]), 128, 0, st>>>(ds, it); break;
      default: kb_collisions<T, 8, S><<<dim3((unsigned)nitems[ST_COLL]), 128, 0, st>>>(ds, it); break;
    }
    pmark(st, "collisions");
  }
  kb_rowsum<S><<<grid(ST_ROWSUM), sizeof(S) == 8 ? 32 * RS_WARPS : 32 * RW_WARPS, 0, st>>>(ds, items[ST_ROWSUM], 1);
  pmark(st, "rowsum_vtemp");
  if (B->is3d) {
    kb_sweep_colm<TC, 1, true><<<grid(ST_Z), COL_T, 0, st>>>(ds, items[ST_Z]);
    kb_sweep_colm<TC, 0, true><<<grid(ST_Y), COL_T, 0, st>>>(ds, items[ST_Y]);
  } else {
    kb_sweep_colm<TC, 0, false><<<grid(ST_Y), COL_T, 0, st>>>(ds, items[ST_Y]);
  }
  pmark(st, "sweep_cols");
  if (B->is3d) kb_sweep_xs<TX, 6, false><<<grid(ST_X), 32 * XS_WARPS, xs_smem<TX, XsC<TX>::C>(6), st>>>(ds, items[ST_X]);
  else kb_sweep_xs<TX, 4, true><<<grid(ST_X), 32 * XS_WARPS, xs_smem<TX, XsC<TX>::C>(4), st>>>(ds, items[ST_X]);
  pmark(st, "sweep_x");
  if (B->is3d) {   // 2D: the new velocities and the state's ghosts are the azimuthal sweep's
    kb_newvel<TN, S><<<grid(ST_NEWVEL), NV_BX, 0, st>>>(ds, items[ST_NEWVEL]);
    pmark(st, "newvel");
    kb_bnd<T, S><<<grid(ST_BND_Z), BND_BX, 0, st>>>(ds, items[ST_BND_Z], 0, 1);
    kb_bnd<T, S><<<grid(ST_BND_Y), BND_BX, 0, st>>>(ds, items[ST_BND_Y], 0, 0);
    pmark(st, "bnd");
  }
  return (int)cudaGetLastError();
}

