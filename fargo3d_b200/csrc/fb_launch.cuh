// fb_launch.cuh -- host-side launchers of the stage kernels for one precision.
// Included once per precision by fb_kernels_f64.cu / fb_kernels_f32.cu with
// FB_REAL and FB_SUF defined.
#include "fb_kernels.cuh"

namespace fb {

// Each launch covers all the disk's fluids (one after the other they would
// cost a launch each, with grids that leave most of the chip idle).  Where the
// grid's third index counts layers or segments as well (per: those of one
// fluid), it ends at 65535: launch(disk, fluids) is then called for as many
// fluids at a time as fit.
template <typename F>
static int by_fluids(const fb_disk_dev *d, int per, F launch) {
  const int nf = d->nfluids, most = per < 65535 ? 65535 / per : 1;
  if (nf <= most) {
    launch(*d, nf);
    return (int)cudaGetLastError();
  }
  fb_disk_dev part = *d;
  for (int f0 = 0; f0 < nf; f0 += most) {
    part.nfluids = nf - f0 < most ? nf - f0 : most;
    for (int f = 0; f < part.nfluids; f++) part.fl[f] = d->fl[f0 + f];
    launch(part, part.nfluids);
    const int e = (int)cudaGetLastError();
    if (e) return e;
  }
  return 0;
}

template <typename T, typename S>
static int launch_rowsum(const fb_disk_dev *d, int which, cudaStream_t st) {
  const int nring = d->sy * d->sz, nf = d->nfluids;
  if (d->precision != FB_FP64) k_rowsum_warp<S><<<dim3(rw_ctas(nring), nf), 32 * RW_WARPS, 0, st>>>(*d, which);
  else k_rowsum<<<dim3(rs_ctas(nring), nf), 32 * RS_WARPS, 0, st>>>(*d, which);
  return (int)cudaGetLastError();
}

template <typename T, typename S>
static int launch_cfl(const fb_disk_dev *d, cudaStream_t st) {
  if constexpr (sizeof(S) == 4) {
    if (!d->is3d) {   // FP32 2D (fb_sources32.cuh)
      if (d->nx % 4 == 0) k_cfl_cyl32q<<<dim3(cfl32q_ctas(d->nx, d->ny), d->nfluids), Q32_T, 0, st>>>(*d);
      else k_cfl_cyl32<<<dim3((d->nx + 127) / 128, (d->ny + CFL32_R - 1) / CFL32_R, d->nfluids), 128, 0, st>>>(*d);
      return (int)cudaGetLastError();
    }
  }
  k_cfl<T, S><<<dim3(d->ny, d->is3d ? d->nz : 1, d->nfluids), 256, 0, st>>>(*d);
  return (int)cudaGetLastError();
}

template <typename T, typename S>
static int launch_sources(const fb_disk_dev *d, cudaStream_t st) {
  const int nx = d->nx, ny = d->ny, nf = d->nfluids;
  if (d->is3d) {
    int dev = 0, e;
    cudaGetDevice(&dev);
    if ((e = s3_allow<k_sources_sph<S>, S>(dev))) return e;
    const int layers = s3_layers((long long)s3_tiles(*d) * d->nz * nf, d->nz);
    const int segs = (d->nz + layers - 1) / layers;
    return by_fluids(d, segs, [&](const fb_disk_dev &D, int n) {
      dim3 grid((nx + S3_TX - 1) / S3_TX, (ny + S3<S>::TY - 1) / S3<S>::TY, segs * n);
      k_sources_sph<S><<<grid, S3<S>::T, sizeof(S3Shared<S>), st>>>(D, layers);
    });
  } else if constexpr (sizeof(S) == 4) {   // FP32 storage: FP32 arithmetic, column-marching warps
    const int rows = s32_rows((long long)nx * ny * nf);
    k_sources_cyl32<<<dim3((nx + S32_COLS - 1) / S32_COLS, (ny + rows - 1) / rows, nf), S32_WARPS * 32, 0, st>>>(*d, rows);
  } else {
    // adiabatic: one more row (the outer edge face, read by SubStep3)
    k_sources_cyl<<<dim3((nx + SRC2_TX - 1) / SRC2_TX, (ny + d->adiabatic + SRC2_TY - 1) / SRC2_TY, nf),
                    SRC2_TX * SRC2_TY, 0, st>>>(*d);
  }
  return (int)cudaGetLastError();
}

template <typename T, typename S>
static int launch_bnd(const fb_disk_dev *d, int vtemp, cudaStream_t st) {
  const int bx = 128, gx = (d->nx + bx - 1) / bx;
  if (d->is3d) k_bnd_z<T, S><<<dim3(gx, d->sy, 6 * d->nfluids), bx, 0, st>>>(*d, vtemp);
  return by_fluids(d, d->sz, [&](const fb_disk_dev &D, int n) {
    k_bnd_y<T, S><<<dim3(gx, 6, D.sz * n), bx, 0, st>>>(D, vtemp);
  });
}

// radial sweep; in 3D the colatitude sweep (V_temp into set A) before it (set
// A into set B)
template <typename T, typename S>
static int launch_sweep_cols(const fb_disk_dev *d, cudaStream_t st) {
  auto sweep = [&](int dir, auto kernel) {
    const int rows = colm_rows(*d, dir);
    const dim3 g = colm_grid(*d, dir, rows);
    return by_fluids(d, (int)g.z, [&](const fb_disk_dev &D, int n) {
      kernel<<<dim3(g.x, g.y, g.z * n), COL_T, 0, st>>>(D, rows);
    });
  };
  if (d->is3d) {
    const int e = sweep(1, k_sweep_colm<T, 1, true, false>);
    return e ? e : sweep(0, k_sweep_colm<T, 0, true, false>);
  }
  if (d->adiabatic) {   // adiabatic disks transport their energy into e_a as a fifth quantity
    if constexpr (sizeof(T) == 8) return sweep(0, k_sweep_colm<T, 0, false, true>);
    return (int)cudaErrorInvalidValue;
  }
  return sweep(0, k_sweep_colm<T, 0, false, false>);
}

// The azimuthal sweep; in 2D with NewVelocity and Stockholm (fb_sweepx.cuh).
template <typename T, typename S>
static int launch_sweep_x(const fb_disk_dev *d, cudaStream_t st) {
  if (!ring_fits(*d)) return (int)cudaErrorInvalidValue;
  constexpr int C = XsC<T>::C, TH = 32 * XS_WARPS;
  const int strips = xs_strips<C>(d->nx), rings = xs_rings(*d);
  const int rows = xs_rows((long long)strips * rings * d->nfluids);
  const dim3 grid(xs_ctas(strips, rings, rows), d->nfluids);
  if (d->is3d) k_sweep_xs<T, 6, false><<<grid, TH, xs_smem<T, C>(6), st>>>(*d, rows);
  else if (!d->adiabatic) k_sweep_xs<T, 4, true><<<grid, TH, xs_smem<T, C>(4), st>>>(*d, rows);
  else if constexpr (sizeof(T) == 8)   // the energy is the fifth transported quantity
    k_sweep_xs<T, 5, true><<<grid, TH, xs_smem<T, C>(5), st>>>(*d, rows);
  return (int)cudaGetLastError();
}

// NewVelocity + Stockholm of 3D disks, from the azimuthal sweep's set A (2D
// disks get their new state from the sweep itself)
template <typename T, typename S>
static int launch_newvel(const fb_disk_dev *d, cudaStream_t st) {
  if (!d->is3d) return 0;
  return by_fluids(d, d->nz, [&](const fb_disk_dev &D, int n) {
    k_newvel<T, S><<<dim3((D.nx + 127) / 128, D.ny, D.nz * n), 128, 0, st>>>(D);
  });
}

// implicit drag of all fluids (fluid count 2..FB_MAXFLUIDS)
template <typename T, typename S>
static int launch_collisions(const fb_disk_dev *d, cudaStream_t st) {
  const dim3 g((d->nx + 127) / 128, d->sy - 1, d->is3d ? d->sz - 1 : 1);
  switch (d->nfluids) {
    case 2: k_collisions<T, 2, S><<<g, 128, 0, st>>>(*d); break;
    case 3: k_collisions<T, 3, S><<<g, 128, 0, st>>>(*d); break;
    case 4: k_collisions<T, 4, S><<<g, 128, 0, st>>>(*d); break;
    case 5: k_collisions<T, 5, S><<<g, 128, 0, st>>>(*d); break;
    case 6: k_collisions<T, 6, S><<<g, 128, 0, st>>>(*d); break;
    case 7: k_collisions<T, 7, S><<<g, 128, 0, st>>>(*d); break;
    case 8: k_collisions<T, 8, S><<<g, 128, 0, st>>>(*d); break;
    default: return (int)cudaErrorInvalidValue;
  }
  return (int)cudaGetLastError();
}

// DustDiffusion_Main of the dust fluids (FP64, 2D): the diffused density into
// rho_a (free until transport), copied back over the active rows, then the
// density's ghosts (FillGhosts(DENS))
template <typename T, typename S>
static int launch_dust_diffusion(const fb_disk_dev *d, cudaStream_t st) {
  if constexpr (sizeof(S) == 8) {
    if (!d->dust_diffusion || d->nfluids < 2 || d->is3d) return (int)cudaErrorInvalidValue;
    const int gx = (d->nx + 127) / 128, nd = d->nfluids - 1;
    k_dust_diffusion<double, double><<<dim3(gx, d->ny, nd), 128, 0, st>>>(*d);
    k_copy_rows<double><<<dim3(gx, d->ny, nd), 128, 0, st>>>(*d);
    k_bnd_rho_y<double, double><<<dim3(gx, 6, nd), 128, 0, st>>>(*d);
    return (int)cudaGetLastError();
  }
  return (int)cudaErrorInvalidValue;
}

// SubStep3 of an adiabatic disk (FP64 storage and arithmetic).
// (The FP32 translation unit, which contracts products and sums, must not hold
// a copy of these FP64 kernels: two copies of one kernel name are one to the
// runtime, and which of them runs is then not defined.)
template <typename T, typename S>
static int launch_substep3(const fb_disk_dev *d, cudaStream_t st) {
  if constexpr (sizeof(S) == 8) {
    if (!d->adiabatic) return (int)cudaErrorInvalidValue;
    k_substep3<double><<<dim3((d->nx + 127) / 128, d->ny, d->nfluids), 128, 0, st>>>(*d);
    return (int)cudaGetLastError();
  }
  return (int)cudaErrorInvalidValue;
}

// the disk's acceleration at the point pt (device: x, y, z, smoothing;
// ComputeAccel), FP64 in every precision
template <typename S>
static int launch_disk_force(const fb_disk_dev *d, const double *pt, double *ring3, double *out3, cudaStream_t st) {
  k_disk_force_rings<S><<<d->ny * (d->is3d ? d->nz : 1), DF_T, 0, st>>>(*d, pt, ring3);
  k_disk_force_fold<<<1, DF_T, 0, st>>>(*d, pt, ring3, out3);
  return (int)cudaGetLastError();
}

// compensated mass of one fluid into out (device double); part: 2 x active
// rings doubles of scratch
template <typename S>
static int launch_mass(const fb_disk_dev *d, int f, double *part, double *out, cudaStream_t st) {
  Dims m = dims_of(*d);
  const int nr = m.ny * (m.is3d ? m.nz : 1);
  k_mass_rings<S><<<(nr + 7) / 8, 256, 0, st>>>(m, geo_of<double>(d->geomd), (const S *)d->fl[f].rho, part);
  k_mass_fold<<<1, 256, 0, st>>>(part, nr, out);
  return (int)cudaGetLastError();
}

}  // namespace fb

#define FB_CAT2(a, b) a##_##b
#define FB_CAT(a, b) FB_CAT2(a, b)

extern "C" {
int FB_CAT(fb_launch_rowsum, FB_SUF)(const fb_disk_dev *d, int which, void *s) {
  return fb::launch_rowsum<FB_REAL, FB_STORE>(d, which, (cudaStream_t)s);
}
int FB_CAT(fb_launch_cfl, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_cfl<FB_REAL_TR, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_sources, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_sources<FB_REAL, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_bnd, FB_SUF)(const fb_disk_dev *d, int vtemp, void *s) {
  return fb::launch_bnd<FB_REAL, FB_STORE>(d, vtemp, (cudaStream_t)s);
}
int FB_CAT(fb_launch_sweep_cols, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_sweep_cols<FB_REAL_TR, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_sweep_x, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_sweep_x<FB_REAL_TR, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_newvel, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_newvel<FB_REAL_TR, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_collisions, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_collisions<FB_REAL, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_dust_diffusion, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_dust_diffusion<FB_REAL, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_substep3, FB_SUF)(const fb_disk_dev *d, void *s) {
  return fb::launch_substep3<FB_REAL, FB_STORE>(d, (cudaStream_t)s);
}
int FB_CAT(fb_launch_mass, FB_SUF)(const fb_disk_dev *d, int fluid, double *part, double *out, void *s) {
  return fb::launch_mass<FB_STORE>(d, fluid, part, out, (cudaStream_t)s);
}
int FB_CAT(fb_launch_disk_force, FB_SUF)(const fb_disk_dev *d, const double *pt, double *ring3, double *out3, void *s) {
  return fb::launch_disk_force<FB_STORE>(d, pt, ring3, out3, (cudaStream_t)s);
}
}
