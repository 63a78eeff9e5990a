// FP32 batched stage kernels: FP32 storage.  2D sources, the transport stages,
// NewVelocity and the CFL's per-cell limits compute in FP32 (approximate
// division and root but for NewVelocity's division, div_rn); 3D sources, ghosts,
// drag, shift, ring means, planets and the CFL minimum in FP64.
#include "fb_batch.cuh"
#ifndef FB_TC
#define FB_TC float
#endif
#ifndef FB_TX
#define FB_TX float
#endif
#ifndef FB_TN
#define FB_TN float
#endif
#ifndef FB_TF
#define FB_TF float
#endif
extern "C" int fb_batch_launch_step_f32(fb_batch *B, double DT, int chain) {
  return launch_step<double, float, FB_TC, FB_TX, FB_TN, FB_TF>(B, DT, chain);
}
