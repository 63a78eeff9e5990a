// FP32 instantiation of the stage kernels (transport, 2D sources and the CFL's
// limits in FP32; 3D sources, ghosts, drag, ring means, shift and the disk force
// stay FP64 inside the kernels).
#define FB_REAL double
#define FB_REAL_TR float
#define FB_STORE float
#define FB_SUF f32
#include "fb_launch.cuh"
