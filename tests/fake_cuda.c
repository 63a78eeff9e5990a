/* A CUDA runtime of the host for tests of the one-disk driver (fb_host.c)
 * without a GPU.  Device memory is host memory.  A stream is a queue of
 * operations that run, in order, when somebody waits for the stream -- the
 * latest moment the runtime promises -- except that a CFL launch runs the
 * queue up to and with itself at once (unless fake_lazy_cfl), as a step's
 * begin waits for its report.  A capture collects the operations of its
 * stream, whoever queues them; what the runtime refuses of a capturing stream
 * (waits, queries, graph launches) is refused.  "Kernels" only do what the
 * driver relies on: the CFL launch reports, the source launch notes the time
 * step it found in the device's scalars. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include "fargo_b200.h"
#include "fb_dev.h"

typedef struct { int kind; void *dst; const void *src; size_t n; const fb_disk_dev *d; fb_disk_dev copy; } Op;
enum { COPY, SOURCES, CFL, COUNT, OTHER, GRAPH };
typedef struct { Op *op; int n, cap; } Ops;
typedef struct { Ops q; Ops *capture; } Stream;

static void add(Ops *q, Op o) {
  if (q->n == q->cap) q->op = (Op *)realloc(q->op, sizeof(Op) * (size_t)(q->cap = q->cap ? 2 * q->cap : 64));
  q->op[q->n++] = o;
}

/* what a test reads and sets */
double fake_dts[256];          /* time steps the source launches found */
int fake_ndts, fake_counted, fake_queries, fake_syncs, fake_yields, fake_lazy_cfl, fake_flags;
void (*fake_on_capture)(void);

static void run_op(const Op *o) {
  int k;
  switch (o->kind) {
    case COPY: memmove(o->dst, o->src, o->n); break;
    case SOURCES: if (fake_ndts < 256) fake_dts[fake_ndts++] = o->copy.scal_dev->dt; break;
    case CFL: {
      volatile double *h = o->copy.pin;
      h[0] = 0.125;
      h[1] = 0.0;
      h[2] = o->copy.pin[PIN_BEGIN / 8 + sizeof(fb_scalars) / 8 + 1];
      break;
    }
    case COUNT: fake_counted++; break;
    case GRAPH:
      for (k = 0; k < ((Ops *)o->src)->n; k++) run_op(&((Ops *)o->src)->op[k]);
      break;
    default: break;
  }
}
static void drain(Stream *s) {
  int k;
  for (k = 0; k < s->q.n; k++) run_op(&s->q.op[k]);
  s->q.n = 0;
}
static void queue(void *stream, Op o) {
  Stream *s = (Stream *)stream;
  int k, cfl = o.kind == CFL;
  if (s->capture) { add(s->capture, o); return; }
  add(&s->q, o);
  if (o.kind == GRAPH)
    for (k = 0; k < ((Ops *)o.src)->n; k++) cfl |= ((Ops *)o.src)->op[k].kind == CFL;
  if (cfl && !fake_lazy_cfl) drain(s);
}
void fake_count(void *stream) { Op o = {COUNT, 0, 0, 0, 0, {0}}; queue(stream, o); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)calloc(1, sizeof(Stream)); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { drain((Stream *)s); free(((Stream *)s)->q.op); free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (((Stream *)s)->capture) return cudaErrorStreamCaptureUnsupported;
  fake_syncs++;
  drain((Stream *)s);
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t s) {
  if (((Stream *)s)->capture) return cudaErrorStreamCaptureUnsupported;
  if (++fake_queries > 1000) drain((Stream *)s);   /* a driver that only polls gets there in the end */
  return ((Stream *)s)->q.n ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *st) {
  *st = ((Stream *)s)->capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) {
  (void)m;
  if (((Stream *)s)->capture) return cudaErrorIllegalState;
  ((Stream *)s)->capture = (Ops *)calloc(1, sizeof(Ops));
  if (fake_on_capture) fake_on_capture();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
  *g = (cudaGraph_t)((Stream *)s)->capture;
  ((Stream *)s)->capture = NULL;
  return *g ? cudaSuccess : cudaErrorIllegalState;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long f) {
  Ops *c = (Ops *)calloc(1, sizeof(Ops));
  int k;
  (void)f;
  for (k = 0; k < ((Ops *)g)->n; k++) add(c, ((Ops *)g)->op[k]);
  *e = (cudaGraphExec_t)c;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(((Ops *)g)->op); free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { free(((Ops *)e)->op); free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
  Op o = {GRAPH, 0, e, 0, 0, {0}};
  if (((Stream *)s)->capture) return cudaErrorStreamCaptureUnsupported;
  queue(s, o);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, enum cudaMemcpyKind k, cudaStream_t s) {
  Op o = {COPY, dst, src, n, 0, {0}};
  (void)k;
  queue(s, o);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, enum cudaMemcpyKind k, cudaStream_t st) {
  size_t r;
  (void)k;
  (void)st;
  for (r = 0; r < h; r++) memmove((char *)d + r * dp, (const char *)s + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) { (void)s; memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { (void)k; memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceFlags(unsigned *f) { *f = (unsigned)fake_flags; return cudaSuccess; }
int fake_yield(void) { fake_yields++; return 0; }   /* fb_host.c is compiled with sched_yield as this */
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorStreamCaptureUnsupported ? "not permitted when stream is capturing" : "error"; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *t = 0; return cudaSuccess; }

static int launch(int kind, const fb_disk_dev *d, void *s) {
  Op o;
  memset(&o, 0, sizeof o);
  o.kind = kind;
  o.copy = *d;   /* kernels take the descriptor by value */
  queue(s, o);
  return 0;
}
#define FAKE(SUF)                                                                                     \
  int fb_launch_rowsum_##SUF(const fb_disk_dev *d, int w, void *s) { (void)w; return launch(OTHER, d, s); } \
  int fb_launch_cfl_##SUF(const fb_disk_dev *d, void *s) { return launch(CFL, d, s); }                \
  int fb_launch_sources_##SUF(const fb_disk_dev *d, void *s) { return launch(SOURCES, d, s); }        \
  int fb_launch_bnd_##SUF(const fb_disk_dev *d, int v, void *s) { (void)v; return launch(OTHER, d, s); } \
  int fb_launch_sweep_cols_##SUF(const fb_disk_dev *d, void *s) { return launch(OTHER, d, s); }       \
  int fb_launch_sweep_x_##SUF(const fb_disk_dev *d, void *s) { return launch(OTHER, d, s); }          \
  int fb_launch_newvel_##SUF(const fb_disk_dev *d, void *s) { return launch(OTHER, d, s); }           \
  int fb_launch_collisions_##SUF(const fb_disk_dev *d, void *s) { return launch(OTHER, d, s); }       \
  int fb_launch_substep3_##SUF(const fb_disk_dev *d, void *s) { return launch(OTHER, d, s); }         \
  int fb_launch_dust_diffusion_##SUF(const fb_disk_dev *d, void *s) { return launch(OTHER, d, s); }   \
  int fb_launch_mass_##SUF(const fb_disk_dev *d, int f, double *p, double *o, void *s) {              \
    (void)f; (void)p; (void)o; return launch(OTHER, d, s); }                                          \
  int fb_launch_disk_force_##SUF(const fb_disk_dev *d, const double *p, double *r, double *o, void *s) { \
    (void)p; (void)r; (void)o; return launch(OTHER, d, s); }
FAKE(f64)
FAKE(f32)
int fb_launch_convert(void *d, const void *s, size_t n, int t, void *st) { (void)d; (void)s; (void)n; (void)t; (void)st; return 0; }
int fb_launch_convert_segs(double *st, const fb_segs *g, int t, void *s) { (void)st; (void)g; (void)t; (void)s; return 0; }
int fb_launch_ring_mean(double *o, const double *s, int nx, int n, void *st) { (void)o; (void)s; (void)nx; (void)n; (void)st; return 0; }
int fb_launch_bg_diffs(const fb_disk_dev *d, int f, void *s) { (void)d; (void)f; (void)s; return 0; }
