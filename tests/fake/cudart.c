/* A stand-in for the CUDA runtime, preloaded in front of it: device memory is
 * host memory, copies run at once, kernels do not run.  It lets the host side
 * of the library (planning, tables, launch configurations, batches) run
 * without a GPU and counts what the tests look at:
 *   fake_live_bytes        bytes allocated and not freed
 *   fake_launches          kernel launches that were accepted
 *   fake_unordered         launches on a non-blocking stream after a copy or
 *                          fill on the legacy stream that nothing waited for
 *                          (such a copy from pageable memory may return before
 *                          its data has arrived)
 *   fake_device_syncs      waits for the whole device, which fail, and spoil the
 *                          capture, while another thread captures a stream
 *   fake_lowered           cudaFuncSetAttribute calls that took dynamic shared
 *                          memory away from a kernel
 *   fake_surplus           launches of a sweep, whose CTAs walk over the tiles,
 *                          with more CTAs than the device holds at once
 *   fake_fail_mallocs(1)   lets every allocation fail
 */
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;
enum { OK = 0, INVALID = 1, OOM = 2 };
typedef struct { unsigned x, y, z; } dim;
typedef struct { int flags; } stream;

static long long live, launches, unordered, lowered, surplus, device_syncs;
static int failing, pending;
static __thread err_t last;

long long fake_live_bytes(void) { return live; }
long long fake_launches(void) { return launches; }
long long fake_unordered(void) { return unordered; }
long long fake_lowered(void) { return lowered; }
long long fake_surplus(void) { return surplus; }
long long fake_device_syncs(void) { return device_syncs; }
void fake_fail_mallocs(int on) { failing = on; }

/* ---- kernels: dynamic shared memory up to 48 KB less the static bytes unless
 * raised, to the opt-in maximum less them (static: a bound on what the batched
 * kernels, whose names start with kb_, and the others hold) */
#define OPTIN_SMEM 232448
#define SM_SMEM (228 * 1024)
static struct { const void *f; int dyn, fixed, sweep; } attr[1 << 16];
static unsigned at(const void *f) {
   unsigned h = (unsigned) (((uintptr_t) f >> 4) * 2654435761u) & 0xffff;
   while (attr[h].f && attr[h].f != f) h = (h + 1) & 0xffff;
   return h;
}
void **__cudaRegisterFatBinary(void *f) { static void *h; (void) f; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void) h; }
void __cudaUnregisterFatBinary(void **h) { (void) h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g) {
   (void) h; (void) v; (void) a; (void) n; (void) e; (void) s; (void) c; (void) g;
}
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *n, int l, void *t, void *b, void *bd, void *gd, int *w) {
   const unsigned k = at(f);
   (void) h; (void) d; (void) l; (void) t; (void) b; (void) bd; (void) gd; (void) w;
   attr[k].f = f;
   attr[k].fixed = strstr(n, "kb_") ? 1152 : 128;
   attr[k].dyn = 48 * 1024 - attr[k].fixed;
   attr[k].sweep = strstr(n, "k_sweep") || strstr(n, "kb_sweep");
}
err_t cudaFuncSetAttribute(const void *f, int a, int v) {
   const unsigned k = at(f);
   if (!attr[k].f || a != 8 || v < 0 || v > OPTIN_SMEM - attr[k].fixed) return INVALID;
   if (v < attr[k].dyn) lowered++;
   attr[k].dyn = v;
   return OK;
}
static err_t launch(const void *f, dim g, dim b, size_t smem, stream *s) {
   if (!g.x || !g.y || !g.z || !b.x || b.x * b.y * b.z > 1024 || smem > (size_t) attr[at(f)].dyn) return last = INVALID;
   if (pending && s && (s->flags & 1)) unordered++;
   if (attr[at(f)].sweep && g.x > 148 * (SM_SMEM / (smem + (size_t) attr[at(f)].fixed + 1024))) surplus++;
   launches++;
   return OK;
}
err_t cudaLaunchKernel(const void *f, dim g, dim b, void **args, size_t smem, stream *s) {
   (void) args;
   return launch(f, g, b, smem, s);
}
typedef struct { dim g, b; size_t smem; stream *s; void *attrs; unsigned n; } config;
err_t cudaLaunchKernelExC(const config *c, const void *f, void **args) { (void) args; return launch(f, c->g, c->b, c->smem, c->s); }
static __thread struct { dim g, b; size_t smem; void *s; } call;
unsigned __cudaPushCallConfiguration(dim g, dim b, size_t smem, void *s) { call.g = g; call.b = b; call.smem = smem; call.s = s; return 0; }
err_t __cudaPopCallConfiguration(dim *g, dim *b, size_t *smem, void *s) {
   *g = call.g; *b = call.b; *smem = call.smem; *(void **) s = call.s;
   return OK;
}

/* ---- memory */
err_t cudaMalloc(void **p, size_t n) {
   char *q;
   *p = NULL;
   if (failing) return OOM;
   q = calloc(1, n + 1024);
   if (!q) return OOM;
   *p = (void *) (((uintptr_t) q + 1023) & ~(uintptr_t) 511);
   ((size_t *) *p)[-1] = n;
   ((char **) *p)[-2] = q;
   live += (long long) n;
   return OK;
}
err_t cudaFree(void *p) {
   if (p) {
      live -= (long long) ((size_t *) p)[-1];
      free(((char **) p)[-2]);
   }
   return OK;
}
err_t cudaMemcpy(void *d, const void *s, size_t n, int kind) {
   memcpy(d, s, n);
   pending = kind != 2; /* a copy to the host waits for all legacy work */
   return OK;
}
err_t cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, stream *st) {
   memcpy(d, s, n);
   if (!st && kind != 2) pending = 1;
   return OK;
}
err_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); pending = 1; return OK; }
err_t cudaMemsetAsync(void *d, int v, size_t n, stream *st) {
   memset(d, v, n);
   if (!st) pending = 1;
   return OK;
}
err_t cudaGetSymbolAddress(void **p, const void *s) { (void) s; *p = NULL; return INVALID; }

/* ---- streams, events, graphs, the device */
err_t cudaStreamCreateWithFlags(stream **s, unsigned f) { *s = calloc(1, sizeof(stream)); (*s)->flags = (int) f; return OK; }
err_t cudaStreamCreateWithPriority(stream **s, unsigned f, int p) { (void) p; return cudaStreamCreateWithFlags(s, f); }
err_t cudaStreamDestroy(stream *s) { free(s); return OK; }
err_t cudaStreamSynchronize(stream *s) { if (!s) pending = 0; return OK; }
err_t cudaStreamWaitEvent(stream *s, void *e, unsigned f) { (void) s; (void) e; (void) f; return OK; }
err_t cudaStreamBeginCapture(stream *s, int m) { (void) s; (void) m; return OK; }
err_t cudaStreamEndCapture(stream *s, void **g) { (void) s; *g = malloc(1); return OK; }
err_t cudaGraphInstantiate(void **x, void *g, unsigned long long f) { (void) g; (void) f; *x = malloc(1); return OK; }
err_t cudaGraphDestroy(void *g) { free(g); return OK; }
err_t cudaGraphExecDestroy(void *x) { free(x); return OK; }
err_t cudaGraphLaunch(void *x, stream *s) { (void) x; (void) s; return OK; }
err_t cudaEventCreate(void **e) { *e = malloc(1); return OK; }
err_t cudaEventCreateWithFlags(void **e, unsigned f) { (void) f; return cudaEventCreate(e); }
err_t cudaEventDestroy(void *e) { free(e); return OK; }
err_t cudaEventRecord(void *e, stream *s) { (void) e; (void) s; return OK; }
err_t cudaEventSynchronize(void *e) { (void) e; return OK; }
err_t cudaEventQuery(void *e) { (void) e; return OK; }
err_t cudaEventElapsedTime(float *ms, void *a, void *b) { (void) a; (void) b; *ms = 1.f; return OK; }
err_t cudaDeviceSynchronize(void) { pending = 0; device_syncs++; return OK; }
err_t cudaSetDevice(int d) { return d == 0 ? OK : 101; }
err_t cudaGetDevice(int *d) { *d = 0; return OK; }
err_t cudaDeviceGetAttribute(int *v, int a, int d) {
   (void) d;
   *v = a == 16 ? 148 : (a == 97 ? OPTIN_SMEM : 0); /* SM count, opt-in shared memory */
   return OK;
}
err_t cudaDeviceGetStreamPriorityRange(int *least, int *greatest) { *least = 0; *greatest = -5; return OK; }
err_t cudaGetLastError(void) { const err_t e = last; last = OK; return e; }
const char *cudaGetErrorString(err_t e) { return e == OOM ? "out of memory" : "invalid value"; }

/* the tensor map encoder: the checks the driver makes of a 3D map */
static int encode(void *m, int type, unsigned rank, void *base, const uint64_t *dims, const uint64_t *strides,
                  const uint32_t *box, const uint32_t *es, int il, int sw, int l2, int fill) {
   const unsigned esz = type == 8 ? 8 : 4; /* FLOAT64, else FLOAT32 */
   (void) es; (void) il; (void) sw; (void) l2; (void) fill;
   memset(m, 0, 128);
   if (rank != 3 || (uintptr_t) base % 16 || box[0] * esz % 16) return 1;
   for (unsigned k = 0; k < 3; k++)
      if (box[k] < 1 || box[k] > 256 || dims[k] < 1) return 1;
   return strides[0] % 16 || strides[1] % 16 ? 1 : 0;
}
err_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long flags, int *q) {
   (void) flags;
   *f = strcmp(name, "cuTensorMapEncodeTiled") == 0 ? (void *) encode : NULL;
   if (q) *q = *f ? 0 : 1;
   return OK;
}
