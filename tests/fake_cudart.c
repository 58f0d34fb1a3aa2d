/* A CUDA runtime without a device, for host-side tests of the library: linked with the library's
 * objects in place of libcudart.  Device memory is host memory that starts as zeros; copies and
 * memsets really happen, and any that leaves a live block is counted and skipped.  Kernels do not run:
 * a launch is logged, with the argument values of the kernels the test watches.  Allocations and graph
 * instantiations can be refused.  Freed blocks are not handed out again before a reset, so an address
 * tells which allocation it came from. */
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

enum { MAXB = 4096, MAXK = 8192, MAXW = 32, MAXLOG = 65536, MAXARG = 24 };

static struct { char *p; size_t n; int live; } blk[MAXB];
static int nblk;
static size_t used, most, room = (size_t)1 << 40;
static long refuse_at = -1, mallocs, violations, instantiations;
static int refuse_graphs, refuse_downloads, blocks_per_sm = 4;
static cudaError_t last;
long long fake_extent(const void *p);

static struct { const void *f; char name[256]; } kern[MAXK];
static int nkern;
static struct { const void *host; size_t n; char *dev; } var[64];
static int nvar;
static struct { char part[64]; char sig[MAXARG + 1]; } watch[MAXW];
static int nwatch;
struct launch { int watch, captured; unsigned grid; long long a[MAXARG], room[MAXARG]; };
static struct launch lg[MAXLOG];
static long nlog, nlaunch, ncaptured;
static int capturing;

/* ---- control, called by the tests */
void fake_reset(void) {
  nlog = nlaunch = ncaptured = violations = mallocs = instantiations = 0;
  refuse_at = -1;
  refuse_graphs = refuse_downloads = 0;
  blocks_per_sm = 4;
  last = cudaSuccess;
  room = (size_t)1 << 40;
  used = most = 0;
  for (int b = 0; b < nblk; ++b) free(blk[b].p);  /* freed ones and what an earlier test left */
  nblk = 0;
}
void fake_room(size_t bytes) { room = bytes; }           /* capacity of the device */
size_t fake_used(void) { return used; }
size_t fake_peak(void) { return most; }
void fake_refuse(long k) { refuse_at = k < 0 ? -1 : mallocs + k; }  /* refuse the k-th allocation from now */
void fake_refuse_graphs(int n) { refuse_graphs = n; }  /* the next n instantiations */
void fake_refuse_downloads(int n) { refuse_downloads = n; }  /* the next n copies to the host */
void fake_blocks_per_sm(int n) { blocks_per_sm = n; }
long fake_violations(void) { return violations; }
long fake_instantiations(void) { return instantiations; }
long fake_launches(void) { return nlaunch; }
long fake_mallocs(void) { return mallocs; }
void fake_clear_watches(void) { nwatch = 0; }
/* log the arguments of kernels whose mangled name contains part: P pointer or long long, i int, f float */
int fake_watch(const char *part, const char *sig) {
  snprintf(watch[nwatch].part, sizeof watch[0].part, "%s", part);
  snprintf(watch[nwatch].sig, sizeof watch[0].sig, "%s", sig);
  return nwatch++;
}
long fake_log(void) { return nlog; }
int fake_log_watch(long k) { return lg[k].watch; }
unsigned fake_log_grid(long k) { return lg[k].grid; }
long long fake_log_arg(long k, int i) { return lg[k].a[i]; }
long long fake_log_room(long k, int i) { return lg[k].room[i]; }  /* fake_extent of argument i at the launch */
/* bytes from p to the end of the live block that holds it, or -1 */
long long fake_extent(const void *p) {
  for (int b = 0; b < nblk; ++b)
    if (blk[b].live && (const char *)p >= blk[b].p && (const char *)p < blk[b].p + blk[b].n)
      return blk[b].p + blk[b].n - (const char *)p;
  for (int v = 0; v < nvar; ++v)
    if (var[v].dev && (const char *)p >= var[v].dev && (const char *)p < var[v].dev + var[v].n)
      return var[v].dev + var[v].n - (const char *)p;
  return -1;
}
static int inside(const void *p, size_t n) {
  long long e = fake_extent(p);
  if (e < 0 || (size_t)e < n) { ++violations; return 0; }
  return 1;
}
static cudaError_t set(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }

/* ---- registration (host_runtime.h signatures) */
void **__cudaRegisterFatBinary(void *f) { static void *h; h = f; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *f, char *df, const char *name, int lim, uint3 *t, uint3 *b, dim3 *bd,
                            dim3 *gd, int *w) {
  (void)h; (void)df; (void)lim; (void)t; (void)b; (void)bd; (void)gd; (void)w;
  if (nkern < MAXK) {
    kern[nkern].f = f;
    snprintf(kern[nkern++].name, sizeof kern[0].name, "%s", name);
  }
}
void __cudaRegisterVar(void **h, char *host, char *dev, const char *name, int ext, size_t size, int constant, int global) {
  (void)h; (void)dev; (void)name; (void)ext; (void)constant; (void)global;
  if (nvar < 64) { var[nvar].host = host; var[nvar++].n = size; }
}
static struct { dim3 g, b; size_t s; void *st; } cfgs[8];
static int ncfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st *st) {
  cfgs[ncfg].g = g; cfgs[ncfg].b = b; cfgs[ncfg].s = s; cfgs[ncfg++].st = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  --ncfg;
  *g = cfgs[ncfg].g; *b = cfgs[ncfg].b; *s = cfgs[ncfg].s; *(void **)st = cfgs[ncfg].st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t s, cudaStream_t st) {
  (void)b; (void)s; (void)st;
  ++nlaunch;
  ncaptured += capturing;
  const char *name = "";
  for (int k = 0; k < nkern; ++k)
    if (kern[k].f == f) { name = kern[k].name; break; }
  for (int w = 0; w < nwatch; ++w)
    if (strstr(name, watch[w].part) && nlog < MAXLOG) {
      struct launch *l = lg + nlog++;
      l->watch = w;
      l->captured = capturing;
      l->grid = g.x;
      for (int i = 0; watch[w].sig[i]; ++i) {
        const char c = watch[w].sig[i];
        l->a[i] = c == 'P' ? *(long long *)args[i] : c == 'i' ? *(int *)args[i] : 0;
        l->room[i] = c == 'P' ? fake_extent((void *)l->a[i]) : 0;
      }
      break;
    }
  return cudaSuccess;
}

/* ---- memory */
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = NULL;
  if (mallocs++ == refuse_at || used + n > room || nblk == MAXB) return set(cudaErrorMemoryAllocation);
  char *q = calloc(1, n ? n : 1);
  if (!q) return set(cudaErrorMemoryAllocation);
  blk[nblk].p = q; blk[nblk].n = n; blk[nblk++].live = 1;
  used += n;
  if (used > most) most = used;
  *p = q;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  for (int b = 0; b < nblk; ++b)
    if (blk[b].p == p && blk[b].live) {
      blk[b].live = 0;
      used -= blk[b].n;
      return cudaSuccess;
    }
  ++violations;
  return set(cudaErrorInvalidValue);
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)st;
  int ok = 1;
  if (k == cudaMemcpyDeviceToHost && refuse_downloads > 0) { --refuse_downloads; return set(cudaErrorUnknown); }
  if (k != cudaMemcpyDeviceToHost) ok &= inside(d, n);
  if (k != cudaMemcpyHostToDevice) ok &= inside(s, n);
  if (ok && !capturing) memmove(d, s, n);
  return ok ? cudaSuccess : set(cudaErrorInvalidValue);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  (void)st;
  if (!inside(d, n)) return set(cudaErrorInvalidValue);
  if (!capturing) memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy3DAsync(const struct cudaMemcpy3DParms *p, cudaStream_t st) {
  (void)st;
  const struct cudaPitchedPtr *s = &p->srcPtr, *d = &p->dstPtr;
  for (size_t z = 0; z < p->extent.depth; ++z)
    for (size_t y = 0; y < p->extent.height; ++y) {
      const char *a = (const char *)s->ptr + s->pitch * (y + s->ysize * z);
      char *b = (char *)d->ptr + d->pitch * (y + d->ysize * z);
      const void *dev = p->kind == cudaMemcpyDeviceToHost ? (const void *)a : (const void *)b;
      if (!inside(dev, p->extent.width)) return set(cudaErrorInvalidValue);
      memcpy(b, a, p->extent.width);
    }
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
  for (int v = 0; v < nvar; ++v)
    if (var[v].host == sym) {
      if (!var[v].dev) var[v].dev = calloc(1, var[v].n);
      *p = var[v].dev;
      return cudaSuccess;
    }
  return set(cudaErrorInvalidSymbol);
}

/* ---- the rest: one device, streams and events that are always done */
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int b, size_t s) { (void)f; (void)b; (void)s; *n = blocks_per_sm; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = malloc(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; *e = malloc(8); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; capturing = 1; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; capturing = 0; *g = malloc(8); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long f) {
  (void)g; (void)f;
  *e = NULL;
  if (refuse_graphs > 0) { --refuse_graphs; return set(cudaErrorMemoryAllocation); }
  ++instantiations;
  *e = malloc(8);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { (void)s; return e ? cudaSuccess : set(cudaErrorInvalidValue); }
