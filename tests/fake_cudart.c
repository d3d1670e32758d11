/* A CUDA runtime for tests of the library's host code without a GPU, put in
 * front of libcudart with LD_PRELOAD: device memory is host memory, copies and
 * memsets happen at once, launches do nothing, and every call that touches a
 * stream is written to the file FAKE_CUDART_LOG names.  Attributes are those
 * of a GB300. */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static FILE *out;
static size_t live, peak, limit = (size_t)-1; /* bytes of device memory */
static int status;                            /* what the next int read from the device says, once */
static struct { void *to; size_t bytes; } up[4096]; /* the latest copies to the device */
static int nup;
static const void *fun[512];
static const char *name[512];
static int nfun;

static FILE *log_file(void) {
  if (!out) {
    const char *f = getenv("FAKE_CUDART_LOG");
    out = f ? fopen(f, "a") : stderr;
    setvbuf(out, NULL, _IOLBF, 0);
  }
  return out;
}

/* ---- control, by ctypes ---- */
void fake_limit(size_t bytes) { limit = bytes; }
void fake_status(int s) { status = s; }
size_t fake_live(void) { return live; }
size_t fake_peak(void) { return peak; }
void *fake_upload(size_t bytes, int back) { /* where the latest copy of that size went, but `back` */
  for (int i = nup; i-- > 0 && i > nup - 4096;)
    if (up[i % 4096].bytes == bytes && back-- == 0) return up[i % 4096].to;
  return NULL;
}
void fake_mark(const char *what) { fprintf(log_file(), "mark %s\n", what); }

/* ---- registration ---- */
void **__cudaRegisterFatBinary(void *b) { return (void **)b; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *d, const char *n, int e, size_t s, int c, int g) {}
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *n, int l, void *t, void *b, void *bd,
                            void *gd, int *w) {
  if (nfun < 512) {
    fun[nfun] = f;
    name[nfun++] = n;
  }
}
static const char *name_of(const void *f) {
  for (int i = 0; i < nfun; i++)
    if (fun[i] == f) return name[i];
  return "?";
}

/* ---- launches ---- */
static cudaError_t launch(const void *f, dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  fprintf(log_file(), "launch %s %u %u %zu %p\n", name_of(f), g.x * g.y * g.z, b.x * b.y * b.z, smem, (void *)st);
  return cudaSuccess;
}
static dim3 cfg_g, cfg_b;
static size_t cfg_s;
static cudaStream_t cfg_st;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st *st) {
  cfg_g = g;
  cfg_b = b;
  cfg_s = s;
  cfg_st = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  *g = cfg_g;
  *b = cfg_b;
  *s = cfg_s;
  *(cudaStream_t *)st = cfg_st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **a, size_t s, cudaStream_t st) {
  return launch((const void *)k, g, b, s, st);
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t s, cudaStream_t st) {
  return launch(f, g, b, s, st);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **a, size_t s, cudaStream_t st) {
  return launch(f, g, b, s, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int threads, size_t smem,
                                                                   unsigned flags) {
  const size_t regs = 65536 / (64 * (size_t)threads), sh = 233472 / (smem + 1024);
  *n = (int)(regs < sh ? regs : sh);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int threads, size_t smem) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, threads, smem, 0);
}

/* ---- device ---- */
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
  *v = a == cudaDevAttrMultiProcessorCount               ? 152
       : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472
       : a == cudaDevAttrMaxSharedMemoryPerBlockOptin     ? 232448
       : a == cudaDevAttrCooperativeLaunch                ? 1
       : a == cudaDevAttrL2CacheSize                      ? 129 << 20
                                                          : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) {
  fprintf(log_file(), "sync device\n");
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "error of the fake runtime"; }

/* ---- memory: the size lies ahead of each block, which starts as 0xAB ---- */
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = NULL;
  if (live + n > limit) return cudaErrorMemoryAllocation;
  char *q = aligned_alloc(256, (n + 511) / 256 * 256 + 256);
  if (!q) return cudaErrorMemoryAllocation;
  *(size_t *)q = n;
  memset(q + 256, 0xAB, n);
  *p = q + 256;
  live += n;
  if (live > peak) peak = live;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (p) {
    live -= *(size_t *)((char *)p - 256);
    free((char *)p - 256);
  }
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned f) { return *d = h, cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
  memset(a, 0, sizeof *a); /* unregistered */
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { return cudaErrorNotSupported; }
static void copied(void *d, size_t n, enum cudaMemcpyKind k) {
  if (k == cudaMemcpyHostToDevice) {
    up[nup % 4096].to = d;
    up[nup++ % 4096].bytes = n;
  }
  if (status && k == cudaMemcpyDeviceToHost && n == sizeof(int)) {
    *(int *)d = status;
    status = 0;
  }
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) {
  fprintf(log_file(), "memcpy %d %zu legacy\n", (int)k, n);
  memcpy(d, s, n);
  copied(d, n, k);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  fprintf(log_file(), "memcpy %d %zu %p\n", (int)k, n, (void *)st);
  memcpy(d, s, n);
  copied(d, n, k);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  fprintf(log_file(), "memset %zu legacy\n", n);
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  fprintf(log_file(), "memset %zu %p\n", n, (void *)st);
  memset(d, v, n);
  return cudaSuccess;
}

/* ---- streams, events, graphs (no capture) ---- */
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) {
  *s = (cudaStream_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  fprintf(log_file(), s == 0 || s == cudaStreamLegacy ? "sync legacy\n" : "sync %p\n", (void *)s);
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { return cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)malloc(1), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { return *ms = 1.0f, cudaSuccess; }
