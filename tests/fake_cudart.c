/* A stand-in for the CUDA runtime, preloaded into a child process so that the
 * library's host code -- what it launches, captures, copies and allocates, and
 * what it does when a call fails -- can be tested without a GPU.  Device memory
 * is host memory, copies are done at once, kernels are recorded and do not run.
 *
 * A test steers it through the fake_* functions:
 *   fake_malloc_limit(n)       device allocations above n bytes fail (0: none do)
 *   fake_status_word(v)        from now on every 4-byte read from the device gives v
 *   fake_cost(f)               f(kernel name, blocks, threads per block, launches so far): ms
 *                              that a launch takes on the clock that events read
 *   fake_launches(name)        launches of kernels whose name holds `name`
 *   fake_instantiations()      CUDA graphs instantiated
 *   fake_allocations(n)        device allocations of at least n bytes, freed ones too
 */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <cuda_runtime_api.h>

#define MAX_KERNELS 4096
static struct {
  const void *fn;
  const char *name;
  unsigned long launches;
} kernels[MAX_KERNELS];
static int nkernels;
static size_t malloc_limit;
static int have_status;
static unsigned status_word;
static unsigned long nlaunches, ninstantiations;
static double now_ms;
static double (*cost_fn)(const char *, unsigned, unsigned, unsigned long);

void fake_malloc_limit(size_t n) { malloc_limit = n; }
void fake_status_word(unsigned v) { have_status = 1; status_word = v; }
void fake_status_clear(void) { have_status = 0; }
void fake_cost(double (*f)(const char *, unsigned, unsigned, unsigned long)) { cost_fn = f; }
unsigned long fake_launches(const char *name) {
  unsigned long n = 0;
  for (int i = 0; i < nkernels; ++i)
    if (strstr(kernels[i].name, name)) n += kernels[i].launches;
  return n;
}
static size_t sizes[1 << 16];
static unsigned nsizes;
unsigned long fake_allocations(size_t n) {
  unsigned long c = 0;
  for (unsigned i = 0; i < nsizes; ++i) c += sizes[i] >= n;
  return c;
}
unsigned long fake_instantiations(void) { return ninstantiations; }

/* ---- registration and launches ---- */
void **__cudaRegisterFatBinary(void *bin) {
  static void *handle;
  (void)bin;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *fn, char *dev, const char *name, int limit, void *tid, void *bid,
                            void *bdim, void *gdim, int *wsize) {
  (void)h; (void)dev; (void)limit; (void)tid; (void)bid; (void)bdim; (void)gdim; (void)wsize;
  if (nkernels == MAX_KERNELS) abort();
  kernels[nkernels].fn = fn;
  kernels[nkernels++].name = name;
}
static struct {
  const void *host;
  void *mem;
} vars[64];
static int nvars;
void __cudaRegisterVar(void **h, char *host, char *dev, const char *name, int ext, size_t size, int constant,
                       int global) {
  (void)h; (void)dev; (void)name; (void)ext; (void)constant; (void)global;
  if (nvars == 64) abort();
  vars[nvars].host = host;
  vars[nvars++].mem = calloc(1, size);
}
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
  for (int i = 0; i < nvars; ++i)
    if (vars[i].host == sym) {
      *p = vars[i].mem;
      return cudaSuccess;
    }
  return cudaErrorInvalidSymbol;
}
static struct {
  dim3 grid, block;
  size_t smem;
  void *stream;
} config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *st) {
  config.grid = grid;
  config.block = block;
  config.smem = smem;
  config.stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *(void **)st = config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) {
  *k = (cudaKernel_t)fn;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t st) {
  (void)args; (void)smem; (void)st;
  for (int i = 0; i < nkernels; ++i)
    if (kernels[i].fn == (const void *)k) {
      kernels[i].launches++;
      now_ms += cost_fn ? cost_fn(kernels[i].name, grid.x, block.x, nlaunches) : 1.0;
      nlaunches++;
      return cudaSuccess;
    }
  return cudaErrorInvalidDeviceFunction;
}
cudaError_t cudaFuncSetAttribute(const void *fn, enum cudaFuncAttribute a, int v) {
  (void)fn; (void)a; (void)v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *fn, int threads, size_t smem,
                                                                   unsigned flags) {
  (void)fn; (void)flags;
  int by_threads = 2048 / (threads > 0 ? threads : 1), by_smem = smem ? (int)((228u << 10) / (smem + 1024)) : 32;
  *n = by_threads < by_smem ? by_threads : by_smem;
  if (*n < 1) *n = 1;
  return cudaSuccess;
}

/* ---- device, memory ---- */
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d == 0 ? cudaSuccess : cudaErrorInvalidDevice; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 << 10 : 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaMalloc(void **p, size_t n) {
  if (malloc_limit && n > malloc_limit) return cudaErrorMemoryAllocation;
  if (nsizes < sizeof sizes / sizeof *sizes) sizes[nsizes++] = n;
  *p = calloc(1, n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)st;
  memmove(d, s, n);
  if (k == cudaMemcpyDeviceToHost && n == sizeof status_word && have_status) memcpy(d, &status_word, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, 0); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  (void)st;
  memset(d, v, n);
  return cudaSuccess;
}

/* ---- streams, events, graphs ---- */
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) {
  (void)s;
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = malloc(1); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f) {
  (void)g; (void)f;
  ninstantiations++;
  *x = malloc(1);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) {
  (void)f;
  *e = calloc(1, sizeof(double));
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  (void)s;
  *(double *)e = now_ms;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(*(double *)b - *(double *)a);
  return cudaSuccess;
}
