/* A CUDA runtime without a GPU, put in front of the real one (LD_PRELOAD) by
 * tests/fake_runtime.py: device memory is host memory, kernels do not run, and
 * every call goes through a hook that can look at it and make it fail.  It
 * shows what the library's host code asks of the runtime, in what order, and
 * what it does when a call fails. */
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

/* hook(call, name, stream, p, q, n, args): name is a kernel's mangled name
 * (launches and attributes); returns the error that the call gives */
typedef int (*hook_fn)(const char*, const char*, uint64_t, uint64_t, uint64_t, uint64_t, void**);
static hook_fn hook;
static cudaError_t last = cudaSuccess;
void fake_set_hook(hook_fn f) { hook = f; }

static cudaError_t call(const char* what, const char* name, const void* stream, const void* p, const void* q, size_t n,
                        void** args) {
  const cudaError_t e =
      hook ? (cudaError_t)hook(what, name, (uint64_t)stream, (uint64_t)p, (uint64_t)q, n, args) : cudaSuccess;
  if (e != cudaSuccess) last = e;
  return e;
}
#define CALL(what, name, stream, p, q, n, args)                            \
  do {                                                                     \
    const cudaError_t e_ = call(what, name, stream, p, q, n, args);        \
    if (e_ != cudaSuccess) return e_;                                      \
  } while (0)

/* ---- kernels ---- */
#define MAXK 1024
static struct {
  const void* f;
  const char* name;
} kern[MAXK];
static int nkern;
static const char* kname(const void* f) {
  for (int i = 0; i < nkern; ++i)
    if (kern[i].f == f) return kern[i].name;
  return "?";
}
void** __cudaRegisterFatBinary(void* b) {
  (void)b;
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void** h, const char* f, char* d, const char* name, int l, void* a, void* b, void* c,
                            void* e, int* w) {
  (void)h, (void)d, (void)l, (void)a, (void)b, (void)c, (void)e, (void)w;
  if (nkern < MAXK) kern[nkern].f = f, kern[nkern++].name = strdup(name);
}
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int c, int g) {
  (void)h, (void)v, (void)d, (void)n, (void)e, (void)s, (void)c, (void)g;
}
static __thread struct {
  dim3 g, b;
  size_t smem;
  void* s;
} cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) {
  cfg.g = g, cfg.b = b, cfg.smem = smem, cfg.s = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = cfg.g, *b = cfg.b, *smem = cfg.smem, *(void**)s = cfg.s;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s) {
  (void)b;
  return call("launch", kname(f), s, (void*)(uintptr_t)g.x, 0, smem, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return call("launch", kname(f), c->stream, (void*)(uintptr_t)c->gridDim.x, 0, c->dynamicSmemBytes, args);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  return call("attribute", kname(f), 0, (void*)(uintptr_t)a, 0, (size_t)v, 0);
}

/* ---- memory ---- */
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = 0;
  CALL("malloc", "", 0, 0, 0, n, 0);
  *p = calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  CALL("free", "", 0, p, 0, 0, 0);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s) {
  *p = 0;
  CALL("malloc_pool", "", s, pool, 0, n, 0);
  *p = calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  CALL("free_pool", "", s, p, 0, 0, 0);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const struct cudaMemPoolProps* props) {
  (void)props;
  *p = (cudaMemPool_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void* v) {
  (void)p, (void)a, (void)v;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t n) { return call("trim_pool", "", 0, p, 0, n, 0); }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int d) {
  (void)d;
  *p = 0;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  CALL(k == cudaMemcpyDeviceToHost ? "copy_down" : "copy_up", "", 0, d, s, n, 0);
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  CALL(k == cudaMemcpyDeviceToHost ? "copy_down_async" : k == cudaMemcpyHostToDevice ? "copy_up_async" : "copy_async", "",
       st, d, s, n, 0);
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  CALL("memset", "", 0, p, 0, n, 0);
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  CALL("memset_async", "", s, p, 0, n, 0);
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = (void*)s;
  return cudaSuccess;
}

/* ---- streams, events, graphs, device ---- */
static cudaError_t handle(void** h) {
  *h = malloc(1);
  return cudaSuccess;
}
static cudaError_t drop(void* h) {
  free(h);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  (void)f;
  return handle((void**)s);
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return call("sync", "", s, 0, 0, 0, 0); }
cudaError_t cudaDeviceSynchronize(void) { return call("sync_device", "", 0, 0, 0, 0, 0); }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) {
  (void)m;
  return call("capture", "", s, 0, 0, 0, 0);
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  CALL("capture_end", "", s, 0, 0, 0, 0);
  return handle((void**)g);
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* st) {
  (void)s;
  *st = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f) {
  (void)g, (void)f;
  return handle((void**)e);
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t e, cudaGraph_t g, cudaGraphExecUpdateResultInfo* i) {
  (void)e, (void)g, (void)i;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { return call("graph", "", s, e, 0, 0, 0); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return drop(e); }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return drop(g); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle((void**)e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  (void)e, (void)s;
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  (void)a, (void)b;
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)a, (void)d;
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) {
  (void)e;
  return "fake";
}
static int ctx_id(void* c, unsigned long long* id) {
  (void)c;
  *id = 1;
  return 0;
}
#undef cudaGetDriverEntryPoint
cudaError_t cudaGetDriverEntryPoint(const char* n, void** f, unsigned long long fl,
                                    enum cudaDriverEntryPointQueryResult* r) {
  (void)n, (void)fl;
  *f = (void*)ctx_id;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
