/* A stand-in for the CUDA runtime with two devices and no kernels, preloaded by
 * test_cpu_devices.py: memory is host memory, a launch does nothing but is refused,
 * as the runtime refuses it, unless its stream belongs to the calling thread's
 * current device. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

typedef int err;
typedef struct { unsigned x, y, z; } dim3;
typedef struct { dim3 grid, block; size_t smem; void* stream; void* attrs; unsigned n; } config;

static __thread int current = 0;
static __thread err last = 0;
static __thread config pushed;
static int foreign_mallocs = 0, expected = -1, launches = 0;

/* what the test sets and reads */
void fake_expect(int device) { expected = device; }  /* where allocations belong */
int fake_foreign_mallocs(void) { return foreign_mallocs; }
int fake_launches(void) { return launches; }

err cudaSetDevice(int d) { if (d < 0 || d > 1) return 101; current = d; return 0; }
err cudaGetDevice(int* d) { *d = current; return 0; }
err cudaGetLastError(void) { err e = last; last = 0; return e; }
const char* cudaGetErrorString(err e) { return e == 400 ? "invalid resource handle" : "error"; }
err cudaDeviceGetAttribute(int* v, int a, int d) { *v = 152; return 0; }

static void allocated(void) { if (expected >= 0 && current != expected) ++foreign_mallocs; }
err cudaMalloc(void** p, size_t n) { allocated(); *p = calloc(1, n); return 0; }
err cudaFree(void* p) { free(p); return 0; }
err cudaHostAlloc(void** p, size_t n, unsigned f) { *p = calloc(1, n); return 0; }
err cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return 0; }
err cudaFreeHost(void* p) { free(p); return 0; }
err cudaMemcpy(void* d, const void* s, size_t n, int k) { memmove(d, s, n); return 0; }
err cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { memmove(d, s, n); return 0; }
err cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, int k) {
  for (size_t r = 0; r < h; ++r) memmove((char*)d + r * dp, (const char*)s + r * sp, w);
  return 0;
}
err cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return 0; }
err cudaMemsetAsync(void* d, int v, size_t n, void* st) { memset(d, v, n); return 0; }
err cudaGetSymbolAddress(void** p, const void* s) { *p = calloc(1, 1 << 20); return 0; }

/* a stream is a pointer to its device */
err cudaStreamCreateWithFlags(void** s, unsigned f) { *s = malloc(sizeof(int)); *(int*)*s = current; return 0; }
err cudaStreamDestroy(void* s) { free(s); return 0; }
err cudaStreamSynchronize(void* s) { return 0; }
err cudaStreamWaitEvent(void* s, void* e, unsigned f) { return 0; }
err cudaStreamBeginCapture(void* s, int m) { return 0; }
err cudaStreamEndCapture(void* s, void** g) { *g = malloc(1); return 0; }
err cudaGraphInstantiate(void** e, void* g, unsigned long long f) { *e = malloc(1); return 0; }
err cudaGraphDestroy(void* g) { free(g); return 0; }
err cudaGraphExecDestroy(void* e) { free(e); return 0; }
err cudaEventCreate(void** e) { *e = malloc(1); return 0; }
err cudaEventCreateWithFlags(void** e, unsigned f) { *e = malloc(1); return 0; }
err cudaEventDestroy(void* e) { free(e); return 0; }
err cudaEventRecord(void* e, void* s) { return 0; }
err cudaEventSynchronize(void* e) { return 0; }
err cudaEventElapsedTime(float* ms, void* a, void* b) { *ms = 1.0f; return 0; }

static err launch(void* stream) {
  ++launches;
  if (stream && *(int*)stream != current) return last = 400;
  return 0;
}
err cudaGraphLaunch(void* e, void* s) { return launch(s); }
err cudaLaunchKernelExC(const config* c, const void* f, void** a) { return launch(c->stream); }
err __cudaLaunchKernel(void* k, dim3 g, dim3 b, void** a, size_t sm, void* s) { return launch(s); }
err cudaLaunchKernel(const void* k, dim3 g, dim3 b, void** a, size_t sm, void* s) { return launch(s); }
err __cudaGetKernel(void** k, const void* f) { *k = (void*)f; return 0; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, void* s) {
  pushed.grid = g; pushed.block = b; pushed.smem = sm; pushed.stream = s;
  return 0;
}
err __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* s) {
  *g = pushed.grid; *b = pushed.block; *sm = pushed.smem; *(void**)s = pushed.stream;
  return 0;
}
err cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }
err cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t sm, unsigned fl) {
  *n = 4;
  return 0;
}
void** __cudaRegisterFatBinary(void* p) { return malloc(8); }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction(void** h, const char* f, char* n, const char* d, int t, void* a, void* b, void* c,
                            void* e, int* w) {}
void __cudaRegisterVar(void** h, char* v, char* a, const char* n, int e, size_t s, int c, int g) {}
