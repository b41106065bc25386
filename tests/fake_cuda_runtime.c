/* A CUDA runtime of two devices for the library's host code, without a GPU: device memory is host memory, copies and
 * clears happen at once, kernels do not run.  It keeps what the host code has to get right:
 *   - the last error: set by a failed call, read and cleared by cudaGetLastError alone;
 *   - the limit of dynamic shared memory, a property of a kernel on one device: a launch of more than 48 KB fails where
 *     cudaFuncSetAttribute has not raised it;
 *   - the order of work: a clear or a copy on the legacy stream, which a non-blocking stream does not wait for, is
 *     pending until something on the host waits for it. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;
typedef void* stream_t;
typedef struct { unsigned x, y, z; } dim3_t;
enum { kInvalidValue = 1, kOutOfMemory = 2 };

static err_t last_error;
static int device;
static int fail_copies, fail_launches, fail_attributes; /* that many of the next calls fail */
static int launches, legacy_pending;
static struct { const void* fn; int device, bytes; } limits[1024];
static int n_limits;

static err_t failed(err_t e) {
  last_error = e;
  return e;
}

/* ---- for the tests ---- */
void fake_fail(int copies, int launches_, int attributes) {
  fail_copies = copies;
  fail_launches = launches_;
  fail_attributes = attributes;
}
int fake_launches(void) { return launches; }
int fake_legacy_pending(void) { return legacy_pending; }

/* ---- devices, errors ---- */
err_t cudaGetDeviceCount(int* n) { *n = 2; return 0; }
err_t cudaGetDevice(int* d) { *d = device; return 0; }
err_t cudaSetDevice(int d) { device = d; return 0; }
err_t cudaDeviceGetAttribute(int* v, int attr, int d) { (void)attr; (void)d; *v = 152; return 0; }
err_t cudaGetLastError(void) {
  const err_t e = last_error;
  last_error = 0;
  return e;
}
const char* cudaGetErrorString(err_t e) { return e ? "fake error" : "no error"; }

/* ---- memory ---- */
err_t cudaMalloc(void** p, size_t n) { return (*p = calloc(1, n + 256)) ? 0 : failed(kOutOfMemory); }
err_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
err_t cudaFree(void* p) { free(p); return 0; }
err_t cudaFreeHost(void* p) { free(p); return 0; }
static void note(stream_t s) { if (!s) legacy_pending = 1; }
err_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); note(0); return 0; }
err_t cudaMemsetAsync(void* p, int v, size_t n, stream_t s) { memset(p, v, n); note(s); return 0; }
err_t cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, stream_t st) {
  (void)kind;
  if (fail_copies > 0) { --fail_copies; return failed(kInvalidValue); }
  memcpy(d, s, n);
  note(st);
  return 0;
}
err_t cudaMemcpy(void* d, const void* s, size_t n, int kind) { return cudaMemcpyAsync(d, s, n, kind, (stream_t)1); }
err_t cudaPointerGetAttributes(void* at, const void* p) { (void)p; memset(at, 0, 24); return 0; }

/* ---- streams, events, graphs ---- */
err_t cudaDeviceSynchronize(void) { legacy_pending = 0; return 0; }
err_t cudaStreamSynchronize(stream_t s) { if (!s) legacy_pending = 0; return 0; }
err_t cudaStreamCreateWithFlags(stream_t* s, unsigned f) { (void)f; *s = (stream_t)64; return 0; }
err_t cudaStreamDestroy(stream_t s) { (void)s; return 0; }
err_t cudaStreamWaitEvent(stream_t s, void* e, unsigned f) { (void)s; (void)e; (void)f; return 0; }
err_t cudaStreamBeginCapture(stream_t s, int m) { (void)s; (void)m; return 0; }
err_t cudaStreamEndCapture(stream_t s, void** g) { (void)s; *g = (void*)64; return 0; }
err_t cudaGraphInstantiate(void** x, void* g, unsigned long long f) { (void)g; (void)f; *x = (void*)64; return 0; }
err_t cudaGraphLaunch(void* x, stream_t s) { (void)x; (void)s; return 0; }
err_t cudaGraphDestroy(void* g) { (void)g; return 0; }
err_t cudaGraphExecDestroy(void* x) { (void)x; return 0; }
err_t cudaEventCreate(void** e) { *e = (void*)64; return 0; }
err_t cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; *e = (void*)64; return 0; }
err_t cudaEventDestroy(void* e) { (void)e; return 0; }
err_t cudaEventRecord(void* e, stream_t s) { (void)e; (void)s; return 0; }
err_t cudaEventSynchronize(void* e) { (void)e; return 0; }
err_t cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a; (void)b; *ms = 1.0f; return 0; }

/* ---- kernels ---- */
err_t cudaFuncSetAttribute(const void* fn, int attr, int value) {
  if (fail_attributes > 0) { --fail_attributes; return failed(kInvalidValue); }
  if (attr == 8 && n_limits < 1024) { /* cudaFuncAttributeMaxDynamicSharedMemorySize */
    limits[n_limits].fn = fn;
    limits[n_limits].device = device;
    limits[n_limits++].bytes = value;
  }
  return 0;
}
static err_t launch(const void* fn, dim3_t grid, size_t smem) {
  int allowed = 48 * 1024, i;
  for (i = 0; i < n_limits; ++i) {
    if (limits[i].fn == fn && limits[i].device == device && limits[i].bytes > allowed) allowed = limits[i].bytes;
  }
  if (fail_launches > 0) { --fail_launches; return failed(kInvalidValue); }
  if (grid.x == 0 || grid.y == 0 || grid.y > 65535 || grid.z == 0 || grid.z > 65535 || smem > (size_t)allowed) return failed(kInvalidValue);
  ++launches;
  return 0;
}
err_t cudaLaunchKernel(const void* fn, dim3_t grid, dim3_t block, void** args, size_t smem, stream_t s) {
  (void)block; (void)args; (void)s;
  return launch(fn, grid, smem);
}
err_t cudaLaunchCooperativeKernel(const void* fn, dim3_t grid, dim3_t block, void** args, size_t smem, stream_t s) {
  return cudaLaunchKernel(fn, grid, block, args, smem, s);
}
struct launch_config { dim3_t grid, block; size_t smem; stream_t stream; void* attrs; unsigned n; };
err_t cudaLaunchKernelExC(const struct launch_config* c, const void* fn, void** args) {
  (void)args;
  return launch(fn, c->grid, c->smem);
}
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* fn, int threads, size_t smem, unsigned f) {
  (void)fn; (void)threads; (void)smem; (void)f;
  *n = 2;
  return 0;
}
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* fn, int threads, size_t smem) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, fn, threads, smem, 0);
}
err_t cudaGetSymbolAddress(void** p, const void* symbol) { *p = (void*)symbol; return 0; }

/* the driver's functions: a tensor map is encoded, an address range is not known */
static int driver_ok(void) { return 0; }
static int driver_unknown(void) { return 1; }
err_t cudaGetDriverEntryPointByVersion(const char* name, void** fn, unsigned v, unsigned long long f, int* q) {
  (void)v; (void)f;
  *fn = strstr(name, "AddressRange") ? (void*)driver_unknown : (void*)driver_ok;
  if (q) *q = 0;
  return 0;
}

/* ---- what nvcc's host code calls ---- */
static struct { dim3_t grid, block; size_t smem; stream_t stream; } pushed;
unsigned __cudaPushCallConfiguration(dim3_t grid, dim3_t block, size_t smem, stream_t s) {
  pushed.grid = grid;
  pushed.block = block;
  pushed.smem = smem;
  pushed.stream = s;
  return 0;
}
err_t __cudaPopCallConfiguration(dim3_t* grid, dim3_t* block, size_t* smem, void* s) {
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *(stream_t*)s = pushed.stream;
  return 0;
}
err_t __cudaGetKernel(const void** kernel, const void* fn) { *kernel = fn; return 0; }
err_t __cudaLaunchKernel(const void* kernel, dim3_t grid, dim3_t block, void** args, size_t smem, stream_t s) {
  return cudaLaunchKernel(kernel, grid, block, args, smem, s);
}
void** __cudaRegisterFatBinary(void* fat) { (void)fat; return (void**)&pushed; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
char __cudaInitModule(void** h) { (void)h; return 0; }
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}
