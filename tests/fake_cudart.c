/* A stand-in for the CUDA runtime calls of libmpsq (preloaded into a process of its own), for tests of
 * host code without a GPU: several devices whose memory is the host's, kernels that do nothing, an
 * account of the device memory held, and the rules that the driver would enforce at a launch. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

enum { OK = 0, INVALID = 1, OUT_OF_MEMORY = 2, DYNAMIC_SMEM = 8, SM_COUNT = 16, RELEASE_THRESHOLD = 4 };
typedef struct { unsigned x, y, z; } dim3_t;

static int device, last_error;
static int64_t held, most, capacity = (int64_t)1 << 40;
static uint64_t default_threshold[2];
static int64_t launches;

void fake_set_device(int d) { device = d; }
void fake_set_capacity(int64_t bytes) { capacity = bytes; }
int64_t fake_held(void) { return held; }
int64_t fake_most(int reset) {
  const int64_t m = most;
  if (reset) most = held;
  return m;
}
uint64_t fake_default_threshold(int d) { return default_threshold[d]; }
int64_t fake_launches(void) { return launches; }

static int fails(int code) { return last_error = code; }
int cudaGetLastError(void) {
  const int e = last_error;
  last_error = OK;
  return e;
}
const char* cudaGetErrorString(int e) { return e == OUT_OF_MEMORY ? "out of memory" : e == INVALID ? "invalid argument" : "error"; }
int cudaGetDevice(int* d) { *d = device; return OK; }
int cudaDeviceGetAttribute(int* v, int attr, int d) { (void)d; *v = attr == SM_COUNT ? 152 : 0; return OK; }

/* ---- memory: its size in front of every block */
int cudaMalloc(void** p, size_t n) {
  *p = NULL;
  if (held + (int64_t)n > capacity) return fails(OUT_OF_MEMORY);
  char* b = malloc(n + 256);
  *(size_t*)b = n;
  held += (int64_t)n;
  if (held > most) most = held;
  *p = b + 256;
  return OK;
}
int cudaFree(void* p) {
  if (p) {
    held -= (int64_t)*(size_t*)((char*)p - 256);
    free((char*)p - 256);
  }
  return OK;
}
int cudaMallocAsync(void** p, size_t n, void* s) { (void)s; return cudaMalloc(p, n); }
int cudaMallocFromPoolAsync(void** p, size_t n, void* pool, void* s) { (void)pool; (void)s; return cudaMalloc(p, n); }
int cudaFreeAsync(void* p, void* s) { (void)s; return cudaFree(p); }
int cudaMemGetInfo(size_t* f, size_t* t) { *f = (size_t)(capacity - held); *t = (size_t)capacity; return OK; }
int cudaMemcpy(void* d, const void* s, size_t n, int k) { (void)k; memcpy(d, s, n); return OK; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { (void)st; return cudaMemcpy(d, s, n, k); }
int cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return OK; }
int cudaMemsetAsync(void* p, int v, size_t n, void* s) { (void)s; return cudaMemset(p, v, n); }

/* ---- memory pools */
static char default_pool[2];
int cudaDeviceGetDefaultMemPool(void** pool, int d) { *pool = &default_pool[d]; return OK; }
int cudaMemPoolSetAttribute(void* pool, int attr, void* v) {
  for (int d = 0; d < 2; ++d)
    if (pool == &default_pool[d] && attr == RELEASE_THRESHOLD) default_threshold[d] = *(uint64_t*)v;
  return OK;
}
int cudaMemPoolGetAttribute(void* pool, int attr, void* v) { (void)pool; (void)attr; *(uint64_t*)v = 0; return OK; }
int cudaMemPoolCreate(void** pool, const void* props) { (void)props; *pool = malloc(1); return OK; }
int cudaMemPoolTrimTo(void* pool, size_t n) { (void)pool; (void)n; return OK; }

/* ---- streams and events */
int cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; *s = malloc(1); return OK; }
int cudaStreamDestroy(void* s) { free(s); return OK; }
int cudaStreamSynchronize(void* s) { (void)s; return OK; }
int cudaStreamWaitEvent(void* s, void* e, unsigned f) { (void)s; (void)e; (void)f; return OK; }
int cudaEventCreate(void** e) { *e = malloc(1); return OK; }
int cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; return cudaEventCreate(e); }
int cudaEventDestroy(void* e) { free(e); return OK; }
int cudaEventRecord(void* e, void* s) { (void)e; (void)s; return OK; }
int cudaEventSynchronize(void* e) { (void)e; return OK; }
int cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a; (void)b; *ms = 1.0f; return OK; }

/* ---- graphs: the work of a capture is done at once */
int cudaStreamBeginCapture(void* s, int mode) { (void)s; (void)mode; return OK; }
int cudaStreamEndCapture(void* s, void** g) { (void)s; *g = malloc(1); return OK; }
int cudaGraphInstantiate(void** e, void* g, unsigned long long f) { (void)g; (void)f; *e = malloc(1); return OK; }
int cudaGraphLaunch(void* e, void* s) { (void)e; (void)s; return OK; }
int cudaGraphDestroy(void* g) { free(g); return OK; }
int cudaGraphExecDestroy(void* e) { free(e); return OK; }

/* ---- kernels: dynamic shared memory above 48 KB needs leave, per device and kernel */
static struct { const void* f; int bytes[2]; } leave[4096];
static int* leave_of(const void* f) {
  for (int i = 0; i < 4096; ++i)
    if (leave[i].f == f || !leave[i].f) {
      leave[i].f = f;
      return leave[i].bytes;
    }
  abort();
}
int cudaFuncSetAttribute(const void* f, int attr, int value) {
  if (attr == DYNAMIC_SMEM) leave_of(f)[device] = value;
  return OK;
}
static struct { dim3_t grid, block; size_t smem; void* stream; } call;
unsigned __cudaPushCallConfiguration(dim3_t grid, dim3_t block, size_t smem, void* stream) {
  call.grid = grid;
  call.block = block;
  call.smem = smem;
  call.stream = stream;
  return 0;
}
int __cudaPopCallConfiguration(dim3_t* grid, dim3_t* block, size_t* smem, void** stream) {
  *grid = call.grid;
  *block = call.block;
  *smem = call.smem;
  *stream = call.stream;
  return OK;
}
int __cudaGetKernel(void** kernel, const void* f) { *kernel = (void*)f; return OK; }
int __cudaLaunchKernel(void* kernel, dim3_t grid, dim3_t block, void** args, size_t smem, void* stream) {
  (void)args;
  (void)stream;
  const uint64_t threads = (uint64_t)block.x * block.y * block.z;
  if (!grid.x || !grid.y || !grid.z || grid.y > 65535 || grid.z > 65535 || !threads || threads > 1024 ||
      smem > 227 * 1024 || (smem > 48 * 1024 && (int64_t)smem > leave_of(kernel)[device]))
    return fails(INVALID);
  ++launches;
  return OK;
}
