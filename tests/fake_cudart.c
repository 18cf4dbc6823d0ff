/* A CUDA runtime without a GPU, preloaded in place of the real one by
 * test_host_runtime.py.  Device memory is host memory, kernels do nothing;
 * what the host code asks of the runtime is checked and written to a log:
 * launch limits, which device and stream an allocation is given back on, and
 * device-wide waits while some thread captures a graph. */
#include <cuda_runtime_api.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define DEVICES 2
#define MAX_ITEMS 4096
#define OPTIN 232448
#define STATIC_SMEM 32768

typedef struct {
  int dev, live, capturing;
  long submitted, done;
} Stream;
typedef struct {
  char* p;
  size_t bytes;
  int dev, pooled, live;
} Block;
typedef struct {
  const void* fn;
  int limit;
} Limit;
typedef struct {
  char name[64];
  int regs;
} Kernel; /* of a library, which fake_registers names beforehand */

static Stream streams[MAX_ITEMS];
static Block blocks[MAX_ITEMS];
static Limit limits[DEVICES][MAX_ITEMS];
static int n_streams, n_blocks, n_limits[DEVICES], current, captures_elsewhere, fail_frees,
    pool_keeps_last;
static Kernel kernels[64];
static int n_kernels;
static char log_text[1 << 20];
static size_t log_len;

static void note(const char* fmt, ...) {
  va_list a;
  va_start(a, fmt);
  if (log_len + 256 < sizeof log_text) {
    log_len += (size_t)vsnprintf(log_text + log_len, 255, fmt, a);
    log_text[log_len++] = '\n';
    log_text[log_len] = 0;
  }
  va_end(a);
}

/* ---- for the test */
const char* fake_log(void) { return log_text; }
void fake_clear(void) { log_len = 0, log_text[0] = 0; }
void fake_set_device(int d) { current = d; }
int fake_device(void) { return current; }
void fake_capture_elsewhere(int on) { captures_elsewhere = on; }
void fake_fail_frees(int on) { fail_frees = on; }
void fake_pool_keeps_last(int on) { pool_keeps_last = on; } /* until it is trimmed */
void fake_registers(const char* name, int regs) {
  snprintf(kernels[n_kernels].name, 64, "%s", name);
  kernels[n_kernels++].regs = regs;
}
long fake_pending(void) {
  long n = 0;
  for (int i = 0; i < n_streams; ++i)
    if (streams[i].live) n += streams[i].submitted - streams[i].done;
  return n;
}
void* fake_block(size_t bytes) { /* the first live block of that size */
  for (int i = 0; i < n_blocks; ++i)
    if (blocks[i].live && blocks[i].bytes == bytes) return blocks[i].p;
  return 0;
}
size_t fake_largest_block(void) {
  size_t m = 0;
  for (int i = 0; i < n_blocks; ++i)
    if (blocks[i].live && blocks[i].bytes > m) m = blocks[i].bytes;
  return m;
}
size_t fake_live_bytes(void) {
  size_t m = 0;
  for (int i = 0; i < n_blocks; ++i)
    if (blocks[i].live) m += blocks[i].bytes;
  return m;
}

/* ---- devices, errors */
cudaError_t cudaGetDeviceCount(int* n) { return *n = DEVICES, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = current, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return current = d, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrComputeCapabilityMajor       ? 10
       : a == cudaDevAttrMultiProcessorCount        ? 148
       : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? OPTIN
                                                    : 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) {
  static char s[32];
  snprintf(s, sizeof s, "fake error %d", (int)e);
  return s;
}
static int fake_encode(void) { return 0; }
cudaError_t cudaGetDriverEntryPoint(const char* s, void** fn, unsigned long long flags,
                                    enum cudaDriverEntryPointQueryResult* q) {
  (void)s, (void)flags;
  *fn = (void*)fake_encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

/* ---- streams and events */
static Stream* stream_of(cudaStream_t s) { return (Stream*)s; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags) {
  (void)flags;
  Stream* x = &streams[n_streams++];
  memset(x, 0, sizeof *x);
  x->dev = current;
  x->live = 1;
  *s = (cudaStream_t)x;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  stream_of(s)->live = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  stream_of(s)->done = stream_of(s)->submitted;
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t s) {
  return stream_of(s)->done == stream_of(s)->submitted ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) {
  (void)s, (void)e, (void)f;
  return cudaSuccess;
}
static void wait_device(int dev) {
  for (int i = 0; i < n_streams; ++i)
    if (streams[i].dev == dev) streams[i].done = streams[i].submitted;
}
cudaError_t cudaDeviceSynchronize(void) {
  note("device %d synchronised", current);
  if (captures_elsewhere) {
    note("VIOLATION: device synchronised while another thread captures");
    return cudaErrorStreamCaptureUnsupported;
  }
  wait_device(current);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) {
  (void)f;
  *e = (cudaEvent_t)calloc(1, sizeof(void*));
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  *(Stream**)e = stream_of(s);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (*(Stream**)e) cudaStreamSynchronize((cudaStream_t) * (Stream**)e);
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }

/* ---- memory */
static cudaError_t allocate(void** p, size_t bytes, int dev, int pooled) {
  Block* b = &blocks[n_blocks++];
  b->p = *p = calloc(bytes ? bytes : 1, 1);
  b->bytes = bytes;
  b->dev = dev;
  b->pooled = pooled;
  b->live = 1;
  note("allocated %zu", bytes);
  return cudaSuccess;
}
static Block* block_of(void* p) {
  for (int i = 0; i < n_blocks; ++i)
    if (blocks[i].live && blocks[i].p == p) return &blocks[i];
  note("VIOLATION: free of an unknown pointer");
  return 0;
}
cudaError_t cudaMalloc(void** p, size_t bytes) {
  return pool_keeps_last ? cudaErrorMemoryAllocation : allocate(p, bytes, current, 0);
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
  (void)p, (void)keep;
  return pool_keeps_last = 0, cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned f) {
  (void)f;
  *p = calloc(bytes, 1);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const struct cudaMemPoolProps* pp) {
  int* d = malloc(sizeof *d);
  *d = pp->location.id;
  *pool = (cudaMemPool_t)d;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void* v) {
  (void)p, (void)a, (void)v;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t bytes, cudaMemPool_t pool, cudaStream_t s) {
  const int dev = *(int*)pool;
  if (stream_of(s)->dev != dev) note("VIOLATION: pool and stream of different devices");
  return allocate(p, bytes, dev, 1);
}
/* A block given back while some stream of its device has work that neither the
 * stream it is freed on nor a wait comes after. */
static void check_idle(const Block* b, const Stream* freed_on) {
  for (int i = 0; i < n_streams; ++i)
    if (streams[i].live && &streams[i] != freed_on && streams[i].dev == b->dev &&
        streams[i].submitted > streams[i].done)
      note("VIOLATION: %zu bytes freed with work pending on another stream", b->bytes);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  Block* b = block_of(p);
  if (!b) return cudaErrorInvalidValue;
  if (fail_frees) return cudaErrorUnknown;
  if (!b->pooled) note("VIOLATION: asynchronous free of a plain allocation");
  if (!stream_of(s)->live) note("VIOLATION: freed on a destroyed stream");
  if (stream_of(s)->dev != b->dev)
    note("VIOLATION: memory of device %d freed on a stream of device %d", b->dev,
         stream_of(s)->dev);
  check_idle(b, stream_of(s));
  note("freed %zu", b->bytes);
  b->live = 0;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  Block* b = block_of(p);
  if (!b) return cudaErrorInvalidValue;
  if (b->pooled) check_idle(b, 0); /* no wait for memory of a pool */
  else wait_device(b->dev);
  note("freed %zu", b->bytes);
  b->live = 0;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k,
                            cudaStream_t st) {
  (void)k;
  memcpy(d, s, n);
  if (!stream_of(st)->capturing) ++stream_of(st)->submitted;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  memset(d, v, n);
  if (!stream_of(st)->capturing) ++stream_of(st)->submitted;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
  (void)p;
  memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) {
  (void)sym;
  static char* scratch;
  if (!scratch) scratch = calloc(16u << 20, 1);
  *p = scratch;
  return cudaSuccess;
}

/* ---- kernels */
static const Kernel* kernel_of(const void* fn) {
  const Kernel* k = fn;
  return k >= kernels && k < kernels + n_kernels ? k : 0;
}
static int static_smem(const void* fn) { return kernel_of(fn) ? 0 : STATIC_SMEM; }
static int* limit_of(const void* fn) {
  int i;
  for (i = 0; i < n_limits[current]; ++i)
    if (limits[current][i].fn == fn) return &limits[current][i].limit;
  limits[current][i].fn = fn;
  limits[current][i].limit = 49152 - static_smem(fn);
  ++n_limits[current];
  return &limits[current][i].limit;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* fn) {
  memset(a, 0, sizeof *a);
  a->sharedSizeBytes = static_smem(fn);
  a->maxDynamicSharedSizeBytes = *limit_of(fn);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* fn, enum cudaFuncAttribute a, int v) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  if (v + static_smem(fn) > OPTIN) return cudaErrorInvalidValue;
  *limit_of(fn) = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* fn, int threads,
                                                          size_t smem) {
  const Kernel* k = kernel_of(fn);
  const int by_smem = (int)(OPTIN / (smem + static_smem(fn) + 1024));
  const int by_regs = k ? 65536 / (((k->regs + 7) & ~7) * threads) : 1024 / threads;
  *n = (long)smem > *limit_of(fn) ? 0 : by_smem < by_regs ? by_smem : by_regs;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void** args, size_t smem,
                             cudaStream_t st) {
  (void)args;
  if ((long)smem > *limit_of(fn)) return cudaErrorInvalidValue;
  note("launch %s grid %u %u %u block %u smem %zu", kernel_of(fn) ? kernel_of(fn)->name : "-",
       g.x, g.y, g.z, b.x, smem);
  if (!stream_of(st)->capturing) ++stream_of(st)->submitted;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) {
  return cudaLaunchKernel(fn, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, c->stream);
}
static dim3 call_grid, call_block;
static size_t call_smem;
static void* call_stream;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
  call_grid = g, call_block = b, call_smem = smem, call_stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = call_grid, *b = call_block, *smem = call_smem, *(void**)st = call_stream;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void* f) {
  (void)f;
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}
cudaError_t cudaLibraryLoadData(cudaLibrary_t* l, const void* c, enum cudaJitOption* jo, void** jv,
                                unsigned nj, enum cudaLibraryOption* lo, void** lv, unsigned nl) {
  (void)l, (void)c, (void)jo, (void)jv, (void)nj, (void)lo, (void)lv, (void)nl;
  return n_kernels ? cudaSuccess : cudaErrorNotSupported;
}
cudaError_t cudaLibraryGetKernel(cudaKernel_t* k, cudaLibrary_t l, const char* name) {
  (void)l;
  for (int i = 0; i < n_kernels; ++i)
    if (!strcmp(kernels[i].name, name)) return *k = (cudaKernel_t)&kernels[i], cudaSuccess;
  fake_registers(name, 64);
  return *k = (cudaKernel_t)&kernels[n_kernels - 1], cudaSuccess;
}
cudaError_t cudaLibraryUnload(cudaLibrary_t l) { return (void)l, cudaSuccess; }

/* ---- graphs */
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) {
  (void)m;
  stream_of(s)->capturing = 1;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  stream_of(s)->capturing = 0;
  *g = (cudaGraph_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long f) {
  (void)g, (void)f;
  *x = (cudaGraphExec_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  (void)x;
  ++stream_of(s)->submitted;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return free(x), cudaSuccess; }
