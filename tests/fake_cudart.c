/* A stand-in for the CUDA runtime library, for tests of the host code on a
 * machine without a GPU: device memory is host memory, copies are made at once,
 * kernels do not run but are counted by name, and a launch on a stream of
 * another device than the current one is refused, as the runtime refuses it. Calls can be made to
 * fail by number (fake_set). It is built as libcudart.so.12 into a test's own
 * directory and put first on the library path of a child process. */
#include <driver_types.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

enum { O_SMS, O_COOP, O_CLUSTERS, O_BLOCKS, O_ENCODE, O_MALLOC_MAX, O_POOL_REFUSED, O_PINNED_MAX, N_OPT };
static long opt[N_OPT] = {148, 1, 64, 1, 0, 1L << 40, -1, 1L << 40};
static const char* opt_name[N_OPT] = {"sms", "cooperative", "max_clusters", "blocks_per_sm", "encode_result", "malloc_max", "pool_refused", "pinned_max"};

int fake_set(const char* name, long v) {
  for (int i = 0; i < N_OPT; i++)
    if (!strcmp(opt_name[i], name)) {
      opt[i] = v;
      return 0;
    }
  return -1;
}

/* bytes of cudaMalloc that are not freed yet */
static size_t held = 0;
size_t fake_held(void) { return held; }

/* called in cudaEventSynchronize, where a program waits for its work */
static void (*on_wait)(void) = NULL;
void fake_on_wait(void (*f)(void)) { on_wait = f; }

/* ---- kernels */
struct kernel {
  const void* host;
  char name[256];
  long launches;
  struct kernel* next;
};
static struct kernel* kernels = NULL;
static long launches = 0;

/* launches of the kernels whose mangled name holds `part`; all: fake_launches("") */
long fake_launches(const char* part) {
  long n = 0;
  for (struct kernel* k = kernels; k; k = k->next)
    if (strstr(k->name, part)) n += k->launches;
  return n;
}
void fake_clear(void) {
  for (struct kernel* k = kernels; k; k = k->next) k->launches = 0;
}

void** __cudaRegisterFatBinary(void* p) {
  (void)p;
  return malloc(sizeof(void*));
}
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void** h, const char* host, char* dev, const char* name, int lim, void* a, void* b, void* c, void* d, int* e) {
  (void)h, (void)dev, (void)lim, (void)a, (void)b, (void)c, (void)d, (void)e;
  struct kernel* k = calloc(1, sizeof(*k));
  k->host = host;
  snprintf(k->name, sizeof(k->name), "%s", name);
  k->next = kernels;
  kernels = k;
}
struct var {
  const void* host;
  void* mem;
  struct var* next;
};
static struct var* vars = NULL;
void __cudaRegisterVar(void** h, char* host, char* dev, const char* name, int ext, size_t size, int constant, int global) {
  (void)h, (void)dev, (void)name, (void)ext, (void)constant, (void)global;
  struct var* v = calloc(1, sizeof(*v));
  v->host = host;
  v->mem = calloc(1, size);
  v->next = vars;
  vars = v;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
  for (struct var* v = vars; v; v = v->next)
    if (v->host == symbol) {
      *p = v->mem;
      return cudaSuccess;
    }
  return cudaErrorInvalidSymbol;
}

static __thread struct {
  dim3 grid, block;
  size_t smem;
  void* stream;
} conf;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
  conf.grid = grid;
  conf.block = block;
  conf.smem = smem;
  conf.stream = stream;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = conf.grid;
  *block = conf.block;
  *smem = conf.smem;
  *(void**)stream = conf.stream;
  return cudaSuccess;
}

/* ---- devices, streams, events */
static __thread int current = 0;
static __thread cudaError_t last = cudaSuccess;
static cudaError_t err(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
struct stream {
  int device, capturing;
};

static cudaError_t launch(const void* f, void* s) {
  if (s && ((struct stream*)s)->device != current) return err(cudaErrorInvalidResourceHandle);
  for (struct kernel* k = kernels; k; k = k->next)
    if (k->host == f) {
      k->launches++;
      launches++;
      return cudaSuccess;
    }
  return err(cudaErrorInvalidDeviceFunction);
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t s) {
  (void)grid, (void)block, (void)args, (void)smem;
  return launch(f, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  (void)args;
  for (unsigned i = 0; i < c->numAttrs; i++) {
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension && opt[O_CLUSTERS] < 1) return err(cudaErrorLaunchOutOfResources);
    if (c->attrs[i].id == cudaLaunchAttributeCooperative && opt[O_SMS] * opt[O_BLOCKS] < (long)c->gridDim.x)
      return err(cudaErrorCooperativeLaunchTooLarge);
  }
  return launch(f, c->stream);
}
cudaError_t cudaSetDevice(int d) {
  current = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = current;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? (int)opt[O_SMS] : a == cudaDevAttrCooperativeLaunch ? (int)opt[O_COOP] : 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) {
  (void)e;
  return "stand-in error";
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  (void)f;
  struct stream* p = calloc(1, sizeof(*p));
  p->device = current;
  *s = (cudaStream_t)p;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  (void)s;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) {
  (void)m;
  ((struct stream*)s)->capturing = 1;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  ((struct stream*)s)->capturing = 0;
  *g = malloc(1);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long f) {
  (void)g, (void)f;
  *x = malloc(1);
  return cudaSuccess;
}
static long graphs = 0;
long fake_graph_launches(void) { return graphs; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  (void)x, (void)s;
  graphs++;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  free(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  free(x);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) {
  (void)f;
  *e = malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  (void)e, (void)s;
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  (void)e;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  (void)e;
  if (on_wait) on_wait();
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  (void)a, (void)b;
  *ms = 0;
  return cudaSuccess;
}

/* ---- memory: a size in front of each block */
#define HEAD 256
static cudaError_t take(void** p, size_t n, long most, int counted) {
  if ((long)n > most) return err(cudaErrorMemoryAllocation);
  char* b = aligned_alloc(256, (HEAD + n + 255) / 256 * 256);
  memset(b, 0, HEAD + n);
  ((size_t*)b)[0] = n;
  ((size_t*)b)[1] = (size_t)counted;
  if (counted) held += n;
  *p = b + HEAD;
  return cudaSuccess;
}
static cudaError_t give(void* p) {
  if (!p) return cudaSuccess;
  char* b = (char*)p - HEAD;
  if (((size_t*)b)[1]) held -= ((size_t*)b)[0];
  free(b);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, opt[O_MALLOC_MAX], 1); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t q, cudaStream_t s) {
  (void)q, (void)s;
  static unsigned char fresh = 0;
  const cudaError_t e = take(p, n, (long)n == opt[O_POOL_REFUSED] ? -1 : 1L << 40, 0); /* this size is refused */
  if (e == cudaSuccess) memset(*p, ++fresh, n); /* not cleared, and no two alike */
  return e;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  (void)s;
  return give(p);
}
/* pinned memory; the last block of an int is the flag that an adaptive run polls */
static int* flag = NULL;
void fake_clear_flag(void) {
  if (flag) *flag = 0;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) {
  (void)f;
  const cudaError_t e = take(p, n, opt[O_PINNED_MAX], 0);
  if (e == cudaSuccess && n == sizeof(int)) flag = *p;
  return e;
}
cudaError_t cudaFreeHost(void* p) { return give(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* q, const struct cudaMemPoolProps* props) {
  (void)props;
  *q = malloc(1);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t q) {
  free(q);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t q, enum cudaMemPoolAttr a, void* v) {
  (void)q, (void)a, (void)v;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* fr, size_t* tot) {
  *fr = (size_t)16 << 30;
  *tot = (size_t)16 << 30;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  (void)k;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)st;
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s) {
  (void)s;
  return cudaMemset(d, v, n);
}

/* ---- limits of a kernel */
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  (void)f, (void)a, (void)v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, size_t smem, unsigned flags) {
  (void)f, (void)threads, (void)smem, (void)flags;
  *n = (int)opt[O_BLOCKS];
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int threads, size_t smem) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, threads, smem, 0);
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
  (void)f, (void)c;
  *n = (int)opt[O_CLUSTERS];
  return cudaSuccess;
}
static int encode_tiled() { return (int)opt[O_ENCODE]; }
cudaError_t cudaGetDriverEntryPoint(const char* symbol, void** p, unsigned long long flags, enum cudaDriverEntryPointQueryResult* r) {
  (void)symbol, (void)flags;
  *p = (void*)encode_tiled;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
