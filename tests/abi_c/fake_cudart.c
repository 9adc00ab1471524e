/* A CUDA runtime for the host side of the library: no device, every call
 * recorded.  Linked with the library's objects in the runtime's place, it
 * answers as a machine of `fake_devices` GPUs would, with the failures a test
 * asks for: a launch whose dynamic shared memory is above the limit set on
 * the current device fails, cooperative launches can be refused. */
#include <cuda_runtime_api.h>
#include <string.h>

#define EXPORT __attribute__((visibility("default")))
enum { kMaxKernels = 512, kMaxLaunches = 65536, kMaxDevices = 4, kMaxMemsets = 4096, kArgBytes = 96 };

static struct { const void* host; char name[512]; int limit[kMaxDevices]; } g_kernel[kMaxKernels];
static int g_kernels;
static struct { int kernel, device, cooperative, overlapped; unsigned grid[3], block; size_t smem; unsigned char arg0[kArgBytes]; }
    g_launch[kMaxLaunches];
static int g_launches;
static struct { const void* p; size_t bytes; } g_memset[kMaxMemsets];
static int g_memsets;
static int g_device, g_sms = 152, g_refuse_cooperative, g_clusters = 1;
static cudaError_t g_last;

static cudaError_t fail(cudaError_t e) { return g_last = e; }
static int find(const void* host) {
  for (int k = 0; k < g_kernels; ++k)
    if (g_kernel[k].host == host) return k;
  return -1;
}

/* ------------------------------------------------------- the test's side */
EXPORT void fake_reset(void) { g_launches = g_memsets = 0; g_last = cudaSuccess; }
EXPORT void fake_set(int device, int sms, int refuse_cooperative, int clusters) {
  g_device = device; g_sms = sms; g_refuse_cooperative = refuse_cooperative; g_clusters = clusters;
}
EXPORT int fake_launches(void) { return g_launches; }
EXPORT const char* fake_launch(int i, int* v, size_t* smem, unsigned char* arg0) {
  v[0] = g_launch[i].device; v[1] = g_launch[i].cooperative; v[2] = (int)g_launch[i].grid[0];
  v[3] = (int)g_launch[i].block; v[4] = g_launch[i].overlapped;
  *smem = g_launch[i].smem;
  memcpy(arg0, g_launch[i].arg0, kArgBytes);
  return g_kernel[g_launch[i].kernel].name;
}
EXPORT int fake_memsets(void) { return g_memsets; }
EXPORT const void* fake_memset(int i, size_t* bytes) { *bytes = g_memset[i].bytes; return g_memset[i].p; }

/* ---------------------------------------------------- registered kernels */
void** __cudaRegisterFatBinary(void* b) { static void* h; (void)b; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void** h, const char* host, char* fun, const char* name, int n, void* a, void* b, void* c,
                            void* d, int* e) {
  (void)h; (void)fun; (void)n; (void)a; (void)b; (void)c; (void)d; (void)e;
  if (g_kernels == kMaxKernels) return;
  g_kernel[g_kernels].host = host;
  strncpy(g_kernel[g_kernels].name, name, sizeof(g_kernel[0].name) - 1);
  for (int k = 0; k < kMaxDevices; ++k) g_kernel[g_kernels].limit[k] = 48 * 1024;
  ++g_kernels;
}
void __cudaRegisterVar(void** h, char* v, char* a, const char* n, int e, size_t s, int c, int g) {
  (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}

/* -------------------------------------------------------------- launches */
static cudaError_t launch(const void* host, dim3 grid, dim3 block, size_t smem, int cooperative, int overlapped,
                          void** args) {
  const int k = find(host);
  if (k < 0) return fail(cudaErrorInvalidDeviceFunction);
  if (smem > (size_t)g_kernel[k].limit[g_device] || grid.x == 0 || grid.y == 0 || grid.z == 0)
    return fail(cudaErrorInvalidValue);
  if (cooperative && g_refuse_cooperative) return fail(cudaErrorCooperativeLaunchTooLarge);
  if (g_launches == kMaxLaunches) return fail(cudaErrorUnknown);
  g_launch[g_launches].kernel = k;
  g_launch[g_launches].device = g_device;
  g_launch[g_launches].cooperative = cooperative;
  g_launch[g_launches].overlapped = overlapped;
  g_launch[g_launches].grid[0] = grid.x; g_launch[g_launches].grid[1] = grid.y; g_launch[g_launches].grid[2] = grid.z;
  g_launch[g_launches].block = block.x;
  g_launch[g_launches].smem = smem;
  /* (the time-blocked kernels' first argument is longer than this) */
  memset(g_launch[g_launches].arg0, 0, kArgBytes);
  if (strstr(g_kernel[k].name, "blk_") || strstr(g_kernel[k].name, "run_"))
    memcpy(g_launch[g_launches].arg0, args[0], kArgBytes);
  ++g_launches;
  return cudaSuccess;
}
static struct { dim3 grid, block; size_t smem; void* st; } g_call;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* st) {
  g_call.grid = grid; g_call.block = block; g_call.smem = smem; g_call.st = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
  *grid = g_call.grid; *block = g_call.block; *smem = g_call.smem; *(void**)st = g_call.st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) { *k = (cudaKernel_t)host; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t st) {
  (void)st;
  return launch((const void*)k, grid, block, smem, 0, 0, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* host, void** args) {
  int coop = 0, overlapped = 0;
  for (unsigned n = 0; n < cfg->numAttrs; ++n) {
    if (cfg->attrs[n].id == cudaLaunchAttributeCooperative) coop = cfg->attrs[n].val.cooperative;
    if (cfg->attrs[n].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      overlapped = cfg->attrs[n].val.programmaticStreamSerializationAllowed;
  }
  return launch(host, cfg->gridDim, cfg->blockDim, cfg->dynamicSmemBytes, coop, overlapped, args);
}

/* ----------------------------------------------------------------- others */
static int encode(void) { return 0; }  /* cuTensorMapEncodeTiled */
cudaError_t cudaGetDriverEntryPointByVersion(const char* s, void** f, unsigned v, unsigned long long flags,
                                             enum cudaDriverEntryPointQueryResult* q) {
  (void)s; (void)v; (void)flags;
  *f = (void*)encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? g_sms : 1;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* host, enum cudaFuncAttribute a, int v) {
  const int k = find(host);
  if (k < 0) return fail(cudaErrorInvalidDeviceFunction);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_kernel[k].limit[g_device] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
  (void)f; (void)c;
  *n = g_clusters;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  (void)v; (void)st;
  if (g_memsets < kMaxMemsets) { g_memset[g_memsets].p = p; g_memset[g_memsets++].bytes = n; }
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)d; (void)s; (void)n; (void)k; (void)st;
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbolAsync(void* d, const void* s, size_t n, size_t o, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)d; (void)s; (void)n; (void)o; (void)k; (void)st;
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void* d, const void* s, size_t n, size_t o, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)d; (void)s; (void)n; (void)o; (void)k; (void)st;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = (void*)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) { (void)st; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = 0; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) { (void)e; (void)st; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 0.f; return cudaSuccess; }
