/* A CUDA runtime without a GPU, preloaded in front of the real one by test_many_row_host_cpu.py: it runs no kernel, it
 * records what the library asks for.  Like the real one it keeps a kernel's shared-memory limit per device and refuses a
 * launch beyond it.  cuBLAS is here too (three calls, looked up by name). */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define MAX 4096
#define API __attribute__((visibility("default")))

static struct { const void* host; char name[256]; } g_fn[MAX];
static struct { const void* fn; int device, value; } g_attr[MAX];
static int n_fn, n_attr, g_device, g_setup_calls, g_refuse_setup, g_refuse_encode, g_resident = 132;
static char g_log[1 << 20];
static size_t g_len;

API void fake_device(int d) { g_device = d; }
API void fake_refuse_setup(int v) { g_refuse_setup = v; }
static char g_refuse_kernel[64];
API void fake_refuse_setup_of(const char* part) { snprintf(g_refuse_kernel, sizeof g_refuse_kernel, "%s", part); }  /* kernels named so */
API void fake_refuse_encode(int v) { g_refuse_encode = v; }
API void fake_resident(int ctas) { g_resident = ctas; }  /* CTAs, one per SM, that clusters can have at once */
static int g_capturing = -1;
API void fake_capturing(int status) { g_capturing = status; }  /* of every stream: a cudaStreamCaptureStatus, or -1: cannot be asked for */
API int fake_setup_calls(void) { return g_setup_calls; }
API const char* fake_log(void) { return g_log; }
API void fake_clear(void) { g_len = 0; g_log[0] = 0; }
static void note(const char* s) { g_len += snprintf(g_log + g_len, sizeof(g_log) - g_len, "%s\n", s); }

static const char* name_of(const void* fn) {
  for (int i = 0; i < n_fn; ++i) if (g_fn[i].host == fn) return g_fn[i].name;
  return "?";
}

/* registration */
static void* g_handle;
API void** __cudaRegisterFatBinary(void* b) { (void)b; return &g_handle; }
API void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
API void __cudaUnregisterFatBinary(void** h) { (void)h; }
API void __cudaRegisterVar(void** h, char* a, char* b, const char* c, int d, size_t e, int f, int g) {
  (void)h; (void)a; (void)b; (void)c; (void)d; (void)e; (void)f; (void)g;
}
API void __cudaRegisterFunction(void** h, const char* host, char* dev, const char* name, int t, void* a, void* b, void* c, void* d, int* e) {
  (void)h; (void)dev; (void)t; (void)a; (void)b; (void)c; (void)d; (void)e;
  if (n_fn < MAX) {
    g_fn[n_fn].host = host;
    snprintf(g_fn[n_fn++].name, 256, "%s", name);
  }
}

/* set-up */
static cudaError_t setup(void) { ++g_setup_calls; return g_refuse_setup ? cudaErrorStreamCaptureUnsupported : cudaSuccess; }
API cudaError_t cudaFuncSetAttribute(const void* fn, enum cudaFuncAttribute a, int v) {
  if (setup() != cudaSuccess) return cudaErrorStreamCaptureUnsupported;
  if (g_refuse_kernel[0] && strstr(name_of(fn), g_refuse_kernel)) return cudaErrorInvalidValue;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && n_attr < MAX) {
    g_attr[n_attr].fn = fn; g_attr[n_attr].device = g_device; g_attr[n_attr++].value = v;
  }
  return cudaSuccess;
}
API cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* fn) { (void)fn; memset(a, 0, sizeof *a); a->sharedSizeBytes = 2048; return cudaSuccess; }
static int cluster_of(const cudaLaunchConfig_t* c) {
  int size = 1;
  for (unsigned i = 0; i < c->numAttrs; ++i) if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) size = c->attrs[i].val.clusterDim.x * c->attrs[i].val.clusterDim.y;
  return size;
}
API cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* fn, const cudaLaunchConfig_t* c) {
  (void)fn;
  *n = g_resident / cluster_of(c);
  return setup();
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* fn, int t, size_t s) { (void)fn; (void)t; (void)s; *n = 1; return cudaSuccess; }
API cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
static int encode(void) { return g_refuse_encode ? 1 : 0; }
API cudaError_t cudaGetDriverEntryPointByVersion(const char* s, void** f, unsigned v, unsigned long long fl, enum cudaDriverEntryPointQueryResult* q) {
  (void)s; (void)v; (void)fl;
  *f = (void*)encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

/* memory */
API cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n < 4096 ? 4096 : 4096); (void)n; return cudaSuccess; }
API cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
API cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { (void)d; (void)s; (void)n; (void)k; return cudaSuccess; }
API cudaError_t cudaMemset(void* p, int v, size_t n) { (void)p; (void)v; (void)n; return cudaSuccess; }
API cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
API cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* status) {
  (void)s;
  if (g_capturing < 0) return cudaErrorStreamCaptureImplicit;
  *status = (enum cudaStreamCaptureStatus)g_capturing;
  return cudaSuccess;
}
API cudaError_t cudaGetLastError(void) { return cudaSuccess; }
API const char* cudaGetErrorString(cudaError_t e) { static char b[32]; snprintf(b, sizeof b, "error %d", (int)e); return b; }

/* launches */
static cudaError_t launch(const void* fn, unsigned x, unsigned y, unsigned threads, size_t smem, int cluster, int pdl) {
  char line[512];
  int limit = 48 * 1024;
  for (int i = 0; i < n_attr; ++i) if (g_attr[i].fn == fn && g_attr[i].device == g_device) limit = g_attr[i].value;
  if (smem > (size_t)limit) return cudaErrorInvalidValue;
  snprintf(line, sizeof line, "launch %s device=%d grid=%u,%u threads=%u smem=%zu cluster=%d pdl=%d", name_of(fn), g_device, x, y, threads, smem, cluster, pdl);
  note(line);
  return cudaSuccess;
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) {
  int pdl = 0;
  (void)args;
  for (unsigned i = 0; i < c->numAttrs; ++i) if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) pdl = c->attrs[i].val.programmaticStreamSerializationAllowed;
  return launch(fn, c->gridDim.x, c->gridDim.y, c->blockDim.x, c->dynamicSmemBytes, cluster_of(c), pdl);
}
static dim3 g_grid, g_block;
static size_t g_smem;
static cudaStream_t g_stream;
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t t) { g_grid = g; g_block = b; g_smem = s; g_stream = t; return 0; }
API cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* t) { *g = g_grid; *b = g_block; *s = g_smem; *(cudaStream_t*)t = g_stream; return cudaSuccess; }
API cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void** args, size_t s, cudaStream_t t) { (void)args; (void)t; return launch(fn, g.x, g.y, b.x, s, 1, 0); }

/* cuBLAS */
API int cublasCreate_v2(void** h) { static int one; *h = &one; return 0; }
API int cublasSetStream_v2(void* h, cudaStream_t s) { (void)h; (void)s; return 0; }
API int cublasGemmEx(void* h, int ta, int tb, int m, int n, int k) {
  char line[128];
  (void)h; (void)ta; (void)tb;
  snprintf(line, sizeof line, "cublas %d,%d,%d", m, n, k);
  note(line);
  return 0;
}
