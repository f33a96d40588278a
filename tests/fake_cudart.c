/* A CUDA runtime without a device, for tests of the library's host side on the CPU (loaded before the real one;
 * see fake_cuda.py): device memory is host memory, copies are memcpy, launches do nothing but are counted and may
 * be refused, and cudaMemset takes effect when the legacy stream is waited for.  Compiled without CUDA's headers: only the names and the argument registers matter. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;
typedef struct { unsigned x, y, z; } dim3_t;
enum { REFUSED = 701 /* cudaErrorLaunchOutOfResources */ };

static err_t last_error;
static long launches, refuse_at, graphs, attribute_queries;
static unsigned long long allocated, uploaded;
static void* copy_dst[4096];
static size_t copy_bytes[4096];
static int copies;
static const char* kernel_name[4096];
static const void* kernel_stub[4096];
static int kernels;
static const char* launched[1 << 16];
static struct { void* p; int v; size_t n; } zeroing[4096];   /* queued on the legacy stream */
static int queued, copying;   /* copying: the last pageable cudaMemcpy to the device may still be on its way */
static void run_legacy_stream(void) {
    for (int i = 0; i < queued; i++) memset(zeroing[i].p, zeroing[i].v, zeroing[i].n);
    queued = copying = 0;
}

#define API __attribute__((visibility("default")))

/* ---- what the tests read and set */
API void fake_reset(long refuse) {   /* refuse the launch of that number (1 the next one; 0: none) */
    launches = graphs = attribute_queries = 0;
    allocated = uploaded = 0;
    copies = 0;
    refuse_at = refuse;
}
API long fake_launches(void) { return launches; }
API long fake_graphs(void) { return graphs; }
API long fake_attribute_queries(void) { return attribute_queries; }
API unsigned long long fake_allocated(void) { return allocated; }
API unsigned long long fake_uploaded(void) { return uploaded; }
API int fake_copies(void) { return copies < 4096 ? copies : 4096; }
API void* fake_copy_dst(int i) { return copy_dst[i]; }
API unsigned long long fake_copy_bytes(int i) { return copy_bytes[i]; }
API int fake_queued(void) { return queued + copying; }   /* writes still queued on the legacy stream, which no other stream waits for */
API const char* fake_kernel(long i) { return launched[i & 0xFFFF] ? launched[i & 0xFFFF] : ""; }

/* ---- registration and launches */
API void** __cudaRegisterFatBinary(void* bin) { return (void**)&bin; }
API void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
API void __cudaUnregisterFatBinary(void** h) { (void)h; }
API void __cudaRegisterFunction(void** h, const char* stub, char* dev, const char* name, int limit, void* a, void* b, void* c,
                                void* d, int* e) {
    if (kernels < 4096) { kernel_stub[kernels] = stub; kernel_name[kernels++] = name; }
}
API void __cudaRegisterVar(void** h, char* var, char* dev, const char* name, int ext, size_t size, int constant, int global) {}
static dim3_t cfg_grid, cfg_block;
static size_t cfg_smem;
static void* cfg_stream;
API unsigned __cudaPushCallConfiguration(dim3_t g, dim3_t b, size_t smem, void* s) {
    cfg_grid = g; cfg_block = b; cfg_smem = smem; cfg_stream = s;
    return 0;
}
API err_t __cudaPopCallConfiguration(dim3_t* g, dim3_t* b, size_t* smem, void* s) {
    *g = cfg_grid; *b = cfg_block; *smem = cfg_smem; *(void**)s = cfg_stream;
    return 0;
}
static err_t launch(const void* stub) {
    launched[launches & 0xFFFF] = 0;
    for (int i = 0; i < kernels; i++)
        if (kernel_stub[i] == stub) launched[launches & 0xFFFF] = kernel_name[i];
    if (++launches == refuse_at) return last_error = REFUSED;
    return 0;
}
API err_t __cudaGetKernel(void** k, const void* stub) { *k = (void*)stub; return 0; }
API err_t __cudaLaunchKernel(void* k, dim3_t g, dim3_t b, void** args, size_t smem, void* s) { return launch(k); }
API err_t cudaLaunchKernelExC(const void* cfg, const void* stub, void** args) { return launch(stub); }
API err_t cudaGetLastError(void) { const err_t e = last_error; last_error = 0; return e; }

/* ---- memory */
API err_t cudaMalloc(void** p, size_t n) { allocated += n; return (*p = calloc(n ? n : 1, 1)) ? 0 : 2; }
API err_t cudaMallocAsync(void** p, size_t n, void* s) { return cudaMalloc(p, n); }
API err_t cudaHostAlloc(void** p, size_t n, unsigned f) { return (*p = calloc(n ? n : 1, 1)) ? 0 : 2; }
API err_t cudaFree(void* p) { run_legacy_stream(); free(p); return 0; }
API err_t cudaFreeAsync(void* p, void* s) { free(p); return 0; }
API err_t cudaFreeHost(void* p) { free(p); return 0; }
static err_t copy(void* d, const void* s, size_t n, int kind) {
    if (n) memmove(d, s, n);
    if (kind == 1) {   /* host to device */
        uploaded += n;
        if (copies < 4096) { copy_dst[copies] = d; copy_bytes[copies] = n; }
        copies++;
    }
    return 0;
}
API err_t cudaMemcpy(void* d, const void* s, size_t n, int kind) {
    run_legacy_stream();
    copying = kind == 1 && n != 0;   /* returns once the pageable source has been staged */
    return copy(d, s, n, kind);
}
API err_t cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) { return copy(d, s, n, kind); }
API err_t cudaMemset(void* d, int v, size_t n) {   /* returns before the device has written */
    if (queued == 4096) run_legacy_stream();
    zeroing[queued].p = d; zeroing[queued].v = v; zeroing[queued++].n = n;
    return 0;
}
API err_t cudaMemsetAsync(void* d, int v, size_t n, void* s) { memset(d, v, n); return 0; }
API err_t cudaGetSymbolAddress(void** p, const void* sym) { *p = (void*)sym; return 0; }

/* ---- device, streams, events, graphs */
API err_t cudaGetDevice(int* d) { *d = 0; return 0; }
API err_t cudaDeviceGetAttribute(int* v, int attr, int dev) { attribute_queries++; *v = 152; return 0; }
API err_t cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }
API err_t cudaStreamCreateWithFlags(void** s, unsigned f) { *s = malloc(1); return 0; }
API err_t cudaStreamDestroy(void* s) { free(s); return 0; }
API err_t cudaStreamSynchronize(void* s) { if (!s) run_legacy_stream(); return 0; }
API err_t cudaStreamWaitEvent(void* s, void* e, unsigned f) { return 0; }
API err_t cudaEventCreate(void** e) { *e = malloc(1); return 0; }
API err_t cudaEventCreateWithFlags(void** e, unsigned f) { return cudaEventCreate(e); }
API err_t cudaEventDestroy(void* e) { free(e); return 0; }
API err_t cudaEventRecord(void* e, void* s) { return 0; }
API err_t cudaEventSynchronize(void* e) { return 0; }
API err_t cudaEventElapsedTime(float* ms, void* a, void* b) { *ms = 1.f; return 0; }
API err_t cudaStreamBeginCapture(void* s, int m) { return 0; }
API err_t cudaStreamEndCapture(void* s, void** g) { *g = malloc(1); return 0; }
API err_t cudaGraphInstantiate(void** x, void* g, unsigned long long f) { graphs++; *x = malloc(1); return 0; }
API err_t cudaGraphDestroy(void* g) { free(g); return 0; }
API err_t cudaGraphExecDestroy(void* g) { free(g); return 0; }
API err_t cudaGraphLaunch(void* x, void* s) { return 0; }
