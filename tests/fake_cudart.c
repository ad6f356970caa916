/* A CUDA runtime without a device, preloaded in place of libcudart by CPU
 * tests of the library's host code: device memory is host memory, kernels are
 * not run, and every event and stream is complete at once.  Calls that matter
 * to a test are logged, event queries can be made to fail, and a stream can be
 * put under capture, where the calls that a capture forbids fail as the
 * runtime's do. */
#include <pthread.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef struct { unsigned x, y, z; } dim;
typedef struct { dim grid, block; size_t smem; void* stream; } config;
enum { OK = 0, NO_MEMORY = 2, CAPTURE_UNSUPPORTED = 900 };

static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static char text[1 << 20];
static size_t used;
static struct { const void* fn; const char* name; } kernels[4096];
static int nkernels, capture, capture_mode, query, cooperative;
static __thread config pushed;

static void note(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    pthread_mutex_lock(&mu);
    if (used < sizeof(text) - 512) used += (size_t)vsnprintf(text + used, 512, fmt, ap);
    pthread_mutex_unlock(&mu);
    va_end(ap);
}
static int forbidden(void) { return capture && capture_mode != 2 ? CAPTURE_UNSUPPORTED : OK; }
static int launch(const void* fn, void** args) {
    const char* name = "?";
    for (int i = 0; i < nkernels; i++)
        if (kernels[i].fn == fn) name = kernels[i].name;
    if (strstr(name, "k_selftest_wait")) **(int**)args[0] = 2; /* all that it does */
    note("launch %s%s\n", name, capture ? " captured" : "");
    return OK;
}

/* For the test: the log so far (emptied), the status of event queries and of
 * cooperative launches, capture. */
size_t fake_log(char* out, size_t n) {
    pthread_mutex_lock(&mu);
    const size_t k = used < n ? used : n;
    memcpy(out, text, k);
    used = 0;
    pthread_mutex_unlock(&mu);
    return k;
}
void fake_event_query(int status) { query = status; }
void fake_capture(int on) { capture = on; }
void fake_cooperative(int status) { cooperative = status; }

/* Registration and launches. */
void** __cudaRegisterFatBinary(void* p) { static void* h; (void)p; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void) {}
void __cudaRegisterFunction(void** h, const char* fn, char* d, const char* name) {
    (void)h, (void)d;
    if (nkernels < 4096) {
        kernels[nkernels].fn = fn;
        kernels[nkernels++].name = name;
    }
}
unsigned __cudaPushCallConfiguration(dim g, dim b, size_t smem, void* s) {
    pushed = (config){g, b, smem, s};
    return OK;
}
int __cudaPopCallConfiguration(dim* g, dim* b, size_t* smem, void** s) {
    *g = pushed.grid, *b = pushed.block, *smem = pushed.smem, *s = pushed.stream;
    return OK;
}
int cudaLaunchKernel(const void* fn, dim g, dim b, void** a, size_t m, void* s) {
    (void)g, (void)b, (void)m, (void)s;
    return launch(fn, a);
}
int cudaLaunchCooperativeKernel(const void* fn, dim g, dim b, void** a, size_t m, void* s) {
    (void)g, (void)b, (void)m, (void)s;
    return cooperative ? cooperative : launch(fn, a);
}
int cudaLaunchKernelExC(const void* cfg, const void* fn, void** a) {
    (void)cfg;
    return launch(fn, a);
}
int cudaFuncSetAttribute(const void* fn, int a, int v) { (void)fn, (void)a, (void)v; return OK; }

/* Device. */
int cudaGetDeviceCount(int* n) { *n = 1; return OK; }
int cudaGetDevice(int* d) { *d = 0; return OK; }
int cudaSetDevice(int d) { (void)d; return OK; }
int cudaDeviceGetAttribute(int* v, int attr, int d) {
    (void)d;
    *v = attr == 16 ? 148 : 1; /* multiprocessors; cooperative launch */
    return OK;
}
int cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = 0, *hi = -5; return OK; }
int cudaGetDriverEntryPoint(const char* s, void** p, uint64_t f, int* q) {
    (void)s, (void)f;
    *p = NULL, *q = 1;
    return OK;
}
int cudaGetSymbolAddress(void** p, const void* s) { *p = (void*)s; return OK; }
int cudaGetLastError(void) { return OK; }
const char* cudaGetErrorString(int e) { (void)e; return "error of the fake runtime"; }

/* Memory. */
static int alloc(void** p, size_t n) {
    if (posix_memalign(p, 256, n ? n : 1)) return NO_MEMORY;
    memset(*p, 0x5a, n);
    return OK;
}
int cudaMalloc(void** p, size_t n) {
    note("malloc\n");
    return forbidden() ? forbidden() : alloc(p, n);
}
int cudaFree(void* p) {
    if (p) note("free\n");
    if (p && forbidden()) return forbidden();
    free(p);
    return OK;
}
int cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; return alloc(p, n); }
int cudaFreeHost(void* p) { free(p); return OK; }
int cudaMemPoolCreate(void** p, const void* a) { (void)a; *p = NULL; return OK; }
int cudaMemPoolSetAttribute(void* p, int a, void* v) { (void)p, (void)a, (void)v; return OK; }
int cudaMemPoolDestroy(void* p) { (void)p; return OK; }
int cudaMallocFromPoolAsync(void** p, size_t n, void* q, void* s) {
    (void)q, (void)s;
    return alloc(p, n);
}
int cudaFreeAsync(void* p, void* s) { (void)s; free(p); return OK; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) {
    (void)kind, (void)st;
    note("copy%s\n", capture ? " captured" : "");
    if (!capture) memcpy(d, s, n);
    return OK;
}
int cudaMemsetAsync(void* d, int v, size_t n, void* st) {
    (void)st;
    note("memset%s\n", capture ? " captured" : "");
    if (!capture) memset(d, v, n);
    return OK;
}

/* Streams and events. */
int cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; return alloc(s, 1); }
int cudaStreamCreateWithPriority(void** s, unsigned f, int p) {
    (void)f, (void)p;
    return alloc(s, 1);
}
int cudaStreamDestroy(void* s) { free(s); return OK; }
int cudaStreamSynchronize(void* s) {
    (void)s;
    note("sync\n");
    return capture ? CAPTURE_UNSUPPORTED : OK;
}
int cudaStreamWaitEvent(void* s, void* e, unsigned f) { (void)s, (void)e, (void)f; return OK; }
int cudaStreamIsCapturing(void* s, int* status) { (void)s; *status = capture; return OK; }
int cudaThreadExchangeStreamCaptureMode(int* mode) {
    const int m = capture_mode;
    capture_mode = *mode;
    *mode = m;
    return OK;
}
int cudaEventCreate(void** e) { return alloc(e, 1); }
int cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; return alloc(e, 1); }
int cudaEventDestroy(void* e) { free(e); return OK; }
int cudaEventRecord(void* e, void* s) { (void)e, (void)s; return OK; }
int cudaEventSynchronize(void* e) { (void)e; return OK; }
int cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a, (void)b; *ms = 0; return OK; }
int cudaEventQuery(void* e) { (void)e; return query; }
