/* The part of the CUDA runtime that libhfgpu.so calls, on host memory and without a GPU: kernels are skipped,
 * allocations can be made to fail.  Preloaded by tests of the engine's host side (error paths that must not be
 * provoked on a device); what is not defined here (module registration) comes from the real runtime. */
#include <stdlib.h>
#include <string.h>

static long fail_after = -1; /* allocations that still succeed; -1: all */
static long uploads    = 0;
static int last_error  = 0;

void fake_fail_malloc(long after) { fail_after = after; }
long fake_uploads(void) { return uploads; }

static int fail(int code) { return last_error = code; }

int cudaMalloc(void** p, size_t n)
{
    if (fail_after == 0)
        return fail(2); /* cudaErrorMemoryAllocation */
    if (fail_after > 0)
        --fail_after;
    *p = calloc(n ? n : 1, 1);
    return *p ? 0 : fail(2);
}
int cudaFree(void* p) { free(p); return 0; }
int cudaHostAlloc(void** p, size_t n, unsigned flags) { (void)flags; return (*p = calloc(n ? n : 1, 1)) ? 0 : fail(2); }
int cudaFreeHost(void* p) { free(p); return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st)
{
    (void)st;
    uploads += kind == 1; /* cudaMemcpyHostToDevice */
    memcpy(d, s, n);
    return 0;
}
int cudaMemcpy(void* d, const void* s, size_t n, int kind) { return cudaMemcpyAsync(d, s, n, kind, 0); }
int cudaMemsetAsync(void* d, int v, size_t n, void* st) { (void)st; memset(d, v, n); return 0; }
int cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 36; return 0; }
int cudaSetDevice(int d) { (void)d; return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaGetDeviceCount(int* n) { *n = 1; return 0; }
int cudaDeviceGetAttribute(int* v, int a, int d) { (void)a; (void)d; *v = 152; return 0; }
int cudaGetLastError(void) { int e = last_error; last_error = 0; return e; }
const char* cudaGetErrorString(int e) { return e == 2 ? "out of memory" : "error"; }
int cudaEventCreate(void** e) { *e = e; return 0; }
int cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; *e = e; return 0; }
int cudaEventDestroy(void* e) { (void)e; return 0; }
int cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a; (void)b; *ms = 0; return 0; }
int cudaEventRecord(void* e, void* s) { (void)e; (void)s; return 0; }
int cudaEventSynchronize(void* e) { (void)e; return 0; }
int cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; *s = s; return 0; }
int cudaStreamDestroy(void* s) { (void)s; return 0; }
int cudaStreamSynchronize(void* s) { (void)s; return 0; }
int cudaStreamWaitEvent(void* s, void* e, unsigned f) { (void)s; (void)e; (void)f; return 0; }
int cudaFuncSetAttribute(const void* f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t m, unsigned fl)
{
    (void)f; (void)b; (void)m; (void)fl;
    *n = 1;
    return 0;
}
/* Non-zero: a <<<>>> launch is skipped. */
unsigned __cudaPushCallConfiguration(void) { return 1; }
