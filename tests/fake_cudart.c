/* Host stand-in for the CUDA runtime calls of libdmrgb200, preloaded by tests of the host logic:
 * device memory is host memory, kernels are not run but their launches recorded, streams, events
 * and graphs are tokens, and the n-th allocation can be made to fail. */
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

enum { OK = 0, ERR_MEMORY = 2 };
typedef struct { unsigned x, y, z; } dim3_;
typedef struct { dim3_ grid, block; size_t smem; void* stream; void* attrs; unsigned n_attrs; } launch_config;

static int last_error, fail_in, allocations;
static long live;
#define MAX_LAUNCHES 65536
static struct { const void* kernel; unsigned grid, block; } launches[MAX_LAUNCHES];
static int n_launches, capturing;

/* test controls */
void fake_fail_in(int n) { fail_in = n; }  /* the n-th allocation from now fails; 0: none */
int fake_allocations(void) { return allocations; }
long fake_live(void) { return live; }  /* allocations not yet freed */
void fake_clear(void) { n_launches = 0; }
int fake_launches(void) { return n_launches; }
void fake_launch(int i, unsigned long* kernel, unsigned* grid, unsigned* block) {
    *kernel = (unsigned long)launches[i].kernel;
    *grid = launches[i].grid;
    *block = launches[i].block;
}

static int allocate(void** p, size_t n) {
    ++allocations;
    if (fail_in && --fail_in == 0) return last_error = ERR_MEMORY;
    *p = calloc(n ? n : 1, 1);
    ++live;
    return OK;
}
static int release(void* p) {
    if (p) --live;
    free(p);
    return OK;
}
static int token(void** p) { return allocate(p, 1); }
static void record(const void* f, unsigned grid, unsigned block) {
    if (n_launches < MAX_LAUNCHES) {
        launches[n_launches].kernel = f;
        launches[n_launches].grid = grid;
        launches[n_launches].block = block;
        ++n_launches;
    }
}

int cudaSetDevice(int d) { (void)d; return OK; }
int cudaGetDevice(int* d) { *d = 0; return OK; }
int cudaDeviceGetAttribute(int* v, int a, int d) { (void)a; (void)d; *v = 148; return OK; }
int cudaGetLastError(void) { int e = last_error; last_error = OK; return e; }
const char* cudaGetErrorString(int e) { return e == ERR_MEMORY ? "out of memory" : "no error"; }
int cudaMalloc(void** p, size_t n) { return allocate(p, n); }
int cudaMallocAsync(void** p, size_t n, void* s) { (void)s; return allocate(p, n); }
int cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; return allocate(p, n); }
int cudaFree(void* p) { return release(p); }
int cudaFreeAsync(void* p, void* s) { (void)s; return release(p); }
int cudaFreeHost(void* p) { return release(p); }
int cudaMemcpy(void* d, const void* s, size_t n, int k) { (void)k; memcpy(d, s, n); return OK; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { (void)k; (void)st; memcpy(d, s, n); return OK; }
int cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return OK; }
int cudaMemsetAsync(void* d, int v, size_t n, void* s) { (void)s; memset(d, v, n); return OK; }
int cudaFuncSetAttribute(const void* f, int a, int v) { (void)f; (void)a; (void)v; return OK; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* o, const void* f, int b, size_t s, unsigned fl) {
    (void)f; (void)b; (void)s; (void)fl;
    *o = 2;
    return OK;
}
int cudaLaunchKernelExC(const launch_config* c, const void* f, void** args) {
    (void)args;
    record(f, c->grid.x, c->block.x);
    return OK;
}
int cudaLaunchKernel(const void* f, dim3_ grid, dim3_ block, void** args, size_t smem, void* s) {
    (void)args; (void)smem; (void)s;
    record(f, grid.x, block.x);
    return OK;
}
int cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; return token(s); }
int cudaStreamDestroy(void* s) { return release(s); }
int cudaStreamSynchronize(void* s) { (void)s; return OK; }
int cudaStreamWaitEvent(void* s, void* e, unsigned f) { (void)s; (void)e; (void)f; return OK; }
int cudaStreamIsCapturing(void* s, int* st) { (void)s; *st = capturing; return OK; }
int cudaStreamBeginCapture(void* s, int m) { (void)s; (void)m; capturing = 1; return OK; }
int cudaStreamEndCapture(void* s, void** g) { (void)s; capturing = 0; return token(g); }
int cudaEventCreate(void** e) { return token(e); }
int cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; return token(e); }
int cudaEventDestroy(void* e) { return release(e); }
int cudaEventRecord(void* e, void* s) { (void)e; (void)s; return OK; }
int cudaEventSynchronize(void* e) { (void)e; return OK; }
int cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a; (void)b; *ms = 1.0f; return OK; }
int cudaGraphInstantiate(void** x, void* g, unsigned long f) { (void)g; (void)f; return token(x); }
int cudaGraphDestroy(void* g) { return release(g); }
int cudaGraphExecDestroy(void* x) { return release(x); }
int cudaGraphLaunch(void* x, void* s) { (void)x; (void)s; return OK; }
