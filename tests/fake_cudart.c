/* A stand-in for the CUDA runtime's entry points that the library calls, preloaded by
 * tests of its host side: device memory is host memory, kernels do nothing, and each
 * call is noted as one letter; FAKE_SMS in the environment is the device's number of
 * SMs (152).  fake_fail_launch(n) makes the n-th kernel launch from
 * then on fail as a launch can. */
#include <stdlib.h>
#include <string.h>

static char log_[1 << 20];
static int n_, fail_, err_;
static void note(char c) { if (n_ < (int)sizeof(log_) - 1) log_[n_++] = c; }
const char* fake_log(void) { log_[n_] = 0; return log_; }
void fake_clear(void) { n_ = 0; }
void fake_fail_launch(int n) { fail_ = n; }

typedef struct { unsigned x, y, z; } dim3_;
static dim3_ g_, b_;
static size_t s_;
static void* st_;

int cudaMalloc(void** p, size_t n) { note('m'); *p = calloc(1, n ? n : 1); return *p ? 0 : 2; }
int cudaFree(void* p) { free(p); return 0; }
int cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; *p = calloc(1, n ? n : 1); return *p ? 0 : 2; }
int cudaFreeHost(void* p) { free(p); return 0; }
static int copy(void* d, const void* s, size_t n, int kind) { note(kind == 1 ? 'u' : kind == 2 ? 'd' : 'c'); memmove(d, s, n); return 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int kind) { return copy(d, s, n, kind); }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) { (void)st; return copy(d, s, n, kind); }
int cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return 0; }
int cudaMemsetAsync(void* d, int v, size_t n, void* st) { (void)st; memset(d, v, n); return 0; }
int cudaDeviceGetAttribute(int* v, int a, int dev) { (void)dev; *v = a == 16 ? (getenv("FAKE_SMS") ? atoi(getenv("FAKE_SMS")) : 152) : 0; return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaEventCreate(void** e) { *e = malloc(1); return 0; }
int cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; return cudaEventCreate(e); }
int cudaEventDestroy(void* e) { free(e); return 0; }
int cudaEventRecord(void* e, void* st) { (void)e; (void)st; note('E'); return 0; }
int cudaEventSynchronize(void* e) { (void)e; return 0; }
int cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a; (void)b; *ms = 1.0f; return 0; }
int cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; *s = malloc(1); return 0; }
int cudaStreamDestroy(void* s) { free(s); return 0; }
int cudaStreamSynchronize(void* s) { (void)s; note('S'); return 0; }
int cudaStreamWaitEvent(void* s, void* e, unsigned f) { (void)s; (void)e; (void)f; return 0; }
int cudaStreamBeginCapture(void* s, int m) { (void)s; (void)m; note('['); return 0; }
int cudaStreamEndCapture(void* s, void** g) { (void)s; note(']'); *g = malloc(1); return 0; }
int cudaGraphInstantiate(void** e, void* g, unsigned long long f) { (void)g; (void)f; *e = malloc(1); return 0; }
int cudaGraphDestroy(void* g) { free(g); return 0; }
int cudaGraphExecDestroy(void* e) { free(e); return 0; }
int cudaGraphLaunch(void* e, void* s) { (void)e; (void)s; note('G'); return 0; }
int cudaGetLastError(void) { int e = err_; err_ = 0; return e; }
int cudaFuncSetAttribute(const void* f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned fl) {
    (void)f; (void)b; (void)s; (void)fl;
    *n = 8;
    return 0;
}
int __cudaGetKernel(void** k, const void* f) { *k = (void*)f; return 0; }
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t s, void* st) { g_ = g; b_ = b; s_ = s; st_ = st; return 0; }
int __cudaPopCallConfiguration(dim3_* g, dim3_* b, size_t* s, void* st) { *g = g_; *b = b_; *s = s_; *(void**)st = st_; return 0; }
static int launch(char c) {
    if (fail_ > 0 && --fail_ == 0) {
        note('!');
        return err_ = 701;   /* cudaErrorLaunchOutOfResources */
    }
    note(c);
    return 0;
}
int __cudaLaunchKernel(void* k, dim3_ g, dim3_ b, void** a, size_t s, void* st) {
    (void)k; (void)g; (void)b; (void)a; (void)s; (void)st;
    return launch('K');
}
static size_t dyn_;
size_t fake_dynamic_smem(void) { size_t d = dyn_; dyn_ = 0; return d; }   /* the largest since the last call */
int cudaLaunchKernelExC(const void* cfg, const void* f, void** a) {
    const size_t d = *(const size_t*)((const char*)cfg + 2 * sizeof(dim3_));   /* cudaLaunchConfig_t: grid, block, dynamic shared memory */
    (void)f; (void)a;
    if (d > dyn_) dyn_ = d;
    return launch('X');
}
