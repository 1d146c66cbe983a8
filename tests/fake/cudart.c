/* A CUDA runtime without a GPU, for tests of the host code's error paths: the
 * library's own objects are linked against it (tests/fake_cuda.py).  Device
 * memory is host memory, copies are done at once, kernels are not run: a launch
 * is handed to fake_check (check.cu), which says whether it would have been
 * safe.  fake_fail makes a chosen call fail. */
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

typedef struct { unsigned x, y, z; } dim3_t;
enum { OK = 0, ERR_VALUE = 1, ERR_MEMORY = 2, ERR_CONFIG = 9, ERR_UNSUPPORTED = 801 };

#define MAX_BLOCKS 4096
static struct { char* p; size_t n; } blocks[MAX_BLOCKS];
static long fail_malloc, fail_launch;     /* calls until one fails (0: none) */
static int last_error, max_cluster = 16;
static long launches, unsafe_launches, clusters[17];
static char why[256];

int fake_check(const void* f, void** args, unsigned grid, char* why, size_t n);
unsigned fake_cluster(const void* config);

void fake_fail(long mallocs, long launch) { fail_malloc = mallocs; fail_launch = launch; }
void fake_max_cluster(int n) { max_cluster = n; }
long fake_launches(void) { return launches; }
long fake_unsafe(void) { return unsafe_launches; }
long fake_clusters(int n) { return clusters[n]; }
const char* fake_why(void) { return why; }
/* bytes from p to the end of the live block that holds it; 0 if none does */
size_t fake_room(const void* p) {
    for (int i = 0; i < MAX_BLOCKS; ++i)
        if (blocks[i].p && (const char*)p >= blocks[i].p && (const char*)p < blocks[i].p + blocks[i].n)
            return (size_t)(blocks[i].p + blocks[i].n - (const char*)p);
    return 0;
}
size_t fake_allocated(void) {
    size_t t = 0;
    for (int i = 0; i < MAX_BLOCKS; ++i) t += blocks[i].p ? blocks[i].n : 0;
    return t;
}

static int err(int e) { if (e) last_error = e; return e; }

int cudaMalloc(void** p, size_t n) {
    *p = NULL;
    if (fail_malloc > 0 && --fail_malloc == 0) return err(ERR_MEMORY);
    for (int i = 0; i < MAX_BLOCKS; ++i)
        if (!blocks[i].p) {
            if (!(blocks[i].p = (char*)malloc(n ? n : 1))) return err(ERR_MEMORY);
            blocks[i].n = n;
            *p = blocks[i].p;
            return OK;
        }
    return err(ERR_MEMORY);
}
int cudaFree(void* p) {
    for (int i = 0; p && i < MAX_BLOCKS; ++i)
        if (blocks[i].p == p) { free(p); blocks[i].p = NULL; }
    return OK;
}
int cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; return (*p = calloc(1, n)) ? OK : err(ERR_MEMORY); }
int cudaFreeHost(void* p) { free(p); return OK; }
int cudaMemcpy(void* d, const void* s, size_t n, int k) { (void)k; memcpy(d, s, n); return OK; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { (void)k; (void)st; memcpy(d, s, n); return OK; }
int cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return OK; }
int cudaMemsetAsync(void* p, int v, size_t n, void* st) { (void)st; memset(p, v, n); return OK; }

static int launch(const void* f, unsigned grid, void** args) {
    if (fail_launch > 0 && --fail_launch == 0) return err(ERR_CONFIG);
    ++launches;
    if (!fake_check(f, args, grid, why, sizeof why)) ++unsafe_launches;
    return OK;
}
int cudaLaunchKernel(const void* f, dim3_t g, dim3_t b, void** args, size_t smem, void* st) {
    (void)b; (void)smem; (void)st;
    return launch(f, g.x, args);
}
int __cudaLaunchKernel(const void* f, dim3_t g, dim3_t b, void** args, size_t smem, void* st) {
    return cudaLaunchKernel(f, g, b, args, smem, st);
}
int cudaLaunchKernelExC(const void* config, const void* f, void** args) {
    const unsigned n = fake_cluster(config);
    if ((int)n > max_cluster) return err(ERR_CONFIG);
    ++clusters[n <= 16 ? n : 0];
    return launch(f, *(const unsigned*)config, args);
}
int __cudaGetKernel(const void** k, const void* f) { *k = f; return OK; }

int cudaGetDeviceCount(int* n) { *n = 1; return OK; }
int cudaGetDevice(int* d) { *d = 0; return OK; }
int cudaSetDevice(int d) { (void)d; return OK; }
int cudaDeviceGetAttribute(int* v, int a, int d) {
    (void)d;
    *v = a == 16 ? 152 : a == 81 ? 233472 : 0;   /* SMs; shared memory per SM */
    return OK;
}
/* every kernel has 6 KB of static shared memory, as the block kernels about have */
#define STATIC_SMEM 6144
#define CTA_SMEM (227 * 1024)
int cudaFuncGetAttributes(size_t* a, const void* f) { (void)f; a[0] = STATIC_SMEM; return OK; }
int cudaFuncSetAttribute(const void* f, int a, int v) {
    (void)f;
    return a == 8 && v + STATIC_SMEM > CTA_SMEM ? err(ERR_VALUE) : OK;   /* 8: dynamic shared memory */
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int threads, size_t smem) {
    (void)f;
    const int by_smem = (int)(233472 / (smem + STATIC_SMEM + 1024)), by_threads = 768 / threads;
    *n = by_smem < by_threads ? by_smem : by_threads;
    return OK;
}
int cudaGetLastError(void) { const int e = last_error; last_error = OK; return e; }
const char* cudaGetErrorString(int e) { return e == ERR_MEMORY ? "out of memory" : e ? "error" : "no error"; }
int cudaGetSymbolAddress(void** p, const void* s) { *p = (void*)s; return OK; }

int cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; *s = (void*)1; return OK; }
int cudaStreamDestroy(void* s) { (void)s; return OK; }
int cudaStreamSynchronize(void* s) { (void)s; return OK; }
int cudaEventCreate(void** e) { *e = (void*)1; return OK; }
int cudaEventDestroy(void* e) { (void)e; return OK; }
int cudaEventRecord(void* e, void* s) { (void)e; (void)s; return OK; }
int cudaEventSynchronize(void* e) { (void)e; return OK; }
/* timing number fast_at is the shortest; the others are the same */
static long fast_at, timings;
void fake_fastest(long n) { fast_at = n; timings = 0; }
long fake_timings(void) { return timings; }
int cudaEventElapsedTime(float* ms, void* a, void* b) {
    (void)a; (void)b;
    *ms = ++timings == fast_at ? 1.0f : 2.0f;
    return OK;
}

#define UNSUPPORTED(name) int name(void) { return err(ERR_UNSUPPORTED); }
UNSUPPORTED(cudaGraphDestroy) UNSUPPORTED(cudaGraphExecDestroy) UNSUPPORTED(cudaGraphExecKernelNodeSetParams)
UNSUPPORTED(cudaGraphInstantiate) UNSUPPORTED(cudaGraphKernelNodeGetParams) UNSUPPORTED(cudaGraphLaunch)
UNSUPPORTED(cudaGraphNodeGetType) UNSUPPORTED(cudaStreamBeginCapture) UNSUPPORTED(cudaStreamEndCapture)
UNSUPPORTED(cudaStreamGetCaptureInfo)

void** __cudaRegisterFatBinary(void* f) { static void* h; (void)f; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
char __cudaInitModule(void** h) { (void)h; return 1; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void** h, const char* f, char* n, const char* d, int t, void* a, void* b, void* c, void* e,
                            int* w) {
    (void)h; (void)f; (void)n; (void)d; (void)t; (void)a; (void)b; (void)c; (void)e; (void)w;
}
void __cudaRegisterVar(void** h, char* a, char* b, const char* n, int e, size_t s, int c, int g) {
    (void)h; (void)a; (void)b; (void)n; (void)e; (void)s; (void)c; (void)g;
}
static struct { dim3_t g, b; size_t smem; void* st; } pushed;
unsigned __cudaPushCallConfiguration(dim3_t g, dim3_t b, size_t smem, void* st) {
    pushed.g = g; pushed.b = b; pushed.smem = smem; pushed.st = st;
    return 0;
}
int __cudaPopCallConfiguration(dim3_t* g, dim3_t* b, size_t* smem, void** st) {
    *g = pushed.g; *b = pushed.b; *smem = pushed.smem; *st = pushed.st;
    return OK;
}
