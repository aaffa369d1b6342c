/* A CUDA runtime that computes nothing, for tests of the library's host code without a GPU:
 * launches and copies do nothing (no host variable is written: results read back keep the
 * zeros they were declared with), allocations succeed up to a limit that the test sets. */
#include <stdlib.h>
#include <string.h>

typedef struct { size_t limit, largest, watch; long nulls; void *watched; } fake_t;
fake_t fake = {(size_t)-1, 0, 0, 0, NULL};
/* allocations of more bytes than limit fail */
void fake_limit(size_t limit) { fake.limit = limit; }
/* largest allocation asked for, and copies from or to a null pointer, since the last call */
size_t fake_largest(void) { size_t v = fake.largest; fake.largest = 0; return v; }
long fake_nulls(void) { long v = fake.nulls; fake.nulls = 0; return v; }
/* keep what the next copies of exactly so many bytes are given, and return the last one */
void fake_watch(size_t bytes) { fake.watch = bytes; free(fake.watched); fake.watched = NULL; }
void *fake_watched(void) { return fake.watched; }

#define OK(name) int name(void) { return 0; }
OK(__cudaPopCallConfiguration) OK(__cudaPushCallConfiguration) OK(__cudaRegisterFatBinaryEnd)
OK(__cudaRegisterFunction) OK(__cudaRegisterVar) OK(__cudaUnregisterFatBinary) OK(cudaLaunchKernel)
OK(cudaEventCreate) OK(cudaEventDestroy) OK(cudaEventRecord) OK(cudaStreamDestroy) OK(cudaStreamSynchronize)
OK(cudaStreamWaitEvent) OK(cudaGetLastError) OK(cudaFuncSetAttribute) OK(cudaMemset2DAsync) OK(cudaMemsetAsync)
OK(cudaGraphDebugDotPrint) OK(cudaGraphDestroy) OK(cudaGraphExecDestroy) OK(cudaGraphInstantiate)
OK(cudaGraphLaunch) OK(cudaStreamBeginCapture) OK(cudaStreamEndCapture)
void **__cudaRegisterFatBinary(void *p) { static void *h; (void)p; return &h; }
int cudaDeviceGetAttribute(int *v, int attr, int dev) {
    (void)dev;
    *v = attr == 16 ? 148 : attr == 97 ? 232448 : 1; /* SMs; opt-in shared memory per block */
    return 0;
}
int cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a; (void)b; *ms = 0; return 0; }
int cudaFree(void *p) { free(p); return 0; }
int cudaFuncGetAttributes(void *a, const void *f) { (void)f; memset(a, 0, 56); return 0; }
int cudaGetDevice(int *dev) { *dev = 0; return 0; }
static int encode(void) { return 0; }
int cudaGetDriverEntryPoint(const char *s, void **f, unsigned long long flags, int *status) {
    (void)s; (void)flags;
    *f = (void *)encode;
    if (status) *status = 0;
    return 0;
}
const char *cudaGetErrorString(int e) { (void)e; return "fake"; }
int cudaGetSymbolAddress(void **p, const void *s) { static char b[256]; (void)s; *p = b; return 0; }
int cudaMalloc(void **p, size_t n) {
    if (n > fake.largest) fake.largest = n;
    if (n > fake.limit) return 2;
    *p = malloc(16);
    return 0;
}
static int copy(const void *d, const void *s, size_t n, int kind) {
    if (!d || !s) fake.nulls++;
    if (n == fake.watch && n && kind == 1) { /* from the host */
        free(fake.watched);
        fake.watched = memcpy(malloc(n), s, n);
    }
    return 0;
}
int cudaMemcpy(void *d, const void *s, size_t n, int k) { return copy(d, s, n, k); }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { (void)st; return copy(d, s, n, k); }
int cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, int k, void *st) {
    (void)dp; (void)sp; (void)w; (void)h; (void)st;
    return copy(d, s, 0, k);
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl) {
    (void)f; (void)b; (void)s; (void)fl;
    *n = 2;
    return 0;
}
int cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; *s = malloc(16); return 0; }
