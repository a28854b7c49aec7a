/* A CUDA runtime for tests without a GPU: loaded in front of libcudart, it backs
 * device memory with host memory, runs no kernel and keeps account of both.
 * Frees on a stream with a kernel in flight are pending until the stream is
 * synchronised or allocates again, as in a stream-ordered memory pool. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define MAXB 4096
static struct { void* p; size_t n; void* pending_on; int live; } blk[MAXB];
static int nblk, fail_in = -1, busy[64], nstream = 1;
static long long launches, total, peak;

/* controls of the tests */
void fake_fail_alloc(int after) { fail_in = after; } /* the allocation after `after` more fails once; -1 none */
long long fake_launches(void) { return launches; }
long long fake_peak(void) { return peak; }
void fake_reset_peak(void) { peak = total; }

static void settle(void* st) {
    for (int i = 0; i < nblk; ++i)
        if (blk[i].p && !blk[i].live && blk[i].pending_on == st) {
            total -= (long long)blk[i].n;
            free(blk[i].p);
            blk[i].p = NULL;
        }
}
static int get(void** p, size_t n) {
    if (fail_in >= 0 && fail_in-- == 0) return 2; /* cudaErrorMemoryAllocation */
    int i = 0;
    while (i < nblk && blk[i].p) ++i;
    if (i == MAXB) return 2;
    if (i == nblk) ++nblk;
    blk[i].p = *p = calloc(1, n ? n : 1);
    blk[i].n = n;
    blk[i].live = 1;
    total += (long long)n;
    if (total > peak) peak = total;
    return 0;
}
static void put(void* p, void* st, int now) {
    for (int i = 0; p && i < nblk; ++i)
        if (blk[i].p == p) {
            blk[i].live = 0;
            blk[i].pending_on = st;
            if (now) {
                total -= (long long)blk[i].n;
                free(p);
                blk[i].p = NULL;
            }
            return;
        }
}
static int ran(void* st) {
    ++launches;
    busy[(uintptr_t)st & 63] = 1;
    return 0;
}

int cudaMalloc(void** p, size_t n) { return get(p, n); }
int cudaFree(void* p) { put(p, 0, 1); return 0; }
int cudaMallocFromPoolAsync(void** p, size_t n, void* pool, void* st) { (void)pool; settle(st); return get(p, n); }
int cudaFreeAsync(void* p, void* st) { put(p, st, !busy[(uintptr_t)st & 63]); return 0; }
int cudaMemPoolCreate(void** pool, const void* props) { (void)props; *pool = &nblk; return 0; }
int cudaMemPoolDestroy(void* pool) { (void)pool; return 0; }
int cudaMemPoolSetAttribute(void* pool, int a, void* v) { (void)pool; (void)a; (void)v; return 0; }
int cudaMemPoolTrimTo(void* pool, size_t n) { (void)pool; (void)n; return 0; }
int cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 34; return 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int k) { (void)k; memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { (void)k; (void)st; memcpy(d, s, n); return 0; }
int cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return 0; }
int cudaMemsetAsync(void* d, int v, size_t n, void* st) { (void)st; memset(d, v, n); return 0; }
int cudaStreamCreateWithFlags(void** st, unsigned f) { (void)f; *st = (void*)(uintptr_t)(nstream++ & 63); return 0; }
int cudaStreamDestroy(void* st) { (void)st; return 0; }
int cudaStreamSynchronize(void* st) { busy[(uintptr_t)st & 63] = 0; settle(st); return 0; }
int cudaStreamIsCapturing(void* st, int* c) { (void)st; *c = 0; return 0; }
int cudaStreamWaitEvent(void* st, void* e, unsigned f) { (void)st; (void)e; (void)f; return 0; }
int cudaEventCreate(void** e) { *e = &launches; return 0; }
int cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; *e = &launches; return 0; }
int cudaEventDestroy(void* e) { (void)e; return 0; }
int cudaEventRecord(void* e, void* st) { (void)e; (void)st; return 0; }
int cudaEventSynchronize(void* e) { (void)e; return 0; }
int cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a; (void)b; *ms = 1.0f; return 0; }
int cudaGetLastError(void) { return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaSetDevice(int d) { (void)d; return 0; }
int cudaDeviceGetAttribute(int* v, int a, int d) { (void)a; (void)d; *v = 148; return 0; }
int cudaFuncSetAttribute(const void* f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned g) {
    (void)f; (void)b; (void)s; (void)g;
    *n = 1;
    return 0;
}
struct config { unsigned grid[3], block[3]; size_t smem; void* stream; };
int cudaLaunchKernelExC(const struct config* c, const void* f, void** a) { (void)f; (void)a; return ran(c->stream); }
struct dim { unsigned x, y, z; };
int cudaLaunchKernel(const void* f, struct dim g, struct dim b, void** a, size_t s, void* st) {
    (void)f; (void)g; (void)b; (void)a; (void)s;
    return ran(st);
}
