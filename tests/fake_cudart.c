/* A CUDA runtime for the CPU, preloaded under liblambda_b200.so: device memory is host
 * memory, kernels do nothing, and every call that allocates, frees, copies, launches or
 * waits is counted. A chosen allocation or launch can be made to fail, as the runtime's
 * does: the call returns the error and leaves it for cudaGetLastError. */
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

#include "driver_types.h"

enum { MALLOC, FREE, HOST_ALLOC, COPY_IN, LAUNCH, SYNC, COUNTERS };
static long counts[COUNTERS];
static long fail_malloc, fail_launch; /* fail the k-th from now on; 0: none */
static cudaError_t pending;
static long copies_waited_for; /* 0 while a copy from host memory may still run */

long fake_count(int what) { return counts[what]; }
void fake_reset(void) { memset(counts, 0, sizeof counts); }
void fake_fail_malloc(long k) { fail_malloc = k; }
void fake_fail_launch(long k) { fail_launch = k; }
int fake_pending(void) { return pending; }
int fake_copies_waited_for(void) { return (int)copies_waited_for; }

static cudaError_t failed(cudaError_t e) {
    pending = e;
    return e;
}
static void *handle(void) { return malloc(1); }

cudaError_t cudaMalloc(void **p, size_t n) {
    counts[MALLOC]++;
    if (fail_malloc && --fail_malloc == 0) return failed(cudaErrorMemoryAllocation);
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    counts[FREE]++;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned flags) {
    (void)flags;
    counts[HOST_ALLOC]++;
    if (fail_malloc && --fail_malloc == 0) return failed(cudaErrorMemoryAllocation);
    *p = calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned flags) {
    (void)flags;
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) {
    (void)k;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)st;
    if (k == cudaMemcpyHostToDevice) {
        counts[COPY_IN]++;
        copies_waited_for = 0;
    }
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    (void)st;
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    (void)s;
    counts[SYNC]++;
    copies_waited_for = 1;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s) {
    (void)f, (void)g, (void)b, (void)a, (void)m, (void)s;
    counts[LAUNCH]++;
    if (fail_launch && --fail_launch == 0) return failed(cudaErrorLaunchOutOfResources);
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void *s) {
    (void)g, (void)b, (void)m, (void)s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
    g->x = g->y = g->z = b->x = b->y = b->z = 1;
    *m = 0;
    *(void **)s = NULL;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    cudaError_t e = pending;
    pending = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError(void) { return pending; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    (void)p;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return (void)d, cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp *p, int d) {
    (void)d;
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
    (void)d;
    switch (a) {
        case cudaDevAttrMaxRegistersPerMultiprocessor: *v = 65536; break;
        case cudaDevAttrMaxThreadsPerMultiProcessor: *v = 2048; break;
        case cudaDevAttrMaxBlocksPerMultiprocessor: *v = 32; break;
        case cudaDevAttrReservedSharedMemoryPerBlock: *v = 1024; break;
        case cudaDevAttrMaxSharedMemoryPerMultiprocessor: *v = 233472; break;
        default: *v = 232448;
    }
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *f) {
    (void)f;
    memset(a, 0, sizeof *a);
    a->numRegs = 64;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
    (void)f, (void)a, (void)v;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = handle(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { return (void)f, *e = handle(), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return (void)e, (void)s, cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { return (void)a, (void)b, *ms = 0, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { return (void)f, *s = handle(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t s) { return (void)s, cudaSuccess; }
