/* A stand-in for the CUDA runtime's host functions, for tests without a GPU (loaded before
 * libcudart): device memory is host memory, copies are done at once, and copies, waits and
 * pointer queries are counted.  The device shares the host's page tables.  Kernels do not run. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

long fake_copies, fake_waits, fake_queries;
size_t fake_fail_bytes; /* a device allocation of this size fails */
int fake_attribute_sms = 152;

struct cudaPointerAttributes { int type, device; void *devicePointer, *hostPointer; long reserved[8]; };

int cudaGetDeviceCount(int *n) { *n = 1; return 0; }
int cudaSetDevice(int d) { (void)d; return 0; }
int cudaDeviceGetAttribute(int *v, int a, int d) { (void)d; *v = a == 16 ? fake_attribute_sms : 1; return 0; }
int cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -1; return 0; }
int cudaStreamCreateWithPriority(void **s, unsigned f, int p) { (void)f; (void)p; *s = malloc(1); return 0; }
int cudaStreamDestroy(void *s) { free(s); return 0; }
int cudaStreamSynchronize(void *s) { (void)s; fake_waits++; return 0; }
int cudaEventCreate(void **e) { *e = malloc(1); return 0; }
int cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; *e = malloc(1); return 0; }
int cudaEventDestroy(void *e) { free(e); return 0; }
int cudaMalloc(void **p, size_t n) {
    *p = NULL;
    if (n == fake_fail_bytes) return 2;
    *p = malloc(n);
    return *p ? 0 : 2;
}
int cudaFree(void *p) { free(p); return 0; }
int cudaMallocHost(void **p, size_t n) { *p = malloc(n); return *p ? 0 : 2; }
int cudaFreeHost(void *p) { free(p); return 0; }
int cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return 0; }
int cudaMemsetAsync(void *p, int v, size_t n, void *s) { (void)s; memset(p, v, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st) {
    (void)kind; (void)st;
    memcpy(d, s, n);
    fake_copies++;
    return 0;
}
int cudaGetLastError(void) { return 0; }
int cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) { /* ordinary memory */
    (void)p;
    fake_queries++;
    a->type = 0;
    a->device = -2;
    a->devicePointer = a->hostPointer = NULL;
    return 0;
}
