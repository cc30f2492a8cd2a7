/* A CUDA runtime of two pretended devices in host memory, preloaded before
 * the real one, for the host-side calls that need no kernel to run.  It keeps
 * one rule of the real runtime: a kernel launch into a stream of another
 * device than the calling thread's current one is refused, a memset or copy
 * is not. */
#include <stdlib.h>
#include <string.h>

typedef int err;
struct stream {
    int device;
};
static __thread int current;
static __thread err last;

err cudaGetDeviceCount(int *n) { return *n = 2, 0; }
err cudaSetDevice(int d) { return d < 0 || d > 1 ? 101 : (current = d, 0); }
err cudaGetDevice(int *d) { return *d = current, 0; }
err cudaGetLastError(void) {
    const err e = last;
    return last = 0, e;
}
err cudaPeekAtLastError(void) { return last; }
const char *cudaGetErrorString(err e) { return e ? "refused" : "ok"; }
err cudaMalloc(void **p, size_t n) { return (*p = malloc(n)) ? 0 : 2; }
err cudaHostAlloc(void **p, size_t n, unsigned f) { return (void)f, (*p = malloc(n)) ? 0 : 2; }
err cudaFree(void *p) { return free(p), 0; }
err cudaFreeHost(void *p) { return free(p), 0; }
err cudaStreamCreateWithFlags(struct stream **s, unsigned f) {
    (void)f;
    *s = malloc(sizeof **s);
    return (*s)->device = current, 0;
}
err cudaStreamDestroy(struct stream *s) { return free(s), 0; }
err cudaStreamSynchronize(struct stream *s) { return (void)s, 0; }
err cudaEventCreate(void **e) { return *e = malloc(1), 0; }
err cudaEventDestroy(void *e) { return free(e), 0; }
err cudaMemsetAsync(void *p, int v, size_t n, struct stream *s) { return (void)s, memset(p, v, n), 0; }
err cudaMemcpyAsync(void *d, const void *a, size_t n, int k, struct stream *s) {
    return (void)k, (void)s, memcpy(d, a, n), 0;
}
struct dim3 {
    unsigned x, y, z;
};
err cudaLaunchKernel(const void *f, struct dim3 g, struct dim3 b, void **args, size_t smem, struct stream *s) {
    (void)f, (void)g, (void)b, (void)args, (void)smem;
    return last = s && s->device != current ? 400 : 0;
}
