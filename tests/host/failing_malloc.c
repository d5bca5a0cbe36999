/* Preloaded where the CUDA runtime is the shared library LIBCUDART: the k-th cudaMalloc from now on finds no memory
 * (it asks the driver for 2^50 bytes, so that the error is a real one in every respect).
 * It also adds up what was asked for. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

static long countdown = 0, asked = 0;

void fail_allocation(long k) { countdown = k; }
long allocations_to_go(void) { return countdown; }
long bytes_asked(void) { return asked; }

int cudaMalloc(void** p, size_t n) {
    static int (*real)(void**, size_t) = 0;
    if (!real) {
        /* The runtime came in with a library opened locally: it is in no scope that RTLD_NEXT sees. */
        void* runtime = dlopen(LIBCUDART, RTLD_LAZY | RTLD_NOLOAD);
        if (runtime) real = (int (*)(void**, size_t))dlsym(runtime, "cudaMalloc");
        if (!real) return 999; /* cudaErrorUnknown */
    }
    asked += (long)n;
    if (countdown > 0 && --countdown == 0) n = (size_t)1 << 50;
    return real(p, n);
}
