/* Preloaded before libcudart: device allocations of exactly one of the sizes in
 * MSET_DENY_BYTES (decimal, each followed by a comma) fail as if no memory were
 * left; every other call goes through. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

int cudaMalloc(void **p, size_t n) {
    static int (*real)(void **, size_t);
    for (const char *d = getenv("MSET_DENY_BYTES"); d && *d; d = strchr(d, ',') + 1)
        if (n == strtoull(d, NULL, 10)) {
            *p = NULL;
            return 2; /* cudaErrorMemoryAllocation */
        }
    /* (the library and its runtime are loaded into a scope of their own) */
    if (!real) real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaMalloc");
    return real(p, n);
}
