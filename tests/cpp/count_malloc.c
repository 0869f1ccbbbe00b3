// Preloaded stand-in for cudaMalloc that counts the calls it passes on.
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

static int calls;

int malloc_calls(void) { return calls; }

int cudaMalloc(void** p, size_t n) {
    void* rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    int (*real)(void**, size_t) = rt ? (int (*)(void**, size_t))dlsym(rt, "cudaMalloc") : 0;
    ++calls;
    return real ? real(p, n) : 999;
}
