// Preloaded stand-in for cudaLaunchCooperativeKernel: refuses launches of at least
// REFUSE_COOP threads a block as too large to be resident, as the runtime does in
// a context with part of the device's SMs; passes the others on.
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>

typedef struct {
    unsigned x, y, z;
} dim3;
typedef int (*launch_fn)(const void*, dim3, dim3, void**, size_t, void*);

int cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem, void* stream) {
    const char* min = getenv("REFUSE_COOP");
    if (min && block.x >= (unsigned)atoi(min)) return 720;  // cudaErrorCooperativeLaunchTooLarge
    void* rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    launch_fn real = rt ? (launch_fn)dlsym(rt, "cudaLaunchCooperativeKernel") : 0;
    return real ? real(f, grid, block, args, smem, stream) : 999;
}
