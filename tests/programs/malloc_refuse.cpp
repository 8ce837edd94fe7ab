// Preloaded by tests/test_gpu_slot_memory.py: cudaMalloc of the byte counts
// that were named fails with cudaErrorMemoryAllocation, as on a device whose
// free memory is in smaller pieces; every other call goes to the runtime.
// Test infrastructure.
#include <dlfcn.h>

#include <cstddef>

static size_t named[8];
static int count = 0, refused = 0;

extern "C" void refuse(size_t bytes) { named[count++ & 7] = bytes; }
extern "C" int refuse_none() {   // and how many calls were refused so far
    for (size_t& b : named) b = 0;
    return refused;
}

extern "C" int cudaMalloc(void** p, size_t bytes) {
    using Fn = int (*)(void**, size_t);
    static const Fn real = (Fn)dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMalloc");
    for (size_t b : named)
        if (b && b == bytes) {
            refused++;
            return 2;   // cudaErrorMemoryAllocation
        }
    return real(p, bytes);
}
