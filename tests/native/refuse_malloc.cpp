// A stand-in for cudaMalloc, preloaded: refuses the allocations of `refuse_from` bytes and more (0: none), as a
// full device does, and passes the others on.
#include <cstddef>
#include <dlfcn.h>

extern "C" {
size_t refuse_from = 0;
int refused = 0;
int cudaMalloc(void** p, size_t bytes) {
    using Fn = int (*)(void**, size_t);
    static Fn real = nullptr;
    if (!real) {
        void* lib = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
        if (lib) real = reinterpret_cast<Fn>(dlsym(lib, "cudaMalloc"));
    }
    if (!real || (refuse_from && bytes >= refuse_from)) {
        ++refused;
        *p = nullptr;
        return 2;   // cudaErrorMemoryAllocation
    }
    return real(p, bytes);
}
}
