// A stand-in for a second GPU, preloaded before the CUDA runtime: devices 0 and 1
// are both the one GPU, and every attribute that is set on a function is printed
// with the device that was current.
#include <dlfcn.h>

#include <cstdio>

#include <cuda_runtime_api.h>

static thread_local int current = 0;

template <class F>
static F real(const char* name, F) {
    return reinterpret_cast<F>(dlsym(RTLD_NEXT, name));
}
#define REAL(f) real(#f, f)

extern "C" {

cudaError_t cudaGetDeviceCount(int* count) {
    *count = 2;
    return cudaSuccess;
}

cudaError_t cudaGetDevice(int* device) {
    *device = current;
    return cudaSuccess;
}

cudaError_t cudaSetDevice(int device) {
    current = device;
    static const auto f = REAL(cudaSetDevice);
    return f(0);
}

cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr attr, int) {
    static const auto f = REAL(cudaDeviceGetAttribute);
    return f(value, attr, 0);
}

cudaError_t cudaFuncSetAttribute(const void* func, cudaFuncAttribute attr, int value) {
    if (attr == cudaFuncAttributeNonPortableClusterSizeAllowed)
        printf("device %d cluster %d\n", current, value);
    fflush(stdout);
    static const auto f = REAL(cudaFuncSetAttribute);
    return f(func, attr, value);
}

}  // extern "C"
