// Compiled before csrc/el_advect.cu (nvcc -include) for tests/test_gpu_tile_failures.py: the tiled
// kernels' set-up fails on request, by a real refusal of the runtime (a shared-memory size no
// device has), and their wait for box copies reports on request that it gave up, after the copies
// have landed.
#pragma once
#include <cuda_runtime.h>

#define EL_TEST_API extern "C" __attribute__((visibility("default")))

EL_TEST_API int el_test_setup_fails;
int el_test_setup_fails = 0;

template <typename F>
static cudaError_t el_test_set_attribute(F* f, cudaFuncAttribute a, int v) {
    return cudaFuncSetAttribute(f, a, el_test_setup_fails ? 1 << 30 : v);
}
#define cudaFuncSetAttribute el_test_set_attribute

#define mbar_wait mbar_wait_real
#include "el_tma.cuh"
#undef mbar_wait

namespace el {
__device__ int test_wait_fails;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    const bool ok = mbar_wait_real(bar, parity);
    return ok && test_wait_fails == 0;
}
}  // namespace el

EL_TEST_API int el_test_set_wait_fails(int v) {
    return cudaMemcpyToSymbol(el::test_wait_fails, &v, sizeof(v)) == cudaSuccess ? 0 : 1;
}
