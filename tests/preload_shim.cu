// The context's kernel settings with the runtime call replaced by one that
// fails where it is told to, for the CPU test (tests/test_preload.py).
#include <cuda_runtime.h>

static int g_calls, g_fail;
template <typename K>
static cudaError_t fake_set_attribute(K, cudaFuncAttribute, int) {
    return ++g_calls == g_fail ? cudaErrorInvalidValue : cudaSuccess;
}
#define cudaFuncSetAttribute fake_set_attribute
#include "../pdf-raster_b200/csrc/rrb_backend.cu"

// Fails call `fail` (0: none); the number of calls in *calls.
extern "C" int pl_preload(int fail, int* calls) {
    g_calls = 0;
    g_fail = fail;
    const cudaError_t e = preload_trial_kernels();
    *calls = g_calls;
    return static_cast<int>(e);
}
