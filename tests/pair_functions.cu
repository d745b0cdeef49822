// The pair arithmetic's reciprocal square root and reciprocal beside CUDA's own
// (tests/test_gpu_pair_functions.py): out[0..3][n].
#include "fj_bs.cuh"

namespace {
__global__ void functions(const double* x, int64_t n, double* out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        out[i] = fj::rsqrt_normal(x[i]);
        out[n + i] = rsqrt(x[i]);
        out[2 * n + i] = fj::rcp_normal(x[i]);
        out[3 * n + i] = 1.0 / x[i];
    }
}
}  // namespace

extern "C" __attribute__((visibility("default"))) int pair_functions(const double* x, int64_t n, double* out, void* s) {
    functions<<<592, 256, 0, (cudaStream_t)s>>>(x, n, out);
    return (int)cudaGetLastError();
}
