// What fj_panel.cu and fj_trsv.cu take from the rest of the library, and their entry points, for a
// build in which every wait expires (tests/test_gpu_expired_waits.py).
#include "fj_panel.cuh"
#include "fj_trsv.cuh"

namespace fj {
int fail(int code, const char*, ...) { return code; }
void note_launch(int) {}
int allow_dynamic_smem(const void* f, size_t bytes) {
    return cuda_status(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), "");
}
}  // namespace fj

#define EXPORT extern "C" __attribute__((visibility("default")))
EXPORT int panel64(double* a, int n, int kb, int32_t* piv, int* info, cudaStream_t s) {
    return fj::panel_factor<double>(a, n, 0, kb, piv, info, nullptr, s);
}
EXPORT int panel32(float* a, int n, int kb, int32_t* piv, int* info, cudaStream_t s) {
    return fj::panel_factor<float>(a, n, 0, kb, piv, info, nullptr, s);
}
EXPORT int solve(const double* lu, int n, const int32_t* piv, double* b, double* work, int transposed, cudaStream_t s) {
    return fj::lu_substitute64(lu, n, piv, b, work, transposed != 0, s);
}
