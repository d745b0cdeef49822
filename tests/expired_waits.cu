// What fj_panel.cu takes from the rest of the library, and its entry points, for a
// build in which every wait expires (tests/test_gpu_expired_waits.py).
#include "fj_panel.cuh"

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
